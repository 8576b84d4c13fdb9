// Gridding (spreading) and degridding (interpolation) with the ES kernel.
//
// Reference: conv_3d_outputdriven_t1 (conv.cu:522-627) -- one thread per grid
// cell tests every point of 9 neighbouring 8x8 hives and evaluates the
// kernel per (cell, point) pair -- and interp_3d_nputsdriven
// (interp.cu:132-210) -- one thread per unsorted point, W^3 gathers.  Both
// compute the periodic 3-D convolution
//   fw[p][g1][g0] = sum_j c_j phi(g0 - X0_j) phi(g1 - X1_j) phi(p - X2_j)
// with phi(d) = exp(beta sqrt(1 - c d^2)) for |d| < W/2.
//
// Method "tiled" (default): gridding by cg_grid_own.cu; degridding here (and in
// cg_degrid_tma.cu): the grid is cut into tiles of TX x TY cells times batches of
// PB planes, handed out by a work queue to persistent CTAs. A CTA stages its tile
// plus the kernel halo (wrapped) in shared memory and interpolates each row of
// its own hives once.
// Method "direct": input-driven over the sorted stream with global atomics /
// global gathers (kept as a cross-check).
#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "cg_coords.cuh"
#include "cg_launch.cuh"
#include "cg_plan.cuh"
#include "cg_tiles.cuh"

namespace cg {

// ======================================================================= direct
template <typename T, int W>
__global__ void __launch_bounds__(256) k_grid_direct(const Rec<T>* __restrict__ recs, int64_t M,
                                                     Geom g, T* __restrict__ fw) {
  const T beta = (T)g.beta, c = (T)g.es_c;
  const T* __restrict__ poly = geom_poly<T>(g);
  const int nf1 = g.nf1, nf2 = g.nf2, nw = g.nw;
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < M;
       s += (int64_t)gridDim.x * blockDim.x) {
    const Rec<T> r = recs[s];
    T kx[W], ky[W], kz[W];
    const int bx = (int)(r.bxy & 0xFFFFu), by = (int)(r.bxy >> 16), bz = (int)r.bz;
    if (bx >= nf1 || by >= nf2 || bz >= nw) continue;  // cells always in range; never indexes wild
    const int ox = bx + taps<T, W>(r.f[0], beta, c, poly, kx);
    const int oy = by + taps<T, W>(r.f[1], beta, c, poly, ky);
    const int oz = bz + taps<T, W>(r.f[2], beta, c, poly, kz);
#pragma unroll 1
    for (int a = 0; a < W; a++) {
      const int zz = wrapi(oz + a, nw);
      const T cr = r.c[0] * kz[a], ci = r.c[1] * kz[a];
#pragma unroll 1
      for (int b = 0; b < W; b++) {
        const int yy = wrapi(oy + b, nf2);
        const T vr = cr * ky[b], vi = ci * ky[b];
        T* row = fw + 2 * (((size_t)zz * nf2 + yy) * nf1);
#pragma unroll
        for (int e = 0; e < W; e++) {
          const int xx = wrapi(ox + e, nf1);
          atomicAdd(row + 2 * xx, vr * kx[e]);
          atomicAdd(row + 2 * xx + 1, vi * kx[e]);
        }
      }
    }
  }
}

template <typename T, int W>
__global__ void __launch_bounds__(256) k_degrid_direct(const Rec<T>* __restrict__ recs,
                                                       const int* __restrict__ perm, int64_t M,
                                                       Geom g, const T* __restrict__ fw,
                                                       T* __restrict__ vis) {
  const T beta = (T)g.beta, c = (T)g.es_c;
  const T* __restrict__ poly = geom_poly<T>(g);
  const int nf1 = g.nf1, nf2 = g.nf2, nw = g.nw;
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < M;
       s += (int64_t)gridDim.x * blockDim.x) {
    const Rec<T> r = recs[s];
    T kx[W], ky[W], kz[W];
    const int bx = (int)(r.bxy & 0xFFFFu), by = (int)(r.bxy >> 16), bz = (int)r.bz;
    if (bx >= nf1 || by >= nf2 || bz >= nw) continue;
    const int ox = bx + taps<T, W>(r.f[0], beta, c, poly, kx);
    const int oy = by + taps<T, W>(r.f[1], beta, c, poly, ky);
    const int oz = bz + taps<T, W>(r.f[2], beta, c, poly, kz);
    T sr = 0, si = 0;
#pragma unroll 1
    for (int a = 0; a < W; a++) {
      const int zz = wrapi(oz + a, nw);
      T pr = 0, pi = 0;
#pragma unroll 1
      for (int b = 0; b < W; b++) {
        const int yy = wrapi(oy + b, nf2);
        const T* row = fw + 2 * (((size_t)zz * nf2 + yy) * nf1);
        T qr = 0, qi = 0;
#pragma unroll
        for (int e = 0; e < W; e++) {
          const int xx = wrapi(ox + e, nf1);
          qr += row[2 * xx] * kx[e];
          qi += row[2 * xx + 1] * kx[e];
        }
        pr += qr * ky[b];
        pi += qi * ky[b];
      }
      sr += pr * kz[a];
      si += pi * kz[a];
    }
    const int64_t i = perm[s];
    if (i < 0 || i >= M) continue;
    vis[2 * i] = sr * r.c[0] - si * r.c[1];
    vis[2 * i + 1] = sr * r.c[1] + si * r.c[0];
  }
}

static int env_int(const char* name, int dflt) {
  const char* v = getenv(name);
  return v ? atoi(v) : dflt;
}

static int num_sms() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n = 148;
  }
  return n;
}


// ---------------------------------------------------------------- degridding
// One degridding tile (work item `item` of tiling tc), staged in `smem`; of its rows
// in order, share `chunk` of `nchunks` (kSplit); nothing of a whole tile with more than `heavy`,
// whose chunks are items of their own.  Called by every thread of the block with the same
// arguments.
template <typename T, int W, bool kSplit>
__device__ __forceinline__ void degrid_tile(const Rec<T>* __restrict__ recs,
                                            const int* __restrict__ perm,
                                            const int* __restrict__ hive_start, int64_t M,
                                            const Geom& g, const TileCfg& tc, int nslots_max,
                                            const T* __restrict__ fw, T* __restrict__ vis,
                                            int item, unsigned char* smem, int* s_warp, int chunk,
                                            int nchunks, int heavy) {
  constexpr int lo = Halo<W>::lo, hi = Halo<W>::hi;
  const int TX = tc.TX, TY = tc.TY, PB = tc.PB;
  const int nw = g.nw, nf1 = g.nf1, nf2 = g.nf2;
  const bool all_planes = (PB >= nw);
  const int SX = TX + lo + hi, SY = TY + lo + hi, SZ = all_planes ? nw : PB + lo + hi;
  const int SXP = SX + 1;  // padded row stride (complex elements)
  const int nstage = SX * SY * SZ;
  T* stg = (T*)smem;
  int* tb = (int*)(stg + 2 * (size_t)SXP * SY * SZ);
  const int ts = nslots_max + 1;
  SegTable t{tb, tb + ts, tb + 2 * ts};
  const T beta = (T)g.beta, c = (T)g.es_c;
  const T* __restrict__ poly = geom_poly<T>(g);
  const size_t plane = (size_t)nf1 * nf2;
  {
    const int tix = tc.bx0 + item % tc.ntx, tiy = tc.by0 + (item / tc.ntx) % tc.nty,
              tib = item / (tc.ntx * tc.nty);
    const int tx0 = tix * TX, ty0 = tiy * TY, p0 = all_planes ? 0 : tib * PB;
    const int tx1 = min(tx0 + TX, nf1), ty1 = min(ty0 + TY, nf2);
    const int p1 = all_planes ? nw : min(p0 + PB, nw);
    const int gx0 = tx0 - lo, gy0 = ty0 - lo, gz0 = all_planes ? 0 : p0 - lo;
    // runs of the tile's own hives (each row belongs to exactly one tile)
    const int nslots = build_segments(g, hive_start, tx0 >> 3, (tx1 - 1) >> 3, ty0 >> 3,
                                      (ty1 - 1) >> 3, p0, p1 - 1, t, s_warp);
    const int total = t.pref[nslots];
    if (total == 0 || (kSplit && nchunks == 1 && total > heavy)) return;  // uniform across the block
    int qb = 0, qe = total;
    if (kSplit && nchunks > 1) {
      qb = (int)((int64_t)total * chunk / nchunks);
      qe = (int)((int64_t)total * (chunk + 1) / nchunks);
    }
    // stage the tile + halo (periodic); row stride SXP = SX + 1 complex
    using V = typename std::conditional<sizeof(T) == 4, float2, double2>::type;
    V* stv = reinterpret_cast<V*>(stg);
    const V* fwv = reinterpret_cast<const V*>(fw);
    const TileDiv div_x(SX), div_xy(SX * SY);
    for (int i = threadIdx.x; i < nstage; i += blockDim.x) {
      const int sz = div_xy(i), r = i - sz * SX * SY, sy = div_x(r), sx = r - sy * SX;
      const int gx = modi(gx0 + sx, nf1), gy = modi(gy0 + sy, nf2), gz = modi(gz0 + sz, nw);
      stv[(sz * SY + sy) * SXP + sx] = fwv[(size_t)gz * plane + (size_t)gy * nf1 + gx];
    }
    __syncthreads();
    for (int q = qb + threadIdx.x; q < qe; q += blockDim.x) {
      const int sgi = find_segment(t.pref, nslots, q);
      const int sidx = t.start[sgi] + (q - t.pref[sgi]);
      const Rec<T> r = recs[sidx];
      const int bx = (int)(r.bxy & 0xFFFFu), by = (int)(r.bxy >> 16), bz = (int)r.bz;
      T kx[W], ky[W], kz[W];
      const int lx = bx + taps<T, W>(r.f[0], beta, c, poly, kx) - gx0;
      const int ly = by + taps<T, W>(r.f[1], beta, c, poly, ky) - gy0;
      const int lz = bz + taps<T, W>(r.f[2], beta, c, poly, kz) - gz0;
      if (lx < 0 || ly < 0 || lx + W > SX || ly + W > SY) continue;  // cannot happen: tile rows only
      T sr = 0, si = 0;
      for (int a = 0; a < W; a++) {
        int zz = lz + a;
        zz = all_planes ? wrapi(zz, nw) : min(max(zz, 0), SZ - 1);
        T pr = 0, pi = 0;
        for (int b = 0; b < W; b++) {
          const T* row = stg + 2 * ((zz * SY + (ly + b)) * SXP + lx);
          T qr = 0, qi = 0;
#pragma unroll
          for (int e = 0; e < W; e++) {
            qr += row[2 * e] * kx[e];
            qi += row[2 * e + 1] * kx[e];
          }
          pr += qr * ky[b];
          pi += qi * ky[b];
        }
        sr += pr * kz[a];
        si += pi * kz[a];
      }
      const int64_t i = perm[sidx];
      if (i < 0 || i >= M) continue;
      vis[2 * i] = sr * r.c[0] - si * r.c[1];
      vis[2 * i + 1] = sr * r.c[1] + si * r.c[0];
    }
    __syncthreads();
  }
}

// counter[0]: queue head; counter[1]: chunk slots.  Items: the chunk slots (kSplit), then
// the tiles.
template <typename T, int W, bool kSplit>
__global__ void __launch_bounds__(512) k_degrid_tiled(const Rec<T>* __restrict__ recs,
                                                      const int* __restrict__ perm,
                                                      const int* __restrict__ hive_start, int64_t M,
                                                      Geom g, TileCfg tc, int nslots_max,
                                                      const T* __restrict__ fw,
                                                      T* __restrict__ vis, int* __restrict__ counter,
                                                      DegridSplit sp) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_warp[33];
  __shared__ int s_item;
  const int nslot = kSplit ? counter[1] : 0;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(counter, 1);
    __syncthreads();
    int item = s_item;
    // a tile's first block-wide barrier orders this read before the next write of s_item
    DegridSlot sl{0, 0, 1};
    if (kSplit && item < nslot) {
      sl = sp.slots[item];
      item = sl.tile;
    } else {
      item -= nslot;
      if (item >= tc.nitems) break;
      const int row = item / tc.ntx, b = row / tc.nty;
      item += (b * tc.nty + center_out(row - b * tc.nty, tc.nty) - row) * tc.ntx;
    }
    degrid_tile<T, W, kSplit>(recs, perm, hive_start, M, g, tc, nslots_max, fw, vis, item, smem, s_warp, sl.chunk,
                              sl.nchunks, sp.heavy);
  }
}

// Many grids in one persistent launch: blocks take (job, tile) items from a
// global queue; every job shares W and the kernel, smem is the largest
// footprint of the jobs' tilings.
template <typename T, int W>
__global__ void __launch_bounds__(512, sizeof(T) == 4 ? 2 : 1) k_degrid_tiled_multi(const GridJob<T>* __restrict__ jobs,
                                                            int njobs, int nitems,
                                                            int* __restrict__ counter) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_warp[33];
  __shared__ int s_item;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(counter, 1);
    __syncthreads();
    const int item = s_item;
    if (item >= nitems) break;
    const int j = find_job(jobs, njobs, item, [](const GridJob<T>& x) { return x.degrid_item0; });
    const GridJob<T>& J = jobs[j];
    degrid_tile<T, W, false>(J.recs, J.perm, J.hive_start, J.M, J.g, J.dt, J.nslots, J.fw, J.vis,
                             item - J.degrid_item0, smem, s_warp, 0, 1, 0);
  }
}

// One warp per tile: its rows from the hive offsets, and slots for a heavy one.  counter[1]
// counts them: every row lies in one tile and heavy >= R, so 2 M / R hold all.
__global__ void __launch_bounds__(256) k_degrid_split(const int* __restrict__ hive_start, Geom g, TileCfg tc, int R,
                                                      int heavy, int cap, int* __restrict__ counter,
                                                      DegridSlot* __restrict__ slots) {
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (t >= tc.nitems) return;
  const int tx0 = (tc.bx0 + t % tc.ntx) * tc.TX, ty0 = (tc.by0 + (t / tc.ntx) % tc.nty) * tc.TY;
  const int p0 = t / (tc.ntx * tc.nty) * tc.PB, p1 = min(p0 + tc.PB, g.nw);
  const int hx0 = tx0 >> 3, hx1 = (min(tx0 + tc.TX, g.nf1) - 1) >> 3;
  const int hy0 = ty0 >> 3, ny = ((min(ty0 + tc.TY, g.nf2) - 1) >> 3) - hy0 + 1;
  int rows = 0;
  for (int r = lane; r < ny * (p1 - p0); r += 32) {
    const int64_t row = ((int64_t)(p0 + r / ny) * g.nhy + hy0 + r % ny) * g.nhx;
    rows += hive_start[row + hx1 + 1] - hive_start[row + hx0];
  }
  rows = __reduce_add_sync(0xffffffffu, rows);
  if (rows > heavy) {
    const int k = (rows + R - 1) / R;  // two at least
    int base = 0;
    if (lane == 0) base = atomicAdd(counter + 1, k);
    base = __shfl_sync(0xffffffffu, base, 0);
    for (int c = lane; c < k && base + c < cap; c += 32) slots[base + c] = DegridSlot{t, c, k};
  }
}

// ======================================================================= launch
// R: half a CTA's share of the rows, so that the last CTA ends soon after the others; at
// least 2048 rows, below which staging the tile once more is no longer small beside them.
// Tiles up to `share` times a CTA's rows stay whole: splitting them gives less than their
// repeated staging takes (TMA variant 2, W = 6, 10M rows around the centre of a 4096^2
// grid: 0.78 ms with no tile split, 0.93 with all above half a CTA's rows).
// Calls of fewer than 131072 rows are not split: the plan costs some 8 us (100k rows evenly
// over a 1024^2 grid 0.050 -> 0.065 ms; all of them in one tile take 0.31 ms, split 0.05).
// CG_SPLIT=0 turns the split off, CG_SPLIT_ROWS sets R.
int plan_degrid_split(const int* d_hive_start, const Geom& g, const TileCfg& tc, int64_t M, int blocks,
                      double share, cg_dev_buf* buf, int* d_counter, cudaStream_t st, DegridSplit* out) {
  *out = DegridSplit{};
  int64_t R = M < 131072 ? M : std::max<int64_t>(2048, M / (2 * (int64_t)std::max(1, blocks)));
  int64_t heavy = std::max<int64_t>(R, (int64_t)(share * (double)M / std::max(1, blocks)));
  if (const char* e = getenv("CG_SPLIT_ROWS")) heavy = R = std::max<int64_t>(1, atoll(e));
  const char* off = getenv("CG_SPLIT");
  const bool split = buf && M > heavy && !(off && atoi(off) == 0);
  CG_CUDA(cudaMemsetAsync(d_counter, 0, 2 * sizeof(int), st));
  if (!split) return CG_OK;
  const int cap = (int)std::min<int64_t>(2147483647, 2 * M / R + 1);
  CG_TRY(ensure(*buf, (size_t)cap * sizeof(DegridSlot)));
  out->slots = (const DegridSlot*)buf->p;
  out->heavy = (int)std::min<int64_t>(heavy, 2147483647);
  k_degrid_split<<<(tc.nitems + 7) / 8, 256, 0, st>>>(d_hive_start, g, tc, (int)R, out->heavy, cap, d_counter,
                                                      (DegridSlot*)buf->p);
  count_launches(1);
  CG_CUDA(cudaGetLastError());
  return CG_OK;
}

static int slots_for(int TY, int PB, int W) { return ((TY >> 3) + 2) * (PB + W + 1) * 3; }

constexpr size_t kDegridBytes = 220 * 1024;
template <typename T>
static size_t degrid_tile_bytes(const Geom& g, int tx, int ty, int pb) {
  const size_t cells = (size_t)(tx + g.kw + 1) * (ty + g.kw) * (pb >= g.nw ? g.nw : pb + g.kw);
  return cells * 2 * sizeof(T) + (size_t)(slots_for(ty, pb, g.kw) + 1) * 4 * kSegInts;
}
// all planes, or their number halved until a tile's batch fits
template <typename T>
static int degrid_planes(const Geom& g, int tx, int ty) {
  int pb = g.nw;
  while (pb > 1 && degrid_tile_bytes<T>(g, tx, ty, pb) > kDegridBytes) pb = (pb + 1) / 2;
  return pb;
}
// Few items of 32 x 16 cells (pb planes; 0: as many as fit): 16 x 8 instead, so that the
// data's tiles fill the SMs (FP64 512^2 x 12 grid, 98 tiles of 32 x 16: 0.165 -> 0.061 ms).
// With many the larger ones stay ahead (FP64 4096^2 x 20, W = 10: 5.9 against 6.5 ms; FP32
// 1024^2 x 190, 378 tiles times 8 plane batches: 0.71 against 0.93 ms).
template <typename T>
bool few_degrid_tiles(const Geom& g, int pb) {
  pb = pb > 0 ? std::min(pb, g.nw) : degrid_planes<T>(g, 32, 16);
  return (int64_t)(g.band_c1 / 32 - g.band_c0 / 32 + 1) * (g.band_r1 / 16 - g.band_r0 / 16 + 1) *
             ((g.nw + pb - 1) / pb) < 4 * num_sms();
}

// Tile shape of the tiled degridding: 32 x 16 cells by default, the plane batch covering all
// planes when the shared-memory footprint allows, otherwise halved until it fits.
// CG_TILE_X / CG_TILE_Y / CG_TILE_PLANES / CG_TILE_THREADS override (tuning).
template <typename T>
TileCfg degrid_tiling(const Geom& g, const TileTune* tt) {
  const size_t budget = kDegridBytes;
  const int W = g.kw;
  TileCfg tc{};
  // 32 x 16 tiles keep two CTAs per SM for FP32 at W <= 7 (one
  // stages its tile while the other interpolates); 32 x 32 left one CTA per SM
  int TX = env_int("CG_TILE_X", 32), TY = env_int("CG_TILE_Y", 16);
  int PB = env_int("CG_TILE_PLANES", 0);
  int threads = env_int("CG_TILE_THREADS", 512);
  if (tt) {
    if (tt->dx > 0) TX = tt->dx;
    if (tt->dy > 0) TY = tt->dy;
    if (tt->dpb > 0) PB = tt->dpb;
    if (tt->dthreads > 0) threads = tt->dthreads;
  }
  TX = std::max(8, (TX / 8) * 8);
  TY = std::max(8, (TY / 8) * 8);
  threads = std::min(512, std::max(64, (threads / 32) * 32));
  auto bytes = [&](int tx, int ty, int pb) { return degrid_tile_bytes<T>(g, tx, ty, pb); };
  if (!(tt && (tt->dx > 0 || tt->dy > 0)) && !getenv("CG_TILE_X") && !getenv("CG_TILE_Y") &&
      few_degrid_tiles<T>(g, PB)) {
    TX = 16;
    TY = 8;
  }
  if (PB <= 0) PB = degrid_planes<T>(g, TX, TY);
  if (PB > g.nw) PB = g.nw;
  // a staged plane batch must not wrap onto itself
  if (PB < g.nw && PB + W > g.nw) PB = g.nw;
  while (bytes(TX, TY, PB) > budget && (TX > 8 || TY > 8)) {
    if (TY >= TX) TY -= 8; else TX -= 8;
  }
  tc.TX = TX;
  tc.TY = TY;
  tc.PB = PB;
  tc.ntx = (g.nf1 + TX - 1) / TX;
  tc.nty = (g.nf2 + TY - 1) / TY;
  // only the tiles of the cells the data can reach (the full grid
  // when the data wraps around an edge); the others hold no rows
  if (0 <= g.band_c0 && g.band_c0 <= g.band_c1 && g.band_c1 < g.nf1) {
    tc.bx0 = g.band_c0 / TX;
    tc.ntx = g.band_c1 / TX - tc.bx0 + 1;
  }
  if (0 <= g.band_r0 && g.band_r0 <= g.band_r1 && g.band_r1 < g.nf2) {
    tc.by0 = g.band_r0 / TY;
    tc.nty = g.band_r1 / TY - tc.by0 + 1;
  }
  tc.npb = (g.nw + PB - 1) / PB;
  tc.nitems = tc.ntx * tc.nty * tc.npb;
  tc.threads = threads;
  tc.smem = bytes(TX, TY, PB);
  return tc;
}

int degrid_slots(const TileCfg& tc, int W) { return slots_for(tc.TY, tc.PB, W); }

// Autotuner candidates.  Gridding has one tiling (cg_grid_own.cu); its time is
// reported.  Degridding tiles (x, y, planes, threads per CTA); every tile that an
// untuned call can take (32 x 16 or, with few_degrid_tiles, 16 x 8, and the TMA variants
// 2 and 4) is among them, so that tuning is never slower than not tuning.
static const int kGridCand[][4] = {{16, 16, 0, 0}};
// threads -1 .. -4: the TMA-staged kernel's variants (all planes; 32 x 16
// tiles with 512 threads and two stages / 256 threads and one stage; 32 x 8
// and 16 x 8 tiles with 128 threads and one stage) where they apply.
static const int kDegridCand[][4] = {{32, 16, 0, 512}, {32, 32, 0, 512}, {32, 8, 0, 512},
                                     {16, 16, 0, 512}, {64, 16, 0, 512}, {32, 16, 0, 256},
                                     {16, 16, 0, 256}, {16, 8, 0, 512}, {32, 16, 8, 512}, {32, 16, 0, -1},
                                     {32, 16, 0, -2}, {32, 8, 0, -3}, {16, 8, 0, -4}};

int tile_candidates(int dir, const int (**cand)[4]) {
  if (dir == 0) {
    *cand = kGridCand;
    return (int)(sizeof(kGridCand) / sizeof(kGridCand[0]));
  }
  *cand = kDegridCand;
  return (int)(sizeof(kDegridCand) / sizeof(kDegridCand[0]));
}

void set_tile_candidate(TileTune& tt, int dir, const int* c) {
  if (dir == 0) {
    tt.wx = c[0]; tt.wy = c[1];
  } else {
    tt.dx = c[0]; tt.dy = c[1]; tt.dpb = c[2]; tt.dthreads = c[3];
  }
}

template <typename T, int W>
static int grid_direct_w(const Rec<T>* d_recs, int64_t M, const Geom& g, T* d_fw, cudaStream_t st) {
  size_t G = (size_t)g.nf1 * g.nf2 * g.nw;
  CG_CUDA(cudaMemsetAsync(d_fw, 0, G * 2 * sizeof(T), st));
  if (M == 0) return CG_OK;
  int blocks = (int)((M + 255) / 256);
  if (blocks > 148 * 64) blocks = 148 * 64;
  k_grid_direct<T, W><<<blocks, 256, 0, st>>>(d_recs, M, g, d_fw);
  count_launches(1);
  CG_CUDA(cudaGetLastError());
  return CG_OK;
}

template <typename T, int W>
static int degrid_w(const Rec<T>* d_recs, const int* d_perm, const int* d_hive_start, int64_t M,
                    const Geom& g, const T* d_fw, T* d_vis, int method, int* d_counter,
                    cudaStream_t st, const TileTune* tt, cg_dev_buf* split) {
  if (M == 0) return CG_OK;
  if (method == kGridDirect) {
    int blocks = (int)((M + 255) / 256);
    if (blocks > 148 * 64) blocks = 148 * 64;
    k_degrid_direct<T, W><<<blocks, 256, 0, st>>>(d_recs, d_perm, M, g, d_fw, d_vis);
    count_launches(1);
    CG_CUDA(cudaGetLastError());
    return CG_OK;
  }
  TileCfg tc = degrid_tiling<T>(g, tt);
  int nslots = slots_for(tc.TY, tc.PB, W);
  int per_sm = 0;
  CG_CUDA(kernel_occupancy((const void*)k_degrid_tiled<T, W, false>, tc.threads, tc.smem, &per_sm));
  if (per_sm < 1) {
    set_last_error("tiled degridding does not fit on an SM");
    return CG_ERR_ARG;
  }
  DegridSplit sp;
  CG_TRY(plan_degrid_split(d_hive_start, g, tc, M, per_sm * num_sms(), 0.5, split, d_counter, st, &sp));
  const int blocks = sp.slots ? per_sm * num_sms() : std::min(tc.nitems, per_sm * num_sms());
  auto* kern = k_degrid_tiled<T, W, false>;
  if (sp.slots) {
    kern = k_degrid_tiled<T, W, true>;
    CG_CUDA(kernel_occupancy((const void*)kern, tc.threads, tc.smem, &per_sm));
    if (per_sm < 1) return CG_ERR_ARG;
  }
  kern<<<blocks, tc.threads, tc.smem, st>>>(d_recs, d_perm, d_hive_start, M, g, tc, nslots, d_fw, d_vis, d_counter, sp);
  count_launches(1);
  CG_CUDA(cudaGetLastError());
  return CG_OK;
}

template <typename T>
int launch_grid(const Rec<T>* d_recs, const int* d_hive_start, int64_t M, const Geom& g, T* d_fw,
                int method, int* d_counter, cudaStream_t st, const SplitScratch* sp) {
  if (method == kGridMma) {
    // tensor-core path: FP32, ES kernel and W <= 8; everything else on the SIMT kernels
    if (sizeof(T) == 4 && !g.polyf) {
      int s = launch_grid_mma((const Rec<float>*)d_recs, d_hive_start, g, (float*)d_fw, st);
      if (s != CG_ERR_ARG) return s;
    }
    method = kGridTiled;
  }
  if (method == kGridTiled) return launch_grid_own<T>(d_recs, d_hive_start, M, g, d_fw, d_counter, st, sp);
#define CG_GRID_CALL(w) grid_direct_w<T, w>(d_recs, M, g, d_fw, st)
  CG_W_SWITCH(g.kw, CG_GRID_CALL)
#undef CG_GRID_CALL
}

template <typename T>
int launch_degrid(const Rec<T>* d_recs, const int* d_perm, const int* d_hive_start, int64_t M,
                  const Geom& g, const T* d_fw, T* d_vis, int method, int* d_counter,
                  cudaStream_t st, const TileTune* tt, cg_dev_buf* split) {
  if (method == kGridMma) method = kGridTiled;
#define CG_DEGRID_CALL(w) \
  degrid_w<T, w>(d_recs, d_perm, d_hive_start, M, g, d_fw, d_vis, method, d_counter, st, tt, split)
  CG_W_SWITCH(g.kw, CG_DEGRID_CALL)
#undef CG_DEGRID_CALL
}

// ================================================================== multi-grid
template <typename T>
int multi_shape(GridJob<T>* jobs, int njobs, MultiShape* sh) {
  if (njobs < 1) return CG_ERR_ARG;
  *sh = MultiShape{};
  sh->kw = jobs[0].g.kw;
  sh->poly = geom_poly_host<T>(jobs[0].g) != nullptr;
  sh->threads = jobs[0].dt.threads;
  int64_t gi = 0, di = 0;
  for (int j = 0; j < njobs; j++) {
    GridJob<T>& J = jobs[j];
    if (J.g.kw != sh->kw || (geom_poly_host<T>(J.g) != nullptr) != sh->poly ||
        J.dt.threads != sh->threads) {
      set_last_error("multi-grid jobs differ in kernel width, kernel or threads");
      return CG_ERR_ARG;
    }
    J.grid_item0 = (int)gi;
    J.degrid_item0 = (int)di;
    gi += J.wt.nitems;
    di += J.dt.nitems;
    sh->grid_slots = std::max(sh->grid_slots, J.wt.slots);
    sh->dsmem = std::max(sh->dsmem, J.dt.smem);
  }
  if (gi > 2147483647LL || di > 2147483647LL) return CG_ERR_SIZE;
  sh->grid_items = (int)gi;
  sh->degrid_items = (int)di;
  return CG_OK;
}

template <typename T, int W>
static int degrid_multi_w(const GridJob<T>* d_jobs, int njobs, const MultiShape& sh,
                          int* d_counter, cudaStream_t st) {
  int per_sm = 0;
  CG_CUDA(kernel_occupancy((const void*)k_degrid_tiled_multi<T, W>, sh.threads, sh.dsmem, &per_sm));
  if (per_sm < 1) {
    set_last_error("multi-grid degridding does not fit on an SM");
    return CG_ERR_ARG;
  }
  const int blocks = std::min(sh.degrid_items, per_sm * num_sms());
  CG_CUDA(cudaMemsetAsync(d_counter, 0, sizeof(int), st));
  k_degrid_tiled_multi<T, W><<<std::max(1, blocks), sh.threads, sh.dsmem, st>>>(
      d_jobs, njobs, sh.degrid_items, d_counter);
  count_launches(1);
  CG_CUDA(cudaGetLastError());
  return CG_OK;
}

template <typename T>
int launch_degrid_multi(const GridJob<T>* d_jobs, int njobs, const MultiShape& sh, int* d_counter,
                        cudaStream_t st) {
  if (njobs < 1 || sh.degrid_items < 1) return CG_OK;
#define CG_DEGRID_MULTI_CALL(w) degrid_multi_w<T, w>(d_jobs, njobs, sh, d_counter, st)
  CG_W_SWITCH(sh.kw, CG_DEGRID_MULTI_CALL)
#undef CG_DEGRID_MULTI_CALL
}

// ================================================================ plane windows
// Memory-limited mode: the grid holds only planes [p0, p1) (plane p at
// fwb + (p - p0) * plane).  Spreading skips taps outside the window; the
// interpolation adds each window's share of a row into vis, so a call
// visits every window once.  Sorted-stream order, one row per thread.
template <typename T, int W>
__global__ void __launch_bounds__(256) k_grid_window(const Rec<T>* __restrict__ recs, int64_t M,
                                                     Geom g, int p0, int p1, T* __restrict__ fwb) {
  const T beta = (T)g.beta, c = (T)g.es_c;
  const T* __restrict__ poly = geom_poly<T>(g);
  const int nf1 = g.nf1, nf2 = g.nf2, nw = g.nw;
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < M;
       s += (int64_t)gridDim.x * blockDim.x) {
    const Rec<T> r = recs[s];
    T kx[W], ky[W], kz[W];
    const int bx = (int)(r.bxy & 0xFFFFu), by = (int)(r.bxy >> 16), bz = (int)r.bz;
    if (bx >= nf1 || by >= nf2 || bz >= nw) continue;
    const int oz = bz + taps<T, W>(r.f[2], beta, c, poly, kz);
    bool any = false;
#pragma unroll
    for (int a = 0; a < W; a++) {
      const int zz = wrapi(oz + a, nw);
      any |= zz >= p0 && zz < p1;
    }
    if (!any) continue;
    const int ox = bx + taps<T, W>(r.f[0], beta, c, poly, kx);
    const int oy = by + taps<T, W>(r.f[1], beta, c, poly, ky);
#pragma unroll 1
    for (int a = 0; a < W; a++) {
      const int zz = wrapi(oz + a, nw);
      if (zz < p0 || zz >= p1) continue;
      const T cr = r.c[0] * kz[a], ci = r.c[1] * kz[a];
#pragma unroll 1
      for (int b = 0; b < W; b++) {
        const int yy = wrapi(oy + b, nf2);
        const T vr = cr * ky[b], vi = ci * ky[b];
        T* row = fwb + 2 * (((size_t)(zz - p0) * nf2 + yy) * nf1);
#pragma unroll
        for (int e = 0; e < W; e++) {
          const int xx = wrapi(ox + e, nf1);
          atomicAdd(row + 2 * xx, vr * kx[e]);
          atomicAdd(row + 2 * xx + 1, vi * kx[e]);
        }
      }
    }
  }
}

template <typename T, int W>
__global__ void __launch_bounds__(256) k_degrid_window(const Rec<T>* __restrict__ recs,
                                                       const int* __restrict__ perm, int64_t M,
                                                       Geom g, int p0, int p1,
                                                       const T* __restrict__ fwb,
                                                       T* __restrict__ vis) {
  const T beta = (T)g.beta, c = (T)g.es_c;
  const T* __restrict__ poly = geom_poly<T>(g);
  const int nf1 = g.nf1, nf2 = g.nf2, nw = g.nw;
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < M;
       s += (int64_t)gridDim.x * blockDim.x) {
    const Rec<T> r = recs[s];
    T kx[W], ky[W], kz[W];
    const int bx = (int)(r.bxy & 0xFFFFu), by = (int)(r.bxy >> 16), bz = (int)r.bz;
    if (bx >= nf1 || by >= nf2 || bz >= nw) continue;
    const int oz = bz + taps<T, W>(r.f[2], beta, c, poly, kz);
    bool any = false;
#pragma unroll
    for (int a = 0; a < W; a++) {
      const int zz = wrapi(oz + a, nw);
      any |= zz >= p0 && zz < p1;
    }
    if (!any) continue;
    const int ox = bx + taps<T, W>(r.f[0], beta, c, poly, kx);
    const int oy = by + taps<T, W>(r.f[1], beta, c, poly, ky);
    T sr = 0, si = 0;
#pragma unroll 1
    for (int a = 0; a < W; a++) {
      const int zz = wrapi(oz + a, nw);
      if (zz < p0 || zz >= p1) continue;
      T pr = 0, pi = 0;
#pragma unroll 1
      for (int b = 0; b < W; b++) {
        const int yy = wrapi(oy + b, nf2);
        const T* row = fwb + 2 * (((size_t)(zz - p0) * nf2 + yy) * nf1);
        T qr = 0, qi = 0;
#pragma unroll
        for (int e = 0; e < W; e++) {
          const int xx = wrapi(ox + e, nf1);
          qr += row[2 * xx] * kx[e];
          qi += row[2 * xx + 1] * kx[e];
        }
        pr += qr * ky[b];
        pi += qi * ky[b];
      }
      sr += pr * kz[a];
      si += pi * kz[a];
    }
    const int64_t i = perm[s];
    if (i < 0 || i >= M) continue;
    vis[2 * i] += sr * r.c[0] - si * r.c[1];
    vis[2 * i + 1] += sr * r.c[1] + si * r.c[0];
  }
}

template <typename T>
int launch_grid_window(const Rec<T>* d_recs, int64_t M, const Geom& g, int p0, int p1, T* d_fwb,
                       cudaStream_t st) {
  CG_CUDA(cudaMemsetAsync(d_fwb, 0, (size_t)(p1 - p0) * g.nf1 * g.nf2 * 2 * sizeof(T), st));
  if (M == 0) return CG_OK;
  const int blocks = (int)std::min<int64_t>((M + 255) / 256, 148 * 64);
#define CG_GW_CALL(w)                                                              \
  (k_grid_window<T, w><<<blocks, 256, 0, st>>>(d_recs, M, g, p0, p1, d_fwb),     \
   count_launches(1), cudaGetLastError() == cudaSuccess ? CG_OK : CG_ERR_CUDA)
  CG_W_SWITCH(g.kw, CG_GW_CALL)
#undef CG_GW_CALL
}

template <typename T>
int launch_degrid_window(const Rec<T>* d_recs, const int* d_perm, int64_t M, const Geom& g,
                         int p0, int p1, const T* d_fwb, T* d_vis, cudaStream_t st) {
  if (M == 0) return CG_OK;
  const int blocks = (int)std::min<int64_t>((M + 255) / 256, 148 * 64);
#define CG_DW_CALL(w)                                                                         \
  (k_degrid_window<T, w><<<blocks, 256, 0, st>>>(d_recs, d_perm, M, g, p0, p1, d_fwb, d_vis), \
   count_launches(1), cudaGetLastError() == cudaSuccess ? CG_OK : CG_ERR_CUDA)
  CG_W_SWITCH(g.kw, CG_DW_CALL)
#undef CG_DW_CALL
}

template int launch_grid_window<float>(const Rec<float>*, int64_t, const Geom&, int, int, float*,
                                       cudaStream_t);
template int launch_grid_window<double>(const Rec<double>*, int64_t, const Geom&, int, int,
                                        double*, cudaStream_t);
template int launch_degrid_window<float>(const Rec<float>*, const int*, int64_t, const Geom&, int,
                                         int, const float*, float*, cudaStream_t);
template int launch_degrid_window<double>(const Rec<double>*, const int*, int64_t, const Geom&,
                                          int, int, const double*, double*, cudaStream_t);

template bool few_degrid_tiles<float>(const Geom&, int);
template bool few_degrid_tiles<double>(const Geom&, int);
template TileCfg degrid_tiling<float>(const Geom&, const TileTune*);
template TileCfg degrid_tiling<double>(const Geom&, const TileTune*);
template int multi_shape<float>(GridJob<float>*, int, MultiShape*);
template int multi_shape<double>(GridJob<double>*, int, MultiShape*);
template int launch_degrid_multi<float>(const GridJob<float>*, int, const MultiShape&, int*,
                                        cudaStream_t);
template int launch_degrid_multi<double>(const GridJob<double>*, int, const MultiShape&, int*,
                                         cudaStream_t);
template int launch_grid<float>(const Rec<float>*, const int*, int64_t, const Geom&, float*, int,
                                int*, cudaStream_t, const SplitScratch*);
template int launch_grid<double>(const Rec<double>*, const int*, int64_t, const Geom&, double*, int,
                                 int*, cudaStream_t, const SplitScratch*);
template int launch_degrid<float>(const Rec<float>*, const int*, const int*, int64_t, const Geom&,
                                  const float*, float*, int, int*, cudaStream_t, const TileTune*, cg_dev_buf*);
template int launch_degrid<double>(const Rec<double>*, const int*, const int*, int64_t,
                                   const Geom&, const double*, double*, int, int*, cudaStream_t,
                                   const TileTune*, cg_dev_buf*);

}  // namespace cg
