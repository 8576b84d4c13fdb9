// Gridding (spreading) with lane-owned grid columns.
//
//   fw[p][g1][g0] = sum_j c_j phi(g0 - X0_j) phi(g1 - X1_j) phi(p - X2_j)
//
// (conv_3d_outputdriven_t1, conv.cu:522-627), periodic in all three axes, every
// grid cell written exactly once, no atomics on data, a deterministic result.
//
// A CTA owns a tile of TX x TY cells (g0, g1) and walks its rows in plane
// order.  Each warp owns a unit of 8 x 4 cells; each half of the warp holds all
// 32 cells of it, two cells per lane, and takes every other row, so two rows are
// spread at a time.  A lane keeps its cells' NZ = W (odd W: W + 1) planes around
// the current plane in registers: all rows of a hive share one plane, so the
// taps along w land on fixed registers.  When the plane advances, the registers
// shift by one and the finished plane's sums (the two halves added) go to HBM.
// Nothing is accumulated in shared memory.
//
// Per chunk of up to S candidate rows (the tile's hives and a ring of one):
//   1. each thread loads kOwnCand candidate records and tests them against the
//      tile; the rows that reach it are compacted in order (the next chunk's candidates
//      load while this chunk's rows are spread);
//   2. the 3 W kernel values of each row are evaluated once per CTA, one
//      (row, axis) per thread, and stored in the row's slot of shared memory;
//      the x and y values sit between zeros, so a lane whose cell a row does
//      not reach reads 0 and needs no test;
//   3. each warp lists the rows that reach its unit, and its halves walk the
//      list: 6 shared loads (list entry, kx, two ky, kz, strength) and 4 W FMAs
//      a row and lane.
// A plane with more than S candidates is cut into chunks by taking every
// n-th candidate, so each chunk covers the tile evenly and the warps finish
// together; planes with few candidates share a chunk.
//
// Bound: instruction issue (0.63 of the cycles; about 190 warp instructions a
// row, 60 of them in the row walk, the rest per chunk and per tile and plane).
// The kernels before this one added each tap to shared memory, a load and a
// store a tap, with 230 warp instructions a row and 0.4 of the cycles issuing.
// Measured, before -> now: 2048^2, 10M rows, W = 6: 7.8 -> 1.9 ms; 4096^2, 20M
// rows, W = 6: 7.8 -> 4.7 ms; FP64 2048^2, 5M rows, W = 10: 24.4 -> 5.8 ms.
// Units of 4 x 4 cells with one cell a lane (64 registers) took 2.9 and 6.9 ms,
// four of them to a warp (128 registers) 2.9 and 8.3, tiles of 32 x 16 cells
// 2.4 and 5.1, two CTAs an SM instead of three 2.3 and 5.7.  FP64 above W = 8
// takes one cell a lane: at W = 10 two need 240 registers (6.75 against 6.47 ms).
#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "cg_coords.cuh"
#include "cg_launch.cuh"
#include "cg_plan.cuh"
#include "cg_tiles.cuh"

namespace cg {
namespace {

constexpr int kOwnUX = 8;                // unit of a warp: 8 columns
constexpr int kOwnCand = 2;              // candidates per thread and chunk
constexpr int kOwnList = 64;             // list entries of a warp
constexpr int kOwnStrip = 4;             // tiles of a strip

template <typename T>
struct OwnC;
template <>
struct OwnC<float> { using type = float2; };
template <>
struct OwnC<double> { using type = double2; };

// Slot of one row in shared memory, in elements of T: zeros, W x values,
// zeros, W y values, zeros, NZ w values, the strength (re, im).  A lane reads
// the x (y) values up to 7 (3) places before and after them.  The slot is an odd
// number of 16-byte words long, so that 16-byte stores of consecutive rows
// fall on different banks.
template <typename T, int W>
struct OwnRow {
  // cells per lane, two rows apart; unit rows, warps and threads of a CTA
  static constexpr int CPL = sizeof(T) == 8 && W > 8 ? 1 : 2;
  static constexpr int UY = 2 * CPL, WARPS = (kOwnTX / kOwnUX) * (kOwnTY / UY), THREADS = 32 * WARPS;
  // CTAs per SM
  static constexpr int CTAS = sizeof(T) == 4 ? (W <= 8 ? 3 : 2) : (W <= 8 ? 2 : 1);
  static constexpr int V = 16 / sizeof(T);
  static constexpr int up(int a) { return (a + V - 1) / V * V; }
  static constexpr int NZ = (W + 1) / 2 * 2;
  static constexpr int KX = kOwnUX;
  static constexpr int KY = up(KX + W + kOwnUX - 1);
  static constexpr int KZ = up(KY + W + UY - 1);
  static constexpr int RAW = up(KZ + NZ + 2);
  static constexpr int ST = (RAW / V) % 2 ? RAW : RAW + V;
};

// Register sums of one lane's two cells (u = 0, 1: rows y and y + 2 of the
// unit): plane j of NZ, two planes per packed register in FP32 (fma.rn.f32x2
// rounds each half as a scalar FMA does).
template <typename T, int NZ, int CPL>
struct OwnAcc;

template <int NZ, int CPL>
struct OwnAcc<float, NZ, CPL> {
  unsigned long long re[CPL][NZ / 2], im[CPL][NZ / 2];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int u = 0; u < CPL; u++)
#pragma unroll
      for (int j = 0; j < NZ / 2; j++) re[u][j] = im[u][j] = 0ull;
  }
  // x, y: shared addresses of this lane's kernel values; z: of the NZ values
  // along w followed by the strength, 16-byte aligned
  __device__ __forceinline__ void add(unsigned x, unsigned y, unsigned z) {
    unsigned long long w[NZ / 2 + 2];
    float kx, ky[CPL], vr, vi;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(kx) : "r"(x) : "memory");
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(ky[0]) : "r"(y) : "memory");
    if constexpr (CPL == 2) asm volatile("ld.shared.f32 %0, [%1+8];" : "=f"(ky[CPL - 1]) : "r"(y) : "memory");
#pragma unroll
    for (int j = 0; j + 1 < NZ / 2 + 1; j += 2)
      asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(w[j]), "=l"(w[j + 1]) : "r"(z + 8 * j) : "memory");
    if constexpr (NZ / 2 % 2 == 0) asm volatile("ld.shared.b64 %0, [%1];" : "=l"(w[NZ / 2]) : "r"(z + 4 * NZ) : "memory");
    asm("mov.b64 {%0, %1}, %2;" : "=f"(vr), "=f"(vi) : "l"(w[NZ / 2]));
    const float xr = vr * kx, xi = vi * kx;
#pragma unroll
    for (int u = 0; u < CPL; u++) {
      const float cr = xr * ky[u], ci = xi * ky[u];
      unsigned long long pr, pi;
      asm("mov.b64 %0, {%1, %1};" : "=l"(pr) : "f"(cr));
      asm("mov.b64 %0, {%1, %1};" : "=l"(pi) : "f"(ci));
#pragma unroll
      for (int j = 0; j < NZ / 2; j++) {
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(re[u][j]) : "l"(pr), "l"(w[j]));
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(im[u][j]) : "l"(pi), "l"(w[j]));
      }
    }
  }
  __device__ __forceinline__ void first(int u, float& r, float& i) const {
    float h;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r), "=f"(h) : "l"(re[u][0]));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(i), "=f"(h) : "l"(im[u][0]));
  }
  __device__ __forceinline__ void shift() {
#pragma unroll
    for (int u = 0; u < CPL; u++)
#pragma unroll
      for (int j = 0; j < NZ / 2; j++) {
        const int k = j + 1 < NZ / 2 ? j + 1 : j;
        re[u][j] = (re[u][j] >> 32) | (k > j ? re[u][k] << 32 : 0ull);
        im[u][j] = (im[u][j] >> 32) | (k > j ? im[u][k] << 32 : 0ull);
      }
  }
};

template <int NZ, int CPL>
struct OwnAcc<double, NZ, CPL> {
  double re[CPL][NZ], im[CPL][NZ];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int u = 0; u < CPL; u++)
#pragma unroll
      for (int j = 0; j < NZ; j++) re[u][j] = im[u][j] = 0.0;
  }
  __device__ __forceinline__ void add(unsigned x, unsigned y, unsigned z) {
    double kx, ky[CPL], vr, vi;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(kx) : "r"(x) : "memory");
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(ky[0]) : "r"(y) : "memory");
    if constexpr (CPL == 2) asm volatile("ld.shared.f64 %0, [%1+16];" : "=d"(ky[CPL - 1]) : "r"(y) : "memory");
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(vr), "=d"(vi) : "r"(z + 8 * NZ) : "memory");
    const double xr = vr * kx, xi = vi * kx;
    double cr[CPL], ci[CPL];
#pragma unroll
    for (int u = 0; u < CPL; u++) {
      cr[u] = xr * ky[u];
      ci[u] = xi * ky[u];
    }
#pragma unroll
    for (int j = 0; j < NZ; j += 2) {
      double q0, q1;
      asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(q0), "=d"(q1) : "r"(z + 8 * j) : "memory");
#pragma unroll
      for (int u = 0; u < CPL; u++) {
        re[u][j] = fma(cr[u], q0, re[u][j]);
        im[u][j] = fma(ci[u], q0, im[u][j]);
        re[u][j + 1] = fma(cr[u], q1, re[u][j + 1]);
        im[u][j + 1] = fma(ci[u], q1, im[u][j + 1]);
      }
    }
  }
  __device__ __forceinline__ void first(int u, double& r, double& i) const {
    r = re[u][0];
    i = im[u][0];
  }
  __device__ __forceinline__ void shift() {
#pragma unroll
    for (int u = 0; u < CPL; u++)
#pragma unroll
      for (int j = 0; j < NZ; j++) {
        const int k = j + 1 < NZ ? j + 1 : j;
        re[u][j] = k > j ? re[u][k] : 0.0;
        im[u][j] = k > j ? im[u][k] : 0.0;
      }
  }
};

// taps() of a polynomial kernel whose coefficients lie 16-byte aligned in shared
// memory, read 16 bytes at a time: left to itself the compiler reads each one
// (gridding 2048^2, 10M rows, W = 6: 2.06 -> 1.90 ms; 4096^2, 20M: 5.14 -> 4.73).
template <int W, typename T>
__device__ __forceinline__ int poly_taps(T f, const T* __restrict__ poly, T* k) {
  constexpr int V = 16 / sizeof(T);
  using Q = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
  const T t = poly_arg<W>(f);
#pragma unroll
  for (int i = 0; i < W; i++) {
    T a[kPolyCoef];
#pragma unroll
    for (int n = 0; n < kPolyCoef; n += V) {
      const Q q = *reinterpret_cast<const Q*>(poly + i * kPolyCoef + n);
      a[n] = q.x;
      a[n + 1] = q.y;
      if constexpr (V == 4) {
        a[n + 2] = q.z;
        a[n + 3] = q.w;
      }
    }
    T v = a[kPolyCoef - 1];
#pragma unroll
    for (int n = kPolyCoef - 2; n >= 0; n--) v = fma(v, t, a[n]);
    k[i] = v;
  }
  return tap_offset<W>(f);
}

// Segment slot of candidate q among the (plane, hive row) entries [lo, hi),
// three slots each.
__device__ __forceinline__ int own_segment(const int* __restrict__ pref, int lo, int hi, int q) {
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (pref[3 * mid] <= q) lo = mid; else hi = mid;
  }
  lo *= 3;
  return lo + (pref[lo + 1] <= q) + (pref[lo + 2] <= q);
}

// n values k[0..n) to p (16-byte aligned), as wide stores as n allows
template <int N, typename T>
__device__ __forceinline__ void store_values(T* p, const T* k) {
  if constexpr (sizeof(T) == 4) {
    constexpr int N4 = N / 4 * 4;
#pragma unroll
    for (int i = 0; i < N4; i += 4)
      *reinterpret_cast<float4*>(p + i) = make_float4(k[i], k[i + 1], k[i + 2], k[i + 3]);
    if constexpr (N - N4 >= 2) *reinterpret_cast<float2*>(p + N4) = make_float2(k[N4], k[N4 + 1]);
    if constexpr (N % 2) p[N - 1] = k[N - 1];
  } else {
#pragma unroll
    for (int i = 0; i + 1 < N; i += 2) *reinterpret_cast<double2*>(p + i) = make_double2(k[i], k[i + 1]);
    if constexpr (N % 2) p[N - 1] = k[N - 1];
  }
}

// Shared memory of a CTA.
template <typename T>
struct OwnSmem {
  T* rows;     // cap + 1 row slots, the last all zero
  T* f;        // 3 x cap fractions of the chunk's rows
  T* poly;     // W x kPolyCoef coefficients (polynomial kernels)
  int4* pre;   // cap: shared addresses of a row's x and y values (for the tile's first cell) and w values
  int4* list;  // kOwnList entries per warp
  int* meta;   // cap: subtiles that a row reaches, and its plane
  int* seg;    // segment table
  int cap;
};

template <typename T, int W>
__host__ __device__ inline size_t own_bytes(int cap, int slots) {
  using R = OwnRow<T, W>;
  return (size_t)(cap + 1) * R::ST * sizeof(T) + (size_t)cap * sizeof(int4) +
         (size_t)R::WARPS * kOwnList * sizeof(int4) + (size_t)3 * cap * sizeof(T) +
         (size_t)W * kPolyCoef * sizeof(T) + (size_t)cap * sizeof(int) +
         (size_t)(slots + 1) * kSegInts * sizeof(int);
}

template <typename T, int W, bool kPoly>
__device__ __forceinline__ OwnSmem<T> own_smem(unsigned char* p, int cap, const T* __restrict__ poly) {
  using R = OwnRow<T, W>;
  OwnSmem<T> m;
  m.cap = cap;
  m.rows = reinterpret_cast<T*>(p);
  p += (size_t)(cap + 1) * R::ST * sizeof(T);
  m.pre = reinterpret_cast<int4*>(p);
  p += (size_t)cap * sizeof(int4);
  m.list = reinterpret_cast<int4*>(p);
  p += (size_t)R::WARPS * kOwnList * sizeof(int4);
  m.f = reinterpret_cast<T*>(p);
  p += (size_t)3 * cap * sizeof(T);
  m.poly = reinterpret_cast<T*>(p);
  p += (size_t)W * kPolyCoef * sizeof(T);
  m.meta = reinterpret_cast<int*>(p);
  m.seg = m.meta + cap;
  // zeros around the values stay: only the values and the strength are rewritten
  for (int i = threadIdx.x; i < (cap + 1) * R::ST; i += R::THREADS) m.rows[i] = (T)0;
  if constexpr (kPoly)
    for (int i = threadIdx.x; i < W * kPolyCoef; i += R::THREADS) m.poly[i] = poly[i];
  __syncthreads();
  return m;
}

// Kernel values of a row along an axis (fraction f) into its slot.
template <typename T, int W, bool kPoly>
__device__ __forceinline__ void own_values(const OwnSmem<T>& sm, int row, int axis, T f, T beta, T c) {
  using R = OwnRow<T, W>;
  constexpr int lo = Halo<W>::lo, NZ = R::NZ;
  T k[W];
  int o;
  if constexpr (kPoly) {
    o = poly_taps<W>(f, sm.poly, k);
  } else {
    o = taps<T, W>(f, beta, c, (const T*)nullptr, k);
  }
  T* p = sm.rows + row * R::ST;
  if (axis < 2) {
    store_values<W>(p + (axis == 0 ? R::KX : R::KY), k);
  } else if constexpr (W == NZ) {
    store_values<W>(p + R::KZ, k);
  } else {  // odd W: the first tap is plane bz - lo or the one above
    const bool up = o + lo > 0;
    T kz[NZ];
#pragma unroll
    for (int i = 0; i < NZ; i++) {
      const T below = i < W ? k[i < W ? i : 0] : (T)0, above = i > 0 ? k[i > 0 ? i - 1 : 0] : (T)0;
      kz[i] = up ? above : below;
    }
    store_values<NZ>(p + R::KZ, kz);
  }
}

// One tile (work item `item` of tiling tc): every cell of it written to fw;
// or, part != nullptr, row chunk `chunk` of `nchunks` of the tile -- rows
// [total * chunk / nchunks, total * (chunk + 1) / nchunks) of its `total` in
// plane order -- written whole into a partial tile at part (cell (x, y, z) at
// (z * TY + y) * TX + x).  Called by all threads with the same arguments.
template <typename T, int W, bool kPoly>
__device__ __forceinline__ void own_tile(const Rec<T>* __restrict__ recs,
                                         const int* __restrict__ hive_start, const Geom& g,
                                         const WarpTile& tc, T* __restrict__ fw, int item,
                                         const OwnSmem<T>& sm, int* s_warp, int* s_cnt, int chunk,
                                         int nchunks, typename OwnC<T>::type* __restrict__ part) {
  using C = typename OwnC<T>::type;
  using R = OwnRow<T, W>;
  constexpr int lo = Halo<W>::lo, hi = Halo<W>::hi, NZ = R::NZ, ST = R::ST;
  constexpr int CPL = R::CPL, UY = R::UY, WARPS = R::WARPS, THREADS = R::THREADS;
  constexpr int NC = kOwnCand, S = THREADS * NC;
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  const int nf1 = g.nf1, nf2 = g.nf2, nw = g.nw;
  const size_t plane = (size_t)nf1 * nf2;
  C* fwc = reinterpret_cast<C*>(fw);
  const int tix = tc.bx0 + item % tc.ntx, tiy = tc.by0 + (item / tc.ntx) % tc.nty, tib = item / (tc.ntx * tc.nty);
  const int tx0 = tix * kOwnTX, ty0 = tiy * kOwnTY, p0 = tib * tc.PB;
  const int tx1 = min(tx0 + kOwnTX, nf1), ty1 = min(ty0 + kOwnTY, nf2), p1 = min(p0 + tc.PB, nw);
  // zeros in every cell of the tile (a partial tile: in all PB planes)
  auto zero_tile = [&]() {
    if (part) {
      for (int i = tid; i < kOwnTX * kOwnTY * tc.PB; i += THREADS) part[i] = C{(T)0, (T)0};
      return;
    }
    // 8 (FP64: 16) threads a tile row; nf1 is even, so pairs never straddle its end
    constexpr int CP = sizeof(T) == 4 ? 2 : 1, TPR = kOwnTX / CP, RPP = THREADS / TPR;
    const int x = tx0 + (tid % TPR) * CP;
    const int wy = ty1 - ty0, nrow = wy * (p1 - p0);
    if (x >= nf1) return;
    for (int r = tid / TPR; r < nrow; r += RPP) {
      const int z = r / wy, y = r - z * wy;
      C* dst = fwc + (size_t)(p0 + z) * plane + (size_t)(ty0 + y) * nf1 + x;
      if constexpr (sizeof(T) == 4)
        *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
      else
        *dst = C{(T)0, (T)0};
    }
  };
  // outside the cells the data can reach
  if (tx0 > g.band_c1 || tx1 <= g.band_c0 || ty0 > g.band_r1 || ty1 <= g.band_r0) {
    zero_tile();
    return;
  }
  const int ts = tc.slots + 1;
  SegTable t{sm.seg, sm.seg + ts, sm.seg + 2 * ts};
  const int hya = raw_hive_lo(ty0 - hi, nf2, g.nhy), hyb = raw_hive_hi(ty1 - 1 + lo, nf2, g.nhy);
  __syncthreads();  // the last tile's table is no longer read
  const int nslots = build_segments(g, hive_start, raw_hive_lo(tx0 - hi, nf1, g.nhx),
                                    raw_hive_hi(tx1 - 1 + lo, nf1, g.nhx), hya, hyb, p0 - hi,
                                    p1 - 1 + lo, t, s_warp);
  const int total = t.pref[nslots];
  int qb = 0, qe = total;
  if (part) {
    qb = (int)((int64_t)total * chunk / nchunks);
    qe = (int)((int64_t)total * (chunk + 1) / nchunks);
  }
  if (qb == qe) {
    zero_tile();
    return;
  }
  const int cap = sm.cap;
  const int hrows = hyb - hya + 1, NP = p1 - p0 + lo + hi;
  // candidates of the planes before raw plane k (plane p0 - hi + k), inside
  // [qb, qe); lane l keeps those of k = l + 1 and l + 33 (NP <= 64)
  auto cut = [&](int k) { return min(max(t.pref[min(k, NP) * hrows * 3], qb), qe); };
  const int cut0 = cut(lane + 1), cut1 = cut(lane + 33);

  const T beta = (T)g.beta, c = (T)g.es_c;
  const int grp = lane >> 4, lx = lane & 7, ly = (lane >> 3) & 1;
  constexpr int NUX = kOwnTX / kOwnUX;
  const int ux = (wib % NUX) * kOwnUX + lx, uy = (wib / NUX) * UY + ly;  // this lane's first cell
  C* dst = part ? part + uy * kOwnTX + ux : fwc + (size_t)p0 * plane + (size_t)(ty0 + uy) * nf1 + tx0 + ux;
  const size_t dplane = part ? (size_t)kOwnTX * kOwnTY : plane;
  const int drow = 2 * (part ? kOwnTX : nf1);  // the second cell is two rows on
  // two cells: the lower half writes the first, the upper half the second
  const bool wr = (CPL == 2 || grp == 0) && (part || (tx0 + ux < nf1 && ty0 + uy + 2 * grp < nf2));
  const unsigned srows = (unsigned)__cvta_generic_to_shared(sm.rows);
  const unsigned offx = ux * sizeof(T), offy = uy * sizeof(T);
  int4* list = sm.list + wib * kOwnList;
  const unsigned zslot = srows + cap * ST * (int)sizeof(T);
  const int4 dummy = make_int4(zslot + (R::KX - (ux - lx)) * (int)sizeof(T),
                               zslot + (R::KY - (uy - ly)) * (int)sizeof(T), zslot + R::KZ * (int)sizeof(T), 0);

  OwnAcc<T, NZ, CPL> acc;
  acc.clear();
  int zc = 0;    // raw plane, from p0 - hi; register j holds plane zc - hi - lo + j of the item
  int live = 0;  // the sums are zero from raw plane `live` on
  // planes finished before raw plane z becomes current
  auto advance = [&](int z) {
    for (; zc < z; zc++) {
      const int p = zc - hi - lo;
      C v = {(T)0, (T)0};
      if (zc < live) {
        // each half adds the other's share of the row that it writes
        T r0, i0, r1, i1;
        acc.first(0, r0, i0);
        acc.first(CPL - 1, r1, i1);
        const T sr = grp ? r0 : r1, si = grp ? i0 : i1;
        const T kr = grp ? r1 : r0, ki = grp ? i1 : i0;
        v.x = kr + __shfl_xor_sync(0xffffffffu, sr, 16);
        v.y = ki + __shfl_xor_sync(0xffffffffu, si, 16);
        acc.shift();
      }
      if (wr && p >= 0 && p < p1 - p0) dst[(size_t)p * dplane + grp * drow] = v;
    }
  };
  // the cnt listed rows of raw plane zc, two at a time per half-warp
  auto spread = [&](int cnt) {
    if (lane == 0) list[cnt] = dummy;
    __syncwarp();
    live = zc + NZ;
    int j = grp;
    for (; j + 2 - grp < cnt; j += 4) {
      const int4 e0 = list[j], e1 = list[j + 2];
      acc.add(offx + e0.x, offy + e0.y, e0.z);
      acc.add(offx + e1.x, offy + e1.y, e1.z);
    }
    if (j - grp < cnt) {
      const int4 e0 = list[j];
      acc.add(offx + e0.x, offy + e0.y, e0.z);
    }
    __syncwarp();
  };

  // chunk sequence: planes [k, knext) or every nch-th candidate of plane k
  int knext = 0, ch = 0, nch = 0, a = 0, n = 0;
  int s_lo = 0, s_hi = 0;  // (plane, hive row) entries of the chunk's planes
  int zone = 0;            // its first plane
  bool one = false;        // a single plane
  auto at = [&](int k) {
    return k <= 32 ? __shfl_sync(0xffffffffu, cut0, (k - 1) & 31) : __shfl_sync(0xffffffffu, cut1, (k - 33) & 31);
  };
  auto next_chunk = [&]() {
    if (ch + 1 < nch) {
      ch++;
      return true;
    }
    if (knext >= NP) return false;
    auto planes = [&](bool lower, bool upper) {
      return (unsigned long long)__ballot_sync(0xffffffffu, lower) |
             (unsigned long long)__ballot_sync(0xffffffffu, upper) << 32;
    };
    a = knext ? at(knext) : qb;
    const int k = __ffsll(planes(cut0 > a, cut1 > a)) - 1;  // first plane with candidates
    if (k < 0) return false;
    // the planes that fit a chunk together, at least one
    const int e = max(k + 1, min(NP, __popcll(planes(cut0 - a <= S, cut1 - a <= S))));
    n = at(e) - a;
    ch = 0;
    nch = (n + S - 1) / S;
    knext = e;
    zone = k;
    one = e == k + 1;
    s_lo = k * hrows;
    s_hi = e * hrows;
    return true;
  };
  // this thread's candidates, consecutive in the chunk
  T cf[NC][3], cv[NC][2];
  int co[NC];  // packed first taps and plane; -1: does not reach the tile
  auto load = [&]() {
#pragma unroll
    for (int i = 0; i < NC; i++) {
      co[i] = -1;
      const int idx = (tid * NC + i) * nch + ch;
      if (idx < n) {
        const int q = a + idx;
        const int sgi = own_segment(t.pref, s_lo, s_hi, q);
        const Rec<T> r = recs[t.start[sgi] + (q - t.pref[sgi])];
        cf[i][0] = r.f[0]; cf[i][1] = r.f[1]; cf[i][2] = r.f[2]; cv[i][0] = r.c[0]; cv[i][1] = r.c[1];
        const int sc = t.shift[sgi];
        int ox = (int)(r.bxy & 0xFFFFu) + tap_offset<W>(r.f[0]) - tx0;
        int oy = (int)(r.bxy >> 16) + tap_offset<W>(r.f[1]) - ty0;
        int z = (int)r.bz - (p0 - hi);
        if (sc) {  // a periodic image
          ox += unpack_shift(sc, nf1);
          oy += unpack_shift(sc >> 2, nf2);
          z += unpack_shift(sc >> 4, nw);
        }
        if (ox + W > 0 && ox < kOwnTX && oy + W > 0 && oy < kOwnTY) co[i] = (ox + 32) | (oy + 32) << 7 | z << 14;
      }
    }
  };

  bool more = next_chunk();
  if (more) load();
  int b0 = 0;  // rows of the chunk done before this pass (more than cap reach the tile)
  while (more) {
    {
      int mine = 0;
#pragma unroll
      for (int i = 0; i < NC; i++) mine += co[i] >= 0;
      int inc = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
      }
      if (lane == 31) s_cnt[wib] = inc;
      __syncthreads();  // also: every warp is done with the last chunk's rows
      const int v = lane < WARPS ? s_cnt[lane] : 0;
      int pos = __reduce_add_sync(0xffffffffu, lane < wib ? v : 0) + inc - mine - b0;
      const int nr = __reduce_add_sync(0xffffffffu, v);
#pragma unroll
      for (int i = 0; i < NC; i++) {
        if (co[i] >= 0) {
          if (pos >= 0 && pos < cap) {
            sm.f[pos] = cf[i][0];
            sm.f[cap + pos] = cf[i][1];
            sm.f[2 * cap + pos] = cf[i][2];
            const int ox = (co[i] & 127) - 32, oy = ((co[i] >> 7) & 127) - 32, z = co[i] >> 14;
            // units along an axis: those with a cell in [o, o + W)
            const int mx = (2 << (min(ox + W - 1, kOwnTX - 1) / kOwnUX)) - (1 << (max(ox, 0) / kOwnUX));
            const int y0 = max(oy, 0) / UY, y1 = min(oy + W - 1, kOwnTY - 1) / UY;
            int units = 0;
#pragma unroll
            for (int y = 0; y < kOwnTY / UY; y++)
              if (y >= y0 && y <= y1) units |= mx << (y * NUX);
            sm.meta[pos] = units | z << 16;
            const unsigned slot = srows + pos * ST * (int)sizeof(T);
            sm.pre[pos] = make_int4(slot + (R::KX - ox) * (int)sizeof(T), slot + (R::KY - oy) * (int)sizeof(T),
                                    slot + R::KZ * (int)sizeof(T), 0);
            *reinterpret_cast<C*>(sm.rows + pos * ST + R::KZ + NZ) = C{cv[i][0], cv[i][1]};
          }
          pos++;
        }
      }
      __syncthreads();
      const int nrow = min(nr - b0, cap);  // rows of this pass
      // kernel values, one (row, axis) per thread: own_values written out (called here, the
      // FP64 instances spill more: W = 7 146 -> 260 bytes, 1M rows on 2048^2 0.51 -> 0.54 ms)
      const int nb = (nrow + 31) >> 5;
      for (int u = wib; u < 3 * nb; u += WARPS) {
        const int axis = u >= 2 * nb ? 2 : (u >= nb ? 1 : 0);
        const int row = ((u - axis * nb) << 5) + lane;
        if (row < nrow) {
          const T f = sm.f[axis * cap + row];
          T k[W];
          int o;
          if constexpr (kPoly) {
            o = poly_taps<W>(f, sm.poly, k);
          } else {
            o = taps<T, W>(f, beta, c, (const T*)nullptr, k);
          }
          T* p = sm.rows + row * ST;
          if (axis < 2) {
            store_values<W>(p + (axis == 0 ? R::KX : R::KY), k);
          } else if constexpr (W == NZ) {
            store_values<W>(p + R::KZ, k);
          } else {  // odd W: the first tap is plane bz - lo or the one above
            const bool up = o + lo > 0;
            T kz[NZ];
#pragma unroll
            for (int i = 0; i < NZ; i++) {
              const T below = i < W ? k[i < W ? i : 0] : (T)0, above = i > 0 ? k[i > 0 ? i - 1 : 0] : (T)0;
              kz[i] = up ? above : below;
            }
            store_values<NZ>(p + R::KZ, kz);
          }
        }
      }
      __syncthreads();
      // the next chunk's candidates (or this chunk's again) while its rows are spread
      const bool one_ = one, last = b0 + cap >= nr;
      const int zone_ = zone;
      if (last) more = next_chunk();
      b0 = last ? 0 : b0 + cap;
      if (more) load();
      // this unit's rows
      const unsigned bit = 1u << wib;
      int cnt = 0;
      if (one_) {
        for (int b = 0; b < nrow; b += 32) {
          const int row = b + lane;
          const bool take = row < nrow && (sm.meta[row] & bit);
          const unsigned sel = __ballot_sync(0xffffffffu, take);
          if (!sel) continue;
          advance(zone_);
          if (take) list[cnt + __popc(sel & ((1u << lane) - 1u))] = sm.pre[row];
          cnt += __popc(sel);
          if (cnt > kOwnList - 33) {
            spread(cnt);
            cnt = 0;
          }
        }
      } else {
        for (int b = 0; b < nrow; b += 32) {
          const int row = b + lane;
          const int m = row < nrow ? sm.meta[row] : 0;
          const bool take = m & bit;
          unsigned rem = __ballot_sync(0xffffffffu, take);
          while (rem) {
            const int z = m >> 16, zf = __shfl_sync(0xffffffffu, z, __ffs(rem) - 1);
            const bool now = take && z == zf;
            const unsigned sel = __ballot_sync(0xffffffffu, now);
            rem &= ~sel;
            if (zf != zc) {
              if (cnt) spread(cnt);
              cnt = 0;
              advance(zf);
            }
            if (now) list[cnt + __popc(sel & ((1u << lane) - 1u))] = sm.pre[row];
            cnt += __popc(sel);
            if (cnt > kOwnList - 33) {
              spread(cnt);
              cnt = 0;
            }
          }
        }
      }
      if (cnt) spread(cnt);
    }
  }
  advance(p1 - p0 + lo + hi);
}

// A strip of up to kOwnStrip tiles side by side (strip `item` of tiling tc) at once, for
// grids with few rows a tile: the table, the candidates and the kernel values are made
// once for all of them, then each warp spreads its unit of every tile in turn.
// False, with nothing written to the grid, where the strip's candidates do not fit one chunk or
// the rows that reach it the row slots.
template <typename T, int W, bool kPoly>
__device__ __forceinline__ bool own_strip(const Rec<T>* __restrict__ recs, const int* __restrict__ hive_start,
                                          const Geom& g, const WarpTile& tc, T* __restrict__ fw, int item,
                                          const OwnSmem<T>& sm, int* s_warp, int* s_cnt) {
  using C = typename OwnC<T>::type;
  using R = OwnRow<T, W>;
  constexpr int lo = Halo<W>::lo, hi = Halo<W>::hi, NZ = R::NZ, ST = R::ST;
  constexpr int CPL = R::CPL, UY = R::UY, WARPS = R::WARPS, THREADS = R::THREADS;
  constexpr int NC = kOwnCand, S = THREADS * NC, NUX = kOwnTX / kOwnUX;
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  const int nf1 = g.nf1, nf2 = g.nf2, nw = g.nw, cap = sm.cap;
  const size_t plane = (size_t)nf1 * nf2;
  C* fwc = reinterpret_cast<C*>(fw);
  const int nsx = (tc.ntx + kOwnStrip - 1) / kOwnStrip, first = item % nsx * kOwnStrip;
  const int nsub = min(kOwnStrip, tc.ntx - first);
  const int tx0 = (tc.bx0 + first) * kOwnTX, ty0 = (tc.by0 + item / nsx % tc.nty) * kOwnTY;
  const int p0 = item / (nsx * tc.nty) * tc.PB;
  const int tx1 = min(tx0 + nsub * kOwnTX, nf1), ty1 = min(ty0 + kOwnTY, nf2), p1 = min(p0 + tc.PB, nw);
  const int ts = tc.slots + 1;
  SegTable t{sm.seg, sm.seg + ts, sm.seg + 2 * ts};
  const int hya = raw_hive_lo(ty0 - hi, nf2, g.nhy), hyb = raw_hive_hi(ty1 - 1 + lo, nf2, g.nhy);
  __syncthreads();  // the last item's table is no longer read
  const int nslots = build_segments(g, hive_start, raw_hive_lo(tx0 - hi, nf1, g.nhx),
                                    raw_hive_hi(tx1 - 1 + lo, nf1, g.nhx), hya, hyb, p0 - hi, p1 - 1 + lo, t, s_warp);
  const int total = t.pref[nslots];
  if (total > S) return false;
  // the rows that reach the strip, in plane order
  T cf[NC][3], cv[NC][2];
  int co[NC];
  int mine = 0;
#pragma unroll
  for (int i = 0; i < NC; i++) {
    co[i] = -1;
    const int q = tid * NC + i;
    if (q < total) {
      const int sgi = own_segment(t.pref, 0, nslots / 3, q);
      const Rec<T> r = recs[t.start[sgi] + (q - t.pref[sgi])];
      cf[i][0] = r.f[0]; cf[i][1] = r.f[1]; cf[i][2] = r.f[2]; cv[i][0] = r.c[0]; cv[i][1] = r.c[1];
      const int sc = t.shift[sgi];
      int ox = (int)(r.bxy & 0xFFFFu) + tap_offset<W>(r.f[0]) - tx0;
      int oy = (int)(r.bxy >> 16) + tap_offset<W>(r.f[1]) - ty0;
      int z = (int)r.bz - (p0 - hi);
      if (sc) {  // a periodic image
        ox += unpack_shift(sc, nf1);
        oy += unpack_shift(sc >> 2, nf2);
        z += unpack_shift(sc >> 4, nw);
      }
      if (ox + W > 0 && ox < nsub * kOwnTX && oy + W > 0 && oy < kOwnTY) co[i] = (ox + 32) | (oy + 32) << 7 | z << 14;
    }
    mine += co[i] >= 0;
  }
  int inc = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) s_cnt[wib] = inc;
  __syncthreads();
  const int v = lane < WARPS ? s_cnt[lane] : 0;
  int pos = __reduce_add_sync(0xffffffffu, lane < wib ? v : 0) + inc - mine;
  const int nrow = __reduce_add_sync(0xffffffffu, v);
  if (nrow > cap) return false;
  const unsigned srows = (unsigned)__cvta_generic_to_shared(sm.rows);
#pragma unroll
  for (int i = 0; i < NC; i++) {
    if (co[i] >= 0) {
      sm.f[pos] = cf[i][0];
      sm.f[cap + pos] = cf[i][1];
      sm.f[2 * cap + pos] = cf[i][2];
      sm.meta[pos] = co[i];
      const unsigned slot = srows + pos * ST * (int)sizeof(T);
      sm.pre[pos] = make_int4(slot + (R::KX - ((co[i] & 127) - 32)) * (int)sizeof(T),
                              slot + (R::KY - (((co[i] >> 7) & 127) - 32)) * (int)sizeof(T),
                              slot + R::KZ * (int)sizeof(T), 0);
      *reinterpret_cast<C*>(sm.rows + pos * ST + R::KZ + NZ) = C{cv[i][0], cv[i][1]};
      pos++;
    }
  }
  __syncthreads();
  // kernel values, one (row, axis) per thread
  const int nb = (nrow + 31) >> 5;
  for (int u = wib; u < 3 * nb; u += WARPS) {
    const int axis = u >= 2 * nb ? 2 : (u >= nb ? 1 : 0);
    const int row = ((u - axis * nb) << 5) + lane;
    if (row < nrow) own_values<T, W, kPoly>(sm, row, axis, sm.f[axis * cap + row], (T)g.beta, (T)g.es_c);
  }
  __syncthreads();
  const int grp = lane >> 4, lx = lane & 7, ly = (lane >> 3) & 1;
  const int uy = wib / NUX * UY;
  int4* list = sm.list + wib * kOwnList;
  const unsigned zslot = srows + cap * ST * (int)sizeof(T);
  for (int ux = wib % NUX * kOwnUX; ux < nsub * kOwnTX; ux += kOwnTX) {
    const int x = tx0 + ux + lx, y = ty0 + uy + ly;  // this lane's first cell
    C* dst = fwc + (size_t)p0 * plane + (size_t)y * nf1 + x + (size_t)(2 * grp) * nf1;
    const bool wr = (CPL == 2 || grp == 0) && x < nf1 && y + 2 * grp < nf2;
    const unsigned offx = (ux + lx) * sizeof(T), offy = (uy + ly) * sizeof(T);
    const int4 dummy = make_int4(zslot + (R::KX - ux) * (int)sizeof(T), zslot + (R::KY - uy) * (int)sizeof(T),
                                 zslot + R::KZ * (int)sizeof(T), 0);
    OwnAcc<T, NZ, CPL> acc;
    acc.clear();
    int zc = 0, live = 0;
    auto advance = [&](int z) {  // as in own_tile
      for (; zc < z; zc++) {
        const int p = zc - hi - lo;
        C s = {(T)0, (T)0};
        if (zc < live) {
          T r0, i0, r1, i1;
          acc.first(0, r0, i0);
          acc.first(CPL - 1, r1, i1);
          s.x = (grp ? r1 : r0) + __shfl_xor_sync(0xffffffffu, grp ? r0 : r1, 16);
          s.y = (grp ? i1 : i0) + __shfl_xor_sync(0xffffffffu, grp ? i0 : i1, 16);
          acc.shift();
        }
        if (wr && p >= 0 && p < p1 - p0) dst[(size_t)p * plane] = s;
      }
    };
    auto spread = [&](int cnt) {
      if (lane == 0) list[cnt] = dummy;
      __syncwarp();
      live = zc + NZ;
      for (int j = grp; j - grp < cnt; j += 2) {
        const int4 e = list[j];
        acc.add(offx + e.x, offy + e.y, e.z);
      }
      __syncwarp();
    };
    int cnt = 0;
    for (int b = 0; b < nrow; b += 32) {
      const int row = b + lane;
      const int m = row < nrow ? sm.meta[row] : 0;
      const int ox = (m & 127) - 32, oy = ((m >> 7) & 127) - 32, z = m >> 14;
      const bool take = row < nrow && ox + W > ux && ox < ux + kOwnUX && oy + W > uy && oy < uy + UY;
      unsigned rem = __ballot_sync(0xffffffffu, take);
      while (rem) {
        const int zf = __shfl_sync(0xffffffffu, z, __ffs(rem) - 1);
        const bool now = take && z == zf;
        const unsigned sel = __ballot_sync(0xffffffffu, now);
        rem &= ~sel;
        if (zf != zc) {
          if (cnt) spread(cnt);
          cnt = 0;
          advance(zf);
        }
        if (now) list[cnt + __popc(sel & ((1u << lane) - 1u))] = sm.pre[row];
        cnt += __popc(sel);
        if (cnt > kOwnList - 33) {
          spread(cnt);
          cnt = 0;
        }
      }
    }
    if (cnt) spread(cnt);
    advance(p1 - p0 + lo + hi);
  }
  return true;
}

// Row split of heavy tiles.  A CTA grids a tile's rows alone, so a tile that
// holds far more than a CTA's share of the launch (the centre of a dense small
// grid) would set its length.  A tile with more than R rows in its hives and
// ring runs as ceil(rows / R) chunks into partial tiles, taken first from the
// queue; the CTA that ends a tile's last chunk sums them in chunk order, so the
// result does not depend on which CTA ran which chunk.
struct OwnSlot {
  int tile, chunk, nchunks, first;  // first: slot of the tile's chunk 0; tile < 0: unused
};
constexpr int kMaxTileChunks = 1024;

// One warp per tile: flags[t] = 1 and slots for a split tile.  counter[1] counts
// slots; a tile whose chunks end beyond cap is gridded whole.
__global__ void __launch_bounds__(256) k_own_split(const int* __restrict__ hive_start, Geom g, WarpTile tc, int R,
                                                   int cap, int* __restrict__ counter, int* __restrict__ flags,
                                                   OwnSlot* __restrict__ slots, int* __restrict__ done) {
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (t >= tc.nitems) return;
  const int tx0 = (tc.bx0 + t % tc.ntx) * kOwnTX, ty0 = (tc.by0 + (t / tc.ntx) % tc.nty) * kOwnTY;
  const int p0 = t / (tc.ntx * tc.nty) * tc.PB, p1 = min(p0 + tc.PB, g.nw);
  int flag = 0;
  if (tx0 <= g.band_c1 && tx0 + kOwnTX > g.band_c0 && ty0 <= g.band_r1 && ty0 + kOwnTY > g.band_r0) {
    const int lo = (g.kw - 1) / 2, hi = (g.kw + 1) / 2;
    const int tx1 = min(tx0 + kOwnTX, g.nf1), ty1 = min(ty0 + kOwnTY, g.nf2);
    const int hxa = raw_hive_lo(tx0 - hi, g.nf1, g.nhx), hxb = raw_hive_hi(tx1 - 1 + lo, g.nf1, g.nhx);
    const int hya = raw_hive_lo(ty0 - hi, g.nf2, g.nhy), ny = raw_hive_hi(ty1 - 1 + lo, g.nf2, g.nhy) - hya + 1;
    int rows = 0;
    for (int r = lane; r < ny * (p1 - p0 + lo + hi); r += 32) {
      const int64_t row = ((int64_t)wrapi(p0 - hi + r / ny, g.nw) * g.nhy + wrapi(hya + r % ny, g.nhy)) * g.nhx;
      rows += hive_start[row + min(hxb, g.nhx - 1) + 1] - hive_start[row + max(hxa, 0)];
      if (hxa < 0) rows += hive_start[row + g.nhx] - hive_start[row + g.nhx + hxa];
      if (hxb >= g.nhx) rows += hive_start[row + hxb - g.nhx + 1] - hive_start[row];
    }
    rows = __reduce_add_sync(0xffffffffu, rows);
    if (rows > R) {
      const int k = min((rows + R - 1) / R, kMaxTileChunks);
      int base = 0;
      if (lane == 0) base = atomicAdd(counter + 1, k);
      base = __shfl_sync(0xffffffffu, base, 0);
      flag = base + k <= cap;
      for (int c = lane; c < k && base + c < cap; c += 32) slots[base + c] = OwnSlot{flag ? t : -1, c, k, base};
      if (flag && lane == 0) done[base] = 0;
    }
  }
  if (lane == 0) flags[t] = flag;
}

// Cells [i0, n) step `step` of a split tile: the sum of its partial tiles
// (slot_cells apart, from `base`) in chunk order, into the grid.
template <typename T>
__device__ __forceinline__ void sum_chunks(const WarpTile& tc, const Geom& g, int item,
                                           const typename OwnC<T>::type* __restrict__ base, int nchunks,
                                           T* __restrict__ fw, int i0, int step) {
  using C = typename OwnC<T>::type;
  const int tix = tc.bx0 + item % tc.ntx, tiy = tc.by0 + (item / tc.ntx) % tc.nty, tib = item / (tc.ntx * tc.nty);
  const int tx0 = tix * kOwnTX, ty0 = tiy * kOwnTY, p0 = tib * tc.PB;
  const int wz = min(p0 + tc.PB, g.nw) - p0;
  const size_t slot = (size_t)kOwnTX * kOwnTY * tc.PB, plane = (size_t)g.nf1 * g.nf2;
  C* fwc = reinterpret_cast<C*>(fw);
  for (int i = i0; i < kOwnTX * kOwnTY * wz; i += step) {
    const int x = tx0 + i % kOwnTX, y = ty0 + i / kOwnTX % kOwnTY, z = i / (kOwnTX * kOwnTY);
    if (x >= g.nf1 || y >= g.nf2) continue;
    C s = __ldcg(base + i);
#pragma unroll 8
    for (int k = 1; k < nchunks; k++) {
      const C v = __ldcg(base + (size_t)k * slot + i);
      s.x += v.x;
      s.y += v.y;
    }
    fwc[(size_t)(p0 + z) * plane + (size_t)y * g.nf1 + x] = s;
  }
}

// counter[0]: queue head; counter[1]: chunk slots.  Items: the chunk slots
// below cap, then the tiles, or (kRest) those that k_grid_strip left: rest[0] tiles, from
// rest[1] on.
template <typename T, int W, bool kPoly, bool kRest>
__global__ void __launch_bounds__(OwnRow<T, W>::THREADS, OwnRow<T, W>::CTAS)
    k_grid_own(const Rec<T>* __restrict__ recs, const int* __restrict__ hive_start, Geom g, WarpTile tc,
               int rows_cap, T* __restrict__ fw, int* __restrict__ counter, const int* __restrict__ flags,
               const OwnSlot* __restrict__ slots, int* __restrict__ done, int cap,
               typename OwnC<T>::type* __restrict__ parts, const int* __restrict__ rest) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_warp[33], s_cnt[OwnRow<T, W>::WARPS], s_item;
  const OwnSmem<T> sm = own_smem<T, W, kPoly>(smem, rows_cap, geom_poly<T>(g));
  const int nslot = flags ? min(cap, counter[1]) : 0;
  const size_t slot_cells = (size_t)kOwnTX * kOwnTY * tc.PB;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(counter, 1);
    __syncthreads();
    int t = s_item;
    __syncthreads();
    OwnSlot sl{0, 0, 1, 0};
    typename OwnC<T>::type* part = nullptr;
    if (t < nslot) {
      sl = slots[t];
      if (sl.tile < 0) continue;
      part = parts + (size_t)t * slot_cells;
      t = sl.tile;
    } else {
      t -= nslot;
      if (t >= (kRest ? rest[0] : tc.nitems)) break;
      if constexpr (kRest) {
        t = rest[1 + t];
      } else {
        if (nslot && flags[t]) continue;  // gridded by its chunks
      }
    }
    own_tile<T, W, kPoly>(recs, hive_start, g, tc, fw, t, sm, s_warp, s_cnt, sl.chunk, sl.nchunks, part);
    if (part) {
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) s_item = atomicAdd(done + sl.first, 1);
      __syncthreads();
      const bool last = s_item == sl.nchunks - 1;
      __syncthreads();
      if (last) {
        __threadfence();
        sum_chunks<T>(tc, g, t, parts + (size_t)sl.first * slot_cells, sl.nchunks, fw, threadIdx.x,
                      OwnRow<T, W>::THREADS);
      }
    }
  }
}

// The strips of tiles; queue[0]: queue head; the tiles of a strip that does not fit are listed,
// queue[1] of them from queue[2] on, for k_grid_own (flags: those that run as chunks).
template <typename T, int W, bool kPoly>
__global__ void __launch_bounds__(OwnRow<T, W>::THREADS, OwnRow<T, W>::CTAS)
    k_grid_strip(const Rec<T>* __restrict__ recs, const int* __restrict__ hive_start, Geom g, WarpTile tc,
                 int rows_cap, T* __restrict__ fw, const int* __restrict__ flags, int* __restrict__ queue) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_warp[33], s_cnt[OwnRow<T, W>::WARPS], s_item;
  const OwnSmem<T> sm = own_smem<T, W, kPoly>(smem, rows_cap, geom_poly<T>(g));
  const int nsx = (tc.ntx + kOwnStrip - 1) / kOwnStrip;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(queue, 1);
    __syncthreads();
    const int strip = s_item;
    __syncthreads();
    if (strip >= nsx * tc.nty * tc.npb) break;
    const int t0 = strip / nsx * tc.ntx + strip % nsx * kOwnStrip, t1 = min(t0 + kOwnStrip, (strip / nsx + 1) * tc.ntx);
    bool whole = true;
    if (flags)
      for (int k = t0; k < t1; k++) whole &= !flags[k];
    if (whole && own_strip<T, W, kPoly>(recs, hive_start, g, tc, fw, strip, sm, s_warp, s_cnt)) continue;
    if (threadIdx.x == 0)
      for (int k = t0; k < t1; k++)
        if (!(flags && flags[k])) queue[2 + atomicAdd(queue + 1, 1)] = k;
  }
}

// Many grids in one persistent launch: CTAs take (job, tile) items from a
// global queue; every job shares W and the kernel.  Items [0, nsplit) are the
// row chunks of the heavy tiles (splits), the others the jobs' tiles in job
// order; a tile with split chunks is skipped there.
template <typename T, int W, bool kPoly>
__global__ void __launch_bounds__(OwnRow<T, W>::THREADS, OwnRow<T, W>::CTAS)
    k_grid_own_multi(const GridJob<T>* __restrict__ jobs, int njobs, int nitems, int rows_cap,
                     int* __restrict__ counter, const SplitItem* __restrict__ splits, int nsplit,
                     typename OwnC<T>::type* __restrict__ parts) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_warp[33], s_cnt[OwnRow<T, W>::WARPS], s_item;
  const OwnSmem<T> sm = own_smem<T, W, kPoly>(smem, rows_cap, geom_poly<T>(jobs[0].g));
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(counter, 1);
    __syncthreads();
    const int item = s_item;
    __syncthreads();
    if (item >= nsplit + nitems) break;
    int j, tile, chunk = 0, nchunks = 1;
    typename OwnC<T>::type* part = nullptr;
    if (item < nsplit) {
      const SplitItem si = splits[item];
      j = si.job;
      tile = si.tile;
      chunk = si.chunk;
      nchunks = si.nchunks;
      part = parts + si.off;
    } else {
      j = find_job(jobs, njobs, item - nsplit, [](const GridJob<T>& x) { return x.grid_item0; });
      tile = item - nsplit - jobs[j].grid_item0;
      if (jobs[j].tile_split && jobs[j].tile_split[tile]) continue;  // gridded by its split items
    }
    const GridJob<T>& J = jobs[j];
    own_tile<T, W, kPoly>(J.recs, J.hive_start, J.g, J.wt, J.fw, tile, sm, s_warp, s_cnt, chunk, nchunks,
                          part);
  }
}

// Sum of the partial tiles of each split tile (tiles[blockIdx.x]: chunk 0 of
// its nchunks, chunks at consecutive slots).
template <typename T>
__global__ void __launch_bounds__(256) k_split_reduce(const GridJob<T>* __restrict__ jobs,
                                                      const SplitItem* __restrict__ tiles,
                                                      const typename OwnC<T>::type* __restrict__ parts) {
  const SplitItem si = tiles[blockIdx.x];
  const GridJob<T>& J = jobs[si.job];
  sum_chunks<T>(J.wt, J.g, si.tile, parts + si.off, si.nchunks, J.fw, threadIdx.x, 256);
}

int device_sms() {
  static const int n = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    return cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess ? v : 148;
  }();
  return n;
}

// Row slots of a CTA: as many as leave CTAS CTAs on an SM, at most a chunk's
// candidates.  Fewer rows than candidates reach a tile (about half at W = 6),
// and a chunk that has more runs in passes.  It sets the order of the sums, so it is a
// function of the kernel and the table size alone.
template <typename T, int W>
int own_rows_cap(int slots, size_t* smem) {
  using R = OwnRow<T, W>;
  const size_t room = (size_t)(227 * 1024) / R::CTAS - 1280;
  int cap = R::THREADS * kOwnCand;
  while (cap > 64 && own_bytes<T, W>(cap, slots) > room) cap -= 16;
  *smem = own_bytes<T, W>(cap, slots);
  return cap;
}

template <typename T, int W>
int own_w(const Rec<T>* recs, const int* hive_start, int64_t M, const Geom& g, T* fw, int* counter,
          cudaStream_t st, const SplitScratch* sp) {
  using C = typename OwnC<T>::type;
  const WarpTile tc = warp_tiling(g);
  size_t smem;
  const int rows_cap = own_rows_cap<T, W>(tc.slots, &smem);
  // Strips where the rows that a strip lists, were they spread evenly over the data's
  // cells, about fit a chunk, and the strips are enough for every CTA to take several.
  // Tiles -> strips, rows a grid column: 4096 x 1024 images, FP32 W = 6, 0.03 rows 0.89 ->
  // 0.55 ms, 0.15 1.08 -> 0.81, 0.2 1.16 -> 1.17; FP64 W = 10 0.15 4.56 -> 3.82, 0.3 5.93 ->
  // 6.01.  Few strips: 1024^2, 30k rows 0.068 -> 0.080 (730 strips), 512^2, 20k 0.037
  // -> 0.103.  CG_GRID_STRIP=0 / 1 overrides.
  const int strips = (tc.ntx + kOwnStrip - 1) / kOwnStrip * tc.nty * tc.npb;
  const double listed = (double)M * (kOwnTX * kOwnStrip + W + 7) * (kOwnTY + W + 7) * (tc.PB + W) / g.nw /
                        ((double)(g.band_c1 - g.band_c0 + 1) * (g.band_r1 - g.band_r0 + 1));
  bool strip = listed <= 1.15 * OwnRow<T, W>::THREADS * kOwnCand && strips >= 4 * OwnRow<T, W>::CTAS * device_sms();
  if (const char* e = getenv("CG_GRID_STRIP")) strip = atoi(e) != 0;
  strip = strip && sp;
  auto* kern = geom_poly_host<T>(g) ? (strip ? k_grid_own<T, W, true, true> : k_grid_own<T, W, true, false>)
                                    : (strip ? k_grid_own<T, W, false, true> : k_grid_own<T, W, false, false>);
  auto* skern = geom_poly_host<T>(g) ? k_grid_strip<T, W, true> : k_grid_strip<T, W, false>;
  int per_sm = 0;
  if (strip) CG_CUDA(kernel_occupancy((const void*)skern, OwnRow<T, W>::THREADS, smem, &per_sm));
  CG_CUDA(kernel_occupancy((const void*)kern, OwnRow<T, W>::THREADS, smem, &per_sm));
  if (per_sm < 1) {
    set_last_error("gridding does not fit on an SM");
    return CG_ERR_ARG;
  }
  const int blocks = per_sm * device_sms();
  // R: about half a CTA's share (a row is in about 4 tiles' hives and rings),
  // so that the last CTA ends soon after the others; at least 2048 rows, some
  // 50 us of a CTA's work, below which a chunk's fixed cost (segment table, all
  // planes of a partial tile written and summed) is no longer small beside it.
  // The chunks of all tiles above R are at most 2 / R times the rows that the
  // tiles list (M, times the tiles that share a hive, 4, and a plane); R is raised
  // until they fit 128 MB of partial tiles, so that which tiles split never
  // depends on the order in which they ask for slots.
  // CG_SPLIT=0 turns the split off, CG_SPLIT_ROWS sets R.
  int* flags = nullptr;
  OwnSlot* slots = nullptr;
  int* done = nullptr;
  int* queue = nullptr;  // of the strips, and the tiles that they leave
  C* parts = nullptr;
  int cap = 0;
  int64_t R = 0;
  const size_t nf = ((size_t)tc.nitems * sizeof(int) + 15) & ~(size_t)15;
  const char* off = getenv("CG_SPLIT");
  if (sp && M > 0 && !(off && atoi(off) == 0)) {
    const size_t slot_bytes = (size_t)tc.TX * tc.TY * tc.PB * sizeof(C);
    const int64_t most = std::max<int64_t>(64, ((int64_t)128 << 20) / (int64_t)slot_bytes);
    // hives and rings of an axis's tiles over its hives: 2 on long axes
    auto times = [](int nf, int nh) { return (4.0 * ((nf + kOwnTX - 1) / kOwnTX) + (nf % 8 ? 2 : 0)) / nh; };
    const double twice = 2.0 * times(g.nf1, g.nhx) * times(g.nf2, g.nhy) * tc.npb * (tc.PB + W + 1) / g.nw;
    R = std::max<int64_t>(2048, 2 * M / blocks);
    R = std::max<int64_t>(R, (int64_t)(twice * (double)M / (double)most));
    if (const char* e = getenv("CG_SPLIT_ROWS")) R = std::max<int64_t>(1, atoll(e));
    if (M > R) {
      cap = (int)std::min<double>((double)most, twice * (double)M / (double)R + 1);
      CG_TRY(ensure(*sp->parts, (size_t)cap * slot_bytes));
      parts = (C*)sp->parts->p;
    }
  }
  if (cap || strip) {
    // flags, chunk slots, chunks done, then the strips' queue and list
    const size_t chunks = cap ? nf + (size_t)cap * (sizeof(OwnSlot) + sizeof(int)) : 0;
    CG_TRY(ensure(*sp->slots, chunks + (strip ? 2 * sizeof(int) + nf : 0)));
    if (strip) queue = (int*)((char*)sp->slots->p + chunks);
    if (cap) {
      flags = (int*)sp->slots->p;
      slots = (OwnSlot*)((char*)sp->slots->p + nf);
      done = (int*)(slots + cap);
    }
  }
  CG_CUDA(cudaMemsetAsync(counter, 0, 2 * sizeof(int), st));
  if (flags) {
    k_own_split<<<(tc.nitems + 7) / 8, 256, 0, st>>>(hive_start, g, tc, (int)std::min<int64_t>(R, 2147483647),
                                                         cap, counter, flags, slots, done);
    count_launches(1);
    CG_CUDA(cudaGetLastError());
  }
  if (strip) {
    CG_CUDA(cudaMemsetAsync(queue, 0, 2 * sizeof(int), st));
    skern<<<std::min(blocks, strips), OwnRow<T, W>::THREADS, smem, st>>>(recs, hive_start, g, tc, rows_cap, fw, flags,
                                                                        queue);
    count_launches(1);
    CG_CUDA(cudaGetLastError());
  }
  kern<<<std::min(blocks, tc.nitems + cap), OwnRow<T, W>::THREADS, smem, st>>>(
      recs, hive_start, g, tc, rows_cap, fw, counter, flags, slots, done, cap, parts, strip ? queue + 1 : nullptr);
  count_launches(1);
  CG_CUDA(cudaGetLastError());
  return CG_OK;
}

template <typename T, int W>
int own_multi_w(const GridJob<T>* d_jobs, int njobs, const MultiShape& sh, int* counter, cudaStream_t st) {
  using C = typename OwnC<T>::type;
  size_t smem;
  const int rows_cap = own_rows_cap<T, W>(sh.grid_slots, &smem);
  auto* kern = sh.poly ? k_grid_own_multi<T, W, true> : k_grid_own_multi<T, W, false>;
  int per_sm = 0;
  CG_CUDA(kernel_occupancy((const void*)kern, OwnRow<T, W>::THREADS, smem, &per_sm));
  if (per_sm < 1) {
    set_last_error("multi-grid gridding does not fit on an SM");
    return CG_ERR_ARG;
  }
  const int blocks = std::min(sh.grid_items + sh.nsplit, per_sm * device_sms());
  CG_CUDA(cudaMemsetAsync(counter, 0, sizeof(int), st));
  kern<<<std::max(1, blocks), OwnRow<T, W>::THREADS, smem, st>>>(d_jobs, njobs, sh.grid_items, rows_cap, counter,
                                                                sh.d_split, sh.nsplit, (C*)sh.d_parts);
  count_launches(1);
  CG_CUDA(cudaGetLastError());
  if (sh.nsplit_tiles > 0) {
    k_split_reduce<T><<<sh.nsplit_tiles, 256, 0, st>>>(d_jobs, sh.d_split_tiles, (const C*)sh.d_parts);
    count_launches(1);
    CG_CUDA(cudaGetLastError());
  }
  return CG_OK;
}

}  // namespace

template <typename T>
int launch_grid_own(const Rec<T>* recs, const int* hive_start, int64_t M, const Geom& g, T* fw, int* counter,
                    cudaStream_t st, const SplitScratch* sp) {
#define CG_OWN_CALL(w) own_w<T, w>(recs, hive_start, M, g, fw, counter, st, sp)
  CG_W_SWITCH(g.kw, CG_OWN_CALL)
#undef CG_OWN_CALL
}

template <typename T>
int launch_grid_multi(const GridJob<T>* d_jobs, int njobs, const MultiShape& sh, int* d_counter,
                      cudaStream_t st) {
  if (njobs < 1 || sh.grid_items < 1) return CG_OK;
#define CG_OWN_MULTI_CALL(w) own_multi_w<T, w>(d_jobs, njobs, sh, d_counter, st)
  CG_W_SWITCH(sh.kw, CG_OWN_MULTI_CALL)
#undef CG_OWN_MULTI_CALL
}

// FP32 here, FP64 in a translation unit of its own (cg_grid_own_f64.cu), so that the two
// compile side by side
#ifdef CG_OWN_FP64
using OwnT = double;
#else
using OwnT = float;
#endif
template int launch_grid_own<OwnT>(const Rec<OwnT>*, const int*, int64_t, const Geom&, OwnT*, int*, cudaStream_t,
                                   const SplitScratch*);
template int launch_grid_multi<OwnT>(const GridJob<OwnT>*, int, const MultiShape&, int*, cudaStream_t);

}  // namespace cg
