// Host functions of the kernels' index arithmetic, exported for the CPU tests.
#include <vector>

#include "cg_band_shape.cuh"
#include "cg_tiles.cuh"

extern "C" {

// slots of a gridding tile's segment table, planes of an item
void t_grid_tiling(int nf1, int nf2, int nw, int kw, int* slots, int* planes) {
  cg::Geom g{};
  g.nf1 = nf1;
  g.nf2 = nf2;
  g.nw = nw;
  g.kw = kw;
  g.band_r1 = nf2 - 1;
  g.band_c1 = nf1 - 1;
  const cg::WarpTile tc = cg::warp_tiling(g);
  *slots = tc.slots;
  *planes = tc.PB;
}

int t_raw_hive_lo(int a, int nf, int nh) { return cg::raw_hive_lo(a, nf, nh); }
int t_raw_hive_hi(int b, int nf, int nh) { return cg::raw_hive_hi(b, nf, nh); }


// Shape of a band transform: false where it does not apply.  v: H, n, NB, apart, threads,
// shared-memory bytes, m0, delta, passes, then each pass's radix and table offset.
static bool shape(cg::band::BandFft& a, int L, int i0, int ni, int o0, int no, int rows, int esz, int* threads,
                  size_t* smem) {
  a = cg::band::BandFft{};
  a.L = L;
  a.i0 = i0;
  a.ni = ni;
  a.o0 = o0;
  a.no = no;
  return cg::band::band_shape(a, rows != 0, esz, threads, smem);
}

int t_band_shape(int L, int i0, int ni, int o0, int no, int rows, int esz, int* v) {
  cg::band::BandFft a;
  int threads;
  size_t smem;
  if (!shape(a, L, i0, ni, o0, no, rows, esz, &threads, &smem)) return 0;
  const int head[9] = {a.H, a.n, a.NB, a.apart, threads, (int)smem, a.m0, a.delta, a.npass};
  for (int i = 0; i < 9; i++) *v++ = head[i];
  for (int i = 0; i < a.npass; i++) {
    *v++ = a.pass[i].R;
    *v++ = a.pass[i].tw;
  }
  return 1;
}

// The kernel's shared-memory indices of every pass and butterfly: 0, or the number of the
// check that fails (1 a pass's stride, 2 out of the line's space, 3 two positions in one
// place, 4 output blocks, 5 butterfly and line indices, 6 the stash, 7 the twiddle table);
// -1 where the shape does not apply.
int t_band_check(int L, int i0, int ni, int o0, int no, int rows, int esz) {
  using namespace cg::band;
  BandFft a;
  int threads;
  size_t smem;
  if (!shape(a, L, i0, ni, o0, no, rows, esz, &threads, &smem)) return -1;
  const int pts = rows ? a.cs : a.stash / a.NB;
  std::vector<char> used(pts, 0), block(a.n / a.pass[a.npass - 1].R, 0);
  for (int i = 0; i < a.n; i++) {
    const int p = padded_at(a, i);
    if (p < 0 || p >= pts) return 2;
    if (used[p]++) return 3;
  }
  int tw = a.L;
  for (int i = 0; i < a.npass; i++) {
    const BandPass& ps = a.pass[i];
    if (ps.tw != tw) return 7;
    tw += ps.blk;
    if (ps.R * ps.sub != ps.blk || ps.R * ps.nbf != a.n || ps.total != ps.nbf * a.NB) return 5;
    for (int b = 0; b < ps.total; b++)
      if (rows ? div_by(b, ps.mnbf, ps.nbf) != b / ps.nbf : (b >> a.logNB) != b / a.NB) return 5;
    for (int bf = 0; bf < ps.nbf; bf++) {
      const int blkid = div_by(bf, ps.msub, ps.sub);
      if (blkid != bf / ps.sub) return 5;
      int base = i == 0 ? bf : blkid * ps.blk + bf - blkid * ps.sub;
      if (i == a.npass - 1) {
        const int k = block_of(a, bf);
        if (k < 0 || k >= (int)block.size() || block[k]++) return 4;
        base = k * ps.R;
      }
      for (int m = 0; m < ps.R; m++)
        if (padded_at(a, base) * a.js + m * ps.step != padded_at(a, base + m * ps.sub) * a.js) return 1;
    }
  }
  if ((size_t)a.stash * esz > smem) return 2;
  if (a.H == 2 && !a.apart && (size_t)(a.stash + (((a.no - 1) >> 1) << a.logNB) + a.NB) * esz > smem) return 6;
  return 0;
}

}
