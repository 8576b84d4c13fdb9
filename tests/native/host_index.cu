// Host functions of the kernels' index arithmetic, exported for the CPU tests.
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

}
