// The FP64 instances of cg_grid_own.cu.
#define CG_OWN_FP64
#include "cg_grid_own.cu"
