// Size-specialised y-/x-pass launchers for lengths 270, 288, 300.
#include "cg_fast_yx.cuh"

CG_YX_INSTANTIATE(270)
CG_YX_INSTANTIATE(288)
CG_YX_INSTANTIATE(300)
