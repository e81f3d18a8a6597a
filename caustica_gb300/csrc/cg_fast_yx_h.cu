// Size-specialised y-/x-pass launchers for lengths 80, 81, 90, 100, 108.
#include "cg_fast_yx.cuh"

CG_YX_INSTANTIATE(80)
CG_YX_INSTANTIATE(81)
CG_YX_INSTANTIATE(90)
CG_YX_INSTANTIATE(100)
CG_YX_INSTANTIATE(108)
