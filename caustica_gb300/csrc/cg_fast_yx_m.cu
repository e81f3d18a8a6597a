// Size-specialised y-/x-pass launchers for lengths 324, 360.
#include "cg_fast_yx.cuh"

CG_YX_INSTANTIATE(324)
CG_YX_INSTANTIATE(360)
