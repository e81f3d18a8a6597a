// Size-specialised y-/x-pass launchers for lengths 120, 125, 135, 144, 150.
#include "cg_fast_yx.cuh"

CG_YX_INSTANTIATE(120)
CG_YX_INSTANTIATE(125)
CG_YX_INSTANTIATE(135)
CG_YX_INSTANTIATE(144)
CG_YX_INSTANTIATE(150)
