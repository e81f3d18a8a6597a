// Size-specialised y-/x-pass launchers for lengths 225, 240, 243, 250.
#include "cg_fast_yx.cuh"

CG_YX_INSTANTIATE(225)
CG_YX_INSTANTIATE(240)
CG_YX_INSTANTIATE(243)
CG_YX_INSTANTIATE(250)
