// Size-specialised y-/x-pass launchers for lengths 162, 180, 200, 216.
#include "cg_fast_yx.cuh"

CG_YX_INSTANTIATE(162)
CG_YX_INSTANTIATE(180)
CG_YX_INSTANTIATE(200)
CG_YX_INSTANTIATE(216)
