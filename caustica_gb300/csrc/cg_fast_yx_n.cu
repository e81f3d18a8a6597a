// Size-specialised y-/x-pass launchers for lengths 375, 384.
#include "cg_fast_yx.cuh"

CG_YX_INSTANTIATE(375)
CG_YX_INSTANTIATE(384)
