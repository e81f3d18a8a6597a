// Persistent z-pass launchers for lengths 270, 288.
#include "cg_fast_z.cuh"

CG_ZP_INSTANTIATE(270)
CG_ZP_INSTANTIATE(288)
