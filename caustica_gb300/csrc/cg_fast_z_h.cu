// Persistent z-pass launchers for lengths 72, 75, 80, 81, 90.
#include "cg_fast_z.cuh"

CG_ZP_INSTANTIATE(72)
CG_ZP_INSTANTIATE(75)
CG_ZP_INSTANTIATE(80)
CG_ZP_INSTANTIATE(81)
CG_ZP_INSTANTIATE(90)
