// Persistent z-pass launchers for lengths 100, 108, 120.
#include "cg_fast_z.cuh"

CG_ZP_INSTANTIATE(100)
CG_ZP_INSTANTIATE(108)
CG_ZP_INSTANTIATE(120)
