// Persistent z-pass launchers for lengths 225, 240.
#include "cg_fast_z.cuh"

CG_ZP_INSTANTIATE(225)
CG_ZP_INSTANTIATE(240)
