// Persistent z-pass launchers for lengths 200, 216.
#include "cg_fast_z.cuh"

CG_ZP_INSTANTIATE(200)
CG_ZP_INSTANTIATE(216)
