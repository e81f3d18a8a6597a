// Persistent z-pass launchers for lengths 243, 250.
#include "cg_fast_z.cuh"

CG_ZP_INSTANTIATE(243)
CG_ZP_INSTANTIATE(250)
