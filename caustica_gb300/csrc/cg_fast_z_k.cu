// Persistent z-pass launchers for lengths 150, 162, 180.
#include "cg_fast_z.cuh"

CG_ZP_INSTANTIATE(150)
CG_ZP_INSTANTIATE(162)
CG_ZP_INSTANTIATE(180)
