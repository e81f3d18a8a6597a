// Persistent z-pass launchers for lengths 125, 135, 144.
#include "cg_fast_z.cuh"

CG_ZP_INSTANTIATE(125)
CG_ZP_INSTANTIATE(135)
CG_ZP_INSTANTIATE(144)
