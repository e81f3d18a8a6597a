// Persistent z-pass launchers for lengths 360, 375.
#include "cg_fast_z.cuh"

CG_ZP_INSTANTIATE(360)
CG_ZP_INSTANTIATE(375)
