// Persistent z-pass launchers for lengths 300, 324.
#include "cg_fast_z.cuh"

CG_ZP_INSTANTIATE(300)
CG_ZP_INSTANTIATE(324)
