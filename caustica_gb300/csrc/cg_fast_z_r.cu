// Persistent z-pass launchers for lengths 384.
#include "cg_fast_z.cuh"

CG_ZP_INSTANTIATE(384)
