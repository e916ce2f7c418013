// Fixed-point kernels of the FP64 form for N = 7 (N+1 = 8 nodes per direction).
#define GX_NP 8
#include "dg_fx_np.cuh"
