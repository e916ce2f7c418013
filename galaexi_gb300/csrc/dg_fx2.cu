// Fixed-point kernels of the FP64 form for N = 1 (N+1 = 2 nodes per direction).
#define GX_NP 2
#include "dg_fx_np.cuh"
