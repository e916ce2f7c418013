// Fixed-point kernels of the FP64 form for N = 2 (N+1 = 3 nodes per direction).
#define GX_NP 3
#include "dg_fx_np.cuh"
