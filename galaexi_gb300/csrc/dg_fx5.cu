// Fixed-point kernels of the FP64 form for N = 4 (N+1 = 5 nodes per direction).
#define GX_NP 5
#include "dg_fx_np.cuh"
