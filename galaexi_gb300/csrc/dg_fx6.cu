// Fixed-point kernels of the FP64 form for N = 5 (N+1 = 6 nodes per direction).
#define GX_NP 6
#include "dg_fx_np.cuh"
