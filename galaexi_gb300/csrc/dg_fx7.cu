// Fixed-point kernels of the FP64 form for N = 6 (N+1 = 7 nodes per direction).
#define GX_NP 7
#include "dg_fx_np.cuh"
