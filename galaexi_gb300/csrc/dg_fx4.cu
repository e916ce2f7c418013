// Fixed-point kernels of the FP64 form for N = 3 (N+1 = 4 nodes per direction).
#define GX_NP 4
#include "dg_fx_np.cuh"
