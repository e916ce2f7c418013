// Fixed-point kernels of the FP64 form for N = 8 (N+1 = 9 nodes per direction).
#define GX_NP 9
#include "dg_fx_np.cuh"
