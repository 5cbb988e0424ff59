// FP32-bulk ensemble kernels, compiled like kernels_fp32.cu (--use_fast_math).
#ifdef MGPU_FLUX_MINB_OVERRIDE
#define MGPU_FLUX_MINB MGPU_FLUX_MINB_OVERRIDE
#else
#define MGPU_FLUX_MINB 5
#endif
// HLLD sweeps (rmhd_face32.cuh) at 6 blocks, 80 registers: 160^3 lean sweeps per RK3 step 3.82 /
// 3.34 / 3.29 ms (PLM) and 5.80 / 4.86 / 4.75 ms (WENO5) at 4 / 5 / 6 blocks
#ifndef MGPU_HLLD_MINB
#define MGPU_HLLD_MINB 6
#endif
// zone c2p at 8 blocks, 64 registers (the FP64 state is live only through two or three Newton
// steps): 160^3 lean c2p per RK3 step 0.74 / 0.68 / 0.64 / 0.62 ms at 5 / 6 / 7 / 8 blocks
#ifdef MGPU_C2P_MINB_OVERRIDE
#define MGPU_C2P_MINB MGPU_C2P_MINB_OVERRIDE
#else
#define MGPU_C2P_MINB 8
#endif
#ifdef MGPU_TC_CTAS_OVERRIDE
#define MGPU_TC_CTAS_PER_SM MGPU_TC_CTAS_OVERRIDE
#endif
#include "c2p_mlp.cuh"
#include "rmhd_ensemble.cuh"
MGPU_DEFINE_ENSEMBLE(fp32, float)
