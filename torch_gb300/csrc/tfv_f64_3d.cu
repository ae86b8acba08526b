// Double-precision 3D step kernels (see tfv_f64.cu; a unit of its own so that
// the two compile in parallel).
#define REAL double
// 128 registers: two 256-thread CTAs per SM.  The integer sequences of
// tfv_soft64.cuh are latency-bound, so 16 resident warps beat 8 without spills
// (160^3: 8.28 against 9.13 ms per step; 2D 1024^2: 1.05 against 1.13).
#define TFV_HYDRO_MIN_BLOCKS 2
#define TFV_FIXED_SHAPES 0
#define TFV_WITH_2D 0
#define TFV_WITH_3D 1
#define TFV_LAUNCH3_NAME launch_step3_f64
#define TFV_WITH_1D 0
#define TFV_STEP1D_MIN_BLOCKS 1
#define TFV_CHECK_READ_NAME check_read_f64_3d
#define TFV_OCC3_NAME occupancy3_f64
#include "tfv_inst.inc"
