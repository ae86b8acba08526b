// Single-precision 2D step kernels (see tfv_f32_3d.cu).
#define REAL float
// 64 registers: eight of the default tile's 128-thread CTAs per SM.  The step is
// bound by latency and instruction issue: the packed fluxes leave 28 B of
// spills (32 grids of 64^2 to 1024^2, ten steps: 4.85 ms with 80 registers and
// six CTAs, 4.65 with 64, 5.09 with 48).
#define TFV_HYDRO_MIN_BLOCKS 4
#define TFV_FIXED_SHAPES 1
#define TFV_WITH_2D 1
#define TFV_WITH_3D 0
#define TFV_LAUNCH2_NAME launch_step2_f32
#define TFV_WITH_1D 1
#define TFV_STEP1D_MIN_BLOCKS 4
#define TFV_LAUNCH1_NAME launch_step1_f32
#define TFV_CHECK_READ_NAME check_read_f32_2d
#define TFV_OCC2_NAME occupancy2_f32
#include "tfv_inst.inc"
