// Double-precision 1D and 2D step kernels (3D: tfv_f64_3d.cu) and the finalize
// kernel: the reference-faithful path.  Built with
// -fmad=false so every product and sum rounds separately, as in NumPy.
#define REAL double
#define TFV_DEFINE_SHARED_KERNELS
// 128 registers: two 256-thread CTAs per SM.  The integer sequences of
// tfv_soft64.cuh are latency-bound, so 16 resident warps beat 8 without spills
// (160^3: 8.28 against 9.13 ms per step; 2D 1024^2: 1.05 against 1.13).
#define TFV_HYDRO_MIN_BLOCKS 2
#define TFV_FIXED_SHAPES 0
#define TFV_WITH_2D 1
#define TFV_WITH_3D 0
#define TFV_LAUNCH2_NAME launch_step2_f64
#define TFV_HLLC_NAME launch_hllc_f64
#define TFV_WITH_1D 1
#define TFV_STEP1D_MIN_BLOCKS 2
#define TFV_LAUNCH1_NAME launch_step1_f64
#define TFV_CHECK_READ_NAME check_read_f64
#define TFV_OCC2_NAME occupancy2_f64
#include "tfv_inst.inc"

namespace tfv {
cudaError_t launch_finalize(const StepArgs& A, int mode, int fp32, double* integrals_out,
                            cudaStream_t s) {
  const dim3 grid(A.fin_slices > 0 ? A.fin_slices : 1, A.ninst);
  return launch_pdl(finalize_kernel, grid, kFinalizeThreads, 0, s, A, mode, fp32, integrals_out);
}
}  // namespace tfv
