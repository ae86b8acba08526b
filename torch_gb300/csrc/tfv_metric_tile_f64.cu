// Tiled metric kernels, double precision (built with -fmad=false: the
// reference's rounding), and the reduction of their tile records.
#define TFV_METRIC_R double
#define TFV_STAGE_MIN_BLOCKS 1
#define TFV_METRIC_TILE_LAUNCH metric_tile_launch_f64
#include "tfv_metric_tile_inst.inc"

namespace tfv {
namespace {
// out[stage][row] = sum over the tiles of part[stage][tile][row], one CTA per
// value, in a fixed order
__global__ void __launch_bounds__(256) tile_reduce_kernel(const double* part, int ntiles,
                                                          double* out) {
  __shared__ double red[32];
  pdl_wait();
  const int row = blockIdx.x % 16, stage = blockIdx.x / 16;
  if (row > 4 && (row < 8 || row > 12)) return;
  const double* p = part + (size_t)stage * ntiles * 16 + row;
  double s = 0.0;
  for (int t = threadIdx.x; t < ntiles; t += blockDim.x) s += p[(size_t)t * 16];
  const double sum = block_sum(s, red);
  if (threadIdx.x == 0) out[blockIdx.x] = sum;
}
}  // namespace
cudaError_t metric_tile_reduce(const double* part, int ntiles, double* out, cudaStream_t s) {
  return launch_pdl(tile_reduce_kernel, 32, 256, 0, s, part, ntiles, out);
}
}  // namespace tfv
