// Tiled metric kernels, single precision.
#define TFV_METRIC_R float
#define TFV_STAGE_MIN_BLOCKS 2
#define TFV_METRIC_TILE_LAUNCH metric_tile_launch_f32
#include "tfv_metric_tile_inst.inc"
