// FP32-mixed instances of the z-streaming kernels (compiled as tile_mixed.cu).
#define RB_TILE_REAL float
#define RB_TILE_IS_MIXED 1
#define RB_STREAM_LAUNCH launch_stream_mixed
#define RB_STREAM_SMEM stream_smem_mixed
#define RB_BATCH_LAUNCH launch_batch_mixed
#include "stream_instances.inc"
