// FP64 drop-in instances of the z-streaming kernels. Compiled with
// --fmad=false, as tile_f64.cu.
#define RB_TILE_REAL double
#define RB_TILE_IS_MIXED 0
#define RB_STREAM_LAUNCH launch_stream_f64
#define RB_STREAM_SMEM stream_smem_f64
#define RB_BATCH_LAUNCH launch_batch_f64
#include "stream_instances.inc"
