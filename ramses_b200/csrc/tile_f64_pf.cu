// The instances of tile_f64.cu with pressure_fix (compiled the same way).
#define RB_TILE_REAL double
#define RB_TILE_PF true
#define RB_TILE_LAUNCH launch_tile_f64_pf
#include "tile_instances.inc"
