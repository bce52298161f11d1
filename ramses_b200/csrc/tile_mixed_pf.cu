// The instances of tile_mixed.cu with pressure_fix (compiled the same way).
#define RB_TILE_REAL float
#define RB_TILE_PF true
#define RB_TILE_LAUNCH launch_tile_mixed_pf
#include "tile_instances.inc"
