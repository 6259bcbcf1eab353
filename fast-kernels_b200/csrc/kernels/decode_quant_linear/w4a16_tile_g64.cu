// The tile kernel for groups of 64.
#define FK_TILE_GROUP 64
#include "w4a16_tile_launch.inc"
