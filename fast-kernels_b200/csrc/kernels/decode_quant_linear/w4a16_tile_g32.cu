// The tile kernel for groups of 32.
#define FK_TILE_GROUP 32
#include "w4a16_tile_launch.inc"
