// The tile kernel for groups of 128.
#define FK_TILE_GROUP 128
#include "w4a16_tile_launch.inc"
