// Launch geometry of the tile kernel (w4a16_gemm_tile.cuh), shared by host planning and device code.
#pragma once

#include "w4a16_common.cuh"

namespace fk_w4a16 {

constexpr int kTileK = 128;            // features of a step: 1, 2 or 4 quantisation groups
constexpr int kTilePair = 2;           // weight tiles of a step: 256 output columns
constexpr int kTileMaxRows = 128;      // batch rows of one pass
constexpr int kTileThreads = 640;      // producer, issuers | 2 unpack warpgroups | 2 promote warpgroups
constexpr int kTileABuffers = 4;       // unpacked weight tiles in tensor memory, 64 columns each
constexpr int kTileDColumn0 = kTileABuffers * 64;
constexpr int kTileDColumns = 256;     // the rest of tensor memory holds accumulators
constexpr int kTileMaxStages = 8;
constexpr int kTileBarrierBytes = 512;

__host__ __device__ constexpr int tile_groups(int group) { return kTileK / group; }
// Above 64 rows a group's accumulators are made in two halves with a buffer each, so that one half
// is read out while the other is multiplied.
__host__ __device__ constexpr int tile_halves(int rows) { return rows > 64 ? 2 : 1; }
__host__ __device__ constexpr int tile_half_rows(int rows) { return rows > 64 ? 64 : rows; }
// Groups whose accumulators share one buffer (and one barrier hand-over): up to 128 columns.
__host__ __device__ constexpr int tile_unit_groups(int group, int rows) {
  const int fit = tile_halves(rows) > 1 ? 1 : 128 / rows;
  return tile_groups(group) < fit ? tile_groups(group) : fit;
}
__host__ __device__ constexpr int tile_d_buffers(int group, int rows) {
  const int fit = kTileDColumns / (tile_unit_groups(group, rows) * tile_half_rows(rows));
  return fit < 4 ? fit : 4;
}
// Staged activations of one (row tile, 128-feature block): operand B, then the group sums.
__host__ __device__ constexpr int tile_block_bytes(int group, int rows) {
  return (rows * kTileK * 2) + (tile_groups(group) * rows * 4);
}
__host__ __device__ constexpr int tile_weight_bytes(int group) {
  return kTilePair * tile_groups(group) * packet_stride(group);
}
__host__ __device__ constexpr int tile_stage_bytes(int group, int rows) {
  return (tile_weight_bytes(group) + tile_block_bytes(group, rows) + 127) & ~127;
}
// Rows of a pass for which a kernel is instantiated.
__host__ __device__ constexpr int tile_rows_template(int rows) {
  return rows <= 16 ? 16 : (rows <= 32 ? 32 : (rows <= 64 ? 64 : 128));
}

}  // namespace fk_w4a16
