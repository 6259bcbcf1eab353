// Interface between the C-ABI translation unit and the kernels compiled in other units.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace fk_w4a16 {

struct GemvParams;

struct UmmaLaunch {
  int group_size;   // 32, 64 or 128
  int rows;         // rows per pass: 1, 2, 4, 8 or 16
  bool bf16;
  int grid_x;       // CTAs = runs of the packet stream
  int row_tiles;
  size_t smem_bytes;
  int max_smem;     // opt-in limit of the device
  bool programmatic;  // launch with programmatic stream serialisation
  cudaStream_t stream;
};

// The pipelined tcgen05 / tensor-memory kernel (w4a16_gemm_umma.cuh).
cudaError_t launch_umma_kernel(const GemvParams& params, const UmmaLaunch& launch);

struct TileLaunch {
  bool bf16;
  int rows;              // rows of a pass, a multiple of 16
  int row_tiles;
  uint32_t blocks;       // steps of a unit
  uint32_t total_steps;
  int ctas;
  int stages;
  size_t smem_bytes;
  int max_smem;
  uint8_t* staged;
  float* slots;
  bool programmatic;
  cudaStream_t stream;
};

// The activation prepass and the tile kernel (w4a16_gemm_tile.cuh) for groups of G.
template <int G>
cudaError_t launch_tile_kernel(const GemvParams& params, const TileLaunch& launch);
template <>
cudaError_t launch_tile_kernel<32>(const GemvParams& params, const TileLaunch& launch);
template <>
cudaError_t launch_tile_kernel<64>(const GemvParams& params, const TileLaunch& launch);
template <>
cudaError_t launch_tile_kernel<128>(const GemvParams& params, const TileLaunch& launch);

}  // namespace fk_w4a16
