// Batches on the fifth-generation tensor cores, up to 128 rows a pass: one read of the weights
// serves the whole batch, and the multiply-adds cost no issue slots.
//
// What bounds it: the hand-overs between its roles. A tcgen05.mma kind::f16 of M = 128 takes ~45 clocks
// for every N up to 64; a step of 128 features x 256 output columns is 16 of them up to 64 rows, 720
// clocks against ~770 clocks of HBM time for its 17 KB of packets, and 32 above (two halves of at most
// 64 rows), 1440 clocks. A step takes ~2000 clocks up to 32 rows, where unpack -> MMA -> unpack is a chain
// through two buffers per tile, ~2800 at 64 rows, and ~4200 at 128, where MMA -> promote -> MMA is one.
// The passes of 16 rows on mma.sync that this replaces pay one whole read and unpack of the layer per
// 16 rows. Measured on 28672 x 8192, bf16, per call: 51 / 57 / 68 / 108 / 204 us at 16 / 32 / 64 / 128 /
// 256 rows (58 / 112 / 221 / 437 / 862 in passes of 16).
//
// Exactness. The unpacked operand is q - 8, exact in bf16 and in fp16, against the activations as
// they are; every quantisation group has an accumulator of its own in tensor memory, and the
// group's scale and offset enter in fp32: y += alpha * D_g + (beta + 8 alpha) * S_g, S_g = sum of
// the group's activations in fp32. Weights are never rounded to 16 bits, and no large constant has
// to cancel (the mma.sync form multiplies 128 + q or 1024 + 16 q).
//
// Work split. A unit is 256 output columns (two packet tiles) x one row tile; its K dimension is
// cut into steps of 128 features, and the steps of all units, unit after unit, into one contiguous
// run per CTA. Two weight tiles share a step's activations, which halves what every SM reads of them
// from L2. A unit that several CTAs share is finished by the last of them through workspace slots,
// added in CTA order: results do not depend on timing.
//
// Roles (640 threads, one CTA per SM, all of its tensor memory; every wait is bounded):
//   producer  1 thread     bulk copies of a step: two packet runs, one block of staged activations
//   issuers   2 threads    G/16 MMAs per group, one thread per tile: A (weights) from tensor
//                          memory, B (activations) from shared memory
//   unpack    2 x 128      warpgroup e unpacks tile e: thread c = column c = TMEM lane c
//   promote   2 x 128      warpgroup e folds tile e's accumulators into fp32 registers, a column per
//                          thread, two rows per packed FMA; stores finished columns
// With 64 to 128 accumulators per thread the promote warps need more registers than an even split
// of the file gives: instances of 64 and 128 rows move them there (2 x 184 + 2 x 40 + 24 = 472 per
// lane position, of the 5 x 96 = 480 that the CTA is launched with). The 128-row instances, and those of
// 64 rows for groups of 32 and 64, still spill 52 to 68 bytes a thread.
#pragma once

#include "w4a16_gemm_umma.cuh"
#include "w4a16_tile_plan.cuh"

namespace fk_w4a16 {

struct TileParams {
  GemvParams base;
  const uint8_t* staged;   // [row_tiles][blocks][tile_block_bytes]
  float* slots;            // [CTAs][2][kTilePair][rows][128] fp32
  int rows;                // rows of a pass, a multiple of 16
  int row_tiles;
  uint32_t blocks;         // steps of a unit: ceil(k / 128)
  uint32_t total_steps;
  int stages;
  int weights_reused;      // more than one row tile reads them
};

struct StageTileParams {
  const uint16_t* act;
  uint8_t* staged;
  int batch;
  int k;
  int rows;
  uint32_t blocks;
};

// Prepass: activations -> operand B blocks (K-major core matrices of 8 rows x 16 bytes; the 8
// features of a word in the order 0 4 1 5 2 6 3 7 that the unpack produces) and fp32 group sums.
// Thread (chunk, row) of a CTA of 128: 16 chunks of 8 features x 8 rows, so that both the loads
// (256 bytes of a row) and the stores (128 bytes) are whole lines.
template <int G, class E>
__global__ void __launch_bounds__(128) stage_activations_tile_kernel(const __grid_constant__ StageTileParams sp) {
  __shared__ float sums[16][8];
  const int r = static_cast<int>(threadIdx.x) & 7;
  const int chunk = static_cast<int>(threadIdx.x) >> 3;
  const uint32_t block = blockIdx.x;
  const int row = (static_cast<int>(blockIdx.y) * 8) + r;
  const int row_tile = row / sp.rows;
  const int n = row - (row_tile * sp.rows);
  const long long feature = (static_cast<long long>(block) * kTileK) + (chunk * 8);
  pdl_launch_dependents();
  pdl_wait_for_prerequisites();
  uint4 w = make_uint4(0u, 0u, 0u, 0u);
  if (row < sp.batch && feature < sp.k) {
    w = __ldg(reinterpret_cast<const uint4*>(sp.act + (static_cast<long long>(row) * sp.k) + feature));
  }
  const uint32_t words[4] = {w.x, w.y, w.z, w.w};
  float sum = 0.0f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    sum += E::to_float(static_cast<unsigned short>(words[i] & 0xffffu));
    sum += E::to_float(static_cast<unsigned short>(words[i] >> 16));
  }
  sums[chunk][r] = sum;
  uint8_t* dst = sp.staged + (((static_cast<size_t>(row_tile) * sp.blocks) + block) *
                              static_cast<size_t>(tile_block_bytes(G, sp.rows)));
  uint4 cells;
  cells.x = __byte_perm(w.x, w.z, 0x5410);
  cells.y = __byte_perm(w.x, w.z, 0x7632);
  cells.z = __byte_perm(w.y, w.w, 0x5410);
  cells.w = __byte_perm(w.y, w.w, 0x7632);
  *reinterpret_cast<uint4*>(dst + ((n >> 3) * (kTileK * 16)) + (chunk * 128) + (r * 16)) = cells;
  __syncthreads();
  if (chunk < tile_groups(G)) {
    float total = 0.0f;
#pragma unroll
    for (int i = 0; i < G / 8; ++i) {
      total += sums[(chunk * (G / 8)) + i][r];
    }
    reinterpret_cast<float*>(dst + (sp.rows * kTileK * 2))[(chunk * sp.rows) + n] = total;
  }
}

namespace tile {

// Word of 8 nibbles -> the four pairs (0,4) (1,5) (2,6) (3,7) of q - 8, exact in the 16-bit type.
template <class E>
__device__ __forceinline__ void unpack_word(uint32_t w, uint32_t* out) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t shifted = w >> (4 * i);
    if constexpr (std::is_same<E, BF16>::value) {
      const uint32_t v = mask_or<0x000f000fu, 0x43004300u>(shifted);  // 128 + q
      asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(out[i]) : "r"(v), "r"(0x43084308u));
    } else {
      const uint32_t v = mask_or<0x000f000fu, 0x64006400u>(shifted);  // 1024 + q
      asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(out[i]) : "r"(v), "r"(0x64086408u));
    }
  }
}

__device__ __forceinline__ void ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// The registers pass through the wait, so that nothing that reads them can move in front of it.
__device__ __forceinline__ void wait_ld16(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
      : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
        "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
      :
      : "memory");
}
__device__ __forceinline__ void ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
// The registers pass through the wait, so that nothing that reads them can move in front of it.
__device__ __forceinline__ void wait_ld32(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
      : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
        "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
        "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
        "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
      :
      : "memory");
}
template <int N>
__device__ __forceinline__ void load_columns(uint32_t taddr, uint32_t (&r)[N]) {
  if constexpr (N == 32) {
    ld32(taddr, r);
  } else {
    ld16(taddr, r);
  }
}
template <int N>
__device__ __forceinline__ void wait_columns(uint32_t (&r)[N]) {
  if constexpr (N == 32) {
    wait_ld32(r);
  } else {
    wait_ld16(r);
  }
}
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo), "r"(hi));
  return v;
}
__device__ __forceinline__ uint64_t broadcast2(float f) {
  return pack2(__float_as_uint(f), __float_as_uint(f));
}
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float half_of(uint64_t v, int which) {
  return __uint_as_float(static_cast<uint32_t>(which == 0 ? v : (v >> 32)));
}
__device__ __forceinline__ uint32_t idesc(bool bf16, int rows) {
  return (1u << 4) | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10) |
         (static_cast<uint32_t>(rows / 8) << 17) | (static_cast<uint32_t>(128 / 16) << 24);
}
// One K = 16 step of B: the two 16-byte K chunks 128 bytes apart, groups of 8 rows 2048 bytes.
__device__ __forceinline__ uint64_t b_desc(uint32_t smem_address) {
  return static_cast<uint64_t>((smem_address & 0x3FFFFu) >> 4) | (static_cast<uint64_t>(128 >> 4) << 16) |
         (static_cast<uint64_t>((kTileK * 16) >> 4) << 32) | (uint64_t{1} << 46);
}
template <int kRegisters>
__device__ __forceinline__ void registers_up() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegisters));
}
template <int kRegisters>
__device__ __forceinline__ void registers_down() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegisters));
}

__host__ __device__ inline uint32_t run_begin(uint32_t cta, uint32_t ctas, uint32_t total) {
  return static_cast<uint32_t>((static_cast<uint64_t>(cta) * total) / ctas);
}
// The CTA whose run holds `step`.
__device__ __forceinline__ uint32_t run_of(uint32_t step, uint32_t ctas, uint32_t total) {
  uint32_t v = static_cast<uint32_t>((static_cast<uint64_t>(step) * ctas) / total);
  while (v + 1 < ctas && run_begin(v + 1, ctas, total) <= step) {
    ++v;
  }
  while (v > 0 && run_begin(v, ctas, total) > step) {
    --v;
  }
  return v;
}

}  // namespace tile

template <int G, int NT, class E>
__global__ void __launch_bounds__(kTileThreads, 1) w4a16_gemm_tile_kernel(const __grid_constant__ TileParams tp) {
  constexpr int kStride = packet_stride(G);
  constexpr int kQBytes = packet_q_bytes(G);
  constexpr int kGroups = tile_groups(G);              // groups of a step
  constexpr int kUnit = tile_unit_groups(G, NT);       // groups of an accumulator buffer
  constexpr int kHalves = tile_halves(NT);
  constexpr int kHalfRows = tile_half_rows(NT);        // MMA N at most
  constexpr int kParts = kGroups / kUnit;              // x kHalves: accumulator hand-overs per step and tile
  constexpr int kDBuffers = tile_d_buffers(G, NT);
  constexpr uint32_t kDHalf = kDBuffers / 2;           // accumulator buffers of one weight tile
  constexpr int kDColumns = kUnit * kHalfRows;
  constexpr int kTileBytes = kGroups * kStride;        // one weight tile of a step
  constexpr bool kMoveRegisters = NT >= 64;
  // Accumulator columns per tcgen05.ld. A load takes some 200 clocks to come back however wide it
  // is (timeline of one CTA: 16 loads of 8 columns, 3600 clocks), so they are as wide as the
  // registers allow.
  constexpr int kChunk = NT < 32 ? NT : 32;
  static_assert(kDBuffers >= 2 && kDBuffers % 2 == 0, "one accumulator buffer per weight tile at least");
  extern __shared__ __align__(128) uint8_t smem[];

  const GemvParams& p = tp.base;
  const int tid = static_cast<int>(threadIdx.x);
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int rows = tp.rows;
  const uint32_t ctas = gridDim.x;
  const uint32_t cta = blockIdx.x;
  const uint32_t stages = static_cast<uint32_t>(tp.stages);
  const uint32_t num_groups = static_cast<uint32_t>(p.num_groups);
  const uint32_t step_begin = tile::run_begin(cta, ctas, tp.total_steps);
  const uint32_t step_end = tile::run_begin(cta + 1, ctas, tp.total_steps);
  const uint32_t count = step_end - step_begin;
  const uint32_t first_unit = step_begin / tp.blocks;
  const uint32_t first_block = step_begin - (first_unit * tp.blocks);

  const uint32_t smem_base = smem_addr(smem);
  const uint32_t full_bar = smem_base + 16;                       // [stages] copies landed
  const uint32_t empty_bar = full_bar + (kTileMaxStages * 8);     // [stages] promote warps are done with it
  const uint32_t aready_bar = empty_bar + (kTileMaxStages * 8);   // [A buffers] unpacked
  const uint32_t afree_bar = aready_bar + (kTileABuffers * 8);    // [A buffers] MMAs complete
  const uint32_t done_bar = afree_bar + (kTileABuffers * 8);      // [D buffers] MMAs complete
  const uint32_t dfree_bar = done_bar + (4 * 8);                  // [D buffers] read out
  const uint32_t drain_bar = dfree_bar + (4 * 8);
  volatile uint32_t* fail_flag = reinterpret_cast<volatile uint32_t*>(smem + 8);
  const uint32_t ring = smem_base + kTileBarrierBytes;
  const uint32_t stage_bytes = static_cast<uint32_t>(tile_stage_bytes(G, rows));
  const uint32_t block_bytes = static_cast<uint32_t>(tile_block_bytes(G, rows));

  if (tid == 0) {
    *fail_flag = 0u;
    for (uint32_t s = 0; s < stages; ++s) {
      mbar_init(full_bar + (s * 8), 1);
      mbar_init(empty_bar + (s * 8), 8);
    }
    for (int i = 0; i < kTileABuffers; ++i) {
      mbar_init(aready_bar + (i * 8), 4);
      mbar_init(afree_bar + (i * 8), 1);
    }
    for (int i = 0; i < kDBuffers; ++i) {
      mbar_init(done_bar + (i * 8), 1);
      mbar_init(dfree_bar + (i * 8), 4);
    }
    mbar_init(drain_bar, 2);
    mbar_init_fence();
  }
  if (warp == 1) {
    umma::tmem_alloc(smem_base, 512);
    umma::tmem_relinquish();
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(smem);

  auto give_up = [&]() {
    *fail_flag = 1u;
    atomicExch(p.status, static_cast<int>(kStatusCopyWaitTimeout));
  };
  // Groups of the step at K block `block`: all, or what is left at the end of K.
  auto groups_of = [&](uint32_t block) -> uint32_t {
    const uint32_t left = num_groups - (block * kGroups);
    return left < kGroups ? left : kGroups;
  };

  if (warp < 4) {
    if constexpr (kMoveRegisters) {
      tile::registers_down<24>();
    }
    if (warp == 0 && lane == 0) {
      // ---- producer --------------------------------------------------------------------------
      const uint64_t weight_policy = tp.weights_reused != 0 ? l2_evict_last_policy() : l2_evict_first_policy();
      const uint64_t act_policy = l2_evict_last_policy();
      uint32_t unit = first_unit;
      uint32_t block = first_block;
      auto copy_weights = [&](uint32_t s) {
        const uint32_t ng = groups_of(block);
        mbar_expect_tx(full_bar + (s * 8), (kTilePair * ng * kStride) + block_bytes);
        const uint32_t pair = unit / static_cast<uint32_t>(tp.row_tiles);
#pragma unroll
        for (uint32_t e = 0; e < kTilePair; ++e) {
          // an odd number of tiles: the last pair reads its only tile twice and stores it once
          uint32_t t = (pair * kTilePair) + e;
          t = t < static_cast<uint32_t>(p.num_tiles) ? t : static_cast<uint32_t>(p.num_tiles) - 1;
          bulk_copy_g2s(ring + (s * stage_bytes) + (e * kTileBytes),
                        p.packets + (((static_cast<size_t>(t) * num_groups) + (block * kGroups)) * kStride),
                        ng * kStride, full_bar + (s * 8), weight_policy);
        }
      };
      auto copy_activations = [&](uint32_t s) {
        const uint32_t row_tile = unit % static_cast<uint32_t>(tp.row_tiles);
        bulk_copy_g2s(ring + (s * stage_bytes) + (kTilePair * kTileBytes),
                      tp.staged + (((static_cast<size_t>(row_tile) * tp.blocks) + block) * block_bytes),
                      block_bytes, full_bar + (s * 8), act_policy);
      };
      auto advance = [&]() {
        if (++block == tp.blocks) {
          block = 0;
          ++unit;
        }
      };
      // The weights do not depend on earlier work in the stream; the staged activations do.
      const uint32_t prefill = count < stages ? count : stages;
      for (uint32_t j = 0; j < prefill; ++j) {
        copy_weights(j);
        advance();
      }
      pdl_launch_dependents();
      pdl_wait_for_prerequisites();
      unit = first_unit;
      block = first_block;
      for (uint32_t j = 0; j < prefill; ++j) {
        copy_activations(j);
        advance();
      }
      uint32_t issued = prefill;
      uint32_t s = 0;
      uint32_t parity = 0;
      for (uint32_t j = prefill; j < count; ++j) {
        if (!mbar_wait_parked(empty_bar + (s * 8), parity)) {
          give_up();
          break;
        }
        proxy_fence_async();
        copy_weights(s);
        copy_activations(s);
        advance();
        issued = j + 1;
        if (++s == stages) {
          s = 0;
          parity ^= 1u;
        }
      }
      // A wait that gave up: let the copies in flight land before the shared memory is handed on.
      for (uint32_t j = issued > stages ? issued - stages : 0; j < issued; ++j) {
        if (!mbar_wait_parked(full_bar + ((j % stages) * 8), use_parity(j / stages))) {
          break;
        }
      }
    } else if ((warp == 1 || warp == 2) && lane == 0) {
      // ---- MMA issuers -----------------------------------------------------------------------
      // One per weight tile: the tensor core takes an issuer's MMAs in as it executes them, so while
      // one issuer is held by its MMAs the other goes through its waits and commits. (A single issuer
      // spent 1900 of 2700 clocks a step on those.) The stage's activations have landed when its
      // packets are unpacked: the unpack warps wait for the one barrier of both.
      // Earlier work may still run, for longer than a bounded wait lasts, and the first of those here
      // ends only after the producer has got past it.
      pdl_wait_for_prerequisites();
      const uint32_t e = static_cast<uint32_t>(warp) - 1;
      const uint32_t idesc_first =
          tile::idesc(std::is_same<E, BF16>::value, rows < kHalfRows ? rows : kHalfRows);
      const uint32_t idesc_second =
          kHalves > 1 ? tile::idesc(std::is_same<E, BF16>::value, rows - kHalfRows) : idesc_first;
      const uint64_t desc_first = tile::b_desc(ring + (kTilePair * kTileBytes));
      const uint64_t desc_stride = stage_bytes >> 4;
      uint64_t desc0 = desc_first;
      uint32_t s = 0;
      uint32_t block = first_block;
      uint32_t dc = 0;  // accumulator hand-overs of this tile so far
      for (uint32_t j = 0; j < count; ++j) {
        const uint32_t ng = groups_of(block);
        block = block + 1 == tp.blocks ? 0 : block + 1;
        const uint32_t a = ((j & 1) * kTilePair) + e;
        bool ok = mbar_wait_parked(aready_bar + (a * 8), use_parity(j >> 1));
#pragma unroll 1
        for (uint32_t x = 0; ok && x < kParts * kHalves; ++x, ++dc) {
          const uint32_t part = x / kHalves;
          const uint32_t half = x % kHalves;
          const uint32_t idesc = half == 0 ? idesc_first : idesc_second;
          const uint32_t d = ((dc % kDHalf) * kTilePair) + e;
          if (dc >= kDHalf) {
            ok = mbar_wait_parked(dfree_bar + (d * 8), use_parity((dc / kDHalf) - 1));
            if (!ok) {
              break;
            }
          }
          umma::fence_after_sync();
#pragma unroll
          for (uint32_t i = 0; i < kUnit; ++i) {
            const uint32_t g = (part * kUnit) + i;
            if (g < ng) {
              const uint32_t d_tmem = tmem_base + kTileDColumn0 + (d * kDColumns) + (i * kHalfRows);
              const uint32_t a_tmem = tmem_base + (a * 64) + (g * (G / 2));
              const uint64_t desc = desc0 + (g * ((G / 8) * 128 / 16)) + (half * ((kHalfRows / 8) * kTileK));
#pragma unroll
              for (uint32_t ks = 0; ks < G / 16; ++ks) {
                umma::mma_f16_ts(d_tmem, a_tmem + (8 * ks), desc + (ks * (256 / 16)), idesc, ks == 0 ? 0u : 1u);
              }
            }
          }
          umma::commit(done_bar + (d * 8));
        }
        if (!ok) {
          give_up();
          break;
        }
        umma::commit(afree_bar + (a * 8));
        desc0 += desc_stride;
        if (++s == stages) {
          s = 0;
          desc0 = desc_first;
        }
      }
    }
  } else if (warp < 12) {
    if constexpr (kMoveRegisters) {
      tile::registers_down<40>();
    }
    // ---- unpack ------------------------------------------------------------------------------
    pdl_wait_for_prerequisites();  // as the issuers: no bounded wait runs while earlier work does
    const uint32_t e = static_cast<uint32_t>(warp - 4) >> 2;
    const uint32_t quarter = static_cast<uint32_t>(warp) & 3;
    const uint32_t col = (quarter * 32) + lane;
    const uint32_t lane_base = tmem_base + ((quarter * 32) << 16);
    uint32_t block = first_block;
    uint32_t s = 0;
    uint32_t parity = 0;
    for (uint32_t j = 0; j < count; ++j) {
      const uint32_t a = ((j & 1) * kTilePair) + e;
      const uint32_t ng = groups_of(block);
      block = block + 1 == tp.blocks ? 0 : block + 1;
      bool ok = mbar_wait_parked(full_bar + (s * 8), parity);
      const uint32_t words_addr = ring + (s * stage_bytes) + (e * kTileBytes) + (col * 4);
      if (ok && j >= 2) {
        ok = mbar_wait_parked(afree_bar + (a * 8), use_parity((j >> 1) - 1));
      }
      if (!ok) {
        give_up();
        break;
      }
      if (++s == stages) {
        s = 0;
        parity ^= 1u;
      }
      umma::fence_after_sync();
#pragma unroll
      for (int half = 0; half < 16; half += 8) {
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = half + i;
          const int g = r / (G / 8);
          w[i] = static_cast<uint32_t>(g) < ng
                     ? umma::lds32(words_addr + (g * kStride) + ((r % (G / 8)) * kTileCols * 4))
                     : 0u;
        }
#pragma unroll
        for (int r = 0; r < 8; r += 4) {
          uint32_t cells[16];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            tile::unpack_word<E>(w[r + i], cells + (4 * i));
          }
          umma::st16(lane_base + (a * 64) + ((half + r) * 4), cells);
        }
      }
      umma::wait_st();
      umma::fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        umma::mbar_arrive(aready_bar + (a * 8));
      }
    }
  } else {
    if constexpr (kMoveRegisters) {
      tile::registers_up<184>();
    }
    // Outputs, slots and tickets are written, and a residual is read, behind earlier work; and no
    // bounded wait runs while it does.
    pdl_wait_for_prerequisites();
    // ---- promote -----------------------------------------------------------------------------
    const uint32_t e = static_cast<uint32_t>(warp - 12) >> 2;
    const uint32_t quarter = static_cast<uint32_t>(warp) & 3;
    const uint32_t col = (quarter * 32) + lane;
    const uint32_t lane_base = tmem_base + ((quarter * 32) << 16) + kTileDColumn0;
    uint64_t acc[NT / 2];
#pragma unroll
    for (int i = 0; i < NT / 2; ++i) {
      acc[i] = 0;
    }

    auto store_column = [&](uint32_t unit) {
      const uint32_t t = ((unit / static_cast<uint32_t>(tp.row_tiles)) * kTilePair) + e;
      const int row0 = static_cast<int>(unit % static_cast<uint32_t>(tp.row_tiles)) * rows;
      if (t >= static_cast<uint32_t>(p.num_tiles)) {
        return;
      }
      const int valid = (p.m - row0) < rows ? (p.m - row0) : rows;
      long long offset = (static_cast<long long>(row0) * p.out_ld) + p.out_col0 +
                         (static_cast<long long>(t) * kTileCols) + col;
#pragma unroll
      for (int m = 0; m < NT; ++m) {
        if (m < valid) {
          float value = tile::half_of(acc[m / 2], m & 1);
          if (p.residual != nullptr) {
            value += E::to_float(__ldcg(static_cast<const unsigned short*>(p.residual) + offset));
          }
          if (p.out_f32 != 0) {
            static_cast<float*>(p.out)[offset] = value;
          } else {
            static_cast<unsigned short*>(p.out)[offset] = E::from_float(value);
          }
          offset += p.out_ld;
        }
      }
    };
    auto slot_of = [&](uint32_t v, uint32_t which) -> float* {
      return tp.slots + ((((static_cast<size_t>(v) * 2) + which) * kTilePair + e) * rows * kTileCols) + col;
    };
    // This CTA's part of `unit` is in the registers: the steps [from, to) of its K dimension.
    auto finish_unit = [&](uint32_t unit, uint32_t from, uint32_t to) {
      if (to - from == tp.blocks) {
        store_column(unit);
        return;
      }
      float* mine = slot_of(cta, unit == first_unit ? 0 : 1);
#pragma unroll
      for (int m = 0; m < NT; ++m) {
        if (m < rows) {
          __stcg(mine + (m * kTileCols), tile::half_of(acc[m / 2], m & 1));
        }
      }
      __threadfence();
      __syncwarp();
      const uint32_t v0 = tile::run_of(unit * tp.blocks, ctas, tp.total_steps);
      const uint32_t v1 = tile::run_of((unit * tp.blocks) + tp.blocks - 1, ctas, tp.total_steps);
      // a ticket per warp: each warp finishes its own 32 columns
      int* ticket = p.tickets + ((((static_cast<size_t>(unit) * kTilePair) + e) * 4) + quarter);
      int drawn = 0;
      if (lane == 0) {
        drawn = atomicAdd(ticket, 1);
      }
      drawn = __shfl_sync(0xffffffffu, drawn, 0);
      if (drawn != static_cast<int>(v1 - v0)) {
        return;
      }
      __threadfence();
#pragma unroll
      for (int i = 0; i < NT / 2; ++i) {
        acc[i] = 0;
      }
      for (uint32_t v = v0; v <= v1; ++v) {
        const float* part = slot_of(v, tile::run_begin(v, ctas, tp.total_steps) / tp.blocks == unit ? 0 : 1);
#pragma unroll
        for (int m0 = 0; m0 < NT; m0 += kChunk) {
          if (m0 < rows) {
            float x[kChunk];  // all in flight at once: the loop is bound by the latency of L2
#pragma unroll
            for (int i = 0; i < kChunk; ++i) {
              x[i] = (i < 16 || m0 + 16 < rows) ? __ldcg(part + ((m0 + i) * kTileCols)) : 0.0f;
            }
#pragma unroll
            for (int i = 0; i < kChunk; i += 2) {
              uint64_t& sum = acc[(m0 + i) / 2];
              const float lo = tile::half_of(sum, 0) + x[i];
              const float hi = tile::half_of(sum, 1) + x[i + 1];
              sum = tile::pack2(__float_as_uint(lo), __float_as_uint(hi));
            }
          }
        }
      }
      store_column(unit);
      if (lane == 0) {
        *ticket = 0;
      }
    };

    uint32_t unit = first_unit;
    uint32_t block = first_block;
    uint32_t from = first_block;
    uint32_t s = 0;
    uint32_t parity = 0;
    uint32_t dc = 0;
    for (uint32_t j = 0; j < count; ++j) {
      const uint32_t ng = groups_of(block);
      bool ok = mbar_wait_parked(full_bar + (s * 8), parity);
      const uint32_t tile_addr = ring + (s * stage_bytes) + (e * kTileBytes) + kQBytes + (col * 2);
      const uint32_t sums_addr = ring + (s * stage_bytes) + (kTilePair * kTileBytes) + (rows * kTileK * 2);
#pragma unroll 1
      for (uint32_t part = 0; ok && part < kParts; ++part) {
        const uint32_t first = part * kUnit;
        const uint32_t valid = ng > first ? (ng - first < kUnit ? ng - first : kUnit) : 0;
#pragma unroll
        for (int half = 0; half < kHalves; ++half) {
          const uint32_t d = ((dc % kDHalf) * kTilePair) + e;
          ok = ok && mbar_wait_parked(done_bar + (d * 8), use_parity(dc / kDHalf));
          ++dc;
          if (ok) {
            umma::fence_after_sync();
            auto read_out = [&]() {  // the accumulators are in registers: the buffer may be overwritten
              umma::fence_before_sync();
              __syncwarp();
              if (lane == 0) {
                umma::mbar_arrive(dfree_bar + (d * 8));
              }
            };
            if (valid == 0) {
              read_out();
            }
#pragma unroll 1
            for (uint32_t i = 0; i < valid; ++i) {
              const uint32_t d_tmem = lane_base + (d * kDColumns) + (i * kHalfRows);
              const uint32_t scale_addr = tile_addr + ((first + i) * kStride);
              unsigned short alpha_bits;
              unsigned short beta_bits;
              asm volatile("ld.shared.u16 %0, [%1];" : "=h"(alpha_bits) : "r"(scale_addr));
              asm volatile("ld.shared.u16 %0, [%1];" : "=h"(beta_bits) : "r"(scale_addr + (kTileCols * 2)));
              const float alpha = E::to_float(alpha_bits);
              const uint64_t alpha2 = tile::broadcast2(alpha);
              const uint64_t offset2 = tile::broadcast2(fmaf(8.0f, alpha, E::to_float(beta_bits)));
              const uint32_t group_sums = sums_addr + ((first + i) * rows * 4);
#pragma unroll
              for (int c = 0; c < kHalfRows; c += kChunk) {
                const int row = (half * kHalfRows) + c;
                if (row < rows) {
                  uint32_t x[kChunk];
                  tile::load_columns(d_tmem + c, x);
                  tile::wait_columns(x);
                  if ((row + kChunk >= rows || c + kChunk == kHalfRows) && i + 1 == valid) {
                    read_out();
                  }
#pragma unroll
                  for (int h = 0; h < kChunk; h += 16) {
                    if (row + h < rows) {  // rows are a multiple of 16: no sums behind the block are read
#pragma unroll
                      for (int q = h; q < h + 16; q += 4) {
                        const uint4 sums = lds128(group_sums + ((row + q) * 4));
                        uint64_t& lo = acc[(row + q) / 2];
                        uint64_t& hi = acc[((row + q) / 2) + 1];
                        tile::fma2(lo, tile::pack2(x[q], x[q + 1]), alpha2);
                        tile::fma2(hi, tile::pack2(x[q + 2], x[q + 3]), alpha2);
                        tile::fma2(lo, tile::pack2(sums.x, sums.y), offset2);
                        tile::fma2(hi, tile::pack2(sums.z, sums.w), offset2);
                      }
                    }
                  }
                }
              }
            }
          }
        }
      }
      if (!ok) {
        give_up();
        break;
      }
      // scales and sums of the stage are read, and its MMAs and unpacks came before: refill it
      __syncwarp();
      if (lane == 0) {
        umma::mbar_arrive(empty_bar + (s * 8));
      }
      if (++s == stages) {
        s = 0;
        parity ^= 1u;
      }
      ++block;
      if (block == tp.blocks || j + 1 == count) {
        finish_unit(unit, from, block);
#pragma unroll
        for (int i = 0; i < NT / 2; ++i) {
          acc[i] = 0;
        }
        block = 0;
        from = 0;
        ++unit;
      }
    }
  }

  umma::fence_before_sync();
  __syncthreads();
  if (*fail_flag != 0u && (warp == 1 || warp == 2) && lane == 0) {
    umma::commit(drain_bar);  // MMAs still in flight, if any
  }
  __syncwarp();
  if (warp == 1) {
    if (*fail_flag != 0u) {
      (void)mbar_wait_parked(drain_bar, 0);
    }
    umma::fence_after_sync();
    umma::tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace fk_w4a16
