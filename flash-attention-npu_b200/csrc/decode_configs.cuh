// Tile configurations of the producer / consumer decode kernel, per tile width (64, 128 or 256 columns; the head dim is
// at most that, columns beyond it are zeros from the TMA unit).
//   X(index, MT, WM, WN, BN, STAGES, SR)   rows per CTA = 16 * MT * WM, consumer warps = WM * WN;
//   SR = 1: the merge slab lies over the ring (never with persistent CTAs)
#pragma once

#include <cuda.h>

#include "fwd_decode.cuh"

// Only the configurations the planner can choose are built (128: measured against the others on the benchmark shapes):
//   3   up to 16 packed rows.  64, 128: two resident CTAs of 1 x 4 consumer warps, 32 KiB stages; 256: one CTA, 64 KiB stages
//   5   17-32 rows, long key ranges or persistent launches.  128: one CTA of 2 x 4 warps, 128-key stages; 64: two such
//       CTAs; 256: one CTA of 2 x 2 warps and five 32-key stages (the fp32 merge slab of 32 rows takes 33 KiB)
//   11  128 only: 17-32 rows, short key ranges (a sliding window): two resident CTAs of 2 x 2 warps, slab over the ring
// Configuration 3 (kDecodeClusterBase) is built a second time with the key splits of a unit in one thread-block cluster
// (kDecodeClusterConfig).
#define FA_DECODE_CONFIGS_64(X) X(3, 1, 1, 4, 128, 3, 0) X(5, 1, 2, 4, 128, 3, 0)
#define FA_DECODE_CONFIGS_128(X) X(3, 1, 1, 4, 64, 3, 0) X(5, 1, 2, 4, 128, 3, 0) X(11, 1, 2, 2, 64, 3, 1)
#define FA_DECODE_CONFIGS_256(X) X(3, 1, 1, 4, 64, 3, 0) X(5, 1, 2, 2, 32, 5, 0)

namespace fa {

// The traits of configuration I, as listed above (the planner and the TMA boxes read the same list).
template <int HD, typename T, int I>
struct DecConfig;
#define FA_X(I_, MT_, WM_, WN_, BN_, ST_, SR_)                              \
  template <typename T>                                                     \
  struct DecConfig<FA_HD_, T, I_> {                                         \
    using Tr = DecTraits<FA_HD_, T, MT_, WM_, WN_, BN_, ST_, SR_>;          \
  };
#define FA_HD_ 64
FA_DECODE_CONFIGS_64(FA_X)
#undef FA_HD_
#define FA_HD_ 128
FA_DECODE_CONFIGS_128(FA_X)
#undef FA_HD_
#define FA_HD_ 256
FA_DECODE_CONFIGS_256(FA_X)
#undef FA_HD_
#undef FA_X

struct DecodeConfigInfo {
  int block_m, block_n, threads, smem_bytes;
  bool slab_in_ring;
};

inline bool decode_config_info(int hd, int cfg, DecodeConfigInfo* out) {
#define FA_X(I_, MT_, WM_, WN_, BN_, ST_, SR_)                                              \
  if (cfg == I_) {                                                                    \
    using Tr = DecTraits<FA_HD_, __nv_bfloat16, MT_, WM_, WN_, BN_, ST_, SR_>;             \
    *out = DecodeConfigInfo{Tr::BM, Tr::BN, Tr::NTHREADS, Tr::SMEM_BYTES, Tr::SLAB_IN_RING}; \
    return true;                                                                      \
  }
#define FA_HD_ 64
  if (hd == 64) { FA_DECODE_CONFIGS_64(FA_X) }
#undef FA_HD_
#define FA_HD_ 128
  if (hd == 128) { FA_DECODE_CONFIGS_128(FA_X) }
#undef FA_HD_
#define FA_HD_ 256
  if (hd == 256) { FA_DECODE_CONFIGS_256(FA_X) }
#undef FA_HD_
#undef FA_X
  return false;
}

#define FA_DECODE_LAUNCHER(NAME_)                                                                                      \
  cudaError_t NAME_(int cfg, const KParams& p, const CUtensorMap& tm_k, const CUtensorMap& tm_v, int grid, cudaStream_t st);
FA_DECODE_LAUNCHER(launch_decode_64_bf16)
FA_DECODE_LAUNCHER(launch_decode_64_fp16)
FA_DECODE_LAUNCHER(launch_decode_128_bf16)
FA_DECODE_LAUNCHER(launch_decode_128_fp16)
FA_DECODE_LAUNCHER(launch_decode_256_bf16)
FA_DECODE_LAUNCHER(launch_decode_256_fp16)
#undef FA_DECODE_LAUNCHER

}  // namespace fa
