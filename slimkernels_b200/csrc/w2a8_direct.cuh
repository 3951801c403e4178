// Decode GEMM without tensor memory: 2-bit weights go from HBM through a small ring of each warp's own into registers,
// where two mask operations and a shift per word make them the operands of warp-level integer MMAs.
//
// For a handful of tokens the GEMM is one pass over the packed weights, and a call lasts a few microseconds: what
// bounds it is how soon the first weights are asked for, how many bytes are in flight, and how long the last ones take
// to turn into outputs.  The tcgen05 kernels pay for their roles there: set-up, four hand-overs per K block, a
// tensor-memory round trip per scale group.  Here a warp owns 16 * MT output features and every WARPS-th 128-wide K block
// of its CTA's range, and shares nothing with the others until the end:
//   * cp.async brings whole blocks (2 KiB of codes at MT = 4, their scales) into DEPTH slots; nobody else reads them, so
//     the only synchronisation is the warp's own wait for its oldest group;
//   * a word holds 16 codes.  code - zero point fits two bits of two's complement (or its negative does: see the kernel), and
//     in the top two bits of a byte that is 64 times its value as int8: a shift and one three-input logic operation take four
//     codes of a word (a byte-permute look-up needs nine operations per 16 codes instead of seven, and prmt issues at half
//     rate; masking without a shift, with the zero point as further rows of MMAs, five, but a quarter more MMAs);
//   * those four registers ARE A fragments of mma.sync m16n8k32: lane (g, q) holds features g and g + 8.  The K order
//     inside an MMA is free as long as both operands use the same one, so the activations are read as they lie (two 16-byte
//     loads per lane and 8 tokens) and four byte permutes per 16 codes put them in the words' order;
//   * the exact int32 sums start at the bits of 1.5 * 2^23, so that they read as floats: a subtraction and an FMA per value
//     take the bias off and scale, exact up to the last rounding.
// The CTA's warps add their sums in shared memory in warp order, the CTAs of a cluster (split K) in rank order through
// distributed shared memory: fixed orders, repeated launches are bit-identical.
//
// Measured, cold weights, tokens x features x K (before: the better tcgen05 decode kernel):
//   8 x 4096 x 4096 2.8 us (6.1), 8 x 22016 x 4096 7.2 us (15.1), 8 x 57344 x 8192 28.7 us = 4.3 TB/s (52.7),
//   16 x 12288 x 4096 8.0 us (10.4), 24 x 4096 x 11008 8.9 us (12.5); group size 64: 8 x 22016 x 4096 10.1 us (46.5).
// mma.sync s8 issues an m16n8k32 every 8 cycles per sub-core, 1.15 POP/s in all, but two or three warps per sub-core do not
// keep it busy (a third of the cycles at 24 tokens), and few CTAs fill whole waves badly: from about 32 tokens on the tcgen05
// kernels win on large weights (see choose_direct).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "activation.cuh"   // the quantiser's rule
#include "ptx_sm100.cuh"

namespace sk {

struct DirectParams {
  const uint8_t* w_tiled;     // [n_tiles][k_blocks][4096]
  const __half* w_scale_tiled;  // [n_tiles][groups][128], zero past N: the plan's copy
  // kernels with LIVE scales read these instead, behind the dependent-launch wait
  const __half* w_scale;      // [groups][N], the caller's, 4-byte aligned
  int scale_pieces;           // 1: its rows are whole 16-byte pieces (base 16-byte aligned, N % 8 == 0)
  int weights_late;           // 1: the codes, too, are read behind that wait (a borrowed buffer)
  const int8_t* x_q;          // [M, ld_x]
  const float* x_scale;       // [M]
  void* out;                  // [M, ld_out] half or bf16
  void* out_extra[7];         // further destinations (peer GPUs' buffers), same ld_out
  int n_extra;
  long long ld_x, ld_out;
  int M, N;
  int K, groups;              // groups = K / G
  int k_blocks;               // ceil(K / 128)
  int blocks_per_group;       // G / 128 (group sizes 64 and 32 are the kernel's GPB = 128 / G instead)
  int zero_point;
  int out_bf16;
  int floor_probe;            // host: launch an empty kernel of this geometry instead
  // kernels that quantise their activations themselves (x_q, ld_x and x_scale are not used then)
  const uint16_t* x_float;    // [M, ld_float] fp16 or bf16, rows 16-byte aligned
  long long ld_float;
  int float_bf16;
};

template <int MT, int NT, int WARPS, int DEPTH, int GPB, bool LIVE>
struct DirectTraits {
  static constexpr int kFeatures = 16 * MT;        // output features per CTA
  static constexpr int kTokens = 8 * NT;           // tokens per CTA
  static constexpr int kThreads = 32 * WARPS;
  // one warp's copy of a K block: the two halves of the features' codes (the second 64 bytes out of step, so that the four
  // lanes of a feature read different banks), then their scales (LIVE: and room for a row that starts mid-word)
  static constexpr int kHalfBytes = 16 * kFeatures;
  static constexpr int kOffHalf = kHalfBytes + 64;
  static constexpr int kOffScales = kOffHalf + kHalfBytes;
  static constexpr int kScalePitch = 2 * kFeatures + (LIVE ? 16 : 0);
  static constexpr int kStageBytes = kOffScales + GPB * kScalePitch;
  static constexpr int kWarpBytes = DEPTH * kStageBytes;
  static constexpr int kPitch = kFeatures + 4;     // floats per token in the reduction buffer: stores are conflict-free
  static constexpr int kRedBytes = WARPS * kTokens * kPitch * 4;    // takes the rings' place
  static constexpr int kDynamicBytes = WARPS * kWarpBytes > kRedBytes ? WARPS * kWarpBytes : kRedBytes;
  static constexpr int kQuantOffset = (kDynamicBytes + 15) / 16 * 16;   // int8 activations of kernels that quantise them
  static_assert(128 % kFeatures == 0, "a CTA's features lie in one weight tile");
  static_assert(GPB * 2 * MT <= 32 && kStageBytes % 16 == 0, "one 16-byte piece of the scales per lane");
};

// d = a . b + c on 16 features x 8 tokens x 32 codes
__device__ __forceinline__ void mma_s8_16832(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                             uint32_t b1, const int (&c)[4]) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]));
}
// The 16 codes of a tiled word as four registers of int8, code k of a nibble pair in the top two bits of its byte: f[0] codes
// {0, 2, 8, 10}, f[1] {4, 6, 12, 14}, f[2] {1, 3, 9, 11}, f[3] {5, 7, 13, 15} (a shift and a three-input logic operation each).
struct CodeBytes {
  uint32_t f[4];
  __device__ __forceinline__ CodeBytes(uint32_t w, uint32_t flip) {
    constexpr uint32_t kTop = 0xC0C0C0C0u;
    f[0] = ((w << 6) ^ flip) & kTop;
    f[1] = ((w << 4) ^ flip) & kTop;
    f[2] = ((w << 2) ^ flip) & kTop;
    f[3] = (w ^ flip) & kTop;
  }
};
// (volatile: never moved above griddepcontrol.wait)
__device__ __forceinline__ uint4 ld_global_v4(const void* p) {
  uint4 v;
  asm volatile("ld.global.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, int bytes) {   // (the rest of the word is zero)
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ uint2 ld_shared_v2(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_shared_b32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float ld_shared_half(uint32_t addr) {
  unsigned short v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr) : "memory");
  return __half2float(__ushort_as_half(v));
}

template <int MT, int NT, int WARPS, int DEPTH, int MIN_CTAS, int GPB, bool LIVE, bool QUANT = false>
__global__ void __launch_bounds__(32 * WARPS, MIN_CTAS) w2a8_direct_kernel(const DirectParams p) {
  using T = DirectTraits<MT, NT, WARPS, DEPTH, GPB, LIVE>;
  static_assert(LIVE || GPB == 1, "the plan has a copy of the scales for group size 128 only");
  extern __shared__ __align__(16) uint8_t direct_smem[];
  float* red = reinterpret_cast<float*>(direct_smem);   // after the main loop: [WARPS][kTokens][kPitch]
  grid_dep_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, q = lane & 3;
  const int n0 = blockIdx.x * T::kFeatures;
  const int m0 = blockIdx.y * T::kTokens;
  const int splits = gridDim.z, rank = blockIdx.z; // a cluster spans the grid's z dimension
  const int kb_end = static_cast<int>(static_cast<long long>(p.k_blocks) * (rank + 1) / splits);
  const int kb0 = static_cast<int>(static_cast<long long>(p.k_blocks) * rank / splits) + warp;
  // This warp's blocks are kb0, kb0 + WARPS, ...: `count` of them, walked in a ring that starts elsewhere in every CTA, so
  // that the CTAs do not all ask L2 for the same activations at the same time.
  const int count = kb0 < kb_end ? (kb_end - kb0 + WARPS - 1) / WARPS : 0;
  const int first = count > 1 ? static_cast<int>(blockIdx.x % static_cast<unsigned>(count)) : 0;

  // ---- weights and scales: DEPTH blocks in flight per warp
  const size_t tile = static_cast<size_t>(n0 >> 7);
  const uint8_t* w_src = p.w_tiled + (tile * p.k_blocks + kb0) * 4096 + ((n0 & 127) + (lane & 15)) * 16;
  const uint32_t ring = smem_u32(direct_smem) + warp * T::kWarpBytes;
  auto fetch_weights = [&](int idx, uint32_t slot) {
    const uint8_t* w = w_src + static_cast<size_t>(idx) * (WARPS * 4096);
    // piece i of a lane: 16 rows of one half per half-warp
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      const int piece = 2 * i + (lane >> 4);       // 16-row group of the two halves' 2 * MT
      const int half = piece / MT, rows = (piece % MT) * 16;
      cp_async16(slot + half * T::kOffHalf + (rows + (lane & 15)) * 16, w + half * 2048 + rows * 16);
    }
  };
  // Where the scales come from (16 bytes per lane and block, unless a row is cut otherwise):
  //   * the plan's copy, a block's features together, for group size 128 and up to 32 tokens.  It is constant and is fetched
  //     with the codes, before the wait below;
  //   * LIVE: the caller's [groups][N], as it is when the call runs, so behind that wait.  The kernel that served group sizes
  //     other than 128 and more than 32 tokens before this one read it then, too.  It costs about a microsecond, most of
  //     it the first loads' latency behind the wait: 8 x 22016 x 4096 with group size 64 8.8 us from a copy, 10.1 from the rows,
  //     8 x 4096 x 4096 with 256 3.1 and 4.3.  That is why the copy stays where it may.  Rows that are not whole 16-byte pieces take words from the one that holds their first scale on:
  //     with N odd every other row starts in the middle of it (scale_shift).
  const uint8_t* s_src = reinterpret_cast<const uint8_t*>(p.w_scale_tiled) + tile * p.groups * 256 + (n0 & 127) * 2 +
                         (lane % (2 * MT)) * 16;
  auto group_of = [&](int idx, int b) {            // the scale group of part b of a block
    const int kb = kb0 + idx * WARPS;
    return GPB > 1 ? min(kb * GPB + b, p.groups - 1) : !LIVE || p.blocks_per_group == 1 ? kb : kb / p.blocks_per_group;
  };
  const uint8_t* s_base = reinterpret_cast<const uint8_t*>(p.w_scale) + 2 * n0;
  // (pieces past N are left out: those features are not stored)
  const bool s_lane = lane < GPB * 2 * MT && (!LIVE || n0 + (lane % (2 * MT)) * 8 < p.N);
  auto piece_src = [&](int idx) {
    if constexpr (!LIVE) return s_src + static_cast<size_t>(group_of(idx, 0)) * 256;
    return s_base + static_cast<size_t>(group_of(idx, lane / (2 * MT))) * (2 * static_cast<size_t>(p.N)) + (lane % (2 * MT)) * 16;
  };
  const uint32_t piece_dst = T::kOffScales + (LIVE ? (lane / (2 * MT)) * T::kScalePitch + (lane % (2 * MT)) * 16 : lane * 16);
  auto fetch_scale_words = [&](int idx, uint32_t slot) {
    constexpr int kWords = T::kFeatures / 2 + 1;
    const long long end = 2LL * p.groups * p.N - 2 * n0;       // of the buffer, from s_base
#pragma unroll 1
    for (int i = lane; i < GPB * kWords; i += 32) {
      const int b = i / kWords, w = i % kWords;
      const long long o = ((2LL * group_of(idx, b) * p.N) & ~3LL) + 4 * w;      // (n0 is even: rows of even N start on words)
      if (o < end) cp_async4(slot + T::kOffScales + b * T::kScalePitch + 4 * w, s_base + o, end - o < 4 ? 2 : 4);
    }
  };
  int idx_fetch = first, to_fetch = count;
  uint32_t slot_fetch = ring;
  auto advance = [&]() {
    --to_fetch;
    if (++idx_fetch == count) idx_fetch = 0;
  };
  auto next_slot = [&]() {
    slot_fetch += T::kStageBytes;
    if (slot_fetch == ring + T::kWarpBytes) slot_fetch = ring;
  };
  auto fetch = [&]() {
    if (to_fetch > 0) {
      fetch_weights(idx_fetch, slot_fetch);
      if (!LIVE || p.scale_pieces) {
        if (s_lane) cp_async16(slot_fetch + piece_dst, piece_src(idx_fetch));
      } else {
        fetch_scale_words(idx_fetch, slot_fetch);
      }
      advance();
    }
    cp_async_commit();                             // (an empty group when there is nothing left: the waits count groups)
    next_slot();
  };
  // The first DEPTH blocks: the plan's codes go out at once, a borrowed buffer's behind the wait.  Live scales are pulled into
  // L2 meanwhile.
  if (LIVE && p.weights_late) grid_dep_wait();
#pragma unroll
  for (int d = 0; d < DEPTH; ++d) {
    if constexpr (!LIVE) {
      fetch();
    } else {
      if (to_fetch > 0) {
        fetch_weights(idx_fetch, slot_fetch);
        if (lane < 2 * GPB) {                      // both ends of each group's row
          const size_t row = static_cast<size_t>(group_of(idx_fetch, lane >> 1)) * (2 * static_cast<size_t>(p.N));
          prefetch_l2(s_base + row + 2 * ((lane & 1) ? min(T::kFeatures, p.N - n0) - 1 : 0));
        }
        advance();
      }
      cp_async_commit();
      next_slot();
    }
  }

  // code - zp as two's complement in the top two bits of a byte is 64 times its value: for zp 2 the code with its upper bit
  // flipped, for zp 1 the code with its lower bit flipped is 1 - code (the scale takes the sign).  Zero points 0 and 3 do not fit
  // two bits: they are zp 2 plus a multiple of the token's sum of codes, another row of MMAs.
  const uint32_t flip = p.zero_point == 1 ? 0x55555555u : 0xAAAAAAAAu;
  const float unit = p.zero_point == 1 ? -0.015625f : 0.015625f;
  const bool offset = p.zero_point == 0 || p.zero_point == 3;
  const uint32_t offset4x = p.zero_point == 0 ? 0x80808080u : 0x40404040u;     // -64 * 2, or -64 * -1
  const int bias[4] = {0x4B400000, 0x4B400000, 0x4B400000, 0x4B400000};   // as a float 12582912 = 1.5 * 2^23
  const int8_t* x_lane[NT];
  if constexpr (!QUANT)
#pragma unroll
    for (int t = 0; t < NT; ++t) x_lane[t] = p.x_q + min(m0 + 8 * t + g, p.M - 1) * p.ld_x + kb0 * 128 + (GPB == 1 ? 32 : 16) * q;
  float acc[MT][NT][4];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[i][t][c] = 0.f;

  // the plan wrote its codes and copies; live scales, activations and outputs may belong to the kernels before this one
  grid_dep_wait();
  // The first blocks' scales with plain loads: as copies behind those of the codes they would hold up the first block until
  // all DEPTH have landed (groups complete in order).
  uint4 s_first[DEPTH];
  if (LIVE && p.scale_pieces) {
#pragma unroll
    for (int d = 0; d < DEPTH; ++d)
      if (s_lane && d < count) s_first[d] = ld_global_v4(piece_src(first + d < count ? first + d : first + d - count));
  }

  const int kb_first = kb0 - warp;                 // the CTA's range is [kb_first, kb_end)
  uint32_t xs_lane = 0;                            // QUANT: this lane's token in shared memory, at the warp's first block
  const float* q_scale = nullptr;
  if constexpr (QUANT) {
    // The activations of the CTA's K range as int8 behind the rings, by the quantiser's rule: the row's largest value (the
    // whole row's), its scale, then the range.  Every CTA reads the rows again -- a few KiB from L2 -- which costs less than a
    // kernel before this one whose only product is those bytes.
    static_assert(NT == 1 && GPB == 1, "few tokens");
    __shared__ float part[T::kTokens][WARPS];
    __shared__ float scale_s[T::kTokens];
    const int tokens = min(T::kTokens, p.M - m0);
    const int nvec = p.K / 8;
    auto row8 = [&](int tok, int v) {
      const uint4 u = ld_global_v4(p.x_float + (m0 + tok) * p.ld_float + 8 * v);
      return p.float_bf16 ? as_half8<true>(u) : u;
    };
    for (int tok = 0; tok < tokens; ++tok) {
      float amax = 0.f;
#pragma unroll 4
      for (int v = threadIdx.x; v < nvec; v += T::kThreads) {
        const uint4 u = row8(tok, v);
        const __half2* h = reinterpret_cast<const __half2*>(&u);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = __half22float2(h[j]);
          amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
      if (lane == 0) part[tok][warp] = amax;
    }
    __syncthreads();
    const int pitch = (kb_end - kb_first) * 128 + 16;    // 16 bytes on: a quarter-warp reads two tokens from different banks
    uint8_t* xq_s = direct_smem + T::kQuantOffset;
    for (int tok = 0; tok < tokens; ++tok) {
      float amax = 0.f;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) amax = fmaxf(amax, part[tok][w]);
      const float s = amax > 0.f ? amax / 127.f : 1.f;
      const float r = 1.f / s;
      if (threadIdx.x == 0) scale_s[tok] = s;
      for (int v = threadIdx.x; v < (kb_end - kb_first) * 16; v += T::kThreads) {
        const uint4 u = row8(tok, kb_first * 16 + v);
        const __half2* h = reinterpret_cast<const __half2*>(&u);
        uint32_t w[2] = {0u, 0u};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = __half22float2(h[j]);
          w[j >> 1] |= (quantize_one_fast(f.x, s, r) | (quantize_one_fast(f.y, s, r) << 8)) << (16 * (j & 1));
        }
        *reinterpret_cast<uint2*>(xq_s + tok * pitch + 8 * v) = make_uint2(w[0], w[1]);
      }
    }
    __syncthreads();
    q_scale = scale_s;
    xs_lane = smem_u32(xq_s) + min(g, tokens - 1) * pitch + warp * 128 + 32 * q;
  }

  uint4 xn[NT][2];                                 // the next block's activations
  int idx_x = first, to_fetch_x = count;
  auto fetch_x = [&]() {
    if (to_fetch_x > 0) {
      const int at = idx_x * (WARPS * 128);
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        if constexpr (QUANT) {
          xn[t][0] = ld_shared_v4(xs_lane + at);
          xn[t][1] = ld_shared_v4(xs_lane + at + 16);
        } else if constexpr (GPB == 1) {
          xn[t][0] = ld_global_v4(x_lane[t] + at);
          xn[t][1] = ld_global_v4(x_lane[t] + at + 16);
        } else {           // K ends inside the last block: what lies past it is read as zero (16-byte pieces: K % 32 == 0)
          const int k = kb0 * 128 + at + 16 * q;
          xn[t][0] = k < p.K ? ld_global_v4(x_lane[t] + at) : make_uint4(0u, 0u, 0u, 0u);
          xn[t][1] = k + 64 < p.K ? ld_global_v4(x_lane[t] + at + 64) : make_uint4(0u, 0u, 0u, 0u);
        }
      }
      --to_fetch_x;
      if (++idx_x == count) idx_x = 0;
    }
  };
  fetch_x();
  if (!LIVE) {
  } else if (p.scale_pieces) {
#pragma unroll
    for (int d = 0; d < DEPTH; ++d)
      if (s_lane && d < count) st_shared_v4(ring + d * T::kStageBytes + piece_dst, s_first[d]);
  } else {
    for (int d = 0; d < min(DEPTH, count); ++d) fetch_scale_words(first + d < count ? first + d : first + d - count, ring + d * T::kStageBytes);
    cp_async_wait_all();
  }
  // A lane's two words of a feature's block: GPB 1 adjacent ones (codes 32 q .. 32 q + 31), else word q of either half
  // (codes 16 q .. and 64 + 16 q ..), so that a half -- one or two scale groups -- is one K step of the warp's MMAs.
  const uint32_t w_off = (GPB == 1 ? (q >> 1) * T::kOffHalf + (q & 1) * 8 : q * 4) + g * 16;
  uint32_t slot = ring;
#pragma unroll 1
  for (int left = count; left > 0; --left) {
    cp_async_wait<DEPTH - 1>();
    __syncwarp();
    uint2 wv[2 * MT];
    float sv[GPB][2 * MT];
#pragma unroll
    for (int j = 0; j < 2 * MT; ++j) {
      if constexpr (GPB == 1) wv[j] = ld_shared_v2(slot + w_off + j * 128);
      else wv[j] = make_uint2(ld_shared_b32(slot + w_off + j * 128), ld_shared_b32(slot + w_off + T::kOffHalf + j * 128));
    }
    const int idx_now = idx_x > 0 ? idx_x - 1 : count - 1;     // (fetch_x is one block ahead)
#pragma unroll
    for (int b = 0; b < GPB; ++b) {
      const uint32_t scale_shift = LIVE && (p.N & 1) ? (group_of(idx_now, b) & 1) * 2 : 0;
#pragma unroll
      for (int j = 0; j < 2 * MT; ++j)
        sv[b][j] = unit * ld_shared_half(slot + T::kOffScales + scale_shift + b * T::kScalePitch + (8 * j + g) * 2);
    }
    __syncwarp();
    fetch();                                   // into the slot just read
    slot += T::kStageBytes;
    if (slot == ring + T::kWarpBytes) slot = ring;
    // B fragments in the order the masks below pick a word's codes: {0,2,8,10}, {1,3,9,11} | {4,6,12,14}, {5,7,13,15}
    uint32_t b_lo[NT][2][2], b_hi[NT][2][2];
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        b_lo[t][h][0] = prmt(xn[t][h].x, xn[t][h].z, 0x6420u);
        b_lo[t][h][1] = prmt(xn[t][h].x, xn[t][h].z, 0x7531u);
        b_hi[t][h][0] = prmt(xn[t][h].y, xn[t][h].w, 0x6420u);
        b_hi[t][h][1] = prmt(xn[t][h].y, xn[t][h].w, 0x7531u);
      }
    fetch_x();
    if constexpr (GPB == 1) {
      float off[NT][2];                            // the bias, and what zero points 0 and 3 add per token
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        off[t][0] = off[t][1] = 12582912.f;
        if (offset) {
          int z[4];
          mma_s8_16832(z, offset4x, offset4x, offset4x, offset4x, b_lo[t][0][0], b_lo[t][0][1], bias);
          mma_s8_16832(z, offset4x, offset4x, offset4x, offset4x, b_hi[t][0][0], b_hi[t][0][1], z);
          mma_s8_16832(z, offset4x, offset4x, offset4x, offset4x, b_lo[t][1][0], b_lo[t][1][1], z);
          mma_s8_16832(z, offset4x, offset4x, offset4x, offset4x, b_hi[t][1][0], b_hi[t][1][1], z);
          off[t][0] = __int_as_float(z[0]);
          off[t][1] = __int_as_float(z[1]);
        }
      }
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        const uint2 lo = wv[2 * i], hi = wv[2 * i + 1];
        const float s_lo = sv[0][2 * i], s_hi = sv[0][2 * i + 1];
        const CodeBytes lx(lo.x, flip), ly(lo.y, flip), hx(hi.x, flip), hy(hi.y, flip);
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          int c[4];
          mma_s8_16832(c, lx.f[0], hx.f[0], lx.f[2], hx.f[2], b_lo[t][0][0], b_lo[t][0][1], bias);
          mma_s8_16832(c, lx.f[1], hx.f[1], lx.f[3], hx.f[3], b_hi[t][0][0], b_hi[t][0][1], c);
          mma_s8_16832(c, ly.f[0], hy.f[0], ly.f[2], hy.f[2], b_lo[t][1][0], b_lo[t][1][1], c);
          mma_s8_16832(c, ly.f[1], hy.f[1], ly.f[3], hy.f[3], b_hi[t][1][0], b_hi[t][1][1], c);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            acc[i][t][k] = fmaf(k < 2 ? s_lo : s_hi, __int_as_float(c[k]) - off[t][k & 1], acc[i][t][k]);
        }
      }
    } else {
      constexpr int kSub = GPB / 2;            // scale groups per half block: one, or the lanes q < 2 and q >= 2
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int sub = 0; sub < kSub; ++sub) {
          const bool mine = kSub == 1 || (q >> 1) == sub;   // the other group's activations count as zero
          uint32_t bl[NT][2], bh[NT][2];
          float off[NT][2];
#pragma unroll
          for (int t = 0; t < NT; ++t) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              bl[t][e] = mine ? b_lo[t][h][e] : 0u;
              bh[t][e] = mine ? b_hi[t][h][e] : 0u;
            }
            off[t][0] = off[t][1] = 12582912.f;
            if (offset) {
              int z[4];
              mma_s8_16832(z, offset4x, offset4x, offset4x, offset4x, bl[t][0], bl[t][1], bias);
              mma_s8_16832(z, offset4x, offset4x, offset4x, offset4x, bh[t][0], bh[t][1], z);
              off[t][0] = __int_as_float(z[0]);
              off[t][1] = __int_as_float(z[1]);
            }
          }
#pragma unroll
          for (int i = 0; i < MT; ++i) {
            const uint32_t lo = h == 0 ? wv[2 * i].x : wv[2 * i].y;
            const uint32_t hi = h == 0 ? wv[2 * i + 1].x : wv[2 * i + 1].y;
            const float s_lo = sv[h * kSub + sub][2 * i], s_hi = sv[h * kSub + sub][2 * i + 1];
            const CodeBytes lb(lo, flip), hb(hi, flip);
#pragma unroll
            for (int t = 0; t < NT; ++t) {
              int c[4];
              mma_s8_16832(c, lb.f[0], hb.f[0], lb.f[2], hb.f[2], bl[t][0], bl[t][1], bias);
              mma_s8_16832(c, lb.f[1], hb.f[1], lb.f[3], hb.f[3], bh[t][0], bh[t][1], c);
#pragma unroll
              for (int k = 0; k < 4; ++k)
                acc[i][t][k] = fmaf(k < 2 ? s_lo : s_hi, __int_as_float(c[k]) - off[t][k & 1], acc[i][t][k]);
            }
          }
        }
    }
  }

  cp_async_wait<0>();
  __syncthreads();                                 // every warp is done with its ring
  // the warps' sums meet in shared memory: element (token, feature) of warp w at red[(w * kTokens + token) * kPitch + feature]
  float* mine = red + warp * T::kTokens * T::kPitch;
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      float* r = mine + (8 * t + 2 * q) * T::kPitch + 16 * i + g;
      r[0] = acc[i][t][0];
      r[T::kPitch] = acc[i][t][1];
      r[8] = acc[i][t][2];
      r[T::kPitch + 8] = acc[i][t][3];
    }
  __syncthreads();
  auto store = [&](int tok, int f, float sum) {
    const int m = m0 + tok, n = n0 + f;
    if (m >= p.M || n >= p.N) return;
    const float y = sum * (QUANT ? q_scale[tok] : ld_global_f32(p.x_scale + m));
    const uint16_t bits = p.out_bf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(y)) : __half_as_ushort(__float2half_rn(y));
    const size_t at = static_cast<size_t>(m) * p.ld_out + n;
    reinterpret_cast<uint16_t*>(p.out)[at] = bits;
    for (int e = 0; e < p.n_extra; ++e) reinterpret_cast<uint16_t*>(p.out_extra[e])[at] = bits;
  };
  const int tokens = min(T::kTokens, p.M - m0);
  for (int i = threadIdx.x; i < tokens * T::kFeatures; i += T::kThreads) {
    const int tok = i / T::kFeatures, f = i % T::kFeatures;
    float* r = red + tok * T::kPitch + f;
    float sum = r[0];
#pragma unroll
    for (int w = 1; w < WARPS; ++w) sum += r[w * T::kTokens * T::kPitch];
    if (splits == 1) store(tok, f, sum);
    else r[0] = sum;                               // (this thread alone reads and writes the element)
  }
  if (splits > 1) {
    cluster_sync_all();
    for (int i = rank * T::kThreads + threadIdx.x; i < tokens * T::kFeatures; i += splits * T::kThreads) {
      const int tok = i / T::kFeatures, f = i % T::kFeatures;
      const uint32_t local = smem_u32(red + tok * T::kPitch + f);
      float part[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) part[r] = r < splits ? ld_dsmem_f32(map_to_cta(local, r)) : 0.f;
      float sum = part[0];
#pragma unroll
      for (int r = 1; r < 8; ++r) sum += part[r];
      store(tok, f, sum);
    }
    cluster_sync_all();                            // peers may still be reading this CTA's shared memory until here
  }
}

}  // namespace sk
