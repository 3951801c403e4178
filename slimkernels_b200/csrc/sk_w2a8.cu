// C ABI of the W2A8 GEMM (declared in include/sk_w2a8.h) plus the small kernels around the main one:
// weight repack / unrepack, and a CUDA-core checker kernel that reads the reference byte layout directly.
#include "../../include/sk_w2a8.h"

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <mutex>
#include <new>
#include <vector>

#include "activation.cuh"
#include "w2a8_umma.cuh"
#include "w2a8_decode.cuh"
#include "w2a8_stream.cuh"
#include "w2a8_direct.cuh"
#include "w2a8_pair.cuh"
#include "weight_prep.cuh"

namespace sk {

constexpr int kChipSms = 148;    // a B200's SMs, for grids and rules that no plan (which asks the device) belongs to

// ------------------------------------------------------------------------------------------------
// Tiled weight order.  Block (tile T, k-block B) is 4096 bytes at ((T * k_blocks + B) * 4096); inside it the
// 32-bit word for (row r, 16-code chunk c) sits at byte (c / 4) * 2048 + r * 16 + (c % 4) * 4 and holds
//   sum_{j=0..3} sum_{b=0..3} code[n = 128 T + r][k = 128 B + 16 c + 4 j + b] << (4 b + 2 (j & 1) + 16 (j >> 1)),
// i.e. nibble b of each 16-bit half holds two codes whose low 2 bits, after a mask, are byte-permute selectors.
// The source byte for codes 4j..4j+3 of that chunk (matrix_packer order: first code in bits 7:6) is
// w_packed[n][(128 B + 16 c) / 4 + j].
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t tiled_word_from_bytes(const uint8_t (&src)[4]) {
  uint32_t w = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const uint32_t code = (src[j] >> (6 - 2 * b)) & 3u;
      w |= code << (4 * b + 2 * (j & 1) + 16 * (j >> 1));
    }
  }
  return w;
}

__global__ void repack_kernel(const uint8_t* __restrict__ w_packed, uint32_t* __restrict__ w_tiled, long long N,
                              long long K, int k_blocks, long long total_words) {
  const long long row_bytes = K / 4;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total_words;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    // idx enumerates destination words in memory order
    const long long block = idx >> 10;             // 1024 words per 4 KiB block
    const int in_block = static_cast<int>(idx & 1023);
    const int half = in_block >> 9;                // 512 words per half
    const int r = (in_block >> 2) & 127;
    const int c = half * 4 + (in_block & 3);
    const long long T = block / k_blocks, B = block % k_blocks;
    const long long n = T * 128 + r;
    const long long k = B * 128 + 16 * c;
    uint8_t src[4] = {0, 0, 0, 0};
    if (n < N) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (k + 4 * j < K) src[j] = w_packed[n * row_bytes + k / 4 + j];
    }
    w_tiled[idx] = tiled_word_from_bytes(src);
  }
}

// The same permutation for plan creation, with the scales of a group-size-128 weight tiled in the same launch: one CTA of
// 128 threads per 4 KiB block, a thread takes one feature's 128 codes (two 16-byte loads, two 16-byte stores; the
// source line's other three blocks are read by neighbouring CTAs and come from L2).  Rows 16-byte aligned, K % 128 == 0.
__global__ void __launch_bounds__(128)
tile_weight_kernel(const uint8_t* __restrict__ w_packed, uint8_t* __restrict__ w_tiled, const __half* __restrict__ w_scale,
                   __half* __restrict__ w_scale_tiled, long long N, long long K, int k_blocks) {
  const int r = threadIdx.x;
  const long long T = blockIdx.y, B = blockIdx.x;
  const long long block = T * k_blocks + B;
  const long long n = T * 128 + r;
  uint4 in[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
  if (n < N) {
    const uint4* src = reinterpret_cast<const uint4*>(w_packed + n * (K / 4) + B * 32);
    in[0] = src[0];
    in[1] = src[1];
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t v[4] = {in[h].x, in[h].y, in[h].z, in[h].w};
    uint32_t o[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const uint8_t b[4] = {static_cast<uint8_t>(v[c]), static_cast<uint8_t>(v[c] >> 8), static_cast<uint8_t>(v[c] >> 16),
                            static_cast<uint8_t>(v[c] >> 24)};
      o[c] = tiled_word_from_bytes(b);
    }
    *reinterpret_cast<uint4*>(w_tiled + block * 4096 + h * 2048 + r * 16) = make_uint4(o[0], o[1], o[2], o[3]);
  }
  if (w_scale_tiled) w_scale_tiled[block * 128 + r] = n < N ? w_scale[static_cast<size_t>(B) * N + n] : __float2half(0.f);
}

// The scales of a group-size-128 weight in the order the split decode kernel (3) streams them: [n_tiles][k_blocks][128
// features] (rows past N are zero), so that the scales of a CTA's K range are one contiguous run.
__global__ void tile_scales_kernel(const __half* __restrict__ w_scale, __half* __restrict__ tiled, long long N,
                                   int k_blocks, long long total) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i % 128);
    const long long t = i / 128;
    const int g = static_cast<int>(t % k_blocks);
    const long long n = (t / k_blocks) * 128 + r;
    tiled[i] = n < N ? w_scale[static_cast<size_t>(g) * N + n] : __float2half(0.f);
  }
}

__global__ void unrepack_kernel(const uint32_t* __restrict__ w_tiled, uint8_t* __restrict__ w_packed, long long N,
                                long long K, int k_blocks, long long total_words) {
  const long long row_bytes = K / 4;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total_words;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long block = idx >> 10;
    const int in_block = static_cast<int>(idx & 1023);
    const int half = in_block >> 9;
    const int r = (in_block >> 2) & 127;
    const int c = half * 4 + (in_block & 3);
    const long long T = block / k_blocks, B = block % k_blocks;
    const long long n = T * 128 + r;
    const long long k = B * 128 + 16 * c;
    if (n >= N) continue;
    const uint32_t w = w_tiled[idx];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (k + 4 * j >= K) continue;
      uint32_t byte = 0;
#pragma unroll
      for (int b = 0; b < 4; ++b) byte |= ((w >> (4 * b + 2 * (j & 1) + 16 * (j >> 1))) & 3u) << (6 - 2 * b);
      w_packed[n * row_bytes + k / 4 + j] = static_cast<uint8_t>(byte);
    }
  }
}

// ------------------------------------------------------------------------------------------------
// CUDA-core checker kernel.  Reads the reference byte layout (uint8 [N, K/4], first code in bits 7:6)
// directly, so it does not depend on the repack, the tensor-core path or TMA.  One thread per output
// (m, n): 32 consecutive n per warp (x loads are warp-uniform), exact int32 group partials via dp4a,
// fp32 scaling in group order.  Used to cross-check the tcgen05 kernel at sizes the CPU oracle cannot reach.
// ------------------------------------------------------------------------------------------------
__global__ void w2a8_simt_kernel(const int8_t* __restrict__ x_q, long long ld_x, const float* __restrict__ x_scale,
                                 const uint8_t* __restrict__ w_packed, const __half* __restrict__ w_scale,
                                 void* __restrict__ out, long long ld_out, int32_t* __restrict__ partials, int M, int N,
                                 int K, int G, int zero_point, int out_bf16) {
  const int n = blockIdx.x * 32 + threadIdx.x;
  const int m = blockIdx.y * blockDim.y + threadIdx.y;
  if (n >= N || m >= M) return;
  const uint8_t* wrow = w_packed + static_cast<size_t>(n) * (K / 4);
  const int8_t* xrow = x_q + static_cast<size_t>(m) * ld_x;
  const int groups = K / G;
  float acc = 0.f;
  for (int g = 0; g < groups; ++g) {
    int32_t part = 0;
    for (int k = g * G; k < (g + 1) * G; k += 4) {
      const uint32_t b = wrow[k >> 2];
      const int c0 = static_cast<int>((b >> 6) & 3u) - zero_point, c1 = static_cast<int>((b >> 4) & 3u) - zero_point;
      const int c2 = static_cast<int>((b >> 2) & 3u) - zero_point, c3 = static_cast<int>(b & 3u) - zero_point;
      const uint32_t wv = (static_cast<uint32_t>(c0) & 0xffu) | ((static_cast<uint32_t>(c1) & 0xffu) << 8) |
                          ((static_cast<uint32_t>(c2) & 0xffu) << 16) | ((static_cast<uint32_t>(c3) & 0xffu) << 24);
      const int xv = *reinterpret_cast<const int*>(xrow + k);
      part = __dp4a(xv, static_cast<int>(wv), part);
    }
    if (partials) partials[(static_cast<size_t>(g) * M + m) * N + n] = part;
    acc = fmaf(__half2float(w_scale[static_cast<size_t>(g) * N + n]), static_cast<float>(part), acc);
  }
  if (out) {
    const float y = acc * x_scale[m];
    uint16_t* o = reinterpret_cast<uint16_t*>(out) + static_cast<size_t>(m) * ld_out + n;
    *o = out_bf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(y)) : __half_as_ushort(__float2half_rn(y));
  }
}

// ------------------------------------------------------------------------------------------------
// Launch-floor probe: what a decode-sized launch costs before it moves a byte.  Same grid, cluster, block size,
// dynamic shared memory and launch attributes as the decode kernel would use, and the same fixed work per CTA
// (barrier initialisation, tensor-memory allocation, one CTA barrier, the cluster barrier of the split-K reduction,
// release); no copies, no arithmetic.  A chain of these in a CUDA graph gives the time per launch below which no
// kernel of this geometry can go.
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(DecodeTraits<16>::kThreads, 2) launch_floor_kernel(int* sink) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint32_t tmem_slot;
  __shared__ __align__(8) unsigned long long bars[16];
  grid_dep_launch_dependents();
  if (threadIdx.x == 0) {
    for (int i = 0; i < 16; ++i) mbar_init(smem_u32(&bars[i]), 1);
    fence_mbar_init();
  }
  if (threadIdx.x / 32 == 1) {
    tmem_alloc(smem_u32(&tmem_slot), 256);
    tmem_relinquish();
  }
  tcgen05_fence_before_sync();
  __syncthreads();
  tcgen05_fence_after_sync();
  grid_dep_wait();
  if (gridDim.z > 1) cluster_sync_all();
  if (sink && smem_raw[threadIdx.x] == 0xff && tmem_slot == 0xffffffffu) *sink = 1;   // keeps the dynamic allocation referenced
  tcgen05_fence_before_sync();
  __syncthreads();
  if (threadIdx.x / 32 == 1) {
    tcgen05_fence_after_sync();
    tmem_dealloc(tmem_slot, 256);
  }
}

// ------------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------------
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

struct CachedMap {
  const void* ptr;
  long long M, ld;
  int block_m;
  CUtensorMap map;
};

}  // namespace sk

struct sk_w2a8_plan {
  int device = 0;
  long long N = 0, K = 0;
  int G = 128, zero_point = 1, out_dtype = SK_OUT_F16;
  int k_blocks = 0, n_tiles = 0, sm_count = sk::kChipSms;
  const uint8_t* w_rowmajor = nullptr;  // borrowed (may be null when created from a tiled buffer)
  const uint8_t* w_tiled = nullptr;     // in the plan's storage, or borrowed
  const __half* w_scale = nullptr;      // borrowed
  __half* w_scale_tiled = nullptr;      // in the plan's storage, group size 128: [n_tiles][k_blocks][128] copy of the scales
  int* status = nullptr;                // device; first in the plan's storage, one block that also holds the tiled copies
  bool external_storage = false;        // that block is the caller's (sk_w2a8_plan_create_in)
  // balanced-split decode kernel: scratch for the partial sums of tiles shared between CTAs, and their counters
  float* stream_scratch = nullptr;      // device, owned; allocated when an option asks for that kernel (stream_setup)
  int* stream_counters = nullptr;       // device, owned; zero between launches
  int stream_ctas = 0, stream_slots = 0;
  bool stream_failed = false;           // there was no memory for them: the split decode kernel takes those calls
  int last_cuda_error = 0;
  int opt_kernel = 0, opt_token_tile = 0, opt_split_k = 0, opt_persistent = 0, opt_pdl = 0, opt_tma_store = 0;
  long long opt_wait_limit = 0;         // 0: the default limit
  int opt_skip_copy = 0;                // failure-path test hook: 1 + index of the K block whose copies are left out
  std::vector<sk::CachedMap> maps;      // small cache of activation tensor maps
  std::mutex mu;
};

namespace sk {

static int cuda_fail(sk_w2a8_plan* plan, cudaError_t e) {
  if (plan) plan->last_cuda_error = static_cast<int>(e);
  (void)cudaGetLastError();
  return e == cudaErrorMemoryAllocation ? SK_ERR_OUT_OF_MEMORY : SK_ERR_CUDA;
}

#ifdef SK_TRACE
static long long* g_trace_buffer = nullptr;
#endif

constexpr size_t kMapCache = 40;   // cached tensor maps per plan (activations and up to 8 output destinations)

struct LaunchChoice {
  int kernel;      // 1 tcgen05 (general), 2 CUDA-core checker, 3 tcgen05 (decode: token tiles 16 / 32, group size 128),
                   // 4 tcgen05 cta_group::2 (pairs of CTAs share a 256-token tile; group size 128, even number of feature tiles),
                   // 5 tcgen05 (decode, one token tile, K range of the whole problem cut into equal CTA ranges)
  int token_tile;  // 16 / 32 / 64 / 128
  int split_k;     // 1 / 2 / 4 / 8
  int persistent;  // 1: one resident set of CTAs walks all tiles
  int ctas;        // CTAs launched
  int mix_tiles1 = 0, mix_split = 0;   // decode kernel 3, mixed launch (see w2a8_decode.cuh); split_k then reports mix_split
};

// Options that take calls away from the direct kernel.
static bool options_force_tcgen05(const sk_w2a8_plan* plan) {
  return plan->opt_kernel || plan->opt_token_tile || plan->opt_split_k || plan->opt_persistent || plan->opt_skip_copy;
}
// Measured on B200 (M = 16): of the tcgen05 decode kernels the balanced split wins once every SM has ~64 K blocks or more to
// stream (70B-class projections: 53 against 70 us on 57344 x 8192); below that its longer tail -- partial sums meet in L2,
// three global round trips -- costs more than the even load saves.  Its 32-token variant is slower throughout.
static bool stream_pays_from(const sk_w2a8_plan* plan) {
  return static_cast<long long>(plan->n_tiles) * plan->k_blocks >= 64LL * plan->sm_count;
}

static LaunchChoice choose(const sk_w2a8_plan* plan, long long M) {
  LaunchChoice c;
  if (plan->opt_token_tile) c.token_tile = plan->opt_token_tile;
  else c.token_tile = M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : M <= 128 ? 128 : 256;
  const bool decode_ok = plan->G == 128 && c.token_tile <= 32;
  // Decode sizes that are one token tile go to the balanced-split kernel (5) where it pays; a forced split (SK_OPT_SPLIT_K) or
  // several token tiles go to the kernel that splits over clusters (3).  Small calls without options are the direct kernel's
  // (choose_direct), so kernel 5 runs only under options, and those that lead here have its scratch allocated (stream_wanted).
  const bool stream_ok = decode_ok && M <= c.token_tile && plan->opt_split_k <= 1 && plan->K % 256 == 0 && !plan->stream_failed;
  const bool stream_pays = stream_ok && c.token_tile == 16 && stream_pays_from(plan);
  c.kernel = plan->opt_kernel && plan->opt_kernel != 6 ? plan->opt_kernel : (stream_pays ? 5 : decode_ok ? 3 : 1);
  if (c.kernel == 5 && !stream_ok) c.kernel = 3;
  if (c.kernel == 3 && !decode_ok) c.kernel = 1;
  const int groups = static_cast<int>(plan->K / plan->G);
  if (c.kernel == 5) {
    c.split_k = 1;
    c.persistent = 0;
    const long long units = static_cast<long long>(plan->n_tiles) * (plan->k_blocks / 2);
    c.ctas = plan->stream_scratch ? plan->stream_ctas : static_cast<int>(units < 2 * plan->sm_count ? units : 2 * plan->sm_count);
    return c;
  }
  if (plan->opt_split_k) c.split_k = plan->opt_split_k;
  else {
    // Fill the machine in ONE wave: split the K range of a tile over a cluster while the CTAs still fit the
    // resident capacity (2 CTAs per SM for token tiles <= 32, else 1) and every CTA keeps enough groups to
    // amortise its prologue (8 = two pipeline stages of the decode kernel, else 4).
    const long long tiles = plan->n_tiles * ((M + c.token_tile - 1) / c.token_tile);
    const long long capacity = static_cast<long long>(plan->sm_count) * (c.token_tile <= 32 ? 2 : 1);
    const int min_groups = c.kernel == 3 ? 8 : 4;
    int s = 1;
    if (c.token_tile <= 64)
      while (s < 8 && tiles * (2 * s) <= capacity && groups / (2 * s) >= min_groups) s *= 2;
    c.split_k = s;
  }
  if (c.split_k > groups || c.token_tile == 192) c.split_k = 1;
  // Decode kernel, one token tile, more feature tiles than SMs (but fewer than CTA slots): with one CTA per tile a
  // few SMs carry two whole tiles and everybody waits for them.  Mixed launch instead: one CTA per tile for as many
  // tiles as there are SMs (rounded down to whole clusters of four), the tiles beyond that split 4 ways (or 2 ways,
  // if there are too many for that) so that they spread over the second CTA slot of many SMs in small pieces.
  if (c.kernel == 3 && !plan->opt_split_k && M <= c.token_tile && c.split_k == 1) {
    const int slots = 2 * plan->sm_count;
    const int tiles1 = (plan->sm_count / 4) * 4;
    const int rest = plan->n_tiles - tiles1;
    if (rest > 0 && plan->n_tiles < slots) {
      if (tiles1 + 4 * rest <= slots && groups >= 16) { c.mix_tiles1 = tiles1; c.mix_split = 4; }
      else if ((rest % 2) == 0 && tiles1 + 2 * rest <= slots && groups >= 8) { c.mix_tiles1 = tiles1; c.mix_split = 2; }
      if (c.mix_split) c.split_k = c.mix_split;
    }
  }
  // With more tiles than the machine holds at once, one resident set of CTAs can walk the tiles instead (option
  // SK_OPT_PERSISTENT = 2): the pipeline of the next tile fills while the previous tile is written out through TMA
  // stores.  Measured on B200 it is not reliably faster than one CTA per tile (all CTAs then move in lock-step and
  // hit L2 in bursts), so it is not the default.
  const long long tiles = plan->n_tiles * ((M + c.token_tile - 1) / c.token_tile);
  const long long capacity = static_cast<long long>(plan->sm_count) * (c.token_tile <= 32 ? 2 : 1);
  c.persistent = (plan->opt_persistent == 2 && tiles > capacity) ? 1 : 0;
  if (c.split_k > 1 || (c.token_tile != 128 && c.token_tile != 256)) c.persistent = 0;
  c.ctas = static_cast<int>(c.persistent ? (tiles < capacity ? tiles : capacity) : tiles * c.split_k);
  if (c.mix_split) c.ctas = c.mix_tiles1 + (plan->n_tiles - c.mix_tiles1) * c.mix_split;
  // Pairs of CTAs (cta_group::2) are an option (SK_OPT_KERNEL = 4), not the default: measured on B200 the pair
  // kernel runs at ~1400 TOP/s where one CTA per tile runs at ~2300.  Its MMAs themselves run at full rate (128.8
  // cycles per 256 x 256 x 32), but every hand-over between the two CTAs costs ~290 cycles (remote mbarrier arrival,
  // multicast commit), two of them sit in the cycle MMA -> epilogue -> MMA of each of the two accumulator buffers that
  // fit tensor memory at 256 tokens, and the epilogue is as long as the MMAs of a group.
  const bool pair_ok = c.token_tile == 256 && plan->G == 128 && (plan->n_tiles % 2) == 0 && !c.persistent && c.split_k == 1;
  if (c.kernel == 4 && !pair_ok) c.kernel = 1;
  return c;
}

template <int BLOCK_M, int EPI_WGS, int EXP_WARPS, int LSTAGES, int ESTAGES, int ACC_BUFS, bool DUMP, bool A_TMEM = false,
          bool PERSIST = false, bool SPLIT = false, bool OTHER_G = false>
static int launch_umma(sk_w2a8_plan* plan, const CUtensorMap& map, const CUtensorMap& out_map,
                       const ExtraOutMaps& extra_maps, const GemmParams& prm, int m_tiles, int split_k,
                       int persistent_ctas, cudaStream_t stream) {
  using L = KernelTraits<BLOCK_M, EPI_WGS, EXP_WARPS, LSTAGES, ESTAGES, ACC_BUFS, A_TMEM, PERSIST>;
  auto kern = w2a8_umma_kernel<BLOCK_M, EPI_WGS, EXP_WARPS, LSTAGES, ESTAGES, ACC_BUFS, DUMP, A_TMEM, PERSIST, SPLIT, OTHER_G>;
  static int configured_device_mask[64] = {0};
  if (plan->device < 64 && !configured_device_mask[plan->device]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kDynamicBytes);
    if (e != cudaSuccess) return cuda_fail(plan, e);
    configured_device_mask[plan->device] = 1;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = PERSIST ? dim3(static_cast<unsigned>(persistent_ctas), 1, 1) : dim3(plan->n_tiles, m_tiles, split_k);
  cfg.blockDim = dim3(L::kThreads, 1, 1);
  cfg.dynamicSmemBytes = L::kDynamicBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (split_k > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = 1;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = split_k;
    ++na;
  }
  // as for the decode kernels; where the tiles take several waves, set-up is nothing and early CTAs of the next kernel in
  // the last wave's free slots cost 2 % (the MLP block of 4096 tokens: 704 us without, 721 with)
  if (!DUMP && plan->opt_pdl != 1 && prm.small_grid) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, map, out_map, extra_maps, prm);
  if (e != cudaSuccess) return cuda_fail(plan, e);
  return SK_OK;
}

template <int TOK, bool DUMP>
static int launch_decode(sk_w2a8_plan* plan, const CUtensorMap& map, const GemmParams& prm, int m_tiles, int split_k,
                         cudaStream_t stream, int mixed_ctas = 0) {
  using L = DecodeTraits<TOK>;
  auto kern = w2a8_decode_kernel<TOK, DUMP>;
  static int configured_device_mask[64] = {0};
  if (plan->device < 64 && !configured_device_mask[plan->device]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kDynamicBytes);
    if (e != cudaSuccess) return cuda_fail(plan, e);
    configured_device_mask[plan->device] = 1;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = mixed_ctas > 0 ? dim3(mixed_ctas, 1, 1) : dim3(plan->n_tiles, m_tiles, split_k);
  cfg.blockDim = dim3(L::kThreads, 1, 1);
  cfg.dynamicSmemBytes = L::kDynamicBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (mixed_ctas > 0) {            // clusters of four along x: four single-tile CTAs, or the shares of one or two tiles
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = 4;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    ++na;
  } else if (split_k > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = 1;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = split_k;
    ++na;
  }
  // Programmatic dependent launch: this kernel's set-up and first weight copies may overlap the tail of the previous
  // kernel in the stream (the kernel itself waits for that kernel before it touches activations or outputs, and its
  // roles sit in griddepcontrol.wait rather than poll).  SK_OPT_DEPENDENT_LAUNCH = 1 launches plainly.
  if (!DUMP && plan->opt_pdl != 1) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, map, prm);
  if (e != cudaSuccess) return cuda_fail(plan, e);
  return SK_OK;
}

template <int TOK, int EXP_WARPS>
static int launch_stream(sk_w2a8_plan* plan, const CUtensorMap& map, const GemmParams& prm, cudaStream_t stream) {
  using L = StreamTraits<TOK, EXP_WARPS>;
  auto kern = w2a8_stream_kernel<TOK, EXP_WARPS>;
  static int configured_device_mask[64] = {0};
  if (plan->device < 64 && !configured_device_mask[plan->device]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kDynamicBytes);
    if (e != cudaSuccess) return cuda_fail(plan, e);
    configured_device_mask[plan->device] = 1;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(plan->stream_ctas, 1, 1);
  cfg.blockDim = dim3(L::kThreads, 1, 1);
  cfg.dynamicSmemBytes = L::kDynamicBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  int na = 0;
  if (plan->opt_pdl != 1) {   // programmatic dependent launch, as for the other decode kernel
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, map, prm);
  if (e != cudaSuccess) return cuda_fail(plan, e);
  return SK_OK;
}

static int dispatch_stream(sk_w2a8_plan* plan, int token_tile, const CUtensorMap& map, const GemmParams& prm,
                           cudaStream_t stream) {
  // (the kernel can be built with 8 or 16 expander warps and one CTA per SM; measured on B200 that is slower than
  // two CTAs of four expander warps per SM)
  return token_tile == 16 ? launch_stream<16, 4>(plan, map, prm, stream) : launch_stream<32, 4>(plan, map, prm, stream);
}

// Geometry of the balanced-split decode kernel for a plan: how many CTAs, and the most CTAs that share one tile.
// want_ctas = 0: two CTAs per SM, but no CTA with less than one half stage.
static void stream_geometry(const sk_w2a8_plan* plan, int want_ctas, int* ctas_out, int* slots_out) {
  const int units_per_tile = plan->k_blocks / 2;
  const long long units = static_cast<long long>(plan->n_tiles) * units_per_tile;
  long long ctas = want_ctas > 0 ? want_ctas : 2LL * plan->sm_count;
  if (ctas > units) ctas = units;
  int slots = 1;
  for (long long t = 0; t < plan->n_tiles; ++t) {
    const int first = stream_owner(units, static_cast<int>(ctas), t * units_per_tile);
    const int last = stream_owner(units, static_cast<int>(ctas), (t + 1) * units_per_tile - 1);
    if (last - first + 1 > slots) slots = last - first + 1;
  }
  *ctas_out = static_cast<int>(ctas);
  *slots_out = slots;
}

// (Re)allocates the scratch buffer and the counters of the balanced-split decode kernel.  Not on the call path:
// sk_w2a8_set_option only.  The device of the plan is current.
static int stream_setup(sk_w2a8_plan* plan, int want_ctas) {
  if (plan->stream_scratch) { cudaFree(plan->stream_scratch); plan->stream_scratch = nullptr; }
  if (plan->stream_counters) { cudaFree(plan->stream_counters); plan->stream_counters = nullptr; }
  plan->stream_ctas = plan->stream_slots = 0;
  plan->stream_failed = true;
  if (plan->G != 128 || (plan->K % 256) != 0) return SK_OK;   // whole half stages only: the other decode kernel serves the rest
  int ctas = 0, slots = 0;
  stream_geometry(plan, want_ctas, &ctas, &slots);
  const size_t bytes = static_cast<size_t>(plan->n_tiles) * slots * StreamTraits<32>::kSlotFloats * sizeof(float);
  cudaError_t e = cudaMalloc(&plan->stream_scratch, bytes);
  if (e != cudaSuccess) { plan->stream_scratch = nullptr; return cuda_fail(plan, e); }
  const size_t cbytes = static_cast<size_t>(plan->n_tiles) * StreamTraits<32>::kEpiWarps * sizeof(int);
  e = cudaMalloc(&plan->stream_counters, cbytes);
  if (e == cudaSuccess) e = cudaMemset(plan->stream_counters, 0, cbytes);
  if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);     // (launches on non-blocking streams are not ordered after it)
  if (e != cudaSuccess) {
    cudaFree(plan->stream_scratch);
    plan->stream_scratch = nullptr;
    if (plan->stream_counters) { cudaFree(plan->stream_counters); plan->stream_counters = nullptr; }
    return cuda_fail(plan, e);
  }
  plan->stream_ctas = ctas;
  plan->stream_slots = slots;
  plan->stream_failed = false;
  return SK_OK;
}

// An option that leads calls of up to 16 tokens to choose(), where large weights get the balanced-split kernel.
static void stream_wanted(sk_w2a8_plan* plan) {
  if (plan->stream_scratch || plan->stream_failed || plan->G != 128 || plan->K % 256 != 0 || !stream_pays_from(plan)) return;
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cudaThreadExchangeStreamCaptureMode(&mode);
  int cur = -1;
  cudaGetDevice(&cur);
  (void)cudaSetDevice(plan->device);
  (void)stream_setup(plan, 0);
  if (cur >= 0 && cur != plan->device) (void)cudaSetDevice(cur);
  cudaThreadExchangeStreamCaptureMode(&mode);
}

// Where a plan's buffers sit in one block of storage (256-byte aligned offsets; -1: the plan has no such buffer).
struct PlanLayout {
  long long status, w_tiled, w_scale_tiled, total;
};
static PlanLayout plan_layout(const sk_w2a8_plan* plan, int w_layout) {
  PlanLayout l;
  long long o = 0;
  auto take = [&o](long long bytes) {
    const long long at = o;
    o += (bytes + 255) & ~255LL;
    return at;
  };
  const long long blocks = static_cast<long long>(plan->n_tiles) * plan->k_blocks;
  l.status = take(sizeof(int));
  l.w_tiled = w_layout == SK_WEIGHT_ROWMAJOR ? take(blocks * kWpBytes) : -1;
  l.w_scale_tiled = plan->G == 128 ? take(blocks * kTileN * static_cast<long long>(sizeof(__half))) : -1;
  l.total = o;
  return l;
}

// ---------------------------------------------------------------------------------------------- direct decode kernel (6)
struct DirectChoice {
  int mt, nt, warps;          // 16-feature tiles per CTA, 8-token tiles per CTA, warps
  int split;                  // CTAs (one cluster) sharing the K range of a tile
  int ctas;
};

// Activations the direct kernel quantises itself: at most this many elements in all, and no more than two CTAs per SM.  Every CTA reads them, so the limit is
// what a CTA can read and convert in less time than a launch (one token through 4096 x 4096, a whole call: 9.4 us against 12.6).
constexpr long long kDirectQuantElements = 8192;

// Whether the kernel takes the scales from the plan's copy: only where the decode kernels, which do, served these calls too.  A
// caller who rewrites the scales in stream order finds them read live everywhere else, as the general kernel does.
static bool direct_reads_copy(const sk_w2a8_plan* plan, long long M) { return plan->G == 128 && M <= 32; }

// The launch-floor probe of the direct kernel: its grid, cluster, threads and dynamic shared memory, and its barriers; nothing
// else (it has no tensor memory to allocate; its registers, which bound the CTAs of an SM, are not imitated).
__global__ void __launch_bounds__(256) direct_floor_kernel(const DirectParams p) {
  extern __shared__ uint8_t smem_raw[];
  grid_dep_launch_dependents();
  grid_dep_wait();
  __syncthreads();
  if (gridDim.z > 1) {
    cluster_sync_all();
    cluster_sync_all();
  }
  if (p.out && smem_raw[threadIdx.x] == 0xff) *static_cast<uint8_t*>(p.out) = 1;   // (never: keeps the allocation referenced)
}

template <int MT, int NT, int WARPS, int DEPTH, int MIN_CTAS, int GPB, bool LIVE, bool QUANT = false>
static int launch_direct(sk_w2a8_plan* plan, const DirectParams& prm, int split, cudaStream_t stream) {
  using T = DirectTraits<MT, NT, WARPS, DEPTH, GPB, LIVE>;
  auto kern = prm.floor_probe ? direct_floor_kernel : w2a8_direct_kernel<MT, NT, WARPS, DEPTH, MIN_CTAS, GPB, LIVE, QUANT>;
  constexpr int kMaxQuant = QUANT ? static_cast<int>(kDirectQuantElements) + 8 * (128 + 16) : 0;   // (a rank's range rounds up to a block)
  if constexpr (T::kQuantOffset + kMaxQuant > 48 * 1024) {
    static int configured_device_mask[64][2] = {};
    if (plan->device < 64 && !configured_device_mask[plan->device][prm.floor_probe]) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           prm.floor_probe ? 227 * 1024 : T::kQuantOffset + kMaxQuant);
      if (e != cudaSuccess) return cuda_fail(plan, e);
      configured_device_mask[plan->device][prm.floor_probe] = 1;
    }
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>((plan->N + T::kFeatures - 1) / T::kFeatures),
                     static_cast<unsigned>((prm.M + T::kTokens - 1) / T::kTokens), static_cast<unsigned>(split));
  cfg.blockDim = dim3(T::kThreads, 1, 1);
  cfg.dynamicSmemBytes = QUANT ? T::kQuantOffset + prm.M * ((prm.k_blocks + split - 1) / split * 128 + 16) : T::kDynamicBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (split > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = 1;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = static_cast<unsigned>(split);
    ++na;
  }
  if (plan->opt_pdl != 1) {   // programmatic dependent launch, as for the other decode kernels
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, prm);
  if (e != cudaSuccess) return cuda_fail(plan, e);
  return SK_OK;
}

// Serves small calls unless an option asks for another kernel (or for its failure-path hook), or scales that are read live do
// not start on a word.  Its time grows with the
// tokens, the tcgen05 kernels' hardly does up to a tile, so the line lies where weights x tokens per SM get large (us, this
// kernel against the better tcgen05 one, group size 128):
//   * up to 24 tokens always: 24 x 57344 x 8192 61 / 80, 24 x 22016 x 4096 15.3 / 17.0, 24 x 4096 x 4096 4.5 / 7.6;
//   * up to 32 tokens below 24 K blocks of a feature tile per SM: 32 x 4096 x 11008 10.4 / 11.5, but 32 x 22016 x 4096 22 / 17.4;
//     with other group sizes always (64: 32 x 22016 x 4096 29 / 52);
//   * up to 128 tokens below 8 such blocks per SM, the weight counted once per 32 tokens: 64 x 2048 x 1024 3.8 / 8.4,
//     64 x 512 x 16384 6.9 / 10.6, but 64 x 4096 x 4096 11.6 / 9.2.
// The shape of a CTA:
//   * 64 features and 4 warps from four such CTAs per SM on (two for 16 tokens): 8 x 57344 x 8192 28.7;
//   * else 32 features and 4 warps from two of those per SM on: 8 x 22016 x 4096 7.2 (9.3 with 64), 24 tokens 15.1 (16.4); with 8
//     tokens and one CTA of 64 per SM, 64 features and 8 warps: 8 x 12288 x 4096 5.2;
//   * else 32 features and 8 warps;
//   * the K range is split over a cluster while the CTAs fit the SMs' slots and every warp keeps four K blocks: 1 x 4096 x
//     11008 in two halves 5.9, but 1 x 4096 x 4096 whole 2.7, in halves 3.7 (the cluster barriers cost more).
static bool choose_direct(const sk_w2a8_plan* plan, long long M, DirectChoice* out) {
  const bool forced = plan->opt_kernel == 6;
  if (!forced && (options_force_tcgen05(plan) || M > 128)) return false;
  if ((reinterpret_cast<uintptr_t>(plan->w_scale) & 3) && !direct_reads_copy(plan, M)) return false;
  DirectChoice c;
  c.nt = M <= 8 ? 1 : M <= 16 ? 2 : M <= 24 ? 3 : 4;
  const long long sms = plan->sm_count;
  const long long token_tiles = (M + 8 * c.nt - 1) / (8 * c.nt);
  const long long work = static_cast<long long>(plan->n_tiles) * plan->k_blocks * token_tiles;
  if (token_tiles > 65535) return false;
  if (!forced && c.nt == 4 && !(M <= 32 && (plan->G != 128 || work < 24 * sms)) && work > 8 * sms) return false;
  const long long per_64 = (plan->N + 63) / 64, per_32 = (plan->N + 31) / 32;
  int slots;                                   // CTAs an SM holds
  if (plan->G < 128) { c.mt = 2; c.warps = 4; slots = 4; }
  else if (c.nt != 3 && per_64 >= (c.nt == 2 ? 2 : 4) * sms) { c.mt = 4; c.warps = 4; slots = 2; }
  else if (c.nt == 1 && per_64 >= sms && per_64 < 2 * sms) { c.mt = 4; c.warps = 8; slots = 2; }
  else if (per_32 >= 2 * sms) { c.mt = 2; c.warps = 4; slots = 2; }
  else { c.mt = 2; c.warps = 8; slots = c.nt <= 2 ? 2 : 1; }
  const long long tiles = (c.mt == 4 ? per_64 : per_32) * token_tiles;
  c.split = 1;
  if (plan->opt_split_k) c.split = plan->opt_split_k;
  else
    while (c.split < 8 && tiles * (2 * c.split) <= slots * sms && plan->k_blocks / (2 * c.split * c.warps) >= 4) c.split *= 2;
  if (c.split > plan->k_blocks) c.split = 1;
  c.ctas = static_cast<int>(tiles * c.split);
  *out = c;
  return true;
}

// <16-feature tiles, 8-token tiles, warps, K blocks in flight per warp, CTAs per SM that registers are kept for, groups per
// K block, scales read from the caller's buffer>
template <int GPB>
static int dispatch_direct_small_groups(sk_w2a8_plan* plan, const DirectChoice& c, const DirectParams& prm, cudaStream_t stream) {
  switch (c.nt) {
    case 1: return launch_direct<2, 1, 4, 4, GPB == 2 ? 5 : 4, GPB, true>(plan, prm, c.split, stream);
    case 2: return launch_direct<2, 2, 4, 4, GPB == 2 ? 4 : 3, GPB, true>(plan, prm, c.split, stream);
    case 3: return launch_direct<2, 3, 4, 4, 2, GPB, true>(plan, prm, c.split, stream);
    default: return launch_direct<2, 4, 4, 4, 2, GPB, true>(plan, prm, c.split, stream);
  }
}
template <bool LIVE>
static int dispatch_direct_blocks(sk_w2a8_plan* plan, const DirectChoice& c, const DirectParams& prm, cudaStream_t stream) {
  if (c.mt == 4 && c.warps == 8) return launch_direct<4, 1, 8, 4, 2, 1, LIVE>(plan, prm, c.split, stream);
  if (c.mt == 4) {
    switch (c.nt) {
      case 1: return launch_direct<4, 1, 4, 4, 3, 1, LIVE>(plan, prm, c.split, stream);
      case 2: return launch_direct<4, 2, 4, 6, 3, 1, LIVE>(plan, prm, c.split, stream);
      default: return launch_direct<4, 4, 4, 4, 2, 1, LIVE>(plan, prm, c.split, stream);
    }
  }
  if (c.warps == 4) {
    switch (c.nt) {
      case 1: return launch_direct<2, 1, 4, 4, LIVE ? 5 : 4, 1, LIVE>(plan, prm, c.split, stream);   // (five CTAs per SM either way)
      case 2: return launch_direct<2, 2, 4, 6, 4, 1, LIVE>(plan, prm, c.split, stream);
      case 3: return launch_direct<2, 3, 4, 6, 3, 1, LIVE>(plan, prm, c.split, stream);
      default: return launch_direct<2, 4, 4, 6, 3, 1, LIVE>(plan, prm, c.split, stream);    // 32 x 12288 x 4096 11.5; two CTAs of four blocks 15.2
    }
  }
  switch (c.nt) {
    case 1: return launch_direct<2, 1, 8, 4, 2, 1, LIVE>(plan, prm, c.split, stream);
    case 2: return launch_direct<2, 2, 8, 4, 2, 1, LIVE>(plan, prm, c.split, stream);
    case 3: return launch_direct<2, 3, 8, 4, 1, 1, LIVE>(plan, prm, c.split, stream);
    default: return launch_direct<2, 4, 8, 4, 1, 1, LIVE>(plan, prm, c.split, stream);
  }
}
static int dispatch_direct(sk_w2a8_plan* plan, const DirectChoice& c, const DirectParams& prm, cudaStream_t stream) {
  if (plan->G == 64) return dispatch_direct_small_groups<2>(plan, c, prm, stream);
  if (plan->G == 32) return dispatch_direct_small_groups<4>(plan, c, prm, stream);
  return direct_reads_copy(plan, prm.M) ? dispatch_direct_blocks<false>(plan, c, prm, stream)
                                        : dispatch_direct_blocks<true>(plan, c, prm, stream);
}

// The same with the activations quantised inside (up to 8 tokens, group sizes from 128 on).
static bool direct_quantises(const sk_w2a8_plan* plan, long long M, const DirectChoice& c) {
  return c.nt == 1 && plan->G >= 128 && M <= 8 && M * plan->K <= kDirectQuantElements && c.ctas <= 2 * plan->sm_count;
}
template <bool LIVE>
static int dispatch_direct_quant_blocks(sk_w2a8_plan* plan, const DirectChoice& c, const DirectParams& prm, cudaStream_t stream) {
  if (c.mt == 4 && c.warps == 8) return launch_direct<4, 1, 8, 4, 2, 1, LIVE, true>(plan, prm, c.split, stream);
  if (c.mt == 4) return launch_direct<4, 1, 4, 4, 3, 1, LIVE, true>(plan, prm, c.split, stream);
  return c.warps == 4 ? launch_direct<2, 1, 4, 4, LIVE ? 5 : 4, 1, LIVE, true>(plan, prm, c.split, stream)
                      : launch_direct<2, 1, 8, 4, 2, 1, LIVE, true>(plan, prm, c.split, stream);
}
static int dispatch_direct_quant(sk_w2a8_plan* plan, const DirectChoice& c, const DirectParams& prm, cudaStream_t stream) {
  return direct_reads_copy(plan, prm.M) ? dispatch_direct_quant_blocks<false>(plan, c, prm, stream)
                                        : dispatch_direct_quant_blocks<true>(plan, c, prm, stream);
}

constexpr int kPairStages = 6;

template <bool DUMP>
static int launch_pair(sk_w2a8_plan* plan, const CUtensorMap& map, const CUtensorMap& out_map,
                       const ExtraOutMaps& extra_maps, const GemmParams& prm, int m_tiles, cudaStream_t stream) {
  using L = PairTraits<kPairStages>;
  auto kern = w2a8_pair_kernel<kPairStages, DUMP>;
  static int configured_device_mask[64] = {0};
  if (plan->device < 64 && !configured_device_mask[plan->device]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kDynamicBytes);
    if (e != cudaSuccess) return cuda_fail(plan, e);
    configured_device_mask[plan->device] = 1;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(plan->n_tiles, m_tiles, 1);
  cfg.blockDim = dim3(L::kThreads, 1, 1);
  cfg.dynamicSmemBytes = L::kDynamicBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;      // the two CTAs of a pair: adjacent feature tiles, same token tile
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, map, out_map, extra_maps, prm);
  if (e != cudaSuccess) return cuda_fail(plan, e);
  return SK_OK;
}

constexpr int kAccBufsSmall = 4;   // accumulator buffers of the token tiles <= 128
constexpr int kAccBufs256 = 2;     // 2 x 256 columns fill the tensor memory
static int acc_bufs_of(int token_tile, int kernel) {
  if (kernel == 3 || kernel == 5) return token_tile == 16 ? DecodeTraits<16>::kAccBufs : DecodeTraits<32>::kAccBufs;
  return token_tile >= 192 ? kAccBufs256 : kAccBufsSmall;
}

// The running sum of one accumulator buffer must stay inside (-2^22, 2^22):
// (K handled per buffer) * 127 * max|code - zp| < 2^22.
static bool running_sum_fits(const sk_w2a8_plan* plan, int token_tile, int split_k, int kernel) {
  const long long groups = plan->K / plan->G;
  const long long groups_cta = (groups + split_k - 1) / split_k;
  const int ab = acc_bufs_of(token_tile, kernel);
  const long long k_per_buf = ((groups_cta + ab - 1) / ab) * plan->G;
  const int mx = plan->zero_point > 3 - plan->zero_point ? plan->zero_point : 3 - plan->zero_point;
  return k_per_buf * 127 * mx < (1LL << 22);
}

// The general kernel's accumulator bias for a launch: the smallest power of two above what a running sum can reach.
static uint32_t accumulator_bias(const sk_w2a8_plan* plan, int token_tile, int split_k) {
  const long long per_block = plan->G < 128 ? 128 / plan->G : 1;
  long long groups_cta = (plan->K / plan->G + split_k - 1) / split_k;
  groups_cta = (groups_cta + per_block - 1) / per_block * per_block;      // (a CTA's range is whole K blocks)
  const int ab = acc_bufs_of(token_tile, 1);
  const int mx = plan->zero_point > 3 - plan->zero_point ? plan->zero_point : 3 - plan->zero_point;
  const long long most = ((groups_cta + ab - 1) / ab) * plan->G * 128 * mx;
  uint32_t bias = 1u << 8;
  while (bias < (1u << 22) && static_cast<long long>(bias) <= most) bias <<= 1;
  return bias;
}

// The launch run_gemm makes for M tokens: the heuristic choice, then the depth check.  A K range too deep for the two
// accumulator buffers of the 256-token tile falls back to 128 tokens (four buffers, half the depth per buffer);
// beyond that the call is refused.
static int resolve_launch(const sk_w2a8_plan* plan, long long M, bool debug_partials, LaunchChoice* out) {
  LaunchChoice ch = choose(plan, M);
  if (debug_partials) {
    if (ch.kernel == 5) { ch.kernel = 3; ch.ctas = static_cast<int>(plan->n_tiles * ((M + ch.token_tile - 1) / ch.token_tile)); }
    ch.split_k = 1; ch.persistent = 0; ch.mix_tiles1 = ch.mix_split = 0;
  }
  // (mixed launch: the CTAs with a tile of their own run the whole depth)
  if (ch.kernel != 2 && !running_sum_fits(plan, ch.token_tile, ch.mix_split ? 1 : ch.split_k, ch.kernel)) {
    if (ch.token_tile >= 192 && !plan->opt_token_tile && running_sum_fits(plan, 128, 1, 1)) {
      ch.token_tile = 128;
      ch.persistent = 0;
      ch.ctas = static_cast<int>(plan->n_tiles * ((M + 127) / 128));
    } else {
      return SK_ERR_BAD_SHAPE;   // K too deep for the int32 running sums of this tile configuration
    }
  }
  *out = ch;
  return SK_OK;
}

// The token tile and K split the general kernel runs M > 32 tokens with: of the tiles up to the heuristic one's size and
// the splits the K range allows, the pair that a simple model gives the least time,
//     waves x (set-up and output + K blocks per CTA x time per K block + cluster reduction),
// with the constants below (one CTA per SM), fitted to sweeps on B200 before the issuers' shorter loop and the epilogue's pairs.
// Against the kernels as they are it is right to 8 % for whole tiles with group size 128 and high elsewhere (medians over 33 to 4096
// tokens, tiles of 64 / 128 / 256 tokens: group size 64 by 22 / 19 / 5 %, 32 by 21 / 8 / 15 %, 256 by 12 / 15 / 20 %), for splits
// 19 % low to 23 % high.  What it is for, the choice, holds: of 280 calls (33 to 4096 tokens, six weights, four group sizes) the launch chosen
// takes within 3 % of the best forced one in all but two kinds.  Where it splits 8 ways into 128 CTAs (96 to 256 x 1024 x 8192) a call
// takes 1.4 to 1.6 times the best launch, as it did before: of these clusters of eight the chip holds 15 at a time.  And 333 x 22016 x 4096
// with group size 128 takes 94.7 us as 256 tokens, 87.1 as 128.
// It replaces "the smallest tile that holds M", which left most SMs idle wherever there are few tiles: 96 x 4096 x 11008
// 38.4 us on 32 CTAs, 15.3 as 128 tokens split 4 ways; 256 x 4096 x 4096 22.4, 13.7 as 64-token tiles; 512 x 4096 x 11008 50.7, 35.2 as
// 128-token tiles (in part the expanders' second group, see w2a8_umma.cuh).
// The launch that resolve_launch names stays where the model sees less than 5 % in it, where its depth check moved it to
// another tile, and where an option forces any part of it.  What is refused is decided before, on that launch.
static void refine_launch(const sk_w2a8_plan* plan, long long M, LaunchChoice* ch) {
  if (ch->kernel != 1 || plan->opt_kernel || plan->opt_token_tile || plan->opt_split_k || plan->opt_persistent) return;
  if (ch->token_tile != (M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : M <= 128 ? 128 : 256)) return;
  struct Tile { int tokens; double us_cta, us_256, us_128, us_64, us_32, us_split; };   // per CTA, per K block by group size, per reduction
  constexpr Tile kTiles[] = {{64, 3.4, 0.50, 0.285, 0.575, 1.04, 3.6}, {128, 4.0, 0.56, 0.365, 0.68, 1.14, 3.8}, {256, 5.3, 0.61, 0.43, 0.87, 1.8, 0.0}};
  const int sms = plan->sm_count;
  auto model = [&](const Tile& t, int split) {
    const long long ctas = static_cast<long long>(plan->n_tiles) * ((M + t.tokens - 1) / t.tokens) * split;
    const long long waves = (ctas + sms - 1) / sms;
    const double us = plan->G > 128 ? t.us_256 : plan->G == 128 ? t.us_128 : plan->G == 64 ? t.us_64 : t.us_32;
    return waves * (t.us_cta + ((plan->k_blocks + split - 1) / split) * us + (split > 1 ? t.us_split : 0.0));
  };
  const Tile* best = nullptr;
  int best_split = 0;
  double best_us = 0.0, now_us = 0.0;
  for (const Tile& t : kTiles) {
    if (t.tokens > ch->token_tile) continue;
    for (int split = 1; split <= 8; split *= 2) {
      if (split > 1 && (plan->k_blocks / split < 4 || t.tokens == 256)) continue;   // (256: the reduction takes longer than it saves)
      if (!running_sum_fits(plan, t.tokens, split, 1)) continue;
      const double us = model(t, split);
      if (t.tokens == ch->token_tile && split == ch->split_k) now_us = us;
      if (!best || us < best_us) { best = &t; best_split = split; best_us = us; }
    }
  }
  if (!best || now_us == 0.0 || best_us > 0.95 * now_us) return;
  ch->token_tile = best->tokens;
  ch->split_k = best_split;
  ch->persistent = 0;
  ch->ctas = static_cast<int>(plan->n_tiles * ((M + best->tokens - 1) / best->tokens) * best_split);
}

// Test aid: the expander's shared-memory image of one 128 x 128 weight block next to the image the TMA writes for the
// same int8 values.  One CTA: (a) copies a 4 KiB tiled block into shared memory and expands it exactly as the general
// kernel's expander threads do (expand16, one row per thread, 16-byte stores into the 128-byte-swizzled K-major
// layout); (b) loads the pre-expanded row-major int8 block through a tensor map with CU_TENSOR_MAP_SWIZZLE_128B -- the
// layout the MMA's shared-memory descriptor expects of both operands; (c) writes both 16 KiB images out and counts
// the bytes that differ.  The wait for the TMA is bounded.
__global__ void __launch_bounds__(128)
expander_image_kernel(const __grid_constant__ CUtensorMap tmap_expanded, const uint8_t* __restrict__ w_tiled_block,
                      int zero_point, uint8_t* __restrict__ image_expander, uint8_t* __restrict__ image_tma,
                      int* __restrict__ mismatches, int* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* wp = smem;                        // [4096] tiled 2-bit block
  uint8_t* wx = smem + 4096;                 // [16384] expander image (1024-aligned: 4096 is)
  uint8_t* wt = smem + 4096 + kWxBytes;      // [16384] TMA image
  __shared__ __align__(8) uint64_t bar;
  __shared__ int abort_flag;
  const uint32_t bar_a = smem_u32(&bar);
  const int row = threadIdx.x;
  if (threadIdx.x == 0) {
    mbar_init(bar_a, 1);
    abort_flag = 0;
    fence_mbar_init();
  }
  for (int i = threadIdx.x; i < kWpBytes / 16; i += blockDim.x)
    reinterpret_cast<uint4*>(wp)[i] = reinterpret_cast<const uint4*>(w_tiled_block)[i];
  __syncthreads();
  if (threadIdx.x == 0) {
    mbar_arrive_expect_tx(bar_a, kWxBytes);
    tma_load_2d(smem_u32(wt), &tmap_expanded, 0, 0, bar_a);
  }
  // (a) as the expander threads of w2a8_umma_kernel, one row per thread
  const uint32_t lut = (static_cast<uint32_t>(0 - zero_point) & 0xffu) | ((static_cast<uint32_t>(1 - zero_point) & 0xffu) << 8) |
                       ((static_cast<uint32_t>(2 - zero_point) & 0xffu) << 16) | ((static_cast<uint32_t>(3 - zero_point) & 0xffu) << 24);
  const uint32_t src = smem_u32(wp) + row * 16;
  const uint4 q0 = ld_shared_v4(src);
  const uint4 q1 = ld_shared_v4(src + 2048);
  const uint32_t words[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
  const uint32_t dst = smem_u32(wx) + row * 128 + ((row & 7) << 4);
#pragma unroll
  for (int c = 0; c < 8; ++c) st_shared_v4(dst ^ (c << 4), expand16(words[c], lut));
  // (b) the TMA image
  const WaitCtx ctx{&abort_flag, status, 200000000ll};
  const bool ok = wait_bounded(bar_a, 0, ctx, kStExpanderFull);
  __syncthreads();
  if (!ok) return;
  // (c)
  int bad = 0;
  for (int i = threadIdx.x; i < kWxBytes / 16; i += blockDim.x) {
    const uint4 a = reinterpret_cast<const uint4*>(wx)[i], b = reinterpret_cast<const uint4*>(wt)[i];
    reinterpret_cast<uint4*>(image_expander)[i] = a;
    reinterpret_cast<uint4*>(image_tma)[i] = b;
    const uint32_t x[4] = {a.x ^ b.x, a.y ^ b.y, a.z ^ b.z, a.w ^ b.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      for (int k = 0; k < 4; ++k) bad += ((x[j] >> (8 * k)) & 0xffu) ? 1 : 0;
  }
  if (bad) atomicAdd(mismatches, bad);
}

// partials[g] holds the running sum of its accumulator buffer; turn it into the group's own partial sum.
__global__ void diff_partials_kernel(int32_t* __restrict__ partials, int groups, long long mn, int acc_bufs) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < mn;
       i += static_cast<long long>(gridDim.x) * blockDim.x)
    for (int g = groups - 1; g >= acc_bufs; --g) partials[g * mn + i] -= partials[(g - acc_bufs) * mn + i];
}

// <tokens, epilogue warpgroups, expander warps, load stages, expanded stages, accumulator buffers>
template <bool SPLIT, bool OTHER_G>
static int dispatch_umma_tile(sk_w2a8_plan* plan, int token_tile, const CUtensorMap& map, const CUtensorMap& out_map,
                              const ExtraOutMaps& extra_maps, const GemmParams& prm, int m_tiles, int split_k, cudaStream_t stream) {
  switch (token_tile) {
    case 16: return launch_umma<16, 1, 8, 4, 4, kAccBufsSmall, false, false, false, SPLIT, OTHER_G>(plan, map, out_map, extra_maps, prm, m_tiles, split_k, 0, stream);
    case 32: return launch_umma<32, 1, 4, 4, 4, kAccBufsSmall, false, false, false, SPLIT, OTHER_G>(plan, map, out_map, extra_maps, prm, m_tiles, split_k, 0, stream);
    case 64: return launch_umma<64, 1, 8, 6, 6, kAccBufsSmall, false, false, false, SPLIT, OTHER_G>(plan, map, out_map, extra_maps, prm, m_tiles, split_k, 0, stream);
    case 128: return launch_umma<128, 2, 8, 6, 6, kAccBufsSmall, false, false, false, SPLIT, OTHER_G>(plan, map, out_map, extra_maps, prm, m_tiles, split_k, 0, stream);
    case 256: return launch_umma<256, 2, 4, 4, 4, kAccBufs256, false, false, false, SPLIT, OTHER_G>(plan, map, out_map, extra_maps, prm, m_tiles, split_k, 0, stream);
    default: return SK_ERR_BAD_ARGUMENT;
  }
}

static int dispatch_umma(sk_w2a8_plan* plan, int token_tile, const CUtensorMap& map, const CUtensorMap& out_map,
                         const ExtraOutMaps& extra_maps, const GemmParams& prm, int m_tiles, int split_k,
                         int persistent_ctas, cudaStream_t stream) {
  if (persistent_ctas > 0 && token_tile == 128)
    return launch_umma<128, 2, 4, 4, 4, kAccBufsSmall, false, false, true>(plan, map, out_map, extra_maps, prm, m_tiles, 1, persistent_ctas, stream);
  if (persistent_ctas > 0 && token_tile == 256)
    return launch_umma<256, 2, 4, 4, 2, kAccBufs256, false, false, true>(plan, map, out_map, extra_maps, prm, m_tiles, 1, persistent_ctas, stream);
  // 192 tokens: the expanded weights live in tensor memory (2 x 192 accumulator columns + 4 x 32 weight columns;
  // no expanded-weight ring in shared memory, so the load ring is 6 stages deep)
  if (token_tile == 192)
    return launch_umma<192, 2, 4, 6, 4, kAccBufs256, false, true>(plan, map, out_map, extra_maps, prm, m_tiles, 1, 0, stream);
  const bool other = plan->G != 128;
  if (split_k > 1)
    return other ? dispatch_umma_tile<true, true>(plan, token_tile, map, out_map, extra_maps, prm, m_tiles, split_k, stream)
                 : dispatch_umma_tile<true, false>(plan, token_tile, map, out_map, extra_maps, prm, m_tiles, split_k, stream);
  return other ? dispatch_umma_tile<false, true>(plan, token_tile, map, out_map, extra_maps, prm, m_tiles, 1, stream)
               : dispatch_umma_tile<false, false>(plan, token_tile, map, out_map, extra_maps, prm, m_tiles, 1, stream);
}

// The debug variants: they store the integer partial sums instead of the scaled output.
static int dispatch_umma_dump(sk_w2a8_plan* plan, int token_tile, const CUtensorMap& map, const ExtraOutMaps& extra_maps,
                              const GemmParams& prm, int m_tiles, cudaStream_t stream) {
  switch (token_tile) {
    case 16: return launch_umma<16, 1, 8, 4, 4, kAccBufsSmall, true>(plan, map, map, extra_maps, prm, m_tiles, 1, 0, stream);
    case 32: return launch_umma<32, 1, 4, 4, 4, kAccBufsSmall, true>(plan, map, map, extra_maps, prm, m_tiles, 1, 0, stream);
    case 64: return launch_umma<64, 1, 8, 6, 6, kAccBufsSmall, true>(plan, map, map, extra_maps, prm, m_tiles, 1, 0, stream);
    case 128: return launch_umma<128, 2, 8, 6, 6, kAccBufsSmall, true>(plan, map, map, extra_maps, prm, m_tiles, 1, 0, stream);
    case 192: return launch_umma<192, 2, 4, 6, 4, kAccBufs256, true, true>(plan, map, map, extra_maps, prm, m_tiles, 1, 0, stream);
    case 256: return launch_umma<256, 2, 4, 4, 4, kAccBufs256, true>(plan, map, map, extra_maps, prm, m_tiles, 1, 0, stream);
    default: return SK_ERR_BAD_ARGUMENT;
  }
}

static int get_x_map(sk_w2a8_plan* plan, const int8_t* x_q, long long M, long long ld_x, int block_m,
                     CUtensorMap* out) {
  std::lock_guard<std::mutex> lock(plan->mu);
  for (const auto& c : plan->maps)
    if (c.ptr == x_q && c.M == M && c.ld == ld_x && c.block_m == block_m) { *out = c.map; return SK_OK; }
  EncodeTiledFn enc = get_encode_fn();
  if (!enc) return SK_ERR_CUDA;
  CachedMap cm;
  cm.ptr = x_q; cm.M = M; cm.ld = ld_x; cm.block_m = block_m;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(plan->K), static_cast<cuuint64_t>(M)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld_x)};
  const cuuint32_t box[2] = {128u, static_cast<cuuint32_t>(block_m)};
  const cuuint32_t estr[2] = {1u, 1u};
  CUresult r = enc(&cm.map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<int8_t*>(x_q), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { plan->last_cuda_error = static_cast<int>(r); return SK_ERR_CUDA; }
  if (plan->maps.size() >= kMapCache) plan->maps.erase(plan->maps.begin());
  plan->maps.push_back(cm);
  *out = cm.map;
  return SK_OK;
}

// Tensor map of an output buffer for TMA stores: 16-bit elements, [M][N] with row pitch ld_out, boxes of 128
// features x box_rows tokens (the whole tile, or 64-token rounds of the persistent kernel), no swizzle.
static int get_out_map(sk_w2a8_plan* plan, const void* out, long long M, long long ld_out, int box_rows,
                       CUtensorMap* res) {
  std::lock_guard<std::mutex> lock(plan->mu);
  for (const auto& c : plan->maps)
    if (c.ptr == out && c.M == M && c.ld == ld_out && c.block_m == -box_rows) { *res = c.map; return SK_OK; }
  EncodeTiledFn enc = get_encode_fn();
  if (!enc) return SK_ERR_CUDA;
  CachedMap cm;
  cm.ptr = out; cm.M = M; cm.ld = ld_out; cm.block_m = -box_rows;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(plan->N), static_cast<cuuint64_t>(M)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld_out) * 2};
  const cuuint32_t box[2] = {128u, static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t estr[2] = {1u, 1u};
  CUresult r = enc(&cm.map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(out), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { plan->last_cuda_error = static_cast<int>(r); return SK_ERR_CUDA; }
  if (plan->maps.size() >= kMapCache) plan->maps.erase(plan->maps.begin());
  plan->maps.push_back(cm);
  *res = cm.map;
  return SK_OK;
}

static DirectParams direct_params(const sk_w2a8_plan* plan, long long M, void* out, long long ld_out) {
  DirectParams prm = {};
  prm.w_tiled = plan->w_tiled;
  prm.w_scale_tiled = plan->w_scale_tiled;
  prm.w_scale = plan->w_scale;
  prm.scale_pieces = (reinterpret_cast<uintptr_t>(plan->w_scale) & 15) == 0 && plan->N % 8 == 0;
  // Borrowed codes are read behind the dependent-launch wait wherever the kernel that took these calls before did, so that a
  // buffer refilled in stream order is seen; the decode kernels (one tile of up to 32 tokens, group size 128) do not wait.
  prm.weights_late = plan->w_rowmajor == nullptr && !direct_reads_copy(plan, M);
  prm.out = out;
  prm.ld_out = ld_out;
  prm.M = static_cast<int>(M);
  prm.N = static_cast<int>(plan->N);
  prm.K = static_cast<int>(plan->K);
  prm.groups = static_cast<int>(plan->K / plan->G);
  prm.k_blocks = plan->k_blocks;
  prm.blocks_per_group = plan->G / 128;
  prm.zero_point = plan->zero_point;
  prm.out_bf16 = plan->out_dtype == SK_OUT_BF16;
  return prm;
}

static int run_gemm(sk_w2a8_plan* plan, long long M, const int8_t* x_q, long long ld_x, const float* x_scale,
                    void* out, long long ld_out, int32_t* partials, cudaStream_t stream,
                    void* const* extra_outs = nullptr, int n_extra = 0, long long scatter_rows = 0,
                    long long scatter_row0 = 0) {
  if (!plan || !x_q) return SK_ERR_NULL_POINTER;
  if (!partials && (!x_scale || !out)) return SK_ERR_NULL_POINTER;
  if (M <= 0 || M > 0x7fffffffLL / 2) return SK_ERR_BAD_SHAPE;
  if (ld_x < plan->K) return SK_ERR_BAD_SHAPE;
  if (!partials && ld_out < plan->N) return SK_ERR_BAD_SHAPE;
  if ((ld_x % 16) != 0 || (reinterpret_cast<uintptr_t>(x_q) & 15) != 0) return SK_ERR_BAD_ALIGNMENT;
  if (out && (reinterpret_cast<uintptr_t>(out) & 1) != 0) return SK_ERR_BAD_ALIGNMENT;

  int cur = -1;
  cudaError_t e = cudaGetDevice(&cur);
  if (e != cudaSuccess) return cuda_fail(plan, e);
  if (cur != plan->device) {
    e = cudaSetDevice(plan->device);
    if (e != cudaSuccess) return cuda_fail(plan, e);
  }
  LaunchChoice ch;
  int rc = resolve_launch(plan, M, partials != nullptr, &ch);
  if (rc != SK_OK) {
    if (cur != plan->device) (void)cudaSetDevice(cur);
    return rc;
  }
  DirectChoice dc;
  if (!partials && scatter_rows == 0 && choose_direct(plan, M, &dc)) {
    DirectParams prm = direct_params(plan, M, out, ld_out);
    prm.x_q = x_q;
    prm.x_scale = x_scale;
    prm.ld_x = ld_x;
    prm.n_extra = n_extra;
    for (int i = 0; i < n_extra; ++i) prm.out_extra[i] = extra_outs[i];
    rc = dispatch_direct(plan, dc, prm, stream);
    if (cur != plan->device) (void)cudaSetDevice(cur);
    return rc;
  }
  if (scatter_rows > 0 && (ch.kernel != 1 || ch.split_k != 1 || (scatter_rows % ch.token_tile) != 0)) {
    // row scatter is the general kernel's: every token tile must belong to one destination
    if (cur != plan->device) (void)cudaSetDevice(cur);
    return SK_ERR_UNAVAILABLE;
  }
  if (!partials) refine_launch(plan, M, &ch);
  if (ch.kernel == 2) {
    if (!plan->w_rowmajor || n_extra > 0) rc = SK_ERR_UNAVAILABLE;
    else {
      dim3 block(32, 8, 1);
      dim3 grid(static_cast<unsigned>((plan->N + 31) / 32), static_cast<unsigned>((M + 7) / 8), 1);
      w2a8_simt_kernel<<<grid, block, 0, stream>>>(x_q, ld_x, x_scale, plan->w_rowmajor, plan->w_scale, out, ld_out,
                                                   partials, static_cast<int>(M), static_cast<int>(plan->N),
                                                   static_cast<int>(plan->K), plan->G, plan->zero_point,
                                                   plan->out_dtype == SK_OUT_BF16);
      e = cudaGetLastError();
      if (e != cudaSuccess) rc = cuda_fail(plan, e);
    }
  } else {
    CUtensorMap map;
    rc = get_x_map(plan, x_q, M, ld_x, ch.kernel == 4 ? 128 : ch.token_tile, &map);
    if (rc == SK_OK) {
      GemmParams prm;
      prm.w_tiled = plan->w_tiled;
      prm.w_scale = plan->w_scale;
      prm.w_scale_tiled = plan->w_scale_tiled;
      prm.x_scale = x_scale;
      prm.out = out;
      prm.n_extra = n_extra;
      prm.scatter_rows = static_cast<int>(scatter_rows);
      prm.scatter_row0 = static_cast<int>(scatter_row0);
      for (int i = 0; i < 7; ++i) prm.out_extra[i] = i < n_extra ? extra_outs[i] : nullptr;
      prm.partials = partials;
      prm.status = plan->status;
      prm.ld_out = ld_out;
      prm.M = static_cast<int>(M);
      prm.N = static_cast<int>(plan->N);
      prm.K = static_cast<int>(plan->K);
      prm.k_blocks = plan->k_blocks;
      prm.steps_per_group = plan->G / 32;
      prm.groups = static_cast<int>(plan->K / plan->G);
      prm.small_grid = ch.ctas <= 2 * plan->sm_count;
      prm.acc_bias = accumulator_bias(plan, ch.token_tile, partials ? 1 : ch.split_k);
      prm.zero_point = plan->zero_point;
      prm.out_bf16 = plan->out_dtype == SK_OUT_BF16;
      prm.wait_limit = plan->opt_wait_limit > 0 ? plan->opt_wait_limit : kWaitLimitCycles;
      prm.fault_skip_kb = plan->opt_skip_copy - 1;
      prm.mix_tiles1 = partials ? 0 : ch.mix_tiles1;
      prm.mix_split = partials ? 0 : ch.mix_split;
      prm.stream_scratch = plan->stream_scratch;
      prm.stream_counters = plan->stream_counters;
      prm.stream_slots = plan->stream_slots;
#ifdef SK_TRACE
      prm.trace = g_trace_buffer;
#endif
      const int m_tiles = static_cast<int>((M + ch.token_tile - 1) / ch.token_tile);
      prm.n_tiles = plan->n_tiles;
      prm.num_tiles = plan->n_tiles * m_tiles;
      // The persistent kernel stores through TMA (and 16-byte vectors for further destinations): the output must be
      // 16-byte aligned with a pitch that is a multiple of 8 elements, N a multiple of 8 (the tensor map's extent in
      // bytes), and with further destinations the feature tiles must be whole.
      bool persist = ch.persistent && scatter_rows == 0 && !partials && (ld_out % 8) == 0 && (plan->N % 8) == 0 &&
                     (reinterpret_cast<uintptr_t>(out) & 15) == 0;
      if (persist && n_extra > 0) {
        if (plan->N % 128) persist = false;
        for (int i = 0; i < n_extra; ++i)
          if (reinterpret_cast<uintptr_t>(extra_outs[i]) & 15) persist = false;
      }
      CUtensorMap out_map = map;   // placeholder where the kernel does not use it
      ExtraOutMaps extra_maps;
      for (int i = 0; i < 7; ++i) extra_maps.map[i] = map;
      if (persist) {
        rc = get_out_map(plan, out, M, ld_out, 64, &out_map);
        if (rc != SK_OK) persist = false, rc = SK_OK;
      }
      // One CTA per tile: the staged tile leaves through one TMA store per destination where the buffers allow it
      // (16-byte aligned, pitch a multiple of 8 elements, N a multiple of 8).
      prm.tma_out = 0;
      if (!persist && !partials && (ch.kernel == 1 || ch.kernel == 4) && ch.split_k == 1 && (ld_out % 8) == 0 && (plan->N % 8) == 0 &&
          (reinterpret_cast<uintptr_t>(out) & 15) == 0 && plan->opt_tma_store != 1) {
        // (row scatter: a destination holds scatter_row0 + scatter_rows rows at least; its map is clipped there)
        const long long map_rows = scatter_rows > 0 ? scatter_row0 + scatter_rows : M;
        bool ok = get_out_map(plan, out, map_rows, ld_out, ch.token_tile, &out_map) == SK_OK;
        for (int i = 0; ok && i < n_extra; ++i)
          ok = (reinterpret_cast<uintptr_t>(extra_outs[i]) & 15) == 0 &&
               get_out_map(plan, extra_outs[i], map_rows, ld_out, ch.token_tile, &extra_maps.map[i]) == SK_OK;
        prm.tma_out = ok ? 1 : 0;
      }
      if (m_tiles > 65535) rc = SK_ERR_BAD_SHAPE;
      else if (partials) {
        if (ch.kernel == 3)
          rc = ch.token_tile == 16 ? launch_decode<16, true>(plan, map, prm, m_tiles, 1, stream)
                                   : launch_decode<32, true>(plan, map, prm, m_tiles, 1, stream);
        else if (ch.kernel == 4) rc = launch_pair<true>(plan, map, out_map, extra_maps, prm, m_tiles, stream);
        else rc = dispatch_umma_dump(plan, ch.token_tile, map, extra_maps, prm, m_tiles, stream);
        if (rc == SK_OK) {
          const long long mn = M * plan->N;
          const int blocks = static_cast<int>(mn / 256 + 1 < sk::kChipSms * 8 ? mn / 256 + 1 : sk::kChipSms * 8);
          diff_partials_kernel<<<blocks, 256, 0, stream>>>(partials, prm.groups, mn, acc_bufs_of(ch.token_tile, ch.kernel));
          e = cudaGetLastError();
          if (e != cudaSuccess) rc = cuda_fail(plan, e);
        }
      }
      else if (ch.kernel == 5)
        rc = dispatch_stream(plan, ch.token_tile, map, prm, stream);
      else if (ch.kernel == 3)
        rc = ch.token_tile == 16 ? launch_decode<16, false>(plan, map, prm, m_tiles, ch.split_k, stream, ch.mix_split ? ch.ctas : 0)
                                 : launch_decode<32, false>(plan, map, prm, m_tiles, ch.split_k, stream, ch.mix_split ? ch.ctas : 0);
      else if (ch.kernel == 4) rc = launch_pair<false>(plan, map, out_map, extra_maps, prm, m_tiles, stream);
      else rc = dispatch_umma(plan, ch.token_tile, map, out_map, extra_maps, prm, m_tiles, ch.split_k, persist ? ch.ctas : 0, stream);
    }
  }
  if (cur != plan->device) (void)cudaSetDevice(cur);
  return rc;
}

// Whether sk_w2a8_linear on M tokens is one kernel that quantises its activations itself.
static bool linear_is_one_kernel(const sk_w2a8_plan* plan, long long M, DirectChoice* dc) {
  LaunchChoice ch;
  return M > 0 && resolve_launch(plan, M, false, &ch) == SK_OK && choose_direct(plan, M, dc) && direct_quantises(plan, M, *dc);
}
static size_t linear_scale_offset(long long M, long long K) { return (static_cast<size_t>(M) * K + 255) & ~static_cast<size_t>(255); }

static int repack_common(bool forward, const uint8_t* src, long long N, long long K, uint8_t* dst,
                         cudaStream_t stream) {
  if (!src || !dst) return SK_ERR_NULL_POINTER;
  if (N <= 0 || K <= 0 || (K % 32) != 0) return SK_ERR_BAD_SHAPE;
  const uint8_t* tiled = forward ? dst : src;
  if ((reinterpret_cast<uintptr_t>(tiled) & 15) != 0) return SK_ERR_BAD_ALIGNMENT;
  const int k_blocks = static_cast<int>((K + 127) / 128);
  const long long n_tiles = (N + 127) / 128;
  const long long total_words = n_tiles * k_blocks * 1024;
  const int threads = 256;
  const long long want = (total_words + threads - 1) / threads;
  const int blocks = static_cast<int>(want < sk::kChipSms * 16 ? want : sk::kChipSms * 16);
  if (forward)
    repack_kernel<<<blocks, threads, 0, stream>>>(src, reinterpret_cast<uint32_t*>(dst), N, K, k_blocks, total_words);
  else
    unrepack_kernel<<<blocks, threads, 0, stream>>>(reinterpret_cast<const uint32_t*>(src), dst, N, K, k_blocks,
                                                    total_words);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return SK_ERR_CUDA;
  return SK_OK;
}

}  // namespace sk

// ================================================================================================
// extern "C"
// ================================================================================================
static bool plan_shape_ok(int64_t N, int64_t K, int group_size) {
  if (N <= 0 || K <= 0 || N > (1LL << 30) || K > (1LL << 30)) return false;
  if (group_size <= 0 || (group_size % 32) != 0 || (K % group_size) != 0 || (K % 32) != 0) return false;
  return (group_size % 128) == 0 || (128 % group_size) == 0;
}

// Plan creation behind both entry points.  storage == nullptr: one cudaMalloc'ed block, the work on the legacy default
// stream, and the device synchronised before it returns.  Otherwise the caller's block, the work ordered on `stream`, and
// no synchronisation.
static int plan_create_common(sk_w2a8_plan** out, int device, int64_t N, int64_t K, int group_size, int zero_point,
                              const uint8_t* w, int w_layout, const void* w_scale_f16, int out_dtype, void* storage,
                              int64_t storage_bytes, cudaStream_t stream) {
  if (!out) return SK_ERR_NULL_POINTER;
  *out = nullptr;
  if (!w || !w_scale_f16) return SK_ERR_NULL_POINTER;
  if (!plan_shape_ok(N, K, group_size)) return SK_ERR_BAD_SHAPE;
  if (zero_point < 0 || zero_point > 3) return SK_ERR_BAD_ARGUMENT;
  if (out_dtype != SK_OUT_F16 && out_dtype != SK_OUT_BF16) return SK_ERR_BAD_ARGUMENT;
  if (w_layout != SK_WEIGHT_ROWMAJOR && w_layout != SK_WEIGHT_TILED) return SK_ERR_BAD_ARGUMENT;
  if ((reinterpret_cast<uintptr_t>(w_scale_f16) & 1) != 0) return SK_ERR_BAD_ALIGNMENT;
  if (w_layout == SK_WEIGHT_TILED && (reinterpret_cast<uintptr_t>(w) & 15) != 0) return SK_ERR_BAD_ALIGNMENT;

  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess) { (void)cudaGetLastError(); return SK_ERR_CUDA; }
  if (device < 0 || device >= ndev) return SK_ERR_BAD_ARGUMENT;
  int major = 0, sms = 0;
  if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
    (void)cudaGetLastError();
    return SK_ERR_CUDA;
  }
  if (major != 10) return SK_ERR_UNSUPPORTED_ARCH;

  sk_w2a8_plan* plan = new (std::nothrow) sk_w2a8_plan();
  if (!plan) return SK_ERR_OUT_OF_MEMORY;
  plan->device = device;
  plan->N = N; plan->K = K; plan->G = group_size; plan->zero_point = zero_point; plan->out_dtype = out_dtype;
  plan->k_blocks = static_cast<int>((K + 127) / 128);
  plan->n_tiles = static_cast<int>((N + 127) / 128);
  plan->sm_count = sms;
  plan->w_scale = static_cast<const __half*>(w_scale_f16);
  plan->external_storage = storage != nullptr;
  const sk::PlanLayout l = sk::plan_layout(plan, w_layout);
  if (storage && storage_bytes < l.total) { delete plan; return SK_ERR_BAD_SHAPE; }
  plan->maps.reserve(sk::kMapCache + 1);   // the tensor-map cache never grows past kMapCache entries: no host reallocation on the call path

  int cur = -1;
  cudaGetDevice(&cur);
  cudaError_t e = cur == device ? cudaSuccess : cudaSetDevice(device);
  char* base = static_cast<char*>(storage);
  if (e == cudaSuccess && !base) {
    void* block = nullptr;
    e = cudaMalloc(&block, static_cast<size_t>(l.total));
    base = e == cudaSuccess ? static_cast<char*>(block) : nullptr;
  }
  int rc = e == cudaSuccess ? SK_OK : sk::cuda_fail(plan, e);
  if (rc == SK_OK) {
    plan->status = reinterpret_cast<int*>(base + l.status);
    if (l.w_scale_tiled >= 0) plan->w_scale_tiled = reinterpret_cast<__half*>(base + l.w_scale_tiled);
    // kernel 3's copy of the scales is made once, here: later changes of w_scale_f16 are not seen by it
    bool scales_tiled = plan->w_scale_tiled == nullptr;
    if (w_layout == SK_WEIGHT_TILED) {
      plan->w_tiled = w;
    } else {
      plan->w_rowmajor = w;
      uint8_t* tiled = reinterpret_cast<uint8_t*>(base + l.w_tiled);
      plan->w_tiled = tiled;
      if (e == cudaSuccess) {
        if ((K % 128) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0 && ((K / 4) % 16) == 0 && plan->n_tiles <= 65535) {
          sk::tile_weight_kernel<<<dim3(plan->k_blocks, plan->n_tiles), 128, 0, stream>>>(
              w, tiled, plan->w_scale, plan->w_scale_tiled, N, K, plan->k_blocks);
          e = cudaGetLastError();
          scales_tiled = true;
        } else {
          rc = sk::repack_common(true, w, N, K, tiled, stream);
        }
      }
    }
    if (rc == SK_OK && e == cudaSuccess && !scales_tiled) {
      const long long total = static_cast<long long>(plan->n_tiles) * plan->k_blocks * sk::kTileN;
      const int blocks = static_cast<int>(total / 256 + 1 < sk::kChipSms * 8 ? total / 256 + 1 : sk::kChipSms * 8);
      sk::tile_scales_kernel<<<blocks, 256, 0, stream>>>(plan->w_scale, plan->w_scale_tiled, N, plan->k_blocks, total);
      e = cudaGetLastError();
    }
    // Last, and not only for its own sake: decode kernels are dependent launches that read the copies before they wait for the
    // kernel in front of them.  Were that a kernel above, they could start when its last CTA exits, before its stores are
    // sure to be visible; this operation starts only after those kernels are complete.
    if (rc == SK_OK && e == cudaSuccess) e = cudaMemsetAsync(plan->status, 0, sizeof(int), stream);
    if (rc == SK_OK && e == cudaSuccess && !storage) e = cudaDeviceSynchronize();
    if (rc == SK_OK && e != cudaSuccess) rc = sk::cuda_fail(plan, e);
  }
  if (cur >= 0 && cur != device) (void)cudaSetDevice(cur);
  if (rc != SK_OK) {
    if (!storage && base) cudaFree(base);
    delete plan;
    return rc;
  }
  *out = plan;
  return SK_OK;
}

extern "C" {

int sk_w2a8_version(void) { return 100; }

const char* sk_status_string(int status) {
  switch (status) {
    case SK_OK: return "ok";
    case SK_ERR_NULL_POINTER: return "null pointer";
    case SK_ERR_BAD_SHAPE: return "bad shape";
    case SK_ERR_BAD_ALIGNMENT: return "bad alignment";
    case SK_ERR_UNSUPPORTED_ARCH: return "unsupported architecture (needs compute capability 10.x)";
    case SK_ERR_CUDA: return "CUDA error";
    case SK_ERR_DEVICE_TIMEOUT: return "a bounded wait inside a kernel expired";
    case SK_ERR_BAD_ARGUMENT: return "bad argument";
    case SK_ERR_OUT_OF_MEMORY: return "out of device memory";
    case SK_ERR_UNAVAILABLE: return "not available for this plan";
    case SK_ERR_STATIC_SCRATCH_TOO_SMALL:
      return "problem needs more scratch than the library's fixed no-allocation buffer holds";
    default: return "unknown status";
  }
}

int64_t sk_w2a8_tiled_bytes(int64_t N, int64_t K) {
  if (N <= 0 || K <= 0) return 0;
  return ((N + 127) / 128) * ((K + 127) / 128) * 4096;
}

int sk_w2a8_repack(const uint8_t* w_packed, int64_t N, int64_t K, uint8_t* w_tiled, sk_stream_t stream) {
  return sk::repack_common(true, w_packed, N, K, w_tiled, static_cast<cudaStream_t>(stream));
}

int sk_w2a8_unrepack(const uint8_t* w_tiled, int64_t N, int64_t K, uint8_t* w_packed, sk_stream_t stream) {
  return sk::repack_common(false, w_tiled, N, K, w_packed, static_cast<cudaStream_t>(stream));
}

int sk_w2a8_plan_create(sk_w2a8_plan** out, int device, int64_t N, int64_t K, int group_size, int zero_point,
                        const uint8_t* w, int w_layout, const void* w_scale_f16, int out_dtype) {
  return plan_create_common(out, device, N, K, group_size, zero_point, w, w_layout, w_scale_f16, out_dtype, nullptr, 0, nullptr);
}

int64_t sk_w2a8_plan_storage_bytes(int device, int64_t N, int64_t K, int group_size, int w_layout) {
  if (!plan_shape_ok(N, K, group_size)) return 0;
  sk_w2a8_plan probe;
  if (cudaDeviceGetAttribute(&probe.sm_count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  probe.N = N; probe.K = K; probe.G = group_size;
  probe.k_blocks = static_cast<int>((K + 127) / 128);
  probe.n_tiles = static_cast<int>((N + 127) / 128);
  return sk::plan_layout(&probe, w_layout).total;
}

int sk_w2a8_plan_create_in(sk_w2a8_plan** out, int device, int64_t N, int64_t K, int group_size, int zero_point,
                           const uint8_t* w, int w_layout, const void* w_scale_f16, int out_dtype, void* storage,
                           int64_t storage_bytes, sk_stream_t stream) {
  if (out) *out = nullptr;
  if (!storage) return SK_ERR_NULL_POINTER;
  if (reinterpret_cast<uintptr_t>(storage) & 255) return SK_ERR_BAD_ALIGNMENT;
  return plan_create_common(out, device, N, K, group_size, zero_point, w, w_layout, w_scale_f16, out_dtype, storage, storage_bytes,
                            static_cast<cudaStream_t>(stream));
}

int sk_w2a8_plan_destroy(sk_w2a8_plan* plan) {
  if (!plan) return SK_ERR_NULL_POINTER;
  if (!plan->external_storage || plan->stream_scratch) {
    int cur = -1;
    cudaGetDevice(&cur);
    (void)cudaSetDevice(plan->device);
    if (plan->stream_scratch) {
      cudaFree(plan->stream_scratch);
      cudaFree(plan->stream_counters);
    }
    if (!plan->external_storage && plan->status) cudaFree(plan->status);   // the block holds all the other buffers
    if (cur >= 0 && cur != plan->device) (void)cudaSetDevice(cur);
  }
  delete plan;
  return SK_OK;
}

int sk_w2a8_plan_info(const sk_w2a8_plan* plan, int64_t* N, int64_t* K, int* group_size, int* zero_point,
                      int* out_dtype, int* device) {
  if (!plan) return SK_ERR_NULL_POINTER;
  if (N) *N = plan->N;
  if (K) *K = plan->K;
  if (group_size) *group_size = plan->G;
  if (zero_point) *zero_point = plan->zero_point;
  if (out_dtype) *out_dtype = plan->out_dtype;
  if (device) *device = plan->device;
  return SK_OK;
}

int sk_w2a8_set_option(sk_w2a8_plan* plan, int key, int64_t value) {
  if (!plan) return SK_ERR_NULL_POINTER;
  switch (key) {
    case SK_OPT_KERNEL:
      if (value < 0 || value > 6) return SK_ERR_BAD_ARGUMENT;
      if (value == 2 && !plan->w_rowmajor) return SK_ERR_UNAVAILABLE;
      if (value == 5 && !plan->stream_scratch) {   // first request
        int cur = -1;
        cudaGetDevice(&cur);
        (void)cudaSetDevice(plan->device);
        const int rc = sk::stream_setup(plan, 0);
        if (cur >= 0 && cur != plan->device) (void)cudaSetDevice(cur);
        if (rc != SK_OK) return rc;
        if (!plan->stream_scratch) return SK_ERR_UNAVAILABLE;   // group size != 128 or K % 256 != 0
      }
      if (value == 4 && plan->G != 128) return SK_ERR_UNAVAILABLE;
      if (value == 3 && plan->G != 128) return SK_ERR_UNAVAILABLE;
      plan->opt_kernel = static_cast<int>(value);
      return SK_OK;
    case SK_OPT_TOKEN_TILE:
      if (value != 0 && value != 16 && value != 32 && value != 64 && value != 128 && value != 192 && value != 256)
        return SK_ERR_BAD_ARGUMENT;
      if (value == 16) sk::stream_wanted(plan);
      plan->opt_token_tile = static_cast<int>(value);
      return SK_OK;
    case SK_OPT_SPLIT_K:
      if (value != 0 && value != 1 && value != 2 && value != 4 && value != 8) return SK_ERR_BAD_ARGUMENT;
      if (value == 1) sk::stream_wanted(plan);
      plan->opt_split_k = static_cast<int>(value);
      return SK_OK;
    case SK_OPT_DEPENDENT_LAUNCH:
      if (value < 0 || value > 2) return SK_ERR_BAD_ARGUMENT;
      plan->opt_pdl = static_cast<int>(value);
      return SK_OK;
    case SK_OPT_TMA_STORE:
      if (value < 0 || value > 2) return SK_ERR_BAD_ARGUMENT;
      plan->opt_tma_store = static_cast<int>(value);
      return SK_OK;
    case SK_OPT_PERSISTENT:
      if (value < 0 || value > 2) return SK_ERR_BAD_ARGUMENT;
      if (value != 0) sk::stream_wanted(plan);
      plan->opt_persistent = static_cast<int>(value);
      return SK_OK;
    case SK_OPT_WAIT_LIMIT_CYCLES:
      if (value < 0 || (value != 0 && value < 1000)) return SK_ERR_BAD_ARGUMENT;
      plan->opt_wait_limit = value;
      return SK_OK;
    case SK_OPT_STREAM_CTAS: {
      if (value < 0 || value > 65535) return SK_ERR_BAD_ARGUMENT;
      if (plan->G != 128 || (plan->K % 256) != 0) return SK_ERR_UNAVAILABLE;
      int cur = -1;
      cudaGetDevice(&cur);
      (void)cudaSetDevice(plan->device);
      const int rc = sk::stream_setup(plan, static_cast<int>(value));   // frees and allocates: orders itself after the plan's launches
      if (cur >= 0 && cur != plan->device) (void)cudaSetDevice(cur);
      return rc;
    }
    case SK_OPT_TEST_SKIP_COPY:
      if (value < 0 || value > (1 << 20)) return SK_ERR_BAD_ARGUMENT;
      if (value != 0) sk::stream_wanted(plan);
      plan->opt_skip_copy = static_cast<int>(value);
      return SK_OK;
    default: return SK_ERR_BAD_ARGUMENT;
  }
}

int sk_w2a8_gemm(sk_w2a8_plan* plan, int64_t M, const int8_t* x_q, int64_t ld_x, const float* x_scale, void* out,
                 int64_t ld_out, sk_stream_t stream) {
  return sk::run_gemm(plan, M, x_q, ld_x, x_scale, out, ld_out, nullptr, static_cast<cudaStream_t>(stream));
}

int64_t sk_w2a8_linear_workspace_bytes(const sk_w2a8_plan* plan, int64_t M) {
  if (!plan || M <= 0) return 0;
  sk::DirectChoice dc;
  if (sk::linear_is_one_kernel(plan, M, &dc)) return 0;
  return static_cast<int64_t>(sk::linear_scale_offset(M, plan->K)) + 4 * M;
}

int sk_w2a8_linear(sk_w2a8_plan* plan, int64_t M, const void* x, int x_bf16, int64_t ld_x, void* out, int64_t ld_out,
                   void* workspace, int64_t workspace_bytes, sk_stream_t stream) {
  if (!plan || !x || !out) return SK_ERR_NULL_POINTER;
  if (M <= 0 || M > 0x7fffffffLL / 2 || ld_x < plan->K || ld_out < plan->N) return SK_ERR_BAD_SHAPE;
  if ((reinterpret_cast<uintptr_t>(x) & 15) || (ld_x % 8) || (reinterpret_cast<uintptr_t>(out) & 1)) return SK_ERR_BAD_ALIGNMENT;
  int cur = -1;
  cudaError_t e = cudaGetDevice(&cur);
  if (e == cudaSuccess && cur != plan->device) e = cudaSetDevice(plan->device);
  if (e != cudaSuccess) return sk::cuda_fail(plan, e);
  int rc;
  sk::DirectChoice dc;
  if (sk::linear_is_one_kernel(plan, M, &dc)) {
    sk::DirectParams prm = sk::direct_params(plan, M, out, ld_out);
    prm.x_float = static_cast<const uint16_t*>(x);
    prm.ld_float = ld_x;
    prm.float_bf16 = x_bf16;
    rc = sk::dispatch_direct_quant(plan, dc, prm, static_cast<cudaStream_t>(stream));
  } else if (!workspace) {
    rc = SK_ERR_NULL_POINTER;
  } else if (workspace_bytes < static_cast<int64_t>(sk::linear_scale_offset(M, plan->K)) + 4 * M) {
    rc = SK_ERR_BAD_SHAPE;
  } else {
    int8_t* x_q = static_cast<int8_t*>(workspace);
    float* x_scale = reinterpret_cast<float*>(x_q + sk::linear_scale_offset(M, plan->K));
    rc = sk_quantize_activation_int8_from(x, x_bf16, ld_x, M, plan->K, x_q, plan->K, x_scale, stream);
    if (rc == SK_OK) rc = sk::run_gemm(plan, M, x_q, plan->K, x_scale, out, ld_out, nullptr, static_cast<cudaStream_t>(stream));
  }
  if (cur != plan->device) (void)cudaSetDevice(cur);
  return rc;
}

int sk_w2a8_gemm_scatter(sk_w2a8_plan* plan, int64_t M, const int8_t* x_q, int64_t ld_x, const float* x_scale,
                         void* const* outs, int n_outs, int64_t ld_out, int64_t col_offset, sk_stream_t stream) {
  if (!outs) return SK_ERR_NULL_POINTER;
  if (n_outs < 1 || n_outs > 8) return SK_ERR_BAD_ARGUMENT;
  if (!plan) return SK_ERR_NULL_POINTER;
  if (col_offset < 0 || col_offset + plan->N > ld_out) return SK_ERR_BAD_SHAPE;
  const size_t esz = 2;   // half and bfloat16
  void* shifted[8];
  for (int i = 0; i < n_outs; ++i) {
    if (!outs[i]) return SK_ERR_NULL_POINTER;
    shifted[i] = static_cast<char*>(outs[i]) + static_cast<size_t>(col_offset) * esz;
  }
  return sk::run_gemm(plan, M, x_q, ld_x, x_scale, shifted[0], ld_out, nullptr, static_cast<cudaStream_t>(stream),
                      shifted + 1, n_outs - 1);
}

int sk_w2a8_gemm_rowscatter(sk_w2a8_plan* plan, int64_t M, const int8_t* x_q, int64_t ld_x, const float* x_scale,
                            void* const* outs, int n_outs, int64_t rows_per_dest, int64_t dst_row0, int64_t ld_out,
                            sk_stream_t stream) {
  if (!outs) return SK_ERR_NULL_POINTER;
  if (n_outs < 1 || n_outs > 8) return SK_ERR_BAD_ARGUMENT;
  if (!plan) return SK_ERR_NULL_POINTER;
  if (rows_per_dest <= 0 || dst_row0 < 0 || M != rows_per_dest * n_outs) return SK_ERR_BAD_SHAPE;
  if (dst_row0 + rows_per_dest > 0x7fffffffLL) return SK_ERR_BAD_SHAPE;
  for (int i = 0; i < n_outs; ++i)
    if (!outs[i]) return SK_ERR_NULL_POINTER;
  return sk::run_gemm(plan, M, x_q, ld_x, x_scale, outs[0], ld_out, nullptr, static_cast<cudaStream_t>(stream),
                      outs + 1, n_outs - 1, rows_per_dest, dst_row0);
}

int sk_w2a8_gemm_debug_partials(sk_w2a8_plan* plan, int64_t M, const int8_t* x_q, int64_t ld_x, int32_t* partials,
                                sk_stream_t stream) {
  if (!partials) return SK_ERR_NULL_POINTER;
  return sk::run_gemm(plan, M, x_q, ld_x, nullptr, nullptr, 0, partials, static_cast<cudaStream_t>(stream));
}

int sk_w2a8_last_device_status(sk_w2a8_plan* plan, int* device_status) {
  if (!plan || !device_status) return SK_ERR_NULL_POINTER;
  int cur = -1;
  cudaGetDevice(&cur);
  (void)cudaSetDevice(plan->device);
  int v = 0;
  cudaError_t e = cudaMemcpy(&v, plan->status, sizeof(int), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && v != 0) e = cudaMemset(plan->status, 0, sizeof(int));
  // a launch that gave up may have left tiles of the balanced-split kernel half counted
  if (e == cudaSuccess && v != 0 && plan->stream_counters)
    e = cudaMemset(plan->stream_counters, 0, static_cast<size_t>(plan->n_tiles) * sk::StreamTraits<32>::kEpiWarps * sizeof(int));
  if (cur >= 0 && cur != plan->device) (void)cudaSetDevice(cur);
  if (e != cudaSuccess) return sk::cuda_fail(plan, e);
  *device_status = v;
  return v == 0 ? SK_OK : SK_ERR_DEVICE_TIMEOUT;
}

int sk_w2a8_last_cuda_error(const sk_w2a8_plan* plan) { return plan ? plan->last_cuda_error : 0; }

int sk_w2a8_launch_floor_probe(sk_w2a8_plan* plan, int64_t M, sk_stream_t stream) {
  if (!plan) return SK_ERR_NULL_POINTER;
  if (M <= 0) return SK_ERR_BAD_SHAPE;
  sk::LaunchChoice ch;
  int rc = sk::resolve_launch(plan, M, false, &ch);
  if (rc != SK_OK) return rc;
  if (ch.kernel != 3 && ch.kernel != 5) return SK_ERR_UNAVAILABLE;   // decode-sized calls only
  int cur = -1;
  if (cudaGetDevice(&cur) != cudaSuccess) return sk::cuda_fail(plan, cudaGetLastError());
  if (cur != plan->device && cudaSetDevice(plan->device) != cudaSuccess) return sk::cuda_fail(plan, cudaGetLastError());
  sk::DirectChoice dc;
  if (sk::choose_direct(plan, M, &dc)) {
    sk::DirectParams prm = sk::direct_params(plan, M, nullptr, 0);
    prm.floor_probe = 1;
    rc = sk::dispatch_direct(plan, dc, prm, static_cast<cudaStream_t>(stream));
    if (cur != plan->device) (void)cudaSetDevice(cur);
    return rc;
  }
  const int dyn = ch.token_tile == 16 ? sk::DecodeTraits<16>::kDynamicBytes : sk::DecodeTraits<32>::kDynamicBytes;
  static int configured[64] = {0};
  cudaError_t e = cudaSuccess;
  if (plan->device < 64 && !configured[plan->device]) {
    e = cudaFuncSetAttribute(sk::launch_floor_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 110 * 1024);
    configured[plan->device] = 1;
  }
  if (e == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    const int m_tiles = static_cast<int>((M + ch.token_tile - 1) / ch.token_tile);
    cfg.gridDim = ch.kernel == 5 ? dim3(ch.ctas, 1, 1)
                  : ch.mix_split ? dim3(ch.ctas, 1, 1) : dim3(plan->n_tiles, m_tiles, ch.split_k);
    cfg.blockDim = dim3(sk::DecodeTraits<16>::kThreads, 1, 1);
    cfg.dynamicSmemBytes = dyn - 1024;
    cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (ch.kernel == 3 && ch.mix_split) {
      attr[na].id = cudaLaunchAttributeClusterDimension;
      attr[na].val.clusterDim.x = 4;
      attr[na].val.clusterDim.y = 1;
      attr[na].val.clusterDim.z = 1;
      ++na;
    } else if (ch.kernel == 3 && ch.split_k > 1) {
      attr[na].id = cudaLaunchAttributeClusterDimension;
      attr[na].val.clusterDim.x = 1;
      attr[na].val.clusterDim.y = 1;
      attr[na].val.clusterDim.z = ch.split_k;
      ++na;
    }
    if (plan->opt_pdl != 1) {
      attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[na].val.programmaticStreamSerializationAllowed = 1;
      ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    e = cudaLaunchKernelEx(&cfg, sk::launch_floor_kernel, static_cast<int*>(nullptr));
  }
  if (cur != plan->device) (void)cudaSetDevice(cur);
  return e == cudaSuccess ? SK_OK : sk::cuda_fail(plan, e);
}

const char* sk_device_status_string(int device_status) {
  switch (device_status) {
    case 0: return "no wait expired";
    case sk::kStProducerEmpty: return "producer: a pipeline stage was never released by the MMAs that read it";
    case sk::kStExpanderFull: return "expander: the copies of a pipeline stage never landed";
    case sk::kStExpanderEmpty: return "expander: a buffer of expanded weights was never released by the MMAs that read it";
    case sk::kStMmaLdFull: return "MMA issuer: the copies of a pipeline stage never landed";
    case sk::kStMmaExFull: return "MMA issuer: the expanded weights of a stage never arrived";
    case sk::kStMmaAccEmpty: return "MMA issuer: an accumulator buffer was never released by the epilogue";
    case sk::kStEpilogueAccFull: return "epilogue: the MMAs of a scale group never completed";
    case sk::kStEpilogueScales: return "epilogue: the copy of the group scales never landed";
    case sk::kStDrain: return "producer: a copy in flight did not land while the CTA was giving up";
    case sk::kStStreamSlots: return "epilogue: a tile is shared by more CTAs than the scratch buffer has slots for";
    default: return "unknown device status";
  }
}

int sk_w2a8_query_route(sk_w2a8_plan* plan, int64_t M, int* token_tile, int* split_k, int* ctas, int* kernel_kind) {
  const int rc = sk_w2a8_query_launch(plan, M, token_tile, split_k, ctas, kernel_kind);
  if (rc != SK_OK) return rc;
  sk::DirectChoice d;
  if (!sk::choose_direct(plan, M, &d)) {
    sk::LaunchChoice c;
    (void)sk::resolve_launch(plan, M, false, &c);
    sk::refine_launch(plan, M, &c);
    if (token_tile) *token_tile = c.token_tile;
    if (split_k) *split_k = c.split_k;
    if (ctas) *ctas = c.ctas;
    return SK_OK;
  }
  if (token_tile) *token_tile = 8 * d.nt;
  if (split_k) *split_k = d.split;
  if (ctas) *ctas = d.ctas;
  if (kernel_kind) *kernel_kind = 6;
  return SK_OK;
}

int sk_w2a8_query_launch(sk_w2a8_plan* plan, int64_t M, int* token_tile, int* split_k, int* ctas, int* kernel_kind) {
  if (!plan) return SK_ERR_NULL_POINTER;
  if (M <= 0) return SK_ERR_BAD_SHAPE;
  sk::LaunchChoice c;
  const int rc = sk::resolve_launch(plan, M, false, &c);
  if (rc != SK_OK) return rc;
  if (token_tile) *token_tile = c.token_tile;
  if (split_k) *split_k = c.split_k;
  if (ctas) *ctas = c.ctas;
  if (kernel_kind) *kernel_kind = c.kernel;
  return SK_OK;
}

// ---------------------------------------------------------------------------------------------- activation side
int sk_w2a8_quantize_weight(const float* w, int64_t ld_w, int64_t K, int64_t N, int group_size, uint8_t* w_packed,
                            float* scale_f32, void* scale_f16, sk_stream_t stream) {
  if (!w || !w_packed || (!scale_f32 && !scale_f16)) return SK_ERR_NULL_POINTER;
  if (K <= 0 || N <= 0 || group_size <= 0 || (group_size % 4) != 0 || (K % group_size) != 0 || ld_w < N ||
      K > (1LL << 30) || N > (1LL << 30) || K / group_size > 65535)
    return SK_ERR_BAD_SHAPE;
  if ((reinterpret_cast<uintptr_t>(w) & 3) || (scale_f16 && (reinterpret_cast<uintptr_t>(scale_f16) & 1)) ||
      (scale_f32 && (reinterpret_cast<uintptr_t>(scale_f32) & 3)))
    return SK_ERR_BAD_ALIGNMENT;
  const dim3 grid(static_cast<unsigned>((N + sk::kPrepThreads - 1) / sk::kPrepThreads), static_cast<unsigned>(K / group_size));
  constexpr int kPrepSmem = sk::kPrepSlab * sk::kPrepThreads * 4;     // 64 KiB
  static int prep_configured[64] = {0};
  int prep_dev = 0;
  if (cudaGetDevice(&prep_dev) != cudaSuccess) return SK_ERR_CUDA;
  if (prep_dev >= 0 && prep_dev < 64 && !prep_configured[prep_dev]) {
    if (cudaFuncSetAttribute(sk::quantize_pack_weight_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPrepSmem) != cudaSuccess) {
      (void)cudaGetLastError();
      return SK_ERR_CUDA;
    }
    prep_configured[prep_dev] = 1;
  }
  sk::quantize_pack_weight_kernel<<<grid, sk::kPrepCtaThreads, kPrepSmem, static_cast<cudaStream_t>(stream)>>>(
      w, ld_w, static_cast<int>(K), static_cast<int>(N), group_size, w_packed, scale_f32, static_cast<__half*>(scale_f16));
  if (cudaGetLastError() != cudaSuccess) return SK_ERR_CUDA;
  return SK_OK;
}

int sk_w2a8_quantize_weight_rows(const void* w, int w_type, int64_t ld_w, int64_t N, int64_t K, int group_size,
                                 uint8_t* w_packed, void* scale_f16, sk_stream_t stream) {
  if (!w || !w_packed || !scale_f16) return SK_ERR_NULL_POINTER;
  if (w_type != sk::kRowsF16 && w_type != sk::kRowsBf16 && w_type != sk::kRowsF32) return SK_ERR_BAD_ARGUMENT;
  if (K <= 0 || N <= 0 || group_size <= 0 || (group_size % 4) != 0 || (K % group_size) != 0 || ld_w < K ||
      K > (1LL << 30) || N > (1LL << 30))
    return SK_ERR_BAD_SHAPE;
  if (reinterpret_cast<uintptr_t>(scale_f16) & 1) return SK_ERR_BAD_ALIGNMENT;
  const int elem = w_type == sk::kRowsF32 ? 4 : 2;
  const int64_t row_ctas = (N + sk::kRowsPerCta - 1) / sk::kRowsPerCta;
  if (group_size < 16 || group_size > sk::kRowsChunk || (group_size & (group_size - 1)) != 0 || row_ctas > 65535 ||
      (reinterpret_cast<uintptr_t>(w) & 15) || ((ld_w * elem) % 16) != 0 || (reinterpret_cast<uintptr_t>(w_packed) & 3))
    return SK_ERR_UNAVAILABLE;
  const dim3 grid(static_cast<unsigned>((K + sk::kRowsChunk - 1) / sk::kRowsChunk), static_cast<unsigned>(row_ctas));
  auto* s16 = static_cast<__half*>(scale_f16);
  const auto st = static_cast<cudaStream_t>(stream);
  const int k = static_cast<int>(K), n = static_cast<int>(N);
  constexpr int threads = 32 * sk::kRowsWarps;
  if (w_type == sk::kRowsF16) sk::quantize_pack_rows_kernel<sk::kRowsF16><<<grid, threads, 0, st>>>(w, ld_w, k, n, group_size, w_packed, s16);
  else if (w_type == sk::kRowsBf16) sk::quantize_pack_rows_kernel<sk::kRowsBf16><<<grid, threads, 0, st>>>(w, ld_w, k, n, group_size, w_packed, s16);
  else sk::quantize_pack_rows_kernel<sk::kRowsF32><<<grid, threads, 0, st>>>(w, ld_w, k, n, group_size, w_packed, s16);
  if (cudaGetLastError() != cudaSuccess) return SK_ERR_CUDA;
  return SK_OK;
}

int sk_quantize_activation_int8(const void* x_f16, int64_t ld_x, int64_t M, int64_t K, int8_t* x_q, int64_t ld_q,
                                float* x_scale, sk_stream_t stream) {
  return sk_quantize_activation_int8_from(x_f16, 0, ld_x, M, K, x_q, ld_q, x_scale, stream);
}

int sk_quantize_activation_int8_from(const void* x, int x_bf16, int64_t ld_x, int64_t M, int64_t K, int8_t* x_q, int64_t ld_q,
                                     float* x_scale, sk_stream_t stream) {
  if (!x || !x_q || !x_scale) return SK_ERR_NULL_POINTER;
  if (M <= 0 || K <= 0 || (K % 8) != 0 || ld_x < K || ld_q < K || M > 0x7fffffffLL) return SK_ERR_BAD_SHAPE;
  if ((reinterpret_cast<uintptr_t>(x) & 15) || (ld_x % 8) || (reinterpret_cast<uintptr_t>(x_q) & 7) || (ld_q % 8))
    return SK_ERR_BAD_ALIGNMENT;
  // launched as a programmatic dependent launch: the kernel waits for its inputs itself (griddepcontrol.wait) and
  // lets the kernel behind it start its set-up early
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(M));
  cfg.blockDim = dim3(sk::kActThreads, 1, 1);
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const uint16_t* src = static_cast<const uint16_t*>(x);
  const long long ldx = ld_x, ldq = ld_q;
  const int k = static_cast<int>(K);
  const int vecs = K <= 8 * sk::kActThreads * 2 ? 2 : K <= 8 * sk::kActThreads * 4 ? 4 : 8;
  auto kern = x_bf16 ? (vecs == 2 ? sk::quantize_activation_kernel<2, true> : vecs == 4 ? sk::quantize_activation_kernel<4, true>
                                                                                        : sk::quantize_activation_kernel<8, true>)
                     : (vecs == 2 ? sk::quantize_activation_kernel<2, false> : vecs == 4 ? sk::quantize_activation_kernel<4, false>
                                                                                         : sk::quantize_activation_kernel<8, false>);
  if (M <= 2 * sk::kChipSms && K > 8 * sk::kActThreads) {      // few rows: more threads per row
    const bool half = K <= 8 * 512;
    cfg.blockDim = dim3(half ? 512 : 1024, 1, 1);
    kern = x_bf16 ? (half ? sk::quantize_activation_kernel<1, true, 512> : sk::quantize_activation_kernel<2, true, 1024>)
                  : (half ? sk::quantize_activation_kernel<1, false, 512> : sk::quantize_activation_kernel<2, false, 1024>);
  }
  const cudaError_t le = cudaLaunchKernelEx(&cfg, kern, src, ldx, x_q, ldq, x_scale, k);
  if (le != cudaSuccess) { (void)cudaGetLastError(); return SK_ERR_CUDA; }
  if (cudaGetLastError() != cudaSuccess) return SK_ERR_CUDA;
  return SK_OK;
}

int sk_silu_mul_quantize_int8(const void* gate_up_f16, int64_t ld_gu, int64_t M, int64_t I, int8_t* h_q, int64_t ld_q,
                              float* h_scale, sk_stream_t stream) {
  if (!gate_up_f16 || !h_q || !h_scale) return SK_ERR_NULL_POINTER;
  if (M <= 0 || I <= 0 || (I % 8) != 0 || ld_gu < 2 * I || ld_q < I || M > 0x7fffffffLL || I > 0x7fffffffLL)
    return SK_ERR_BAD_SHAPE;
  if ((reinterpret_cast<uintptr_t>(gate_up_f16) & 15) || (ld_gu % 8) || (reinterpret_cast<uintptr_t>(h_q) & 7) || (ld_q % 8))
    return SK_ERR_BAD_ALIGNMENT;
  const auto st = static_cast<cudaStream_t>(stream);
  const __half* gu = static_cast<const __half*>(gate_up_f16);
  // Many rows: CTAs that stay and take a row each at a time.  A row is one CTA's work here and up to eight CTAs' in the cluster kernel
  // below.  Where which is the faster one, in us by which an MLP block of 512 to 8192 hidden features gets shorter with resident CTAs
  // (a range: with the hidden size):
  //   * from 64 rows on: 64 x 14336 .3 to 1.0, 64 x 8320 1.6 to 2.0, 128 x 8320 1.7 to 2.0, 444 x 5504 1.4 to 1.7, 1024 x 6144 1.0 to 1.9, 2048 x
  //     11008 8, 4096 x 11008 19.  Under 64 rows it is nothing or less (48 x 13312 -.2 to -.8).  Single sizes lose a little still (88 x
  //     13824 -.3 to -.9, 128 x 12288 up to -.6, 960 x 4224 -.2 to -.6, with 8192 hidden features -2.4);
  //   * up to 2048 features, where half the threads or more have nothing, with more than 384 Ki values: 192 x 2048 -.6, 208 x 2048 up to .7,
  //     256 x 1536 -.4 to -.8, 272 x 1536 .2 to .7, 256 x 1024 -.9 to .3, 416 x 1024 .2 to .5, 592 x 512 .1;
  //   * up to 4096 features, where a cluster is one CTA too, only while every row has a CTA of its own: 592 x 3072 .5 to 1.1, 640 x 3072 -1.3 to
  //     -1.9, 4096 x 4096 -2.8;
  //   * with two vectors a wave holds 444 resident CTAs or 592 clusters of two.  Between and somewhat above the cluster is the better one:
  //     up to 4608 features for 445 to 600 rows (480 x 4224 -.5 to -1.3, 576 x 4480 -.4 to -2.9, 640 x 4224 -.6 to 1.5), up to 6144 for 513 to 768
  //     (512 x 5504 .7 to 1.0, 520 x 5504 -.7 to -4.2, 720 x 5504 .2 to -1.9, 832 x 5504 1.2 to 2.2), above 7168 for 481 to 512 (512 x 8192 -.3 to -2.2,
  //     520 x 8192 1.0; 512 x 7168 .7 to -1.1).
  const int vecs = static_cast<int>(I <= 8LL * sk::kRowsThreads * 4 ? (I / 8 + sk::kRowsThreads - 1) / sk::kRowsThreads : 5);
  bool resident = vecs <= 4 && M >= 64;
  if (vecs == 1) resident = resident && M <= 4 * sk::kChipSms && (I > 2048 || M * I > (384 << 10));
  if (vecs == 2)
    resident = resident && !(I <= 4608   ? M > 3 * sk::kChipSms && M <= 600
                             : I <= 6144 ? M > 512 && M <= 768
                                         : I > 7168 && M > 480 && M <= 512);
  if (resident) {
    auto kern = vecs == 1   ? sk::silu_mul_quantize_rows_kernel<1>
                : vecs == 2 ? sk::silu_mul_quantize_rows_kernel<2>
                : vecs == 3 ? sk::silu_mul_quantize_rows_kernel<3>
                            : sk::silu_mul_quantize_rows_kernel<4>;
    const int smem = static_cast<int>(I) * 4, grid = sk::kChipSms * sk::rows_ctas_per_sm(vecs);
    if (vecs >= 3) {                      // more than 48 KB of shared memory with the longest rows
      // Always the most that the instantiation takes: the attribute belongs to the kernel, so a size of this call's own would be
      // taken from under another thread's launch with longer rows.
      static std::atomic<int> configured[2][64];
      int dev = 0;
      if (cudaGetDevice(&dev) != cudaSuccess) return SK_ERR_CUDA;
      const bool known = dev >= 0 && dev < 64;
      if (!known || !configured[vecs - 3][dev].load(std::memory_order_acquire)) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, vecs * sk::kRowsThreads * 8 * 4) != cudaSuccess) {
          (void)cudaGetLastError();
          return SK_ERR_CUDA;
        }
        if (known) configured[vecs - 3][dev].store(1, std::memory_order_release);
      }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(M < grid ? M : grid));
    cfg.blockDim = dim3(sk::kRowsThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // see sk_quantize_activation_int8
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, kern, gu, static_cast<long long>(ld_gu), h_q, static_cast<long long>(ld_q), h_scale,
                           static_cast<long long>(M), static_cast<int>(I)) != cudaSuccess) {
      (void)cudaGetLastError();
      return SK_ERR_CUDA;
    }
    return SK_OK;
  }
  // one pass over HBM: the row split over a cluster of 1..8 CTAs whose threads keep their fp32 values in registers
  // As many CTAs as the row needs, whether or not that is a power of two: 11008 features are 3 x 1.8 vectors per thread, in
  // four CTAs a third of the second vectors' threads would idle (12 us of 697 of the MLP block of 4096 tokens).  Few rows leave SMs
  // idle instead: then up to eight CTAs, one vector per thread.
  const long long per_cta = 8LL * sk::kActThreads * sk::kClusterVecs;
  int csize = static_cast<int>(I / per_cta < 8 ? (I + per_cta - 1) / per_cta : 9);
  if (csize <= 8 && M * 8 <= sk::kChipSms) csize = static_cast<int>((I + 8LL * sk::kActThreads - 1) / (8LL * sk::kActThreads));
  if (csize > 8) csize = 8;
  if (I <= per_cta * csize) {
    for (int64_t m0 = 0; m0 < M; m0 += 65535) {       // gridDim.y holds at most 65535 rows per launch
      const int64_t rows = M - m0 < 65535 ? M - m0 : 65535;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(static_cast<unsigned>(csize), static_cast<unsigned>(rows), 1);
      cfg.blockDim = dim3(sk::kActThreads, 1, 1);
      cfg.stream = st;
      cudaLaunchAttribute attr[2];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = static_cast<unsigned>(csize);
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // see sk_quantize_activation_int8
      attr[1].val.programmaticStreamSerializationAllowed = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 2;
      if (cudaLaunchKernelEx(&cfg, sk::silu_mul_quantize_cluster_kernel, gu + m0 * ld_gu, static_cast<long long>(ld_gu),
                             h_q + m0 * ld_q, static_cast<long long>(ld_q), h_scale + m0, static_cast<int>(I)) != cudaSuccess) {
        (void)cudaGetLastError();
        return SK_ERR_CUDA;
      }
    }
    return SK_OK;
  }
  // longer rows still: read twice and recompute (same values), full occupancy
  sk::silu_mul_quantize_twopass_kernel<<<static_cast<unsigned>(M), sk::kActThreads, 0, st>>>(
      gu, ld_gu, h_q, ld_q, h_scale, static_cast<int>(I));
  if (cudaGetLastError() != cudaSuccess) return SK_ERR_CUDA;
  return SK_OK;
}

// workspace layout of the MLP block (all offsets 256-byte aligned)
namespace {
struct MlpLayout {
  size_t x_q, x_scale, gate_up, h_q, h_scale, total;
};
inline size_t up256(size_t v) { return (v + 255) & ~static_cast<size_t>(255); }
inline MlpLayout mlp_layout(int64_t M, int64_t hidden, int64_t inter) {
  MlpLayout l;
  size_t o = 0;
  l.x_q = o;     o = up256(o + static_cast<size_t>(M) * hidden);
  l.x_scale = o; o = up256(o + static_cast<size_t>(M) * 4);
  l.gate_up = o; o = up256(o + static_cast<size_t>(M) * 2 * inter * 2);
  l.h_q = o;     o = up256(o + static_cast<size_t>(M) * inter);
  l.h_scale = o; o = up256(o + static_cast<size_t>(M) * 4);
  l.total = o;
  return l;
}
// The caller has made the plans' device current: the two side kernels launch on the current device.
int mlp_run(sk_w2a8_plan* gu, sk_w2a8_plan* down, int64_t M, const void* x, int x_bf16, int64_t ld_x, void* out, int64_t ld_out,
            char* ws, sk_stream_t stream) {
  const int64_t hidden = gu->K, inter = down->K;
  const MlpLayout l = mlp_layout(M, hidden, inter);
  void* gate_up = ws + l.gate_up;
  int8_t* h_q = reinterpret_cast<int8_t*>(ws + l.h_q);
  float* h_scale = reinterpret_cast<float*>(ws + l.h_scale);
  // (int8 activations and their scales lie next to each other at the start of the workspace)
  int rc = sk_w2a8_linear(gu, M, x, x_bf16, ld_x, gate_up, 2 * inter, ws + l.x_q, static_cast<int64_t>(l.gate_up - l.x_q), stream);
  if (rc == SK_OK) rc = sk_silu_mul_quantize_int8(gate_up, 2 * inter, M, inter, h_q, inter, h_scale, stream);
  if (rc == SK_OK) rc = sk_w2a8_gemm(down, M, h_q, inter, h_scale, out, ld_out, stream);
  return rc;
}
int mlp_check(const sk_w2a8_plan* gu, const sk_w2a8_plan* down, int64_t M) {
  if (!gu || !down) return SK_ERR_NULL_POINTER;
  if (M <= 0) return SK_ERR_BAD_SHAPE;
  if (gu->N != 2 * down->K || down->N != gu->K || gu->device != down->device) return SK_ERR_BAD_SHAPE;
  if (gu->out_dtype != SK_OUT_F16) return SK_ERR_BAD_ARGUMENT;   // the SiLU kernel reads fp16
  if ((gu->K % 16) != 0 || (down->K % 16) != 0) return SK_ERR_BAD_SHAPE;
  return SK_OK;
}
}  // namespace

int64_t sk_w2a8_mlp_workspace_bytes(const sk_w2a8_plan* gate_up, const sk_w2a8_plan* down, int64_t M) {
  if (mlp_check(gate_up, down, M) != SK_OK) return 0;
  return static_cast<int64_t>(mlp_layout(M, gate_up->K, down->K).total);
}

int sk_w2a8_mlp_forward(sk_w2a8_plan* gate_up, sk_w2a8_plan* down, int64_t M, const void* x_f16, int64_t ld_x,
                        void* out, int64_t ld_out, void* workspace, int64_t workspace_bytes, sk_stream_t stream) {
  return sk_w2a8_mlp_forward_from(gate_up, down, M, x_f16, 0, ld_x, out, ld_out, workspace, workspace_bytes, stream);
}

int sk_w2a8_mlp_forward_from(sk_w2a8_plan* gate_up, sk_w2a8_plan* down, int64_t M, const void* x, int x_bf16, int64_t ld_x,
                             void* out, int64_t ld_out, void* workspace, int64_t workspace_bytes, sk_stream_t stream) {
  int rc = mlp_check(gate_up, down, M);
  if (rc != SK_OK) return rc;
  if (!x || !out || !workspace) return SK_ERR_NULL_POINTER;
  if (reinterpret_cast<uintptr_t>(workspace) & 255) return SK_ERR_BAD_ALIGNMENT;
  if (workspace_bytes < static_cast<int64_t>(mlp_layout(M, gate_up->K, down->K).total)) return SK_ERR_BAD_SHAPE;
  // a plan is bound to one device: run there whatever device the calling thread has current, and put that back
  const int dev = gate_up->device;
  int cur = -1;
  if (cudaGetDevice(&cur) != cudaSuccess) return sk::cuda_fail(gate_up, cudaGetLastError());
  if (cur != dev && cudaSetDevice(dev) != cudaSuccess) return sk::cuda_fail(gate_up, cudaGetLastError());
  rc = mlp_run(gate_up, down, M, x, x_bf16, ld_x, out, ld_out, static_cast<char*>(workspace), stream);
  if (cur != dev) (void)cudaSetDevice(cur);
  return rc;
}

// ------------------------------------------------------------------------------------------------
// MLP block without any allocation: the intermediates live in a fixed array that is part of the library image.
// ------------------------------------------------------------------------------------------------
namespace {
constexpr size_t kMlpStaticBytes = 8u << 20;   // 8 MiB per GPU that loads the library, held until the process exits
static __device__ __align__(256) unsigned char g_mlp_static_scratch[kMlpStaticBytes];
std::mutex g_static_mu;
void* g_static_addr[64] = {nullptr};           // device address of the array, per device ordinal
}  // namespace

int64_t sk_w2a8_mlp_static_scratch_bytes(void) { return static_cast<int64_t>(kMlpStaticBytes); }

int sk_w2a8_mlp_forward_static(sk_w2a8_plan* gate_up, sk_w2a8_plan* down, int64_t M, const void* x_f16, int64_t ld_x,
                               void* out, int64_t ld_out, sk_stream_t stream) {
  int rc = mlp_check(gate_up, down, M);
  if (rc != SK_OK) return rc;
  if (!x_f16 || !out) return SK_ERR_NULL_POINTER;
  if (mlp_layout(M, gate_up->K, down->K).total > kMlpStaticBytes) return SK_ERR_STATIC_SCRATCH_TOO_SMALL;
  const int dev = gate_up->device;
  if (dev < 0 || dev >= 64) return SK_ERR_BAD_ARGUMENT;
  int cur = -1;
  if (cudaGetDevice(&cur) != cudaSuccess) return sk::cuda_fail(gate_up, cudaGetLastError());
  if (cur != dev && cudaSetDevice(dev) != cudaSuccess) return sk::cuda_fail(gate_up, cudaGetLastError());
  void* scratch = nullptr;
  {
    // In host code the array's name is only a handle; the address a kernel can use has to be asked for, once
    // per device and with that device current.
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (!g_static_addr[dev]) {
      void* p = nullptr;
      const cudaError_t e = cudaGetSymbolAddress(&p, g_mlp_static_scratch);
      if (e != cudaSuccess || !p) {
        if (cur != dev) (void)cudaSetDevice(cur);
        return sk::cuda_fail(gate_up, e);
      }
      g_static_addr[dev] = p;
    }
    scratch = g_static_addr[dev];
  }
  rc = mlp_run(gate_up, down, M, x_f16, 0, ld_x, out, ld_out, static_cast<char*>(scratch), stream);
  if (cur != dev) (void)cudaSetDevice(cur);
  return rc;
}

int sk_w2a8_debug_expander_image(const uint8_t* w_tiled_block, int zero_point, const int8_t* expanded_rowmajor,
                                 uint8_t* image_expander, uint8_t* image_tma, int* mismatches, int* device_status,
                                 sk_stream_t stream) {
  if (!w_tiled_block || !expanded_rowmajor || !image_expander || !image_tma || !mismatches || !device_status)
    return SK_ERR_NULL_POINTER;
  if (zero_point < 0 || zero_point > 3) return SK_ERR_BAD_ARGUMENT;
  if ((reinterpret_cast<uintptr_t>(w_tiled_block) & 15) || (reinterpret_cast<uintptr_t>(expanded_rowmajor) & 15) ||
      (reinterpret_cast<uintptr_t>(image_expander) & 15) || (reinterpret_cast<uintptr_t>(image_tma) & 15))
    return SK_ERR_BAD_ALIGNMENT;
  sk::EncodeTiledFn enc = sk::get_encode_fn();
  if (!enc) return SK_ERR_CUDA;
  CUtensorMap map;
  const cuuint64_t dims[2] = {128, 128};
  const cuuint64_t strides[1] = {128};
  const cuuint32_t box[2] = {128u, 128u};
  const cuuint32_t estr[2] = {1u, 1u};
  if (enc(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<int8_t*>(expanded_rowmajor), dims, strides, box, estr,
          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return SK_ERR_CUDA;
  const int dyn = 4096 + 2 * sk::kWxBytes + 1024;
  static int configured[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return SK_ERR_CUDA;
  if (dev < 64 && !configured[dev]) {
    if (cudaFuncSetAttribute(sk::expander_image_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) != cudaSuccess) {
      (void)cudaGetLastError();
      return SK_ERR_CUDA;
    }
    configured[dev] = 1;
  }
  sk::expander_image_kernel<<<1, 128, dyn, static_cast<cudaStream_t>(stream)>>>(map, w_tiled_block, zero_point, image_expander,
                                                                          image_tma, mismatches, device_status);
  if (cudaGetLastError() != cudaSuccess) return SK_ERR_CUDA;
  return SK_OK;
}

int sk_w2a8_debug_stream_cut(int64_t units, int ctas, int cta, int64_t unit, int64_t* range_begin, int64_t* range_end,
                             int* owner_of_unit) {
  if (units <= 0 || ctas <= 0 || ctas > units || cta < 0 || cta >= ctas || unit < 0 || unit >= units) return SK_ERR_BAD_ARGUMENT;
  if (range_begin) *range_begin = sk::stream_range_begin(units, ctas, cta);
  if (range_end) *range_end = sk::stream_range_begin(units, ctas, cta + 1);
  if (owner_of_unit) *owner_of_unit = sk::stream_owner(units, ctas, unit);
  return SK_OK;
}

int sk_sum_row_blocks(const void* blocks, int n_blocks, int64_t block_stride, int64_t ld, int64_t rows, int64_t N,
                      void* out, int64_t ld_out, int out_dtype, sk_stream_t stream) {
  if (!blocks || !out) return SK_ERR_NULL_POINTER;
  if (n_blocks < 1 || n_blocks > 64) return SK_ERR_BAD_ARGUMENT;
  if (out_dtype != SK_OUT_F16 && out_dtype != SK_OUT_BF16) return SK_ERR_BAD_ARGUMENT;
  if (rows <= 0 || N <= 0 || (N % 8) != 0 || ld < N || ld_out < N || N > 0x7fffffffLL) return SK_ERR_BAD_SHAPE;
  if ((reinterpret_cast<uintptr_t>(blocks) & 15) || (reinterpret_cast<uintptr_t>(out) & 15) || (ld % 8) || (ld_out % 8) ||
      (block_stride % 8))
    return SK_ERR_BAD_ALIGNMENT;
  const long long total = rows * (N / 8);
  const int threads = 256;
  const long long want = (total + threads - 1) / threads;
  const int grid = static_cast<int>(want < sk::kChipSms * 16 ? want : sk::kChipSms * 16);
  const auto st = static_cast<cudaStream_t>(stream);
  if (out_dtype == SK_OUT_BF16)
    sk::sum_row_blocks_kernel<true><<<grid, threads, 0, st>>>(static_cast<const uint16_t*>(blocks), block_stride, ld, n_blocks,
                                                             rows, static_cast<int>(N), static_cast<uint16_t*>(out), ld_out);
  else
    sk::sum_row_blocks_kernel<false><<<grid, threads, 0, st>>>(static_cast<const uint16_t*>(blocks), block_stride, ld, n_blocks,
                                                              rows, static_cast<int>(N), static_cast<uint16_t*>(out), ld_out);
  if (cudaGetLastError() != cudaSuccess) return SK_ERR_CUDA;
  return SK_OK;
}

#ifdef SK_TRACE
// Diagnostic build only: device buffer of 5 x 64 clock stamps written by CTA (0,0,0) of the next launches.
int sk_w2a8_set_trace_buffer(long long* device_buffer) {
  sk::g_trace_buffer = device_buffer;
  return SK_OK;
}
#endif

}  // extern "C"
