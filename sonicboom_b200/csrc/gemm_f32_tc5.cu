// float32 products of more than a few rows on the tensor cores: out[M,N] = A[M,K] . W[N,K]^T, every operand value split
// into two TF32 values.
//
// x = hi + lo with hi = x rounded to TF32 (11 significant bits) and lo = x - hi, exact in float32, cut to TF32:
// 22 to 23 bits of x.  A product is hi hi + hi lo + lo hi (lo lo is below float32's rounding), three MMAs
// (`tcgen05.mma kind::tf32`) on one float32 accumulator in tensor memory.  The accumulator covers 32 values of K only;
// its sums are then added up in registers with float32's own rounding, so that the tensor cores' accumulation, which may
// not round to nearest, stays a chain of twelve.
// Error against 64 bits, 2-norm, here / one term after the other: K = 256 1.4e-7 / 2.9e-7, 1,536 1.5e-7 / 7.0e-7, 8,960 1.8e-7 / 1.7e-6; with positive,
// long-tailed and gated operands at most a tenth more.  Splitting an operand into two values of a shorter type and leaving
// out the product of the small halves is a published method (Ootomo and Yokota, "Recovering single precision accuracy from
// Tensor Cores while surpassing the FP32 theoretical peak performance", 2022).
//
// A block computes 128 weight rows (the MMA's rows) x up to 224 tokens.  Warp 0 loads float32 tiles by TMA (128-byte
// swizzle, 32 values of K), warp 1 issues the MMAs, and eight warps do the arithmetic: they split a stage's
// values (hi over the loaded value, lo into a buffer of its own; the order of the values does not matter, so the swizzle is left as it is), and while its
// MMAs run drain the stage before it from the other of two accumulators.  Where the tiles leave SMs idle a cluster of blocks
// shares K; the partial tiles meet in distributed shared memory and are added in rank order, so no workspace is needed.
//
// Bound by the tensor cores (three TF32 products) and, close to it, by shared memory, which the MMAs and the splitting share.
// 201 rows, us, packed FMA tiles / here: 17920 x 1536 with the gate 327 / 100, 1536 x 8960 278 / 74, 2048 x 1536 48 / 26, 1536 x 1536 55 / 25;
// a prompt of 201 tokens of the 1.5B model 22.6 to 8.5 ms, now 7.2 (the plain kernel: 110).  What is left is a stage's chain of
// loading, splitting, MMAs and draining: 2 us for 32 values of K at 224 tokens, of which the MMAs take 0.7.
//
// A value that is not finite, or that rounds to infinity as TF32, makes its sums NaN here (infinity times a lo of 0): a result that is not
// finite is computed once more term by term in float32, and is then what the plain kernel gives.  So is a result below TC_SMALL:
// below 2^-112 an operand is off by up to 2^-136, its last bit as TF32, more than the 2^-24 of it that a float32 result may be off
// (512 terms with operands around 2^-126: 3.0e-4, term by term 4.0e-7).  Over K terms that is at most K 2^-135 times the largest
// operand: below 2^-24 of a result of TC_SMALL for operands up to 2^41 / K.  What is left are products of operands beyond that
// with ones below 2^-112, and operands below 2^-136, which count as 0 where nothing else is in the sum.  (Looking for small operands
// while they are split closes that too, but cost the gate/up product of 201 rows 5 % and the down product 7.)
#include <cooperative_groups.h>
#include <float.h>

#include "device_cache.h"
#include "tc5.cuh"

namespace cg = cooperative_groups;

namespace {

// 224 tokens: three stages beside the two of lo, and 112 sums a thread; with 256 two stages would be left.
constexpr int TC_ROWS = 128, TC_K = 32, TC_MAX_TOKENS = 224, TC_ACC = 256;        // weight rows, values of K of a stage, tokens, columns between accumulators
constexpr int TC_ROW_BYTES = TC_K * 4;                              // a swizzled row
constexpr int TC_W_BYTES = TC_ROWS * TC_ROW_BYTES;
constexpr int TC_WARPS = 8, TC_THREADS = 64 + 32 * TC_WARPS;
constexpr int TC_PITCH = TC_ROWS + 4;                               // of a token's sums in the partial tile
constexpr int TC_MAX_STAGES = 6, TC_SMEM = 225 * 1024;

constexpr float TC_SMALL = 0x1p-70f;

struct TcArgs {
  const float* A;
  const float* W;
  int M, N, K, epilogue;
  const void* bias;
  int bias_dtype;
  const float* residual;
  int tokens, tiles_m, stages;                       // tokens of a tile (a multiple of 32), token tiles, ring stages
};

// W and A of a stage.  The ring's stages are loaded and become hi in place; two more of the same size hold lo of the last two.
__host__ __device__ inline int tc_stage_bytes(int tokens) { return TC_W_BYTES + tokens * TC_ROW_BYTES; }

// K-major rows of 128 bytes with the 128-byte swizzle, groups of 8 rows 1024 bytes apart
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void umma_tf32(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// In whole-number arithmetic, at four times the rate of the conversion instruction: hi rounds half away from zero (a carry into the
// exponent is the right next value), lo is cut.  An infinity, or a value that rounds to one, leaves a lo that is not finite, and so
// does a NaN whose bits the carry turned into a zero.
__device__ __forceinline__ void split_value(float x, float& hi, float& lo) {
  hi = __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
  lo = __uint_as_float(__float_as_uint(x - hi) & 0xffffe000u);
}

template <typename TO>
__global__ void __launch_bounds__(TC_THREADS, 1)
gemm_f32_tc5_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const TcArgs p,
                    TO* out) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bars[3 * TC_MAX_STAGES + 4];
  __shared__ uint32_t tmem_slot;
  const uint32_t raw = (uint32_t)__cvta_generic_to_shared(smem_raw);
  const uint32_t ring = (raw + 1023u) & ~1023u;
  unsigned char* ring_ptr = smem_raw + (ring - raw);
  const uint32_t bar0 = (uint32_t)__cvta_generic_to_shared(bars);
  // loaded[s], split[s], empty[s]; the accumulators' full[2] and drained[2]
  auto loaded = [&](int s) { return bar0 + 8 * s; };
  auto split = [&](int s) { return bar0 + 8 * (TC_MAX_STAGES + s); };
  auto empty = [&](int s) { return bar0 + 8 * (2 * TC_MAX_STAGES + s); };
  auto full = [&](int a) { return bar0 + 8 * (3 * TC_MAX_STAGES + a); };
  auto drained = [&](int a) { return bar0 + 8 * (3 * TC_MAX_STAGES + 2 + a); };
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = (int)(blockIdx.x % p.tiles_m) * p.tokens, n0 = (int)(blockIdx.x / p.tiles_m) * TC_ROWS;
  const int k_tiles = (p.K + TC_K - 1) / TC_K, splits = gridDim.z, rank = blockIdx.z;
  const int t0 = (int)((long)k_tiles * rank / splits), n_k = (int)((long)k_tiles * (rank + 1) / splits) - t0;
  const int stage_bytes = tc_stage_bytes(p.tokens), a_bytes = p.tokens * TC_ROW_BYTES, S = p.stages;

  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(loaded(s), 1);
      mbar_init(split(s), TC_WARPS / 2);
      mbar_init(empty(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(full(a), 1);
      mbar_init(drained(a), TC_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    fence_async_smem();
  }
  if (warp == 1) tmem_alloc((uint32_t)__cvta_generic_to_shared(&tmem_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *(volatile uint32_t*)&tmem_slot;

  float acc[TC_MAX_TOKENS / 2];                        // this thread's weight row, its group's half of the tokens
  const int half = p.tokens / 2;
  bool ok = true;
  if (warp == 0) {
    if (lane == 0) {
      // ---- loads: weights first, they wait for nobody
      const int head = min(S, n_k);
      for (int i = 0; i < head; ++i) {
        mbar_expect_tx(loaded(i), TC_W_BYTES + a_bytes);
        tma_load_2d(ring + i * stage_bytes, &map_w, (t0 + i) * TC_K, n0, loaded(i));
      }
      sb_pdl_wait();
      for (int i = 0; i < head; ++i) tma_load_2d(ring + i * stage_bytes + TC_W_BYTES, &map_a, (t0 + i) * TC_K, m0, loaded(i));
      int issued = head;
      for (int i = head; i < n_k; ++i) {
        const int s = i % S;
        ok = mbar_wait(empty(s), ((i / S) & 1) ^ 1, 11);
        if (!ok) break;
        mbar_expect_tx(loaded(s), TC_W_BYTES + a_bytes);
        tma_load_2d(ring + s * stage_bytes, &map_w, (t0 + i) * TC_K, n0, loaded(s));
        tma_load_2d(ring + s * stage_bytes + TC_W_BYTES, &map_a, (t0 + i) * TC_K, m0, loaded(s));
        issued = i + 1;
      }
      sb_pdl_launch();
      if (!ok)                                         // copies in flight land before the block's memory goes away
        for (int i = max(0, issued - S); i < issued; ++i) mbar_wait(loaded(i % S), (i / S) & 1, 12);
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      // ---- MMAs: float32 accumulator, TF32 operands, both K-major, 128 rows x tokens
      const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(p.tokens >> 3) << 17) | ((uint32_t)(TC_ROWS >> 4) << 24);
      for (int i = 0; i < n_k; ++i) {
        const int s = i % S, a = i & 1;
        ok = mbar_wait(split(s), (i / S) & 1, 13) && mbar_wait(drained(a), ((i >> 1) & 1) ^ 1, 14);
        if (!ok) break;
        tc_fence_after();
        const uint32_t w_hi = ring + s * stage_bytes, a_hi = w_hi + TC_W_BYTES, w_lo = ring + (S + a) * stage_bytes, a_lo = w_lo + TC_W_BYTES;
        const uint32_t d = tmem + a * TC_ACC;
        // the small products first
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const uint64_t wd = tc_desc(j == 0 ? w_lo : w_hi), ad = tc_desc(j == 1 ? a_lo : a_hi);
#pragma unroll
          for (int k = 0; k < TC_K / 8; ++k) umma_tf32(d, wd + (uint64_t)(k * 2), ad + (uint64_t)(k * 2), idesc, j > 0 || k > 0);
        }
        umma_commit(empty(s));
        umma_commit(full(a));
      }
    }
    __syncwarp();
  } else {
    // ---- splitting and draining; thread: lanes 32 q ... of tensor memory, half `group` of the tokens
    const int w = warp - 2, q = warp & 3, group = w >> 2, t = tid - 64;
#pragma unroll
    for (int j = 0; j < TC_MAX_TOKENS / 2; ++j) acc[j] = 0.0f;
    auto drain = [&](int i) {
      const int a = i & 1;
      if (!__all_sync(0xffffffffu, mbar_wait(full(a), (i >> 1) & 1, 15))) return false;
      tc_fence_after();
      const uint32_t col = tmem + ((uint32_t)(q * 32) << 16) + a * TC_ACC + group * half;
#pragma unroll
      for (int c = 0; c < TC_MAX_TOKENS / 32; ++c) {
        if (c * 16 >= half) break;
        uint32_t r[32];
        tmem_ld16(col + c * 16, r);
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[c * 16 + j] += __uint_as_float(r[j]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(drained(a));
      return true;
    };
    for (int i = 0; i < n_k; ++i) {
      // the two groups split every second stage each, so that one's waits and fences overlap the other's work
      if ((i & 1) == group) {
        const int s = i % S;
        ok = __all_sync(0xffffffffu, mbar_wait(loaded(s), (i / S) & 1, 16));
        if (!ok) break;
        // the lo stage was last read by the MMAs of two stages ago, which this warp has drained
        unsigned char* base = ring_ptr + (size_t)s * stage_bytes;
        unsigned char* low = ring_ptr + (size_t)(S + (i & 1)) * stage_bytes;
#pragma unroll 4
        for (int o = (t & 127) * 16; o < stage_bytes; o += 16 * TC_WARPS * 16) {
          float4* at = reinterpret_cast<float4*>(base + o);
          const float4 x = *at;
          float4 hi, lo;
          split_value(x.x, hi.x, lo.x);
          split_value(x.y, hi.y, lo.y);
          split_value(x.z, hi.z, lo.z);
          split_value(x.w, hi.w, lo.w);
          *at = hi;
          *reinterpret_cast<float4*>(low + o) = lo;
        }
        fence_async_smem();                            // the MMAs read what was written here
        __syncwarp();
        if (lane == 0) mbar_arrive(split(s));
      }
      if (i > 0) {
        ok = drain(i - 1);
        if (!ok) break;
      }
    }
    if (ok && n_k > 0) ok = drain(n_k - 1);
  }

  // the partial tile over the ring (every load and every MMA has ended), then the cluster's blocks share out its tokens
  sb_pdl_wait();                                       // the residual
  tc_fence_before();
  __syncthreads();
  float* part = reinterpret_cast<float*>(ring_ptr);
  if (warp >= 2) {
    const int q = warp & 3, group = (warp - 2) >> 2;
#pragma unroll
    for (int j = 0; j < TC_MAX_TOKENS / 2; ++j)
      if (j < half) part[(group * half + j) * TC_PITCH + q * 32 + lane] = acc[j];
  }
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  const float* peer[8];
#pragma unroll
  for (int s = 0; s < 8; ++s) peer[s] = s < splits ? cluster.map_shared_rank(part, s) : part;
  // the sum of token r and weight row c of the tile
  auto sum_at = [&](int r, int c) {
    float v = 0.0f;
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (s < splits) v += peer[s][r * TC_PITCH + c];
    const float size = fabsf(v);
    if (!(size <= FLT_MAX) || (size < TC_SMALL && size > 0.0f)) {
      const float4* a = reinterpret_cast<const float4*>(p.A + (size_t)(m0 + r) * p.K);
      const float4* w = reinterpret_cast<const float4*>(p.W + (size_t)(n0 + c) * p.K);
      v = 0.0f;
      for (int k = 0; k < p.K / 4; ++k) v = fmaf(a[k].w, w[k].w, fmaf(a[k].z, w[k].z, fmaf(a[k].y, w[k].y, fmaf(a[k].x, w[k].x, v))));
    }
    return v;
  };
  const int live = min(p.tokens, p.M - m0);
  if (p.epilogue == SB_EPI_SWIGLU) {
    const int c = tid & 63, at = c / SB_SWIGLU_BLOCK * 2 * SB_SWIGLU_BLOCK + c % SB_SWIGLU_BLOCK, j = n0 / 2 + c;
    if (tid < 256 && j < p.N / 2)
      for (int r = rank * 4 + (tid >> 6); r < live; r += 4 * splits)
        out[(size_t)(m0 + r) * (p.N / 2) + j] = sb_from_f32<TO>(sb_silu(sum_at(r, at)) * sum_at(r, at + SB_SWIGLU_BLOCK));
  } else {
    const int c = tid & 127, n = n0 + c;
    if (tid < 256 && n < p.N) {
      float add = 0.0f;
      if (p.epilogue == SB_EPI_BIAS)
        add = p.bias_dtype == SB_F32 ? ((const float*)p.bias)[n] : __bfloat162float(((const __nv_bfloat16*)p.bias)[n]);
      for (int r = rank * 2 + (tid >> 7); r < live; r += 2 * splits) {
        float v = sum_at(r, c);
        if (p.epilogue == SB_EPI_BIAS) v += add;
        else if (p.epilogue == SB_EPI_RESIDUAL) v += p.residual[(size_t)(m0 + r) * p.N + n];
        else if (p.epilogue == SB_EPI_RELU2) v = sb_relu2(v);
        out[(size_t)(m0 + r) * p.N + n] = sb_from_f32<TO>(v);
      }
    }
  }
  cluster.sync();                                      // nobody's tile goes while another block reads it
  if (warp == 1) tmem_dealloc(tmem, 512);
}

bool tc_map(CUtensorMap* map, const float* base, int rows, int K, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)K * 4};
  const cuuint32_t box[2] = {(cuuint32_t)TC_K, (cuuint32_t)box_rows};
  const cuuint32_t elem[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Clusters of `blocks` blocks that the current device runs at once.
template <typename TO>
int tc_clusters(int blocks) {
  static SbDeviceCache most[9];
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) device = -1;
  return most[blocks].get(device, [&] {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1, 1, blocks);
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = TC_SMEM;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = blocks;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_f32_tc5_kernel<TO>, &cfg) == cudaSuccess) return n;
    cudaGetLastError();
    return -1;
  });
}

// Blocks that share a tile's K: as many as run at once, at most eight, with at least four stages of K each.  A block has an SM
// to itself and a cluster's blocks lie in one group of SMs, so fewer than (SMs / 8) clusters of eight may fit: 16 tiles with eight
// blocks each ran in two waves.
template <typename TO>
int tc_splits(long tiles, int K, int n_sms) {
  const long k_tiles = (K + TC_K - 1) / TC_K;
  for (int s = 8; s > 1; --s)
    if (k_tiles >= 4 * s && tiles * s <= n_sms && tiles <= tc_clusters<TO>(s)) return s;
  return 1;
}

template <typename TO>
int tc_launch(TcArgs p, TO* out, int n_sms, cudaStream_t stream) {
  p.tiles_m = (p.M + TC_MAX_TOKENS - 1) / TC_MAX_TOKENS;
  p.tokens = ((p.M + p.tiles_m - 1) / p.tiles_m + 31) / 32 * 32;
  p.tiles_m = (p.M + p.tokens - 1) / p.tokens;
  const long tiles = (long)p.tiles_m * ((p.N + TC_ROWS - 1) / TC_ROWS);
  if (tiles > 2147483647L) SB_FAIL(SB_ERR_UNSUPPORTED, "sb_gemm_f32: too many tiles");
  p.stages = (TC_SMEM - 1024) / tc_stage_bytes(p.tokens) - 2;
  if (p.stages > TC_MAX_STAGES) p.stages = TC_MAX_STAGES;
  CUtensorMap map_w, map_a;
  if (!tc_map(&map_w, p.W, p.N, p.K, TC_ROWS) || !tc_map(&map_a, p.A, p.M, p.K, p.tokens))
    SB_FAIL(SB_ERR_CUDA, "sb_gemm_f32: cuTensorMapEncodeTiled failed");
  // every call sets it, as it belongs to the current device's copy of the kernel; it costs nothing beside the product
  if (cudaError_t e = cudaFuncSetAttribute(gemm_f32_tc5_kernel<TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM))
    SB_FAIL(SB_ERR_CUDA, "sb_gemm_f32: %s", cudaGetErrorString(e));
  const int splits = tc_splits<TO>(tiles, p.K, n_sms);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)tiles, 1, splits);
  cfg.blockDim = dim3(TC_THREADS);
  cfg.dynamicSmemBytes = TC_SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = splits;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (sb_pdl_enabled() & SB_K_OTHER) ? 2 : 1;
  cudaLaunchKernelEx(&cfg, gemm_f32_tc5_kernel<TO>, map_w, map_a, p, out);
  return SB_OK;
}

}  // namespace

int sb_gemm_f32_tc5(const float* A, const float* W, int M, int N, int K, int epilogue, const void* bias, int bias_dtype,
                    const float* residual, void* out, int out_dtype, int n_sms, cudaStream_t stream) {
  TcArgs p{};
  p.A = A; p.W = W; p.M = M; p.N = N; p.K = K; p.epilogue = epilogue; p.bias = bias; p.bias_dtype = bias_dtype; p.residual = residual;
  const int rc = out_dtype == SB_F32 ? tc_launch(p, (float*)out, n_sms, stream) : tc_launch(p, (__nv_bfloat16*)out, n_sms, stream);
  if (rc) return rc;
  SB_CHECK_LAUNCH("sb_gemm_f32 (tensor cores)");
  return SB_OK;
}

int sb_gemm_f32_tc5_status() { return tc5_read_status(); }
