// The float32 products of the 32-bit path: out[M,N] = A[M,K] . W[N,K]^T with float32 operands.  More than 32 rows (16 of wide
// products) at K of 256 or more run on the tensor cores with operands split in two (gemm_f32_tc5.cu); here are two FFMA
// forms, chosen in sb_gemm_f32:
//
// * gemm_f32_rows_kernel, few rows: bound by reading W once.  A block takes R weight rows; its warps share K in
//   chunks of 128 values, a lane reads 16 bytes of every weight row past L1 and 16 bytes of every activation row
//   (which the SM's blocks keep in L1), so that a warp's loads run along the rows.  Sums: a lane's terms in
//   ascending order, then the lanes in a fixed tree, then the warps in order.
// * gemm_f32_tile_kernel, many rows at a K below 256: bound by FFMA issue and shared-memory loads.  128 threads compute 16 TM x 128
//   outputs, TM x 16 a thread: a load from shared memory costs its bytes times its lanes whether lanes share the
//   address or not, so a thread's tile is as large as the registers allow (TM 8: 24 values loaded for 128 FMA) and
//   two products go into one packed FMA.  Tiles lie [k][row] in shared memory.  Every output is one chain over K in
//   ascending order: the bits of the plain kernel.
//
// Measured on one B200 inside a step of the 1.5B layers (28 layers: 2048, 1536 and 17920 x 1536, 1536 x 8960): three rows
// 15.5 us a product on average where the plain kernel took 636 (one row of 151936 x 1536: 140 us, 6.6 TB/s).
// The tile form and the plain kernel, us a product: 64 rows of 512 x 128 10.5 and 20.8, 201 of 4096 x 128 19.0 and 43.0,
// 1,000 of 1000 x 252 34.8 and 81.7, 2,048 of 4096 x 64 36.6 and 59.9.
// Error of the rows form against float64 at K = 8960: 1.2e-7, of terms one after the other 9e-7.
//
// A row's rounding depends on the number of rows in the launch: its form changes at 17 and 33 rows, and on the tensor cores
// the blocks that share K with the number of tiles.  Up to 16 rows it does not.
// Epilogues as in gemm_plain.cu, which computes the same sums in another order and takes the sizes and
// alignments that these forms do not (K a multiple of 4, rows on 16 bytes).
#include "common.cuh"

namespace {

struct F32Args {
  const float* A;
  const float* W;
  int M, N, K, epilogue;
  const void* bias;
  int bias_dtype;
  const float* residual;
};

// out[m, n] from the finished sum (every epilogue but SWIGLU)
template <typename TO>
__device__ __forceinline__ void f32_store(const F32Args& p, TO* out, int m, int n, float v) {
  if (p.epilogue == SB_EPI_BIAS)
    v += p.bias_dtype == SB_F32 ? ((const float*)p.bias)[n] : __bfloat162float(((const __nv_bfloat16*)p.bias)[n]);
  else if (p.epilogue == SB_EPI_RESIDUAL)
    v += p.residual[(size_t)m * p.N + n];
  else if (p.epilogue == SB_EPI_RELU2)
    v = sb_relu2(v);
  out[(size_t)m * p.N + n] = sb_from_f32<TO>(v);
}

// ---------------------------------------------------------------------------- few rows
constexpr int ROWS_WARPS = 4;
constexpr int ROWS_MAX = 32;              // rows that stream the weights, in groups of eight

__device__ __forceinline__ float4 load_weights(const float* p) {       // read once: past L1
  float4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];\n"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

// Sums of n (a power of two) values over the lanes of a warp in a fixed tree.  With n >= 32 lane l ends with the sums
// of values l * n/32 ... in v[0 ...]; with fewer, lanes 32/n * i ... hold value i in v[0].
template <int N, int O>
__device__ __forceinline__ void lanes_sum(float* v, int lane) {
  if constexpr (O > 0) {
    if constexpr (N > 1) {
      const bool high = lane & O;
#pragma unroll
      for (int i = 0; i < N / 2; ++i) {
        const float other = __shfl_xor_sync(0xffffffffu, high ? v[i] : v[i + N / 2], O);
        v[i] = (high ? v[i + N / 2] : v[i]) + other;
      }
      lanes_sum<N / 2, O / 2>(v, lane);
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], O);
      lanes_sum<1, O / 2>(v, lane);
    }
  }
}

// MT activation rows (rows beyond M repeat the last one and are not stored) times R weight rows; blocks of the same
// weight rows follow each other.  With SWIGLU the R rows are R/2 gate rows and the up rows of the same outputs.
template <int MT, int R, typename TO>
__global__ void __launch_bounds__(ROWS_WARPS * 32)
gemm_f32_rows_kernel(F32Args p, TO* out) {
  constexpr int V = MT * R;
  __shared__ float part[ROWS_WARPS][V];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int groups = (p.M + MT - 1) / MT;
  const int m0 = (int)(blockIdx.x % groups) * MT, b = blockIdx.x / groups;
  const bool swiglu = p.epilogue == SB_EPI_SWIGLU;
  const float* w[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    int n;
    if (swiglu) {
      const int j = b * (R / 2) + r % (R / 2);
      n = j / SB_SWIGLU_BLOCK * 2 * SB_SWIGLU_BLOCK + j % SB_SWIGLU_BLOCK + (r < R / 2 ? 0 : SB_SWIGLU_BLOCK);
    } else {
      n = b * R + r;
    }
    w[r] = p.W + (size_t)min(n, p.N - 1) * p.K;
  }
  const float* a[MT];
#pragma unroll
  for (int i = 0; i < MT; ++i) a[i] = p.A + (size_t)min(m0 + i, p.M - 1) * p.K;

  float acc[V] = {};
  sb_pdl_wait();
  int k = warp * 128 + lane * 4;
#pragma unroll 2
  for (; k < p.K; k += ROWS_WARPS * 128) {
    float4 wv[R];
#pragma unroll
    for (int r = 0; r < R; ++r) wv[r] = load_weights(w[r] + k);
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      const float4 av = *reinterpret_cast<const float4*>(a[i] + k);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float& s = acc[i * R + r];
        s = fmaf(av.x, wv[r].x, s);
        s = fmaf(av.y, wv[r].y, s);
        s = fmaf(av.z, wv[r].z, s);
        s = fmaf(av.w, wv[r].w, s);
      }
    }
  }
  sb_pdl_launch();
  lanes_sum<V, 16>(acc, lane);
  if constexpr (V >= 32) {
#pragma unroll
    for (int i = 0; i < V / 32; ++i) part[warp][lane * (V / 32) + i] = acc[i];
  } else {
    if (lane % (32 / V) == 0) part[warp][lane / (32 / V)] = acc[0];
  }
  __syncthreads();
  if ((int)threadIdx.x >= V) return;
  float s = 0.0f;
#pragma unroll
  for (int i = 0; i < ROWS_WARPS; ++i) s += part[i][threadIdx.x];
  const int m = m0 + threadIdx.x / R, r = threadIdx.x % R;
  if (swiglu) {
    // the up value's thread sits R/2 further on, in the same warp
    const unsigned mask = V >= 32 ? 0xffffffffu : (1u << V) - 1u;
    const float up = __shfl_down_sync(mask, s, R / 2);
    const int j = b * (R / 2) + r;
    if (r < R / 2 && m < p.M && j < p.N / 2) out[(size_t)m * (p.N / 2) + j] = sb_from_f32<TO>(sb_silu(s) * up);
    return;
  }
  const int n = b * R + r;
  if (m < p.M && n < p.N) f32_store(p, out, m, n, s);
}

// ---------------------------------------------------------------------------- many rows
constexpr int BN = 128, BK = 16, TILE_THREADS = 128;
constexpr int W_PITCH = BN + 4;           // 4 more: the 16 rows x 2 columns a warp writes at once fall on 32 banks

template <int TM>
struct Tile {
  static constexpr int BM = 16 * TM, PITCH = BM + 4;
  static constexpr int STAGE = BK * (PITCH + W_PITCH);
  static constexpr int FLOATS = 2 * STAGE > BM * W_PITCH ? 2 * STAGE : BM * W_PITCH;     // the finished tile lies over the stages
  static constexpr int A_UNITS = BM / 16 * 2, W_UNITS = BN / 16 * 2;      // 16 rows x 2 columns of 16 bytes, a warp's load
  static constexpr int A_LOADS = (A_UNITS + 3) / 4, W_LOADS = W_UNITS / 4;
};

struct Pair {
  unsigned long long v;
};
__device__ __forceinline__ Pair pack(float a, float b) {
  Pair r;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack(Pair p, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;\n" : "=f"(a), "=f"(b) : "l"(p.v));
}
__device__ __forceinline__ void fma_pair(Pair& c, Pair a, Pair b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(c.v) : "l"(a.v), "l"(b.v));
}

template <int TM, typename TO>
__global__ void __launch_bounds__(TILE_THREADS, 2)
gemm_f32_tile_kernel(F32Args p, TO* out) {
  using T = Tile<TM>;
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tiles_m = (p.M + T::BM - 1) / T::BM;       // tiles of the same weight rows follow each other
  const int m0 = (int)(blockIdx.x % tiles_m) * T::BM, n0 = (int)(blockIdx.x / tiles_m) * BN;
  const int tiles = (p.K + BK - 1) / BK;
  const int r_in = lane >> 1, c_in = lane & 1;          // a warp's load: 16 rows, two neighbouring 16-byte columns

  float4 ra[T::A_LOADS], rw[T::W_LOADS];
  auto fetch = [&](int t) {
    const int kb = t * BK;
#pragma unroll
    for (int i = 0; i < T::A_LOADS; ++i) {
      const int u = i * 4 + warp, k = kb + ((u & 1) * 2 + c_in) * 4;
      const int m = m0 + (u >> 1) * 16 + r_in;
      ra[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (u < T::A_UNITS && m < p.M && k < p.K) ra[i] = *reinterpret_cast<const float4*>(p.A + (size_t)m * p.K + k);
    }
#pragma unroll
    for (int i = 0; i < T::W_LOADS; ++i) {
      const int u = i * 4 + warp, k = kb + ((u & 1) * 2 + c_in) * 4;
      const int n = n0 + (u >> 1) * 16 + r_in;
      rw[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (n < p.N && k < p.K) rw[i] = __ldg(reinterpret_cast<const float4*>(p.W + (size_t)n * p.K + k));
    }
  };
  auto put = [&](int stage) {
    float* sa = smem + stage * T::STAGE;
    float* sw = sa + BK * T::PITCH;
#pragma unroll
    for (int i = 0; i < T::A_LOADS; ++i) {
      const int u = i * 4 + warp, r = (u >> 1) * 16 + r_in, k = ((u & 1) * 2 + c_in) * 4;
      if (u >= T::A_UNITS) continue;
      sa[k * T::PITCH + r] = ra[i].x;
      sa[(k + 1) * T::PITCH + r] = ra[i].y;
      sa[(k + 2) * T::PITCH + r] = ra[i].z;
      sa[(k + 3) * T::PITCH + r] = ra[i].w;
    }
#pragma unroll
    for (int i = 0; i < T::W_LOADS; ++i) {
      const int u = i * 4 + warp, r = (u >> 1) * 16 + r_in, k = ((u & 1) * 2 + c_in) * 4;
      sw[k * W_PITCH + r] = rw[i].x;
      sw[(k + 1) * W_PITCH + r] = rw[i].y;
      sw[(k + 2) * W_PITCH + r] = rw[i].z;
      sw[(k + 3) * W_PITCH + r] = rw[i].w;
    }
  };

  const int tx = tid & 7, ty = tid >> 3;               // columns tx * 4 + 32 j, rows ty * TM + i
  Pair acc[TM][8];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = pack(0.0f, 0.0f);

  sb_pdl_wait();
  fetch(0);
  put(0);
  __syncthreads();
  for (int t = 0; t < tiles; ++t) {
    const int stage = t & 1;
    if (t + 1 < tiles) fetch(t + 1);
    const float* sa = smem + stage * T::STAGE + ty * TM;
    const float* sw = smem + stage * T::STAGE + BK * T::PITCH + tx * 4;
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      Pair a[TM], w[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 v = *reinterpret_cast<const float4*>(sw + k * W_PITCH + 32 * j);
        w[2 * j] = pack(v.x, v.y);
        w[2 * j + 1] = pack(v.z, v.w);
      }
      if constexpr (TM % 4 == 0) {
#pragma unroll
        for (int i = 0; i < TM; i += 4) {
          const float4 v = *reinterpret_cast<const float4*>(sa + k * T::PITCH + i);
          a[i] = pack(v.x, v.x); a[i + 1] = pack(v.y, v.y); a[i + 2] = pack(v.z, v.z); a[i + 3] = pack(v.w, v.w);
        }
      } else {
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          const float v = sa[k * T::PITCH + i];
          a[i] = pack(v, v);
        }
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) fma_pair(acc[i][j], a[i], w[j]);
    }
    // the other stage was last read before the barrier that ended the previous round
    if (t + 1 < tiles) put(stage ^ 1);
    __syncthreads();
  }
  sb_pdl_launch();

  // the tile through shared memory, so that a warp writes along a row
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float4 v;
      unpack(acc[i][2 * j], v.x, v.y);
      unpack(acc[i][2 * j + 1], v.z, v.w);
      *reinterpret_cast<float4*>(smem + (ty * TM + i) * W_PITCH + tx * 4 + 32 * j) = v;
    }
  __syncthreads();
  if (p.epilogue == SB_EPI_SWIGLU) {
    const int c = tid & 63, at = c / SB_SWIGLU_BLOCK * 2 * SB_SWIGLU_BLOCK + c % SB_SWIGLU_BLOCK, j = n0 / 2 + c;
    if (j < p.N / 2)
      for (int r = tid >> 6; r < T::BM && m0 + r < p.M; r += 2)
        out[(size_t)(m0 + r) * (p.N / 2) + j] =
            sb_from_f32<TO>(sb_silu(smem[r * W_PITCH + at]) * smem[r * W_PITCH + at + SB_SWIGLU_BLOCK]);
  } else if (n0 + tid < p.N) {
    for (int r = 0; r < T::BM && m0 + r < p.M; ++r) f32_store(p, out, m0 + r, n0 + tid, smem[r * W_PITCH + tid]);
  }
}

template <int MT, int R, typename TO>
void launch_rows(const F32Args& p, TO* out, cudaStream_t stream) {
  const int per = p.epilogue == SB_EPI_SWIGLU ? R / 2 : R, n = p.epilogue == SB_EPI_SWIGLU ? p.N / 2 : p.N;
  sb_launch<SB_K_OTHER>(gemm_f32_rows_kernel<MT, R, TO>, dim3((unsigned)((p.M + MT - 1) / MT) * (unsigned)((n + per - 1) / per)), dim3(ROWS_WARPS * 32), 0,
                        stream, p, out);
}

template <int TM>
long tile_blocks(const F32Args& p) { return (long)((p.M + Tile<TM>::BM - 1) / Tile<TM>::BM) * ((p.N + BN - 1) / BN); }

template <int TM, typename TO>
int launch_tile(const F32Args& p, TO* out, cudaStream_t stream) {
  const size_t smem = Tile<TM>::FLOATS * sizeof(float);
  // every call sets it, as it belongs to the current device's copy of the kernel; it costs nothing beside the product
  if (cudaError_t e = cudaFuncSetAttribute(gemm_f32_tile_kernel<TM, TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem))
    SB_FAIL(SB_ERR_CUDA, "sb_gemm_f32: %s", cudaGetErrorString(e));
  sb_launch<SB_K_OTHER>(gemm_f32_tile_kernel<TM, TO>, dim3((unsigned)tile_blocks<TM>(p)), dim3(TILE_THREADS), smem, stream, p, out);
  return SB_OK;
}

template <typename TO>
int run_f32(const F32Args& p, TO* out, int n_sms, cudaStream_t stream) {
  if (p.M <= ROWS_MAX) {
    if (p.M == 1) launch_rows<1, 4, TO>(p, out, stream);
    else if (p.M == 2) launch_rows<2, 4, TO>(p, out, stream);
    else if (p.M <= 4) launch_rows<4, 4, TO>(p, out, stream);
    else launch_rows<8, 4, TO>(p, out, stream);
    return SB_OK;
  }
  // the largest tile that gives every SM a block, else the smallest
  if (tile_blocks<8>(p) >= n_sms) return launch_tile<8, TO>(p, out, stream);
  if (tile_blocks<4>(p) >= n_sms) return launch_tile<4, TO>(p, out, stream);
  return launch_tile<2, TO>(p, out, stream);
}

}  // namespace

// The tensor-core form (gemm_f32_tc5.cu).  Its splitting of the operands (22 to 23 bits) makes an error of 1.4e-7 whatever K is; terms
// added one after the other have 2.0e-7 at K = 128, 2.9e-7 at 256, and a short K leaves its stages no time to overlap.
// Streaming the weights / the tensor cores, us at 17 and 28 rows: 2048 x 1536 11.0, 13.9 / 12.2, 12.7; 1536 x 8960 32.9, 47.9 / 36.3, 36.8;
// 3584 x 3584 32.9, 44.5 / 30.7, 31.4; 6144 x 1536 27.0, 35.2 / 26.9, 27.6; 8192 x 1536 35.5, 45.9 / 27.9, 28.6; 17920 x 1536 73.9, 96.9 /
// 50.5, 51.2; 37888 x 3584 299, 405 / 209, 211.  8,192 columns is where the tensor cores gain a fifth and more at every count from 17 on
// (64 tiles of 128 columns); below it the two lie within a tenth of each other at 17 rows, and the line stays at 33.
constexpr int SPLIT_MIN_K = 256, SPLIT_WIDE_ROWS = 16, SPLIT_WIDE_N = 8192;
int sb_gemm_f32_tc5(const float* A, const float* W, int M, int N, int K, int epilogue, const void* bias, int bias_dtype,
                    const float* residual, void* out, int out_dtype, int n_sms, cudaStream_t stream);

int sb_check_linear_args(const char* who, int M, int N, int K, int epilogue, const void* bias, const float* residual, int out_dtype);

extern "C" int sb_gemm_f32(const float* A, const float* W, int M, int N, int K, int epilogue, const void* bias, int bias_dtype,
                           const float* residual, void* out, int out_dtype, int n_sms, cudaStream_t stream) {
  if (!sb_valid_dtype(out_dtype) || (bias && !sb_valid_dtype(bias_dtype)))
    SB_FAIL(SB_ERR_ARG, "sb_gemm_f32: dtype codes %d %d", out_dtype, bias_dtype);
  if (int rc = sb_check_linear_args("sb_gemm_f32", M, N, K, epilogue, bias, residual, out_dtype)) return rc;
  if (!A || !W || n_sms <= 0) SB_FAIL(SB_ERR_ARG, "sb_gemm_f32: operands missing, or %d SMs", n_sms);
  if (K % 4 || (((uintptr_t)A | (uintptr_t)W) & 15))
    SB_FAIL(SB_ERR_UNSUPPORTED, "sb_gemm_f32: rows must start on 16 bytes (K = %d): sb_gemm_plain takes the others", K);
  if (M > 65535 * 64) SB_FAIL(SB_ERR_UNSUPPORTED, "sb_gemm_f32: M=%d is too many rows", M);
  if (K >= SPLIT_MIN_K && (M > ROWS_MAX || (M > SPLIT_WIDE_ROWS && N >= SPLIT_WIDE_N)))
    return sb_gemm_f32_tc5(A, W, M, N, K, epilogue, bias, bias_dtype, residual, out, out_dtype, n_sms, stream);
  const F32Args p{A, W, M, N, K, epilogue, bias, bias_dtype, residual};
  const int rc = out_dtype == SB_F32 ? run_f32(p, (float*)out, n_sms, stream) : run_f32(p, (__nv_bfloat16*)out, n_sms, stream);
  if (rc) return rc;
  SB_CHECK_LAUNCH("sb_gemm_f32");
  return SB_OK;
}
