// Token selection on the device: greedy argmax and the seeded sampler, a cluster of blocks per row.
//
// Bound by latency: a row is 0.6 MB that the head's product has just left in L2.  The blocks of a cluster share it.  For
// stage 3 every thread takes the largest of its values; the least of the blocks' RANK_SHARE-th largest such maxima is
// a value that at least CANDIDATES of the row reach, and only those that reach it (about 400 of a row of
// random logits) are collected in the first block and sorted.  Rows where more than MAX_LIST reach it (many equal logits) go through a
// radix select in the first block instead, with the same result.  Measured at a vocabulary of 152,064 on one B200, us: 8
// rows sampled at temperature 0.7 23.3, 64 rows 36 (one block per row, five passes over it for a radix select and the
// filters by one thread took 342 and 389); greedy, one row 4.0, 64 rows 7.2, 256 rows 31 (7.0, 10.0 and 30).
//
// The order of stages is the reference's (capi/include/sonicboom/capi.h:629-645,
// core/src/nn/sampling.cpp:157-203, 257-352):
//   1. repetition / presence / frequency penalties over the row's history window;
//   2. temperature <= 0: the argmax of the penalized logits, ties toward the lowest id;
//   3. otherwise z = logit / T (one float division); the 256 highest z, ties toward the lower
//      id, in (z descending, id ascending) order;
//   4. candidates more than 30 below the maximum are dropped; top_k; min_p (z < max + ln(min_p)
//      dropped); nucleus (shortest prefix whose normalized mass reaches top_p);
//   5. Gumbel-max draw: u = (bits[0] + 0.5) / 2^32 with bits = Philox4x32-10(counter =
//      {pos_lo, pos_hi, id, 0}, key = seed); the highest z - log(-log u) wins, ties toward the
//      lower id.  `position` is the absolute position of the token being produced, so a
//      sequence's draws do not depend on its row in the batch.
// Penalties are applied to the logits row in place and undone before the kernel returns.
#include <cooperative_groups.h>
#include <math.h>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int THREADS = 512;
constexpr int MOST = 8;              // blocks that share a row, at most
constexpr int CANDIDATES = 256;      // core/include/sonicboom/nn/sampling.h:68
constexpr float LOGIT_WINDOW = 30.0f;  // core/include/sonicboom/nn/sampling.h:61
constexpr int MAX_HISTORY = 1024;    // the reference's device penalty window (capi.cpp:2711-2715)
constexpr int MAX_LIST = 2048;       // values collected for the sort

__device__ __forceinline__ uint32_t order_key(float z) {
  // Monotone map float -> uint32 (larger z, larger key); NaN sorts lowest.
  if (z != z) return 0u;
  const uint32_t b = __float_as_uint(z);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// The float an order key stands for (a NaN for the key of every NaN).
__device__ __forceinline__ float key_value(uint32_t k) {
  if (k == 0u) return __uint_as_float(0x7fffffffu);
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

__device__ void philox4x32_10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, uint64_t key,
                              uint32_t out[4]) {
  // Random123 constants (core/src/nn/sampling.cpp:207-227).
  const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
  uint32_t k0 = (uint32_t)key, k1 = (uint32_t)(key >> 32);
  for (int r = 0; r < 10; ++r) {
    const uint32_t hi0 = __umulhi(M0, c0), lo0 = M0 * c0;
    const uint32_t hi1 = __umulhi(M1, c2), lo1 = M1 * c2;
    const uint32_t n0 = hi1 ^ c1 ^ k0, n1 = lo1, n2 = hi0 ^ c3 ^ k1, n3 = lo0;
    c0 = n0; c1 = n1; c2 = n2; c3 = n3;
    k0 += W0; k1 += W1;
  }
  out[0] = c0; out[1] = c1; out[2] = c2; out[3] = c3;
}

// The largest of a block's 64-bit values (every thread returns it); `red` holds 32.
__device__ unsigned long long block_max(unsigned long long v, unsigned long long* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  if (lane == 0) red[warp] = v;
  __syncthreads();
  v = lane < THREADS / 32 ? red[lane] : 0ull;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  return v;
}

// A value and its id as one number: the larger value first, ties toward the lower id.
__device__ __forceinline__ unsigned long long key_and_id(uint32_t key, int id) {
  return ((unsigned long long)key << 32) | (uint32_t)(~(uint32_t)id);
}

// The CANDIDATES highest z of the row into `cand` (any order) by a radix select of the threshold key: for rows where
// too many values are equal to be listed.  One block; `hist` holds 256.
__device__ void select_by_radix(const float* lg, int vocab, float T, unsigned long long* cand, uint32_t* hist) {
  __shared__ uint32_t s_prefix, s_need, s_count, s_running;
  const int tid = threadIdx.x;
  const uint32_t want = (uint32_t)min(vocab, CANDIDATES);
  if (tid == 0) { s_prefix = 0u; s_need = want; }
  __syncthreads();
  for (int shift = 24; shift >= 0; shift -= 8) {
    if (tid < 256) hist[tid] = 0u;
    __syncthreads();
    const uint32_t prefix = s_prefix;
    const uint32_t mask = shift == 24 ? 0u : (0xffffffffu << (shift + 8));
    for (int i = tid; i < vocab; i += THREADS) {
      const uint32_t k = order_key(__fdiv_rn(lg[i], T));
      if ((k & mask) == prefix) atomicAdd(&hist[(k >> shift) & 255u], 1u);
    }
    __syncthreads();
    if (tid == 0) {
      uint32_t need = s_need, b = 255u;
      for (;; --b) {                       // highest digit whose suffix count reaches `need`
        if (hist[b] >= need || b == 0u) break;
        need -= hist[b];
      }
      s_need = need;                       // how many of the ties at this digit are wanted
      s_prefix = prefix | (b << shift);
    }
    __syncthreads();
  }
  const uint32_t kth = s_prefix;           // key of the last candidate
  const uint32_t n_ties = s_need;          // how many ids with exactly that key are taken
  if (tid == 0) { s_count = 0u; s_running = 0u; }
  __syncthreads();
  for (int i = tid; i < vocab; i += THREADS) {
    const uint32_t k = order_key(__fdiv_rn(lg[i], T));
    if (k > kth) cand[atomicAdd(&s_count, 1u)] = key_and_id(k, i);
  }
  __syncthreads();
  const uint32_t n_gt = s_count;
  // ties at the threshold key: the lowest ids, found by an ordered scan over the row
  for (int base = 0; base < vocab; base += THREADS) {
    if (s_running >= n_ties) break;
    const int i = base + tid;
    const bool flag = i < vocab && order_key(__fdiv_rn(lg[i], T)) == kth;
    const uint32_t ballot = __ballot_sync(0xffffffffu, flag);
    const int lane = tid & 31, warp = tid >> 5;
    if (lane == 0) hist[warp] = __popc(ballot);
    __syncthreads();
    uint32_t before = s_running;
    for (int w = 0; w < warp; ++w) before += hist[w];
    const uint32_t rank = before + __popc(ballot & ((1u << lane) - 1u));
    if (flag && rank < n_ties) cand[n_gt + rank] = key_and_id(kth, i);
    __syncthreads();
    if (tid == 0) {
      uint32_t total = 0;
      for (int w = 0; w < THREADS / 32; ++w) total += hist[w];
      s_running += total;
    }
    __syncthreads();
  }
}

template <int CLUSTER>
__global__ void __launch_bounds__(THREADS, 2)
sample_kernel(float* logits, int vocab, const SbSampleParams* params, const int32_t* history,
              int history_stride, const int32_t* fed_pos, int32_t* out_tokens) {
  constexpr int RANK_SHARE = CANDIDATES / CLUSTER;
  static_assert(RANK_SHARE <= THREADS && CLUSTER <= MOST, "a block has a maximum a thread");
  __shared__ int32_t h_tok[MAX_HISTORY];
  __shared__ float h_old[MAX_HISTORY];
  __shared__ uint32_t hist[256];
  __shared__ __align__(16) unsigned long long cand[MAX_LIST];     // key_and_id: sorts z desc, id asc
  __shared__ unsigned long long red[32];
  __shared__ double score[CANDIDATES];
  __shared__ unsigned long long best_of[CLUSTER];
  __shared__ uint32_t s_share, s_count;
  __shared__ int s_keep;
  __shared__ double win_score[32];
  __shared__ int win_id[32];

  sb_pdl_launch();
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();                                   // every block of the cluster runs: its memory can be written
  sb_pdl_wait();
  const int row = blockIdx.x / CLUSTER, rank = blockIdx.x % CLUSTER, tid = threadIdx.x;
  // the thread's values: first, first + CLUSTER * THREADS, ...; the blocks take 32 values in turn, so that a short row
  // is shared out too
  const int first = ((tid >> 5) * CLUSTER + rank) * 32 + (tid & 31);
  SbSampleParams p = params[row];
  // with `fed_pos`, the token produced follows the one fed at fed_pos[row] in this step
  if (fed_pos) p.position = (uint64_t)fed_pos[row] + 1u;
  float* lg = logits + (size_t)row * vocab;

  // 1. penalties, in place (undone at the end).  h_tok[i] >= 0 marks a first occurrence.
  const bool penal = p.history_len > 0 && (p.repeat_penalty != 1.0f || p.presence_penalty != 0.0f ||
                                           p.frequency_penalty != 0.0f);
  const int win = penal ? min(p.history_len, MAX_HISTORY) : 0;
  if (penal) {
    const int32_t* hrow = history + (size_t)row * history_stride;
    // The blocks share the window's places out; the first one keeps what they changed.  The window lies in every block's shared
    // memory (over the candidates' list), filled up with ids that no token has.  (1,024 tokens and 152,064 greedy values, counted by one
    // block of 512 threads from memory: 8 rows 51 us, 64 rows 98; shared out 15.6 and 33.)
    int32_t* window = reinterpret_cast<int32_t*>(cand);
    int32_t* kept_tok = cluster.map_shared_rank(h_tok, 0);
    float* kept_old = cluster.map_shared_rank(h_old, 0);
    const int fours = (win + 3) / 4;
    for (int i = tid; i < 4 * fours; i += THREADS) window[i] = i < win ? hrow[i] : -1;
    __syncthreads();
    for (int i = tid * CLUSTER + rank; i < win; i += THREADS * CLUSTER) {
      const int32_t t = window[i];
      int count = 0, before = 0;                     // places of the token, those ahead of this one
      for (int j = 0; j < fours; ++j) {
        const int4 w = reinterpret_cast<const int4*>(window)[j];
        const int at = 4 * j;
        count += (w.x == t) + (w.y == t) + (w.z == t) + (w.w == t);
        before += (w.x == t && at < i) + (w.y == t && at + 1 < i) + (w.z == t && at + 2 < i) + (w.w == t && at + 3 < i);
      }
      const bool first_one = before == 0;
      kept_tok[i] = -1;
      if (first_one && t >= 0 && t < vocab) {
        const float old = lg[t];
        float v = old;
        if (p.repeat_penalty != 1.0f)
          v = v > 0.0f ? __fdiv_rn(v, p.repeat_penalty) : __fmul_rn(v, p.repeat_penalty);
        const float adjust = __fmaf_rn(p.frequency_penalty, (float)count, p.presence_penalty);
        kept_tok[i] = t;
        kept_old[i] = old;
        lg[t] = __fsub_rn(v, adjust);
      }
    }
    cluster.sync();                                  // the whole cluster reads the row as it is now
  }

  int result = -1;
  if (!(p.temperature > 0.0f)) {
    // 2. greedy (the two zeros are equal; NaN loses against everything): the group of eight values that holds the thread's
    // largest first, then its first place in the group
    constexpr int STEP = CLUSTER * THREADS, GROUP = 8;
    float top = -INFINITY;
    int group = -1;
    int at = first;
    for (; at + (GROUP - 1) * STEP < vocab; at += GROUP * STEP) {
      float v[GROUP], largest;
#pragma unroll
      for (int j = 0; j < GROUP; ++j) v[j] = lg[at + j * STEP];
      largest = v[0];
#pragma unroll
      for (int j = 1; j < GROUP; ++j) largest = fmaxf(largest, v[j]);        // passes over NaN
      if (largest > top) { top = largest; group = at; }
    }
    for (; at < vocab; at += STEP)
      if (lg[at] > top) { top = lg[at]; group = at; }
    unsigned long long best = 0ull;
    if (group >= 0) {
      while (lg[group] != top) group += STEP;
      best = key_and_id(order_key(top + 0.0f), group);
    } else {                                          // nothing above minus infinity
      for (int i = first; i < vocab; i += STEP) best = max(best, key_and_id(order_key(lg[i]), i));
    }
    best = block_max(best, red);
    if (tid == 0) *cluster.map_shared_rank(&best_of[rank], 0) = best;
    cluster.sync();
    if (rank != 0) return;
    best = 0ull;
    for (int i = 0; i < CLUSTER; ++i) best = max(best, best_of[i]);
    result = (int)(~(uint32_t)(best & 0xffffffffull));
  } else {
    // 3. the CANDIDATES highest z
    const float T = p.temperature;
    uint32_t mine = 0u;
#pragma unroll 8
    for (int i = first; i < vocab; i += CLUSTER * THREADS) mine = max(mine, order_key(lg[i]));
    if (mine != 0u) mine = order_key(__fdiv_rn(key_value(mine), T));     // the division keeps the order
    uint32_t share = 0u;                             // the RANK_SHARE-th largest of the block's maxima, its upper half
    for (int bit = 31; bit >= 16; --bit) {
      const uint32_t t = share | (1u << bit);
      if (__syncthreads_count(mine >= t) >= RANK_SHARE) share = t;
    }
    if (tid == 0) { s_share = share; s_count = 0u; }
    cluster.sync();
    for (int i = 0; i < CLUSTER; ++i) share = min(share, *cluster.map_shared_rank(&s_share, i));
    if (mine >= share) {
      uint32_t* count = cluster.map_shared_rank(&s_count, 0);
      unsigned long long* list = cluster.map_shared_rank(cand, 0);
#pragma unroll 4
      for (int i = first; i < vocab; i += CLUSTER * THREADS) {
        const uint32_t k = order_key(__fdiv_rn(lg[i], T));
        if (k < share) continue;
        const uint32_t slot = atomicAdd(count, 1u);
        if (slot < MAX_LIST) list[slot] = key_and_id(k, i);
      }
    }
    cluster.sync();
    if (rank != 0) return;
    int n = (int)min(s_count, (uint32_t)MAX_LIST + 1u);
    if (n > MAX_LIST) {
      n = min(vocab, CANDIDATES);
      select_by_radix(lg, vocab, T, cand, hist);
      __syncthreads();
    }
    // bitonic sort, descending (empty slots are 0 and sink to the end)
    int size = CANDIDATES;
    while (size < n) size <<= 1;
    for (int i = n + tid; i < size; i += THREADS) cand[i] = 0ull;
    __syncthreads();
    for (int k = 2; k <= size; k <<= 1) {
      for (int j = k >> 1; j > 0; j >>= 1) {
        for (int i = tid; i < size / 2; i += THREADS) {
          const int at = 2 * i - (i & (j - 1)), partner = at + j;
          const unsigned long long a = cand[at], b = cand[partner];
          if ((at & k) == 0 ? a < b : a > b) { cand[at] = b; cand[partner] = a; }
        }
        __syncthreads();
      }
    }
    // 4. filters: each keeps a prefix of the sorted list
    const int n_cand = min(vocab, CANDIDATES);
    const bool held = tid < n_cand;
    const float z = held ? key_value((uint32_t)(cand[tid] >> 32)) : 0.0f;
    const int id = held ? (int)(~(uint32_t)(cand[tid] & 0xffffffffull)) : -1;
    const float zmax = key_value((uint32_t)(cand[0] >> 32));
    int keep = __syncthreads_count(held && z >= zmax - LOGIT_WINDOW);
    if (p.top_k > 0u && (uint32_t)keep > p.top_k) keep = (int)p.top_k;
    if (p.min_p > 0.0f) keep = __syncthreads_count(tid < keep && z >= zmax + logf(p.min_p));
    if (p.top_p > 0.0f && p.top_p < 1.0f && keep > 0) {
      if (tid < keep) score[tid] = exp((double)z - (double)zmax);
      __syncthreads();
      if (tid == 0) {                                // the sums in ascending order
        double total = 0.0;
        for (int c = 0; c < keep; ++c) total += score[c];
        s_keep = keep;
        if (total > 0.0) {
          double acc = 0.0;
          int k2 = 0;
          while (k2 < keep) {
            acc += score[k2];
            ++k2;
            if (acc / total >= (double)p.top_p) break;
          }
          s_keep = k2 < 1 ? 1 : k2;
        }
      }
      __syncthreads();
      keep = s_keep;
    }
    // 5. Gumbel-max over the kept prefix: the highest score, ties toward the lower id
    double s = 0.0;
    int si = -1;
    if (tid < keep) {
      uint32_t bits[4];
      philox4x32_10((uint32_t)p.position, (uint32_t)(p.position >> 32), (uint32_t)id, 0u, p.seed, bits);
      const double u = ((double)bits[0] + 0.5) / 4294967296.0;
      s = (double)z + (-log(-log(u)));
      si = id;
    }
    auto better = [](double os, int oi, double s_, int i_) { return oi >= 0 && (i_ < 0 || os > s_ || (os == s_ && oi < i_)); };
    for (int o = 16; o > 0; o >>= 1) {
      const double os = __shfl_xor_sync(0xffffffffu, s, o);
      const int oi = __shfl_xor_sync(0xffffffffu, si, o);
      if (better(os, oi, s, si)) { s = os; si = oi; }
    }
    if ((tid & 31) == 0) { win_score[tid >> 5] = s; win_id[tid >> 5] = si; }
    __syncthreads();
    for (int w = 0; w < CANDIDATES / 32; ++w)
      if (better(win_score[w], win_id[w], s, si)) { s = win_score[w]; si = win_id[w]; }
    result = si;                                     // thread 0 has compared every warp's
  }

  __syncthreads();
  if (penal) {
    for (int i = tid; i < win; i += THREADS)
      if (h_tok[i] >= 0) lg[h_tok[i]] = h_old[i];
  }
  if (tid == 0) out_tokens[row] = result;
}

__global__ void add_kernel(int32_t* x, int n, int delta) {
  sb_pdl_launch();
  sb_pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] += delta;
}

// x[i] = min(x[i] + 1, last[i]): a row of a captured decode batch moves to its next position
// but never past the last position it holds pages for; a row that has finished stays there.
__global__ void advance_kernel(int32_t* x, const int32_t* __restrict__ last, int n) {
  sb_pdl_launch();
  sb_pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] = min(x[i] + 1, last[i]);
}

}  // namespace

extern "C" int sb_advance_rows(int32_t* x, const int32_t* last, int n, cudaStream_t stream) {
  if (n <= 0 || !x || !last) SB_FAIL(SB_ERR_ARG, "sb_advance_rows: n=%d", n);
  sb_launch(advance_kernel, dim3((n + 255) / 256), dim3(256), 0, stream, x, last, n);
  SB_CHECK_LAUNCH("sb_advance_rows");
  return SB_OK;
}

// x[i] += delta: advances the positions of a decode loop that stays on the device.
extern "C" int sb_add_i32(int32_t* x, int n, int delta, cudaStream_t stream) {
  if (n <= 0) SB_FAIL(SB_ERR_ARG, "sb_add_i32: n=%d", n);
  sb_launch(add_kernel, dim3((n + 255) / 256), dim3(256), 0, stream, x, n, delta);
  SB_CHECK_LAUNCH("sb_add_i32");
  return SB_OK;
}

extern "C" int sb_sample_params_size() { return (int)sizeof(SbSampleParams); }

// logits [n_rows, vocab] float32 (penalties touch it in place and restore it); params: one
// SbSampleParams per row in device memory; history [n_rows, history_stride] int32 (may be null
// when no row has history); fed_pos, when given, holds the position of the token each row was
// fed in this step and overrides the records' `position` with fed_pos + 1 (a loop that runs
// on the device advances it there); out_tokens int32 [n_rows].
extern "C" int sb_sample(float* logits, int n_rows, int vocab, const void* params,
                         const int32_t* history, int history_stride, const int32_t* fed_pos,
                         int32_t* out_tokens, cudaStream_t stream) {
  if (n_rows <= 0 || vocab <= 0) SB_FAIL(SB_ERR_ARG, "sb_sample: n_rows=%d vocab=%d", n_rows, vocab);
  if (history_stride < 0 || history_stride > MAX_HISTORY)
    SB_FAIL(SB_ERR_UNSUPPORTED, "sb_sample: a penalty window of %d tokens is above the cap of %d",
            history_stride, MAX_HISTORY);
  auto launch = [&](auto* kernel, unsigned cluster) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)n_rows * cluster);
    cfg.blockDim = dim3(THREADS);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = (sb_pdl_enabled() & SB_K_OTHER) ? 2 : 1;
    cudaLaunchKernelEx(&cfg, kernel, logits, vocab, (const SbSampleParams*)params, history, history_stride, fed_pos, out_tokens);
  };
  // Blocks a row: eight, while all rows' blocks run at once (two fit an SM) and have 4,096 values each.  A vocabulary of 152,064,
  // greedy / sampled, us, with eight blocks and with the rule's: 64 rows 14.5 / 53.8 and 7.2 / 36.3, 128 rows 31.4 / 93.1 and 11.6 / 64.7, 256 rows
  // 76.5 / 193 and 30.9 / 192; of 1,000, 32 rows 3.1 / 16.5 and 2.6 / 11.5.
  int device = 0, sms = 0;
  if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) sms = 0;
  int cluster = MOST;
  while (cluster > 1 && ((long)n_rows * cluster > 2 * sms || vocab < 4096 * cluster)) cluster /= 2;
  if (cluster == 8) launch(sample_kernel<8>, 8);
  else if (cluster == 4) launch(sample_kernel<4>, 4);
  else if (cluster == 2) launch(sample_kernel<2>, 2);
  else launch(sample_kernel<1>, 1);
  SB_CHECK_LAUNCH("sb_sample");
  return SB_OK;
}
