// Float32 attention over the paged cache for the 32-bit path: FFMA only, a block per tile of query rows of one
// key/value head of one sequence.
//
// A query row is a (token, head in group) pair, so that all query heads of a key/value head share its tiles.  Three
// forms: 16 rows (a decode step: one token's heads), 64 rows (prompts), 32 rows (prompts whose 64-row tiles leave SMs idle).
// Keys come in tiles of 64 at absolute positions.  Tile t belongs to part t % 8; every part has a running softmax of its own
// and the eight are merged in order, in every form, so a row's bits depend on its own keys and position alone: not on the
// form, and so not on the cut or on what else the step holds.  A cluster of blocks shares the parts out and merges
// them through distributed shared memory; no workspace is needed.  Its size, which changes no bit either, is the number of
// key tiles that the step's longest sequence has, up to 8 blocks for 16 rows, where a step has few blocks and the sequence is
// long, else up to 4, with two parts each, one after the other; a row that sees one tile of keys takes one block, and the others leave.
//
// What attn_plain.cu says about masks, caps, biases and sinks holds here; that kernel (a block per row and head, a
// warp per key) stays for head sizes this one does not take.  The kernel alone, us, there / here, 12/2 heads of 128: one token at 20, 64
// keys 16.4 / 7.3, 36.4 / 12.6; 256 tokens at 30 keys 73.6 / 21.0 (225 with clusters of eight whatever the length); three at 100 to 400
// 324 / 13.9; prompts of 10 in 64 sequences 69 / 17.8, of 201 183 / 24 (40 while blocks without a tile of keys stayed to the end), of
// 4,000 2,467.  8/8 heads of 256, one row a tile of 16: 256 tokens at 30 keys 105 / 184, 64 at 50 51 / 71, a sequence of 64 47 / 19.5.
#include <cooperative_groups.h>
#include <math.h>
#include <type_traits>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int THREADS = 256, KEYS = 64, LOADS = 4, PARTS = 8;

struct F32Attn {
  const float* q;
  float* out;
  const int32_t* seq_row0;
  const int32_t* seq_pos0;
  const int32_t* page_off;
  const int32_t* page_ids;
  const float* cache;
  int n_rows, max_len, page_size, n_pages, n_q_heads, n_kv_heads, hd, window, chunk, bias_len;
  float scale, softcap;
  const float* sink;
  const float* bias;
};

// TQ query rows a thread in the scores and the output (16 threads of neighbouring lanes share a row's keys or
// dimensions); head sizes up to 64 ND.
template <int TQ, int ND>
struct Form {
  static constexpr int QB = 16 * TQ;
  static constexpr int MOST = TQ == 1 ? 8 : 4, MINE = PARTS / MOST;           // blocks of a cluster, parts of a block
  static int floats(int hd) {      // queries, keys (later probabilities), values, maximum and sum, their merge
    const int kp = KEYS * (hd + 4), pp = QB * (KEYS + 4), op = QB * hd;
    const int first = kp > pp ? kp : pp;
    return QB * hd + (first > op ? first : op) + KEYS * hd + 2 * MINE * QB;
  }
};

template <int TQ, int ND>
__global__ void __launch_bounds__(THREADS, ND <= 2 ? 2 : 1)           // two blocks fit an SM's shared memory at head sizes up to 128
attn_f32_kernel(F32Attn p, int tiles_per_seq) {
  using F = Form<TQ, ND>;
  constexpr int QB = F::QB;
  extern __shared__ __align__(16) float smem[];
  const int hd = p.hd, kpitch = hd + 4, ppitch = KEYS + 4;
  float* qs = smem;
  float* ks = qs + QB * hd;
  float* ps = ks;                                       // over the keys, once the scores are made
  const int first = max(max(KEYS * kpitch, QB * ppitch), QB * hd);
  float* vs = ks + first;
  float* stat = vs + KEYS * hd;                         // maximum and sum per part and row, for the merge
  static_assert(F::MINE <= 2 && QB <= KEYS, "a block's parts lie over its keys and values");
  __shared__ int bad_values;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = blockIdx.z, tid = threadIdx.x;
  const int seq = blockIdx.x / tiles_per_seq, tile = blockIdx.x % tiles_per_seq, g = blockIdx.y;
  const int group = p.n_q_heads / p.n_kv_heads;
  // the step's plan was written before the step's first kernel, which triggers after its own wait
  // (n_rows may be less than the plan's: the caller wants its first rows)
  const int row0 = p.seq_row0[seq], n_new = min(p.seq_row0[seq + 1], p.n_rows) - row0, pos0 = p.seq_pos0[seq];
  const int pairs = n_new * group, pair0 = tile * QB;
  if (pair0 >= pairs) return;                           // the same for the whole cluster
  const int32_t* pages = p.page_ids + p.page_off[seq];
  const int held = (p.page_off[seq + 1] - p.page_off[seq]) * p.page_size;      // positions with a page

  const int tx = tid & 15, ty = tid >> 4;               // rows ty * TQ + i
  // what each of the thread's rows sees: keys lo ... pos (none where the position has no page: the row is zeros)
  int pos[TQ], lo[TQ];
  bool live[TQ];
#pragma unroll
  for (int i = 0; i < TQ; ++i) {
    const int pair = pair0 + ty * TQ + i;
    pos[i] = pos0 + pair / group;
    live[i] = pair < pairs && pos[i] >= 0 && pos[i] / p.page_size < held / p.page_size;
    lo[i] = max(p.window > 0 ? max(0, pos[i] - p.window + 1) : 0, p.chunk > 0 ? max(pos[i], 0) / p.chunk * p.chunk : 0);
  }
  // the tile's keys: from the first row's first to the last row's last
  const int first_pos = pos0 + pair0 / group, last_pos = pos0 + (min(pair0 + QB, pairs) - 1) / group;
  const int k_lo = max(p.window > 0 ? max(0, first_pos - p.window + 1) : 0,
                       p.chunk > 0 ? max(first_pos, 0) / p.chunk * p.chunk : 0);
  const int k_hi = min(min(last_pos, held - 1), p.max_len - 1);
  // Tile t_lo + i is block (t_lo + i) % splits's; `mine` is this block's first i.  Fewer blocks than MOST have no second part: there
  // are no more tiles than blocks.
  const int t_lo = k_lo / KEYS, t_hi = k_hi >= k_lo ? k_hi / KEYS : -1;
  const int splits = gridDim.z, used = min(max(t_hi - t_lo + 1, 1), splits), mine = (rank - t_lo) & (splits - 1);
  if (used == 1 && mine != 0) return;                   // a block alone meets nobody

  sb_pdl_wait();
  const int quads = hd / 4;
  if (mine < used)
  for (int i = tid; i < QB * quads; i += THREADS) {
    const int r = i / quads, c = i % quads, pair = pair0 + r;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (pair < pairs)
      v = *reinterpret_cast<const float4*>(p.q + ((size_t)(row0 + pair / group) * p.n_q_heads + g * group + pair % group) * hd + 4 * c);
    *reinterpret_cast<float4*>(qs + r * hd + 4 * c) = v;
  }

  float m[TQ], l[TQ];
  float4 acc[TQ][ND];
  // The block's parts.  The first of two is set aside in local memory (an index that the compiler does not know): kept in
  // registers, or in a copy of the loop each, it cost 4,000 tokens 13 and 10 % more.
  const bool two = F::MINE > 1 && splits == F::MOST && t_lo + mine + splits <= t_hi;
  float4 kept[F::MINE][TQ][ND];
  float2 kept_stat[F::MINE][TQ];
  int last = 0;                                         // the part whose sums are in registers
#pragma unroll 1
  for (int j = 0; j < F::MINE; ++j) {
  if (j > 0 && !two) break;
  last = j;
#pragma unroll
  for (int i = 0; i < TQ; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.0f;
#pragma unroll
    for (int d = 0; d < ND; ++d) acc[i][d] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
  for (int t = t_lo + mine + j * splits; t <= t_hi; t += PARTS) {
    const int base = t * KEYS, n_keys = min(KEYS, k_hi - base + 1);     // the rest of the tile is neither loaded nor looked at
    const int load = (n_keys + 15) / 16 * 16 * quads;
    __syncthreads();                                    // the tile before this one has been read
    if (tid == 0) bad_values = 0;
    __syncthreads();
    bool bad = false;
    // LOADS keys' and values' 16 bytes a thread at once: one after the other they were most of a decode step's time
    for (int i0 = tid; i0 < load; i0 += LOADS * THREADS) {
      float4 kv[LOADS], vv[LOADS];
      int page[LOADS];
#pragma unroll
      for (int u = 0; u < LOADS; ++u) {
        const int i = i0 + u * THREADS, j = base + i / quads;
        page[u] = i < load && j >= k_lo && j <= k_hi ? pages[j / p.page_size] : -1;
      }
#pragma unroll
      for (int u = 0; u < LOADS; ++u) {
        const int i = i0 + u * THREADS, j = base + i / quads, c = i % quads;
        kv[u] = vv[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (page[u] >= 0 && page[u] < p.n_pages) {
          const float* at = p.cache + (((size_t)page[u] * 2 * p.n_kv_heads + g) * p.page_size + j % p.page_size) * hd + 4 * c;
          kv[u] = *reinterpret_cast<const float4*>(at);
          vv[u] = *reinterpret_cast<const float4*>(at + (size_t)p.n_kv_heads * p.page_size * hd);
        }
      }
#pragma unroll
      for (int u = 0; u < LOADS; ++u) {
        const int i = i0 + u * THREADS, r = i / quads, c = i % quads;
        if (i >= load) continue;
        *reinterpret_cast<float4*>(ks + r * kpitch + 4 * c) = kv[u];
        *reinterpret_cast<float4*>(vs + r * hd + 4 * c) = vv[u];
        const float s = fabsf(vv[u].x) + fabsf(vv[u].y) + fabsf(vv[u].z) + fabsf(vv[u].w);
        bad |= !(s < INFINITY);
      }
    }
    if (bad) bad_values = 1;
    __syncthreads();

    // scores: rows ty * TQ + i, keys tx + 16 j
    float s[TQ][4] = {};
    auto scores = [&](auto columns) {                   // of the first 16 `columns` keys
      constexpr int NJ = decltype(columns)::value;
      for (int c = 0; c < quads; ++c) {
        float4 kq[NJ];
#pragma unroll
        for (int j = 0; j < NJ; ++j) kq[j] = *reinterpret_cast<const float4*>(ks + (tx + 16 * j) * kpitch + 4 * c);
#pragma unroll
        for (int i = 0; i < TQ; ++i) {
          const float4 qv = *reinterpret_cast<const float4*>(qs + (ty * TQ + i) * hd + 4 * c);
#pragma unroll
          for (int j = 0; j < NJ; ++j) {
            s[i][j] = fmaf(qv.x, kq[j].x, s[i][j]);
            s[i][j] = fmaf(qv.y, kq[j].y, s[i][j]);
            s[i][j] = fmaf(qv.z, kq[j].z, s[i][j]);
            s[i][j] = fmaf(qv.w, kq[j].w, s[i][j]);
          }
        }
      }
    };
    if (TQ == 1 && n_keys <= 32) scores(std::integral_constant<int, 2>());
    else scores(std::integral_constant<int, 4>());
    __syncthreads();                                    // the keys have been read: the probabilities take their place
#pragma unroll
    for (int i = 0; i < TQ; ++i) {
      float tile_max = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = base + tx + 16 * j;
        float v = s[i][j] * p.scale;
        if (p.softcap > 0.0f) v = p.softcap * tanhf(v / p.softcap);
        const bool sees = live[i] && key >= lo[i] && key <= pos[i];
        if (p.bias && sees) {
          const int h = g * group + (pair0 + ty * TQ + i) % group;
          v += p.bias[(size_t)h * p.bias_len + min(pos[i] - key, p.bias_len - 1)];
        }
        s[i][j] = sees ? v : -INFINITY;
        tile_max = fmaxf(tile_max, s[i][j]);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, o));
      const float m_new = fmaxf(m[i], tile_max);
      float sum = 0.0f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float e = s[i][j] == -INFINITY ? 0.0f : expf(s[i][j] - m_new);
        ps[(ty * TQ + i) * ppitch + tx + 16 * j] = e;
        sum += e;
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      const float alpha = m[i] == -INFINITY ? 0.0f : expf(m[i] - m_new);
      l[i] = l[i] * alpha + sum;
      m[i] = m_new;
#pragma unroll
      for (int d = 0; d < ND; ++d) {
        acc[i][d].x *= alpha; acc[i][d].y *= alpha; acc[i][d].z *= alpha; acc[i][d].w *= alpha;
      }
    }
    __syncwarp();                                       // a row's probabilities are read by the lanes that wrote them
    // output: rows ty * TQ + i, dimensions tx * 4 + 64 d.  A value that is not finite must not reach rows that do not
    // see its key, so a tile that holds one takes the keys one by one.
    const bool check = bad_values != 0;
    for (int k4 = 0; k4 < n_keys; k4 += 4) {
      float4 pr[TQ];
#pragma unroll
      for (int i = 0; i < TQ; ++i) pr[i] = *reinterpret_cast<const float4*>(ps + (ty * TQ + i) * ppitch + k4);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
#pragma unroll
        for (int d = 0; d < ND; ++d) {
          if (tx * 4 + 64 * d >= hd) continue;
          const float4 v = *reinterpret_cast<const float4*>(vs + (k4 + c) * hd + tx * 4 + 64 * d);
#pragma unroll
          for (int i = 0; i < TQ; ++i) {
            const float w = c == 0 ? pr[i].x : c == 1 ? pr[i].y : c == 2 ? pr[i].z : pr[i].w;
            if (check) {
              const int key = base + k4 + c;
              if (!(live[i] && key >= lo[i] && key <= pos[i])) continue;
            }
            acc[i][d].x = fmaf(w, v.x, acc[i][d].x);
            acc[i][d].y = fmaf(w, v.y, acc[i][d].y);
            acc[i][d].z = fmaf(w, v.z, acc[i][d].z);
            acc[i][d].w = fmaf(w, v.w, acc[i][d].w);
          }
        }
      }
    }
  }
  if (two && j == 0) {
#pragma unroll
    for (int i = 0; i < TQ; ++i) {
      kept_stat[j][i] = make_float2(m[i], l[i]);
#pragma unroll
      for (int d = 0; d < ND; ++d) kept[j][i][d] = acc[i][d];
    }
  }
  }

  // merge: every block leaves its parts' sums over its keys' space, then takes a share of the rows
  sb_pdl_launch();
  __syncthreads();
  float* os = ks;
  auto leave = [&](int j, const float4 (&sums)[TQ][ND], auto stat_of) {
#pragma unroll
    for (int i = 0; i < TQ; ++i) {
      const int r = j * QB + ty * TQ + i;
#pragma unroll
      for (int d = 0; d < ND; ++d)
        if (tx * 4 + 64 * d < hd) *reinterpret_cast<float4*>(os + r * hd + tx * 4 + 64 * d) = sums[i][d];
      if (tx == 0) *reinterpret_cast<float2*>(stat + 2 * r) = stat_of(i);
    }
  };
  if (mine < used) leave(last, acc, [&](int i) { return make_float2(m[i], l[i]); });
  if (two) leave(0, kept[last - 1], [&](int i) { return kept_stat[last - 1][i]; });
  // part s begins with tile t_lo + i and is the (i / splits)-th of block s % splits (i beyond the last tile: the part is empty)
  auto begins = [&](int s) { return (s - t_lo) & (PARTS - 1); };
  auto holds = [&](int s) { return t_lo + begins(s) <= t_hi; };
  auto row_of = [&](int s, int r) { return (begins(s) >= splits ? QB : 0) + r; };
  if (used > 1) cluster.sync();
  else __syncthreads();
  const int share = (QB + used - 1) / used;
  for (int r = mine * share + ty; r < min((mine + 1) * share, QB); r += 16) {
    const int pair = pair0 + r;
    if (pair >= pairs) continue;
    const int h = g * group + pair % group, at = pos0 + pair / group;
    const bool row_live = at >= 0 && at / p.page_size < held / p.page_size;
    float2 st[PARTS];
#pragma unroll
    for (int s = 0; s < PARTS; ++s)
      st[s] = holds(s) ? *reinterpret_cast<const float2*>(cluster.map_shared_rank(stat, s & (splits - 1)) + 2 * row_of(s, r))
                       : make_float2(-INFINITY, 0.0f);
    float m_all = p.sink ? p.sink[h] : -INFINITY, total = 0.0f;
#pragma unroll
    for (int s = 0; s < PARTS; ++s) m_all = fmaxf(m_all, st[s].x);
    float f[PARTS];
#pragma unroll
    for (int s = 0; s < PARTS; ++s) {
      f[s] = st[s].x == -INFINITY ? 0.0f : expf(st[s].x - m_all);
      total += st[s].y * f[s];
    }
    if (p.sink) total += expf(p.sink[h] - m_all);
    const float inv = 1.0f / total;
    float* to = p.out + ((size_t)(row0 + pair / group) * p.n_q_heads + h) * hd;
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      const int at_d = tx * 4 + 64 * d;
      if (at_d >= hd) continue;
      float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (row_live) {
#pragma unroll
        for (int s = 0; s < PARTS; ++s) {
          float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if (holds(s))
            v = *reinterpret_cast<const float4*>(cluster.map_shared_rank(os, s & (splits - 1)) + row_of(s, r) * hd + at_d);
          o.x = fmaf(v.x, f[s], o.x); o.y = fmaf(v.y, f[s], o.y); o.z = fmaf(v.z, f[s], o.z); o.w = fmaf(v.w, f[s], o.w);
        }
        o.x *= inv; o.y *= inv; o.z *= inv; o.w *= inv;
      }
      *reinterpret_cast<float4*>(to + at_d) = o;
    }
  }
  if (used > 1) cluster.sync();                         // nobody's sums go while another block reads them
}

template <int TQ, int ND>
int launch(const F32Attn& p, int n_seqs, int max_new, cudaStream_t stream) {
  using F = Form<TQ, ND>;
  const int group = p.n_q_heads / p.n_kv_heads;
  const int tiles = (int)(((long)max_new * group + F::QB - 1) / F::QB);
  const size_t smem = (size_t)F::floats(p.hd) * sizeof(float);
  if (cudaError_t e = cudaFuncSetAttribute(attn_f32_kernel<TQ, ND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           F::floats(64 * ND) * (int)sizeof(float)))
    SB_FAIL(SB_ERR_CUDA, "sb_attention_f32: %s", cudaGetErrorString(e));
  cudaLaunchConfig_t cfg = {};
  const int key_tiles = (p.max_len + KEYS - 1) / KEYS;
  int splits = 1;
  while (splits < key_tiles && splits < F::MOST) splits *= 2;
  cfg.gridDim = dim3((unsigned)n_seqs * (unsigned)tiles, p.n_kv_heads, splits);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = splits;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (sb_pdl_enabled() & SB_K_OTHER) ? 2 : 1;
  cudaLaunchKernelEx(&cfg, attn_f32_kernel<TQ, ND>, p, tiles);
  SB_CHECK_LAUNCH("sb_attention_f32");
  return SB_OK;
}

}  // namespace

int sb_check_attention_args(const char* who, int n_rows, int n_q_heads, int n_kv_heads, int hd, int window, int page_size);

extern "C" int sb_attention_f32(const float* q, float* out, int n_rows, int n_seqs, int max_new, int max_len, const int32_t* seq_row0,
                                const int32_t* seq_pos0, const int32_t* page_off, const int32_t* page_ids, int page_size,
                                const float* cache, int n_pages, int n_q_heads, int n_kv_heads, int hd, int window,
                                float scale, const float* sink, float softcap, int chunk, const float* bias, int bias_len,
                                int n_sms, cudaStream_t stream) {
  if (chunk < 0 || (bias && bias_len < 1))
    SB_FAIL(SB_ERR_ARG, "sb_attention_f32: chunk %d, a distance bias of %d entries", chunk, bias_len);
  if (softcap < 0.0f) SB_FAIL(SB_ERR_ARG, "sb_attention_f32: score cap %g (0: none)", softcap);
  if (int rc = sb_check_attention_args("sb_attention_f32", n_rows, n_q_heads, n_kv_heads, hd, window, page_size)) return rc;
  if (n_seqs <= 0 || max_new <= 0 || max_len <= 0)
    SB_FAIL(SB_ERR_ARG, "sb_attention_f32: %d sequences, at most %d new rows and %d positions", n_seqs, max_new, max_len);
  if (hd % 4 || hd > 256 || n_kv_heads > 65535)
    SB_FAIL(SB_ERR_UNSUPPORTED, "sb_attention_f32: head size %d (a multiple of 4 up to 256), %d key/value heads", hd, n_kv_heads);
  const F32Attn p{q, out, seq_row0, seq_pos0, page_off, page_ids, cache, n_rows, max_len, page_size, n_pages, n_q_heads, n_kv_heads, hd, window,
                  chunk, bias_len, scale, softcap, sink, bias};
  if (n_sms <= 0) SB_FAIL(SB_ERR_ARG, "sb_attention_f32: %d SMs", n_sms);
  // one token's heads fit the 16-row form; a row of a longer stretch sees up to 64 rows' keys loaded once, or 32 where 64
  // leave SMs idle (a prompt of 201 tokens: 38 tiles of 64 rows, 152 blocks with a tile of keys each, or 304 with half the work)
  const long rows = (long)max_new * (n_q_heads / n_kv_heads), tiles = (rows + 63) / 64 * n_kv_heads * n_seqs;
#define SB_F32_FORMS(ND)                                              \
  if (rows <= 16) return launch<1, ND>(p, n_seqs, max_new, stream);   \
  if (2 * tiles < n_sms) return launch<2, ND>(p, n_seqs, max_new, stream); \
  return launch<4, ND>(p, n_seqs, max_new, stream);
  if (hd <= 64) { SB_F32_FORMS(1) }
  if (hd <= 128) { SB_F32_FORMS(2) }
  SB_F32_FORMS(4)
#undef SB_F32_FORMS
}
