// Attention over the paged cache for any batch of tokens: one block per
// (token, query head).  It serves the float32 path and every size the tiled
// bfloat16 kernels do not take.  A token at position p sees the keys at
// positions lo..p of its own request, lo = max(0, p - window + 1) with a
// window and 0 without, wherever the pages lie
// (python/helios/exec/paged_attn.py:264-295, 368-408; GQA mapping :248-261).
//
// Options, each off by default: values of another size than the keys (`vd`); a bias on the
// score that grows with the distance, score - slopes[h] * (p - j); a bias looked up by the
// distance, score + bias_table[min(p - j, bias_rows - 1), h]; first tokens that a window
// keeps (`keep_first`: j visible if j <= p and (p - j < window or j < keep_first)); a sink in
// the softmax, a key without a value whose score is 0 or sink_values[h], so that the weights
// are exp(s_j) / (exp(sink) + sum exp(s_j)); a gate per (token, head), the head's output times
// sigmoid(gate[t, h]), or per output value (`gate_wide`: gate[t, h * vd + d]); means of whole blocks
// of `pool` tokens behind the window (`pooled`: a key and a value a block in pages of their own,
// block b seen if (b + 1) * pool <= p - window + 1); a constant `factor` on the output.
//
// Scores, softmax and the weighted sum are float32.  The keys are walked in runs of 32 from
// `lo`; the runs are dealt to the block's eight warps in turn, and the warps' sums are merged
// in order, so the order of every sum depends on the token's position alone: not on how the
// request was cut into steps, nor on the rest of the batch.
//
// Bound by the latency of its loads: a decode step has a few dozen rows of some hundred keys.
// So a row has a block of eight warps where its keys make as many runs (below: SHARE), and a run's loads are independent: eight lanes share a
// key (four elements a lane and load, the key's dot product finished by three shuffles), a
// warp's four groups of eight lanes walk eight keys of the run each, and values the same way.
// In chains, 14 heads of 64 on 2 KV heads, float32, one warp a row with a key a lane / this:
// 3 decode rows of 313 keys 132 / 8.1 µs, 24 of 1,000 420 / 29, one of 4,096 1,676 / 49;
// prompts of 37, 128 and 301 tokens 345 / 99, one of 2,048 8,646 / 1,455.
#include "common.cuh"

// Keys and values that stand for whole blocks of tokens; all null / 0: none.
template <typename T>
struct PooledPages {
  const T* k;             // [page, kv head, slot, hd]
  const T* v;             // [page, kv head, slot, vd]
  const int* table;       // [requests, table_stride]
  int table_stride;
  int pool;
};

constexpr int ATTN_WARPS = 8;
constexpr int ATTN_MAX_HD = 256;

// four neighbouring elements of a row of `n`, as float; zeros behind its end
template <typename T, bool VEC>
__device__ __forceinline__ float4 load_four(const T* row, int d, int n) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if constexpr (VEC) {
    if (d < n) {
      if constexpr (sizeof(T) == 4) {
        v = *reinterpret_cast<const float4*>(row + d);
      } else {
        const uint2 raw = *reinterpret_cast<const uint2*>(row + d);
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
        const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
        v = make_float4(a.x, a.y, b.x, b.y);
      }
    }
  } else {
    if (d < n) v.x = to_float(row[d]);
    if (d + 1 < n) v.y = to_float(row[d + 1]);
    if (d + 2 < n) v.z = to_float(row[d + 2]);
    if (d + 3 < n) v.w = to_float(row[d + 3]);
  }
  return v;
}

// NJ: 32 * NJ >= hd, vd.  VEC: rows of keys and values are whole 4-element pieces.
// SHARE: a token whose keys make one, two or three to four runs has 8, 4 or 2 of its heads in one block,
// with 1, 2 or 4 warps each, and the blocks of the other heads end at once (the position is on the
// device).  The sums are the same ones in the same order.  A row of at most 32 keys alone keeps one warp of
// eight, and two blocks fit an SM.  14 heads of 64 on 2 KV heads, float32, a block a row / shared, µs: 67 prompts
// of 30 tokens 347 / 67, 2,048 tokens with a window of 16 356 / 69 and of 128 383 / 236, 600 decode rows of 30
// keys 116 / 25; but 600 of 250 keys 223 / 246 (half a microsecond a block until the position is there
// and the warps are dealt), and one row of 30 5.6 / 6.1.  So it is for launches of many rows that may be short.
// AHEAD: for launches of at most a block an SM.  All keys and values of a run are asked for at once, before its
// scores: one trip to memory a run instead of four, for registers that leave an SM one block.  14 heads of 64 on 2 KV
// heads, float32, µs: 3 rows of 20 keys 4.6 / 3.7, of 313 7.8 / 6.2, of 4,096 49 / 36; 10 of 1,000 14.9 / 11.0.  Heads
// of at most 32 values have all of it under way as it is (5.56 / 5.60), and of 128 it does not fit the registers.
template <typename T, int NJ, bool VEC, bool SHARE, bool AHEAD>
__global__ void __launch_bounds__(ATTN_WARPS * 32) attention_generic_kernel(
    T* __restrict__ out, const T* __restrict__ q, int q_stride,
    const T* __restrict__ k_pages, const T* __restrict__ v_pages,
    const int* __restrict__ block_table, int bt_stride, const int* __restrict__ seq_of_token,
    const int* __restrict__ positions, int head_blocks, int head_step, int nh, int nkv, int hd, int vd, int page_size,
    int window, float scale, const float* __restrict__ slopes, int sink,
    const T* __restrict__ gate, int gate_stride, const float* __restrict__ bias_table, int bias_rows,
    const float* __restrict__ sink_values, int keep_first, int gate_wide, PooledPages<T> pooled,
    int out_stride, float factor) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float part_acc[ATTN_WARPS][32 * NJ];
  __shared__ float part_m[ATTN_WARPS], part_l[ATTN_WARPS];
  constexpr int KEYS = AHEAD ? 8 : NJ <= 4 ? 8 / NJ : 1;     // keys a group has in flight: eight loads a lane
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = lane >> 3, gl = lane & 7;
  const int t = blockIdx.x / head_blocks;
  int h = (blockIdx.x - t * head_blocks) * head_step, kvh = h / (nh / nkv);
  const int pos = positions[t];
  const int* token_table = block_table + (size_t)seq_of_token[t] * bt_stride;
  const int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;

  // this lane's pieces of a row: elements 4 (8 j + gl) .. + 3
  float4 qr[NJ], acc[NJ];
  auto load_query = [&] {
    const T* qrow = q + (size_t)t * q_stride + (size_t)h * hd;
#pragma unroll
    for (int j = 0; j < NJ; ++j) qr[j] = load_four<T, false>(qrow, 4 * (8 * j + gl), hd);
  };
  int wpr = ATTN_WARPS;                                // warps of a row
  if constexpr (SHARE) {
    if constexpr (NJ == 8) load_query();               // (while the position is on its way; smaller heads are slower so)
    const int total = (pos - lo) / 32 + 1 + (min(keep_first, lo) + 31) / 32 +
                      (pooled.pool > 0 ? (lo / pooled.pool + 31) / 32 : 0);
    wpr = total <= 1 ? 1 : total <= 2 ? 2 : total <= 4 ? 4 : ATTN_WARPS;
    if (h & (ATTN_WARPS / wpr - 1)) return;            // another block has this head
    if (wpr < ATTN_WARPS) {
      h += warp / wpr;
      if (h >= nh) return;
      kvh = h / (nh / nkv);
      if constexpr (NJ == 8) load_query();
    }
    if constexpr (NJ < 8) load_query();
  } else {
    load_query();
  }
  const int part = warp & (wpr - 1), row_warp = warp - part;
#pragma unroll
  for (int j = 0; j < NJ; ++j) acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
  float m = -INFINITY, l = 0.f;
  const float slope = slopes ? slopes[h] : 0.f;

  // three stretches of keys: the means of the blocks behind the window, the first tokens a
  // window keeps (those it has passed), then the window itself; each in runs of 32 from its own
  // first key
  int run = 0;                                         // runs of the row so far
  for (int stretch = pooled.pool > 0 ? -1 : 0; stretch < 2; ++stretch) {
    const int first = stretch <= 0 ? 0 : lo;
    const int last = stretch < 0 ? lo / pooled.pool - 1 : stretch == 0 ? min(keep_first, lo) - 1 : pos;
    const int* table = stretch < 0 ? pooled.table + (size_t)seq_of_token[t] * pooled.table_stride : token_table;
    const T* kp = stretch < 0 ? pooled.k : k_pages;
    const T* vp = stretch < 0 ? pooled.v : v_pages;
    const int runs = last >= first ? (last - first) / 32 + 1 : 0;
    for (int r = (part - run % ATTN_WARPS + ATTN_WARPS) % ATTN_WARPS; r < runs; r += ATTN_WARPS) {
      const int base = first + 32 * r;
      const int key = base + lane;
      const bool valid = key <= last;
      // the key's place in the pages, in rows
      size_t place = 0;
      if (valid) place = ((size_t)table[key / page_size] * nkv + kvh) * page_size + key % page_size;
      float score = -INFINITY;
      float4 values[AHEAD ? 8 : 1][NJ];
#pragma unroll 1
      for (int i0 = 0; i0 < 8; i0 += KEYS) {           // the group's keys 8 group + i
        float4 kv[KEYS][NJ];
#pragma unroll
        for (int u = 0; u < KEYS; ++u) {
          const size_t at = __shfl_sync(0xffffffffu, (unsigned long long)place, 8 * group + i0 + u);
          const int n = base + 8 * group + i0 + u <= last ? hd : 0;
#pragma unroll
          for (int j = 0; j < NJ; ++j) kv[u][j] = load_four<T, VEC>(kp + at * hd, 4 * (8 * j + gl), n);
        }
        if constexpr (AHEAD) {
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const size_t at = __shfl_sync(0xffffffffu, (unsigned long long)place, 8 * group + u);
            const int n = base + 8 * group + u <= last ? vd : 0;
#pragma unroll
            for (int j = 0; j < NJ; ++j) values[u][j] = load_four<T, VEC>(vp + at * vd, 4 * (8 * j + gl), n);
          }
        }
#pragma unroll
        for (int u = 0; u < KEYS; ++u) {
          float dot = 0.f;
#pragma unroll
          for (int j = 0; j < NJ; ++j) {
            dot = fmaf(qr[j].x, kv[u][j].x, dot);
            dot = fmaf(qr[j].y, kv[u][j].y, dot);
            dot = fmaf(qr[j].z, kv[u][j].z, dot);
            dot = fmaf(qr[j].w, kv[u][j].w, dot);
          }
          dot += __shfl_xor_sync(0xffffffffu, dot, 1);
          dot += __shfl_xor_sync(0xffffffffu, dot, 2);
          dot += __shfl_xor_sync(0xffffffffu, dot, 4);
          if (gl == i0 + u) score = dot;
        }
      }
      if (valid) {
        score = score * scale - slope * (float)(pos - key);
        if (bias_table) score += bias_table[(size_t)min(pos - key, bias_rows - 1) * nh + h];
      } else {
        score = -INFINITY;
      }
      const float m_new = fmaxf(m, warp_max(score));
      const float p = score == -INFINITY ? 0.f : expf(score - m_new);
      const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
      l = l * corr + warp_sum(p);
      m = m_new;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        acc[j].x *= corr;
        acc[j].y *= corr;
        acc[j].z *= corr;
        acc[j].w *= corr;
      }
#pragma unroll 1
      for (int i0 = 0; i0 < 8; i0 += KEYS) {
        float4 kv[KEYS][NJ];
        float pj[KEYS];
#pragma unroll
        for (int u = 0; u < KEYS; ++u) {
          pj[u] = __shfl_sync(0xffffffffu, p, 8 * group + i0 + u);
          if constexpr (AHEAD) {
#pragma unroll
            for (int j = 0; j < NJ; ++j) kv[u][j] = values[u][j];
          } else {
            const size_t at = __shfl_sync(0xffffffffu, (unsigned long long)place, 8 * group + i0 + u);
            const int n = base + 8 * group + i0 + u <= last ? vd : 0;
#pragma unroll
            for (int j = 0; j < NJ; ++j) kv[u][j] = load_four<T, VEC>(vp + at * vd, 4 * (8 * j + gl), n);
          }
        }
#pragma unroll
        for (int u = 0; u < KEYS; ++u)
#pragma unroll
          for (int j = 0; j < NJ; ++j) {
            acc[j].x = fmaf(pj[u], kv[u][j].x, acc[j].x);
            acc[j].y = fmaf(pj[u], kv[u][j].y, acc[j].y);
            acc[j].z = fmaf(pj[u], kv[u][j].z, acc[j].z);
            acc[j].w = fmaf(pj[u], kv[u][j].w, acc[j].w);
          }
      }
    }
    run += runs;
  }

  // the four groups' sums, then the warps' in order
  auto groups_sum = [](float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    return v + __shfl_xor_sync(0xffffffffu, v, 16);
  };
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const float4 a = make_float4(groups_sum(acc[j].x), groups_sum(acc[j].y), groups_sum(acc[j].z), groups_sum(acc[j].w));
    if (group == 0) *reinterpret_cast<float4*>(&part_acc[warp][4 * (8 * j + gl)]) = a;
  }
  if (lane == 0) { part_m[warp] = m; part_l[warp] = l; }
  __syncthreads();
  m = -INFINITY;
#pragma unroll
  for (int w = 0; w < ATTN_WARPS; ++w)
    if (w < wpr) m = fmaxf(m, part_m[row_warp + w]);
  for (int d = threadIdx.x - 32 * row_warp; d < vd; d += 32 * wpr) {
    l = 0.f;
    float y = 0.f;
#pragma unroll
    for (int w = 0; w < ATTN_WARPS; ++w) {
      if (w >= run) break;                             // the warps behind the last run have seen no key
      const float pm = part_m[row_warp + w], f = pm == -INFINITY ? 0.f : expf(pm - m);
      l = fmaf(part_l[row_warp + w], f, l);
      y = fmaf(part_acc[row_warp + w][d], f, y);
    }
    if (sink) {                     // a key without a value: it adds exp(s - m) to the sum only (s = 0 unless given)
      const float sv = sink_values ? sink_values[h] : 0.f;
      const float m_new = fmaxf(m, sv);
      const float corr = expf(m - m_new);
      l = l * corr + expf(sv - m_new);
      y *= corr;
    }
    float inv = factor / l;
    if (gate && !gate_wide) inv /= 1.f + expf(-to_float(gate[(size_t)t * gate_stride + h]));
    y *= inv;
    if (gate && gate_wide) y /= 1.f + expf(-to_float(gate[(size_t)t * gate_stride + (size_t)h * vd + d]));
    out[(size_t)t * out_stride + (size_t)h * vd + d] = from_float<T>(y);
  }
}

HB_EXPORT int hb_attention_generic(void* out, const void* q, int q_stride, const void* k_pages,
                                   const void* v_pages, const int* block_table, int bt_stride,
                                   const int* seq_of_token, const int* positions, int T, int nh,
                                   int nkv, int hd, int vd, int page_size, int window, float scale,
                                   const float* slopes, int sink, const void* gate,
                                   int gate_stride, const float* bias_table, int bias_rows,
                                   const float* sink_values, int keep_first, int gate_wide,
                                   const void* pooled_k, const void* pooled_v, const int* pooled_table,
                                   int pooled_table_stride, int pool, int out_stride, float factor, int act_dt,
                                   int sms, cudaStream_t stream) {
  if (T <= 0) return HB_OK;
  if (hd <= 0 || hd > ATTN_MAX_HD || vd <= 0 || vd > ATTN_MAX_HD || nkv <= 0 || nh % nkv != 0 ||
      page_size <= 0 || keep_first < 0 || pool < 0 || out_stride < nh * vd ||
      (pool > 0 && (window <= 0 || !pooled_k || !pooled_v || !pooled_table)) || (bias_table != nullptr && bias_rows <= 0))
    return HB_BAD_ARGUMENT;
  if ((long)T * nh > 0x7fffffffL) return HB_BAD_ARGUMENT;
  const int most = hd > vd ? hd : vd;
  // The runs of keys a row can have, as far as the arguments say: by the window, or the table's width
  // (in a captured step that is what a request may grow to, so that many rows may be short all the same).
  // Up to four, the heads that share a block are known here, and the others get no blocks.
  const long keys_of_table = (long)bt_stride * page_size;
  long keys = keys_of_table;
  if (window > 0 && window < keys) keys = window;
  long runs = (keys + 31) / 32 + (window > 0 ? (keep_first + 31) / 32 : 0);
  if (pool > 0) runs += ((long)pooled_table_stride * page_size + 31) / 32;
  const long rows = (long)T * nh;
  const bool share = runs <= 4 ? rows > 2L * sms : rows > 8L * sms && (window <= 0 || window >= keys_of_table);
  const int head_step = !share ? 1 : runs <= 1 ? 8 : runs <= 2 ? 4 : runs <= 4 ? 2 : 1;
  const int head_blocks = (nh + head_step - 1) / head_step;
#define HB_GENERIC_SHARE(NJ, VEC, SHARE, AHEAD)                                                                       \
    hb_launch(attention_generic_kernel<TA, NJ, VEC, SHARE, AHEAD>, dim3((unsigned)(T * head_blocks)),                 \
        dim3(ATTN_WARPS * 32), 0, stream,                                                                      \
        (TA*)out, (const TA*)q, q_stride, (const TA*)k_pages, (const TA*)v_pages, block_table,                 \
        bt_stride, seq_of_token, positions, head_blocks, head_step, nh, nkv, hd, vd, page_size, window, scale, \
        slopes, sink, (const TA*)gate, gate_stride, bias_table, bias_rows, sink_values, keep_first,            \
        gate_wide,                                                                                             \
        PooledPages<TA>{(const TA*)pooled_k, (const TA*)pooled_v, pooled_table, pooled_table_stride, pool},    \
        out_stride, factor)
#define HB_GENERIC_LAUNCH(NJ, VEC)                                                                             \
    do {                                                                                                       \
      constexpr bool MAY = VEC && NJ == 2;                                                                     \
      if (share) HB_GENERIC_SHARE(NJ, VEC, true, false);                                                       \
      else if (MAY && rows <= sms) HB_GENERIC_SHARE(NJ, VEC, false, MAY);                                      \
      else HB_GENERIC_SHARE(NJ, VEC, false, false);                                                            \
    } while (0)
  HB_DISPATCH_DTYPE(act_dt, TA,
    const uintptr_t addresses = reinterpret_cast<uintptr_t>(k_pages) | reinterpret_cast<uintptr_t>(v_pages) |
                                (pool > 0 ? reinterpret_cast<uintptr_t>(pooled_k) | reinterpret_cast<uintptr_t>(pooled_v) : 0);
    const bool vec = hd % 4 == 0 && vd % 4 == 0 && addresses % (4 * sizeof(TA)) == 0;
    if (!vec) HB_GENERIC_LAUNCH(8, false);
    else if (most <= 32) HB_GENERIC_LAUNCH(1, true);
    else if (most <= 64) HB_GENERIC_LAUNCH(2, true);
    else if (most <= 128) HB_GENERIC_LAUNCH(4, true);
    else HB_GENERIC_LAUNCH(8, true));
#undef HB_GENERIC_LAUNCH
#undef HB_GENERIC_SHARE
  return hb_check_launch();
}
