// The recurrence of `delta_rule.cu` for 16-bit activations and portions of many tokens, sixteen tokens (a
// chunk) at a time.  With c_i = g_1 .. g_i (products of the decays from the chunk's first token on) and
// S the state before the chunk, the writes of a chunk are the solution of a triangular system:
//
//   u_i = beta_i (v_i - S^T (c_i k_i) - sum_{j<i} A_ij u_j),   A_ij = sum_d k_i k_j g_{j+1} .. g_i
//   U   = T (V - S^T Kc),                                      T = (I + diag(beta) A)^-1 diag(beta)
//   o_i = S^T (c_i q_i) + sum_{j<=i} B_ij u_j,                 B_ij = sum_d q_i k_j g_{j+1} .. g_i
//   S   = g_1 .. g_16 (.) S + sum_j (k_j g_{j+1} .. g_16) u_j
//
// so that the only chain left is one of chunks: `delta_chunk_prepare` makes Kc, Qc, the keys of the last
// line, T and B for all chunks side by side, and `delta_chunk` walks a request's chunks with three small
// products each.  No decay is ever divided by: every product of decays is a product.
//
// The products with S run on mma.sync in bfloat16, each float32 factor as the sum of three bfloat16 values
// (x = x0 + x1 + x2, exact: 24 bits are 3 x 8), so six products of a pair (those below 2^-24 of the whole
// are left out), by size in accumulators of their own: the large one holds products of 16 bits, which its
// 24 take nearly without rounding.  S itself is float32 and takes two fused multiply-adds a chunk instead of
// two roundings a token.  A sum of a chunk has roundings that the walk by tokens has not, so what costs little is
// made better than there: 1 / |k|, 1 / |q|, k . q and beta in 64 bits (a unit vector's element is rounded once), the
// decays' rate as the sum of two, and the term of a token's own write, mostly the largest of its sum, is added last
// (into o, u and, for a chunk's last token, S): 7 of 180 µs.  Errors against 64 bits, 2,048 tokens of 128 x 128,
// relative 2-norms in e-7, walk by tokens / this, where the decays are 0.02, 0.46, 0.82, 0.995 and 0.9999 on average:
// after silu outputs 1.31 / 0.50, 1.30 / 0.63, 1.28 / 0.87, 6.46 / 6.39, 24.1 / 18.9, states 0.73 / 0.50, 0.86 / 0.73,
// 1.25 / 1.02, 8.69 / 8.29, 30.6 / 23.7; normal inputs, 0.02 and 0.82: outputs 1.46 / 0.51, 1.67 / 1.21, states 0.70 /
// 0.50, 1.22 / 1.05, and without those measures 1.63, 1.85 and 0.90, 1.21.  Keys that are alike (a cosine of 0.8), dk
// of 24: 0.98 to 1.06 of the walk's.  TF32 and its rest instead, three products: 1.5 to 2.1.
// 32-bit activations keep the walk by tokens, whose numbers do not depend on how a prompt was cut.
#pragma once
#include "common.cuh"

constexpr int DC_TOKENS = 16;       // tokens of a chunk
constexpr int DC_COLS = 16;         // columns of S a group of warps owns
// A block owns GROUPS times 16 columns; for each 16, four warps hold S and four solve, stage and write outputs.
constexpr int DC_GROUP_THREADS = 256;

// What a (chunk, head) leaves for the walk, as it lies in the walk's shared memory (words of 32 bits): c k,
// c q and the last line's keys as fragments of mma.sync's B operand, a plane for each of the three bfloat16
// values, 8 bytes a lane; the products of all decays [DK]; T and B [16][16].
//   c k, c q: [16 dk][8 tokens][plane][lane][2], k = dk
//   last line: [8 dk][plane][lane][2], k = token (2 i, 2 i + 1 of a k group are tokens i and
//   i + 4 of the group's eight, on both operands)
template <int DK>
struct DeltaChunk {
  static constexpr int PLANE = 64;                    // words a fragment's plane
  static constexpr int ROWS = 3 * DC_TOKENS * DK / 2; // words of one of the three
  static constexpr int Q = ROWS, E = 2 * ROWS, G = 3 * ROWS, L = G + DK;
  static constexpr int TI = L + DK, BI = TI + DC_TOKENS * DC_TOKENS;
  static constexpr int WORDS = BI + DC_TOKENS * DC_TOKENS;
  static_assert(WORDS % 4 == 0 && DK % 64 == 0, "");
};
// x and y as three bfloat16 values each, x in the low halves: the nearest one (ties away from zero), the
// nearest one to the rest, and what is left, which has eight bits
__device__ __forceinline__ void dc_split(float x, float y, uint32_t (&p)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const uint32_t a = __float_as_uint(x) + (i < 2 ? 0x8000u : 0u), b = __float_as_uint(y) + (i < 2 ? 0x8000u : 0u);
    p[i] = __byte_perm(a, b, 0x7632);
    if (i < 2) {
      x -= __uint_as_float(a & 0xffff0000u);
      y -= __uint_as_float(b & 0xffff0000u);
    }
  }
}
// Chunk c of request s is number cu_tokens[s] / 16 + s + c: that grows by one from chunk to chunk of a request
// and by at least one from request to request, so no two share a number and none is above this.
__host__ __device__ __forceinline__ long dc_chunks(long n_tokens, long n_seqs) {
  return (n_tokens - 1) / DC_TOKENS + n_seqs;
}

// g of a raw decay; the rate exp(a_log) as the sum of two
__device__ __forceinline__ float dc_decay(float a, float rate_hi, float rate_lo) {
  const float sp = a > 20.f ? a : log1pf(expf(a)), y = rate_hi * sp, g = expf(-y);
  return g > 0.f ? fmaf(-g, fmaf(rate_lo, sp, fmaf(rate_hi, sp, -y)), g) : g;       // (y may be infinite)
}

// One block a (chunk, head).  Bound by its instructions: 256 dot products over dk with a running product of
// decays each, and the splitting.  Sixteen threads a dot product, the pairs (i, j) of two rows j and 15 - j by the
// same threads, so that all walk 17; the sums of four rows i go over the lanes together, eight shuffles for 32.  Six
// blocks an SM (80 registers; four 1 % slower with the walk, eight, with their spills, 6 %).  Under ncu, 2,048 tokens of 16
// heads of 128 x 128: 51 µs, issue slots 65 % busy, the way from shared memory 64 %, the 64-bit pipe 2 %.
template <typename T, int DK>
__global__ void __launch_bounds__(128, 6)
delta_chunk_prepare_kernel(uint32_t* __restrict__ chunks, const T* __restrict__ qkv, int qkv_ld, int q_off, int k_off,
                           const T* __restrict__ beta_raw, int beta_ld, const T* __restrict__ a_raw, int a_ld,
                           const float* __restrict__ a_log, const float* __restrict__ dt_bias,
                           const int* __restrict__ cu_tokens, int n_seqs, int heads, int kv_heads, int dk) {
  pdl_launch_dependents();
  pdl_wait();
  using C = DeltaChunk<DK>;
  constexpr int N = DC_TOKENS, LD = DK + 4;
  __shared__ __align__(16) float ks[N][LD], qs[N][LD], gs[N][LD];
  __shared__ float am[N][N + 1], bm[N][N + 1], bs[N], kqs[N];
  const int id = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int lo = 0, hi = n_seqs - 1;                        // the last request whose first chunk is not above id
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (cu_tokens[mid] / N + mid <= id) lo = mid;
    else hi = mid - 1;
  }
  const int t_seq = cu_tokens[lo], c = id - (t_seq / N + lo);
  const int nc = min(N, cu_tokens[lo + 1] - t_seq - c * N);
  if (c < 0 || nc <= 0) return;
  const int t0 = t_seq + c * N;
  const int kh = h / (heads / kv_heads);
  {
    // a warp's four tokens: everything is asked for before anything is summed
    constexpr int M = DK / 32;
    float kx[4][M], qx[4][M], ax[4][M], bias[M], beta = 0.f;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const size_t t = t0 + min(warp + 4 * r, nc - 1);
      const T* kr = qkv + t * qkv_ld + k_off + (size_t)kh * dk;
      const T* qr = qkv + t * qkv_ld + q_off + (size_t)kh * dk;
      const T* ar = a_raw + t * a_ld + (size_t)h * dk;
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const int d = lane + 32 * m;
        const bool in = d < dk;
        kx[r][m] = in ? to_float(kr[d]) : 0.f;
        qx[r][m] = in ? to_float(qr[d]) : 0.f;
        ax[r][m] = in ? to_float(ar[d]) : 0.f;
      }
    }
    const int of = lane >> 3, own = warp + 4 * (lane >> 1 & 3);       // what this lane finishes below, and the token
    if (of == 3) beta = to_float(beta_raw[(size_t)(t0 + min(own, nc - 1)) * beta_ld + h]);
#pragma unroll
    for (int m = 0; m < M; ++m) bias[m] = lane + 32 * m < dk ? dt_bias[(size_t)h * dk + lane + 32 * m] : 0.f;
    const double rate = exp((double)a_log[h]);
    const float rate_hi = (float)rate, rate_lo = (float)(rate - (double)rate_hi);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int m = 0; m < M; ++m) {                   // (rows behind the last token: k = q = 0, g = 1, beta = 0)
        const int d = lane + 32 * m;
        gs[warp + 4 * r][d] = warp + 4 * r < nc && d < dk ? dc_decay(ax[r][m] + bias[m], rate_hi, rate_lo) : 1.f;
      }
    // |k|^2, |q|^2 and k . q of the four tokens: a lane's few products in 32 bits, the lanes' in 64; of two partners
    // each goes on with half of the sums, and lane 8 of + 2 r ends up with sum `of` of token r
    double sums[16];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      float kk = 0.f, qq = 0.f, kq = 0.f;
#pragma unroll
      for (int m = 0; m < M; ++m) {
        kk = fmaf(kx[r][m], kx[r][m], kk);
        qq = fmaf(qx[r][m], qx[r][m], qq);
        kq = fmaf(kx[r][m], qx[r][m], kq);
      }
      sums[r] = kk;
      sums[4 + r] = qq;
      sums[8 + r] = kq;
      sums[12 + r] = 0.;
    }
#pragma unroll
    for (int left = 8, o = 16; left > 0; left /= 2, o /= 2)
#pragma unroll
      for (int x = 0; x < left; ++x) {
        const bool upper = lane & o;
        const double got = __shfl_xor_sync(0xffffffffu, upper ? sums[x] : sums[x + left], o);
        sums[x] = (upper ? sums[x + left] : sums[x]) + got;
      }
    double value = sums[0] + __shfl_xor_sync(0xffffffffu, sums[0], 1);
    // 1 / |k|, dk^-1/2 / |q|, k . q of the unit vectors, beta
    if (of < 2) value = rsqrt((value + 1e-6) * (of ? (double)dk : 1.));
    if (of == 3) value = 1. / (1. + exp(-(double)beta));
    const double kn = __shfl_sync(0xffffffffu, value, lane & 6), qn = __shfl_sync(0xffffffffu, value, 8 + (lane & 6));
    if (of == 2) value *= kn * qn;
    const float hi = (float)value, lo = (float)(value - (double)hi);
    if (of >= 2 && !(lane & 1)) (of == 2 ? kqs : bs)[own] = own < nc ? hi : 0.f;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = warp + 4 * r;
      const float k_hi = __shfl_sync(0xffffffffu, hi, 2 * r), k_lo = __shfl_sync(0xffffffffu, lo, 2 * r);
      const float q_hi = __shfl_sync(0xffffffffu, hi, 8 + 2 * r), q_lo = __shfl_sync(0xffffffffu, lo, 8 + 2 * r);
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const int d = lane + 32 * m;
        ks[i][d] = i < nc ? fmaf(kx[r][m], k_hi, kx[r][m] * k_lo) : 0.f;
        qs[i][d] = i < nc ? fmaf(qx[r][m], q_hi, qx[r][m] * q_lo) : 0.f;
      }
    }
  }
  __syncthreads();
  uint32_t* dst = chunks + ((size_t)id * heads + h) * C::WORDS;
  {
    constexpr int M = DK / 64;                        // pieces of four values a thread
    const int part = tid & 15, pair = tid >> 4;
#pragma unroll 1
    for (int side = 0; side < 2; ++side) {
      const int j = side ? N - 1 - pair : pair;
      float4 w[M];
#pragma unroll
      for (int m = 0; m < M; ++m) w[m] = *reinterpret_cast<const float4*>(&ks[j][4 * part + 64 * m]);
#pragma unroll 1
      for (int i0 = j; i0 < N; i0 += 4) {             // (the two halves of a warp may be at different rows)
        float sums[8];                                // of k, then of q
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int i = min(i0 + r, N - 1);
          float a = 0.f, b = 0.f;
#pragma unroll
          for (int m = 0; m < M; ++m) {
            if (i0 + r > j) {
              const float4 g = *reinterpret_cast<const float4*>(&gs[i][4 * part + 64 * m]);
              w[m].x *= g.x; w[m].y *= g.y; w[m].z *= g.z; w[m].w *= g.w;
            }
            const float4 k = *reinterpret_cast<const float4*>(&ks[i][4 * part + 64 * m]);
            const float4 q = *reinterpret_cast<const float4*>(&qs[i][4 * part + 64 * m]);
            a = fmaf(w[m].x, k.x, fmaf(w[m].y, k.y, fmaf(w[m].z, k.z, fmaf(w[m].w, k.w, a))));
            b = fmaf(w[m].x, q.x, fmaf(w[m].y, q.y, fmaf(w[m].z, q.z, fmaf(w[m].w, q.w, b))));
          }
          sums[r] = a;
          sums[4 + r] = b;
        }
        // eight sums over sixteen lanes: half of them to the other half of the lanes at each step
#pragma unroll
        for (int o = 8, left = 4; o > 1; o /= 2, left /= 2)
#pragma unroll
          for (int x = 0; x < left; ++x) {
            const bool upper = part & o;
            const float got = __shfl_xor_sync(0xffffu << (lane & 16), upper ? sums[x] : sums[x + left], o);
            sums[x] = (upper ? sums[x + left] : sums[x]) + got;
          }
        sums[0] += __shfl_xor_sync(0xffffu << (lane & 16), sums[0], 1);
        const int i = i0 + (part >> 1 & 1) + (part >> 1 & 2);
        if (!(part & 1) && i < N) (part & 8 ? bm : am)[i][j] = sums[0];
      }
    }
  }
  // the products of decays up to every token, two channels of eight tokens a thread, and behind it, a channel
  // a thread
  for (int x = tid; x < DK; x += 128) {
    const int d = 2 * x % DK, first = 2 * x / DK * 8;
    float px = 1.f, py = 1.f;
    for (int i = 0; i < first; ++i) {
      px *= gs[i][d];
      py *= gs[i][d + 1];
    }
    uint32_t* at = dst + (d / 16) * 2 * 3 * C::PLANE + d % 8 + (d % 16) / 8 + (first / 8) * 3 * C::PLANE;
#pragma unroll
    for (int i = 0; i < 8; ++i, at += 8) {
      px *= gs[first + i][d];
      py *= gs[first + i][d + 1];
      uint32_t w[3];
      dc_split(ks[first + i][d] * px, ks[first + i][d + 1] * py, w);
#pragma unroll
      for (int p = 0; p < 3; ++p) at[p * C::PLANE] = w[p];
      dc_split(qs[first + i][d] * px, qs[first + i][d + 1] * py, w);
#pragma unroll
      for (int p = 0; p < 3; ++p) at[C::Q + p * C::PLANE] = w[p];
    }
    if (first) {
      reinterpret_cast<float*>(dst)[C::G + d] = px;
      reinterpret_cast<float*>(dst)[C::G + d + 1] = py;
    }
  }
  for (int d = 127 - tid; d < DK; d += 128) {         // (of 64 channels, by the threads that had none above)
    float p = 1.f, e[N];
#pragma unroll
    for (int i = N - 1; i >= 0; --i) {
      e[i] = i == nc - 1 ? 0.f : ks[i][d] * p;        // (the last token's write has no product of decays)
      p *= gs[i][d];
    }
    reinterpret_cast<float*>(dst)[C::L + d] = ks[nc - 1][d];
    uint32_t* to = dst + C::E + (d / 8) * 3 * C::PLANE + (d % 8) * 8;
    uint32_t w[N / 2][3];                             // [2 kappa + half of the tokens]
#pragma unroll
    for (int i = 0; i < N / 2; ++i) dc_split(e[i / 2 + 8 * (i % 2)], e[i / 2 + 8 * (i % 2) + 4], w[i]);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      *reinterpret_cast<uint4*>(to + q * C::PLANE) = make_uint4(w[0][q], w[1][q], w[2][q], w[3][q]);
      *reinterpret_cast<uint4*>(to + q * C::PLANE + 4) = make_uint4(w[4][q], w[5][q], w[6][q], w[7][q]);
    }
  }
  __syncthreads();
  for (int idx = tid; idx < N * N; idx += 128) {
    const int i = idx / N, j = idx % N;
    reinterpret_cast<float*>(dst)[C::BI + idx] = j < i ? bm[i][j] : j == i ? kqs[i] : 0.f;
  }
  if (tid < N) {                                      // a column of T a thread
    float x[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      float s = i == tid ? 1.f : 0.f;
#pragma unroll
      for (int m = 0; m < i; ++m) s = fmaf(-am[i][m], x[m], s);
      x[i] = bs[i] * s;
      reinterpret_cast<float*>(dst)[C::TI + i * N + tid] = x[i];
    }
  }
}

// ---------------------------------------------------------------- the walk over chunks
// D += A B, 16 x 8 x 16
__device__ __forceinline__ void dc_mma(float (&d)[4], const uint32_t (&a)[4], const uint2& b) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y));
}
// the six products of two factors of three planes each, by size: sums[0] += a0 b0, ...; of two results in turn, so
// that a product's sums are there when the next one adds to them
__device__ __forceinline__ void dc_mma_split(float (&x)[3][4], float (&y)[3][4], const uint32_t (&a)[3][4],
                                             const uint32_t* frag_x, const uint32_t* frag_y, int lane) {
  uint2 b[3], c[3];
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    b[p] = *reinterpret_cast<const uint2*>(frag_x + 64 * p + 2 * lane);
    c[p] = *reinterpret_cast<const uint2*>(frag_y + 64 * p + 2 * lane);
  }
#pragma unroll
  for (int p = 0; p < 3; ++p)
#pragma unroll
    for (int q = 0; q + p < 3; ++q) {
      dc_mma(x[p + q], a[q], b[p]);
      dc_mma(y[p + q], a[q], c[p]);
    }
}
__device__ __forceinline__ float dc_total(const float (&sums)[3][4], int e) { return sums[0][e] + (sums[1][e] + sums[2][e]); }
template <int BARRIER, int THREADS>
__device__ __forceinline__ void dc_bar_sync() { asm volatile("bar.sync %0, %1;" ::"n"(BARRIER), "n"(THREADS) : "memory"); }
template <int BARRIER, int THREADS>
__device__ __forceinline__ void dc_bar_arrive() { asm volatile("bar.arrive %0, %1;" ::"n"(BARRIER), "n"(THREADS) : "memory"); }

template <int DK, int GROUPS, int STAGES>
struct DeltaChunkSmem {
  static constexpr int PLD = 24;                      // floats a column of partial sums (16) or a row of U takes
  static constexpr int PART = DC_COLS * PLD;
  static constexpr int PK = 0;                        // of a group: [4][cols][tokens]: S^T Kc by warp
  static constexpr int PQ = PK + 4 * PART;                       // [2][4][cols][tokens]: S^T Qc
  static constexpr int R = PQ + 8 * PART;                        // [cols][20]: V - S^T Kc
  static constexpr int U = R + DC_COLS * 20;                     // [tokens][cols]
  static constexpr int GROUP = U + DC_TOKENS * PLD;
  static constexpr int CHUNKS = STAGES * DeltaChunk<DK>::WORDS;
  static constexpr size_t BYTES = (size_t)(CHUNKS + GROUPS * GROUP) * 4;
};

// v at qkv[t, v_off + h * dv + col]; S of a slot at state + slot * state_stride, [heads, dk, dv]; o [T, heads * dv].
// Block = (request, head, 16 GROUPS columns).  S^T lies in the accumulator fragments of a group's first four warps, a
// quarter of dk each (columns of S on the rows of the fragment), which are as they stand the A operand of S^T Kc and
// S^T Qc.  The other four own the solution: four columns each, two tokens of a column a thread.  A chunk's
// chain is S^T Kc -> barrier -> sums of the four quarters, U = T R -> barrier -> the write into S; S^T Qc runs beside
// the solution, the outputs and the copies beside the write.  Bound by that chain, 1,880 cycles
// a chunk under ncu (2,048 tokens, 16 heads of 128 x 128: 143 µs, issue slots 47 % busy, tensor pipe 31 %, the way from
// shared memory 49 %); eight warps of 16 dk each instead of four take as long (and 5 % longer where blocks share SMs).
template <typename T, int DK, int GROUPS, int STAGES>
__global__ void __launch_bounds__(GROUPS * DC_GROUP_THREADS)
delta_chunk_kernel(float* __restrict__ o, const uint32_t* __restrict__ chunks, const T* __restrict__ qkv, int qkv_ld,
                   int v_off, float* __restrict__ state, long state_stride, const int* __restrict__ cu_tokens,
                   const int* __restrict__ slots, int heads, int dk, int dv) {
  pdl_wait();                                         // (nor launched early: see `delta_rule_kernel`)
  using C = DeltaChunk<DK>;
  using M = DeltaChunkSmem<DK, GROUPS, STAGES>;
  constexpr int N = DC_TOKENS, ND = DK / 32, PLD = M::PLD, THREADS = GROUPS * DC_GROUP_THREADS, HALF = THREADS / 2;
  extern __shared__ __align__(16) uint32_t dc_sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = (tid >> 5) & 3, group = (tid >> 7) % GROUPS;
  const int col_blocks = (dv + GROUPS * DC_COLS - 1) / (GROUPS * DC_COLS);
  const int s = blockIdx.x / col_blocks / heads, h = blockIdx.x / col_blocks - s * heads;
  const int col0 = (blockIdx.x % col_blocks * GROUPS + group) * DC_COLS;
  const int t0 = cu_tokens[s], n = cu_tokens[s + 1] - t0;
  if (n <= 0) return;
  const int n_chunks = (n + N - 1) / N;
  float* gm = reinterpret_cast<float*>(dc_sm) + M::CHUNKS + group * M::GROUP;

  if (tid < HALF) {
    // ------------------------------------------------------------ S
    const int kap = lane & 3, row = lane >> 2, d0 = warp * (DK / 4);
    float* S_g = state + (size_t)slots[s] * state_stride + (size_t)h * dk * dv + col0;
    float S[ND][4];                                   // tiles of 8 dk
#pragma unroll
    for (int m = 0; m < ND; ++m)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int d = d0 + 8 * m + 2 * kap + (e & 1), c = row + 8 * (e >> 1);
        S[m][e] = d < dk && col0 + c < dv ? S_g[(size_t)d * dv + c] : 0.f;
      }
    uint32_t a[ND / 2][3][4];                         // [16 dk][plane]: rows col, col + 8 of two tiles
    auto split_tiles = [&](int m) {                   // tiles m, m + 1
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          uint32_t w[3];
          dc_split(S[m + t][2 * e], S[m + t][2 * e + 1], w);
#pragma unroll
          for (int p = 0; p < 3; ++p) a[m / 2][p][2 * t + e] = w[p];
        }
    };
#pragma unroll
    for (int m = 0; m < ND; m += 2) split_tiles(m);
    dc_bar_sync<2, THREADS>();                        // the first chunk is there
    for (int ch = 0; ch < n_chunks; ++ch) {
      const uint32_t* st = dc_sm + ch % STAGES * C::WORDS;
      auto product = [&](const uint32_t* frags, float* part) {
        float sums[2][3][4] = {};
#pragma unroll
        for (int m = 0; m < ND / 2; ++m) {
          const uint32_t* frag = frags + (warp * (ND / 2) + m) * 2 * 3 * C::PLANE;
          dc_mma_split(sums[0], sums[1], a[m], frag, frag + 3 * C::PLANE, lane);
        }
        float* p = part + warp * M::PART + row * PLD + 2 * kap;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          *reinterpret_cast<float2*>(p + 8 * t) = make_float2(dc_total(sums[t], 0), dc_total(sums[t], 1));
          *reinterpret_cast<float2*>(p + 8 * t + 8 * PLD) = make_float2(dc_total(sums[t], 2), dc_total(sums[t], 3));
        }
      };
      product(st, gm + M::PK);
      dc_bar_arrive<1, THREADS>();
      product(st + C::Q, gm + M::PQ + (ch & 1) * 4 * M::PART);
      dc_bar_sync<2, THREADS>();
      const float* u_last = gm + M::U + (min(N, n - ch * N) - 1) * PLD + row;
      const float last[2] = {u_last[0], u_last[8]};
      // U^T [columns, tokens]; k = 2 kap, 2 kap + 1 of eight tokens are tokens kap and kap + 4
      uint32_t u[3][4];
      const float* us = gm + M::U + kap * PLD + row;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        uint32_t w[3];
        const float* x = us + 8 * (e >> 1) * PLD + 8 * (e & 1);
        dc_split(x[0], x[4 * PLD], w);
#pragma unroll
        for (int p = 0; p < 3; ++p) u[p][e] = w[p];
      }
#pragma unroll
      for (int m = 0; m < ND; m += 2) {
        float sums[2][3][4] = {};
        const uint32_t* frag = st + C::E + (warp * ND + m) * 3 * C::PLANE;
        dc_mma_split(sums[0], sums[1], u, frag, frag + 3 * C::PLANE, lane);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const float2 g = *reinterpret_cast<const float2*>(st + C::G + d0 + 8 * (m + t) + 2 * kap);
          const float2 k = *reinterpret_cast<const float2*>(st + C::L + d0 + 8 * (m + t) + 2 * kap);
#pragma unroll
          for (int e = 0; e < 4; ++e)                 // (the last token's write comes last, with one rounding)
            S[m + t][e] = fmaf((e & 1) ? k.y : k.x, last[e >> 1],
                               fmaf(S[m + t][e], (e & 1) ? g.y : g.x, dc_total(sums[t], e)));
        }
        split_tiles(m);                               // for the next chunk, beside the other tiles' products
      }
    }
#pragma unroll
    for (int m = 0; m < ND; ++m)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int d = d0 + 8 * m + 2 * kap + (e & 1), c = row + 8 * (e >> 1);
        if (d < dk && col0 + c < dv) S_g[(size_t)d * dv + c] = S[m][e];
      }
  } else {
    // ------------------------------------------------------------ copies, the solution, outputs
    const int own = 4 * warp + (lane & 3), tok = lane >> 2;          // column; tokens tok, tok + 8
    const bool live = col0 + own < dv;
    const uint32_t* src = chunks + ((size_t)(t0 / N + s) * heads + h) * C::WORDS;
    const size_t chunk_step = (size_t)heads * C::WORDS;
    const T* v_col = qkv + v_off + (size_t)h * dv + (live ? col0 + own : 0);
    float* o_col = o + (size_t)h * dv + col0 + own;
    const size_t o_step = (size_t)heads * dv;
    auto stage = [&](int ch) {
      if (ch < n_chunks) {
        uint32_t* to = dc_sm + ch % STAGES * C::WORDS;
        const uint32_t* from = src + (size_t)ch * chunk_step;
#pragma unroll 5
        for (int i = tid - HALF; i < C::WORDS / 4; i += HALF) dr_cp_async16(to + 4 * i, from + 4 * i);
      }
      asm volatile("cp.async.commit_group;\n" ::);
    };
    T v_next[2];
    auto fetch_v = [&](int ch) {                      // (a token beyond the request's last is not read from)
#pragma unroll
      for (int e = 0; e < 2; ++e) v_next[e] = v_col[(size_t)(t0 + min(ch * N + tok + 8 * e, n - 1)) * qkv_ld];
    };
#pragma unroll
    for (int ch = 0; ch < STAGES - 1; ++ch) stage(ch);
    fetch_v(0);
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2));
    dc_bar_sync<2, THREADS>();
    float* rs = gm + M::R;
    float* us = gm + M::U;
    // a + the row of T or B left of its own token, times a column (a token that holds NaN must not reach the ones
    // before it, as zero times NaN would).  The own token's term, mostly the largest, is added last by the callers:
    // one rounding of its size.
    auto row_sum = [&](float first, const float (&w)[N], const float (&x)[N], int token) {
      float a[4] = {first};
#pragma unroll
      for (int j = 0; j < N - 1; ++j)
        if (j < token) a[(j + 1) & 3] = fmaf(w[j], x[j], a[(j + 1) & 3]);
      return (a[0] + a[1]) + (a[2] + a[3]);
    };
    auto parts_sum = [&](const float* p) { return (p[0] + p[M::PART]) + (p[2 * M::PART] + p[3 * M::PART]); };
    auto load_row = [&](float (&w)[N], const float* from) {
#pragma unroll
      for (int j = 0; j < N; j += 4) *reinterpret_cast<float4*>(&w[j]) = *reinterpret_cast<const float4*>(from + j);
    };
    for (int ch = 0; ch < n_chunks; ++ch) {
      const float* st = reinterpret_cast<const float*>(dc_sm + ch % STAGES * C::WORDS);
      const int nc = min(N, n - ch * N);
      float v[2], t_row[2][N], t_own[2], b_own[2], sum[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        v[e] = tok + 8 * e < nc ? to_float(v_next[e]) : 0.f;
        load_row(t_row[e], st + C::TI + (tok + 8 * e) * N);
        t_own[e] = st[C::TI + (tok + 8 * e) * (N + 1)];
        b_own[e] = st[C::BI + (tok + 8 * e) * (N + 1)];
      }
      fetch_v(ch + 1);
      dc_bar_sync<1, THREADS>();
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        sum[e] = tok + 8 * e < nc ? parts_sum(gm + M::PK + own * PLD + tok + 8 * e) : 0.f;
        rs[own * 20 + tok + 8 * e] = v[e] - sum[e];
      }
      __syncwarp();
      float r[N];
      load_row(r, rs + own * 20);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        sum[e] = fmaf(t_own[e], v[e], row_sum(-t_own[e] * sum[e], t_row[e], r, tok + 8 * e));
        us[(tok + 8 * e) * PLD + own] = sum[e];
      }
      asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 3));
      dc_bar_sync<2, THREADS>();
      float u[N];
#pragma unroll
      for (int j = 0; j < N; ++j) u[j] = us[j * PLD + own];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int i = tok + 8 * e;
        float b_row[N];
        load_row(b_row, st + C::BI + i * N);
        const float before = row_sum(parts_sum(gm + M::PQ + (ch & 1) * 4 * M::PART + own * PLD + i), b_row, u, i);
        if (live && i < nc) o_col[(size_t)(t0 + ch * N + i) * o_step] = fmaf(b_own[e], sum[e], before);
      }
      // the stage of the chunk before: its last reads were made before this chunk's first barrier
      stage(ch + STAGES - 1);
    }
    asm volatile("cp.async.wait_group 0;\n" ::);
  }
}
