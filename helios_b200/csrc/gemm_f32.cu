// True float32 matrix product on the FMA pipes: C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]).
// No tensor cores and no reduced-precision mode.  Every output element is summed in one order
// that depends on K alone: runs of RUN consecutive k, in each the even k and the odd k from zero in
// their order, then the two; the runs of a quarter of K in order; and (q0 + q1) + (q2 + q3).  Both kernels
// below keep that order, so a row's result does not depend on the other rows of the launch.
// Even and odd k are the halves of `fma.rn.f32x2`, two multiply-adds an instruction.
// (python/helios/exec/model.py:236-238, 250-251, 336-337, 493-496: y = x W^T + b with W
// stored [out, in].)
#include "common.cuh"

constexpr int RUN = 16;             // consecutive k of one partial sum
constexpr int BK = 32;              // k of a tile of the kernel for many rows: a quarter is whole tiles
static_assert(BK % RUN == 0, "");
// k of a quarter (the last ones may be short or empty)
__host__ __device__ __forceinline__ int quarter_k(int K) { return (K + 4 * BK - 1) / (4 * BK) * BK; }

// 16 bytes, of zeros where `in` does not hold (nothing is read then)
__device__ __forceinline__ void cp_async16_if(void* smem, const void* gmem, bool in) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(in ? 16 : 0));
}
__device__ __forceinline__ void cp_async4_if(void* smem, const void* gmem, bool in) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(s), "l"(gmem), "r"(in ? 4 : 0));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ float both(f32x2 v) {
  return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}

// Lets a kernel take up to BYTES of dynamic shared memory.  Once per device, and the same for every
// call: the limit belongs to the function, and a call that set its own size could lower it between
// another thread's setting and launch.
template <auto KERNEL, int BYTES>
static bool allow_shared_memory() {
  constexpr int MOST_DEVICES = 64;
  static bool done[MOST_DEVICES] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MOST_DEVICES) return false;
  if (!done[dev]) {
    if (cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, BYTES) != cudaSuccess) return false;
    done[dev] = true;
  }
  return true;
}

// ---------------------------------------------------------------- few rows
// Bound by reading W once.  A warp takes ROWS_W rows of W and 32 runs of k, a run a lane: the 64
// bytes of a lane's run come straight into registers; with AHEAD, those of the warp's next rows before the
// sums of the present ones are made, so that loads are on their way all the time.  A's rows lie in shared
// memory for the whole of K, runs RUN + 4 floats apart so that neighbouring lanes read different banks.  The
// `wpg` warps that share rows of W are a group with a barrier of its own; the groups of all blocks, which
// are as many as are resident, take the rows in turn.
constexpr int ROWS_RUN = RUN + 4;
constexpr int ROWS_MOST_WARPS = 8;
constexpr int ROWS_MOST_SMEM = 200 * 1024;       // what a block may take of shared memory

__device__ __forceinline__ void group_sync(int group, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(threads) : "memory");
}

template <int MT, int ROWS_W, bool AHEAD>
__global__ void __launch_bounds__(32 * ROWS_MOST_WARPS, MT > 4 && ROWS_W > 2 ? 1 : 2)
gemm_f32_rows_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W,
                     const float* __restrict__ bias, int M, int N, int K, int lda, int ldw, int ldc,
                     int wpg) {
  extern __shared__ __align__(16) float rows_sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, threads = blockDim.x;
  const int groups = (threads >> 5) / wpg, g = warp / wpg, first_rb = warp - g * wpg;
  const int q_runs = quarter_k(K) / RUN, runs = 4 * q_runs;
  const int rounds = (runs + 32 * wpg - 1) / (32 * wpg);                          // 32-run pieces a warp takes
  const int line = runs * ROWS_RUN;                // floats of one row of A
  const int part_line = runs + 1;                  // floats of one output's partial sums
  constexpr int OUTS = ROWS_W * MT;
  float* part = rows_sm + MT * line + g * 2 * OUTS * part_line;     // [2][OUTS][part_line]
  const int m0 = blockIdx.y * MT;
  const int units = (N + ROWS_W - 1) / ROWS_W, step_units = gridDim.x * groups;
  const int u0 = blockIdx.x * groups + g;
  const int steps = u0 < units ? ((units - 1 - u0) / step_units + 1) * rounds : 0;

  pdl_launch_dependents();
  int next_n = u0 * ROWS_W, next_round = 0;        // what `load` fetches next
  auto load = [&](ulonglong2 (&w)[ROWS_W][RUN / 4]) {
    const int k0 = ((first_rb + next_round * wpg) * 32 + lane) * RUN;
#pragma unroll
    for (int r = 0; r < ROWS_W; ++r) {
      const float* src = W + (size_t)(next_n + r) * ldw + k0;
#pragma unroll
      for (int i = 0; i < RUN / 4; ++i)
        w[r][i] = (next_n + r < N && k0 + 4 * i < K) ? __ldg(reinterpret_cast<const ulonglong2*>(src) + i)
                                                     : make_ulonglong2(0ull, 0ull);
    }
    if (++next_round == rounds) {
      next_round = 0;
      next_n = next_n < N ? next_n + step_units * ROWS_W : next_n;
    }
  };
  {  // the first rows of W on their way to L2 under the kernel before (no further: W need not be a
     // weight that nobody writes)
    const int k0 = (first_rb * 32 + lane) * RUN;
    for (int i = 0; i < (AHEAD ? 2 : 1); ++i)
      for (int r = 0; r < ROWS_W; ++r) {
        const int n = (u0 + i * step_units) * ROWS_W + r;
        if (k0 < K && n < N) asm volatile("prefetch.global.L2 [%0];" ::"l"(W + (size_t)n * ldw + k0));
      }
  }
  pdl_wait();
  ulonglong2 w0[ROWS_W][RUN / 4], w1[AHEAD ? ROWS_W : 1][RUN / 4];
  load(w0);
#pragma unroll
  for (int m = 0; m < MT; ++m) {
    const float* src = A + (size_t)(m0 + m < M ? m0 + m : 0) * lda;
    for (int v = tid; v < runs * (RUN / 4); v += threads) {
      const bool in = m0 + m < M && 4 * v < K;
      cp_async16_if(rows_sm + m * line + (v / (RUN / 4)) * ROWS_RUN + (v % (RUN / 4)) * 4, in ? src + 4 * v : A, in);
    }
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();

  int n0 = u0 * ROWS_W, round = 0, half = 0, turn = 0;
  auto take = [&](auto& w, auto& ahead) {
    float* sums = part + half * OUTS * part_line;
    const int run = (first_rb + round * wpg) * 32 + lane;
    if constexpr (AHEAD) load(ahead);
    f32x2 acc[ROWS_W][MT];
#pragma unroll
    for (int r = 0; r < ROWS_W; ++r)
#pragma unroll
      for (int m = 0; m < MT; ++m) acc[r][m] = 0ull;
    if (run < runs) {
      const float* a_run = rows_sm + run * ROWS_RUN;
#pragma unroll
      for (int i = 0; i < RUN / 4; ++i)
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(a_run + m * line + 4 * i);
#pragma unroll
          for (int r = 0; r < ROWS_W; ++r) acc[r][m] = fma2(a.x, w[r][i].x, acc[r][m]);
#pragma unroll
          for (int r = 0; r < ROWS_W; ++r) acc[r][m] = fma2(a.y, w[r][i].y, acc[r][m]);
        }
    }
    if constexpr (!AHEAD) load(w);
    if (run < runs) {
#pragma unroll
      for (int r = 0; r < ROWS_W; ++r)
#pragma unroll
        for (int m = 0; m < MT; ++m) sums[(r * MT + m) * part_line + run] = both(acc[r][m]);
    }
    if (++round < rounds) return;
    round = 0;
    group_sync(g, 32 * wpg);
    // a thread a quarter, the four of an output side by side; the group's warps take the rows in turn, with four rows
    // in groups of many warps (long rows, and so long sums) eight outputs each: 1,024 x 4,096 at four rows 9.9 -> 8.8 µs, but 151,936 x 896
    // at eight 190 -> 203
    auto finish = [&](int base) {
      const int idx = base + lane, out = idx / 4;
      const bool in = out < OUTS;
      const float* p = sums + (in ? out : 0) * part_line + (idx % 4) * q_runs;
      float q = 0.f;
#pragma unroll 8
      for (int r = 0; r < q_runs; ++r) q += p[r];
      q += __shfl_xor_sync(0xffffffffu, q, 1);
      q += __shfl_xor_sync(0xffffffffu, q, 2);
      const int n = n0 + out / MT, m = m0 + out % MT;
      if (in && idx % 4 == 0 && n < N && m < M) C[(size_t)m * ldc + n] = q + (bias ? bias[n] : 0.f);
    };
    if (AHEAD || wpg <= 2) {
      if (first_rb == turn) {
#pragma unroll
        for (int base = 0; base < 4 * OUTS; base += 32) finish(base);
      }
      turn = turn + 1 == wpg ? 0 : turn + 1;
    } else {
#pragma unroll 1
      for (int base = 32 * (first_rb >= turn ? first_rb - turn : first_rb - turn + wpg); base < 4 * OUTS; base += 32 * wpg)
        finish(base);
      for (turn += (4 * OUTS + 31) / 32; turn >= wpg;) turn -= wpg;
    }
    // (the next rows' sums go to the other half of `part`; this half is written again only behind the
    // group's next barrier)
    n0 += step_units * ROWS_W;
    half ^= 1;
  };
  if constexpr (AHEAD) {
    for (int step = 0; step < steps; step += 2) {
      take(w0, w1);
      if (step + 1 < steps) take(w1, w0);
    }
  } else {
    for (int step = 0; step < steps; ++step) take(w0, w0);
  }
}

// ---------------------------------------------------------------- many rows
// Bound by the FMA pipes and by the operands' way from shared memory to registers.  Operands stay [row][k] in
// shared memory (rows 36 floats apart, so that neighbouring rows start in different banks).  KS = 4: the four blocks
// of a cluster have a quarter of K each, three tiles in flight, and add their quarters through distributed shared
// memory.  KS = 1: a block has all of K, two tiles in flight, and keeps the quarters that wait for another one in
// shared memory (in C they cost 14 to 21 % of the time).  `launch_tiles` says which.
constexpr int LINE = BK + 4, TILE_THREADS = 128;
template <int TM, int TN, int KS>
struct Tile {                                      // 8 threads along M, 16 along N
  static constexpr int BM = 8 * TM, BN = 16 * TN, STAGE_FLOATS = (BM + BN) * LINE, STAGES = KS == 1 ? 2 : 3;
  static constexpr int BYTES = (STAGES * STAGE_FLOATS + (KS == 1 ? 2 * BM * BN : 0)) * (int)sizeof(float);
  static_assert(KS == 1 || STAGES * STAGE_FLOATS >= BM * (BN + 1), "the sums of a block lie where its tiles were");
};

__device__ __forceinline__ float peer_f32(const float* mine, uint32_t rank) {
  uint32_t remote;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote)
               : "r"((uint32_t)__cvta_generic_to_shared(mine)), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int TM, int TN, bool VEC, int KS>
__global__ void __launch_bounds__(TILE_THREADS, TM * TN > 16 ? 3 : 4)
gemm_f32_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W,
                const float* __restrict__ bias, int M, int N, int K, int lda, int ldw, int ldc) {
  pdl_wait();
  using Tl = Tile<TM, TN, KS>;
  constexpr int BM = Tl::BM, BN = Tl::BN, STAGE_FLOATS = Tl::STAGE_FLOATS, STAGES = Tl::STAGES;
  extern __shared__ __align__(16) float tile_sm[];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tx = tid % 16, ty = tid / 16;          // rows ty + 8 i of A, tx + 16 j of W
  constexpr int QUARTERS = 4 / KS;
  const int qk = quarter_k(K);
  const int k_first = (int)blockIdx.z * QUARTERS * qk;             // the cluster lies along z: rank = blockIdx.z
  const int k_end = min(K, k_first + QUARTERS * qk);
  const int tiles = k_end > k_first ? (k_end - k_first + BK - 1) / BK : 0;
  auto load = [&](int it) {
    const int k0 = k_first + it * BK;
    float* to = tile_sm + (it % STAGES) * STAGE_FLOATS;            // A's rows, then W's
    if (it < tiles) {
      if constexpr (VEC) {
#pragma unroll
        for (int idx = tid; idx < (BM + BN) * (BK / 4); idx += TILE_THREADS) {
          const int r = idx / (BK / 4), c = (idx % (BK / 4)) * 4, k = k0 + c;
          const bool of_a = r < BM;
          const int row = of_a ? m0 + r : n0 + r - BM;
          const bool in = row < (of_a ? M : N) && k < K;
          const float* src = of_a ? A : W;
          cp_async16_if(to + r * LINE + c, in ? src + (size_t)row * (of_a ? lda : ldw) + k : src, in);
        }
      } else {
#pragma unroll 4
        for (int idx = tid; idx < (BM + BN) * BK; idx += TILE_THREADS) {
          const int r = idx / BK, c = idx % BK, k = k0 + c;
          const bool of_a = r < BM;
          const int row = of_a ? m0 + r : n0 + r - BM;
          const bool in = row < (of_a ? M : N) && k < K;
          const float* src = of_a ? A : W;
          cp_async4_if(to + r * LINE + c, in ? src + (size_t)row * (of_a ? lda : ldw) + k : src, in);
        }
      }
    }
    cp_async_commit();
  };
  float sum[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) sum[i][j] = 0.f;
  for (int it = 0; it < STAGES - 1; ++it) load(it);
  // A thread has one run's and one quarter's sums in registers; what it has beside them lies in shared memory: the first
  // of a pair of quarters, and, of a block with all four, the first pair.
  float* kept = tile_sm + STAGES * STAGE_FLOATS + tid;             // [2][TM TN][TILE_THREADS]
  auto each = [&](auto&& f) {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) f(sum[i][j], kept[(i * TN + j) * TILE_THREADS], kept[(TM * TN + i * TN + j) * TILE_THREADS]);
  };
  int it = 0;
#pragma unroll 1
  for (int q = 0; q < QUARTERS; ++q) {
#pragma unroll 1
    for (const int end = min(tiles, (q + 1) * (qk / BK)); it < end; ++it) {
      cp_async_wait<STAGES - 2>();
      __syncthreads();
      load(it + STAGES - 1);
      const float* as = tile_sm + (it % STAGES) * STAGE_FLOATS + ty * LINE;
      const float* ws = tile_sm + (it % STAGES) * STAGE_FLOATS + (BM + tx) * LINE;
#pragma unroll 1
      for (int run = 0; run < BK; run += RUN) {
        f32x2 acc[TM][TN];
#pragma unroll
        for (int k = 0; k < RUN; k += 4) {
          ulonglong2 w[TN];
#pragma unroll
          for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(ws + 16 * j * LINE + run + k);
#pragma unroll
          for (int i = 0; i < TM; ++i) {
            const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(as + 8 * i * LINE + run + k);
            // (a sum's next step comes TN instructions later, past the latency of this one)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = fma2(a.x, w[j].x, k == 0 ? 0ull : acc[i][j]);
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = fma2(a.y, w[j].y, acc[i][j]);
          }
        }
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) sum[i][j] += both(acc[i][j]);
      }
    }
    if constexpr (QUARTERS == 4) {
      const bool last = it >= tiles;               // quarters behind it are empty: zeros, added as such
      if (q == 3) each([](float& v, float& one, float& pair) { v = pair + (one + v); });
      else if (q == 2 && last) each([](float& v, float&, float& pair) { v = pair + (v + 0.f); });
      else if (q == 1 && last) each([](float& v, float& one, float&) { v = (one + v) + 0.f; });
      else if (q == 1) each([](float& v, float& one, float& pair) { pair = one + v; v = 0.f; });
      else if (last) each([](float& v, float&, float&) { v += 0.f; });
      else each([](float& v, float& one, float&) { one = v; v = 0.f; });
      if (last) break;
    }
  }
  cp_async_wait<0>();
  if constexpr (KS == 1) {
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + 16 * j;
      if (n >= N) break;
      const float add = bias ? bias[n] : 0.f;
#pragma unroll
      for (int i = 0; i < TM; ++i)
        if (m0 + ty + 8 * i < M) C[(size_t)(m0 + ty + 8 * i) * ldc + n] = sum[i][j] + add;
    }
    return;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) tile_sm[(ty + 8 * i) * (BN + 1) + tx + 16 * j] = sum[i][j];
  cluster_sync();
  // each block of the cluster finishes its share of the rows
  constexpr int SHARE = BM / KS;
#pragma unroll 4
  for (int idx = tid; idx < SHARE * BN; idx += TILE_THREADS) {
    const int r = (int)blockIdx.z * SHARE + idx / BN, c = idx % BN;
    const float* p = tile_sm + r * (BN + 1) + c;
    const float v = (peer_f32(p, 0) + peer_f32(p, 1)) + (peer_f32(p, 2) + peer_f32(p, 3));
    if (m0 + r < M && n0 + c < N) C[(size_t)(m0 + r) * ldc + n0 + c] = v + (bias ? bias[n0 + c] : 0.f);
  }
  cluster_sync();                                  // nobody leaves while a peer may still read its sums
}

template <int TM, int TN, bool VEC, int KS>
static int launch_tile(float* C, const float* A, const float* W, const float* bias, int M, int N, int K, int lda,
                       int ldw, int ldc, cudaStream_t stream) {
  using Tl = Tile<TM, TN, KS>;
  constexpr int smem = Tl::BYTES;
  if (!allow_shared_memory<gemm_f32_kernel<TM, TN, VEC, KS>, smem>()) return HB_LAUNCH_FAILED;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((N + Tl::BN - 1) / Tl::BN, (M + Tl::BM - 1) / Tl::BM, KS);
  if (cfg.gridDim.y > 65535) return HB_BAD_ARGUMENT;
  cfg.blockDim = dim3(TILE_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = KS;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  // (no early launch: blocks that came while the kernel before holds the SMs would crowd where
  // room is and stay there for their long walk)
  cudaLaunchKernelEx(&cfg, gemm_f32_kernel<TM, TN, VEC, KS>, C, A, W, bias, M, N, K, lda, ldw, ldc);
  return hb_check_launch();
}

// Which of four: 4 x 4 outputs a thread (four blocks an SM) or 8 x 4 (three), a quarter of K a block (clusters of four)
// or all of it.  A block takes a time for each of its tiles and one beside them, of which a first block alone on an SM
// takes the part `alone` and the last round of blocks its part; `steps` is how far rounds of blocks stay together
// (the rest runs on evenly).  Microseconds (but for a constant), fitted to products of 17 to 4,096 rows, 64 to 151,936
// features and K of 17 to 4,864: what it chooses takes 1.004 of the best one's time on average, 1.10 at most.  One block a tile /
// four, µs, 8 x 4: 4,096 rows of 32,000 x 64 505 / 1,771, of 32,000 x 256 1,686 / 2,487, of 9,728 x 896 1,686 / 1,943; 4 x 4:
// 466 rows of 896 x 4,864 185 / 124, 64 rows of 1,000 x 333, whose rows are no whole 16-byte pieces, 21.0 / 8.1 (copied as they came, not
// under way beside the products, 42 / 14).
struct TileCost { int tile, ks; float each, block, alone, steps; };
template <bool VEC>
static int launch_tiles(float* C, const float* A, const float* W, const float* bias, int M, int N, int K, int lda,
                        int ldw, int ldc, int form, int sms, cudaStream_t stream) {
  static constexpr TileCost costs[] = {{44, 1, 1.93f, 1.8f, .28f, .66f}, {44, 4, 1.79f, 2.6f, .36f, .6f},
                                       {84, 1, 2.52f, 2.7f, .26f, .66f}, {84, 4, 2.49f, 3.2f, .89f, .73f}};
  int tile = form < 100 ? 84 : form / 10, ks = form % 10;
  if (form < 100) {
    float best = INFINITY;
    for (const TileCost& c : costs) {
      const int bm = c.tile == 44 ? 32 : 64, a_sm = c.tile == 44 ? 4 : 3, q = quarter_k(K) / BK, all = (K + BK - 1) / BK;
      if (((form == 44 || form == 84) && c.tile != form) || (M + bm - 1) / bm > 65535) continue;
      const int tiles = c.ks == 4 ? (q < all ? q : all) : all;
      const long blocks = (long)((N + 63) / 64) * ((M + bm - 1) / bm) * c.ks, slots = (long)sms * a_sm;
      const long full = blocks / slots, rest = blocks - full * slots;
      float rounds = (float)full;
      if (rest) rounds += c.alone + (1.f - c.alone) * ((rest + sms - 1) / sms) / a_sm;
      if (full) rounds = c.steps * rounds + (1.f - c.steps) * blocks / slots;
      const float time = rounds * (c.each * tiles + c.block);
      if (time < best) {
        best = time;
        tile = c.tile;
        ks = c.ks;
      }
    }
  }
  if (tile == 44) return ks == 1 ? launch_tile<4, 4, VEC, 1>(C, A, W, bias, M, N, K, lda, ldw, ldc, stream)
                                 : launch_tile<4, 4, VEC, 4>(C, A, W, bias, M, N, K, lda, ldw, ldc, stream);
  return ks == 1 ? launch_tile<8, 4, VEC, 1>(C, A, W, bias, M, N, K, lda, ldw, ldc, stream)
                 : launch_tile<8, 4, VEC, 4>(C, A, W, bias, M, N, K, lda, ldw, ldc, stream);
}

// MT rows of A a block: 0 if they do not fit its shared memory
template <int MT, int ROWS_W, bool AHEAD>
static int launch_rows_as(float* C, const float* A, const float* W, const float* bias, int M, int N, int K,
                          int lda, int ldw, int ldc, int sms, cudaStream_t stream, bool* fits) {
  const long runs = 4L * (quarter_k(K) / RUN);
  const long pieces = (runs + 31) / 32, rounds = (pieces + ROWS_MOST_WARPS - 1) / ROWS_MOST_WARPS;
  const int wpg = (int)((pieces + rounds - 1) / rounds);
  const int units = (N + ROWS_W - 1) / ROWS_W;
  auto smem_of = [&](int groups) {
    return ((long)MT * runs * ROWS_RUN + 2L * groups * ROWS_W * MT * (runs + 1)) * (long)sizeof(float);
  };
  // as many groups a block as eight warps hold, fewer where the blocks would leave SMs without one
  int groups = wpg >= 8 ? 1 : 8 / wpg;
  while (groups > 1 && ((long)units < (long)sms * groups || smem_of(groups) > ROWS_MOST_SMEM / 2)) --groups;
  const long smem = smem_of(groups);
  *fits = smem <= ROWS_MOST_SMEM;
  if (!*fits) return HB_OK;
  if (!allow_shared_memory<gemm_f32_rows_kernel<MT, ROWS_W, AHEAD>, ROWS_MOST_SMEM>()) return HB_LAUNCH_FAILED;
  const int resident = sms * (smem <= ROWS_MOST_SMEM / 2 && (MT <= 4 || ROWS_W <= 2) ? 2 : 1);
  const int blocks = (units + groups - 1) / groups;
  const dim3 grid(blocks < resident ? blocks : resident, (M + MT - 1) / MT);
  hb_launch(gemm_f32_rows_kernel<MT, ROWS_W, AHEAD>, grid, dim3(32 * wpg * groups), (size_t)smem, stream, C, A, W, bias,
            M, N, K, lda, ldw, ldc, wpg);
  return hb_check_launch();
}
// Four rows of W a warp where W is large, where A's rows leave an SM one block anyway, or where two would be more
// blocks of one warp, each with all of A, than SMs; else two with the next two on their way: less to wait for where a
// group has a few rows in all.  Two / four rows, µs: 9,728 x 896 at one row of A 9.6 / 8.5, three 11.6 / 10.7, six 15.8 /
// 15.2, but eight 17.4 / 18.6, and 151,936 x 896 at six 169 / 175 (one block an SM); 896 x 4,864 at one 9.0 / 6.7, six
// 15.7 / 13.4, eight 19.7 / 19.0; 1,024 x 4,096 at six 14.3 / 11.1; 512 x 128 at two 2.9 / 2.4; but 2,048 x 1,024 at one 3.4 / 3.5, three 3.8 / 4.3, 1,152 x 896 3.1 / 3.4, 3.8 / 4.2,
// 768 x 256 at two 2.5 / 2.6, 128 x 128 at three 1.8 / 2.1.
template <int MT>
static int launch_rows(float* C, const float* A, const float* W, const float* bias, int M, int N, int K,
                       int lda, int ldw, int ldc, int form, int sms, cudaStream_t stream, bool* fits) {
  const long runs = 4L * (quarter_k(K) / RUN);
  const bool large = (long)N * K >= 3 << 20 && (MT <= 4 || (MT <= 6 && (long)N * K < 32 << 20));
  const bool one_block = MT > 6 && 2 * MT * runs * ROWS_RUN * (long)sizeof(float) > ROWS_MOST_SMEM;
  const bool one_warp = MT <= 6 && runs <= 32 && N >= 256 && N < 4L * sms;
  if (form == 4 || (form != 2 && (large || one_block || one_warp)))
    return launch_rows_as<MT, 4, false>(C, A, W, bias, M, N, K, lda, ldw, ldc, sms, stream, fits);
  return launch_rows_as<MT, 2, true>(C, A, W, bias, M, N, K, lda, ldw, ldc, sms, stream, fits);
}

// few_rows: up to this many rows of A go through the kernel that streams W (16-byte rows only,
// K up to what a row of A may take of shared memory).  form: 0, or the one to take where there is a
// choice (2, 4: rows of W a warp; 44, 84: outputs a thread, M x N; 441, 444, 841, 844: and blocks a tile): the
// results are the same.
HB_EXPORT int hb_gemm_f32_as(float* C, const float* A, const float* W, const float* bias, int M, int N,
                             int K, int lda, int ldw, int ldc, int few_rows, int form, int sms, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return HB_OK;
  if (K <= 0 || sms <= 0) return HB_BAD_ARGUMENT;
  const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 &&
                   ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) == 0;
  // (more than eight rows read W twice, or, of a W with many rows, once in tiles: 9,728 x 896 at 16 rows 31 / 24 µs,
  // 1,152 x 896 9.2 / 9.0, but 12 8.4 / 9.0, and 1,024 x 512 at 16 5.0 / 6.8)
  if (vec && M <= few_rows && (M <= 8 || N < (M <= 12 ? 2048 : 1025) || form == 2 || form == 4)) {
    bool fits = false;
    int rc = HB_OK;
#define HB_ROWS(MT) rc = launch_rows<MT>(C, A, W, bias, M, N, K, lda, ldw, ldc, form, sms, stream, &fits)
    if (M > 12 || M == 7 || M == 8) HB_ROWS(8);
    else if (M > 4) HB_ROWS(6);
    if (!fits && M > 12) HB_ROWS(6);
    if (!fits && M > 3) HB_ROWS(4);
    if (!fits && M > 2) HB_ROWS(3);
    if (!fits && M > 1) HB_ROWS(2);
    if (!fits) HB_ROWS(1);
#undef HB_ROWS
    if (fits) return rc;
  }
  return vec ? launch_tiles<true>(C, A, W, bias, M, N, K, lda, ldw, ldc, form, sms, stream)
             : launch_tiles<false>(C, A, W, bias, M, N, K, lda, ldw, ldc, form, sms, stream);
}

HB_EXPORT int hb_gemm_f32(float* C, const float* A, const float* W, const float* bias, int M, int N,
                          int K, int lda, int ldw, int ldc, int few_rows, int sms, cudaStream_t stream) {
  return hb_gemm_f32_as(C, A, W, bias, M, N, K, lda, ldw, ldc, few_rows, 0, sms, stream);
}
