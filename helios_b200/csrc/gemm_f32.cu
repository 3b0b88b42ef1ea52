// True float32 matrix product on the FMA pipes: C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]).
// No tensor cores and no reduced-precision mode.  Every output element is summed in one order
// that depends on K alone: runs of RUN consecutive k, each from zero in the order of k; the runs
// of a quarter of K in order; and (q0 + q1) + (q2 + q3).  Both kernels below keep that order, so
// a row's result does not depend on the other rows of the launch.
// (python/helios/exec/model.py:236-238, 250-251, 336-337, 493-496: y = x W^T + b with W
// stored [out, in].)
#include "common.cuh"

constexpr int RUN = 16;             // consecutive k of one partial sum
constexpr int BK = 32;              // k of a tile of the kernel for many rows: a quarter is whole tiles
static_assert(BK % RUN == 0, "");
// k of a quarter (the last ones may be short or empty)
__host__ __device__ __forceinline__ int quarter_k(int K) { return (K + 4 * BK - 1) / (4 * BK) * BK; }

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
// ... of 16 bytes of zeros where `in` does not hold (nothing is read then)
__device__ __forceinline__ void cp_async16_if(void* smem, const void* gmem, bool in) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(in ? 16 : 0));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

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
// Bound by reading W once.  A warp takes four rows of W and 32 runs of k, a run a lane: the 64
// bytes of a lane's run come straight into registers (16 loads of 16 bytes a lane, 8 KB a warp
// in flight), those of the warp's next rows before the sums of the present ones are put
// together.  A's rows lie in shared memory for the whole of K, runs RUN + 4 floats apart so that
// neighbouring lanes read different banks; each load of A serves four rows of W.  `wpg` warps
// share four rows of W; a block has up to eight warps.
// Chains over cold weights, one 64 x 64 tile a block walking K alone / this, µs: 151,936 x 896 (bound
// by memory at 83) 477 / 89 at one row, 133 at 4, 210 at 8; 9,728 x 896 76 / 11.5, 15, 23;
// 896 x 4,864 200 / 7.1, 13, 23; 896 x 896 38 / 3.5, 5.3, 6.5.
constexpr int ROWS_W = 4;                        // rows of W a warp
constexpr int ROWS_RUN = RUN + 4;
constexpr int ROWS_MOST_THREADS = 256;
constexpr int ROWS_MOST_SMEM = 200 * 1024;       // what a block may take of shared memory

template <int MT>
__global__ void __launch_bounds__(ROWS_MOST_THREADS, 2)
gemm_f32_rows_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W,
                     const float* __restrict__ bias, int M, int N, int K, int lda, int ldw, int ldc,
                     int wpg, int tiles) {
  extern __shared__ __align__(16) float rows_sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, threads = blockDim.x;
  const int groups = (threads >> 5) / wpg, g = warp / wpg, first_rb = warp - g * wpg;
  const int q_runs = quarter_k(K) / RUN, runs = 4 * q_runs;
  const int rounds = (runs + 32 * wpg - 1) / (32 * wpg);                          // 32-run pieces a warp takes
  const int tile_rows = groups * ROWS_W;
  const int line = runs * ROWS_RUN;                // floats of one row of A
  const int part_line = runs + 1;                  // floats of one output's partial sums
  float* part = rows_sm + MT * line;               // [2][tile_rows * MT][part_line]
  const int part_size = tile_rows * MT * part_line;
  const int m0 = blockIdx.y * MT;
  const int my_tiles = ((int)blockIdx.x < tiles) ? (tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;

  pdl_launch_dependents();
  float4 w[ROWS_W][RUN / 4];
  auto load = [&](int t, int round) {
    const int n0 = (blockIdx.x + t * gridDim.x) * tile_rows + g * ROWS_W;
    const int k0 = ((first_rb + round * wpg) * 32 + lane) * RUN;
#pragma unroll
    for (int r = 0; r < ROWS_W; ++r) {
      const float* src = W + (size_t)(n0 + r) * ldw + k0;
#pragma unroll
      for (int i = 0; i < RUN / 4; ++i)
        w[r][i] = (t < my_tiles && n0 + r < N && k0 + 4 * i < K) ? __ldg(reinterpret_cast<const float4*>(src) + i)
                                                                 : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  {  // the first rows of W on their way to L2 under the kernel before (no further: W need not be a
     // weight that nobody writes)
    const int n0 = blockIdx.x * tile_rows + g * ROWS_W, k0 = (first_rb * 32 + lane) * RUN;
    if (k0 < K)
      for (int r = 0; r < ROWS_W; ++r)
        if (n0 + r < N) asm volatile("prefetch.global.L2 [%0];" ::"l"(W + (size_t)(n0 + r) * ldw + k0));
  }
  pdl_wait();
  load(0, 0);
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

  for (int t = 0; t < my_tiles; ++t) {
    float* sums = part + (t & 1) * part_size;
    for (int round = 0; round < rounds; ++round) {
      const int run = (first_rb + round * wpg) * 32 + lane;
      float acc[ROWS_W][MT];
#pragma unroll
      for (int r = 0; r < ROWS_W; ++r)
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[r][m] = 0.f;
      if (run < runs) {
        const float* a_run = rows_sm + run * ROWS_RUN;
#pragma unroll
        for (int i = 0; i < RUN / 4; ++i)
#pragma unroll
          for (int m = 0; m < MT; ++m) {
            const float4 a = *reinterpret_cast<const float4*>(a_run + m * line + 4 * i);
#pragma unroll
            for (int r = 0; r < ROWS_W; ++r) acc[r][m] = fmaf(a.x, w[r][i].x, acc[r][m]);
#pragma unroll
            for (int r = 0; r < ROWS_W; ++r) acc[r][m] = fmaf(a.y, w[r][i].y, acc[r][m]);
#pragma unroll
            for (int r = 0; r < ROWS_W; ++r) acc[r][m] = fmaf(a.z, w[r][i].z, acc[r][m]);
#pragma unroll
            for (int r = 0; r < ROWS_W; ++r) acc[r][m] = fmaf(a.w, w[r][i].w, acc[r][m]);
          }
      }
      if (round + 1 < rounds) load(t, round + 1);
      else load(t + 1, 0);
      if (run < runs) {
#pragma unroll
        for (int r = 0; r < ROWS_W; ++r)
#pragma unroll
          for (int m = 0; m < MT; ++m) sums[((g * ROWS_W + r) * MT + m) * part_line + run] = acc[r][m];
      }
    }
    __syncthreads();
    // a thread a quarter, the four of an output side by side
    for (int base = tid - lane; base < 4 * tile_rows * MT; base += threads) {
      const int idx = base + lane, out = idx / 4;
      const bool in = out < tile_rows * MT;
      const float* p = sums + (in ? out : 0) * part_line + (idx % 4) * q_runs;
      float q = 0.f;
#pragma unroll 4
      for (int r = 0; r < q_runs; ++r) q += p[r];
      q += __shfl_xor_sync(0xffffffffu, q, 1);
      q += __shfl_xor_sync(0xffffffffu, q, 2);
      const int n = (blockIdx.x + t * gridDim.x) * tile_rows + out / MT, m = m0 + out % MT;
      if (in && idx % 4 == 0 && n < N && m < M) C[(size_t)m * ldc + n] = q + (bias ? bias[n] : 0.f);
    }
    // (the next tile's sums go to the other half of `part`; this half is written again only
    // behind the next tile's barrier)
  }
}

// ---------------------------------------------------------------- many rows
// Bound by the FMA pipes.  64 x 64 outputs a block of four warps, 8 x 4 a thread (8 x 8 takes all
// registers: two warps a scheduler, and slower).  Operands stay [row][k] in shared memory
// (rows 36 floats apart, so that neighbouring rows start in different banks), three tiles in
// flight.  `ks` blocks of a cluster share the quarters of K, where the tiles alone would leave
// SMs idle, and add their sums through distributed shared memory.
// 466 rows, µs, one block a tile with 4 x 4 outputs a thread / this: 9,728 x 896 392 / 259 (31
// TFLOP/s), 896 x 4,864 350 / 170, 1,152 x 896 72 / 45; 64 rows: 200 / 60 at 896 x 4,864.
constexpr int BM = 64, BN = 64, TM = 8, TN = 4, LINE = BK + 4, STAGES = 3;
constexpr int TILE_THREADS = (BM / TM) * (BN / TN);
constexpr int STAGE_FLOATS = (BM + BN) * LINE;
static_assert(STAGES * STAGE_FLOATS >= BM * (BN + 1), "the sums of a block lie where its tiles were");

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

template <bool VEC>
__global__ void __launch_bounds__(TILE_THREADS, 3)
gemm_f32_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W,
                const float* __restrict__ bias, int M, int N, int K, int lda, int ldw, int ldc, int ks) {
  pdl_wait();
  extern __shared__ __align__(16) float tile_sm[];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tx = tid % (BN / TN), ty = tid / (BN / TN);   // rows ty + 8 i of A, tx + 16 j of W
  const int qk = quarter_k(K), q_tiles = qk / BK, quarters = 4 / ks;
  const int k_first = (int)blockIdx.z * quarters * qk;     // the cluster lies along z: rank = blockIdx.z
  const int k_end = min(K, k_first + quarters * qk);
  const int tiles = k_end > k_first ? (k_end - k_first + BK - 1) / BK : 0;
  auto load = [&](int it) {
    const int k0 = k_first + it * BK;
    float* as = tile_sm + (it % STAGES) * STAGE_FLOATS;
    float* ws = as + BM * LINE;
    if (it < tiles) {
      if constexpr (VEC) {
        for (int idx = tid; idx < BM * (BK / 4); idx += TILE_THREADS) {
          const int r = idx / (BK / 4), c = (idx % (BK / 4)) * 4, k = k0 + c;
          const bool a_in = m0 + r < M && k < K, w_in = n0 + r < N && k < K;
          cp_async16_if(as + r * LINE + c, a_in ? A + (size_t)(m0 + r) * lda + k : A, a_in);
          cp_async16_if(ws + r * LINE + c, w_in ? W + (size_t)(n0 + r) * ldw + k : W, w_in);
        }
      } else {
        for (int idx = tid; idx < BM * BK; idx += TILE_THREADS) {
          const int r = idx / BK, c = idx % BK, k = k0 + c;
          as[r * LINE + c] = (m0 + r < M && k < K) ? A[(size_t)(m0 + r) * lda + k] : 0.f;
          ws[r * LINE + c] = (n0 + r < N && k < K) ? W[(size_t)(n0 + r) * ldw + k] : 0.f;
        }
      }
    }
    cp_async_commit();
  };
  static_assert(BM == BN, "one loop fills both tiles");
  float acc[TM][TN], sum[TM][TN], pair[TM][TN], first[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = sum[i][j] = pair[i][j] = first[i][j] = 0.f;
  for (int it = 0; it < STAGES - 1; ++it) load(it);
  int it = 0;
  for (int q = 0; q < quarters; ++q) {
    for (int end = min(tiles, (q + 1) * q_tiles); it < end; ++it) {
      cp_async_wait<STAGES - 2>();
      __syncthreads();
      load(it + STAGES - 1);
      const float* as = tile_sm + (it % STAGES) * STAGE_FLOATS + ty * LINE;
      const float* ws = tile_sm + (it % STAGES) * STAGE_FLOATS + (BM + tx) * LINE;
#pragma unroll 1
      for (int run = 0; run < BK; run += RUN) {
#pragma unroll
        for (int k = run; k < run + RUN; k += 4) {
          float4 w[TN];
#pragma unroll
          for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const float4*>(ws + (BN / TN) * j * LINE + k);
#pragma unroll
          for (int i = 0; i < TM; ++i) {
            const float4 a = *reinterpret_cast<const float4*>(as + (BM / TM) * i * LINE + k);
            // (a sum's next step comes TN instructions later, past the latency of this one)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.x, w[j].x, acc[i][j]);
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.y, w[j].y, acc[i][j]);
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.z, w[j].z, acc[i][j]);
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.w, w[j].w, acc[i][j]);
          }
        }
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) {
            sum[i][j] += acc[i][j];
            acc[i][j] = 0.f;
          }
      }
    }
    // quarters 0 and 2 begin a pair (a block that has one quarter passes it on as it is)
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        pair[i][j] = (q & 1) ? pair[i][j] + sum[i][j] : sum[i][j];
        if (q == 1) first[i][j] = pair[i][j];
        sum[i][j] = 0.f;
      }
  }
  cp_async_wait<0>();
  if (ks == 1) {
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int m = m0 + ty + (BM / TM) * i;
      if (m >= M) continue;
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const int n = n0 + tx + (BN / TN) * j;
        if (n < N) C[(size_t)m * ldc + n] = (first[i][j] + pair[i][j]) + (bias ? bias[n] : 0.f);
      }
    }
    return;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) tile_sm[(ty + (BM / TM) * i) * (BN + 1) + tx + (BN / TN) * j] = pair[i][j];
  cluster_sync();
  // each block of the cluster finishes its share of the rows
  const int share = BM / ks;
  for (int idx = tid; idx < share * BN; idx += TILE_THREADS) {
    const int r = (int)blockIdx.z * share + idx / BN, c = idx % BN;
    const float* p = tile_sm + r * (BN + 1) + c;
    float v = peer_f32(p, 0) + peer_f32(p, 1);
    if (ks == 4) v += peer_f32(p, 2) + peer_f32(p, 3);
    if (m0 + r < M && n0 + c < N) C[(size_t)(m0 + r) * ldc + n0 + c] = v + (bias ? bias[n0 + c] : 0.f);
  }
  cluster_sync();                                  // nobody leaves while a peer may still read its sums
}

template <bool VEC>
static int launch_tiles(float* C, const float* A, const float* W, const float* bias, int M, int N, int K, int lda,
                        int ldw, int ldc, int sms, cudaStream_t stream) {
  constexpr int smem = STAGES * STAGE_FLOATS * (int)sizeof(float);
  if (!allow_shared_memory<gemm_f32_kernel<VEC>, smem>()) return HB_LAUNCH_FAILED;
  const long tiles = (long)((N + BN - 1) / BN) * ((M + BM - 1) / BM);
  // three blocks fit an SM: the quarters go to blocks of their own until all SMs are full a few
  // times over, if each then still has some tiles to walk
  int ks = 1;
  while (ks < 4 && tiles * ks < 8L * sms && K >= ks * 4 * BK) ks *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((N + BN - 1) / BN, (M + BM - 1) / BM, ks);
  if (cfg.gridDim.y > 65535) return HB_BAD_ARGUMENT;
  cfg.blockDim = dim3(TILE_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = ks;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  // (no early launch: blocks that came while the kernel before holds the SMs would crowd where
  // room is and stay there for their long walk)
  cudaLaunchKernelEx(&cfg, gemm_f32_kernel<VEC>, C, A, W, bias, M, N, K, lda, ldw, ldc, ks);
  return hb_check_launch();
}

// MT rows of A a block: 0 if they do not fit its shared memory
template <int MT>
static int launch_rows(float* C, const float* A, const float* W, const float* bias, int M, int N, int K,
                       int lda, int ldw, int ldc, int sms, cudaStream_t stream, bool* fits) {
  const long runs = 4L * (quarter_k(K) / RUN);
  const long pieces = (runs + 31) / 32, rounds = (pieces + 7) / 8;
  const int wpg = (int)((pieces + rounds - 1) / rounds);
  // more rows of W a block where the blocks still cover the SMs
  int groups = 1;
  while (2 * groups * wpg <= 8 && (long)N >= (long)sms * 2 * groups * ROWS_W) groups *= 2;
  const long smem = ((long)MT * runs * ROWS_RUN + 2L * groups * ROWS_W * MT * (runs + 1)) * (long)sizeof(float);
  *fits = smem <= ROWS_MOST_SMEM;
  if (!*fits) return HB_OK;
  if (!allow_shared_memory<gemm_f32_rows_kernel<MT>, ROWS_MOST_SMEM>()) return HB_LAUNCH_FAILED;
  const int tiles = (N + groups * ROWS_W - 1) / (groups * ROWS_W);
  // a block takes up to four tiles (A is staged once for them), fewer where that leaves SMs idle
  int per_block = tiles / (2 * sms);
  per_block = per_block < 1 ? 1 : per_block > 4 ? 4 : per_block;
  const dim3 grid((tiles + per_block - 1) / per_block, (M + MT - 1) / MT);
  hb_launch(gemm_f32_rows_kernel<MT>, grid, dim3(32 * wpg * groups), (size_t)smem, stream, C, A, W, bias, M, N, K,
            lda, ldw, ldc, wpg, tiles);
  return hb_check_launch();
}

// few_rows: up to this many rows of A go through the kernel that streams W (16-byte rows only,
// K up to what a row of A may take of shared memory)
HB_EXPORT int hb_gemm_f32(float* C, const float* A, const float* W, const float* bias, int M, int N,
                          int K, int lda, int ldw, int ldc, int few_rows, int sms, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return HB_OK;
  if (K <= 0 || sms <= 0) return HB_BAD_ARGUMENT;
  const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 &&
                   ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) == 0;
  if (vec && M <= few_rows) {
    bool fits = false;
    int rc = HB_OK;
#define HB_ROWS(MT) rc = launch_rows<MT>(C, A, W, bias, M, N, K, lda, ldw, ldc, sms, stream, &fits)
    if (M > 6) HB_ROWS(8);
    else if (M > 4) HB_ROWS(6);
    if (!fits && M > 3) HB_ROWS(4);
    if (!fits && M > 2) HB_ROWS(3);
    if (!fits && M > 1) HB_ROWS(2);
    if (!fits) HB_ROWS(1);
#undef HB_ROWS
    if (fits) return rc;
  }
  return vec ? launch_tiles<true>(C, A, W, bias, M, N, K, lda, ldw, ldc, sms, stream)
             : launch_tiles<false>(C, A, W, bias, M, N, K, lda, ldw, ldc, sms, stream);
}
