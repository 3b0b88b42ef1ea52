// True float32 matrix product on the FMA pipes: C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]).
// No tensor cores and no reduced-precision mode.  Every output element is summed in one order
// that depends on K alone: runs of RUN consecutive k, each from zero in the order of k; eight
// runs in order make a block's sum, and the blocks' sums are added in order.  Both kernels below
// keep that order, so a row's result does not depend on the other rows of the launch.
// (python/helios/exec/model.py:236-238, 250-251, 336-337, 493-496: y = x W^T + b with W
// stored [out, in].)
#include "common.cuh"

constexpr int RUN = 16;             // consecutive k of one partial sum
constexpr int RUNS = 8;             // runs of a block's sum

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

// ---------------------------------------------------------------- few rows
// Bound by reading W once.  A warp takes four rows of W and 32 runs of k, a run a lane: the 64
// bytes of a lane's run come straight into registers (16 loads of 16 bytes a lane, 8 KB a warp
// in flight), those of the warp's next rows before the sums of the present ones are put
// together.  A's rows lie in shared memory for the whole of K, runs RUN + 4 floats apart so that
// neighbouring lanes read different banks; each load of A serves four rows of W.  `wpg` warps
// share four rows of W; a block has up to eight warps.
// Chains over cold weights, 64 x 64 tiles with one order of k / this, µs: 151,936 x 896 (bound by
// memory at 83) 477 / 90 at one row, 116 at 4, 190 at 8; 9,728 x 896 76 / 12, 14.5, 21;
// 896 x 4,864 200 / 7.0, 14.6, 26; 896 x 896 38 / 3.7, 5.8, 6.5.
constexpr int ROWS_W = 4;                        // rows of W a warp
constexpr int ROWS_RUN = RUN + 4;
constexpr int ROWS_MOST_THREADS = 256;

template <int MT>
__global__ void __launch_bounds__(ROWS_MOST_THREADS, 2)
gemm_f32_rows_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W,
                     const float* __restrict__ bias, int M, int N, int K, int lda, int ldw, int ldc,
                     int wpg, int tiles) {
  extern __shared__ __align__(16) float rows_sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, threads = blockDim.x;
  const int groups = (threads >> 5) / wpg, g = warp / wpg, first_rb = warp - g * wpg;
  const int blocks = (K + RUN * RUNS - 1) / (RUN * RUNS), runs = blocks * RUNS;   // whole blocks of runs
  const int rounds = (runs + 32 * wpg - 1) / (32 * wpg);                          // 32-run pieces a warp takes
  const int tile_rows = groups * ROWS_W;
  const int line = runs * ROWS_RUN;                // floats of one row of A
  const int part_line = runs + 4;                  // floats of one output's partial sums
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
  for (int idx = tid; idx < MT * runs * (RUN / 4); idx += threads) {
    const int m = idx / (runs * (RUN / 4)), v = idx - m * (runs * (RUN / 4));
    const bool in = m0 + m < M && 4 * v < K;
    cp_async16_if(rows_sm + m * line + (v / (RUN / 4)) * ROWS_RUN + (v % (RUN / 4)) * 4,
                  in ? A + (size_t)(m0 + m) * lda + 4 * v : A, in);
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
            for (int r = 0; r < ROWS_W; ++r) {
              acc[r][m] = fmaf(a.x, w[r][i].x, acc[r][m]);
              acc[r][m] = fmaf(a.y, w[r][i].y, acc[r][m]);
              acc[r][m] = fmaf(a.z, w[r][i].z, acc[r][m]);
              acc[r][m] = fmaf(a.w, w[r][i].w, acc[r][m]);
            }
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
    // a block's eight runs, in order; the sum takes the first run's place
    for (int idx = tid; idx < tile_rows * MT * blocks; idx += threads) {
      float* p = sums + (idx / blocks) * part_line + (idx % blocks) * RUNS;
      const float4 u = *reinterpret_cast<const float4*>(p), v = *reinterpret_cast<const float4*>(p + 4);
      *p = ((((((u.x + u.y) + u.z) + u.w) + v.x) + v.y) + v.z) + v.w;
    }
    __syncthreads();
    for (int idx = tid; idx < tile_rows * MT; idx += threads) {
      const float* p = sums + idx * part_line;
      float total = 0.f;
      for (int b = 0; b < blocks; ++b) total += p[b * RUNS];
      const int n = (blockIdx.x + t * gridDim.x) * tile_rows + idx / MT, m = m0 + idx % MT;
      if (n < N && m < M) C[(size_t)m * ldc + n] = total + (bias ? bias[n] : 0.f);
    }
    // (the next tile's sums go to the other half of `part`; this half is written again only
    // behind two barriers of the next tile)
  }
}

// ---------------------------------------------------------------- many rows
// Bound by the FMA pipes.  64 x 64 outputs a block, 8 x 4 a thread; operands stay [row][k] in
// shared memory (rows 36 floats apart, so that neighbouring rows start in different banks),
// and a thread reads four k of a row at once: 12 loads for 128 multiply-adds.
constexpr int BM = 64, BN = 64, BK = 32, TM = 8, TN = 4, LINE = BK + 4;
constexpr int TILE_THREADS = (BM / TM) * (BN / TN);

template <bool VEC>
__global__ void __launch_bounds__(TILE_THREADS, 3)
gemm_f32_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W,
                const float* __restrict__ bias, int M, int N, int K, int lda, int ldw, int ldc) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ __align__(16) float As[2][BM][LINE];
  __shared__ __align__(16) float Ws[2][BN][LINE];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tx = tid % (BN / TN), ty = tid / (BN / TN);   // rows ty + 8 i of A, tx + 16 j of W
  auto load = [&](int k0, int b) {
    if constexpr (VEC) {
      for (int idx = tid; idx < BM * (BK / 4); idx += TILE_THREADS) {
        const int r = idx / (BK / 4), k = k0 + (idx % (BK / 4)) * 4;
        const bool a_in = m0 + r < M && k < K, w_in = n0 + r < N && k < K;
        cp_async16_if(&As[b][r][k - k0], a_in ? A + (size_t)(m0 + r) * lda + k : A, a_in);
        cp_async16_if(&Ws[b][r][k - k0], w_in ? W + (size_t)(n0 + r) * ldw + k : W, w_in);
      }
    } else {
      for (int idx = tid; idx < BM * BK; idx += TILE_THREADS) {
        const int r = idx / BK, k = k0 + idx % BK;
        As[b][r][k - k0] = (m0 + r < M && k < K) ? A[(size_t)(m0 + r) * lda + k] : 0.f;
        Ws[b][r][k - k0] = (n0 + r < N && k < K) ? W[(size_t)(n0 + r) * ldw + k] : 0.f;
      }
    }
    cp_async_commit();
  };
  static_assert(BM == BN, "one loop fills both tiles");
  float acc[TM][TN], block[TM][TN], total[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = block[i][j] = total[i][j] = 0.f;
  auto carry = [](float (&from)[TM][TN], float (&to)[TM][TN]) {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        to[i][j] += from[i][j];
        from[i][j] = 0.f;
      }
  };
  load(0, 0);
  int b = 0;
  for (int k0 = 0; k0 < K; k0 += BK) {
    cp_async_wait<0>();
    __syncthreads();
    if (k0 + BK < K) load(k0 + BK, b ^ 1);
#pragma unroll
    for (int run = 0; run < BK; run += RUN) {
#pragma unroll
      for (int k = run; k < run + RUN; k += 4) {
        float4 w[TN];
#pragma unroll
        for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const float4*>(&Ws[b][tx + (BN / TN) * j][k]);
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          const float4 a = *reinterpret_cast<const float4*>(&As[b][ty + (BM / TM) * i][k]);
#pragma unroll
          for (int j = 0; j < TN; ++j) {
            acc[i][j] = fmaf(a.x, w[j].x, acc[i][j]);
            acc[i][j] = fmaf(a.y, w[j].y, acc[i][j]);
            acc[i][j] = fmaf(a.z, w[j].z, acc[i][j]);
            acc[i][j] = fmaf(a.w, w[j].w, acc[i][j]);
          }
        }
      }
      carry(acc, block);
    }
    if ((k0 + BK) % (RUN * RUNS) == 0 || k0 + BK >= K) carry(block, total);
    b ^= 1;
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty + (BM / TM) * i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + (BN / TN) * j;
      if (n < N) C[(size_t)m * ldc + n] = total[i][j] + (bias ? bias[n] : 0.f);
    }
  }
}

// MT rows of A a block: 0 if they do not fit its shared memory
template <int MT>
static int launch_rows(float* C, const float* A, const float* W, const float* bias, int M, int N, int K,
                       int lda, int ldw, int ldc, int sms, cudaStream_t stream, bool* fits) {
  const long runs = (long)(K + RUN * RUNS - 1) / (RUN * RUNS) * RUNS;
  const long pieces = (runs + 31) / 32, rounds = (pieces + 7) / 8;
  const int wpg = (int)((pieces + rounds - 1) / rounds);
  // more rows of W a block where the blocks still cover the SMs
  int groups = 1;
  while (2 * groups * wpg <= 8 && (long)N >= (long)sms * 2 * groups * ROWS_W) groups *= 2;
  const long smem = ((long)MT * runs * ROWS_RUN + 2L * groups * ROWS_W * MT * (runs + 4)) * (long)sizeof(float);
  *fits = smem <= 200 * 1024;
  if (!*fits) return HB_OK;
  if (cudaFuncSetAttribute(gemm_f32_rows_kernel<MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return HB_LAUNCH_FAILED;
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
    if (M > 4) HB_ROWS(8);
    if (!fits && M > 2) HB_ROWS(4);
    if (!fits && M > 1) HB_ROWS(2);
    if (!fits) HB_ROWS(1);
#undef HB_ROWS
    if (fits) return rc;
  }
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (grid.y > 65535) return HB_BAD_ARGUMENT;
  if (vec) hb_launch(gemm_f32_kernel<true>, grid, dim3(TILE_THREADS), 0, stream, C, A, W, bias, M, N, K, lda, ldw, ldc);
  else hb_launch(gemm_f32_kernel<false>, grid, dim3(TILE_THREADS), 0, stream, C, A, W, bias, M, N, K, lda, ldw, ldc);
  return hb_check_launch();
}
