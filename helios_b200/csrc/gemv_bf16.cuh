// Products of one to four tokens with a small weight matrix, on the FMA pipes: y[t, n] = x[t] . w[n],
// with the epilogues that decode steps use of the tensor-core kernel (same meaning, see there).
//
// A step of a small model is a chain of such products, each over in less time than the tensor-core
// kernel takes around its sums (barriers, tensor memory, copies through shared memory, a cluster's
// two barriers).  Here a warp takes two rows of w (four for a gated unit, two features' gate and up
// rows), a lane 16 bytes of a row at a time, straight into registers, and asks for its first rows before
// the kernel before is done, as the tensor-core kernel does; then x, the sums, one barrier, and a thread a
// feature and token finishes.  A block has 16 features, or eight with twice the warps a row where blocks of 16 leave SMs
// idle (`gemv_block_features`, ops.py), or 18 or 20 of a gated unit where those need a round of blocks less (two blocks
// an SM); its features share a slot of the sums of squares.  Chains over cold weights, tensor cores / this, µs at one
// token: 1,152 x 896 4.95 / 2.05, 896 x 896 4.05 / 2.03, 896 x 4,864 6.06 / 3.56, 2,048 x 8,192 9.98 / 8.69.  Gated units, 16
// features a block / this: 2 x 4,864 x 896 6.7 / 6.1, 2 x 5,300 x 1,024 7.2 / 6.6, 2 x 5,900 x 512 5.3 / 4.2.  Beyond one round
// the last blocks run alone, and the tensor-core kernel is ahead; which products come here, and both sides'
// figures, stand at `gemv_features` (ops.py).
#pragma once
#include "common.cuh"

namespace {

struct GemvArgs {
  void* out;                   // [T, ldo] bfloat16 or float32
  const __nv_bfloat16* x;      // [T, ldx]
  const __nv_bfloat16* w;      // [N or 2 N, ldw]
  const float* bias;
  float* residual;
  const float* norm_weight;
  float* sumsq_out;            // [T, slots_out]
  const float* sumsq_in;       // [T, slots_in]
  int T, N, K, ldx, ldw, ldo, up_row, out_f32, slots_in, slots_out;
  float eps;
};

__device__ __forceinline__ float gemv_dot8(const uint4& a, const uint4& b, float acc) {
  const uint32_t u[4] = {a.x, a.y, a.z, a.w}, v[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    acc = fmaf(__uint_as_float(u[i] << 16), __uint_as_float(v[i] << 16), acc);
    acc = fmaf(__uint_as_float(u[i] & 0xffff0000u), __uint_as_float(v[i] & 0xffff0000u), acc);
  }
  return acc;
}

// TT: tokens (T <= TT); WF: warps side by side, two features each; KS: warps that share a row; EPI: EPI_STORE,
// EPI_GLU or EPI_GELU
template <int TT, int WF, int KS, int EPI>
__global__ void __launch_bounds__(32 * WF * KS, WF * KS <= 10 && TT == 1 ? 2 : 1)
gemv_bf16_kernel(GemvArgs a) {
  constexpr int GEMV_F = 2 * WF;                 // features a block
  constexpr bool GATED = EPI != EPI_STORE;
  constexpr int ROWS = GATED ? 4 : 2;            // rows a warp: features f, f + 1, then their up rows
  constexpr int PRE = GATED ? 2 : 4;             // 256-element steps a register buffer holds
  __shared__ float part[KS][ROWS / 2][TT][GEMV_F];
  __shared__ float scale[TT];
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ks = warp / WF, f0 = 2 * (warp % WF), n0 = blockIdx.x * GEMV_F;
  const int steps = (a.K + 255) / 256;
  uint4 w[2][PRE][ROWS];
  auto load_w = [&](uint4 (&buf)[PRE][ROWS], int s0) {      // this warp's steps s0 .. s0 + PRE - 1
#pragma unroll
    for (int i = 0; i < PRE; ++i) {
      const int k = ((s0 + i) * KS + ks) * 256 + 8 * lane;
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const int n = n0 + f0 + (r & 1);
        const size_t row = (size_t)(n + (r >= 2 ? a.up_row : 0));
        buf[i][r] = (k < a.K && n < a.N) ? __ldg(reinterpret_cast<const uint4*>(a.w + row * a.ldw + k))
                                         : make_uint4(0, 0, 0, 0);
      }
    }
  };
  float acc[ROWS][TT];
#pragma unroll
  for (int r = 0; r < ROWS; ++r)
#pragma unroll
    for (int t = 0; t < TT; ++t) acc[r][t] = 0.f;
  auto multiply = [&](const uint4 (&buf)[PRE][ROWS], int s0) {
    uint4 x[PRE][TT];
#pragma unroll
    for (int i = 0; i < PRE; ++i) {
      const int k = ((s0 + i) * KS + ks) * 256 + 8 * lane;
#pragma unroll
      for (int t = 0; t < TT; ++t)
        x[i][t] = (k < a.K && t < a.T) ? __ldcg(reinterpret_cast<const uint4*>(a.x + (size_t)t * a.ldx + k))
                                       : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int i = 0; i < PRE; ++i)
#pragma unroll
      for (int t = 0; t < TT; ++t)
#pragma unroll
        for (int r = 0; r < ROWS; ++r) acc[r][t] = gemv_dot8(buf[i][r], x[i][t], acc[r][t]);
  };
  const int mine = (steps - ks + KS - 1) / KS;             // steps of this warp
  load_w(w[0], 0);
  load_w(w[1], PRE);
  pdl_wait();
  // what a finishing thread needs from memory beyond the sums goes out under them
  const int et = tid / GEMV_F, ef = tid % GEMV_F, en = n0 + ef;
  const bool finishes = tid < TT * GEMV_F && et < a.T && en < a.N;
  float old = 0.f, bias_n = 0.f, weight_n = 0.f;
  if (finishes) {
    if (a.residual) old = __ldcg(a.residual + (size_t)et * a.N + en);
    if (a.bias) bias_n = a.bias[en];
    if (a.norm_weight) weight_n = a.norm_weight[en];
  }
  float squares = 0.f;
  if (a.sumsq_in && warp < a.T) {
#pragma unroll 4
    for (int j = lane; j < a.slots_in; j += 32) squares += __ldcg(a.sumsq_in + (size_t)warp * a.slots_in + j);
  }
  for (int s = 0; s < mine; s += 2 * PRE) {
    multiply(w[0], s);
    if (s + 2 * PRE < mine) load_w(w[0], s + 2 * PRE);
    if (s + PRE < mine) {
      multiply(w[1], s + PRE);
      if (s + 3 * PRE < mine) load_w(w[1], s + 3 * PRE);
    }
  }
  if (a.sumsq_in && warp < a.T) {
    squares = warp_sum(squares);
    if (lane == 0) scale[warp] = rsqrtf(squares / (float)a.K + a.eps);
  }
#pragma unroll
  for (int r = 0; r < ROWS; ++r)
#pragma unroll
    for (int t = 0; t < TT; ++t) {
      const float v = warp_sum(acc[r][t]);
      if (lane == 0) part[ks][r >> 1][t][f0 + (r & 1)] = v;
    }
  __syncthreads();
  if (tid >= TT * GEMV_F) return;                          // whole warps, or part of the first one
  float val = 0.f, up = 0.f;
#pragma unroll
  for (int i = 0; i < KS; ++i) {
    val += part[i][0][et][ef];
    if (GATED) up += part[i][ROWS / 2 - 1][et][ef];
  }
  if (a.sumsq_in && et < a.T) {
    val *= scale[et];
    up *= scale[et];
  }
  if (GATED) val = finishes ? glu_value<EPI>(val, up) : 0.f;
  val += bias_n;
  if (a.residual) {
    val += old;
    if (finishes) a.residual[(size_t)et * a.N + en] = val;
    if (a.norm_weight) {
      if (finishes) reinterpret_cast<__nv_bfloat16*>(a.out)[(size_t)et * a.ldo + en] = __float2bfloat16_rn(val * weight_n);
      float sq = finishes ? val * val : 0.f;
      constexpr uint32_t lanes = TT * GEMV_F >= 32 ? 0xffffffffu : (1u << (TT * GEMV_F % 32)) - 1u;
      static_assert(GATED || GEMV_F == 8 || GEMV_F == 16, "a token's features are neighbouring lanes");
#pragma unroll
      for (int o = GEMV_F / 2; o > 0; o >>= 1) sq += __shfl_xor_sync(lanes, sq, o);
      if (ef == 0 && et < a.T) a.sumsq_out[(size_t)et * a.slots_out + blockIdx.x] = sq;
    }
  } else if (finishes) {
    if (a.out_f32) reinterpret_cast<float*>(a.out)[(size_t)et * a.ldo + en] = val;
    else reinterpret_cast<__nv_bfloat16*>(a.out)[(size_t)et * a.ldo + en] = __float2bfloat16_rn(val);
  }
}

template <int TT, int WF, int KS, int EPI>
int launch_gemv_as(const GemvArgs& a, cudaStream_t stream) {
  // with sums of squares all slots of the last 128 features are written
  const int features = a.sumsq_out ? (a.N + 127) / 128 * 128 : a.N;
  hb_launch(gemv_bf16_kernel<TT, WF, KS, EPI>, dim3((features + 2 * WF - 1) / (2 * WF)), dim3(32 * WF * KS), 0, stream, a);
  return hb_check_launch();
}
template <int TT>
int launch_gemv(const GemvArgs& a, int block_features, cudaStream_t stream) {
  if (block_features == 8)
    return a.K > 2048 ? launch_gemv_as<TT, 4, 4, EPI_STORE>(a, stream) : launch_gemv_as<TT, 4, 2, EPI_STORE>(a, stream);
  return a.K > 2048 ? launch_gemv_as<TT, 8, 2, EPI_STORE>(a, stream) : launch_gemv_as<TT, 8, 1, EPI_STORE>(a, stream);
}
template <int EPI>
int launch_gemv_gated(const GemvArgs& a, int sms, cudaStream_t stream) {
  if (a.K > 2048) return launch_gemv_as<1, 8, 2, EPI>(a, stream);
  // blocks of nine or ten warps where those need a round less (two blocks an SM)
  auto rounds = [&](int features) { return ((a.N + features - 1) / features + 2 * sms - 1) / (2 * sms); };
  if (rounds(16) > rounds(18)) return launch_gemv_as<1, 9, 1, EPI>(a, stream);
  if (rounds(16) > rounds(20)) return launch_gemv_as<1, 10, 1, EPI>(a, stream);
  return launch_gemv_as<1, 8, 1, EPI>(a, stream);
}

}  // namespace

// As hb_gemm_bf16_fused, for 1 to 4 tokens (one with a gated unit); rows of x and w in whole 16-byte pieces.
// block_features: 16, or 8 (not for a gated unit); a block leaves one partial sum of squares a token,
// 128 / block_features to 128 features.
HB_EXPORT int hb_gemv_bf16(void* out, const void* x, const void* w, const float* bias, int T, int N, int K, int ldx,
                           int ldw, int ldo, int glu, int up_row, int out_f32, float* residual,
                           const float* norm_weight, float* sumsq_out, const float* sumsq_in, int slots_in, float eps,
                           int block_features, int sms, cudaStream_t stream) {
  if (T <= 0 || N <= 0) return HB_OK;
  if ((block_features != 8 && block_features != 16) || sms <= 0) return HB_BAD_ARGUMENT;
  if (T > 4 || K <= 0 || K % 8 || ldx % 8 || ldw % 8 || glu < 0 || glu > 2 ||
      (glu && (T > 1 || bias || residual || out_f32)) || (residual && out_f32) || (norm_weight && (!residual || !sumsq_out || !out)) || (!residual && !out) ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15))
    return HB_BAD_ARGUMENT;
  GemvArgs a;
  a.out = out; a.x = (const __nv_bfloat16*)x; a.w = (const __nv_bfloat16*)w; a.bias = bias;
  a.residual = residual; a.norm_weight = norm_weight; a.sumsq_out = norm_weight ? sumsq_out : nullptr;
  a.sumsq_in = sumsq_in; a.T = T; a.N = N; a.K = K; a.ldx = ldx; a.ldw = ldw; a.ldo = ldo; a.up_row = up_row;
  a.out_f32 = out_f32; a.slots_in = slots_in; a.slots_out = 128 / block_features * ((N + 127) / 128); a.eps = eps;
  if (glu) return glu == 1 ? launch_gemv_gated<EPI_GLU>(a, sms, stream) : launch_gemv_gated<EPI_GELU>(a, sms, stream);
  return T == 1 ? launch_gemv<1>(a, block_features, stream)
       : T == 2 ? launch_gemv<2>(a, block_features, stream) : launch_gemv<4>(a, block_features, stream);
}
