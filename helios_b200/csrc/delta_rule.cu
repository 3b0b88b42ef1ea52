// A recurrent mixer with a matrix state per head, written by the gated delta rule with one
// decay per key channel.  Per token and head (k, q unit vectors, q also times dk^-1/2):
//
//   S <- g (.) S            (g in (0,1)^dk scales the rows of S [dk, dv])
//   u  = beta (v - S^T k)
//   S <- S + k u^T
//   o  = S^T q              (the read-out sees this token's write)
//
// The columns of S never mix: eight threads own a column (or two), an eighth of its dk values in
// registers each, and walk the request's tokens in order, so a request's numbers do not depend on
// how its tokens were cut into steps or on the rest of the batch.  In bfloat16 that holds on each side of one
// boundary only: long portions go by chunks of tokens (`delta_chunk.cuh`, `delta_rule_by_chunks` in ops.py says
// which), whose sums have another order.  State, decays, gates, unit norms and
// the recurrence are float32.
//
// Kernels: `causal_conv_silu` (short causal convolution over time per channel + silu, the
// taps - 1 inputs before a step's first token taken from the request's slot),
// `causal_conv_state` (leaves the last taps - 1 inputs in the slot; steps of single tokens do both in
// `causal_conv_step`), `delta_prepare` and `delta_rule` (the recurrence; `delta_step` both for single tokens;
// `delta_chunk.cuh` for 16-bit activations and portions of many tokens) and `gated_rmsnorm` (o / rms(o) * weight * sigmoid(gate) per head).
#include "common.cuh"
#include "causal_conv.cuh"

// ---------------------------------------------------------------- short convolution
// x [T, ld] (the first `channels` columns), w [channels, taps] (the last column is the
// current token's), bias [channels] or null, conv state of a slot at state + slot * state_stride: [channels, taps - 1],
// oldest first.  out [T, channels].
template <typename T>
__global__ void causal_conv_silu_kernel(T* __restrict__ out, const T* __restrict__ x, int ld,
                                        const float* __restrict__ w, const float* __restrict__ bias,
                                        const float* __restrict__ state,
                                        long state_stride, const int* __restrict__ seq_of_token,
                                        const int* __restrict__ cu_tokens,
                                        const int* __restrict__ slots, int n_tokens, int channels,
                                        int taps) {
  pdl_launch_dependents();
  pdl_wait();
  const size_t total = (size_t)n_tokens * channels;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (size_t)gridDim.x * blockDim.x) {
    const int t = (int)(idx / channels), c = (int)(idx - (size_t)t * channels);
    const int s = seq_of_token[t];
    const int local = t - cu_tokens[s];
    const float* st = state + (size_t)slots[s] * state_stride + (size_t)c * (taps - 1);
    float acc = bias ? bias[c] : 0.f;
    for (int j = 0; j < taps; ++j) {
      const int src = local - (taps - 1) + j;
      const float v = src >= 0 ? to_float(x[(size_t)(t - (taps - 1) + j) * ld + c])
                               : st[(taps - 1) + src];
      acc = fmaf(w[(size_t)c * taps + j], v, acc);
    }
    out[idx] = from_float<T>(acc / (1.f + expf(-acc)));
  }
}

// The same for bfloat16 rows that come in 16-byte pieces (channels, row stride and addresses
// multiples of eight values) and 2 to 4 taps: a thread takes eight neighbouring channels of
// CONV_TOKENS consecutive tokens, so that the channels' weights (16-byte loads) and the rows
// the tokens share are read once; each channel's sum in the order of the kernel above.
constexpr int CONV_TOKENS = 4;

template <int TAPS>
__global__ void __launch_bounds__(128)
causal_conv_silu_bf16x8_kernel(__nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ x,
                               int ld, const float* __restrict__ w, const float* __restrict__ bias,
                               const float* __restrict__ state, long state_stride,
                               const int* __restrict__ seq_of_token,
                               const int* __restrict__ cu_tokens, const int* __restrict__ slots,
                               int n_tokens, int channels) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int ROWS = CONV_TOKENS + TAPS - 1;
  const int pieces = channels / 8;
  const int groups = (n_tokens + CONV_TOKENS - 1) / CONV_TOKENS;
  const size_t total = (size_t)groups * pieces;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (size_t)gridDim.x * blockDim.x) {
    const int tg = (int)(idx / pieces), c = (int)(idx - (size_t)tg * pieces) * 8;
    const int t0 = tg * CONV_TOKENS;
    // where the tokens stand in their requests: two loads, one after the other, so they go out first and
    // together, not token by token between the sums
    int seq[CONV_TOKENS];
#pragma unroll
    for (int u = 0; u < CONV_TOKENS; ++u) seq[u] = seq_of_token[min(t0 + u, n_tokens - 1)];
    // the eight channels' weights are 8 x TAPS consecutive floats from a 32-byte boundary
    float wr[8 * TAPS];
#pragma unroll
    for (int i = 0; i < 2 * TAPS; ++i) {
      const float4 q = *reinterpret_cast<const float4*>(w + (size_t)c * TAPS + 4 * i);
      wr[4 * i] = q.x; wr[4 * i + 1] = q.y; wr[4 * i + 2] = q.z; wr[4 * i + 3] = q.w;
    }
    float b8[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) b8[e] = bias ? bias[c + e] : 0.f;
    // rows t0 - (TAPS - 1) .. t0 + CONV_TOKENS - 1 of the step, where they exist
    float v[ROWS][8];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const int row = t0 - (TAPS - 1) + r;
      if (row >= 0 && row < n_tokens) {
        const uint4 raw = *reinterpret_cast<const uint4*>(x + (size_t)row * ld + c);
        const uint32_t in[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&in[e]));
          v[r][2 * e] = f.x;
          v[r][2 * e + 1] = f.y;
        }
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[r][e] = 0.f;
      }
    }
    int place[CONV_TOKENS];
#pragma unroll
    for (int u = 0; u < CONV_TOKENS; ++u) place[u] = t0 + u - cu_tokens[seq[u]];
#pragma unroll
    for (int u = 0; u < CONV_TOKENS; ++u) {
      const int t = t0 + u;
      if (t >= n_tokens) break;
      const int s = seq[u], local = place[u];
      float acc[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = b8[e];
      if (local >= TAPS - 1) {
#pragma unroll
        for (int j = 0; j < TAPS; ++j) {
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[e] = fmaf(wr[e * TAPS + j], v[u + j][e], acc[e]);
        }
      } else {
        // the request's first tokens of this step: the inputs before them are in its slot
        const float* st = state + (size_t)slots[s] * state_stride + (size_t)c * (TAPS - 1);
#pragma unroll
        for (int j = 0; j < TAPS; ++j) {
          const int src = local - (TAPS - 1) + j;
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float in = src >= 0 ? v[u + j][e] : st[(size_t)e * (TAPS - 1) + (TAPS - 1) + src];
            acc[e] = fmaf(wr[e * TAPS + j], in, acc[e]);
          }
        }
      }
      uint32_t res[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const __nv_bfloat162 o = __floats2bfloat162_rn(acc[2 * e] / (1.f + expf(-acc[2 * e])),
                                                       acc[2 * e + 1] / (1.f + expf(-acc[2 * e + 1])));
        res[e] = *reinterpret_cast<const uint32_t*>(&o);
      }
      *reinterpret_cast<uint4*>(out + (size_t)t * channels + c) = make_uint4(res[0], res[1], res[2], res[3]);
    }
  }
}

// Steps of single tokens: the sum and the shift of the slot's inputs in one launch, four neighbouring
// channels a thread, whose inputs, weights and outputs are whole pieces (`causal_conv_silu` and
// `causal_conv_state` read the same inputs one after the other, value by value: 64 requests of 6,144
// channels 13.4 µs, so 5.1).  A request's sum per channel has the same order.
template <typename T, int TAPS>
__global__ void __launch_bounds__(128)
causal_conv_step_kernel(T* __restrict__ out, const T* __restrict__ x, int ld, const float* __restrict__ w,
                        const float* __restrict__ bias, float* __restrict__ state, long state_stride,
                        const int* __restrict__ cu_tokens, const int* __restrict__ slots, int channels) {
  pdl_launch_dependents();
  pdl_wait();
  const int s = blockIdx.y, c = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (c >= channels) return;
  const int t0 = cu_tokens[s], t1 = cu_tokens[s + 1];
  if (t0 >= t1) return;
  float* st = state + (size_t)slots[s] * state_stride + (size_t)c * (TAPS - 1);
  __align__(16) float in[4 * (TAPS - 1)];
  __align__(16) float wr[4 * TAPS];
#pragma unroll
  for (int i = 0; i < TAPS; ++i) *reinterpret_cast<float4*>(wr + 4 * i) = *reinterpret_cast<const float4*>(w + (size_t)c * TAPS + 4 * i);
#pragma unroll
  for (int i = 0; i < TAPS - 1; ++i) *reinterpret_cast<float4*>(in + 4 * i) = *reinterpret_cast<const float4*>(st + 4 * i);
  for (int t = t0; t < t1; ++t) {
    float v[4], y[4];
    const T* xr = x + (size_t)t * ld + c;
    if constexpr (sizeof(T) == 4) {
      const float4 a = *reinterpret_cast<const float4*>(xr);
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    } else {
      const uint2 raw = *reinterpret_cast<const uint2*>(xr);
      const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
      const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
      v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float* own = in + e * (TAPS - 1);
      float acc = bias ? bias[c + e] : 0.f;
#pragma unroll
      for (int j = 0; j < TAPS - 1; ++j) acc = fmaf(wr[e * TAPS + j], own[j], acc);
      acc = fmaf(wr[e * TAPS + TAPS - 1], v[e], acc);
      y[e] = acc / (1.f + expf(-acc));
#pragma unroll
      for (int j = 0; j + 1 < TAPS - 1; ++j) own[j] = own[j + 1];
      own[TAPS - 2] = v[e];
    }
    T* dst = out + (size_t)t * channels + c;
    if constexpr (sizeof(T) == 4) {
      *reinterpret_cast<float4*>(dst) = make_float4(y[0], y[1], y[2], y[3]);
    } else {
      const __nv_bfloat162 a = __floats2bfloat162_rn(y[0], y[1]), b = __floats2bfloat162_rn(y[2], y[3]);
      uint2 packed;
      packed.x = *reinterpret_cast<const uint32_t*>(&a);
      packed.y = *reinterpret_cast<const uint32_t*>(&b);
      *reinterpret_cast<uint2*>(dst) = packed;
    }
  }
#pragma unroll
  for (int i = 0; i < TAPS - 1; ++i) *reinterpret_cast<float4*>(st + 4 * i) = *reinterpret_cast<const float4*>(in + 4 * i);
}

HB_EXPORT int hb_causal_conv_silu(void* out, const void* x, int ld, const float* w, const float* bias,
                                  float* state,
                                  long state_stride, const int* seq_of_token, const int* cu_tokens,
                                  const int* slots, int n_tokens, int n_seqs, int channels, int taps,
                                  int act_dt, cudaStream_t stream) {
  if (n_tokens <= 0 || channels <= 0) return HB_OK;
  if (taps < 1 || ld < channels) return HB_BAD_ARGUMENT;
  const size_t piece = act_dt == HB_BF16 ? 8 : 16;
  if (n_tokens == n_seqs && n_seqs <= 65535 && taps >= 2 && taps <= 4 && channels % 4 == 0 && ld % 4 == 0 &&
      state_stride % 4 == 0 && ((reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(state)) & 15) == 0 &&
      (reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(x)) % piece == 0) {
    const dim3 grid1((channels / 4 + 127) / 128, n_seqs);
#define HB_CONV_STEP(TP)                                                                                        \
    HB_DISPATCH_DTYPE(act_dt, TA,                                                                               \
      hb_launch(causal_conv_step_kernel<TA, TP>, grid1, dim3(128), 0, stream, (TA*)out, (const TA*)x, ld, w,     \
                bias, state, state_stride, cu_tokens, slots, channels))
    if (taps == 2) HB_CONV_STEP(2);
    else if (taps == 3) HB_CONV_STEP(3);
    else HB_CONV_STEP(4);
#undef HB_CONV_STEP
    return hb_check_launch();
  }
  const size_t total = (size_t)n_tokens * channels;
  // steps of few tokens keep a thread a (token, channel): more threads, shorter chains of loads
  if (act_dt == HB_BF16 && n_tokens >= 64 && channels % 8 == 0 && ld % 8 == 0 && taps >= 2 && taps <= 4 &&
      ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0) {
    size_t vblocks = ((size_t)((n_tokens + CONV_TOKENS - 1) / CONV_TOKENS) * (channels / 8) + 127) / 128;
    if (vblocks > 148 * 32) vblocks = 148 * 32;
#define HB_CONV8(TP)                                                                                          \
    hb_launch(causal_conv_silu_bf16x8_kernel<TP>, dim3((unsigned)vblocks), dim3(128), 0, stream,              \
              (__nv_bfloat16*)out, (const __nv_bfloat16*)x, ld, w, bias, (const float*)state, state_stride,   \
              seq_of_token, cu_tokens, slots, n_tokens, channels)
    if (taps == 2) HB_CONV8(2);
    else if (taps == 3) HB_CONV8(3);
    else HB_CONV8(4);
#undef HB_CONV8
  } else {
    size_t blocks = (total + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    HB_DISPATCH_DTYPE(act_dt, TA,
      hb_launch(causal_conv_silu_kernel<TA>, dim3((unsigned)blocks), dim3(256), 0, stream, (TA*)out,
                (const TA*)x, ld, w, bias, (const float*)state, state_stride, seq_of_token, cu_tokens, slots,
                n_tokens, channels, taps));
  }
  if (taps > 1) {
    const size_t total2 = (size_t)n_seqs * channels;
    size_t blocks2 = (total2 + 255) / 256;
    if (blocks2 > 148 * 16) blocks2 = 148 * 16;
    HB_DISPATCH_DTYPE(act_dt, TA,
      hb_launch(causal_conv_state_kernel<TA>, dim3((unsigned)blocks2), dim3(256), 0, stream, state,
                state_stride, (const TA*)x, ld, cu_tokens, slots, n_seqs, channels, taps));
  }
  return hb_check_launch();
}

// ---------------------------------------------------------------- the recurrence
// Two kernels, and one that does both for steps of single tokens.  `delta_prepare` is parallel over
// (token, head): unit-norm k and q (q also times dk^-1/2), the decays g = exp(-exp(A_log) softplus(a + dt_bias)) and the write strength
// beta = sigmoid(b), all float32, left as kqg [T, heads, 3, dkp] (dkp = dk rounded up to 4;
// the padding holds k = q = 0, g = 1) and (beta, k . q) [T, heads, 2].  `delta_rule` then walks each
// request's tokens in order: a block owns 16 (or 32) columns of one head's S, eight threads one
// column (or two) in registers (an eighth of its dk rows each); the staged rows of 16 tokens arrive in
// shared memory by 16-byte cp.async one chunk ahead, the values of the next chunk wait in
// registers, and the two sums over dk run as four partial sums a thread and three shuffles
// (their order depends on dk alone, not on the step or the batch).
// Bound by the chain of a token: products, shuffles, the write.  So the columns of one request
// are spread over as many SMs as there are (one prompt of 16 heads of 128 x 128: 128 blocks of
// four warps; with 64 columns a block and four threads a column it was 32 blocks), and the
// products go two an instruction.  2,048 tokens 1,428 -> 447 µs, of 8 heads of 64 x 64 912 -> 314 (with
// conversions of the next chunk's values, and its beta stored from registers, 527 and 372).
constexpr int DR_CHUNK = 16;        // tokens staged in shared memory at a time
constexpr int DR_PARTS = 8;         // threads a column of S is spread over
// Columns of S a block owns, and columns a thread has a share of.  Where every block has an SM of its
// own, 16 and one: a token's chain bounds the walk, and is shortest so.  With several blocks an SM its
// shared-memory path does (a 16-byte load takes four cycles whatever it broadcasts; 212 of 345 cycles
// a token), and a row's piece is read once for two columns; 32 columns a block where that leaves two
// blocks an SM.  One column a thread / two, µs: one request of 2,048 tokens 447 / 498; 3 of 700 328 /
// 284; 24 of 40 150 / 110; 64 of 8 130 / 103.  Keys of more than 128 values take one column a thread (two
// do not fit its registers) and are padded to 160, 192 or 256 (8 heads of 160 x 160, padded to 256 / 160,
// µs: one request of 2,048 tokens 770 / 491, 24 of 40 187 / 114, 64 of 8 175 / 92).
constexpr int DR_COLS = 16, DR_COLS_WIDE = 32;

__device__ __forceinline__ void dr_cp_async16(void* smem, const void* gmem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void dr_cp_async8(void* smem, const void* gmem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem));
}

// A warp's norms of one (token, head): 1 / |k|, dk^-1/2 / |q| and k . q of the unit vectors
// (the scan reads o = (g (.) S)^T q + u (k . q) off ONE pass over S).
struct DeltaNorms { float kn, qn, kq; };
template <typename T>
__device__ __forceinline__ DeltaNorms delta_norms(const T* kr, const T* qr, int dk, int lane) {
  float kk = 0.f, qq = 0.f, kq = 0.f;
  for (int i = lane; i < dk; i += 32) {
    const float kv = to_float(kr[i]), qv = to_float(qr[i]);
    kk = fmaf(kv, kv, kk);
    qq = fmaf(qv, qv, qq);
    kq = fmaf(kv, qv, kq);
  }
  DeltaNorms n;
  n.kn = rsqrtf(warp_sum(kk) + 1e-6f);
  n.qn = rsqrtf(warp_sum(qq) + 1e-6f) * rsqrtf((float)dk);
  n.kq = warp_sum(kq) * n.kn * n.qn;
  return n;
}
__device__ __forceinline__ float delta_decay(float a, float rate) {
  const float sp = a > 20.f ? a : log1pf(expf(a));
  return expf(-rate * sp);
}
__device__ __forceinline__ float delta_beta(float raw) { return 1.f / (1.f + expf(-raw)); }

// qkv [T, qkv_ld]: q at q_off + kh * dk, k at k_off + kh * dk (after convolution and silu).
// beta_raw [T, beta_ld] at column h (before the sigmoid), a_raw [T, a_ld] at column h * dk
// (before dt_bias and softplus).
template <typename T>
__global__ void __launch_bounds__(128)
delta_prepare_kernel(float* __restrict__ kqg, float* __restrict__ beta, const T* __restrict__ qkv,
                     int qkv_ld, int q_off, int k_off, const T* __restrict__ beta_raw, int beta_ld,
                     const T* __restrict__ a_raw, int a_ld, const float* __restrict__ a_log,
                     const float* __restrict__ dt_bias, int n_rows, int heads, int kv_heads, int dk,
                     int dkp) {
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= n_rows) return;
  const int t = row / heads, h = row - t * heads;
  const int kh = h / (heads / kv_heads);
  const T* kr = qkv + (size_t)t * qkv_ld + k_off + (size_t)kh * dk;
  const T* qr = qkv + (size_t)t * qkv_ld + q_off + (size_t)kh * dk;
  const DeltaNorms nm = delta_norms(kr, qr, dk, lane);
  const float rate = expf(a_log[h]);
  float* dst = kqg + (size_t)row * 3 * dkp;
  for (int i = lane; i < dkp; i += 32) {
    float kv = 0.f, qv = 0.f, gv = 1.f;
    if (i < dk) {
      kv = to_float(kr[i]) * nm.kn;
      qv = to_float(qr[i]) * nm.qn;
      gv = delta_decay(to_float(a_raw[(size_t)t * a_ld + (size_t)h * dk + i]) + dt_bias[(size_t)h * dk + i], rate);
    }
    dst[i] = kv;
    dst[dkp + i] = qv;
    dst[2 * dkp + i] = gv;
  }
  if (lane == 0) {
    beta[2 * row] = delta_beta(to_float(beta_raw[(size_t)t * beta_ld + h]));
    beta[2 * row + 1] = nm.kq;
  }
}

// Two float32 operations an instruction, each rounded as the single one is.
__device__ __forceinline__ uint64_t dr_fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t dr_mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t dr_pack(float x, float y) {
  return (uint64_t)__float_as_uint(x) | ((uint64_t)__float_as_uint(y) << 32);
}
__device__ __forceinline__ float dr_lo(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float dr_hi(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }

// v at qkv[t, v_off + h * dv + col].  S of a slot at state + slot * state_stride,
// [heads, dk, dv].  o [T, heads * dv] float32.  A column of S is held by DR_PARTS neighbouring
// threads: thread `part` keeps the rows 4 (DR_PARTS m + part) .. + 3, and the two sums over dk
// are finished with shuffles.  A thread has W (1 or 2) columns.  COLS and W change which block and
// thread own a column, never a sum's order.
// MANY: for launches of more blocks than SMs.  A request's blocks follow one another, so that those of a
// long request lie on SMs of their own; and the state's columns go in whole 16-byte pieces (`in_pieces`) by
// way of the second staging buffer.  A warp's threads hold four (or eight) neighbouring columns of eight rows,
// so that their own loads fetch half a sector each, which is most of the time of a few tokens a request.
// Value by value / so, 16 heads of 128 x 128, µs: 64 requests of 4 tokens 70 / 56, of 2 62 / 47, of 8 95 / 77; 7 of one
// token beside one of 500 223 / 139.  4 heads of 256 x 256: 64 of 8 123 / 109.  Keys of at most 64 values gain less
// than the longer code costs their walk (3 requests of 700 tokens, 8 heads of 64 x 64, 112 / 122).
template <typename T, int DK, int COLS, int W, bool MANY>
__global__ void __launch_bounds__(COLS * DR_PARTS / W)
delta_rule_kernel(float* __restrict__ o, const float* __restrict__ kqg, const float* __restrict__ beta,
                  const T* __restrict__ qkv, int qkv_ld, int v_off, float* __restrict__ state,
                  long state_stride, const int* __restrict__ cu_tokens, const int* __restrict__ slots,
                  int heads, int dk, int dkp, int dv, int in_pieces) {
  // Neither launched early nor releasing the next kernel early: a long prompt of one request
  // is a few blocks that run for a long time.  Launched while the kernel before still holds
  // the SMs they land two to an SM wherever room is, and share its issue slots for all that
  // time; the blocks of a dependent released at the start would wait beside them as long.
  pdl_wait();
  extern __shared__ __align__(16) float dr_sm[];
  constexpr int THREADS = COLS * DR_PARTS / W, STEP = 4 * DR_PARTS;
  constexpr int G = DK / STEP;                      // float4 groups a thread holds
  constexpr int VT = DR_CHUNK / DR_PARTS;           // values of a chunk a thread fetches
  constexpr int ROW = 3 * DK;                       // staged floats a token: k, q, g of DK rows each
  static_assert(DK % STEP == 0 && DR_CHUNK % DR_PARTS == 0, "");
  float* stage_buf = dr_sm;                         // [2][CHUNK][ROW]
  float* bs = dr_sm + 2 * DR_CHUNK * ROW;           // [2][CHUNK][2]: beta, k . q
  float* vs = bs + 4 * DR_CHUNK;                    // [2][CHUNK][COLS]
  int s = blockIdx.x, h = blockIdx.y, col_block = blockIdx.z;
  if constexpr (MANY) {
    const int col_blocks = (dv + COLS - 1) / COLS;
    s = blockIdx.x / col_blocks / heads;
    h = blockIdx.x / col_blocks - s * heads;
    col_block = blockIdx.x % col_blocks;
  }
  const int part = threadIdx.x % DR_PARTS, lcol = threadIdx.x / DR_PARTS;
  const int col = col_block * COLS + W * lcol;
  bool live[W];
#pragma unroll
  for (int w = 0; w < W; ++w) live[w] = col + w < dv;
  const int t0 = cu_tokens[s], n = cu_tokens[s + 1] - t0;
  float* S_g = state + (size_t)slots[s] * state_stride + (size_t)h * dk * dv;
  const T* v_head = qkv + v_off + (size_t)h * dv;

  uint64_t S[W][G][2];
  if constexpr (!MANY) {
#pragma unroll
  for (int m = 0; m < G; ++m)
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int w = 0; w < W; ++w) {
        const int i = STEP * m + 4 * part + 2 * e;
        S[w][m][e] = dr_pack((live[w] && i < dk) ? S_g[(size_t)i * dv + col + w] : 0.f,
                             (live[w] && i + 1 < dk) ? S_g[(size_t)(i + 1) * dv + col + w] : 0.f);
      }
  }
  // the staged rows behind dkp hold nothing: k = q = g = 0 there, once for all tokens
  auto clear_padding = [&] {
  for (int idx = threadIdx.x; idx < 2 * DR_CHUNK * 3 * (DK - dkp); idx += THREADS)
    stage_buf[idx / (DK - dkp) * DK + dkp + idx % (DK - dkp)] = 0.f;
  };
  if constexpr (!MANY) clear_padding();

  // (nothing here waits for a load: a warp issues in order, and a conversion or a store of what was
  // just asked for would hold up the tokens of the chunk that is there)
  auto stage = [&](int c0, int b) {
    const int nc = min(DR_CHUNK, n - c0);
    float* dst = stage_buf + b * DR_CHUNK * ROW;
    const float* src = kqg + ((size_t)(t0 + c0) * heads + h) * 3 * dkp;
    const size_t token_step = (size_t)heads * 3 * dkp;
    if (dkp == DK) {
      for (int idx = threadIdx.x; idx < nc * (ROW / 4); idx += THREADS) {
        const int j = idx / (ROW / 4), v = idx % (ROW / 4);
        dr_cp_async16(dst + j * ROW + v * 4, src + j * token_step + v * 4);
      }
    } else {
      const int vecs = dkp / 4;
      for (int idx = threadIdx.x; idx < nc * 3 * vecs; idx += THREADS) {
        const int r = idx / vecs, v = idx - r * vecs, j = r / 3;    // r = 3 j + (k, q or g)
        dr_cp_async16(dst + r * DK + v * 4, src + j * token_step + (r - 3 * j) * dkp + v * 4);
      }
    }
    for (int j = threadIdx.x; j < nc; j += THREADS)
      dr_cp_async8(bs + 2 * (b * DR_CHUNK + j), beta + 2 * ((size_t)(t0 + c0 + j) * heads + h));
  };
  // the columns' thread `part` fetches the values of tokens part, part + DR_PARTS, ... of a chunk
  T v_next[VT][W];
  auto fetch_v = [&](int c0) {
#pragma unroll
    for (int jj = 0; jj < VT; ++jj) {
      const T* v = v_head + (size_t)(t0 + min(c0 + DR_PARTS * jj + part, n - 1)) * qkv_ld;
#pragma unroll
      for (int w = 0; w < W; ++w) v_next[jj][w] = v[live[w] ? col + w : 0];
    }
  };

  const bool pieces = MANY && in_pieces;
  constexpr int TLINE = COLS + 4;
  static_assert(!MANY || DK * TLINE <= DR_CHUNK * ROW, "");
  if constexpr (MANY) {
    if (n <= 0) return;
    float* tile = stage_buf + DR_CHUNK * ROW;
    if (pieces) {
      for (int idx = threadIdx.x; idx < dk * (COLS / 4); idx += THREADS) {
        const int i = idx / (COLS / 4), c = 4 * (idx % (COLS / 4));
        if (col_block * COLS + c < dv)
          dr_cp_async16(tile + i * TLINE + c, S_g + (size_t)i * dv + col_block * COLS + c);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::);
    stage(0, 0);
    fetch_v(0);
    asm volatile("cp.async.commit_group;\n" ::);
    if (pieces) {
      asm volatile("cp.async.wait_group 1;\n" ::);
      __syncthreads();
    }
    const float* from = pieces ? tile + W * lcol : S_g + col;
    const int line = pieces ? TLINE : dv;
#pragma unroll
    for (int m = 0; m < G; ++m)
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int w = 0; w < W; ++w) {
          const int i = STEP * m + 4 * part + 2 * e;
          S[w][m][e] = dr_pack((live[w] && i < dk) ? from[(size_t)i * line + w] : 0.f,
                               (live[w] && i + 1 < dk) ? from[(size_t)(i + 1) * line + w] : 0.f);
        }
    if (pieces && dkp < DK) __syncthreads();           // the zeros go where the tile lies
    clear_padding();
  } else {
    if (n > 0) {
      stage(0, 0);
      fetch_v(0);
    }
    asm volatile("cp.async.commit_group;\n" ::);
  }
  int b = 0;
  float* o_next = o + (size_t)t0 * heads * dv + (size_t)h * dv + col;
  const size_t o_step = (size_t)heads * dv;
  for (int c0 = 0; c0 < n; c0 += DR_CHUNK) {
    const int nc = min(DR_CHUNK, n - c0);
    asm volatile("cp.async.wait_group 0;\n" ::);
#pragma unroll
    for (int jj = 0; jj < VT; ++jj)
#pragma unroll
      for (int w = 0; w < W; ++w)
        vs[(b * DR_CHUNK + DR_PARTS * jj + part) * COLS + W * lcol + w] = to_float(v_next[jj][w]);
    __syncthreads();
    if (c0 + DR_CHUNK < n) {
      stage(c0 + DR_CHUNK, b ^ 1);
      fetch_v(c0 + DR_CHUNK);
    }
    asm volatile("cp.async.commit_group;\n" ::);
    const float* rows = stage_buf + b * DR_CHUNK * ROW + 4 * part;
    const float* bq = bs + 2 * b * DR_CHUNK;
    const float* vc = vs + b * DR_CHUNK * COLS + W * lcol;
    // a token's row pieces are read one token ahead, so that the chain of a token is the
    // products, the shuffles and the write alone
    struct Token { ulonglong2 k[G], q[G], g[G]; float2 bq; float v[W]; };
    auto fetch = [&](Token& x, int j) {
      const float* r = rows + j * ROW;
#pragma unroll
      for (int m = 0; m < G; ++m) {
        x.k[m] = *reinterpret_cast<const ulonglong2*>(r + STEP * m);
        x.q[m] = *reinterpret_cast<const ulonglong2*>(r + DK + STEP * m);
        x.g[m] = *reinterpret_cast<const ulonglong2*>(r + 2 * DK + STEP * m);
      }
      x.bq = *reinterpret_cast<const float2*>(bq + 2 * j);
      if constexpr (W == 2) {
        const float2 v = *reinterpret_cast<const float2*>(vc + j * COLS);
        x.v[0] = v.x;
        x.v[1] = v.y;
      } else {
        x.v[0] = vc[j * COLS];
      }
    };
    // one pass: S <- g (.) S with the sums S^T k and S^T q; then u, the read-out
    // o = S^T q + u (k . q) (what S^T q is after the write), and the write S += k u, which
    // nothing waits for until the next token's pass
    auto token = [&](const Token& x, Token& ahead, int j_ahead) {
      uint64_t d01[W] = {}, d23[W] = {}, e01[W] = {}, e23[W] = {};
#pragma unroll
      for (int m = 0; m < G; ++m)
#pragma unroll
        for (int w = 0; w < W; ++w) {
          S[w][m][0] = dr_mul2(S[w][m][0], x.g[m].x);
          S[w][m][1] = dr_mul2(S[w][m][1], x.g[m].y);
          d01[w] = dr_fma2(S[w][m][0], x.k[m].x, d01[w]);
          d23[w] = dr_fma2(S[w][m][1], x.k[m].y, d23[w]);
          e01[w] = dr_fma2(S[w][m][0], x.q[m].x, e01[w]);
          e23[w] = dr_fma2(S[w][m][1], x.q[m].y, e23[w]);
        }
      fetch(ahead, j_ahead);
      float dot[W], rd[W], u[W];
#pragma unroll
      for (int w = 0; w < W; ++w) {
        dot[w] = (dr_lo(d01[w]) + dr_hi(d01[w])) + (dr_lo(d23[w]) + dr_hi(d23[w]));
        rd[w] = (dr_lo(e01[w]) + dr_hi(e01[w])) + (dr_lo(e23[w]) + dr_hi(e23[w]));
      }
#pragma unroll
      for (int p = 1; p < DR_PARTS; p *= 2) {
#pragma unroll
        for (int w = 0; w < W; ++w) dot[w] += __shfl_xor_sync(0xffffffffu, dot[w], p);
#pragma unroll
        for (int w = 0; w < W; ++w) rd[w] += __shfl_xor_sync(0xffffffffu, rd[w], p);
      }
#pragma unroll
      for (int w = 0; w < W; ++w) {
        u[w] = x.bq.x * (x.v[w] - dot[w]);
        const uint64_t uu = dr_pack(u[w], u[w]);
#pragma unroll
        for (int m = 0; m < G; ++m) {
          S[w][m][0] = dr_fma2(x.k[m].x, uu, S[w][m][0]);
          S[w][m][1] = dr_fma2(x.k[m].y, uu, S[w][m][1]);
        }
        if (live[w] && part == 0) o_next[w] = fmaf(u[w], x.bq.y, rd[w]);
      }
      o_next += o_step;
    };
    Token x0, x1;
    fetch(x0, 0);
    int j = 0;
    for (; j + 1 < nc; j += 2) {
      token(x0, x1, j + 1);
      token(x1, x0, min(j + 2, nc - 1));
    }
    if (j < nc) token(x0, x1, j);
    b ^= 1;
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  if (pieces) {
    __syncthreads();                                   // nobody reads staged rows any more
    float* to = stage_buf + W * lcol;
#pragma unroll
    for (int w = 0; w < W; ++w)
      if (live[w]) {
#pragma unroll
        for (int m = 0; m < G; ++m)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int i = STEP * m + 4 * part + 2 * e;
            if (i < dk) to[i * TLINE + w] = dr_lo(S[w][m][e]);
            if (i + 1 < dk) to[(i + 1) * TLINE + w] = dr_hi(S[w][m][e]);
          }
      }
    __syncthreads();
    for (int idx = threadIdx.x; idx < dk * (COLS / 4); idx += THREADS) {
      const int i = idx / (COLS / 4), c = 4 * (idx % (COLS / 4));
      if (col_block * COLS + c < dv)
        *reinterpret_cast<float4*>(S_g + (size_t)i * dv + col_block * COLS + c) =
            *reinterpret_cast<const float4*>(stage_buf + i * TLINE + c);
    }
    return;
  }
#pragma unroll
  for (int w = 0; w < W; ++w)
    if (live[w]) {
#pragma unroll
      for (int m = 0; m < G; ++m)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int i = STEP * m + 4 * part + 2 * e;
          if (i < dk) S_g[(size_t)i * dv + col + w] = dr_lo(S[w][m][e]);
          if (i + 1 < dk) S_g[(size_t)(i + 1) * dv + col + w] = dr_hi(S[w][m][e]);
        }
    }
}

// Steps of single tokens (decode), bound by reading and writing the states once: a block owns
// the whole S of a (request, head), 4 LANES columns of it, the LANES threads of a `part` the rows a
// thread of that part owns above, four neighbouring columns a thread, so that a row is one access of
// up to 512 bytes and all of a block's rows are in flight at once.  The preparation is done here as
// well (every warp computes the norms; nothing goes through memory), and every sum has the order of the
// two kernels above: dot products by element of a group of four, then the parts pairwise.  LANES is 32, or
// 16 or 8 where the values of a head are 64 or 32 columns, so that no lane is idle (160 requests, two
// kernels / 32 lanes / this, µs: 16 heads of 24 x 24 14.3 / 25.2 / 9.2,
// 8 of 64 x 64 15.8 / 17.4 / 12.0).
// 16 heads of 128 x 128, preparation and recurrence: 42 -> 34 µs at 64 requests, 100 -> 81 at 160,
// 9.7 -> 7.5 at 8, 7.8 -> 5.5 at one.
template <typename T, int G, int LANES>
__global__ void __launch_bounds__(LANES * DR_PARTS, G <= 4 ? 2 : 1)
delta_step_kernel(float* __restrict__ o, const T* __restrict__ qkv, int qkv_ld, int q_off, int k_off, int v_off,
                  const T* __restrict__ beta_raw, int beta_ld, const T* __restrict__ a_raw, int a_ld,
                  const float* __restrict__ a_log, const float* __restrict__ dt_bias, float* __restrict__ state,
                  long state_stride, const int* __restrict__ cu_tokens, const int* __restrict__ slots, int heads,
                  int kv_heads, int dk, int dv) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int STEP = 4 * DR_PARTS, DK = STEP * G;
  __shared__ __align__(16) float kqg[3][DK];
  __shared__ __align__(16) float sums[2][DR_PARTS][4 * LANES];
  const int s = blockIdx.x, h = blockIdx.y, part = threadIdx.x / LANES, piece = threadIdx.x % LANES;
  const int col = (blockIdx.z * LANES + piece) * 4;
  const bool live = col < dv;                         // dv is a multiple of four here
  const int t0 = cu_tokens[s], n = cu_tokens[s + 1] - t0;
  if (n <= 0) return;
  float* S_g = state + (size_t)slots[s] * state_stride + (size_t)h * dk * dv + col;
  float4 S[G][4];
#pragma unroll
  for (int m = 0; m < G; ++m)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = STEP * m + 4 * part + e;
      S[m][e] = live && i < dk ? *reinterpret_cast<const float4*>(S_g + (size_t)i * dv) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  const float rate = expf(a_log[h]);
  const int kh = h / (heads / kv_heads);
  for (int t = t0; t < t0 + n; ++t) {
    const T* kr = qkv + (size_t)t * qkv_ld + k_off + (size_t)kh * dk;
    const T* qr = qkv + (size_t)t * qkv_ld + q_off + (size_t)kh * dk;
    const float4 v = [&] {
      const T* p = qkv + (size_t)t * qkv_ld + v_off + (size_t)h * dv + col;
      return live ? make_float4(to_float(p[0]), to_float(p[1]), to_float(p[2]), to_float(p[3]))
                  : make_float4(0.f, 0.f, 0.f, 0.f);
    }();
    const DeltaNorms nm = delta_norms(kr, qr, dk, threadIdx.x & 31);
    for (int i = threadIdx.x; i < DK; i += LANES * DR_PARTS) {
      kqg[0][i] = i < dk ? to_float(kr[i]) * nm.kn : 0.f;
      kqg[1][i] = i < dk ? to_float(qr[i]) * nm.qn : 0.f;
      kqg[2][i] = i < dk ? delta_decay(to_float(a_raw[(size_t)t * a_ld + (size_t)h * dk + i]) + dt_bias[(size_t)h * dk + i], rate) : 0.f;
    }
    const float beta = delta_beta(to_float(beta_raw[(size_t)t * beta_ld + h]));
    __syncthreads();
    float4 d[4], r[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) d[e] = r[e] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int m = 0; m < G; ++m) {
      const float4 k4 = *reinterpret_cast<const float4*>(&kqg[0][STEP * m + 4 * part]);
      const float4 q4 = *reinterpret_cast<const float4*>(&kqg[1][STEP * m + 4 * part]);
      const float4 g4 = *reinterpret_cast<const float4*>(&kqg[2][STEP * m + 4 * part]);
      const float k[4] = {k4.x, k4.y, k4.z, k4.w}, q[4] = {q4.x, q4.y, q4.z, q4.w}, g[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float4& x = S[m][e];
        x.x *= g[e]; x.y *= g[e]; x.z *= g[e]; x.w *= g[e];
        d[e].x = fmaf(x.x, k[e], d[e].x); r[e].x = fmaf(x.x, q[e], r[e].x);
        d[e].y = fmaf(x.y, k[e], d[e].y); r[e].y = fmaf(x.y, q[e], r[e].y);
        d[e].z = fmaf(x.z, k[e], d[e].z); r[e].z = fmaf(x.z, q[e], r[e].z);
        d[e].w = fmaf(x.w, k[e], d[e].w); r[e].w = fmaf(x.w, q[e], r[e].w);
      }
    }
    auto add = [](float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); };
    *reinterpret_cast<float4*>(&sums[0][part][4 * piece]) = add(add(d[0], d[1]), add(d[2], d[3]));
    *reinterpret_cast<float4*>(&sums[1][part][4 * piece]) = add(add(r[0], r[1]), add(r[2], r[3]));
    __syncthreads();
    auto parts_sum = [&](int which) {
      float4 p[DR_PARTS];
#pragma unroll
      for (int i = 0; i < DR_PARTS; ++i) p[i] = *reinterpret_cast<const float4*>(&sums[which][i][4 * piece]);
#pragma unroll
      for (int x = 1; x < DR_PARTS; x *= 2)
#pragma unroll
        for (int i = 0; i < DR_PARTS; i += 2 * x) p[i] = add(p[i], p[i + x]);
      return p[0];
    };
    const float4 dot = parts_sum(0);
    const float4 u = make_float4(beta * (v.x - dot.x), beta * (v.y - dot.y), beta * (v.z - dot.z), beta * (v.w - dot.w));
#pragma unroll
    for (int m = 0; m < G; ++m) {
      const float4 k4 = *reinterpret_cast<const float4*>(&kqg[0][STEP * m + 4 * part]);
      const float k[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float4& x = S[m][e];
        x.x = fmaf(k[e], u.x, x.x); x.y = fmaf(k[e], u.y, x.y);
        x.z = fmaf(k[e], u.z, x.z); x.w = fmaf(k[e], u.w, x.w);
      }
    }
    if (part == 0 && live) {
      const float4 rd = parts_sum(1);
      *reinterpret_cast<float4*>(o + ((size_t)t * heads + h) * dv + col) =
          make_float4(fmaf(u.x, nm.kq, rd.x), fmaf(u.y, nm.kq, rd.y), fmaf(u.z, nm.kq, rd.z), fmaf(u.w, nm.kq, rd.w));
    }
    if (t + 1 < t0 + n) __syncthreads();               // the next token's rows and sums go to the same places
  }
#pragma unroll
  for (int m = 0; m < G; ++m)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = STEP * m + 4 * part + e;
      if (live && i < dk) *reinterpret_cast<float4*>(S_g + (size_t)i * dv) = S[m][e];
    }
}

// scratch: n_tokens * heads * (3 * dkp + 2) floats, dkp = dk rounded up to a multiple of 4
HB_EXPORT int hb_delta_rule(float* o, float* scratch, const void* qkv, int qkv_ld, int q_off, int k_off,
                            int v_off, const void* beta_raw, int beta_ld, const void* a_raw, int a_ld,
                            const float* a_log, const float* dt_bias, float* state,
                            long state_stride, const int* cu_tokens, const int* slots, int n_tokens,
                            int n_seqs, int heads, int kv_heads, int dk, int dv, int act_dt,
                            int sms, cudaStream_t stream) {
  if (n_seqs <= 0 || n_tokens <= 0) return HB_OK;
  if (heads <= 0 || kv_heads <= 0 || heads % kv_heads || dk <= 0 || dk > 256 || dv <= 0 ||
      heads > 65535 || scratch == nullptr || sms <= 0)
    return HB_BAD_ARGUMENT;
  // one token a request: the state's rows in whole 16-byte pieces, everything in one launch
  const int pieces = dv % 4 == 0 && state_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(state) & 15) == 0 ? 1 : 0;
  if (n_tokens == n_seqs && pieces && (reinterpret_cast<uintptr_t>(o) & 15) == 0) {
    const int lanes = dv <= 32 ? 8 : dv <= 64 ? 16 : 32;
    const dim3 grid1(n_seqs, heads, (dv + 4 * lanes - 1) / (4 * lanes));
#define HB_DR_STEP_LANES(G, LANES)                                                                           \
    HB_DISPATCH_DTYPE(act_dt, TA,                                                                            \
      hb_launch(delta_step_kernel<TA, G, LANES>, grid1, dim3(LANES * DR_PARTS), 0, stream, o,                \
                (const TA*)qkv, qkv_ld, q_off, k_off, v_off, (const TA*)beta_raw, beta_ld,                   \
                (const TA*)a_raw, a_ld, a_log, dt_bias, state, state_stride, cu_tokens, slots, heads,        \
                kv_heads, dk, dv))
#define HB_DR_STEP(G)                                                                                        \
    if (lanes == 8) HB_DR_STEP_LANES(G, 8);                                                                  \
    else if (lanes == 16) HB_DR_STEP_LANES(G, 16);                                                           \
    else HB_DR_STEP_LANES(G, 32)
    if (grid1.z > 65535) return HB_BAD_ARGUMENT;
    if (dk <= 32) { HB_DR_STEP(1); }
    else if (dk <= 64) { HB_DR_STEP(2); }
    else if (dk <= 128) { HB_DR_STEP(4); }
    else { HB_DR_STEP(8); }
#undef HB_DR_STEP
#undef HB_DR_STEP_LANES
    return hb_check_launch();
  }
  const int dkp = (dk + 3) / 4 * 4;
  float* kqg = scratch;
  float* beta = scratch + (size_t)n_tokens * heads * 3 * dkp;
  const int n_rows = n_tokens * heads;
  HB_DISPATCH_DTYPE(act_dt, TA,
    hb_launch(delta_prepare_kernel<TA>, dim3((n_rows + 3) / 4), dim3(128), 0, stream, kqg, beta,
              (const TA*)qkv, qkv_ld, q_off, k_off, (const TA*)beta_raw, beta_ld, (const TA*)a_raw, a_ld,
              a_log, dt_bias, n_rows, heads, kv_heads, dk, dkp));
  const bool alone = (long)n_seqs * heads * ((dv + DR_COLS - 1) / DR_COLS) <= sms;
  const int cols = dk <= 128 && (long)n_seqs * heads * ((dv + DR_COLS_WIDE - 1) / DR_COLS_WIDE) >= 2L * sms ? DR_COLS_WIDE : DR_COLS;
  const long blocks = (long)n_seqs * heads * ((dv + cols - 1) / cols);
  if (blocks > 0x7fffffffL) return HB_BAD_ARGUMENT;
#define HB_DR_LAUNCH_COLS(DKMAX, COLS, W, MANY)                                                      \
  HB_DISPATCH_DTYPE(act_dt, TA,                                                                   \
    const size_t smem = (2 * DR_CHUNK * 3 * DKMAX + 4 * DR_CHUNK + 2 * DR_CHUNK * COLS) * sizeof(float); \
    if (smem > 48 * 1024)                                                                         \
      cudaFuncSetAttribute(delta_rule_kernel<TA, DKMAX, COLS, W, MANY>,                           \
                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);               \
    const dim3 grid = MANY ? dim3((unsigned)blocks) : dim3(n_seqs, heads, (dv + cols - 1) / cols); \
    delta_rule_kernel<TA, DKMAX, COLS, W, MANY><<<grid, dim3(COLS * DR_PARTS / W), smem, stream>>>(   \
        o, (const float*)kqg, (const float*)beta, (const TA*)qkv, qkv_ld, v_off, state,           \
        state_stride, cu_tokens, slots, heads, dk, dkp, dv, pieces))
#define HB_DR_LAUNCH(DKMAX)                                                                       \
  if (alone) HB_DR_LAUNCH_COLS(DKMAX, DR_COLS, 1, false);                                         \
  else if (cols == DR_COLS) HB_DR_LAUNCH_COLS(DKMAX, DR_COLS, 2, (DKMAX >= 128));                 \
  else HB_DR_LAUNCH_COLS(DKMAX, DR_COLS_WIDE, 2, (DKMAX >= 128))
#define HB_DR_LAUNCH_LONG(DKMAX)                                                                  \
  if (alone) HB_DR_LAUNCH_COLS(DKMAX, DR_COLS, 1, false);                                         \
  else HB_DR_LAUNCH_COLS(DKMAX, DR_COLS, 1, true)
  if (dk <= 32) { HB_DR_LAUNCH(32); }
  else if (dk <= 64) { HB_DR_LAUNCH(64); }
  else if (dk <= 128) { HB_DR_LAUNCH(128); }
  else if (dk <= 160) { HB_DR_LAUNCH_LONG(160); }
  else if (dk <= 192) { HB_DR_LAUNCH_LONG(192); }
  else { HB_DR_LAUNCH_LONG(256); }
#undef HB_DR_LAUNCH_LONG
#undef HB_DR_LAUNCH_COLS
#undef HB_DR_LAUNCH
  return hb_check_launch();
}

#include "delta_chunk.cuh"

// The 32-bit words a (chunk, head) takes of `hb_delta_chunk`'s scratch; 0: this key size goes by `hb_delta_rule`
HB_EXPORT int hb_delta_chunk_words(int dk) {
  return dk <= 0 || dk > 128 ? 0 : dk <= 64 ? DeltaChunk<64>::WORDS : DeltaChunk<128>::WORDS;
}

// scratch: dc_chunks(n_tokens, n_seqs) * heads * hb_delta_chunk_words(dk) words, 16-byte aligned.  39,936 bytes a chunk and
// head of 128 values, 2,496 a token where `hb_delta_rule` takes 1,544; a request of one token takes a whole chunk, so the
// callers ask for 24 tokens a request (at most 4.2 KB a token and head).
HB_EXPORT int hb_delta_chunk(float* o, uint32_t* scratch, const void* qkv, int qkv_ld, int q_off, int k_off,
                             int v_off, const void* beta_raw, int beta_ld, const void* a_raw, int a_ld,
                             const float* a_log, const float* dt_bias, float* state,
                             long state_stride, const int* cu_tokens, const int* slots, int n_tokens,
                             int n_seqs, int heads, int kv_heads, int dk, int dv, int sms, cudaStream_t stream) {
  if (n_seqs <= 0 || n_tokens <= 0) return HB_OK;
  if (heads <= 0 || kv_heads <= 0 || heads % kv_heads || hb_delta_chunk_words(dk) == 0 || dv <= 0 ||
      heads > 65535 || scratch == nullptr || (reinterpret_cast<uintptr_t>(scratch) & 15) || sms <= 0)
    return HB_BAD_ARGUMENT;
  const long ids = dc_chunks(n_tokens, n_seqs);
  // one group of 16 columns a block where every block has an SM; else two, which share the staged chunks
  const long alone = (long)n_seqs * heads * ((dv + DC_COLS - 1) / DC_COLS);
  const int cols = alone <= sms ? DC_COLS : 2 * DC_COLS;
  const long blocks = (long)n_seqs * heads * ((dv + cols - 1) / cols);
  if (blocks > 0x7fffffffL || ids > 0x7fffffffL) return HB_BAD_ARGUMENT;
  using TA = __nv_bfloat16;
#define HB_DC_LAUNCH(DK, GROUPS, STAGES)                                                                      \
  do {                                                                                                        \
    hb_launch(delta_chunk_prepare_kernel<TA, DK>, dim3((unsigned)ids, heads), dim3(128), 0, stream, scratch,  \
              (const TA*)qkv, qkv_ld, q_off, k_off, (const TA*)beta_raw, beta_ld, (const TA*)a_raw, a_ld,     \
              a_log, dt_bias, cu_tokens, n_seqs, heads, kv_heads, dk);                                        \
    auto kernel = delta_chunk_kernel<TA, DK, GROUPS, STAGES>;                                                 \
    constexpr size_t smem = DeltaChunkSmem<DK, GROUPS, STAGES>::BYTES;                                        \
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);                     \
    kernel<<<(unsigned)blocks, GROUPS * DC_GROUP_THREADS, smem, stream>>>(                                    \
        o, (const uint32_t*)scratch, (const TA*)qkv, qkv_ld, v_off, state, state_stride, cu_tokens, slots,    \
        heads, dk, dv);                                                                                       \
  } while (0)
  if (dk <= 64) {
    if (cols == DC_COLS) HB_DC_LAUNCH(64, 1, 4);
    else HB_DC_LAUNCH(64, 2, 3);
  } else {
    if (cols == DC_COLS) HB_DC_LAUNCH(128, 1, 4);
    else HB_DC_LAUNCH(128, 2, 3);
  }
#undef HB_DC_LAUNCH
  return hb_check_launch();
}

// ---------------------------------------------------------------- output norm and gate
// out[t, h, :] = o[t, h, :] / sqrt(mean(o[t, h, :]^2) + eps) * weight * sigmoid(gate[t, h, :]);
// one warp per (token, head); the weight (dv values) is shared by the heads.
// VEC: four neighbouring values a lane at a time (rows in whole pieces).
template <typename T, bool VEC>
__global__ void gated_rmsnorm_kernel(T* __restrict__ out, const float* __restrict__ o,
                                     const T* __restrict__ gate, int gate_ld,
                                     const float* __restrict__ weight, int n_rows, int heads, int dv,
                                     float eps) {
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= n_rows) return;
  const int t = row / heads, h = row - t * heads;
  const float* orow = o + (size_t)row * dv;
  const T* grow = gate + (size_t)t * gate_ld + (size_t)h * dv;
  float ss = 0.f;
  T* dst = out + (size_t)row * dv;
  if constexpr (VEC) {
    for (int d = 4 * lane; d < dv; d += 128) {
      const float4 x = *reinterpret_cast<const float4*>(orow + d);
      ss = fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, fmaf(x.w, x.w, ss))));
    }
    const float rstd = rsqrtf(warp_sum(ss) / (float)dv + eps);
    for (int d = 4 * lane; d < dv; d += 128) {
      const float4 x = *reinterpret_cast<const float4*>(orow + d);
      const float4 w = *reinterpret_cast<const float4*>(weight + d);
      float gt[4];
      if constexpr (sizeof(T) == 4) {
        const float4 g = *reinterpret_cast<const float4*>(grow + d);
        gt[0] = g.x; gt[1] = g.y; gt[2] = g.z; gt[3] = g.w;
      } else {
        const uint2 raw = *reinterpret_cast<const uint2*>(grow + d);
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
        const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
        gt[0] = a.x; gt[1] = a.y; gt[2] = b.x; gt[3] = b.y;
      }
      const float v[4] = {x.x * rstd * w.x, x.y * rstd * w.y, x.z * rstd * w.z, x.w * rstd * w.w};
      float y[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) y[e] = v[e] * (1.f / (1.f + expf(-gt[e])));
      if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4*>(dst + d) = make_float4(y[0], y[1], y[2], y[3]);
      } else {
        const __nv_bfloat162 a = __floats2bfloat162_rn(y[0], y[1]), b = __floats2bfloat162_rn(y[2], y[3]);
        uint2 packed;
        packed.x = *reinterpret_cast<const uint32_t*>(&a);
        packed.y = *reinterpret_cast<const uint32_t*>(&b);
        *reinterpret_cast<uint2*>(dst + d) = packed;
      }
    }
    return;
  }
  for (int d = lane; d < dv; d += 32) ss += orow[d] * orow[d];
  const float rstd = rsqrtf(warp_sum(ss) / (float)dv + eps);
  for (int d = lane; d < dv; d += 32) {
    const float gt = 1.f / (1.f + expf(-to_float(grow[d])));
    dst[d] = from_float<T>(orow[d] * rstd * weight[d] * gt);
  }
}

HB_EXPORT int hb_gated_rmsnorm(void* out, const float* o, const void* gate, int gate_ld,
                               const float* weight, int T, int heads, int dv, float eps, int act_dt,
                               cudaStream_t stream) {
  if (T <= 0) return HB_OK;
  if (heads <= 0 || dv <= 0 || gate_ld < heads * dv) return HB_BAD_ARGUMENT;
  const int n_rows = T * heads;
  HB_DISPATCH_DTYPE(act_dt, TA,
    const size_t piece = 4 * sizeof(TA);
    const bool vec = dv % 4 == 0 && gate_ld % 4 == 0 &&
                     ((reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(weight)) & 15) == 0 &&
                     reinterpret_cast<uintptr_t>(out) % piece == 0 && reinterpret_cast<uintptr_t>(gate) % piece == 0;
    auto kernel = vec ? gated_rmsnorm_kernel<TA, true> : gated_rmsnorm_kernel<TA, false>;
    hb_launch(kernel, dim3((n_rows + 3) / 4), dim3(128), 0, stream, (TA*)out, o,
              (const TA*)gate, gate_ld, weight, n_rows, heads, dv, eps));
  return hb_check_launch();
}
