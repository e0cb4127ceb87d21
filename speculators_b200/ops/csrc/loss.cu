// Row-wise distillation losses between draft logits and verifier logits.
//
// One CTA per row.  Forward streams over the row pair and collects the online-softmax statistics (max, sum-exp) and the
// argmax of both rows, and for the KL divergence its cross term; the other divergences are reduced in a second pass.  Nothing of size [rows, V] is
// written.  Backward recomputes both softmaxes from the saved statistics and
// writes d(logits) in bf16 with the closed forms
//     kl   : dp - tp
//     rkl  : dp * (log dp - log tp - L)
//     jsd  : 0.5 * dp * (log(dp / mix) - KL(dp || mix)),  mix = (dp + tp) / 2
//     ce   : dp - onehot(argmax tp)
//     tv   : -dp * (1[dp <= tp] - s),  s = sum of dp over {dp <= tp}
// (dp = softmax(logits), tp = softmax(targets), L the row loss).  The same five
// reductions exist as Triton programs in the reference
// (src/speculators/losses/fused.py:91-235); this file is an independent CUDA
// implementation with two additions: the row pairing takes a `shift`
// (logits row r is compared with targets row r + shift, which is how the TTT
// steps of EAGLE-3 align their targets) and both argmaxes are by-products, so the
// accuracy metrics need no extra pass over the vocabulary.
#include "common.cuh"
#include "loss_stats.cuh"

namespace sb200 {

enum LossOp : int { kOpKL = 0, kOpRKL = 1, kOpJSD = 2, kOpCE = 3, kOpTV = 4 };
constexpr int kLossThreads = 512, kFwdThreads = 256;
constexpr int kNumStats = 5;  // m_d, z_d, m_t, z_t, per-op extra

// One thread's share of a row: running maximum, sum of exponentials against it, and the column at which the vector of eight
// starts that holds the maximum first (which of the eight is looked up once, at the end of the row).  KL: and the cross term.
struct Share {
  float m = -INFINITY, z = 0.f, A = 0.f;
  int col = 0x7fffffff;
};
__device__ __forceinline__ float max8(const bf16x8& v) {
  const __nv_bfloat162 m = __hmax2(__hmax2(v.v[0], v.v[1]), __hmax2(v.v[2], v.v[3]));
  return fmaxf(__low2float(m), __high2float(m));
}
// A new maximum moves the sums; most vectors bring none.
__device__ __forceinline__ void raise(Share& s, float to, int col) {
  if (to > s.m) {
    const float by = __expf(s.m - to);
    s.z *= by;
    s.A *= by;
    s.m = to;
    s.col = col;
  }
}
__device__ __forceinline__ float reference(const Share& s) { return s.m == -INFINITY ? 0.f : s.m; }

// Two fp32 values in a register pair: one instruction for both.
typedef unsigned long long float2x;
__device__ __forceinline__ float2x both(float lo, float hi) {
  float2x r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 apart(float2x v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ float2x fma2(float2x a, float2x b, float2x c) {
  float2x r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ float2x add2(float2x a, float2x b) {
  float2x r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float2x widen(const __nv_bfloat162& v) {
  const uint32_t w = *reinterpret_cast<const uint32_t*>(&v);
  return both(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
__device__ __forceinline__ float exp_base2(float v) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
constexpr float kLog2E = 1.4426950408889634f;
// e^(x - m) = 2^(x log2 e - m log2 e) in one multiply-add needs m log2 e to be finite: not where everything so far is -inf or the
// type's lowest value
constexpr float kFiniteFrom = -1e38f;
__device__ __forceinline__ float2x exp2x(float2x x, float2x log2e, float2x minus_m) {
  const float2 a = apart(fma2(x, log2e, minus_m));
  return both(exp_base2(a.x), exp_base2(a.y));
}

__device__ __forceinline__ void add8(Share& s, const bf16x8& v, int col) {
  raise(s, max8(v), col);
  if (s.m < kFiniteFrom) {
    float x[8];
    unpack8(v, x);
    const float m = reference(s);
    for (int j = 0; j < 8; ++j) s.z += __expf(x[j] - m);
    return;
  }
  const float2x log2e = both(kLog2E, kLog2E), minus_m = both(-s.m * kLog2E, -s.m * kLog2E);
  float2x add = both(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < 4; ++i) add = add2(add, exp2x(widen(v.v[i]), log2e, minus_m));
  const float2 sum = apart(add);
  s.z += sum.x + sum.y;
}
// The target row's, with A = sum_v e^{t_v - m}(t_v - x_v): sum_v p_v (t_v - x_v) = A / Z needs no second read of the rows.
__device__ __forceinline__ void add8_kl(Share& s, const bf16x8& tv, const bf16x8& xv, int col) {
  raise(s, max8(tv), col);
  if (s.m >= kFiniteFrom) {
    const float2x log2e = both(kLog2E, kLog2E), minus_m = both(-s.m * kLog2E, -s.m * kLog2E), minus = both(-1.f, -1.f);
    float2x add = both(0.f, 0.f), add_a = both(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2x t = widen(tv.v[i]), e = exp2x(t, log2e, minus_m);
      add = add2(add, e);
      add_a = fma2(e, fma2(widen(xv.v[i]), minus, t), add_a);
    }
    const float2 a = apart(add_a), sum = apart(add);
    if (fabsf(a.x + a.y) <= 3.4e38f) {  // else an infinite logit is among them
      s.z += sum.x + sum.y;
      s.A += a.x + a.y;
      return;
    }
  }
  float t[8], x[8];
  unpack8(tv, t);
  unpack8(xv, x);
  const float m = reference(s);
  for (int j = 0; j < 8; ++j) {
    const float e = __expf(t[j] - m);
    s.z += e;
    if (e > 0.f) s.A += e * (t[j] - x[j]);  // zero-probability targets contribute nothing
  }
}
__device__ __forceinline__ void add1(Share& s, float x, float other, int col, bool cross) {
  raise(s, x, col);
  const float e = __expf(x - reference(s));
  s.z += e;
  if (cross && e > 0.f) s.A += e * (x - other);
}
__device__ __forceinline__ void merge(Share& a, const Share& b) {
  const float m = fmaxf(a.m, b.m), ra = a.m == -INFINITY ? 0.f : __expf(a.m - m), rb = b.m == -INFINITY ? 0.f : __expf(b.m - m);
  a.z = a.z * ra + b.z * rb;
  a.A = a.A * ra + b.A * rb;
  if (b.m > a.m || (b.m == a.m && b.col < a.col)) a.col = b.col;
  a.m = m;
}
// Over the block, the same in every thread: shuffles, one exchange, and the warps' shares in order.
template <int WARPS>
__device__ __forceinline__ void merge_block(Share& s, Share (&slots)[WARPS]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    Share b;
    b.m = __shfl_xor_sync(0xffffffffu, s.m, o);
    b.z = __shfl_xor_sync(0xffffffffu, s.z, o);
    b.A = __shfl_xor_sync(0xffffffffu, s.A, o);
    b.col = __shfl_xor_sync(0xffffffffu, s.col, o);
    merge(s, b);
  }
  if ((threadIdx.x & 31) == 0) slots[threadIdx.x >> 5] = s;
  __syncthreads();
  s = slots[0];
#pragma unroll
  for (int w = 1; w < WARPS; ++w) merge(s, slots[w]);
}
// Column of the row's maximum (the first one).
__device__ __forceinline__ int first_max(const Share& s, const __nv_bfloat16* row, int vec_end) {
  if (s.col >= vec_end) return s.col;
  for (int j = 0; j < 8; ++j)
    if (__bfloat162float(row[s.col + j]) == s.m) return s.col + j;
  return s.col;
}

// Bound by issue and the special-function units before memory: an exponential per column and row, and beside it what the
// maximum, its column and the sums take.  So the maximum comes from packed comparisons and its column is kept per vector of
// eight, the sums are packed pairs, rescaling waits for a new maximum, two vectors are in flight, and the block meets once a row.  us before and after:
// KL 1280 x 32000 56 and 47, 4096 x 32000 161 and 122; total variation (a second pass) 222 and 185; labels 2460 x 151936
// 172 and 150 (reading takes 25, 80, 160 and 114).
template <int OP, int THREADS>
__global__ void __launch_bounds__(THREADS, 1536 / THREADS)
loss_fwd_kernel(const __nv_bfloat16* __restrict__ logits, const __nv_bfloat16* __restrict__ targets,
                const uint8_t* __restrict__ active, const uint8_t* __restrict__ also, const int64_t* __restrict__ labels,
                float* __restrict__ loss, float* __restrict__ stats, int* __restrict__ argmax_d,
                int* __restrict__ argmax_t, int rows, int V, int64_t ld_logits, int64_t ld_targets,
                int shift, const int* __restrict__ target_row) {
  pdl_begin();
  __shared__ Share slots[2][THREADS / 32];
  __shared__ float scratch[33];
  const int r = blockIdx.x;
  if (r >= rows) return;
  float* st = stats + r;
  const int tr = target_row != nullptr ? target_row[r] : r + shift;
  if (tr < 0 || (active && !active[r] && !(also && also[r]))) {
    if (threadIdx.x == 0) {
      loss[r] = 0.f;
#pragma unroll
      for (int k = 0; k < kNumStats; ++k) st[(int64_t)k * rows] = 0.f;
      if (argmax_d) argmax_d[r] = -1;
      if (argmax_t) argmax_t[r] = -2;
    }
    return;
  }
  const __nv_bfloat16* x = logits + (int64_t)r * ld_logits;
  // with integer labels (token cross-entropy) there is no target row to read
  const bool has_t = targets != nullptr;
  const __nv_bfloat16* t = has_t ? targets + (int64_t)tr * ld_targets : x;
  const bool vec_ok = ((V & 7) == 0) && ((ld_logits & 7) == 0) && ((ld_targets & 7) == 0);
  const int nvec = vec_ok ? (V >> 3) : 0;

  Share sd, stt;
  auto take = [&](const bf16x8& a, const bf16x8& b, int v) {
    add8(sd, a, v << 3);
    if (has_t) {
      if (OP == kOpKL) add8_kl(stt, b, a, v << 3);
      else add8(stt, b, v << 3);
    }
  };
  int v = threadIdx.x;
  for (; v + THREADS < nvec; v += 2 * THREADS) {
    const bf16x8 a0 = ld8(x + (v << 3)), a1 = ld8(x + ((v + THREADS) << 3));
    bf16x8 b0 = a0, b1 = a1;
    if (has_t) {
      b0 = ld8(t + (v << 3));
      b1 = ld8(t + ((v + THREADS) << 3));
    }
    take(a0, b0, v);
    take(a1, b1, v + THREADS);
  }
  if (v < nvec) {
    const bf16x8 a0 = ld8(x + (v << 3));
    take(a0, has_t ? ld8(t + (v << 3)) : a0, v);
  }
  for (int c = (nvec << 3) + threadIdx.x; c < V; c += THREADS) {
    const float xc = __bfloat162float(x[c]);
    add1(sd, xc, 0.f, c, false);
    if (has_t) add1(stt, __bfloat162float(t[c]), xc, c, OP == kOpKL);
  }
  if (has_t) merge_block(stt, slots[1]);
  merge_block(sd, slots[0]);
  const float lse_d = sd.m + __logf(sd.z);
  float lse_t = 0.f;
  if (has_t) lse_t = stt.m + __logf(stt.z);

  float acc0 = 0.f, acc1 = 0.f;
  if (OP != kOpCE && OP != kOpKL) {
    auto body = [&](float xv, float tv) {
      const float ldp = xv - lse_d, ltp = tv - lse_t;
      const float dp = __expf(ldp), tp = __expf(ltp);
      if (OP == kOpRKL) {
        if (dp > 0.f) acc0 += dp * (ldp - ltp);
      } else if (OP == kOpJSD) {
        const float mx = fmaxf(ldp, ltp);
        const float lm = mx + __logf(__expf(ldp - mx) + __expf(ltp - mx)) - 0.6931471805599453f;
        if (tp > 0.f) acc0 += tp * (ltp - lm);
        if (dp > 0.f) acc1 += dp * (ldp - lm);
      } else {  // TV
        acc0 += fminf(dp, tp);
        if (dp <= tp) acc1 += dp;
      }
    };
    for (int v = threadIdx.x; v < nvec; v += THREADS) {
      float a[8], b[8];
      unpack8(ld8(x + (v << 3)), a);
      unpack8(ld8(t + (v << 3)), b);
#pragma unroll
      for (int j = 0; j < 8; ++j) body(a[j], b[j]);
    }
    for (int c = (nvec << 3) + threadIdx.x; c < V; c += THREADS)
      body(__bfloat162float(x[c]), __bfloat162float(t[c]));
    acc0 = block_sum(acc0, scratch);
    if (OP == kOpJSD || OP == kOpTV) acc1 = block_sum(acc1, scratch);
  }
  if (threadIdx.x == 0) {
    int best_t;
    if (has_t) {
      best_t = first_max(stt, t, nvec << 3);
    } else {
      const int64_t lab = labels ? labels[tr] : 0;
      best_t = lab < 0 ? 0 : (lab >= V ? V - 1 : (int)lab);
      stt.m = 0.f;
      stt.z = 1.f;
    }
    float L, extra;
    if (OP == kOpKL) {
      L = extra = stt.A / stt.z + lse_d - lse_t;  // sum_v p_v (t_v - x_v) and the normalisers
    } else if (OP == kOpRKL) {
      L = acc0;
      extra = acc0;
    } else if (OP == kOpJSD) {
      L = 0.5f * (acc0 + acc1);
      extra = acc1;
    } else if (OP == kOpCE) {
      L = lse_d - __bfloat162float(x[best_t]);
      extra = (float)best_t;
    } else {
      L = 1.f - acc0;
      extra = acc1;
    }
    loss[r] = L;
    st[0] = sd.m;
    st[(int64_t)rows] = sd.z;
    st[(int64_t)2 * rows] = stt.m;
    st[(int64_t)3 * rows] = stt.z;
    st[(int64_t)4 * rows] = extra;
    if (argmax_d) argmax_d[r] = first_max(sd, x, nvec << 3);
    if (argmax_t) argmax_t[r] = best_t;
  }
}

// grid.x = total_rows (rows of the d(logits) buffer); rows >= `rows` or with a zero
// upstream gradient are zero-filled.
template <int OP>
__global__ void __launch_bounds__(kLossThreads)
loss_bwd_kernel(const __nv_bfloat16* __restrict__ logits, const __nv_bfloat16* __restrict__ targets,
                const float* __restrict__ grad_out, const float* __restrict__ grad_scale, const float* __restrict__ stats,
                __nv_bfloat16* __restrict__ dlogits, int rows, int total_rows, int V,
                int64_t ld_logits, int64_t ld_targets, int64_t ld_dlogits, int shift, const int* __restrict__ target_row,
                const int* __restrict__ live) {
  pdl_begin();
  const int r = blockIdx.x;
  if (r >= live_rows(live, total_rows)) return;
  __nv_bfloat16* d = dlogits + (int64_t)r * ld_dlogits;
  const bool vec_ok =
      ((V & 7) == 0) && ((ld_logits & 7) == 0) && ((ld_targets & 7) == 0) && ((ld_dlogits & 7) == 0);
  const int nvec = vec_ok ? (V >> 3) : 0;
  const float go = r < rows ? grad_out[r] * (grad_scale != nullptr ? *grad_scale : 1.f) : 0.f;
  // a row the forward skipped (inactive) has all-zero statistics; its sum-exp would be >= 1
  // otherwise.  Such a row gets no gradient whatever the upstream value is.
  const bool skipped = r < rows && stats[(int64_t)rows + r] == 0.f;
  if (go == 0.f || skipped) {
    bf16x8 z;
#pragma unroll
    for (int i = 0; i < 4; ++i) z.v[i] = __floats2bfloat162_rn(0.f, 0.f);
    for (int v = threadIdx.x; v < nvec; v += kLossThreads) st8(d + (v << 3), z);
    for (int c = (nvec << 3) + threadIdx.x; c < V; c += kLossThreads) d[c] = __float2bfloat16(0.f);
    return;
  }
  const __nv_bfloat16* x = logits + (int64_t)r * ld_logits;
  const __nv_bfloat16* t = targets + (int64_t)(target_row != nullptr ? target_row[r] : r + shift) * ld_targets;  // not negative: the forward did not skip it
  const float* st = stats + r;
  const float lse_d = st[0] + __logf(st[(int64_t)rows]);
  const float lse_t = (OP == kOpCE) ? 0.f : st[(int64_t)2 * rows] + __logf(st[(int64_t)3 * rows]);
  const float extra = st[(int64_t)4 * rows];
  const int label = (OP == kOpCE) ? (int)extra : -1;

  auto grad = [&](float xv, float tv, int col) -> float {
    const float ldp = xv - lse_d;
    const float dp = __expf(ldp);
    if (OP == kOpCE) return go * (dp - (col == label ? 1.f : 0.f));
    const float ltp = tv - lse_t;
    const float tp = __expf(ltp);
    if (OP == kOpKL) return go * (dp - tp);
    if (OP == kOpRKL) return dp > 0.f ? go * dp * (ldp - ltp - extra) : 0.f;
    if (OP == kOpJSD) {
      const float mx = fmaxf(ldp, ltp);
      const float lm = mx + __logf(__expf(ldp - mx) + __expf(ltp - mx)) - 0.6931471805599453f;
      return dp > 0.f ? go * 0.5f * dp * ((ldp - lm) - extra) : 0.f;
    }
    return -go * dp * ((dp <= tp ? 1.f : 0.f) - extra);  // TV
  };
  for (int v = threadIdx.x; v < nvec; v += kLossThreads) {
    float a[8], b[8], o[8];
    unpack8(ld8(x + (v << 3)), a);
    if (OP != kOpCE) unpack8(ld8(t + (v << 3)), b);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = grad(a[j], OP != kOpCE ? b[j] : 0.f, (v << 3) + j);
    st8(d + (v << 3), pack8(o));
  }
  for (int c = (nvec << 3) + threadIdx.x; c < V; c += kLossThreads)
    d[c] = __float2bfloat16(
        grad(__bfloat162float(x[c]), OP != kOpCE ? __bfloat162float(t[c]) : 0.f, c));
}

// active / also (optional): rows marked in neither are skipped.  target_row (optional): the row of `targets` that each row is
// compared with, instead of its own + shift; rows with a negative one are skipped.
int launch_loss_fwd(int op, const void* logits, const void* targets, const uint8_t* active, const uint8_t* also,
                    const int64_t* labels, float* loss, float* stats, int* argmax_d, int* argmax_t, int rows, int V,
                    int64_t ld_logits, int64_t ld_targets, int shift, const int* target_row, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (targets == nullptr && (labels == nullptr || op != kOpCE)) return -3;
  count_launch(1);
#define SB200_LF(OPV)                                                                            \
  launch_pdl(loss_fwd_kernel<OPV, kFwdThreads>, rows, kFwdThreads, 0, stream,                              \
      (const __nv_bfloat16*)logits, (const __nv_bfloat16*)targets, active, also, labels, loss, stats,   \
      argmax_d, argmax_t, rows, V, ld_logits, ld_targets, shift, target_row)
  switch (op) {
    case kOpKL: SB200_LF(kOpKL); break;
    case kOpRKL: SB200_LF(kOpRKL); break;
    case kOpJSD: SB200_LF(kOpJSD); break;
    case kOpCE: SB200_LF(kOpCE); break;
    case kOpTV: SB200_LF(kOpTV); break;
    default: return -1;
  }
#undef SB200_LF
  return 0;
}

// grad_scale (optional, device): a factor of every grad_out; target_row as in launch_loss_fwd; live (optional, device): rows of
// dlogits in use, those behind are not written
int launch_loss_bwd(int op, const void* logits, const void* targets, const float* grad_out,
                    const float* grad_scale, const float* stats, void* dlogits, int rows, int total_rows, int V,
                    int64_t ld_logits, int64_t ld_targets, int64_t ld_dlogits, int shift, const int* target_row,
                    const int* live, cudaStream_t stream) {
  if (total_rows <= 0) return 0;
  count_launch(1);
#define SB200_LB(OPV)                                                                         \
  launch_pdl(loss_bwd_kernel<OPV>, total_rows, kLossThreads, 0, stream,                                \
      (const __nv_bfloat16*)logits, (const __nv_bfloat16*)targets, grad_out, grad_scale, stats,            \
      (__nv_bfloat16*)dlogits, rows, total_rows, V, ld_logits, ld_targets, ld_dlogits, shift, target_row, live)
  switch (op) {
    case kOpKL: SB200_LB(kOpKL); break;
    case kOpRKL: SB200_LB(kOpRKL); break;
    case kOpJSD: SB200_LB(kOpJSD); break;
    case kOpCE: SB200_LB(kOpCE); break;
    case kOpTV: SB200_LB(kOpTV); break;
    default: return -1;
  }
#undef SB200_LB
  return 0;
}

}  // namespace sb200
