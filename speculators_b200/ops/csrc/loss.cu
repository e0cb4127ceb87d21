// Row-wise distillation losses between draft logits and verifier logits.
//
// One CTA per row.  Forward makes two streaming passes over the row pair: pass 1
// collects the online-softmax statistics (max, sum-exp) and the argmax of both
// rows, pass 2 reduces the selected divergence.  Nothing of size [rows, V] is
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
#include "packed_f32.cuh"

namespace sb200 {

// kOpKLTV: the KL divergence, and the total variation next to it (forward only)
enum LossOp : int { kOpKL = 0, kOpRKL = 1, kOpJSD = 2, kOpCE = 3, kOpTV = 4, kOpKLTV = 5 };
constexpr int kLossThreads = 512;
constexpr int kNumStats = 5;  // m_d, z_d, m_t, z_t, per-op extra

// One thread's share of a row: running maximum, sum of exponentials against it, and the column where the vector of eight starts
// that brought the maximum (which of the eight is looked up once a row); columns behind the last whole vector on their own.
// Sums are formed in the order of the columns, eight at a time, as online_update (loss_stats.cuh) forms them.
struct Share {
  float m = -INFINITY, z = 0.f;
  int col = 0x7fffffff;
};
__device__ __forceinline__ float max8(const bf16x8& v) {
  const __nv_bfloat162 m = __hmax2(__hmax2(v.v[0], v.v[1]), __hmax2(v.v[2], v.v[3]));
  return fmaxf(__low2float(m), __high2float(m));
}
__device__ __forceinline__ float2x widen(const __nv_bfloat162& v) {
  const uint32_t w = *reinterpret_cast<const uint32_t*>(&v);
  return both(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
// e^v = 2^(v log2 e) of two differences
__device__ __forceinline__ float2 exp_pair(float2x v) {
  constexpr float kLog2E = 1.4426950408889634f;
  const float2 s = apart(mul2(v, both(kLog2E, kLog2E)));
  float2 e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.x) : "f"(s.x));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.y) : "f"(s.y));
  return e;
}
// The new maximum and what it makes of the sums so far.
__device__ __forceinline__ float raise(Share& s, float vmax, int col) {
  const float m_new = fmaxf(s.m, vmax), by = __expf(s.m - m_new);
  s.col = vmax > s.m ? col : s.col;
  s.m = m_new;
  return by;
}
__device__ __forceinline__ void add8(Share& s, const bf16x8& v, int col) {
  const float by = raise(s, max8(v), col);
  const float2x minus_m = both(-s.m, -s.m);
  float add = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 e = exp_pair(add2(widen(v.v[i]), minus_m));
    add += e.x;
    add += e.y;
  }
  s.z = fmaf(s.z, by, add);
}
// The target row's, with A = sum_v e^{t_v - m}(t_v - x_v) (see online_update_kl in loss_stats.cuh).
__device__ __forceinline__ void add8_kl(Share& s, float& A, const bf16x8& tv, const bf16x8& xv, int col) {
  const float by = raise(s, max8(tv), col);
  const float2x minus_m = both(-s.m, -s.m), minus = both(-1.f, -1.f);
  float add = 0.f, add_a = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2x t = widen(tv.v[i]);
    const float2 e = exp_pair(add2(t, minus_m)), d = apart(fma2(widen(xv.v[i]), minus, t));
    add += e.x;
    add += e.y;
    add_a = fmaf(e.x, d.x, add_a);
    add_a = fmaf(e.y, d.y, add_a);
  }
  if (add_a != add_a) {  // an infinite logit is among them: zero-probability targets contribute nothing
    float t[8], x[8];
    unpack8(tv, t);
    unpack8(xv, x);
    add = add_a = 0.f;
    for (int j = 0; j < 8; ++j) {
      const float e = __expf(t[j] - s.m);
      add += e;
      if (e > 0.f) add_a = fmaf(e, t[j] - x[j], add_a);
    }
  }
  s.z = fmaf(s.z, by, add);
  A = fmaf(A, by, add_a);
}
__device__ __forceinline__ void add1(Share& s, float x, int col) {
  const float by = raise(s, x, col);
  s.z = fmaf(s.z, by, __expf(x - s.m));
}
__device__ __forceinline__ void add1_kl(Share& s, float& A, float t, float x, int col) {
  const float by = raise(s, t, col), e = __expf(t - s.m);
  s.z = fmaf(s.z, by, e);
  A = fmaf(A, by, e > 0.f ? e * (t - x) : 0.f);
}

// Meetings of the block.  Every warp finishes the reduction for itself, in the order block_sum takes, so that a meeting is one barrier.
constexpr int kLossWarps = kLossThreads / 32;
struct Meeting {
  float m[2][kLossWarps], z[2][kLossWarps], acc[2][kLossWarps];
  int col[2][kLossWarps];
};
__device__ __forceinline__ float over_warps_sum(const float* of) {
  const int lane = threadIdx.x & 31;
  return warp_sum(lane < kLossWarps ? of[lane] : 0.f);
}
// Row `i`'s share over the block; meet_max, a barrier, meet_sum, a barrier, met.
__device__ __forceinline__ void meet_max(const Share& s, Meeting& at, int i) {
  const float m = warp_max(s.m);
  const int col = __reduce_min_sync(0xffffffffu, s.m == m ? s.col : 0x7fffffff);
  if ((threadIdx.x & 31) == 0) {
    at.m[i][threadIdx.x >> 5] = m;
    at.col[i][threadIdx.x >> 5] = col;
  }
}
__device__ __forceinline__ void meet_sum(Share& s, Meeting& at, int i) {
  const int lane = threadIdx.x & 31;
  const float wm = lane < kLossWarps ? at.m[i][lane] : -INFINITY, M = warp_max(wm);
  s.col = __reduce_min_sync(0xffffffffu, lane < kLossWarps && wm == M ? at.col[i][lane] : 0x7fffffff);
  const float z = warp_sum((s.m == -INFINITY) ? 0.f : s.z * __expf(s.m - M));
  if (lane == 0) at.z[i][threadIdx.x >> 5] = z;
  s.m = M;
}
__device__ __forceinline__ void met(Share& s, const Meeting& at, int i) { s.z = over_warps_sum(at.z[i]); }
__device__ __forceinline__ float block_sum_in(float v, float* of) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) of[threadIdx.x >> 5] = v;
  __syncthreads();
  return over_warps_sum(of);
}
// Column of the row's maximum, the first one.
__device__ __forceinline__ int first_max(const Share& s, const __nv_bfloat16* row, int vec_end) {
  if (s.col >= vec_end) return s.col;
  for (int j = 0; j < 8; ++j)
    if (__bfloat162float(row[s.col + j]) == s.m) return s.col + j;
  return s.col;
}

// Bound by issue and the special-function units before memory: an exponential per column and row, and beside it what the maximum,
// its column and the sums take.  So the maximum comes from packed comparisons, its column is kept per vector of eight and looked up
// once a row, differences and scalings are packed pairs, and a row takes two to four barriers, by loss (23 before).  Sums keep their order.  The
// KL divergence does best with three blocks an SM and one vector of each row in flight, the others with two and what registers
// the compiler likes (us, two vectors and one: KL 4096 x 32000 143 and 130, total variation 168 and 195, labels 2460 x 151936 144 and
// 175; bounded to 32 registers the labels took 268).  us before and after: KL 1001 x 32000 45.7 and 38.7, 4096 x 32000 159 and 129,
// total variation 220 and 168, cross-entropy 8192 x 32000 253 and 205, labels 300 x 151936 38.5 and 29.8, 2460 x 151936 170 and 144
// (reading takes 20, 80, 80, 160, 14 and 114).
template <int OP>
__global__ void __launch_bounds__(kLossThreads, OP == kOpKL || OP == kOpKLTV ? 3 : 0)
loss_fwd_kernel(const __nv_bfloat16* __restrict__ logits, const __nv_bfloat16* __restrict__ targets,
                const uint8_t* __restrict__ active, const uint8_t* __restrict__ also, const int64_t* __restrict__ labels,
                float* __restrict__ loss, float* __restrict__ stats, int* __restrict__ argmax_d,
                int* __restrict__ argmax_t, int rows, int V, int64_t ld_logits, int64_t ld_targets,
                int shift, const int* __restrict__ target_row, float* __restrict__ tv) {
  pdl_begin();
  constexpr bool KL = OP == kOpKL || OP == kOpKLTV;
  __shared__ Meeting at;
  const int r = blockIdx.x;
  if (r >= rows) return;
  float* st = stats + r;
  const int tr = target_row != nullptr ? target_row[r] : r + shift;
  if (tr < 0 || (active && !active[r] && !(also && also[r]))) {
    if (threadIdx.x == 0) {
      loss[r] = 0.f;
      if (OP == kOpKLTV) tv[r] = 0.f;
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
  float kl_a = 0.f;  // KL: the cross term, accumulated in the same pass
  auto take = [&](const bf16x8& a, const bf16x8& b, int v) {
    add8(sd, a, v << 3);
    if (has_t) {
      if (KL) add8_kl(stt, kl_a, b, a, v << 3);
      else add8(stt, b, v << 3);
    }
  };
  int v = threadIdx.x;
  if constexpr (KL) {
    for (; v < nvec; v += kLossThreads) {
      const bf16x8 a0 = ld8(x + (v << 3));
      take(a0, has_t ? ld8(t + (v << 3)) : a0, v);
    }
  } else {
    for (; v + kLossThreads < nvec; v += 2 * kLossThreads) {
      const bf16x8 a0 = ld8(x + (v << 3)), a1 = ld8(x + ((v + kLossThreads) << 3));
      bf16x8 b0 = a0, b1 = a1;
      if (has_t) {
        b0 = ld8(t + (v << 3));
        b1 = ld8(t + ((v + kLossThreads) << 3));
      }
      take(a0, b0, v);
      take(a1, b1, v + kLossThreads);
    }
    if (v < nvec) {
      const bf16x8 a0 = ld8(x + (v << 3));
      take(a0, has_t ? ld8(t + (v << 3)) : a0, v);
    }
  }
  for (int c = (nvec << 3) + threadIdx.x; c < V; c += kLossThreads) {
    const float xc = __bfloat162float(x[c]);
    add1(sd, xc, c);
    if (has_t) {
      if (KL) add1_kl(stt, kl_a, __bfloat162float(t[c]), xc, c);
      else add1(stt, __bfloat162float(t[c]), c);
    }
  }
  const float my_mt = stt.m;  // this thread's running max of the target row, before the block-wide combine
  meet_max(sd, at, 0);
  if (has_t) meet_max(stt, at, 1);
  __syncthreads();
  meet_sum(sd, at, 0);
  if (has_t) meet_sum(stt, at, 1);
  __syncthreads();
  met(sd, at, 0);
  if (has_t) {
    met(stt, at, 1);
  } else {
    stt.m = 0.f;
    stt.z = 1.f;
    int lab = labels ? (int)labels[tr] : 0;
    stt.col = lab < 0 ? 0 : (lab >= V ? V - 1 : lab);
  }
  auto best_of_target = [&]() { return has_t ? first_max(stt, t, nvec << 3) : stt.col; };
  const float lse_d = sd.m + __logf(sd.z);
  const float lse_t = stt.m + __logf(stt.z);

  float acc0 = 0.f, acc1 = 0.f;
  if (OP == kOpCE) {
    if (threadIdx.x == 0) {
      const int c = best_of_target();  // none in a row of nothing but -inf or NaN
      acc0 = c < V ? lse_d - __bfloat162float(x[c]) : __int_as_float(0x7fffffff);
    }
  } else if (KL) {
    // sum_v p_v (t_v - x_v) = (sum over threads of A rescaled to the row max) / Z_t; thread 0 adds
    // the normaliser terms once so that the block sum below yields the row's KL directly
    acc0 = (my_mt == -INFINITY) ? 0.f : kl_a * __expf(my_mt - stt.m) / stt.z;
    if (threadIdx.x == 0) acc0 += lse_d - lse_t;
  }
  if (OP != kOpCE && OP != kOpKL) {
    float acc0b = 0.f;
    float& acc = OP == kOpKLTV ? acc0b : acc0;
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
        acc += fminf(dp, tp);
        if (OP == kOpTV && dp <= tp) acc1 += dp;
      }
    };
    for (int v = threadIdx.x; v < nvec; v += kLossThreads) {
      float a[8], b[8];
      unpack8(ld8(x + (v << 3)), a);
      unpack8(ld8(t + (v << 3)), b);
#pragma unroll
      for (int j = 0; j < 8; ++j) body(a[j], b[j]);
    }
    for (int c = (nvec << 3) + threadIdx.x; c < V; c += kLossThreads)
      body(__bfloat162float(x[c]), __bfloat162float(t[c]));
    if (OP == kOpKLTV) acc1 = acc0b;
  }
  if (OP != kOpCE) acc0 = block_sum_in(acc0, at.acc[0]);
  if (OP == kOpJSD || OP == kOpTV || OP == kOpKLTV) acc1 = block_sum_in(acc1, at.acc[1]);
  if (threadIdx.x == 0) {
    float L, extra;
    const int best_t = OP == kOpCE || argmax_t ? best_of_target() : 0;
    if (KL || OP == kOpRKL) {
      L = acc0;
      extra = acc0;
    } else if (OP == kOpJSD) {
      L = 0.5f * (acc0 + acc1);
      extra = acc1;
    } else if (OP == kOpCE) {
      L = acc0;
      extra = (float)best_t;
    } else {
      L = 1.f - acc0;
      extra = acc1;
    }
    loss[r] = L;
    if (OP == kOpKLTV) tv[r] = 1.f - acc1;
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
// compared with, instead of its own + shift; rows with a negative one are skipped.  tv (optional, with the KL divergence): the rows'
// total variation, 0 where skipped.
int launch_loss_fwd(int op, const void* logits, const void* targets, const uint8_t* active, const uint8_t* also,
                    const int64_t* labels, float* loss, float* stats, int* argmax_d, int* argmax_t, int rows, int V,
                    int64_t ld_logits, int64_t ld_targets, int shift, const int* target_row, float* tv, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (tv != nullptr) {
    if (op != kOpKL || targets == nullptr) return -4;
    op = kOpKLTV;
  }
  if (targets == nullptr && (labels == nullptr || op != kOpCE)) return -3;
  count_launch(1);
#define SB200_LF(OPV)                                                                            \
  launch_pdl(loss_fwd_kernel<OPV>, rows, kLossThreads, 0, stream,                                         \
      (const __nv_bfloat16*)logits, (const __nv_bfloat16*)targets, active, also, labels, loss, stats,   \
      argmax_d, argmax_t, rows, V, ld_logits, ld_targets, shift, target_row, tv)
  switch (op) {
    case kOpKL: SB200_LF(kOpKL); break;
    case kOpRKL: SB200_LF(kOpRKL); break;
    case kOpJSD: SB200_LF(kOpJSD); break;
    case kOpCE: SB200_LF(kOpCE); break;
    case kOpTV: SB200_LF(kOpTV); break;
    case kOpKLTV: SB200_LF(kOpKLTV); break;
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
