// Flat-buffer optimizer kernels: squared-norm reduction and fused AdamW.
//
// The trainable parameters of a model live in one contiguous bf16 buffer (the
// compute weights) with a parallel bf16 gradient buffer; the optimizer keeps fp32
// master weights and both moments for the slice of that buffer this rank owns.
// One AdamW launch therefore updates every parameter: read grad (+ clip scale),
// master, m, v; write master, m, v and the bf16 compute weight.  All scalar
// inputs that change from step to step (learning rate, bias corrections, the
// gradient norm) are read from device memory so the launch can sit inside a
// captured CUDA graph.
#include "common.cuh"

namespace sb200 {

constexpr int kOptThreads = 256;

// hyper layout (fp32): [0] lr  [1] beta1  [2] beta2  [3] eps  [4] weight_decay
//                      [5] bias_correction1  [6] bias_correction2  [7] max_grad_norm (<=0: off)
//                      [8] grad_scale (multiplied into every gradient, e.g. 1/world_size)
constexpr int kHyperLen = 16;

template <typename T>
__device__ __forceinline__ float to_f(T v);
template <>
__device__ __forceinline__ float to_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// Stage 1: per-CTA partial sums of squares into partial[blockIdx.x].
template <typename T>
__global__ void __launch_bounds__(kOptThreads)
sumsq_partial_kernel(const T* __restrict__ g, int64_t n, float* __restrict__ partial) {
  pdl_begin();
  __shared__ float scratch[33];
  float acc = 0.f;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float v = to_f<T>(g[i]);
    acc += v * v;
  }
  acc = block_sum(acc, scratch);
  if (threadIdx.x == 0) partial[blockIdx.x] = acc;
}

template <>
__global__ void __launch_bounds__(kOptThreads)
sumsq_partial_kernel<__nv_bfloat16>(const __nv_bfloat16* __restrict__ g, int64_t n,
                                     float* __restrict__ partial) {
  pdl_begin();
  __shared__ float scratch[33];
  float acc = 0.f;
  const int64_t nvec = n >> 3;  // buffer base is 16-byte aligned by construction
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nvec;
       v += (int64_t)gridDim.x * blockDim.x) {
    float f[8];
    unpack8(ld8(g + (v << 3)), f);
#pragma unroll
    for (int j = 0; j < 8; ++j) acc += f[j] * f[j];
  }
  for (int64_t i = (nvec << 3) + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float v = __bfloat162float(g[i]);
    acc += v * v;
  }
  acc = block_sum(acc, scratch);
  if (threadIdx.x == 0) partial[blockIdx.x] = acc;
}

// Stage 2: out[0] (+)= sum(partial[0:P]) in a fixed order (deterministic).
__global__ void sumsq_final_kernel(const float* __restrict__ partial, int P, float* __restrict__ out,
                                   int accumulate) {
  pdl_begin();
  __shared__ float scratch[33];
  float acc = 0.f;
  for (int i = threadIdx.x; i < P; i += blockDim.x) acc += partial[i];
  acc = block_sum(acc, scratch);
  if (threadIdx.x == 0) out[0] = accumulate ? out[0] + acc : acc;
}

// Eight consecutive fp32 / gradient values with 16-byte accesses.  The optimizer's buffers are read and written once
// per step and are gigabytes: evict-first, so that they do not displace the weights in L2.
struct f32x8 {
  float v[8];
};
__device__ __forceinline__ f32x8 ld8s(const float* p) {
  const float4 a = __ldcs(reinterpret_cast<const float4*>(p)), b = __ldcs(reinterpret_cast<const float4*>(p) + 1);
  return f32x8{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
}
__device__ __forceinline__ f32x8 ld8s(const __nv_bfloat16* p) {
  const uint4 q = __ldcs(reinterpret_cast<const uint4*>(p));
  f32x8 r;
  unpack8(*reinterpret_cast<const bf16x8*>(&q), r.v);
  return r;
}
__device__ __forceinline__ void st8s(float* p, const f32x8& x) {
  __stcs(reinterpret_cast<float4*>(p), make_float4(x.v[0], x.v[1], x.v[2], x.v[3]));
  __stcs(reinterpret_cast<float4*>(p) + 1, make_float4(x.v[4], x.v[5], x.v[6], x.v[7]));
}

struct AdamScalars {
  float keep, b1, b2, gscale, step_size, inv_sqrt_bc2, eps;
};
__device__ __forceinline__ void adam_update(const AdamScalars& s, float g, float& p, float& m, float& v) {
  g *= s.gscale;
  p *= s.keep;
  m = s.b1 * m + (1.f - s.b1) * g;
  v = s.b2 * v + (1.f - s.b2) * g * g;
  const float denom = sqrtf(v) * s.inv_sqrt_bc2 + s.eps;
  p -= s.step_size * (m / denom);
}

// norm_sq: device scalar holding the (already all-reduced) sum of squares of the
// *unscaled* gradients; clip coefficient = min(1, max_norm / (grad_scale*sqrt(norm_sq) + 1e-6)).
//
// Bound by memory: 28 bytes per parameter (bf16 gradient, fp32 master and two moments read and written, bf16
// weight).  A thread owns eight consecutive parameters and a block 2048, one block per chunk: seven independent
// 16-byte loads are in flight per thread.  With one parameter per thread and loop step (2- and 4-byte accesses)
// 1.14 G parameters took 5.58 ms, 5.7 TB/s; this form takes 5.17 ms, 6.2 TB/s (96 % of a plain copy).
template <typename G, bool VEC>
__global__ void __launch_bounds__(kOptThreads)
adamw_kernel(float* __restrict__ master, float* __restrict__ m, float* __restrict__ v,
             const G* __restrict__ grad, __nv_bfloat16* __restrict__ w16, int64_t n,
             const float* __restrict__ hyper, const float* __restrict__ norm_sq) {
  pdl_begin();
  AdamScalars s;
  s.b1 = hyper[1];
  s.b2 = hyper[2];
  s.eps = hyper[3];
  s.keep = 1.f - hyper[0] * hyper[4];
  s.gscale = hyper[8];
  if (hyper[7] > 0.f && norm_sq) {
    const float total = s.gscale * sqrtf(norm_sq[0]);
    const float coef = hyper[7] / (total + 1e-6f);
    if (coef < 1.f) s.gscale *= coef;
  }
  s.step_size = hyper[0] / hyper[5];
  s.inv_sqrt_bc2 = rsqrtf(hyper[6]);
  const int64_t i0 = ((int64_t)blockIdx.x * kOptThreads + threadIdx.x) * 8;
  if (VEC && i0 + 8 <= n) {
    const f32x8 g = ld8s(grad + i0);
    f32x8 p = ld8s(master + i0), a = ld8s(m + i0), b = ld8s(v + i0);
#pragma unroll
    for (int j = 0; j < 8; ++j) adam_update(s, g.v[j], p.v[j], a.v[j], b.v[j]);
    st8s(master + i0, p);
    st8s(m + i0, a);
    st8s(v + i0, b);
    if (w16) st8(w16 + i0, pack8(p.v));
    return;
  }
  for (int64_t i = i0; i < n && i < i0 + 8; ++i) {
    float p = master[i], a = m[i], b = v[i];
    adam_update(s, to_f<G>(grad[i]), p, a, b);
    master[i] = p;
    m[i] = a;
    v[i] = b;
    if (w16) w16[i] = __float2bfloat16(p);
  }
}

// ---- Muon ------------------------------------------------------------------------------
// Matrix update of Muon around its Newton-Schulz iteration (which runs as stacks of GEMMs over the matrices of one
// shape), for all matrices of this rank in one launch each:
//   muon_momentum: g' = g * grad_scale * clip;  buf = lerp(buf, g', 1 - momentum);
//                  u = nesterov ? lerp(g', buf, momentum) : buf;  out = bf16(u), and the sums of u^2 per chunk
//   muon_norms:    inv_norm[matrix] = bf16(1 / (|u| + 1e-7)), summed over the matrix's chunks in order
//   muon_scale:    x = bf16(u * inv_norm), where the iteration starts
//   muon_apply:    w = w * (1 - lr * wd) - lr * adjust * o;  w16 = bf16(w)
// with lr = hyper[0] * lr_ratio (the matrix group follows the schedule of the AdamW group), read from device memory
// so that the launches can be captured.  A block handles one chunk of one matrix:
//   table[matrix] = {offset in the flat gradient / weight buffers, elements, offset in the state buffers},
//   chunks[block] = {matrix, chunk inside it}.
// Bound by memory (12 and 12 bytes per parameter plus the gradient): 16-byte accesses, one launch instead of one per
// matrix (the small matrices of a narrow draft are a few microseconds each).
constexpr int kMuonChunk = 4 * 8 * kOptThreads;

struct MuonChunk {
  int64_t flat, state, count;  // first element in the flat / state buffers, elements of the chunk
  int matrix;
};
__device__ __forceinline__ MuonChunk muon_chunk(const int64_t* __restrict__ table, const int2* __restrict__ chunks) {
  const int2 c = chunks[blockIdx.x];
  const int64_t first = (int64_t)c.y * kMuonChunk, n = table[c.x * 3 + 1] - first;
  return MuonChunk{table[c.x * 3] + first, table[c.x * 3 + 2] + first, n < kMuonChunk ? n : kMuonChunk, c.x};
}

template <typename G>
__global__ void __launch_bounds__(kOptThreads)
muon_momentum_kernel(const G* __restrict__ grad, float* __restrict__ buf, __nv_bfloat16* __restrict__ out, const int64_t* __restrict__ table,
                     const int2* __restrict__ chunks, const float* __restrict__ hyper, const float* __restrict__ norm_sq, float momentum,
                     int nesterov, float* __restrict__ partial) {
  pdl_begin();
  __shared__ float scratch[33];
  const MuonChunk c = muon_chunk(table, chunks);
  const float max_norm = hyper[7];
  float gscale = hyper[8];
  if (max_norm > 0.f && norm_sq) {
    const float coef = max_norm / (gscale * sqrtf(norm_sq[0]) + 1e-6f);
    if (coef < 1.f) gscale *= coef;
  }
  float acc = 0.f;
  auto update = [&](float g, float& b) -> float {
    g *= gscale;
    b += (g - b) * (1.f - momentum);
    return nesterov ? g + (b - g) * momentum : b;
  };
#pragma unroll
  for (int it = 0; it < 4; ++it) {
    const int64_t i = (int64_t)(it * kOptThreads + threadIdx.x) * 8;
    if (i + 8 <= c.count) {
      const f32x8 g = ld8s(grad + c.flat + i);
      f32x8 b = ld8s(buf + c.state + i), u;
#pragma unroll
      for (int j = 0; j < 8; ++j) u.v[j] = update(g.v[j], b.v[j]);
      st8s(buf + c.state + i, b);
      const bf16x8 r = pack8(u.v);
      st8(out + c.state + i, r);
      unpack8(r, u.v);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc += u.v[j] * u.v[j];
    } else {
      for (int64_t k = i; k < c.count; ++k) {
        float b = buf[c.state + k];
        const __nv_bfloat16 r = __float2bfloat16(update(to_f<G>(grad[c.flat + k]), b));
        buf[c.state + k] = b;
        out[c.state + k] = r;
        acc += __bfloat162float(r) * __bfloat162float(r);
      }
    }
  }
  acc = block_sum(acc, scratch);
  if (threadIdx.x == 0) partial[blockIdx.x] = acc;
}

__global__ void __launch_bounds__(kOptThreads)
muon_norms_kernel(const float* __restrict__ partial, const int* __restrict__ first_chunk, float* __restrict__ inv_norm) {
  pdl_begin();
  __shared__ float scratch[33];
  float acc = 0.f;
  for (int i = first_chunk[blockIdx.x] + threadIdx.x; i < first_chunk[blockIdx.x + 1]; i += blockDim.x) acc += partial[i];
  acc = block_sum(acc, scratch);
  if (threadIdx.x == 0) inv_norm[blockIdx.x] = __bfloat162float(__float2bfloat16(1.f / (sqrtf(acc) + 1e-7f)));
}

__global__ void __launch_bounds__(kOptThreads)
muon_scale_kernel(__nv_bfloat16* __restrict__ x, const int64_t* __restrict__ table, const int2* __restrict__ chunks, const float* __restrict__ inv_norm) {
  pdl_begin();
  const MuonChunk c = muon_chunk(table, chunks);
  const float s = inv_norm[c.matrix];
#pragma unroll
  for (int it = 0; it < 4; ++it) {
    const int64_t i = (int64_t)(it * kOptThreads + threadIdx.x) * 8;
    if (i + 8 <= c.count) {
      float u[8];
      unpack8(ld8(x + c.state + i), u);
#pragma unroll
      for (int j = 0; j < 8; ++j) u[j] *= s;
      st8(x + c.state + i, pack8(u));
    } else {
      for (int64_t k = i; k < c.count; ++k) x[c.state + k] = __float2bfloat16(__bfloat162float(x[c.state + k]) * s);
    }
  }
}

__global__ void __launch_bounds__(kOptThreads)
muon_apply_kernel(float* __restrict__ master, const __nv_bfloat16* __restrict__ update, __nv_bfloat16* __restrict__ w16,
                  const int64_t* __restrict__ table, const int2* __restrict__ chunks, const float* __restrict__ adjust,
                  const float* __restrict__ hyper, float lr_ratio, float weight_decay) {
  pdl_begin();
  const MuonChunk c = muon_chunk(table, chunks);
  const float lr = hyper[0] * lr_ratio;
  const float keep = 1.f - lr * weight_decay, step = lr * adjust[c.matrix];
#pragma unroll
  for (int it = 0; it < 4; ++it) {
    const int64_t i = (int64_t)(it * kOptThreads + threadIdx.x) * 8;
    if (i + 8 <= c.count) {
      const f32x8 u = ld8s(update + c.state + i);
      f32x8 w = ld8s(master + c.state + i);
#pragma unroll
      for (int j = 0; j < 8; ++j) w.v[j] = w.v[j] * keep - step * u.v[j];
      st8s(master + c.state + i, w);
      st8(w16 + c.flat + i, pack8(w.v));
    } else {
      for (int64_t k = i; k < c.count; ++k) {
        const float w = master[c.state + k] * keep - step * __bfloat162float(update[c.state + k]);
        master[c.state + k] = w;
        w16[c.flat + k] = __float2bfloat16(w);
      }
    }
  }
}

int muon_chunk_elements() { return kMuonChunk; }

// partial: fp32[num_chunks] scratch; inv_norm: fp32[num_matrices]
void launch_muon_momentum(const void* grad, int grad_is_bf16, float* buf, void* out, const int64_t* table, const int* chunks, int num_chunks,
                          const int* first_chunk, int num_matrices, const float* hyper, const float* norm_sq, float momentum, int nesterov,
                          float* partial, float* inv_norm, cudaStream_t stream) {
  if (num_chunks <= 0) return;
  count_launch(3);
  if (grad_is_bf16)
    launch_pdl(muon_momentum_kernel<__nv_bfloat16>, num_chunks, kOptThreads, 0, stream, (const __nv_bfloat16*)grad, buf, (__nv_bfloat16*)out, table,
               (const int2*)chunks, hyper, norm_sq, momentum, nesterov, partial);
  else
    launch_pdl(muon_momentum_kernel<float>, num_chunks, kOptThreads, 0, stream, (const float*)grad, buf, (__nv_bfloat16*)out, table, (const int2*)chunks,
               hyper, norm_sq, momentum, nesterov, partial);
  launch_pdl(muon_norms_kernel, num_matrices, kOptThreads, 0, stream, partial, first_chunk, inv_norm);
  launch_pdl(muon_scale_kernel, num_chunks, kOptThreads, 0, stream, (__nv_bfloat16*)out, table, (const int2*)chunks, inv_norm);
}

void launch_muon_apply(float* master, const void* update, void* w16, const int64_t* table, const int* chunks, int num_chunks, const float* adjust,
                       const float* hyper, float lr_ratio, float weight_decay, cudaStream_t stream) {
  if (num_chunks <= 0) return;
  count_launch(1);
  launch_pdl(muon_apply_kernel, num_chunks, kOptThreads, 0, stream, master, (const __nv_bfloat16*)update, (__nv_bfloat16*)w16, table, (const int2*)chunks,
             adjust, hyper, lr_ratio, weight_decay);
}

// Hyper-parameters travel as kernel arguments (copied at launch), so the host can
// prepare step k+1 while step k is still queued: no staging buffer to overwrite.
struct HyperVals {
  float v[16];
};
__global__ void set_hyper_kernel(float* __restrict__ hyper, const HyperVals vals) {
  pdl_begin();
  if (threadIdx.x < 16) hyper[threadIdx.x] = vals.v[threadIdx.x];
}

void launch_set_hyper(float* hyper, const float* host_vals16, cudaStream_t stream) {
  HyperVals vals;
  for (int i = 0; i < 16; ++i) vals.v[i] = host_vals16[i];
  count_launch(1);
  launch_pdl(set_hyper_kernel, 1, 32, 0, stream, hyper, vals);
}

int sumsq_num_partials() { return 4 * kNumSM; }

void launch_sumsq(const void* g, int is_bf16, int64_t n, float* partial, float* out, int accumulate,
                  cudaStream_t stream) {
  const int P = sumsq_num_partials();
  count_launch(2);
  if (is_bf16)
    launch_pdl(sumsq_partial_kernel<__nv_bfloat16>, P, kOptThreads, 0, stream, (const __nv_bfloat16*)g, n,
                                                                        partial);
  else
    launch_pdl(sumsq_partial_kernel<float>, P, kOptThreads, 0, stream, (const float*)g, n, partial);
  launch_pdl(sumsq_final_kernel, 1, 256, 0, stream, partial, P, out, accumulate);
}

template <typename G>
static void launch_adamw_as(float* master, float* m, float* v, const G* grad, __nv_bfloat16* w16, int64_t n, const float* hyper,
                            const float* norm_sq, cudaStream_t stream) {
  const uintptr_t bits = reinterpret_cast<uintptr_t>(master) | reinterpret_cast<uintptr_t>(m) | reinterpret_cast<uintptr_t>(v) |
                         reinterpret_cast<uintptr_t>(grad) | reinterpret_cast<uintptr_t>(w16);
  const int64_t grid = (n + 8 * kOptThreads - 1) / (8 * kOptThreads);
  if ((bits & 15) == 0) launch_pdl(adamw_kernel<G, true>, (unsigned)grid, kOptThreads, 0, stream, master, m, v, grad, w16, n, hyper, norm_sq);
  else launch_pdl(adamw_kernel<G, false>, (unsigned)grid, kOptThreads, 0, stream, master, m, v, grad, w16, n, hyper, norm_sq);
}

void launch_adamw(float* master, float* m, float* v, const void* grad, int grad_is_bf16, void* w16,
                  int64_t n, const float* hyper, const float* norm_sq, cudaStream_t stream) {
  if (n <= 0) return;
  count_launch(1);
  if (grad_is_bf16) launch_adamw_as(master, m, v, (const __nv_bfloat16*)grad, (__nv_bfloat16*)w16, n, hyper, norm_sq, stream);
  else launch_adamw_as(master, m, v, (const float*)grad, (__nv_bfloat16*)w16, n, hyper, norm_sq, stream);
}

}  // namespace sb200
