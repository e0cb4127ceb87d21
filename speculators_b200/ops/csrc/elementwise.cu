// SwiGLU and rotary-embedding kernels (bf16 in/out, fp32 math).
#include "common.cuh"

namespace sb200 {

// rows_used (optional, device): how many of the rows hold anything (a mixture-of-experts buffer sized for the worst case).
// gate_up is [rows, 2*I] with the gate in columns [0, I) and up in [I, 2I)
// (the gate and up projections run as one GEMM).  h = silu(gate) * up.
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gate_up,
                                  __nv_bfloat16* __restrict__ h, int64_t rows, int I, const int* __restrict__ rows_used) {
  pdl_begin();
  if (rows_used != nullptr) rows = min(rows, (int64_t)*rows_used);
  const int nvec = I >> 3;
  const int64_t total = rows * nvec;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = idx / nvec;
    const int c = (int)(idx - r * nvec) << 3;
    const __nv_bfloat16* base = gate_up + r * 2 * (int64_t)I;
    float g[8], u[8], o[8];
    unpack8(ld8(base + c), g);
    unpack8(ld8(base + I + c), u);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float s = 1.f / (1.f + __expf(-g[j]));
      // eager order: act(gate) rounded to bf16, then times up
      o[j] = __bfloat162float(__float2bfloat16(g[j] * s)) * u[j];
    }
    st8(h + r * (int64_t)I + c, pack8(o));
  }
}

// d(gate_up) from dh: dgate = dh * up * (s + g*s*(1-s)), dup = dh * silu(g)
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ dh,
                                  const __nv_bfloat16* __restrict__ gate_up,
                                  __nv_bfloat16* __restrict__ dgate_up, int64_t rows, int I, const int* __restrict__ rows_used) {
  pdl_begin();
  if (rows_used != nullptr) rows = min(rows, (int64_t)*rows_used);
  const int nvec = I >> 3;
  const int64_t total = rows * nvec;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = idx / nvec;
    const int c = (int)(idx - r * nvec) << 3;
    const __nv_bfloat16* base = gate_up + r * 2 * (int64_t)I;
    __nv_bfloat16* obase = dgate_up + r * 2 * (int64_t)I;
    float g[8], u[8], d[8], dg[8], du[8];
    unpack8(ld8(base + c), g);
    unpack8(ld8(base + I + c), u);
    unpack8(ld8(dh + r * (int64_t)I + c), d);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float s = 1.f / (1.f + __expf(-g[j]));
      dg[j] = d[j] * u[j] * (s + g[j] * s * (1.f - s));
      du[j] = d[j] * g[j] * s;
    }
    st8(obase + c, pack8(dg));
    st8(obase + I + c, pack8(du));
  }
}

// In-place neox rotary embedding on `heads` consecutive heads of width `hd`
// inside a row of `row_stride` elements (q and k live side by side in the fused
// qkv projection output, so one launch rotates both).  Only the first `rot`
// channels of a head rotate (partial rotary).  cos/sin tables are fp32
// [max_pos, rot/2]; `positions` selects the table row per token.  `sign` = +1
// forward, -1 backward (the transpose of a rotation is the inverse rotation).
__global__ void rope_kernel(__nv_bfloat16* __restrict__ x, const int64_t* __restrict__ positions,
                            const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                            int64_t tokens, int heads, int hd, int rot, int64_t row_stride,
                            int64_t max_pos, float sign, const int* __restrict__ live) {
  pdl_begin();
  tokens = live_rows(live, (int)tokens);
  const int half = rot >> 1;
  const int64_t total = tokens * heads * half;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(idx % half);
    const int64_t th = idx / half;
    const int h = (int)(th % heads);
    const int64_t t = th / heads;
    int64_t pos = positions[t];
    pos = pos < 0 ? 0 : (pos >= max_pos ? max_pos - 1 : pos);
    const float c = cos_t[pos * half + i];
    const float s = sign * sin_t[pos * half + i];
    __nv_bfloat16* p = x + t * row_stride + (int64_t)h * hd;
    const float x1 = __bfloat162float(p[i]);
    const float x2 = __bfloat162float(p[i + half]);
    p[i] = __float2bfloat16(rotate_first(x1, x2, c, s));
    p[i + half] = __float2bfloat16(rotate_second(x1, x2, c, s));
  }
}

// Same rotation, eight channel pairs per thread (16-byte accesses); needs rot/2 % 8 == 0
// and 16-byte aligned rows/heads (row_stride % 8 == 0, hd % 8 == 0, aligned base).
__global__ void rope_vec8_kernel(__nv_bfloat16* __restrict__ x, const int64_t* __restrict__ positions,
                                 const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                                 int64_t tokens, int heads, int hd, int rot, int64_t row_stride,
                                 int64_t max_pos, float sign, const int* __restrict__ live) {
  pdl_begin();
  tokens = live_rows(live, (int)tokens);
  const int half = rot >> 1;
  const int hv = half >> 3;
  const int64_t total = tokens * heads * hv;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(idx % hv) << 3;
    const int64_t th = idx / hv;
    const int h = (int)(th % heads);
    const int64_t t = th / heads;
    int64_t pos = positions[t];
    pos = pos < 0 ? 0 : (pos >= max_pos ? max_pos - 1 : pos);
    const float4* c4 = reinterpret_cast<const float4*>(cos_t + pos * half + i);
    const float4* s4 = reinterpret_cast<const float4*>(sin_t + pos * half + i);
    const float4 ca = c4[0], cb = c4[1], sa = s4[0], sb = s4[1];
    const float c[8] = {ca.x, ca.y, ca.z, ca.w, cb.x, cb.y, cb.z, cb.w};
    const float sn[8] = {sa.x, sa.y, sa.z, sa.w, sb.x, sb.y, sb.z, sb.w};
    __nv_bfloat16* p = x + t * row_stride + (int64_t)h * hd + i;
    float x1[8], x2[8], y1[8], y2[8];
    unpack8(ld8(p), x1);
    unpack8(ld8(p + half), x2);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float sj = sign * sn[j];
      y1[j] = rotate_first(x1[j], x2[j], c[j], sj);
      y2[j] = rotate_second(x1[j], x2[j], c[j], sj);
    }
    st8(p, pack8(y1));
    st8(p + half, pack8(y2));
  }
}

// Gradient side of the rotation: up to three column blocks (q | k | v gradients, each with rows of its own stride) are
// rotated back and laid side by side into one buffer, in one pass instead of a concatenation and a rotation in place (or
// a copy and a rotation, where the gradient may be shared).  A head is hd channels, of which the first `rot` rotate in
// the blocks marked so; everything else is copied.
struct RopePart {
  const __nv_bfloat16* src;
  int64_t stride;
  int heads, rotate;
};
struct RopeMerge {
  RopePart part[3];
  __nv_bfloat16* dst;
  int64_t dst_stride;
  const int64_t* positions;
  const float* cos_t;
  const float* sin_t;
  int64_t max_pos;
  int tokens, hd, rot;
  float sign;
  const int* live;  // optional: tokens in use
};
__global__ void __launch_bounds__(256) rope_merge_kernel(const RopeMerge a) {
  pdl_begin();
  const int half = a.rot >> 1, pairs = half >> 3, rotated = pairs + ((a.hd - a.rot) >> 3), plain = a.hd >> 3;
  int units[3], all = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i) { units[i] = a.part[i].heads * (a.part[i].rotate ? rotated : plain); all += units[i]; }
  const int64_t total = (int64_t)live_rows(a.live, a.tokens) * all;
  for (int64_t idx = (int64_t)blockIdx.x * 256 + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * 256) {
    const int t = (int)(idx / all);
    int u = (int)(idx - (int64_t)t * all), col = 0, which = 0;
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (which == i && u >= units[i]) { u -= units[i]; col += a.part[i].heads * a.hd; ++which; }
    const RopePart& p = which == 0 ? a.part[0] : which == 1 ? a.part[1] : a.part[2];
    const __nv_bfloat16* src = p.src + (int64_t)t * p.stride;
    __nv_bfloat16* dst = a.dst + (int64_t)t * a.dst_stride + col;
    if (!p.rotate) {
      st8(dst + u * 8, ld8(src + u * 8));
      continue;
    }
    const int h = u / rotated, r = u - h * rotated;
    if (r >= pairs) {
      const int c = h * a.hd + a.rot + (r - pairs) * 8;
      st8(dst + c, ld8(src + c));
      continue;
    }
    int64_t pos = a.positions[t];
    pos = pos < 0 ? 0 : (pos >= a.max_pos ? a.max_pos - 1 : pos);
    const float4* c4 = reinterpret_cast<const float4*>(a.cos_t + pos * half + r * 8);
    const float4* s4 = reinterpret_cast<const float4*>(a.sin_t + pos * half + r * 8);
    const float4 ca = c4[0], cb = c4[1], sa = s4[0], sb = s4[1];
    const float c[8] = {ca.x, ca.y, ca.z, ca.w, cb.x, cb.y, cb.z, cb.w};
    const float sn[8] = {sa.x, sa.y, sa.z, sa.w, sb.x, sb.y, sb.z, sb.w};
    float x1[8], x2[8], y1[8], y2[8];
    const int at = h * a.hd + r * 8;
    unpack8(ld8(src + at), x1);
    unpack8(ld8(src + at + half), x2);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float sj = a.sign * sn[j];
      y1[j] = rotate_first(x1[j], x2[j], c[j], sj);
      y2[j] = rotate_second(x1[j], x2[j], c[j], sj);
    }
    st8(dst + at, pack8(y1));
    st8(dst + at + half, pack8(y2));
  }
}

// Gated attention: y = out * sigmoid(gate) and its gradients; the gate of head h sits at gate + t * gate_stride + h * head_stride
// (the second half of each head's [query | gate] projection), and so does its gradient.
__global__ void __launch_bounds__(256)
gate_mul_fwd_kernel(const __nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ gate, __nv_bfloat16* __restrict__ y, int tokens, int heads,
                    int hd, int64_t gate_stride, int head_stride) {
  pdl_begin();
  const int per_head = hd >> 3, per_row = heads * per_head;
  const int64_t total = (int64_t)tokens * per_row;
  for (int64_t idx = (int64_t)blockIdx.x * 256 + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * 256) {
    const int t = (int)(idx / per_row), u = (int)(idx - (int64_t)t * per_row), h = u / per_head, c = (u - h * per_head) * 8;
    float o[8], g[8];
    unpack8(ld8(out + idx * 8), o);
    unpack8(ld8(gate + t * gate_stride + h * head_stride + c), g);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] *= __bfloat162float(__float2bfloat16(1.f / (1.f + __expf(-g[j]))));
    st8(y + idx * 8, pack8(o));
  }
}
__global__ void __launch_bounds__(256)
gate_mul_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ gate,
                    __nv_bfloat16* __restrict__ dout, __nv_bfloat16* __restrict__ dgate, int tokens, int heads, int hd, int64_t gate_stride,
                    int head_stride, int64_t dgate_stride) {
  pdl_begin();
  const int per_head = hd >> 3, per_row = heads * per_head;
  const int64_t total = (int64_t)tokens * per_row;
  for (int64_t idx = (int64_t)blockIdx.x * 256 + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * 256) {
    const int t = (int)(idx / per_row), u = (int)(idx - (int64_t)t * per_row), h = u / per_head, c = (u - h * per_head) * 8;
    float d[8], o[8], g[8];
    unpack8(ld8(dy + idx * 8), d);
    unpack8(ld8(out + idx * 8), o);
    unpack8(ld8(gate + t * gate_stride + h * head_stride + c), g);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float s = 1.f / (1.f + __expf(-g[j]));
      g[j] = d[j] * o[j] * s * (1.f - s);
      d[j] *= s;
    }
    st8(dout + idx * 8, pack8(d));
    st8(dgate + t * dgate_stride + h * head_stride + c, pack8(g));
  }
}

static inline int grid_for(int64_t total, int threads) {
  int64_t g = (total + threads - 1) / threads;
  const int64_t cap = (int64_t)kNumSM * 16;
  return (int)(g < cap ? (g > 0 ? g : 1) : cap);
}

void launch_swiglu_fwd(const void* gate_up, void* h, int64_t rows, int I, const int* rows_used, cudaStream_t stream) {
  if (rows <= 0) return;
  count_launch(1);
  launch_pdl(swiglu_fwd_kernel, grid_for(rows * (I >> 3), 256), 256, 0, stream, 
      (const __nv_bfloat16*)gate_up, (__nv_bfloat16*)h, rows, I, rows_used);
}
void launch_swiglu_bwd(const void* dh, const void* gate_up, void* dgate_up, int64_t rows, int I,
                       const int* rows_used, cudaStream_t stream) {
  if (rows <= 0) return;
  count_launch(1);
  launch_pdl(swiglu_bwd_kernel, grid_for(rows * (I >> 3), 256), 256, 0, stream, 
      (const __nv_bfloat16*)dh, (const __nv_bfloat16*)gate_up, (__nv_bfloat16*)dgate_up, rows, I, rows_used);
}
void launch_rope(void* x, const int64_t* positions, const float* cos_t, const float* sin_t,
                 int64_t tokens, int heads, int hd, int rot, int64_t row_stride, int64_t max_pos,
                 float sign, const int* live, cudaStream_t stream) {
  if (tokens <= 0) return;
  count_launch(1);
  const int half = rot >> 1;
  const bool vec = (half % 8 == 0) && (hd % 8 == 0) && (row_stride % 8 == 0) && ((uintptr_t)x % 16 == 0) &&
                   ((uintptr_t)cos_t % 16 == 0) && ((uintptr_t)sin_t % 16 == 0);
  if (vec) {
    launch_pdl(rope_vec8_kernel, grid_for(tokens * heads * (half >> 3), 256), 256, 0, stream, 
        (__nv_bfloat16*)x, positions, cos_t, sin_t, tokens, heads, hd, rot, row_stride, max_pos, sign, live);
    return;
  }
  launch_pdl(rope_kernel, grid_for(tokens * heads * half, 256), 256, 0, stream, 
      (__nv_bfloat16*)x, positions, cos_t, sin_t, tokens, heads, hd, rot, row_stride, max_pos, sign, live);
}

// srcs / strides / heads / rotate: three column blocks (heads 0: absent).  rot and hd multiples of 16 and 8, rows 16-byte aligned.
void launch_rope_merge(const void* const* srcs, const int64_t* strides, const int* heads, const int* rotate, void* dst, int64_t dst_stride,
                       const int64_t* positions, const float* cos_t, const float* sin_t, int64_t max_pos, int tokens, int hd, int rot, float sign,
                       const int* live, cudaStream_t stream) {
  if (tokens <= 0) return;
  RopeMerge a{};
  int64_t units = 0;
  for (int i = 0; i < 3; ++i) {
    a.part[i] = RopePart{(const __nv_bfloat16*)srcs[i], strides[i], heads[i], rotate[i]};
    units += (int64_t)heads[i] * (hd >> 3);
  }
  a.dst = (__nv_bfloat16*)dst;
  a.dst_stride = dst_stride;
  a.positions = positions;
  a.cos_t = cos_t;
  a.sin_t = sin_t;
  a.max_pos = max_pos;
  a.tokens = tokens;
  a.hd = hd;
  a.rot = rot;
  a.sign = sign;
  a.live = live;
  count_launch(1);
  launch_pdl(rope_merge_kernel, grid_for(tokens * units, 256), 256, 0, stream, a);
}

void launch_gate_mul_fwd(const void* out, const void* gate, void* y, int tokens, int heads, int hd, int64_t gate_stride, int head_stride, cudaStream_t stream) {
  if (tokens <= 0) return;
  count_launch(1);
  launch_pdl(gate_mul_fwd_kernel, grid_for((int64_t)tokens * heads * (hd >> 3), 256), 256, 0, stream, (const __nv_bfloat16*)out, (const __nv_bfloat16*)gate,
             (__nv_bfloat16*)y, tokens, heads, hd, gate_stride, head_stride);
}
void launch_gate_mul_bwd(const void* dy, const void* out, const void* gate, void* dout, void* dgate, int tokens, int heads, int hd, int64_t gate_stride,
                         int head_stride, int64_t dgate_stride, cudaStream_t stream) {
  if (tokens <= 0) return;
  count_launch(1);
  launch_pdl(gate_mul_bwd_kernel, grid_for((int64_t)tokens * heads * (hd >> 3), 256), 256, 0, stream, (const __nv_bfloat16*)dy, (const __nv_bfloat16*)out,
             (const __nv_bfloat16*)gate, (__nv_bfloat16*)dout, (__nv_bfloat16*)dgate, tokens, heads, hd, gate_stride, head_stride, dgate_stride);
}

}  // namespace sb200
