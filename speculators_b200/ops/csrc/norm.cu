// RMSNorm forward / backward for bf16 activations (fp32 statistics).
//
// Forward:  y[r, :] = x[src(r), :] * rsqrt(mean(x^2) + eps) * w
//   * `row_index` (optional) gathers the input row, which turns the kernel into
//     "embedding lookup + RMSNorm" for the EAGLE-3 first layer;
//   * separate row strides for x and y let the caller write straight into one half
//     of a [T, 2H] buffer, so the concat of normalised embeddings and normalised
//     hidden states never exists as a separate copy.
// Backward: dx = rstd * (g - xhat * mean(g * xhat)),  g = dy * w,  xhat = x * rstd
//           dw[c] = sum_r dy[r, c] * xhat[r, c]   (two-stage: per-CTA partials,
//           then a column reduce; the partial buffer is caller-provided scratch).
//   What autograd would do in passes of its own rides along, rounded as those passes round:
//   * dy may come in two parts (a consumer of one half of a concatenation beside one of the whole),
//   * the gradient that reaches x directly (a residual branch) is added to dx,
//   * dw is stored in bf16 or added to the bf16 gradient of earlier calls.
// `centred`: the weight is 1 + w (zero-centred norms), applied in fp32 without rounding xhat first.
#include "common.cuh"

namespace sb200 {

constexpr int kNormThreads = 256;
// Vectors (8 x bf16) handled per thread are a template parameter NV, the block's threads another:
// H <= threads * 8 * NV.  256 threads at NV 2, 4, 8 serve 4096 / 8192 / 16384 columns, 512 threads at NV 8 serve
// 32768 (the concatenated auxiliary states of a 70B-class verifier: 3 x 8192).
constexpr int kNormMaxH = 32768;

struct NormWeight {
  bool centred;
  __device__ __forceinline__ void load(const __nv_bfloat16* w, float (&wv)[8]) const {
    unpack8(ld8(w), wv);
    if (centred) {
#pragma unroll
      for (int j = 0; j < 8; ++j) wv[j] += 1.f;
    }
  }
  // the plain module normalises in fp32, rounds to bf16, then scales
  __device__ __forceinline__ float apply(float xhat, float w) const { return centred ? xhat * w : __bfloat162float(__float2bfloat16(xhat)) * w; }
};
__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16(v)); }

SB200_BOUNDS_RECORD

template <int NV, int THREADS>
__global__ void __launch_bounds__(THREADS)
rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                   const int64_t* __restrict__ row_index, __nv_bfloat16* __restrict__ y,
                   float* __restrict__ rstd_out, int rows, int H, int64_t x_stride,
                   int64_t y_stride, float eps, int64_t src_rows, NormWeight nw) {
  pdl_begin();
  __shared__ float scratch[33];
  const int nvec = H >> 3;
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    const int64_t src = row_index ? row_index[r] : (int64_t)r;
    if (!SB200_IN_RANGE(src, src_rows, 1)) continue;  // debug build only
    const __nv_bfloat16* xr = x + src * x_stride;
    float cache[NV][8];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = threadIdx.x + i * THREADS;
      if (v < nvec) {
        unpack8(ld8(xr + (v << 3)), cache[i]);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += cache[i][j] * cache[i][j];
      }
    }
    ss = block_sum(ss, scratch);
    const float rstd = rsqrtf(ss / (float)H + eps);
    if (threadIdx.x == 0 && rstd_out) rstd_out[r] = rstd;
    __nv_bfloat16* yr = y + (int64_t)r * y_stride;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = threadIdx.x + i * THREADS;
      if (v < nvec) {
        float wv[8], o[8];
        nw.load(w + (v << 3), wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = nw.apply(cache[i][j] * rstd, wv[j]);
        st8(yr + (v << 3), pack8(o));
      }
    }
  }
}

// One CTA walks rows blockIdx.x, +gridDim.x, ... and keeps its dw partial in registers.
// A row's x and dy stay in registers (packed bf16) between the reduction and the dx pass,
// and the next row is fetched before the block-wide reduction of the current one, so the
// loads of one row overlap the synchronisation of the previous row.
struct NormBwdArgs {
  const __nv_bfloat16* dy;
  const __nv_bfloat16* dy2;  // optional second part of dy
  const __nv_bfloat16* x;
  const __nv_bfloat16* w;
  const float* rstd;
  const __nv_bfloat16* add;  // optional gradient that reaches x directly
  __nv_bfloat16* dx;         // optional
  float* dw_partial;         // optional
  int rows, H;
  int64_t dy_stride, dy2_stride, x_stride, add_stride, dx_stride;
  NormWeight nw;
};
__device__ __forceinline__ bf16x8 load_dy(const NormBwdArgs& p, int64_t r, int c) {
  const bf16x8 d = ld8(p.dy + r * p.dy_stride + c);
  if (p.dy2 == nullptr) return d;
  float a[8], b[8];
  unpack8(d, a);
  unpack8(ld8(p.dy2 + r * p.dy2_stride + c), b);
#pragma unroll
  for (int j = 0; j < 8; ++j) a[j] += b[j];
  return pack8(a);
}
__device__ __forceinline__ void store_dx(const NormBwdArgs& p, int64_t r, int c, const float (&d)[8]) {
  if (p.dx == nullptr) return;
  float o[8];
  if (p.add != nullptr) {
    unpack8(ld8(p.add + r * p.add_stride + c), o);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] += round_bf16(d[j]);
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = d[j];
  }
  st8(p.dx + r * p.dx_stride + c, pack8(o));
}

template <int NV, int THREADS, bool DW>
__global__ void __launch_bounds__(THREADS)
rmsnorm_bwd_kernel(const NormBwdArgs p) {
  pdl_begin();
  __shared__ float scratch[33];
  const int nvec = p.H >> 3;
  float dwacc[DW ? NV : 1][8];
  bf16x8 wreg[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = threadIdx.x + i * THREADS;
    if (v < nvec) wreg[i] = ld8(p.w + (v << 3));
    if (DW) {
#pragma unroll
      for (int j = 0; j < 8; ++j) dwacc[i][j] = 0.f;
    }
  }

  constexpr bool kPrefetch = NV <= 4;  // wider rows would spill: fetch each row when it is due
  constexpr int NB = kPrefetch ? NV : 1;
  bf16x8 xa[NV], da[NV], xb[NB], db[NB];
  auto fetch = [&](int r, bf16x8* xr_, bf16x8* dr_) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = threadIdx.x + i * THREADS;
      if (v < nvec) {
        xr_[i] = ld8(p.x + (int64_t)r * p.x_stride + (v << 3));
        dr_[i] = load_dy(p, r, v << 3);
      }
    }
  };
  int r = blockIdx.x;
  if (kPrefetch && r < p.rows) fetch(r, xa, da);
  for (; r < p.rows; r += gridDim.x) {
    if constexpr (kPrefetch) {
      const int rn = r + gridDim.x;
      if (rn < p.rows) fetch(rn, xb, db);
    } else {
      fetch(r, xa, da);
    }
    const float rstd = p.rstd[r];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = threadIdx.x + i * THREADS;
      if (v < nvec) {
        float xv[8], dv[8], wv[8];
        unpack8(xa[i], xv);
        unpack8(da[i], dv);
        unpack8(wreg[i], wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xh = xv[j] * rstd;
          dot += dv[j] * (p.nw.centred ? 1.f + wv[j] : wv[j]) * xh;
          if (DW) dwacc[i][j] += dv[j] * xh;
        }
      }
    }
    dot = block_sum(dot, scratch) / (float)p.H;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = threadIdx.x + i * THREADS;
      if (v < nvec) {
        float xv[8], dv[8], wv[8], d[8];
        unpack8(xa[i], xv);
        unpack8(da[i], dv);
        unpack8(wreg[i], wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) d[j] = rstd * (dv[j] * (p.nw.centred ? 1.f + wv[j] : wv[j]) - xv[j] * rstd * dot);
        store_dx(p, r, v << 3, d);
      }
    }
    if constexpr (kPrefetch) {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        xa[i] = xb[i];
        da[i] = db[i];
      }
    }
  }
  if (DW) {
    float* out = p.dw_partial + (int64_t)blockIdx.x * p.H;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = threadIdx.x + i * THREADS;
      if (v < nvec) {
        float4* o4 = reinterpret_cast<float4*>(out + (v << 3));
        o4[0] = make_float4(dwacc[i][0], dwacc[i][1], dwacc[i][2], dwacc[i][3]);
        o4[1] = make_float4(dwacc[i][4], dwacc[i][5], dwacc[i][6], dwacc[i][7]);
      }
    }
  }
}

// dw alone: the norm of an input that needs no gradient (the auxiliary states of the verifier), and the weight half of
// rows too wide for the accumulators above.  Nothing has to meet across a row, so a thread owns eight columns and walks
// rows: x and dy are read once, 256 columns x 8 row groups per block.
constexpr int kDwGroups = 8;
__global__ void __launch_bounds__(32 * kDwGroups)
rmsnorm_dw_kernel(const NormBwdArgs p) {
  pdl_begin();
  __shared__ float tile[kDwGroups][32 * 8 + 8];
  const int c = (blockIdx.x * 32 + threadIdx.x) * 8;
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  if (c < p.H) {
#pragma unroll 4
    for (int r = blockIdx.y * kDwGroups + threadIdx.y; r < p.rows; r += gridDim.y * kDwGroups) {
      float xv[8], dv[8];
      const float rstd = p.rstd[r];
      unpack8(ld8(p.x + (int64_t)r * p.x_stride + c), xv);
      unpack8(load_dy(p, r, c), dv);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += dv[j] * (xv[j] * rstd);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) tile[threadIdx.y][threadIdx.x * 8 + j] = acc[j];
  __syncthreads();
  const int t = threadIdx.y * 32 + threadIdx.x, col = blockIdx.x * 256 + t;
  if (col < p.H) {
    float sum = 0.f;
#pragma unroll
    for (int g = 0; g < kDwGroups; ++g) sum += tile[g][t];
    p.dw_partial[(int64_t)blockIdx.y * p.H + col] = sum;
  }
}

// ---- narrow rows (H <= 256: per-head q / k norms) ---------------------------------------------
// One warp per row, lane v holds the row's v-th vector of eight: no shared memory and no block
// barrier per row.  The block-per-row kernels above spend a 256-thread CTA and two barriers on a
// 128-element row (16 active lanes); for the [tokens x heads, head_dim] norms of Qwen3-style
// attention that was 0.3-1.2 ms per launch against about 20 us of memory traffic.
constexpr int kNarrowMaxH = 256;
constexpr int kNarrowWarps = kNormThreads / 32;

__global__ void __launch_bounds__(kNormThreads)
rmsnorm_fwd_narrow_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                          float* __restrict__ rstd_out, int rows, int H, int64_t x_stride, int64_t y_stride, float eps, NormWeight nw) {
  pdl_begin();
  const int lane = threadIdx.x & 31, nvec = H >> 3;
  const bool on = lane < nvec;
  float wv[8];
  if (on) nw.load(w + (lane << 3), wv);
  const int warps = gridDim.x * kNarrowWarps;
  for (int r = blockIdx.x * kNarrowWarps + (threadIdx.x >> 5); r < rows; r += warps) {
    float xv[8], ss = 0.f;
    if (on) {
      unpack8(ld8(x + (int64_t)r * x_stride + (lane << 3)), xv);
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += xv[j] * xv[j];
    }
    ss = warp_sum(ss);
    const float rstd = rsqrtf(ss / (float)H + eps);
    if (lane == 0 && rstd_out) rstd_out[r] = rstd;
    if (on) {
      float o[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = nw.apply(xv[j] * rstd, wv[j]);
      st8(y + (int64_t)r * y_stride + (lane << 3), pack8(o));
    }
  }
}

// dw partials: one row of H floats per warp of the grid (summed by colsum_kernel).
__global__ void __launch_bounds__(kNormThreads)
rmsnorm_bwd_narrow_kernel(const NormBwdArgs p) {
  pdl_begin();
  const int lane = threadIdx.x & 31, nvec = p.H >> 3;
  const bool on = lane < nvec;
  float wv[8], dwacc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) { wv[j] = 0.f; dwacc[j] = 0.f; }
  if (on) p.nw.load(p.w + (lane << 3), wv);
  const int warps = gridDim.x * kNarrowWarps, warp_id = blockIdx.x * kNarrowWarps + (threadIdx.x >> 5);
  for (int r = warp_id; r < p.rows; r += warps) {
    float xv[8], dv[8], dot = 0.f;
    const float rstd = p.rstd[r];
    if (on) {
      unpack8(ld8(p.x + (int64_t)r * p.x_stride + (lane << 3)), xv);
      unpack8(load_dy(p, r, lane << 3), dv);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xh = xv[j] * rstd;
        dot += dv[j] * wv[j] * xh;
        dwacc[j] += dv[j] * xh;
      }
    }
    dot = warp_sum(dot) / (float)p.H;
    if (on) {
      float d[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) d[j] = rstd * (dv[j] * wv[j] - xv[j] * rstd * dot);
      store_dx(p, r, lane << 3, d);
    }
  }
  if (p.dw_partial && on) {
    float4* o4 = reinterpret_cast<float4*>(p.dw_partial + (int64_t)warp_id * p.H + (lane << 3));
    o4[0] = make_float4(dwacc[0], dwacc[1], dwacc[2], dwacc[3]);
    o4[1] = make_float4(dwacc[4], dwacc[5], dwacc[6], dwacc[7]);
  }
}

static int narrow_grid(int rows) {
  const int blocks = (rows + kNarrowWarps - 1) / kNarrowWarps;
  return blocks < 4 * kNumSM ? blocks : 4 * kNumSM;
}

// dw[c] (+)= bf16(sum_p partial[p, c]).  Block = 32 columns x 32 row-groups; the row-groups
// split P (a handful of independent loads per thread) and meet in shared memory, so
// each column is summed in a fixed order (deterministic) by H/32 CTAs.
constexpr int kColsumGroups = 32;
__global__ void __launch_bounds__(32 * kColsumGroups)
colsum_kernel(const float* __restrict__ partial, __nv_bfloat16* __restrict__ dw, int P, int H, int accumulate) {
  pdl_begin();
  __shared__ float tile[kColsumGroups][33];
  const int c = blockIdx.x * 32 + threadIdx.x;
  float s = 0.f;
  if (c < H) {
#pragma unroll 4
    for (int p = threadIdx.y; p < P; p += kColsumGroups) s += partial[(int64_t)p * H + c];
  }
  tile[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && c < H) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < kColsumGroups; ++i) t += tile[i][threadIdx.x];
    dw[c] = __float2bfloat16(accumulate ? __bfloat162float(dw[c]) + round_bf16(t) : t);
  }
}

static bool norm_dw_alone(int H, bool with_dx) { return H > kNarrowMaxH && (!with_dx || H > 16384); }
// rows of the dw partials that launch_rmsnorm_bwd writes
int rmsnorm_bwd_partial_rows(int rows, int H, bool with_dx) {
  if (H <= kNarrowMaxH) return narrow_grid(rows) * kNarrowWarps;  // one partial row per warp
  if (norm_dw_alone(H, with_dx)) {
    const int columns = (H + 255) / 256, slices = (8 * kNumSM + columns - 1) / columns, most = (rows + 4 * kDwGroups - 1) / (4 * kDwGroups);
    return slices < most ? slices : most;
  }
  const int g = 2 * kNumSM;
  return rows < g ? rows : g;
}

SB200_BOUNDS_READER(read_bounds_norm)

// src_rows: number of rows of `x` (what `row_index` may address).
void launch_rmsnorm_fwd(const void* x, const void* w, const int64_t* row_index, void* y,
                        float* rstd, int rows, int H, int64_t x_stride, int64_t y_stride, float eps,
                        int64_t src_rows, int centred, cudaStream_t stream) {
  if (rows <= 0) return;
  const NormWeight nw{centred != 0};
  count_launch(1);
  if (H <= kNarrowMaxH && row_index == nullptr) {
    launch_pdl(rmsnorm_fwd_narrow_kernel, narrow_grid(rows), kNormThreads, 0, stream, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w,
               (__nv_bfloat16*)y, rstd, rows, H, x_stride, y_stride, eps, nw);
    return;
  }
  const int grid = rows < 8 * kNumSM ? rows : 8 * kNumSM;
#define SB200_FWD(NVV, THREADS)                                                                                          \
  launch_pdl(rmsnorm_fwd_kernel<NVV, THREADS>, grid, THREADS, 0, stream, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, row_index, \
             (__nv_bfloat16*)y, rstd, rows, H, x_stride, y_stride, eps, src_rows, nw)
  if (H <= 4096) SB200_FWD(2, 256);
  else if (H <= 8192) SB200_FWD(4, 256);
  else if (H <= 16384) SB200_FWD(8, 256);
  else SB200_FWD(8, 512);
#undef SB200_FWD
}

void launch_rmsnorm_bwd(const void* dy, int64_t dy_stride, const void* dy2, int64_t dy2_stride, const void* x, int64_t x_stride, const void* w,
                        const float* rstd, const void* add, int64_t add_stride, void* dx, int64_t dx_stride, float* dw_partial, void* dw, int rows,
                        int H, int accumulate_dw, int centred, cudaStream_t stream) {
  if (rows <= 0) return;
  typedef const __nv_bfloat16* In;
  const NormBwdArgs p{(In)dy, (In)dy2, (In)x, (In)w, rstd, (In)add, (__nv_bfloat16*)dx, dw_partial, rows, H, dy_stride, dy2_stride, x_stride,
                      add_stride, dx_stride, NormWeight{centred != 0}};
  const int partial_rows = rmsnorm_bwd_partial_rows(rows, H, dx != nullptr), grid = rows < 2 * kNumSM ? rows : 2 * kNumSM;
  const bool alone = norm_dw_alone(H, dx != nullptr);
#define SB200_BWD(NVV, THREADS)                                                                                            \
  do {                                                                                                                     \
    if (dw_partial && !alone) launch_pdl(rmsnorm_bwd_kernel<NVV, THREADS, true>, partial_rows, THREADS, 0, stream, p);      \
    else launch_pdl(rmsnorm_bwd_kernel<NVV, THREADS, false>, grid, THREADS, 0, stream, p);                                  \
  } while (0)
  count_launch((dw_partial && dw ? 2 : 1) + (alone && dx != nullptr && dw_partial ? 1 : 0));
  if (H <= kNarrowMaxH) launch_pdl(rmsnorm_bwd_narrow_kernel, narrow_grid(rows), kNormThreads, 0, stream, p);
  else if (dx != nullptr && H <= 4096) SB200_BWD(2, 256);
  else if (dx != nullptr && H <= 8192) SB200_BWD(4, 256);
  else if (dx != nullptr && H <= 16384) SB200_BWD(8, 256);
  else if (dx != nullptr) launch_pdl(rmsnorm_bwd_kernel<8, 512, false>, grid, 512, 0, stream, p);
#undef SB200_BWD
  if (alone && dw_partial) launch_pdl(rmsnorm_dw_kernel, dim3((H + 255) / 256, partial_rows), dim3(32, kDwGroups), 0, stream, p);
  if (dw_partial && dw)
    launch_pdl(colsum_kernel, (H + 31) / 32, dim3(32, kColsumGroups), 0, stream, dw_partial, (__nv_bfloat16*)dw, partial_rows, H, accumulate_dw);
}

}  // namespace sb200
