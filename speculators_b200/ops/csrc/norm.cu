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

SB200_BOUNDS_RECORD

// Sum over the block with one barrier: `slot` alternates, so that a slot is written again only after everybody has passed
// the barrier behind its last reading.  The order of the additions is block_sum's.
template <int THREADS>
__device__ __forceinline__ float row_sum(float v, float (&scratch)[2][THREADS / 32], int slot) {
  constexpr int W = THREADS / 32;
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) scratch[slot][threadIdx.x >> 5] = v;
  __syncthreads();
  float s[W];
#pragma unroll
  for (int i = 0; i < W; ++i) s[i] = scratch[slot][i];
#pragma unroll
  for (int half = W / 2; half > 0; half >>= 1)
#pragma unroll
    for (int i = 0; i < half; ++i) s[i] += s[i + half];
  return s[0];
}

// Blocks an SM runs at once, by registers; the grid is no larger (a second, part-filled wave took as long as the first),
// and evens out how many rows its blocks walk.
template <int NV, int THREADS> constexpr int kFwdBlocks = THREADS == 512 ? 1 : NV == 2 ? 5 : NV == 4 ? 4 : 2;

// ADD: the row is x + add, rounded as a sum of its own would be, kept in `sum` and normalised from registers: a block of a decoder
// hands its result to the next norm without reading it back, and a launch less.  Its two reads take the registers that hold the next row
// otherwise; with that too, rows went through local memory (us: a sum and a norm apart, with the next row, now: 1777 x 4096 21.5, 20.5,
// 18.5; 8192 x 4096 73, 74, 59; 500 x 8192 15.4, 20.4, 14.4; 8192 x 8192 128, 170, 105; 8192 x 32768 484, 720, 448).
struct NormAdd {
  const __nv_bfloat16* add;
  __nv_bfloat16* sum;
};
template <int NV, int THREADS, bool ADD = false>
__global__ void __launch_bounds__(THREADS, kFwdBlocks<NV, THREADS>)
rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                   const int64_t* __restrict__ row_index, __nv_bfloat16* __restrict__ y,
                   float* __restrict__ rstd_out, int rows, int H, int64_t x_stride,
                   int64_t y_stride, float eps, int64_t src_rows, NormWeight nw, const int* __restrict__ live, const NormAdd ad) {
  pdl_begin();
  rows = live_rows(live, rows);
  __shared__ float scratch[2][THREADS / 32];
  const int nvec = H >> 3;
  bf16x8 cur[NV], next[ADD ? 1 : NV], cur_add[ADD ? NV : 1];
  bool ok = false, next_ok = false;  // false only in the debug build
  auto fetch = [&](int r, bf16x8 (&to)[NV], bf16x8 (&to_add)[ADD ? NV : 1]) -> bool {
    const int64_t src = row_index ? row_index[r] : (int64_t)r;
    if (!SB200_IN_RANGE(src, src_rows, 1)) return false;
    const __nv_bfloat16* xr = x + src * x_stride;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = threadIdx.x + i * THREADS;
      if (v < nvec) to[i] = ld8(xr + (v << 3));
      if (ADD && v < nvec) to_add[ADD ? i : 0] = ld8(ad.add + (int64_t)r * H + (v << 3));
    }
    return true;
  };
  int r = blockIdx.x, slot = 0;
  if (!ADD && r < rows) ok = fetch(r, cur, cur_add);
  for (; r < rows; r += gridDim.x, slot ^= 1) {
    if constexpr (!ADD) {
      if (r + (int)gridDim.x < rows) next_ok = fetch(r + gridDim.x, next, cur_add);  // in flight during this row's reduction
    } else {
      ok = fetch(r, cur, cur_add);
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int v = threadIdx.x + i * THREADS;
        if (v < nvec) {
          float a[8], b[8];
          unpack8(cur[i], a);
          unpack8(cur_add[ADD ? i : 0], b);
#pragma unroll
          for (int j = 0; j < 8; ++j) a[j] += b[j];
          cur[i] = pack8(a);
          st8(ad.sum + (int64_t)r * H + (v << 3), cur[i]);
        }
      }
    }
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = threadIdx.x + i * THREADS;
      if (ok && v < nvec) {
        float xv[8];
        unpack8(cur[i], xv);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += xv[j] * xv[j];
      }
    }
    ss = row_sum<THREADS>(ss, scratch, slot);
    const float rstd = rsqrtf(ss / (float)H + eps);
    if (ok && threadIdx.x == 0 && rstd_out) rstd_out[r] = rstd;
    __nv_bfloat16* yr = y + (int64_t)r * y_stride;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = threadIdx.x + i * THREADS;
      if (ok && v < nvec) {
        float xv[8], wv[8], o[8];
        unpack8(cur[i], xv);
        nw.load(w + (v << 3), wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = nw.apply(xv[j] * rstd, wv[j]);
        st8(yr + (v << 3), pack8(o));
      }
      if (!ADD) cur[i] = next[ADD ? 0 : i];
    }
    if (!ADD) ok = next_ok;
  }
}

// One CTA walks rows blockIdx.x, +gridDim.x, ... and keeps its dw partial in registers.
// The row's direct gradient and the next row's scale are loaded before the reduction too, which takes one barrier:
// 2048 x 4096 27 -> 18.9 us, 8192 x 4096 92 -> 57.5 (copy bandwidth: 41.6), 1536 x 8192 58 -> 33.6.
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
  const int* live;  // optional: rows in use
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
__device__ __forceinline__ void store_dx(const NormBwdArgs& p, int64_t r, int c, const float (&d)[8], const bf16x8* add = nullptr) {
  if (p.dx == nullptr) return;
  float o[8];
  if (p.add != nullptr) {
    unpack8(add != nullptr ? *add : ld8(p.add + r * p.add_stride + c), o);
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
  const int rows = live_rows(p.live, p.rows);
  __shared__ float scratch[2][THREADS / 32];
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
  int r = blockIdx.x, slot = 0;
  float rstd_next = r < rows ? p.rstd[r] : 0.f;
  if (kPrefetch && r < rows) fetch(r, xa, da);
  for (; r < rows; r += gridDim.x, slot ^= 1) {
    const float rstd = rstd_next;
    const int rn = r + gridDim.x;
    if (rn < rows) rstd_next = p.rstd[rn];
    if constexpr (kPrefetch) {
      if (rn < rows) fetch(rn, xb, db);
    } else {
      fetch(r, xa, da);
    }
    bf16x8 addv[NB];  // this row's direct gradient: its load passes during the reduction too
    if (kPrefetch && p.add != nullptr) {
#pragma unroll
      for (int i = 0; i < NB; ++i) {
        const int v = threadIdx.x + i * THREADS;
        if (v < nvec) addv[i] = ld8(p.add + (int64_t)r * p.add_stride + (v << 3));
      }
    }
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
    dot = row_sum<THREADS>(dot, scratch, slot) / (float)p.H;
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
        store_dx(p, r, v << 3, d, kPrefetch ? &addv[kPrefetch ? i : 0] : nullptr);
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
  const int rows = live_rows(p.live, p.rows);
  __shared__ float tile[kDwGroups][32 * 8 + 8];
  const int c = (blockIdx.x * 32 + threadIdx.x) * 8;
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  if (c < p.H) {
#pragma unroll 4
    for (int r = blockIdx.y * kDwGroups + threadIdx.y; r < rows; r += gridDim.y * kDwGroups) {
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

// The arithmetic of a narrow row's eight elements, rounding by rounding: the kernels below and the ones that do head norms and
// rotation at once share it and give the same bits.  Sums take one fused multiply-add per element; x-hat = x rstd rounds, and
// so does dy w; dx = rstd (dy w - x-hat dot) rounds x-hat dot, fuses dy w into the difference and rounds the product with rstd.
__device__ __forceinline__ float narrow_squares(const float (&x)[8]) {
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) ss = __fmaf_rn(x[j], x[j], ss);
  return ss;
}
__device__ __forceinline__ float narrow_sums(const float (&dy)[8], const float (&w)[8], const float (&x)[8], float rstd, float (&dw)[8]) {
  float dot = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float xh = __fmul_rn(x[j], rstd);
    dot = __fmaf_rn(__fmul_rn(dy[j], w[j]), xh, dot);
    dw[j] = __fmaf_rn(dy[j], xh, dw[j]);
  }
  return dot;
}
__device__ __forceinline__ void narrow_dx(const float (&dy)[8], const float (&w)[8], const float (&x)[8], float rstd, float dot, float (&dx)[8]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) dx[j] = __fmul_rn(rstd, __fmaf_rn(dy[j], w[j], -__fmul_rn(__fmul_rn(x[j], rstd), dot)));
}

__global__ void __launch_bounds__(kNormThreads)
rmsnorm_fwd_narrow_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                          float* __restrict__ rstd_out, int rows, int H, int64_t x_stride, int64_t y_stride, float eps, NormWeight nw, const int* __restrict__ live) {
  pdl_begin();
  rows = live_rows(live, rows);
  const int lane = threadIdx.x & 31, nvec = H >> 3;
  const bool on = lane < nvec;
  float wv[8];
  if (on) nw.load(w + (lane << 3), wv);
  const int warps = gridDim.x * kNarrowWarps;
  for (int r = blockIdx.x * kNarrowWarps + (threadIdx.x >> 5); r < rows; r += warps) {
    float xv[8], ss = 0.f;
    if (on) {
      unpack8(ld8(x + (int64_t)r * x_stride + (lane << 3)), xv);
      ss = narrow_squares(xv);
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
  const int rows = live_rows(p.live, p.rows);
  const int lane = threadIdx.x & 31, nvec = p.H >> 3;
  const bool on = lane < nvec;
  float wv[8], dwacc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) { wv[j] = 0.f; dwacc[j] = 0.f; }
  if (on) p.nw.load(p.w + (lane << 3), wv);
  const int warps = gridDim.x * kNarrowWarps, warp_id = blockIdx.x * kNarrowWarps + (threadIdx.x >> 5);
  for (int r = warp_id; r < rows; r += warps) {
    float xv[8], dv[8], dot = 0.f;
    const float rstd = p.rstd[r];
    if (on) {
      unpack8(ld8(p.x + (int64_t)r * p.x_stride + (lane << 3)), xv);
      unpack8(load_dy(p, r, lane << 3), dv);
      dot = narrow_sums(dv, wv, xv, rstd, dwacc);
    }
    dot = warp_sum(dot) / (float)p.H;
    if (on) {
      float d[8];
      narrow_dx(dv, wv, xv, rstd, dot, d);
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

// dw[c] (+)= bf16(sum_p partial[p, c]).  Block = COLS columns x 32 row-groups; the row-groups split P and meet in shared
// memory, so each column is summed in a fixed order (deterministic), the same for any COLS.  Bound by latency: sixteen loads of a
// thread are issued before the first is added (spelled out: left to the compiler, unrolled loops had three or four in flight
// whatever their depth).  Few columns over thousands of rows (per-head norms) take blocks of 8 columns, whole 32-byte sectors, where 32
// columns a block make four blocks.  us: 4736 x 128 14.3 -> 6.8, 4736 x 256 14.6 -> 10.9; 296 x 1024 .. 8192 as before.
constexpr int kColsumGroups = 32;
struct ColsumJobs {  // blockIdx.y picks one
  const float* partial[2];
  __nv_bfloat16* dw[2];
  int rows[2], accumulate[2];
};
template <int COLS>
__global__ void __launch_bounds__(COLS * kColsumGroups)
colsum_kernel(const ColsumJobs jobs, int H) {
  pdl_begin();
  const float* __restrict__ partial = jobs.partial[blockIdx.y];
  __nv_bfloat16* __restrict__ dw = jobs.dw[blockIdx.y];
  const int P = jobs.rows[blockIdx.y], accumulate = jobs.accumulate[blockIdx.y];
  __shared__ float tile[kColsumGroups][COLS + 1];
  const int c = blockIdx.x * COLS + threadIdx.x;
  float s = 0.f;
  if (c < H) {
    constexpr int FLIGHT = 16;
    const float* at = partial + (int64_t)threadIdx.y * H + c;
    const int64_t step = (int64_t)kColsumGroups * H;
    int left = P > (int)threadIdx.y ? (P - (int)threadIdx.y + kColsumGroups - 1) / kColsumGroups : 0;
    for (; left >= FLIGHT; left -= FLIGHT, at += FLIGHT * step) {
      float v[FLIGHT];
#pragma unroll
      for (int j = 0; j < FLIGHT; ++j) asm volatile("ld.global.f32 %0, [%1];" : "=f"(v[j]) : "l"(at + j * step));
#pragma unroll
      for (int j = 0; j < FLIGHT; ++j) s += v[j];
    }
#pragma unroll 4
    for (; left > 0; --left, at += step) s += *at;
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
static void launch_colsum(const ColsumJobs& jobs, int n, int H, cudaStream_t stream) {
  if (H <= 256) launch_pdl(colsum_kernel<8>, dim3((H + 7) / 8, n), dim3(8, kColsumGroups), 0, stream, jobs, H);
  else launch_pdl(colsum_kernel<32>, dim3((H + 31) / 32, n), dim3(32, kColsumGroups), 0, stream, jobs, H);
}

// ---- per-head norms and rotation of a projection ---------------------------------------------------------------------
// [a heads | b heads | plain heads] per token.  Forward: y = rope(bf16(norm(x))) of the a and b heads into a buffer of
// their own.  Backward: the gradients of all three blocks, each in up to two tensors (rows below `split` and from it on),
// are rotated back, taken through the norm and laid into one buffer of the projection's layout.  One launch each way
// replaces a norm and a rotation per block, and backward the rotation, the norm, the zero-filled slice gradients and
// their sums: 19 passes over the heads of a layer in DFlash's attention.  hd / 8 lanes hold a head (16 bytes each), the
// partner of a rotated pair is hd / 2 channels or less away and comes by shuffle.  Every rounding of the separate
// kernels is kept, and so is the order of every sum (the row groups of the weight gradient are the warps of the narrow
// kernel), so that both forms give the same bits.  Bound by memory; DSpark's five layers at 3000 tokens + 4096 draft
// rows: 11.8 -> 10.95 ms for the step.
struct HeadsRope {
  const int64_t* positions;
  const float* cos_t;
  const float* sin_t;
  int64_t max_pos;
  int rot;
};
// rotate the 8 channels of a lane (index `l` of the head's lanes); all lanes of the warp take part
__device__ __forceinline__ void rotate8(const HeadsRope& p, int64_t t, bool on, int l, float sign, float (&v)[8]) {
  const int half = p.rot >> 1, hl = half >> 3;  // lanes of one half
  const bool first = l < hl, in = l < 2 * hl;
  float other[8];
  const int lane = threadIdx.x & 31, from = in ? (first ? lane + hl : lane - hl) : lane;
#pragma unroll
  for (int j = 0; j < 8; ++j) other[j] = __shfl_sync(0xffffffffu, v[j], from);
  if (!on || !in) return;
  int64_t pos = p.positions[t];
  pos = pos < 0 ? 0 : (pos >= p.max_pos ? p.max_pos - 1 : pos);
  const int64_t at = pos * half + (first ? l : l - hl) * 8;
  const float4 ca = *reinterpret_cast<const float4*>(p.cos_t + at), cb = *reinterpret_cast<const float4*>(p.cos_t + at + 4);
  const float4 sa = *reinterpret_cast<const float4*>(p.sin_t + at), sb = *reinterpret_cast<const float4*>(p.sin_t + at + 4);
  const float c[8] = {ca.x, ca.y, ca.z, ca.w, cb.x, cb.y, cb.z, cb.w};
  const float sn[8] = {sa.x, sa.y, sa.z, sa.w, sb.x, sb.y, sb.z, sb.w};
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float sj = sign * sn[j];
    const float x1 = first ? v[j] : other[j], x2 = first ? other[j] : v[j];
    v[j] = first ? rotate_first(x1, x2, c[j], sj) : rotate_second(x1, x2, c[j], sj);
  }
}
template <int L>
__device__ __forceinline__ float lanes_sum(float v) {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

struct HeadsFwdArgs {
  const __nv_bfloat16* src;
  int64_t src_stride;
  const __nv_bfloat16* w[2];
  int heads[2];
  __nv_bfloat16* out;  // [T, (heads[0] + heads[1]) * hd]
  float* rstd;         // [T * heads[0]] then [T * heads[1]]
  int tokens, src_last;  // tokens from src_last on read that row of src
  float eps;
  HeadsRope rope;
  const int* live;  // optional: tokens in use
};
template <int L>
__global__ void __launch_bounds__(256) heads_fwd_kernel(const HeadsFwdArgs p) {
  pdl_begin();
  constexpr int HD = L * 8;
  const int l = threadIdx.x % L, all = p.heads[0] + p.heads[1];
  const int64_t rows = (int64_t)live_rows(p.live, p.tokens) * all, groups = (int64_t)gridDim.x * (256 / L);
  const NormWeight nw{false};
  for (int64_t base = (int64_t)blockIdx.x * (256 / L) + (threadIdx.x & ~31) / L; base < rows; base += groups) {
    const int64_t r = base + (threadIdx.x & 31) / L;
    const bool on = r < rows;
    const int64_t t = on ? r / all : 0;
    const int c = on ? (int)(r - t * all) : 0, which = c >= p.heads[0], h = which ? c - p.heads[0] : c;
    float xv[8], wv[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) xv[j] = 0.f;
    if (on) unpack8(ld8(p.src + min(t, (int64_t)p.src_last) * p.src_stride + c * HD + l * 8), xv);
    const float ss = narrow_squares(xv);
    nw.load(p.w[which] + l * 8, wv);
    const float rstd = rsqrtf(lanes_sum<L>(ss) / (float)HD + p.eps);
    if (on && l == 0) p.rstd[(which ? (int64_t)p.tokens * p.heads[0] : 0) + t * p.heads[which] + h] = rstd;
#pragma unroll
    for (int j = 0; j < 8; ++j) xv[j] = round_bf16(nw.apply(xv[j] * rstd, wv[j]));
    rotate8(p.rope, t, on, l, 1.f, xv);
    if (on) st8(p.out + r * HD + l * 8, pack8(xv));
  }
}

struct HeadsBwdArgs {
  const __nv_bfloat16* d[3][2];
  int64_t d_stride[3][2];
  int split[3];
  const __nv_bfloat16* src;
  int64_t src_stride;
  const __nv_bfloat16* w[2];
  const float* rstd[2];
  float* partial[2];  // weight gradient sums, one row per group
  int heads[3], groups[3];
  __nv_bfloat16* dst;
  int64_t dst_stride;
  int tokens;
  HeadsRope rope;
  const int* live;  // optional: tokens in use
};
template <int L>
__global__ void __launch_bounds__(256) heads_bwd_kernel(const HeadsBwdArgs p) {
  pdl_begin();
  constexpr int HD = L * 8;
  const int l = threadIdx.x % L;
  int g = (blockIdx.x * 256 + threadIdx.x) / L, which = 0;  // the groups of a block of heads are whole warps
#pragma unroll
  for (int i = 0; i < 2; ++i)
    if (which == i && g >= p.groups[i]) { g -= p.groups[i]; ++which; }
  if (g >= p.groups[which]) return;  // whole warps
  const int heads = which == 0 ? p.heads[0] : which == 1 ? p.heads[1] : p.heads[2], groups = p.groups[which], split = p.split[which];
  const int col0 = (which > 0 ? p.heads[0] * HD : 0) + (which > 1 ? p.heads[1] * HD : 0);
  const int64_t rows = (int64_t)live_rows(p.live, p.tokens) * heads;
  const __nv_bfloat16* d0 = p.d[which][0];
  const __nv_bfloat16* d1 = p.d[which][1];
  const int64_t s0 = p.d_stride[which][0], s1 = p.d_stride[which][1];
  auto gradient = [&](int64_t r, bool on, int64_t& t, int& h) -> bf16x8 {
    t = on ? r / heads : 0;
    h = on ? (int)(r - t * heads) : 0;
    const bool low = t < split;
    const __nv_bfloat16* src = low ? d0 : d1;
    if (on && src != nullptr) return ld8(src + (low ? t * s0 : (t - split) * s1) + h * HD + l * 8);
    const float z[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    return pack8(z);
  };
  if (which == 2) {
    for (int64_t r = g; r < rows; r += groups) {
      int64_t t;
      int h;
      const bf16x8 v = gradient(r, true, t, h);
      st8(p.dst + t * p.dst_stride + col0 + h * HD + l * 8, v);
    }
    return;
  }
  const NormWeight nw{false};
  float wv[8], dwacc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) dwacc[j] = 0.f;
  nw.load(p.w[which] + l * 8, wv);
  const float* rstd_of = p.rstd[which];
  const int trips = (int)((rows + groups - 1) / groups);  // the same in all groups: every lane shuffles
  int64_t t;
  int h;
  bool on = g < rows;
  bf16x8 dn = gradient(g, on, t, h);
  bf16x8 xn = ld8(p.src + t * p.src_stride + col0 + h * HD + l * 8);
  float rn = rstd_of[on ? g : 0];
  for (int i = 0; i < trips; ++i) {
    const bool cur_on = on;
    const int64_t ct = t;
    const int ch = h;
    const float rstd = rn;
    float xv[8], dv[8];
    unpack8(dn, dv);
    unpack8(xn, xv);
    if (i + 1 < trips) {  // the next row's loads are in flight during this one's sums
      const int64_t r = g + (int64_t)(i + 1) * groups;
      on = r < rows;
      dn = gradient(r, on, t, h);
      xn = ld8(p.src + t * p.src_stride + col0 + h * HD + l * 8);
      rn = rstd_of[on ? r : 0];
    }
    rotate8(p.rope, ct, cur_on, l, -1.f, dv);
#pragma unroll
    for (int j = 0; j < 8; ++j) dv[j] = cur_on ? round_bf16(dv[j]) : 0.f;
    const float dot = lanes_sum<L>(narrow_sums(dv, wv, xv, rstd, dwacc)) / (float)HD;
    if (cur_on) {
      float d[8];
      narrow_dx(dv, wv, xv, rstd, dot, d);
      st8(p.dst + ct * p.dst_stride + col0 + ch * HD + l * 8, pack8(d));
    }
  }
  if (p.partial[which] != nullptr) {
    float4* o4 = reinterpret_cast<float4*>(p.partial[which] + (int64_t)g * HD + l * 8);
    o4[0] = make_float4(dwacc[0], dwacc[1], dwacc[2], dwacc[3]);
    o4[1] = make_float4(dwacc[4], dwacc[5], dwacc[6], dwacc[7]);
  }
}

// Rows that were one row of the projection (P-EAGLE's deeper samples all read the same mask token and mask state, so the
// products are formed once): their gradients, rotated back, are summed in fp32 and taken through the norm as one row.
// The result is kept as two bf16 rows, the rounded sum and what the rounding left over, so that the products of the
// backward pass see it at twice the precision.  Two launches: slices of rows by 2048 columns, then one block per head.
struct RepeatedArgs {
  const __nv_bfloat16* d[3];  // gradients of the repeated rows
  int64_t d_stride[3];
  int heads[3], hd, rows, slices;
  float* part;  // [slices][all columns]
  HeadsRope rope;  // positions of the repeated rows
  const __nv_bfloat16* w[2];
  const __nv_bfloat16* src;  // the row of the projection they read
  const float* rstd[2];      // of its heads
  float* dw_part[2];         // one row of hd floats per head
  __nv_bfloat16* dst;        // two rows
  int64_t dst_stride;
};
__global__ void __launch_bounds__(256) repeated_sum_kernel(const RepeatedArgs p) {
  pdl_begin();
  const int64_t cols = (int64_t)(p.heads[0] + p.heads[1] + p.heads[2]) * p.hd, c = ((int64_t)blockIdx.x * 256 + threadIdx.x) * 8;
  if (c >= cols) return;
  int head = (int)(c / p.hd), which = 0;
  const int at = (int)(c - (int64_t)head * p.hd), half = p.rope.rot >> 1;
#pragma unroll
  for (int i = 0; i < 2; ++i)
    if (which == i && head >= p.heads[i]) { head -= p.heads[i]; ++which; }
  const __nv_bfloat16* d = p.d[which];
  const int64_t stride = p.d_stride[which];
  const int col = head * p.hd + at;
  const bool rotated = which < 2 && at < p.rope.rot, first = at < half;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (d != nullptr) {
    for (int r = blockIdx.y; r < p.rows; r += gridDim.y) {
      float v[8];
      unpack8(ld8(d + (int64_t)r * stride + col), v);
      if (!rotated) {
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += v[j];
        continue;
      }
      float o[8];
      unpack8(ld8(d + (int64_t)r * stride + (first ? col + half : col - half)), o);
      int64_t pos = p.rope.positions[r];
      pos = pos < 0 ? 0 : (pos >= p.rope.max_pos ? p.rope.max_pos - 1 : pos);
      const float* cs = p.rope.cos_t + pos * half + (first ? at : at - half);
      const float* sn = p.rope.sin_t + pos * half + (first ? at : at - half);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += first ? v[j] * cs[j] + o[j] * sn[j] : v[j] * cs[j] - o[j] * sn[j];
    }
  }
  float4* out = reinterpret_cast<float4*>(p.part + (int64_t)blockIdx.y * cols + c);
  out[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
  out[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
}
__global__ void __launch_bounds__(256) repeated_finish_kernel(const RepeatedArgs p) {
  pdl_begin();
  __shared__ float scratch[33];
  int head = blockIdx.x, which = 0;
  const int64_t cols = (int64_t)gridDim.x * p.hd;
#pragma unroll
  for (int i = 0; i < 2; ++i)
    if (which == i && head >= p.heads[i]) { head -= p.heads[i]; ++which; }
  for (int at = threadIdx.x; at < ((p.hd + 255) & ~255); at += 256) {
    const int64_t c = (int64_t)blockIdx.x * p.hd + at;
    const bool on = at < p.hd;
    float s = 0.f;
    if (on)
      for (int i = 0; i < p.slices; ++i) s += p.part[(int64_t)i * cols + c];
    if (which < 2) {  // a head is at most 256 wide: one trip
      const float rstd = p.rstd[which][head], w = on ? __bfloat162float(p.w[which][at]) : 0.f;
      const float xh = on ? __bfloat162float(p.src[c]) * rstd : 0.f;
      const float dot = block_sum(s * w * xh, scratch) / (float)p.hd;
      if (on && p.dw_part[which] != nullptr) p.dw_part[which][(int64_t)head * p.hd + at] = s * xh;
      s = rstd * (s * w - xh * dot);
    }
    if (on) {
      const __nv_bfloat16 hi = __float2bfloat16(s);
      p.dst[c] = hi;
      p.dst[p.dst_stride + c] = __float2bfloat16(s - __bfloat162float(hi));
    }
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

static int norm_fwd_grid(int rows, int H, int blocks) {
  if (H <= 4096 && rows <= 16 * kNumSM) return rows;
  const int most = blocks * kNumSM, rounds = (rows + most - 1) / most;
  return (rows + rounds - 1) / rounds;
}

// sum = x + add, y = norm(sum); dense rows of H elements (above kNarrowMaxH, a multiple of 8)
void launch_add_rmsnorm_fwd(const void* x, const void* add, const void* w, void* sum, void* y, int rows, int H, float eps, cudaStream_t stream) {
  if (rows <= 0) return;
  count_launch(1);
#define SB200_ADD(NVV, THREADS)                                                                                                                   \
  launch_pdl(rmsnorm_fwd_kernel<NVV, THREADS, true>, norm_fwd_grid(rows, H, kFwdBlocks<NVV, THREADS>), THREADS, 0, stream, (const __nv_bfloat16*)x, \
             (const __nv_bfloat16*)w, (const int64_t*)nullptr, (__nv_bfloat16*)y, (float*)nullptr, rows, H, (int64_t)H, (int64_t)H, eps, (int64_t)rows, \
             NormWeight{false}, (const int*)nullptr, NormAdd{(const __nv_bfloat16*)add, (__nv_bfloat16*)sum})
  if (H <= 4096) SB200_ADD(2, 256);
  else if (H <= 8192) SB200_ADD(4, 256);
  else if (H <= 16384) SB200_ADD(8, 256);
  else SB200_ADD(8, 512);
#undef SB200_ADD
}

// src_rows: number of rows of `x` (what `row_index` may address).
// live (optional, device): how many of the rows are in use.
void launch_rmsnorm_fwd(const void* x, const void* w, const int64_t* row_index, void* y,
                        float* rstd, int rows, int H, int64_t x_stride, int64_t y_stride, float eps,
                        int64_t src_rows, int centred, const int* live, cudaStream_t stream) {
  if (rows <= 0) return;
  const NormWeight nw{centred != 0};
  count_launch(1);
  if (H <= kNarrowMaxH && row_index == nullptr) {
    launch_pdl(rmsnorm_fwd_narrow_kernel, narrow_grid(rows), kNormThreads, 0, stream, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w,
               (__nv_bfloat16*)y, rstd, rows, H, x_stride, y_stride, eps, nw, live);
    return;
  }
  // A block a row, or blocks that walk rows with the next one in flight.  Measured at 512 to 24576 columns, 128 to 16384 rows
  // (us, a block each and walking).  From L2, back to back: up to 4096 columns walking never gains up to 2368 rows and loses
  // up to a third (1536 x 4096 7.2 and 9.7, 2048 x 2048 6.2 and 6.4), behind them 2 to 20 % (3000 x 2048 8.4 and 9.9, 8192 x
  // 4096 33.8 and 35.9).  From memory it is level or gains a tenth there (8192 x 2048 28.7 and 26.8, 2368 x 4096 18.4 and
  // 16.4) and 15 to 20 % on wide rows, where a block's loads are long (1536 x 24576 57 and 47, from L2 51 and 42).  The line
  // gives few narrow rows, which the step's kernels find in L2, a block each.
  auto grid = [&](int blocks) { return norm_fwd_grid(rows, H, blocks); };
#define SB200_FWD(NVV, THREADS)                                                                                          \
  launch_pdl(rmsnorm_fwd_kernel<NVV, THREADS>, grid(kFwdBlocks<NVV, THREADS>), THREADS, 0, stream, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, row_index, \
             (__nv_bfloat16*)y, rstd, rows, H, x_stride, y_stride, eps, src_rows, nw, live, NormAdd{nullptr, nullptr})
  if (H <= 4096) SB200_FWD(2, 256);
  else if (H <= 8192) SB200_FWD(4, 256);
  else if (H <= 16384) SB200_FWD(8, 256);
  else SB200_FWD(8, 512);
#undef SB200_FWD
}

void launch_rmsnorm_bwd(const void* dy, int64_t dy_stride, const void* dy2, int64_t dy2_stride, const void* x, int64_t x_stride, const void* w,
                        const float* rstd, const void* add, int64_t add_stride, void* dx, int64_t dx_stride, float* dw_partial, void* dw, int rows,
                        int H, int accumulate_dw, int centred, const int* live, cudaStream_t stream) {
  if (rows <= 0) return;
  typedef const __nv_bfloat16* In;
  const NormBwdArgs p{(In)dy, (In)dy2, (In)x, (In)w, rstd, (In)add, (__nv_bfloat16*)dx, dw_partial, rows, H, dy_stride, dy2_stride, x_stride,
                      add_stride, dx_stride, NormWeight{centred != 0}, live};
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
    launch_colsum(ColsumJobs{{dw_partial, nullptr}, {(__nv_bfloat16*)dw, nullptr}, {partial_rows, 0}, {accumulate_dw, 0}}, 1, H, stream);
}

#define SB200_HEADS(KERNEL, BLOCKS, ARGS)                                                   \
  do {                                                                                      \
    if (hd == 64) launch_pdl(KERNEL<8>, BLOCKS, 256, 0, stream, ARGS);                      \
    else if (hd == 128) launch_pdl(KERNEL<16>, BLOCKS, 256, 0, stream, ARGS);               \
    else launch_pdl(KERNEL<32>, BLOCKS, 256, 0, stream, ARGS);                              \
  } while (0)

// heads: a, b; hd 64, 128 or 256; rot a multiple of 16
// src_last: tokens from there on read that row of src (tokens or more: every token its own)
void launch_heads_fwd(const void* src, int64_t src_stride, const void* const* w, const int* heads, void* out, float* rstd, int tokens, int src_last, float eps,
                      const int64_t* positions, const float* cos_t, const float* sin_t, int64_t max_pos, int hd, int rot, const int* live, cudaStream_t stream) {
  if (tokens <= 0) return;
  typedef const __nv_bfloat16* In;
  const HeadsFwdArgs a{(In)src, src_stride, {(In)w[0], (In)w[1]}, {heads[0], heads[1]}, (__nv_bfloat16*)out, rstd, tokens, src_last, eps,
                       HeadsRope{positions, cos_t, sin_t, max_pos, rot}, live};
  const int64_t blocks = ((int64_t)tokens * (heads[0] + heads[1]) * (hd / 8) + 255) / 256;
  const int grid = (int)(blocks < 16 * kNumSM ? blocks : 16 * kNumSM);
  count_launch(1);
  SB200_HEADS(heads_fwd_kernel, grid, a);
}

int heads_bwd_groups(int tokens, int heads) { return heads > 0 ? narrow_grid(tokens * heads) * kNarrowWarps : 0; }

static int repeated_slices(int rows) { return rows < 96 ? rows : 96; }
int64_t repeated_part_floats(int rows, int heads, int hd) { return (int64_t)repeated_slices(rows) * heads * hd; }

// d / d_stride: [3][2] gradients of the a, b and plain blocks below and from `split` on; rstd: [all_tokens * a] then
// [all_tokens * b]; partial[i]: heads_bwd_groups rows of hd floats, and one more per head with repeated rows.
// all_tokens > tokens: the gradients of the rest (the second of each pair; the a block's rows follow its first ones)
// belong to row `tokens` of src, positions go on, and two more rows of dst receive their sum; part: repeated_part_floats.
void launch_heads_bwd(const void* const* d, const int64_t* d_stride, const int* split, const void* src, int64_t src_stride, const void* const* w,
                      const float* rstd, float* const* partial, void* const* dw, const int* accumulate, const int* heads, void* dst, int64_t dst_stride,
                      int tokens, int all_tokens, float* part, const int64_t* positions, const float* cos_t, const float* sin_t, int64_t max_pos, int hd,
                      int rot, const int* live, cudaStream_t stream) {
  if (tokens <= 0) return;
  typedef const __nv_bfloat16* In;
  const bool repeated = all_tokens > tokens;
  HeadsBwdArgs a{};
  RepeatedArgs q{};
  int64_t groups = 0;
  for (int i = 0; i < 3; ++i) {
    for (int k = 0; k < 2; ++k) {
      a.d[i][k] = (In)d[2 * i + k];
      a.d_stride[i][k] = d_stride[2 * i + k];
    }
    q.d[i] = i == 0 ? (d[0] != nullptr ? (In)d[0] + (int64_t)tokens * d_stride[0] : nullptr) : (In)d[2 * i + 1];
    q.d_stride[i] = d_stride[i == 0 ? 0 : 2 * i + 1];
    q.heads[i] = a.heads[i] = heads[i];
    a.split[i] = repeated ? tokens : split[i];
    a.groups[i] = heads_bwd_groups(tokens, heads[i]);
    groups += a.groups[i];
  }
  for (int i = 0; i < 2; ++i) {
    q.w[i] = a.w[i] = (In)w[i];
    a.partial[i] = partial[i];
    a.rstd[i] = rstd + (i ? (int64_t)all_tokens * heads[0] : 0);
    q.rstd[i] = a.rstd[i] + (int64_t)tokens * heads[i];
    q.dw_part[i] = partial[i] != nullptr ? partial[i] + (int64_t)a.groups[i] * hd : nullptr;
  }
  a.src = (In)src;
  a.src_stride = src_stride;
  a.dst = (__nv_bfloat16*)dst;
  a.dst_stride = dst_stride;
  a.tokens = tokens;
  a.rope = HeadsRope{positions, cos_t, sin_t, max_pos, rot};
  a.live = live;
  const int grid = (int)((groups * (hd / 8) + 255) / 256);
  count_launch(1);
  SB200_HEADS(heads_bwd_kernel, grid, a);
  if (repeated) {
    q.hd = hd;
    q.rows = all_tokens - tokens;
    q.slices = repeated_slices(q.rows);
    q.part = part;
    q.rope = HeadsRope{positions + tokens, cos_t, sin_t, max_pos, rot};
    q.src = (In)src + (int64_t)tokens * src_stride;
    q.dst = a.dst + (int64_t)tokens * dst_stride;
    q.dst_stride = dst_stride;
    const int all = heads[0] + heads[1] + heads[2];
    count_launch(2);
    launch_pdl(repeated_sum_kernel, dim3((all * hd + 2047) / 2048, q.slices), 256, 0, stream, q);
    launch_pdl(repeated_finish_kernel, all, 256, 0, stream, q);
  }
  ColsumJobs jobs{};
  int n = 0;
  for (int i = 0; i < 2; ++i)
    if (partial[i] != nullptr && dw[i] != nullptr) {
      jobs.partial[n] = partial[i];
      jobs.dw[n] = (__nv_bfloat16*)dw[i];
      jobs.rows[n] = a.groups[i] + (repeated ? heads[i] : 0);
      jobs.accumulate[n++] = accumulate[i];
    }
  if (n > 0) {
    count_launch(1);
    launch_colsum(jobs, n, hd, stream);
  }
}

// dst[0 .. 2): the sum of `rows` rows of d in fp32, as a rounded row and the rest; width a multiple of 8
void launch_repeated_rows_sum(const void* d, int64_t d_stride, int rows, int width, float* part, void* dst, int64_t dst_stride, cudaStream_t stream) {
  RepeatedArgs q{};
  q.d[2] = (const __nv_bfloat16*)d;
  q.d_stride[2] = d_stride;
  q.hd = width % 256 == 0 ? 256 : 8;
  q.heads[2] = width / q.hd;
  q.rows = rows;
  q.slices = repeated_slices(rows);
  q.part = part;
  q.dst = (__nv_bfloat16*)dst;
  q.dst_stride = dst_stride;
  count_launch(2);
  launch_pdl(repeated_sum_kernel, dim3((width + 2047) / 2048, q.slices), 256, 0, stream, q);
  launch_pdl(repeated_finish_kernel, q.heads[2], 256, 0, stream, q);
}
#undef SB200_HEADS

}  // namespace sb200
