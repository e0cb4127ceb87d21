// Row movement of a mixture-of-experts layer whose experts all live on this GPU.
//
// A slot is one (token, choice) pair, slot = token * k + j.  The expert products run over a padded row order
// (expert e owns rows seg[e] .. seg[e + 1], a multiple of 128, of which the first count[e] hold slots in slot order);
// the plan gives both directions of the map, slot_row[slot] and row_slot[row] (-1: padding), so that every pass below
// is a gather: no atomics, no sort, no intermediate copies, and the same bits on every run.
//
//   moe_plan          counts, segment offsets, 256-row tile prefix and both maps, two launches
//   moe_gather        x_pad[row] = x[token(row)], zeros in padding rows
//   moe_gather_bwd    dx[token] = sum_j dx_pad[slot_row]
//   moe_combine       out[token] = sum_j p[slot] y_pad[slot_row] + sigmoid(g[token]) shared[token] + residual[token]
//   moe_combine_bwd   dy_pad[row] = p[slot] dout[token], dp[slot] = <y_pad[row], dout[token]>;
//                     dshared = sigmoid(g) dout, dg = <shared, dout> sigmoid'(g)
//
// All of them are bound by memory: a row is read and written once, 16 bytes per thread and access, one block per row.
// `live` (optional, device): tokens in use; the slots of the others are not placed.  Rows past seg[E] exist in the buffers (their capacity is the worst case) but are neither read nor written.
#include "common.cuh"

namespace sb200 {
namespace moe {

constexpr int kThreads = 256;
constexpr int kPlanThreads = 1024;
constexpr int kMaxExperts = 1024;

// The k largest of a row's values, descending, equal ones by index (NaN counts as the largest, as torch.topk has it).  A warp a
// row, PER values a lane in registers as keys that order like the values; k rounds of a warp-wide maximum.  Bound by the rounds'
// shuffles: 4092 rows of 256, 10 of them, 7 us; a top-k and its sort took 74.  The routing does not call it: equal probabilities are
// common there and keep the order that torch.topk gives them.
template <int PER>
__global__ void __launch_bounds__(256) topk_rows_kernel(const float* __restrict__ p, int rows, int E, int k, int64_t* __restrict__ index) {
  pdl_begin();
  const int r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= rows) return;
  unsigned key[PER];
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int e = j * 32 + lane;
    const unsigned b = e < E ? __float_as_uint(p[(int64_t)r * E + e]) : 0xffffffffu;  // (a place behind the row: the lowest key)
    const bool nan = (b & 0x7fffffffu) > 0x7f800000u;
    key[j] = e >= E ? 0u : nan ? 0xffffffffu : b > 0x80000000u ? ~b : b | 0x80000000u;  // (-0 equals 0)
  }
  for (int i = 0; i < k; ++i) {
    unsigned best = 0;
    int at = 0;
#pragma unroll
    for (int j = PER - 1; j >= 0; --j)
      if (key[j] >= best) {  // the lowest of equal ones
        best = key[j];
        at = j * 32 + lane;
      }
    const unsigned top = __reduce_max_sync(0xffffffffu, best);
    const int e = (int)__reduce_min_sync(0xffffffffu, best == top ? (unsigned)at : 0xffffffffu);
#pragma unroll
    for (int j = 0; j < PER; ++j)
      if (j * 32 + lane == e) key[j] = 0u;
    if (lane == 0) index[(int64_t)r * k + i] = e;
  }
}

__global__ void __launch_bounds__(kPlanThreads)
count_kernel(const int64_t* __restrict__ expert, int n_slots, int E, int* __restrict__ hist, const int* __restrict__ live, int k) {
  pdl_begin();
  n_slots = live_rows(live, n_slots / k) * k;
  __shared__ int count[kMaxExperts];
  for (int e = threadIdx.x; e < E; e += kPlanThreads) count[e] = 0;
  __syncthreads();
  const int i = blockIdx.x * kPlanThreads + threadIdx.x;
  if (i < n_slots) atomicAdd(&count[min(max((int)expert[i], 0), E - 1)], 1);
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += kPlanThreads) hist[blockIdx.x * E + e] = count[e];
}

// Exclusive prefix sums of pad128(total[e]) and of its 256-row tiles by one warp.
__device__ __forceinline__ void scan_segments(const int* total, int E, int* seg, int* tiles) {
  const int lane = threadIdx.x & 31;
  int base = 0, tbase = 0;
  for (int e0 = 0; e0 < E; e0 += 32) {
    const int e = e0 + lane;
    const int rows = e < E ? (total[e] + 127) & ~127 : 0, t = (rows + 255) >> 8;
    int a = rows, b = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, a, o), v = __shfl_up_sync(0xffffffffu, b, o);
      if (lane >= o) { a += u; b += v; }
    }
    if (e < E) { seg[e] = base + a - rows; tiles[e] = tbase + b - t; }
    base += __shfl_sync(0xffffffffu, a, 31);
    tbase += __shfl_sync(0xffffffffu, b, 31);
  }
  if (lane == 0) { seg[E] = base; tiles[E] = tbase; }
}

__global__ void __launch_bounds__(kPlanThreads)
place_kernel(const int64_t* __restrict__ expert, int n_slots, int E, int capacity, const int* __restrict__ hist, int* __restrict__ seg_out,
             int* __restrict__ tiles_out, int* __restrict__ slot_row, int* __restrict__ row_slot, const int* __restrict__ live, int k) {
  pdl_begin();
  n_slots = live_rows(live, n_slots / k) * k;
  __shared__ int total[kMaxExperts], before[kMaxExperts], seg[kMaxExperts + 1], tiles[kMaxExperts + 1];
  extern __shared__ unsigned short warp_count[];  // [32][E]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int e = threadIdx.x; e < E; e += kPlanThreads) {
    int all = 0, mine = 0;
    for (int b = 0; b < (int)gridDim.x; ++b) {
      const int c = hist[b * E + e];
      if (b < (int)blockIdx.x) mine += c;
      all += c;
    }
    total[e] = all;
    before[e] = mine;
  }
  for (int i = threadIdx.x; i < 32 * E; i += kPlanThreads) warp_count[i] = 0;
  __syncthreads();
  if (warp == 0) scan_segments(total, E, seg, tiles);
  const int i = blockIdx.x * kPlanThreads + threadIdx.x;
  const int e = i < n_slots ? min(max((int)expert[i], 0), E - 1) : E;
  const unsigned same = __match_any_sync(0xffffffffu, e);
  const int rank = __popc(same & ((1u << lane) - 1u));
  if (e < E && rank == 0) warp_count[warp * E + e] = (unsigned short)__popc(same);
  __syncthreads();
  for (int x = threadIdx.x; x < E; x += kPlanThreads) {  // slots of the expert in earlier warps of this block
    int run = 0;
    for (int w = 0; w < 32; ++w) {
      const int c = warp_count[w * E + x];
      warp_count[w * E + x] = (unsigned short)run;
      run += c;
    }
  }
  __syncthreads();
  if (e < E) {
    const int row = seg[e] + before[e] + warp_count[warp * E + e] + rank;
    slot_row[i] = row;
    row_slot[row] = i;
  }
  // padding rows: the blocks share the experts, then what lies past the last segment
  for (int x = blockIdx.x * 32 + warp; x < E; x += gridDim.x * 32)
    for (int r = seg[x] + total[x] + lane; r < seg[x + 1]; r += 32) row_slot[r] = -1;
  for (int r = seg[E] + i; r < capacity; r += gridDim.x * kPlanThreads) row_slot[r] = -1;
  if (blockIdx.x == 0) {
    for (int x = threadIdx.x; x <= E; x += kPlanThreads) {
      seg_out[x] = seg[x];
      tiles_out[x] = tiles[x];
    }
  }
}

__global__ void __launch_bounds__(kThreads)
gather_kernel(const __nv_bfloat16* __restrict__ x, int64_t x_stride, const int* __restrict__ row_slot, const int* __restrict__ rows_used, int k,
              __nv_bfloat16* __restrict__ out, int H) {
  pdl_begin();
  const int used = *rows_used;
  for (int row = blockIdx.x; row < used; row += gridDim.x) {
    const int slot = row_slot[row];
    const __nv_bfloat16* src = x + (int64_t)(slot < 0 ? 0 : slot / k) * x_stride;
    for (int c = threadIdx.x * 8; c < H; c += kThreads * 8) {
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (slot >= 0) v = *reinterpret_cast<const uint4*>(src + c);
      *reinterpret_cast<uint4*>(out + (int64_t)row * H + c) = v;
    }
  }
}

__global__ void __launch_bounds__(kThreads)
gather_bwd_kernel(const __nv_bfloat16* __restrict__ d_pad, const int* __restrict__ slot_row, int k, __nv_bfloat16* __restrict__ dx, int H,
                  const int* __restrict__ live) {
  pdl_begin();
  const int64_t t = blockIdx.x;
  if (live != nullptr && t >= *live) return;
  for (int c = threadIdx.x * 8; c < H; c += kThreads * 8) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 5
    for (int j = 0; j < k; ++j) {
      float v[8];
      unpack8(ld8(d_pad + (int64_t)slot_row[t * k + j] * H + c), v);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += v[i];
    }
    st8(dx + t * H + c, pack8(acc));
  }
}

__device__ __forceinline__ float sigmoid(float g) { return 1.f / (1.f + __expf(-g)); }

__global__ void __launch_bounds__(kThreads)
combine_kernel(const __nv_bfloat16* __restrict__ y_pad, const int* __restrict__ slot_row, const __nv_bfloat16* __restrict__ p, int k,
               const __nv_bfloat16* __restrict__ shared, const __nv_bfloat16* __restrict__ gate, const __nv_bfloat16* __restrict__ residual,
               __nv_bfloat16* __restrict__ out, int H, const int* __restrict__ live) {
  pdl_begin();
  const int64_t t = blockIdx.x;
  if (live != nullptr && t >= *live) return;
  const float s = shared != nullptr ? sigmoid(__bfloat162float(gate[t])) : 0.f;
  for (int c = threadIdx.x * 8; c < H; c += kThreads * 8) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, v[8];
#pragma unroll 5
    for (int j = 0; j < k; ++j) {
      const float w = __bfloat162float(p[t * k + j]);
      unpack8(ld8(y_pad + (int64_t)slot_row[t * k + j] * H + c), v);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = fmaf(w, v[i], acc[i]);
    }
    if (shared != nullptr) {
      unpack8(ld8(shared + t * H + c), v);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = fmaf(s, v[i], acc[i]);
    }
    if (residual != nullptr) {
      unpack8(ld8(residual + t * H + c), v);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += v[i];
    }
    st8(out + t * H + c, pack8(acc));
  }
}

// Blocks 0 .. : one padded row each; the last `tokens` blocks (with a shared expert): one token each.
__global__ void __launch_bounds__(kThreads)
combine_bwd_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ y_pad, const int* __restrict__ row_slot,
                   const int* __restrict__ rows_used, const __nv_bfloat16* __restrict__ p, int k, __nv_bfloat16* __restrict__ dy_pad,
                   __nv_bfloat16* __restrict__ dp, const __nv_bfloat16* __restrict__ shared, const __nv_bfloat16* __restrict__ gate,
                   __nv_bfloat16* __restrict__ dshared, __nv_bfloat16* __restrict__ dgate, int tokens, int H,
                   const int* __restrict__ live) {
  pdl_begin();
  __shared__ float scratch[33];
  if ((int)blockIdx.x < tokens) {  // shared expert
    const int64_t t = blockIdx.x;
    if (live != nullptr && t >= *live) return;
    const float s = sigmoid(__bfloat162float(gate[t]));
    float dot = 0.f;
    for (int c = threadIdx.x * 8; c < H; c += kThreads * 8) {
      float d[8], y[8];
      unpack8(ld8(dout + t * H + c), d);
      unpack8(ld8(shared + t * H + c), y);
#pragma unroll
      for (int i = 0; i < 8; ++i) { dot += d[i] * y[i]; d[i] *= s; }
      st8(dshared + t * H + c, pack8(d));
    }
    dot = block_sum(dot, scratch);
    if (threadIdx.x == 0) dgate[t] = __float2bfloat16(dot * s * (1.f - s));
    return;
  }
  const int used = *rows_used;
  for (int row = blockIdx.x - tokens; row < used; row += gridDim.x - tokens) {
    const int slot = row_slot[row];
    const int64_t t = slot < 0 ? 0 : slot / k;
    const float w = slot < 0 ? 0.f : __bfloat162float(p[slot]);
    float dot = 0.f;
    for (int c = threadIdx.x * 8; c < H; c += kThreads * 8) {
      float d[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (slot >= 0) {
        float y[8];
        unpack8(ld8(dout + t * H + c), d);
        unpack8(ld8(y_pad + (int64_t)row * H + c), y);
#pragma unroll
        for (int i = 0; i < 8; ++i) { dot += d[i] * y[i]; d[i] *= w; }
      }
      st8(dy_pad + (int64_t)row * H + c, pack8(d));
    }
    if (slot >= 0) {  // uniform over the block
      dot = block_sum(dot, scratch);
      if (threadIdx.x == 0) dp[slot] = __float2bfloat16(dot);
    }
  }
}

}  // namespace moe

static int row_blocks(int rows) { return rows < 16 * kNumSM ? rows : 16 * kNumSM; }

int launch_topk_rows(const float* p, int rows, int E, int k, int64_t* index, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (E < 1 || E > moe::kMaxExperts || k < 1 || k > E) return -1;
  count_launch(1);
  const int grid = (rows + 7) / 8;
  if (E <= 64) launch_pdl(moe::topk_rows_kernel<2>, grid, 256, 0, stream, p, rows, E, k, index);
  else if (E <= 128) launch_pdl(moe::topk_rows_kernel<4>, grid, 256, 0, stream, p, rows, E, k, index);
  else if (E <= 256) launch_pdl(moe::topk_rows_kernel<8>, grid, 256, 0, stream, p, rows, E, k, index);
  else if (E <= 512) launch_pdl(moe::topk_rows_kernel<16>, grid, 256, 0, stream, p, rows, E, k, index);
  else launch_pdl(moe::topk_rows_kernel<32>, grid, 256, 0, stream, p, rows, E, k, index);
  return 0;
}
int moe_plan_blocks(int n_slots) { return (n_slots + moe::kPlanThreads - 1) / moe::kPlanThreads; }

// hist: int[moe_plan_blocks(n_slots) * E] scratch; k: slots per token
int launch_moe_plan(const int64_t* expert, int n_slots, int E, int capacity, int* hist, int* seg, int* tiles, int* slot_row, int* row_slot,
                    const int* live, int k, cudaStream_t stream) {
  using namespace moe;
  if (E < 1 || E > kMaxExperts || n_slots < 1 || k < 1) return -1;
  const int blocks = moe_plan_blocks(n_slots), smem = 32 * E * (int)sizeof(unsigned short);
  static PerDeviceOnce configured;
  if (configured.needed()) {
    if (cudaFuncSetAttribute(place_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 32 * kMaxExperts * (int)sizeof(unsigned short)) != cudaSuccess) return -2;
    configured.mark();
  }
  count_launch(2);
  launch_pdl(count_kernel, blocks, kPlanThreads, 0, stream, expert, n_slots, E, hist, live, k);
  launch_pdl(place_kernel, blocks, kPlanThreads, smem, stream, expert, n_slots, E, capacity, hist, seg, tiles, slot_row, row_slot, live, k);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

typedef const __nv_bfloat16* In;
typedef __nv_bfloat16* Out;

void launch_moe_gather(const void* x, int64_t x_stride, const int* row_slot, const int* rows_used, int k, void* out, int capacity, int H, cudaStream_t stream) {
  count_launch(1);
  launch_pdl(moe::gather_kernel, row_blocks(capacity), moe::kThreads, 0, stream, (In)x, x_stride, row_slot, rows_used, k, (Out)out, H);
}

void launch_moe_gather_bwd(const void* d_pad, const int* slot_row, int k, void* dx, int tokens, int H, const int* live, cudaStream_t stream) {
  count_launch(1);
  launch_pdl(moe::gather_bwd_kernel, tokens, moe::kThreads, 0, stream, (In)d_pad, slot_row, k, (Out)dx, H, live);
}

void launch_moe_combine(const void* y_pad, const int* slot_row, const void* p, int k, const void* shared, const void* gate, const void* residual,
                        void* out, int tokens, int H, const int* live, cudaStream_t stream) {
  count_launch(1);
  launch_pdl(moe::combine_kernel, tokens, moe::kThreads, 0, stream, (In)y_pad, slot_row, (In)p, k, (In)shared, (In)gate, (In)residual, (Out)out, H, live);
}

void launch_moe_combine_bwd(const void* dout, const void* y_pad, const int* row_slot, const int* rows_used, const void* p, int k, void* dy_pad, void* dp,
                            const void* shared, const void* gate, void* dshared, void* dgate, int tokens, int capacity, int H, const int* live,
                            cudaStream_t stream) {
  count_launch(1);
  const int shared_blocks = shared != nullptr ? tokens : 0;
  launch_pdl(moe::combine_bwd_kernel, shared_blocks + row_blocks(capacity), moe::kThreads, 0, stream, (In)dout, (In)y_pad, row_slot, rows_used, (In)p, k,
             (Out)dy_pad, (Out)dp, (In)shared, (In)gate, (Out)dshared, (Out)dgate, shared_blocks, H, live);
}

}  // namespace sb200
