// Row bookkeeping of the drafts' steps: document intervals, P-EAGLE's sampling and mask, embedding gradients.
//
// All of it is latency, not bandwidth: the torch formulations were 10 to 60 launches of 2 us each (and, in the sampler,
// two host synchronisations per depth) on a few thousand indices.  Single-block kernels scan 8 consecutive entries per
// thread, 8192 per round, so a packed row of ordinary length takes one round.
#include "common.cuh"

namespace sb200 {
namespace rows {

constexpr int kT = 1024, kPer = 8;

// inclusive scan over the block; `scratch`: 32 values
template <typename Op>
__device__ __forceinline__ int block_scan(int v, Op op, int* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v = op(v, u);
  }
  __syncthreads();
  if (lane == 31) scratch[warp] = v;
  __syncthreads();
  int up_to = scratch[lane];  // every warp scans the 32 sums itself: no serial walk over them
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, up_to, o);
    if (lane >= o) up_to = op(up_to, u);
  }
  const int before = __shfl_sync(0xffffffffu, up_to, max(warp - 1, 0));
  return warp > 0 ? op(v, before) : v;
}

// lo / hi of every row under causal + same-document (+ window) masking: equal ids form runs, -1 is padding.
__global__ void __launch_bounds__(kT) document_interval_kernel(const int64_t* __restrict__ doc, int T, int window, int* __restrict__ lo, int* __restrict__ hi) {
  pdl_begin();
  __shared__ int scratch[32], carry;
  if (threadIdx.x == 0) carry = 0;
  for (int base = 0; base < T; base += kT * kPer) {
    const int i0 = base + threadIdx.x * kPer;
    int start[kPer], last = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const int i = i0 + j;
      if (i < T && (i == 0 || doc[i] != doc[i - 1])) last = i;
      start[j] = last;
    }
    __syncthreads();  // carry of the round before
    const int from = carry;
    const int all = block_scan(last, [](int a, int b) { return max(a, b); }, scratch);
    // what the threads before this one reached
    const int up = __shfl_up_sync(0xffffffffu, all, 1);
    int before = from;
    if ((threadIdx.x & 31) != 0) before = max(before, up);
    else for (int w = 0; w < (int)(threadIdx.x >> 5); ++w) before = max(before, scratch[w]);
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const int i = i0 + j;
      if (i < T) {
        int l = max(start[j], before);
        if (window > 0) l = max(l, i - window + 1);
        lo[i] = doc[i] == -1 ? i : l;
        hi[i] = i + 1;
      }
    }
    __syncthreads();
    if (threadIdx.x == kT - 1) carry = max(from, all);
  }
}

// Ordered compaction over n candidates: put(rank, i) for every i with keep(i); returns how many (valid in all threads).
template <typename Keep, typename Put>
__device__ __forceinline__ int compact(int n, Keep keep, Put put, int* scratch, int* total) {
  __syncthreads();
  if (threadIdx.x == 0) *total = 0;
  for (int base = 0; base < n; base += kT * kPer) {
    const int i0 = base + threadIdx.x * kPer;
    unsigned bits = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j)
      if (i0 + j < n && keep(i0 + j)) bits |= 1u << j;
    const int mine = __popc(bits);
    __syncthreads();
    const int from = *total;
    const int upto = block_scan(mine, [](int a, int b) { return a + b; }, scratch);
    int rank = from + upto - mine;
#pragma unroll
    for (int j = 0; j < kPer; ++j)
      if (bits >> j & 1) put(rank++, i0 + j);
    __syncthreads();
    if (threadIdx.x == kT - 1) *total = from + upto;
  }
  __syncthreads();
  return *total;
}

__global__ void __launch_bounds__(kT) compact_kernel(const bool* __restrict__ valid, int T, int64_t* __restrict__ list, int* __restrict__ count) {
  pdl_begin();
  __shared__ int scratch[32], total;
  const int n = compact(T, [&](int i) { return valid[i]; }, [&](int rank, int i) { list[rank] = i; }, scratch, &total);
  if (threadIdx.x == 0) *count = n;
}

// One depth of the sampler: the `take` entries of `pool` that `perm` puts first, ascending (all of it as it is without a
// permutation); their anchors and depths; the successors that are still inside the mask as the next pool.
__global__ void __launch_bounds__(kT)
cod_step_kernel(const int64_t* __restrict__ pool, const int64_t* __restrict__ perm, int take, const bool* __restrict__ valid, int T, int depth, int filter_zero,
                unsigned char* __restrict__ flags, int64_t* __restrict__ picked, int64_t* __restrict__ anchor, int64_t* __restrict__ depths,
                int64_t* __restrict__ next, int* __restrict__ count) {
  pdl_begin();
  __shared__ int scratch[32], total;
  auto put = [&](int rank, int64_t at) {
    picked[rank] = at;
    anchor[rank] = at - depth;
    depths[rank] = depth;
  };
  if (perm != nullptr) {
    for (int i = threadIdx.x; i < T; i += kT) flags[i] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < take; i += kT) flags[pool[perm[i]]] = 1;
    __syncthreads();
    compact(T, [&](int i) { return flags[i] != 0; }, [&](int rank, int i) { put(rank, i); }, scratch, &total);
  } else {
    for (int i = threadIdx.x; i < take; i += kT) put(i, pool[i]);
  }
  __syncthreads();
  auto successor = [&](int i) { const int64_t s = picked[i] + 1; return s >= T ? s - T : s; };
  const int n = compact(take, [&](int i) { const int64_t s = successor(i); return (s != 0 || !filter_zero) && valid[s]; },
                        [&](int rank, int i) { next[rank] = successor(i); }, scratch, &total);
  if (threadIdx.x == 0) *count = n;
}

// table[depth, anchor] = row - T for the rows of depth >= 1 (the caller has filled it with -1)
__global__ void __launch_bounds__(256)
peagle_table_kernel(const int64_t* __restrict__ anchor, const int64_t* __restrict__ depth, const bool* __restrict__ row_valid, int n, int T, int num_depths,
                    int* __restrict__ table) {
  pdl_begin();
  const int r = blockIdx.x * 256 + threadIdx.x;
  if (r >= n || (row_valid != nullptr && !row_valid[r])) return;
  const int64_t d = depth[r], a = anchor[r] < 0 ? anchor[r] + T : anchor[r];
  if (d >= 1 && d < num_depths && a >= 0 && a < T) table[d * T + a] = r - T;
}
__global__ void __launch_bounds__(256)
peagle_spec_kernel(const int64_t* __restrict__ anchor, const int64_t* __restrict__ depth, const bool* __restrict__ row_valid, const int64_t* __restrict__ doc,
                   const int* __restrict__ doc_lo, int n, int T, int num_depths, int window, const int* __restrict__ table, int* __restrict__ lo,
                   int* __restrict__ hi, int* __restrict__ extra) {
  pdl_begin();
  const int r = blockIdx.x * 256 + threadIdx.x;
  if (r >= n) return;
  const int64_t d = depth[r], a0 = anchor[r];
  const int64_t a = min(max(a0 < 0 ? a0 + T : a0, (int64_t)0), (int64_t)T - 1);
  const bool pad = doc[a] == -1 || (row_valid != nullptr && !row_valid[r]);
  int64_t l = doc_lo[a];
  if (window > 0) l = max(l, a0 + d - window + 1);
  lo[r] = pad ? 0 : (int)l;
  hi[r] = pad ? 0 : (int)(a0 + 1);
  if (extra != nullptr)
    for (int e = 1; e < num_depths; ++e) extra[(int64_t)r * (num_depths - 1) + e - 1] = d >= e && !pad ? table[(int64_t)e * T + a] : -1;
}

// ---- rows that a step needs --------------------------------------------------------------------------------------
// In a training-time-test step row t is wanted where its loss in some pass s < S (label and target row t + s, loss_mask[t + s])
// or its run of correct passes (loss_mask[t]) counts; every other row only serves as context keys of pass 0.  The verifier's
// row u is wanted where some wanted comparison reads it.  Block 0 lists the first, block 1 the second, ascending, as
// index (row of the step -> row of the batch) and inverse (-1: not listed).  Labels may reach past the rows (N >= T of them; there
// is no verifier's list then).  The count is rounded up to 256, so that no GEMM
// or attention tile and no contraction step of 128 straddles it, by rows that nobody asked for (the last ones): they are
// computed like any other and their gradients are exact zeros.
constexpr int kKept = 16;  // rounds of which the flags stay in shared memory: 131072 rows
__global__ void __launch_bounds__(kT)
wanted_rows_kernel(const uint8_t* __restrict__ mask, int T, int N, int S, int64_t* __restrict__ index, int* __restrict__ inverse, int* __restrict__ count) {
  pdl_begin();
  __shared__ int scratch[32], total, carry;
  __shared__ uint8_t kept[kKept * kT];
  const int dir = blockIdx.x == 0 ? 1 : -1, rounds = (T + kT * kPer - 1) / (kT * kPer);
  index += (int64_t)blockIdx.x * T;
  inverse += (int64_t)blockIdx.x * T;
  auto wanted = [&](int round) {  // bit j: row i0 + j
    const int i0 = (round * kT + threadIdx.x) * kPer;
    unsigned bits = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j)
      for (int s = 0; s < S; ++s) {
        const int u = i0 + j + dir * s;
        if (i0 + j < T && u >= 0 && u < N && mask[u] != 0) bits |= 1u << j;
      }
    return bits;
  };
  int mine = 0;
  for (int round = 0; round < rounds; ++round) {
    const unsigned bits = wanted(round);
    if (round < kKept) kept[round * kT + threadIdx.x] = (uint8_t)bits;
    mine += __popc(bits);
  }
  const auto plus = [](int a, int b) { return a + b; };
  const int up_to = block_scan(mine, plus, scratch);
  if (threadIdx.x == kT - 1) total = up_to;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int n = total, live = min(T, max(256, (n + 255) & ~255)), drop = T - live;  // the first `drop` unwanted rows stay out
  for (int round = 0; round < rounds; ++round) {
    const unsigned bits = round < kKept ? kept[round * kT + threadIdx.x] : wanted(round);
    const int here = __popc(bits), from = carry, upto = rounds == 1 ? up_to : block_scan(here, plus, scratch);
    int rank = from + upto - here;  // wanted rows before this one
    const int i0 = (round * kT + threadIdx.x) * kPer;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const int i = i0 + j, unwanted = i - rank;
      if (i >= T) break;
      const bool want = bits >> j & 1, in = want || unwanted >= drop;
      const int at = rank + max(0, unwanted - drop);
      inverse[i] = in ? at : -1;
      if (in) index[at] = i;
      rank += want;
    }
    __syncthreads();
    if (threadIdx.x == kT - 1) carry = from + upto;
    __syncthreads();
  }
  if (threadIdx.x == 0) count[blockIdx.x] = live;
}

// What the passes read of the listed rows: ids, positions and label masks shifted by the pass, the verifier's listed row to
// compare with (-1: none), the first run of correct passes, key intervals, and each later pass's own keys of the earlier ones.
struct StepRows {
  const uint8_t* mask;
  const int64_t *ids, *positions;
  const int* interval[2];  // [2, T] lo and hi (optional)
  const int64_t* index;
  const int *inverse, *count;  // of both lists
  int T, N, S;
  int64_t *ids_out, *positions_out;  // [S, T]
  uint8_t *mask_out, *prev_out;      // [S, T], [T]
  int* target_row;                   // [S, T]
  int* interval_out[2];              // [2, T]
  int* extra;                        // pass s from row T s (s - 1) / 2 on: [T, s]
};
__global__ void __launch_bounds__(256) step_rows_kernel(const StepRows p) {
  pdl_begin();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= p.T) return;
  const bool on = i < p.count[0];
  const int64_t t = on ? p.index[i] : 0;
  p.prev_out[i] = on && p.mask[t] != 0;
#pragma unroll
  for (int k = 0; k < 2; ++k)
    if (p.interval[k] != nullptr) {
      p.interval_out[k][i] = on ? p.interval[k][t] : 0;
      p.interval_out[k][p.T + i] = on ? p.interval[k][p.T + t] : 0;
    }
  for (int s = 0; s < p.S; ++s) {
    const int64_t u = t + s, at = (int64_t)s * p.T + i;
    const bool in = on && u < p.N;
    p.ids_out[at] = in ? p.ids[u] : 0;
    p.positions_out[at] = on ? p.positions[t] + s : 0;
    p.mask_out[at] = in && p.mask[u] != 0;
    if (p.target_row != nullptr) p.target_row[at] = in ? p.inverse[p.T + u] : -1;
    int* extra = p.extra + (int64_t)p.T * (s * (s - 1) / 2) + (int64_t)i * s;
    for (int j = 0; j < s; ++j) extra[j] = on ? j * p.T + i : -1;
  }
}

// Rows of up to two matrices at once (blockIdx.y), 16 bytes per thread.  Taken: out[r] = x[index[r]] for the rows in use.
struct RowCopies {
  const __nv_bfloat16* from[2];
  int64_t stride[2];
  __nv_bfloat16* to[2];
  int W[2];
  int rows;
};
__global__ void __launch_bounds__(256) take_rows_kernel(const RowCopies p, const int64_t* __restrict__ index, const int* __restrict__ live) {
  pdl_begin();
  const bool second = blockIdx.y != 0;
  const __nv_bfloat16* x = second ? p.from[1] : p.from[0];
  __nv_bfloat16* out = second ? p.to[1] : p.to[0];
  const int64_t stride = second ? p.stride[1] : p.stride[0];
  const int W = second ? p.W[1] : p.W[0], per = W >> 3;
  const int64_t total = (int64_t)live_rows(live, p.rows) * per;
  for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < total; e += (int64_t)gridDim.x * 256) {
    const int64_t r = e / per;
    const int c = (int)(e - r * per) * 8;
    st8(out + r * W + c, ld8(x + index[r] * stride + c));
  }
}
// the way back: out[t] = d[inverse[t]], zero where the row was not taken
__global__ void __launch_bounds__(256) put_rows_kernel(const RowCopies p, const int* __restrict__ inverse) {
  pdl_begin();
  const bool second = blockIdx.y != 0;
  const __nv_bfloat16* d = second ? p.from[1] : p.from[0];
  __nv_bfloat16* out = second ? p.to[1] : p.to[0];
  const int64_t stride = second ? p.stride[1] : p.stride[0];
  const int W = second ? p.W[1] : p.W[0], per = W >> 3;
  const int64_t total = (int64_t)p.rows * per;
  const float zero[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < total; e += (int64_t)gridDim.x * 256) {
    const int64_t t = e / per;
    const int c = (int)(e - t * per) * 8, from = inverse[t];
    st8(out + t * W + c, from >= 0 ? ld8(d + (int64_t)from * stride + c) : pack8(zero));
  }
}

// Gradient rows of an embedding from ids in ascending order (`order`: where each came from), summed in fp32 in a fixed order
// and stored into, or added to, the id's row of dw.  Rows of other ids are not touched.
//
// The positions are cut into slices of 32, and a block sums what one id has in one slice: its loads do not depend on one
// another, and however often an id comes (frequent tokens, the padding of a batch) no block walks more than 32 rows.  An id
// that lies in one slice is done then; one that crosses into others leaves a partial row per slice (an id has at most two
// kinds in a slice: it starts there, row 2 k + 1, or it comes from the slice before, row 2 k), and embedding_join_kernel
// sums those.  As one block per id, the loop's exit hanging on a load, a step with real text waited for its most frequent id:
// added to a 152k x 4096 table, 8194 rows with Zipf's frequencies (673 of one id) 841 -> 46 us, a quarter of them padding
// 2545 -> 50, all one id 9926 -> 50; ids that hardly repeat 47 -> 52 (2050 rows: 18.5 -> 21.5), the second launch.
constexpr int kSlice = 32;
__device__ __forceinline__ bool embedding_id_ok(int64_t id, int64_t vocab, int64_t padding) { return id != padding && id >= 0 && id < vocab; }

__global__ void __launch_bounds__(256)
embedding_bwd_kernel(const int64_t* __restrict__ ids, const int64_t* __restrict__ order, const __nv_bfloat16* __restrict__ d, int64_t d_stride, int n, int H,
                     int64_t vocab, int64_t padding, __nv_bfloat16* __restrict__ dw, int accumulate, float* __restrict__ part) {
  pdl_begin();
  __shared__ int64_t rows[kSlice];
  const int i = blockIdx.x, slice = i / kSlice, stop = slice * kSlice + min(n - slice * kSlice, kSlice), lane = threadIdx.x & 31;
  // one round of loads for all that the block has to know, whether it needs it or not
  const int at = i + min(lane, stop - i - 1);
  const int64_t id = ids[i], before = ids[max(i - 1, 0)], mine = ids[at], next = ids[min(stop, n - 1)], row = order[at];
  const bool starts = i == 0 || before != id;
  if ((!starts && i % kSlice != 0) || !embedding_id_ok(id, vocab, padding)) return;
  const bool same = lane < stop - i && mine == id, more = stop < n && next == id;
  const int len = __popc(__ballot_sync(0xffffffffu, same));  // ascending: the equal ones come first
  if (threadIdx.x < len) rows[threadIdx.x] = row;
  __syncthreads();
  const bool whole = starts && !(more && i + len == stop);
  for (int c = threadIdx.x * 8; c < H; c += 256 * 8) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, v[8];
#pragma unroll 4
    for (int j = 0; j < len; ++j) {
      unpack8(ld8(d + rows[j] * d_stride + c), v);
#pragma unroll
      for (int u = 0; u < 8; ++u) acc[u] += v[u];
    }
    if (!whole) {
      float4* out = reinterpret_cast<float4*>(part + (2 * (int64_t)slice + starts) * H + c);
      out[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
      out[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
      continue;
    }
    __nv_bfloat16* out = dw + id * (int64_t)H + c;
    if (accumulate) {
      unpack8(ld8(out), v);
#pragma unroll
      for (int u = 0; u < 8; ++u) acc[u] = round_bf16(acc[u]) + v[u];
    }
    st8(out, pack8(acc));
  }
}

// One block: 128 columns of the ids that start in one of 8 slices and cross into the next.  A warp takes a slice and sums an id
// that comes into few others by itself; for longer ones the eight warps share the partial rows and meet in shared memory (8194 rows in runs of 40: 46 us, 58 where the
// block took one id after the other).
constexpr int kJoinSlices = 8, kJoinAlone = 8;
__device__ __forceinline__ void add4(float4& a, const float4& b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }
__device__ __forceinline__ void embedding_store4(__nv_bfloat16* dw, int accumulate, float4 v) {
  __nv_bfloat162* out = reinterpret_cast<__nv_bfloat162*>(dw);
  if (accumulate) {
    const float2 a = __bfloat1622float2(out[0]), b = __bfloat1622float2(out[1]);
    v = make_float4(round_bf16(v.x) + a.x, round_bf16(v.y) + a.y, round_bf16(v.z) + b.x, round_bf16(v.w) + b.y);
  }
  out[0] = __floats2bfloat162_rn(v.x, v.y);
  out[1] = __floats2bfloat162_rn(v.z, v.w);
}
__global__ void __launch_bounds__(32 * kJoinSlices)
embedding_join_kernel(const int64_t* __restrict__ ids, const float* __restrict__ part, int n, int H, int64_t vocab, int64_t padding,
                      __nv_bfloat16* __restrict__ dw, int accumulate) {
  pdl_begin();
  constexpr int kThreads = 32 * kJoinSlices;
  __shared__ float4 tile[kJoinSlices][32];
  __shared__ int shared_by_all[kJoinSlices];
  const int slices = (n - 1) / kSlice + 1, k0 = blockIdx.x * kJoinSlices, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.y * 128 + lane * 4;
  // the warp's slice: what starts in it and comes into `further` others, as far as 32 lanes see
  const int mine = k0 + warp;
  int further = 0;
  if (mine + 1 < slices) {
    const int begin = mine * kSlice;
    const int64_t id = ids[begin + kSlice], last = ids[begin + kSlice - 1], before = ids[max(begin - 1, 0)];
    const int m = mine + 1 + min(lane, slices - 2 - mine);
    const bool same = lane < slices - 1 - mine && ids[m * kSlice] == id;
    if (last == id && (begin == 0 || before != id) && embedding_id_ok(id, vocab, padding)) further = __popc(__ballot_sync(0xffffffffu, same));
    if (further > 0 && further <= kJoinAlone && c < H) {
      float4 acc = *reinterpret_cast<const float4*>(part + (2 * (int64_t)mine + 1) * H + c);
#pragma unroll
      for (int r = 1; r <= kJoinAlone; ++r)
        if (r <= further) add4(acc, *reinterpret_cast<const float4*>(part + 2 * (int64_t)(mine + r) * H + c));
      embedding_store4(dw + id * (int64_t)H + c, accumulate, acc);
    }
  }
  if (lane == 0) shared_by_all[warp] = further > kJoinAlone;
  __syncthreads();
  for (int s = 0; s < kJoinSlices; ++s) {
    if (!shared_by_all[s]) continue;
    const int k = k0 + s;
    const int64_t id = ids[(k + 1) * kSlice];
    int got;
    further = 0;
    do {
      const int m = k + 1 + further + threadIdx.x;
      got = __syncthreads_count(m < slices && ids[min(m, slices - 1) * kSlice] == id);
      further += got;
    } while (got == kThreads);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < H) {
#pragma unroll 4
      for (int r = warp; r <= further; r += kJoinSlices) add4(acc, *reinterpret_cast<const float4*>(part + (2 * (int64_t)(k + r) + (r == 0)) * H + c));
    }
    tile[warp][lane] = acc;
    __syncthreads();
    if (warp == 0 && c < H) {
#pragma unroll
      for (int w = 1; w < kJoinSlices; ++w) add4(acc, tile[w][lane]);
      embedding_store4(dw + id * (int64_t)H + c, accumulate, acc);
    }
    __syncthreads();  // the tile is written again
  }
}

// ---- anchored blocks (DFlash, DSpark) ------------------------------------------------------------
// Up to `take_most` of the valid rows, the ones with the smallest keys (keys in [0, 1), ties to the lower row), ascending, padded with
// zeros; a flag per slot.  The last `block` rows are never anchors.  One block: the k-th smallest key by its bits, eight at a time
// (positive floats order like their bits), then an ordered compaction.  As a top-k of the keys, a sort of the picks and the
// arithmetic around them it was 25 launches: 512 of 3000 rows, blocks of 8, took 85 us, now 11, and with the two specs and the slots' indices
// (70 launches) 190 us, now 27.
__global__ void __launch_bounds__(kT)
select_anchors_kernel(const bool* __restrict__ mask, const float* __restrict__ keys, int T, int block, int slots, int take_most, int64_t* __restrict__ anchors,
                      bool* __restrict__ picked) {
  pdl_begin();
  __shared__ int scratch[32], total, hist[256], sh_digit, sh_below, cutoff;
  const int usable = T - block;  // rows from there on are never anchors
  auto valid = [&](int i) { return i < usable && mask[i]; };
  auto bits = [&](int i) { return __float_as_uint(keys[i]); };
  for (int i = threadIdx.x; i < slots; i += kT) {
    anchors[i] = 0;
    picked[i] = false;
  }
  int mine = 0;
  for (int i = threadIdx.x; i < usable; i += kT) mine += mask[i] ? 1 : 0;
  block_scan(mine, [](int a, int b) { return a + b; }, scratch);
  __syncthreads();
  int n = 0;
  for (int w = 0; w < 32; ++w) n += scratch[w];
  const int take = min(take_most, n);
  unsigned thr = 0xffffffffu;
  int last = T;  // equal keys count up to this row
  if (take < n && take > 0) {
    unsigned prefix = 0, known = 0;
    int need = take;  // of the keys that share the digits found so far
    for (int shift = 24; shift >= 0; shift -= 8) {
      for (int i = threadIdx.x; i < 256; i += kT) hist[i] = 0;
      __syncthreads();
      for (int i = threadIdx.x; i < usable; i += kT)
        if (mask[i] && (bits(i) & known) == prefix) atomicAdd(&hist[(bits(i) >> shift) & 255], 1);
      __syncthreads();
      const int h = threadIdx.x < 256 ? hist[threadIdx.x] : 0;
      const int upto = block_scan(h, [](int a, int b) { return a + b; }, scratch);
      if (threadIdx.x < 256 && upto >= need && upto - h < need) {
        sh_digit = threadIdx.x;
        sh_below = upto - h;
      }
      __syncthreads();
      prefix |= (unsigned)sh_digit << shift;
      known |= 255u << shift;
      need -= sh_below;
      if (shift == 0) total = hist[sh_digit];
      __syncthreads();
    }
    thr = prefix;
    if (total > need) {  // more keys equal the last one taken than are wanted
      compact(usable, [&](int i) { return mask[i] && bits(i) == thr; }, [&](int rank, int i) { if (rank == need - 1) cutoff = i; }, scratch, &total);
      last = cutoff;
    }
  }
  if (take > 0)
    compact(usable, [&](int i) { return valid(i) && (bits(i) < thr || (bits(i) == thr && i <= last)); },
            [&](int rank, int i) { anchors[rank] = i; picked[rank] = true; }, scratch, &total);
}

// Context interval of a block's rows - the anchor's document before the anchor, inside the window if there is one - and the rows of the
// block as extra keys (up to the row itself with `causal`).  One thread an extra key.
__global__ void __launch_bounds__(256)
anchor_spec_kernel(const int64_t* __restrict__ doc, const int* __restrict__ doc_lo, int T, const int64_t* __restrict__ anchors, int n, int block, int window,
                   int causal, int* __restrict__ lo, int* __restrict__ hi, int* __restrict__ extra) {
  pdl_begin();
  const int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x;
  const int64_t row = e / block;
  if (row >= (int64_t)n * block) return;
  const int slot = (int)(e - row * block);
  const int64_t blk = row / block;
  extra[e] = !causal || slot <= (int)(row - blk * block) ? (int)(blk * block) + slot : -1;
  if (slot != 0) return;
  const int64_t a = anchors[blk];
  const bool seen = a >= 0 && a < T && doc[a] != -1;
  const int first = seen ? doc_lo[a] : 0;
  lo[row] = !seen ? 0 : window >= 0 ? max(first, (int)a - window) : first;
  hi[row] = seen ? (int)a : 0;
}

// What a block's slots read: token, position, row of the packed sequence, row of the targets, and whether a loss counts there.
__global__ void __launch_bounds__(256)
anchor_slots_kernel(const int64_t* __restrict__ anchors, const bool* __restrict__ picked, const int64_t* __restrict__ ids, const int64_t* __restrict__ positions,
                    const bool* __restrict__ mask, int T, int n, int block, int64_t mask_token, int from_anchor, int64_t* __restrict__ token,
                    int64_t* __restrict__ position, int64_t* __restrict__ index, int64_t* __restrict__ target, bool* __restrict__ counts) {
  pdl_begin();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n * block) return;
  const int blk = i / block, slot = i - blk * block;
  const int64_t a = anchors[blk], at = a + slot;
  token[i] = slot == 0 ? ids[a] : mask_token;
  position[i] = positions[a] + slot;
  index[i] = at;
  const int64_t t = from_anchor ? at : at - 1;
  target[i] = t < 0 ? t + T : t % T;
  counts[i] = picked[blk] && at < T && mask[at] && (from_anchor || slot != 0);
}

}  // namespace rows

void launch_select_anchors(const bool* mask, const float* keys, int T, int block, int slots, int take_most, int64_t* anchors, bool* picked, cudaStream_t stream) {
  count_launch(1);
  launch_pdl(rows::select_anchors_kernel, 1, rows::kT, 0, stream, mask, keys, T, block, slots, take_most, anchors, picked);
}
void launch_anchor_spec(const int64_t* doc, const int* doc_lo, int T, const int64_t* anchors, int n, int block, int window, int causal, int* lo, int* hi,
                        int* extra, cudaStream_t stream) {
  const int64_t elements = (int64_t)n * block * block;
  if (elements <= 0) return;
  count_launch(1);
  launch_pdl(rows::anchor_spec_kernel, (int)((elements + 255) / 256), 256, 0, stream, doc, doc_lo, T, anchors, n, block, window, causal, lo, hi, extra);
}
void launch_anchor_slots(const int64_t* anchors, const bool* picked, const int64_t* ids, const int64_t* positions, const bool* mask, int T, int n, int block,
                         int64_t mask_token, int from_anchor, int64_t* token, int64_t* position, int64_t* index, int64_t* target, bool* counts,
                         cudaStream_t stream) {
  if (n * block <= 0) return;
  count_launch(1);
  launch_pdl(rows::anchor_slots_kernel, (n * block + 255) / 256, 256, 0, stream, anchors, picked, ids, positions, mask, T, n, block, mask_token, from_anchor, token,
             position, index, target, counts);
}

void launch_document_interval(const int64_t* doc, int T, int window, int* lo, int* hi, cudaStream_t stream) {
  if (T <= 0) return;
  count_launch(1);
  launch_pdl(rows::document_interval_kernel, 1, rows::kT, 0, stream, doc, T, window, lo, hi);
}
void launch_compact(const bool* valid, int T, int64_t* list, int* count, cudaStream_t stream) {
  count_launch(1);
  launch_pdl(rows::compact_kernel, 1, rows::kT, 0, stream, valid, T, list, count);
}
void launch_cod_step(const int64_t* pool, const int64_t* perm, int take, const bool* valid, int T, int depth, int filter_zero, unsigned char* flags,
                     int64_t* picked, int64_t* anchor, int64_t* depths, int64_t* next, int* count, cudaStream_t stream) {
  count_launch(1);
  launch_pdl(rows::cod_step_kernel, 1, rows::kT, 0, stream, pool, perm, take, valid, T, depth, filter_zero, flags, picked, anchor, depths, next, count);
}
void launch_peagle_spec(const int64_t* anchor, const int64_t* depth, const bool* row_valid, const int64_t* doc, const int* doc_lo, int n, int T, int num_depths,
                        int window, int* table, int* lo, int* hi, int* extra, cudaStream_t stream) {
  if (n <= 0) return;
  const int grid = (n + 255) / 256;
  if (extra != nullptr) {
    count_launch(1);
    launch_pdl(rows::peagle_table_kernel, grid, 256, 0, stream, anchor, depth, row_valid, n, T, num_depths, table);
  }
  count_launch(1);
  launch_pdl(rows::peagle_spec_kernel, grid, 256, 0, stream, anchor, depth, row_valid, doc, doc_lo, n, T, num_depths, window, (const int*)table, lo, hi, extra);
}
// target_row == nullptr: no list of the verifier's rows (needed where N > T)
void launch_step_rows(const uint8_t* mask, const int64_t* ids, const int64_t* positions, const int* const* interval, int T, int N, int S, int64_t* index,
                      int* inverse, int* count, int64_t* ids_out, int64_t* positions_out, uint8_t* mask_out, uint8_t* prev_out, int* target_row,
                      int* const* interval_out, int* extra, cudaStream_t stream) {
  if (T <= 0) return;
  count_launch(2);
  launch_pdl(rows::wanted_rows_kernel, target_row != nullptr ? 2 : 1, rows::kT, 0, stream, mask, T, N, S, index, inverse, count);
  const rows::StepRows p{mask, ids, positions, {interval[0], interval[1]}, index, inverse, count, T, N, S, ids_out, positions_out, mask_out, prev_out,
                         target_row, {interval_out[0], interval_out[1]}, extra};
  launch_pdl(rows::step_rows_kernel, (T + 255) / 256, 256, 0, stream, p);
}
static rows::RowCopies row_copies(int n, const void* const* from, const int64_t* stride, const int* W, void* const* to, int rows, dim3* grid) {
  rows::RowCopies p{};
  int64_t most = 0;
  for (int i = 0; i < n; ++i) {
    p.from[i] = (const __nv_bfloat16*)from[i];
    p.stride[i] = stride[i];
    p.to[i] = (__nv_bfloat16*)to[i];
    p.W[i] = W[i];
    const int64_t blocks = ((int64_t)rows * (W[i] >> 3) + 255) / 256;
    most = blocks > most ? blocks : most;
  }
  p.rows = rows;
  *grid = dim3((unsigned)(most < 16 * kNumSM ? (most > 0 ? most : 1) : 16 * kNumSM), n);
  return p;
}
// n: 1 or 2 matrices of the same rows
void launch_take_rows(int n, const void* const* x, const int64_t* stride, const int* W, void* const* out, const int64_t* index, const int* live, int rows,
                      cudaStream_t stream) {
  if (rows <= 0) return;
  dim3 grid;
  const rows::RowCopies p = row_copies(n, x, stride, W, out, rows, &grid);
  count_launch(1);
  launch_pdl(rows::take_rows_kernel, grid, 256, 0, stream, p, index, live);
}
void launch_put_rows(int n, const void* const* d, const int64_t* stride, const int* W, void* const* out, const int* inverse, int rows, cudaStream_t stream) {
  if (rows <= 0) return;
  dim3 grid;
  const rows::RowCopies p = row_copies(n, d, stride, W, out, rows, &grid);
  count_launch(1);
  launch_pdl(rows::put_rows_kernel, grid, 256, 0, stream, p, inverse);
}
int embedding_bwd_partial_rows(int n) { return n > rows::kSlice ? ((n - 1) / rows::kSlice + 1) * 2 : 0; }
void launch_embedding_bwd(const int64_t* ids, const int64_t* order, const void* d, int64_t d_stride, int n, int H, int64_t vocab, int64_t padding, void* dw,
                          int accumulate, float* part, cudaStream_t stream) {
  if (n <= 0) return;
  const int slices = (n - 1) / rows::kSlice + 1;
  count_launch(slices > 1 ? 2 : 1);
  launch_pdl(rows::embedding_bwd_kernel, n, 256, 0, stream, ids, order, (const __nv_bfloat16*)d, d_stride, n, H, vocab, padding, (__nv_bfloat16*)dw, accumulate,
             part);
  if (slices > 1)
    launch_pdl(rows::embedding_join_kernel, dim3((slices - 1 + rows::kJoinSlices - 1) / rows::kJoinSlices, (H + 127) / 128), 256, 0, stream, ids,
               (const float*)part, n, H, vocab, padding, (__nv_bfloat16*)dw, accumulate);
}

}  // namespace sb200
