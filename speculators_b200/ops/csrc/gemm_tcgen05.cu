// bf16 GEMM on the 5th-generation tensor cores:  C[M,N] = A[M,K] * B[N,K]^T  (+ epilogue)
//
// This is the nn.Linear forward shape: both operands are K-major (row-major with K
// contiguous), the accumulator is fp32.  Roles of a CTA's warps:
//
//   warp 0  TMA producer : cp.async.bulk.tensor (128B-swizzled boxes, no multicast) into a
//                          shared-memory ring, completion counted on mbarriers
//   warp 1  MMA issuer   : allocates TMEM (two 256-column fp32 accumulators in the persistent
//                          kernel), one elected thread issues tcgen05.mma from
//                          shared-memory descriptors and tcgen05.commit's to free ring slots
//   warps 2.. epilogue   : tcgen05.ld the finished accumulator (each warp its own 32 TMEM
//                          lanes = 32 output rows), convert to bf16, apply the epilogue and
//                          store; the MMA warp meanwhile fills the other accumulator
//
// Tiles are walked n-major so that CTAs running at the same time share B (weight) tiles in
// L2.  Ragged M / N / K are handled by TMA zero fill and masked stores.
//
// Three kernels share this structure.  gemm_tn_2cta_kernel (large products) pairs two SMs (a cluster
// of two CTAs, tcgen05 cta_group::2) on a 256x256 tile, persistent over tiles: each CTA stages its own 128
// rows of A and 128 of the tile's 256 rows of B, the even CTA's elected thread issues M=256 MMAs that read
// both CTAs' shared memory and write both CTAs' TMEM, and completion is multicast to the barriers of both
// CTAs.  Halving the B traffic per SM is what the L2-to-SM path needs to keep the tensor pipe fed.
// gemm_split_kernel runs the same tile on a cluster of two or four pairs that divide the contraction (few
// tiles, long contraction), gemm_small_kernel one 128x64 tile per CTA (few tiles, short contraction).
//
// Operand layouts.  The forward product has both operands K-major (rows of A and of B run
// along the contraction).  The backward products of a linear layer do not:
//   dgrad  dX[T,in]  = dY[T,out] * W[out,in]        B is read as stored, [K, N] with N contiguous
//   wgrad  dW[out,in] (+)= dY[T,out]^T * X[T,in]    A is [K, M] with M contiguous, B is [K, N]
// The kernels therefore take each operand either K-major or MN-major (template flags):
// an MN-major operand is staged by TMA as boxes of 64 MN-elements x 128 contraction rows (the
// same 16 KB, 128-byte swizzle) and described to the tensor core with an MN-major shared-memory
// descriptor plus the transpose bit of the instruction descriptor, so no operand is ever
// transposed in memory.
//
// Every wait is bounded: a thread that exhausts its poll budget records a code in the
// caller's status word and leaves its loop; the other roles then run out of budget (or
// see the status word) too, the CTA meets at the final barrier, frees its TMEM and
// returns.  Nothing traps and nothing spins forever.
#include <atomic>

#include "gemm_split.h"
#include "loss_stats.cuh"
#include "remember.h"
#include "tcgen05_utils.cuh"

namespace sb200 {

namespace tc {

constexpr int BM = 128, BN = 256, BK = 64;
constexpr int TMEM_COLS = 512;

// kSwiGLU: the weight is the stack [gate rows | up rows] of a gated MLP (N = 2 I).  A tile pairs 128 gate columns
// with the same 128 up columns (the leader CTA loads the gate rows, its peer the up rows, so the accumulator holds
// gate in columns 0..127 and up in 128..255); the epilogue stores both halves into C[M, 2 I] (kept for the backward
// pass) and silu(gate) * up into h[M, I].
enum Epilogue : int { kStore = 0, kAccumulate = 1, kAddResidual = 2, kSwiGLU = 3 };
enum Status : int { kOk = kStatusOk, kTimeoutProducer = 1, kTimeoutMma = 2, kTimeoutEpilogue = 3, kTimeoutPartial = 4 };

// Row statistics in the epilogue (the lm_head product fused with the row loss): next to
// storing the logits tile, every thread reduces its row's 256 columns of the tile, together with
// the same columns of the target logits row `row + shift`, to the online-softmax statistics of
// both and the cross term of the KL divergence, and writes them as one record of kStatWords
// floats at partial[(row * tiles_n + tile_n) * kStatWords].  A second kernel merges a row's
// records.  The statistics are taken from the bf16-rounded logits, i.e. from the values the
// backward pass reads back.
constexpr int kStatWords = 12;  // m_d z_d best_d idx_d | m_t z_t A best_t | idx_t - - -   (one record per row and 128-column half tile)
struct RowStatsOut {
  const __nv_bfloat16* targets;  // nullptr: plain GEMM
  int64_t ldt;
  int t_rows;   // rows of the target matrix
  int shift;    // logits row r pairs with target row r + shift
  float* partial;
};

// Grouped products (mixture-of-experts): rows sorted by expert, expert e owning the rows
// seg[e] .. seg[e+1] of the activation matrices, every seg[e] a multiple of 128 (the rows
// between an expert's last token and the next boundary are zero).  All sizes that depend on the
// routing are read from device memory, so the launch is fixed-shape and can be captured.
//   kGroupRows  C[r, :] = A[r, :] . B_e^T for r in expert e (forward and input gradient): tiles are
//               enumerated per expert through tile_start (prefix sum of ceil(rows_e / 256) * tiles_n);
//               B is the stack of the experts' matrices ([E * N, K] K-major or [E * K, N] MN-major).
//   kGroupK     C_e (+)= A[seg_e, :]^T . B[seg_e, :] (weight gradient): the contraction runs over
//               expert e's rows, C is the stack [E * M, N]; an expert without rows yields zeros.
enum GroupMode : int { kGroupNone = 0, kGroupRows = 1, kGroupK = 2 };
struct Grouping {
  int mode;
  int num_groups;
  const int* seg;         // [num_groups + 1] padded row offsets
  const int* tile_start;  // [num_groups + 1] prefix sum of ceil(rows_e / 256) (kGroupRows); tiles of expert e: that x tiles_n
};

// Row-parallel product of a tensor-parallel layer: the ranks hold slices of the contraction, so
// every rank's product is a partial sum of the whole [M, N] output.  Rank `owner = column /
// cols` reduces the columns owner * cols .. + cols - 1; instead of storing its partial tile at home
// and handing the buffer to a collective, the epilogue stores each tile straight into the owner's
// staging area over NVLink (plain stores to peer-mapped memory, issued while the tensor core works
// on the next tile): stage of rank o = [world][M][cols], slot `rank` written by this rank.
// cols is a multiple of 256, so a tile has one owner.
constexpr int kMaxScatterRanks = 8;
struct Scatter {
  int world;  // 0: off
  int rank;
  int cols;   // N / world
  __nv_bfloat16* stage[kMaxScatterRanks];
};

struct Params {
  __nv_bfloat16* c;
  const __nv_bfloat16* residual;
  int M, N, K;
  int64_t ldc, ldr;
  int epilogue;
  int* status;
  RowStatsOut rs;
  Grouping grp;
  Scatter sc;
  __nv_bfloat16* h;  // kSwiGLU: [M, N / 2] output, row stride ldh
  int64_t ldh;
  int staged;        // 1: C (and h) leave through shared memory and TMA stores (map_c, map_h)
  // result = alpha * product (+ beta * addend), rounded where separate element-wise passes over bf16 tensors would round:
  // alpha * bf16(product) and beta * addend each to bf16 before the sum; alpha = beta = 1 is the plain epilogue.
  // once: alpha * product + beta * addend + diagonal on its diagonal, in fp32 and rounded once
  float alpha, beta, diagonal;
  int once;
  // a stack of `batch` products: the z-th of each operand's stack, elements apart
  int batch;
  int64_t c_batch, r_batch;
  int symmetric;  // the product is symmetric: tiles above the diagonal are computed and stored twice (map_h: transposed stores)
  // Device-side row count of the activations (live_rows).  It bounds M, and where both operands are MN-major (a weight
  // gradient, which sums over the rows) K.  A multiple of 256 or all rows: no tile and no contraction step straddles it.
  const int* live;
  // Tiles divided between pairs (SplitPlan): partial sums [round][pair][CTA][epilogue warp][1024] float4 and, zero at launch, one
  // flag per (round, pair, CTA, epilogue warp) behind a start counter.  nullptr: none are.
  float4* partial;
  int* sync;
};

// ---- a part-filled last wave, its tiles divided -------------------------------------------------------------------
// 74 pairs walk the tiles in whole waves, and the last one is usually part-filled: 80 tiles take as long as 148.  What is left
// over after the whole waves is divided instead (us before and after: 1280 x 4096 x 4096 43.9 and 34.7, 1280 x 4096 x 14336
// 141 and 104, 1280 x 4096 x 151936 1572 and 1041, 2560 x 4096 x 14336 229 and 196, 1777 x 6144 x 4096 67 and 63): `parts` pairs take a tile, each an equal part of its contraction, in one or
// two rounds (left[0], then left[1] tiles).  All parts but the last leave their sums in fp32 in global memory (256 KB a pair, which
// stay in L2) and raise a flag per epilogue warp; the counterparts in the pair with the last part add them to their
// accumulator, in the order of the contraction, before the epilogue.  The same bits on every run.
//   The pairs of one part walk neighbouring tiles in step, as in a whole wave, and so share operand panels in L2.  Dividing
// all steps evenly (each pair a contiguous range of the tiles' contraction steps) balances better and loses that: 1024 x
// 8192 x 28672 took 465 us so, 321 undivided - every panel came from memory once per tile.
//   The rounds come first.  A pair waits for pairs with a lower number only, and numbers go by the order in which pairs start
// (a counter): whoever is waited for is running already, and waits for nobody who is not.
constexpr int kMostParts = 8;
constexpr int kSplitSync = 1 + 2 * 74 * 16;  // ints of `sync`: the counter, then flags of (round, pair, CTA, epilogue warp)
struct SplitPlan {
  int whole;    // tiles in whole waves; the rest are divided
  int left[2];  // tiles of the two rounds
  int parts[2];
  int steps;    // contraction steps of a pair on its way through (the longest part of each round)
  float us;     // predicted, above a launch's fixed part
};
// Round i of `left` tiles in `parts` parts: 0.56 us a step, and for writing, waiting for and adding sums 2.5 us and 1.2 a part.
// Without whole waves behind them the rounds have nothing to hide that behind (256 x 4096 x 14336: 46.6 us where this says 31).
constexpr float kStepUs = 0.56f, kRoundUs = 2.5f, kPartUs = 1.2f, kSplitGainUs = 2.f, kAloneUs = 20.f;
__host__ __device__ inline SplitPlan split_plan(int tiles, int kb, int pairs) {
  const int waves = tiles / pairs, rest = tiles - waves * pairs;
  SplitPlan s{tiles, {0, 0}, {1, 1}, kb * (waves + (rest > 0)), 0.f};
  s.us = kStepUs * s.steps;
  if (rest == 0) return s;
  auto consider = [&](int n0, int c0, int n1, int c1) {
    if (c0 < 2 || kb < 2 * c0 || n0 * c0 > pairs || (n1 > 0 && (c1 < 2 || kb < 2 * c1 || n1 * c1 > pairs))) return;
    const int steps = kb * waves + (kb + c0 - 1) / c0 + (n1 > 0 ? (kb + c1 - 1) / c1 : 0);
    const float us = kStepUs * steps + kRoundUs + kPartUs * c0 + (n1 > 0 ? kRoundUs + kPartUs * c1 : 0.f);
    if (us + (waves > 0 ? kSplitGainUs : kAloneUs) < kStepUs * kb * (waves + 1) && (s.left[0] == 0 || us < s.us)) s = SplitPlan{waves * pairs, {n0, n1}, {c0, n1 > 0 ? c1 : 1}, steps, us};
  };
  const int fit = pairs / rest;
  for (int c = 2; c <= kMostParts; ++c) {
    if (c <= fit) consider(rest, c, 0, 0);
    const int half = pairs / 2, behind = rest - half;  // two parts for as many tiles as that takes, then the others
    if (behind > 0 && c <= pairs / behind) consider(half, 2, behind, c);
  }
  return s;
}

// The pieces of tiles that one pair works on, in order: its parts of divided tiles, then whole tiles.
template <bool DIVIDE>
struct Pieces {  // whole tiles only
  int tile;
  static constexpr int k0 = 0, steps = 0, round = -1, part = 0;
  int next;
  __device__ __forceinline__ explicit Pieces(int number) : next(number) {}
  __device__ __forceinline__ bool advance(const SplitPlan& s, int, int, int pairs) {
    tile = next;
    next += pairs;
    return tile < s.whole;
  }
};
template <>
struct Pieces<true> {
  int tile, k0, steps;  // this piece: contraction steps k0 .. k0 + steps of the tile
  int round, part;      // of a divided tile; round -1: a whole one
  int at, next;
  __device__ __forceinline__ explicit Pieces(int number) : round(-1), part(0), at(0), next(number) {}
  __device__ __forceinline__ bool advance(const SplitPlan& s, int kb, int number, int pairs) {
    while (at < 2) {
      const int i = at++, n = i == 0 ? s.left[0] : s.left[1], c = i == 0 ? s.parts[0] : s.parts[1];
      if (number >= n * c) continue;
      round = i;
      part = number / n;
      tile = s.whole + (i == 0 ? 0 : s.left[0]) + number - part * n;
      k0 = part * kb / c;
      steps = (part + 1) * kb / c - k0;
      return true;
    }
    round = -1;
    if (next >= s.whole) return false;
    tile = next;
    k0 = 0;
    steps = kb;
    next += pairs;
    return true;
  }
};

// A warp's 32 rows x 128 columns of the accumulator, four columns at a time, lanes (rows) side by side.
__device__ __forceinline__ void split_put(float4* to, uint32_t tmem, int lane) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t r[32];
    tmem_ld32(tmem + c * 32, r);
    tmem_ld_wait();
#pragma unroll
    for (int v = 0; v < 8; ++v)
      __stcg(to + (c * 8 + v) * 32 + lane, make_float4(__uint_as_float(r[v * 4]), __uint_as_float(r[v * 4 + 1]), __uint_as_float(r[v * 4 + 2]), __uint_as_float(r[v * 4 + 3])));
  }
}
__device__ __forceinline__ void split_add(const float4* from, uint32_t tmem, int lane) {
#pragma unroll 1
  for (int c = 0; c < 4; ++c) {
    uint32_t r[32];
    float4 o[8];
#pragma unroll
    for (int v = 0; v < 8; ++v) o[v] = __ldcg(from + (c * 8 + v) * 32 + lane);
    tmem_ld32(tmem + c * 32, r);
    tmem_ld_wait();
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      const float add[4] = {o[v].x, o[v].y, o[v].z, o[v].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) r[v * 4 + j] = __float_as_uint(__uint_as_float(r[v * 4 + j]) + add[j]);
    }
    tmem_st32(tmem + c * 32, r);
  }
  tmem_st_wait();
}
// One lane's bounded wait for a flag; false = gave up (status word set) or another role already failed.
__device__ __forceinline__ bool flag_wait(const int* flag, int* status, int code) {
  for (uint32_t i = 0; i < POLL_LIMIT; ++i) {
    int up;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(up) : "l"(flag) : "memory");
    if (up != 0) return true;
    if ((i & 0xfff) == 0xfff && *reinterpret_cast<volatile int*>(status) != kStatusOk) return false;
  }
  atomicCAS(status, kStatusOk, code);
  return false;
}

// both rounded to bf16
__device__ __forceinline__ void bf16_round2(float& a, float& b) {
  const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
  const uint32_t w = *reinterpret_cast<const uint32_t*>(&t);
  a = __uint_as_float(w << 16);
  b = __uint_as_float(w & 0xffff0000u);
}
struct Scaling {
  float alpha, beta, diagonal;
  int once;
  bool plain;
  __device__ __forceinline__ explicit Scaling(const Params& p)
      : alpha(p.alpha), beta(p.beta), diagonal(p.diagonal), once(p.once), plain(!p.once && p.alpha == 1.f && p.beta == 1.f) {}
  // (the plain epilogue skips the arithmetic as a whole behind one uniform test each: with the other forms' tests in between split
  // products took 1 to 2 % more, 2048 x 1024 x 3072 with a residual 22.7 us instead of 22.2)
  template <int N>
  __device__ __forceinline__ void product(float (&f)[N], int row, int col) const {  // N columns from col on
    if (plain) return;
    if (once) {
#pragma unroll
      for (int j = 0; j < N; ++j) f[j] *= alpha;
      if ((unsigned)(row - col) < (unsigned)N) {
#pragma unroll
        for (int j = 0; j < N; ++j) f[j] += row == col + j ? diagonal : 0.f;
      }
    } else if (alpha != 1.f) {
#pragma unroll
      for (int j = 0; j < N; j += 2) {
        float pad = 0.f, &second = j + 1 < N ? f[j + 1 < N ? j + 1 : j] : pad;
        bf16_round2(f[j], second);
        f[j] *= alpha;
        second *= alpha;
        bf16_round2(f[j], second);
      }
    }
  }
  template <int N>
  __device__ __forceinline__ void add(float (&f)[N], const float (&o)[N]) const {
    if (plain) {
#pragma unroll
      for (int j = 0; j < N; ++j) f[j] += o[j];
      return;
    }
    if (once) {
#pragma unroll
      for (int j = 0; j < N; ++j) f[j] = fmaf(beta, o[j], f[j]);
      return;
    }
#pragma unroll
    for (int j = 0; j < N; j += 2) {
      float a = o[j], b = j + 1 < N ? o[j + 1 < N ? j + 1 : j] : 0.f;
      if (beta != 1.f) {
        a *= beta;
        b *= beta;
        bf16_round2(a, b);
      }
      f[j] += a;
      if (j + 1 < N) f[j + 1 < N ? j + 1 : j] += b;
    }
  }
};

// First element of the W-column chunk at (row, n0) of the output.
__device__ __forceinline__ __nv_bfloat16* c_chunk(const Params& p, int row, int n0, int z) {
  if (p.sc.world > 0) {
    const int owner = n0 / p.sc.cols;
    return p.sc.stage[owner] + ((int64_t)p.sc.rank * p.M + row) * p.sc.cols + (n0 - owner * p.sc.cols);
  }
  return p.c + z * p.c_batch + (int64_t)row * p.ldc + n0;
}

// Where one 256x256 tile (or this CTA's half of it) sits in the operands.
struct TileInfo {
  int a_m, a_k0;   // A: first MN index of this CTA's 128, first contraction index
  int b_n, b_k0;   // B: the same
  int num_kb;      // 128-wide contraction steps
  int c_row0;      // C row of this CTA's first accumulator row
  int row_end;     // C rows >= row_end do not exist (for this tile)
  int n0;          // first C column
  int tile_n;      // column-tile index (row statistics)
  int z;           // which product of the stack
  bool mirror;     // symmetric product: the tile's transpose is stored too
};

constexpr int kBandRows = 8;

template <bool B_MN>
__device__ __forceinline__ TileInfo decode_tile(const Params& p, int M, int tile, int tiles_m, int tiles_n, int num_kb, int rank) {
  TileInfo t;
  t.z = 0;
  t.mirror = false;
  if (p.grp.mode == kGroupNone && p.symmetric) {
    const int per = tiles_m * (tiles_m + 1) / 2;
    t.z = tile / per;
    const int local = tile - t.z * per;
    int j = (int)((sqrtf(8.f * local + 1.f) - 1.f) * 0.5f);  // local = j (j + 1) / 2 + i, i <= j
    while (j * (j + 1) / 2 > local) --j;
    while ((j + 1) * (j + 2) / 2 <= local) ++j;
    const int i = local - j * (j + 1) / 2, m0 = i * 256 + rank * 128;
    t.mirror = i != j;
    t.tile_n = j;
    t.n0 = j * 256;
    t.a_m = m0; t.a_k0 = 0; t.b_n = t.n0 + rank * 128; t.b_k0 = 0; t.num_kb = num_kb; t.c_row0 = m0; t.row_end = M;
  } else if (p.grp.mode == kGroupNone) {
    t.z = tile / (tiles_m * tiles_n);
    tile -= t.z * tiles_m * tiles_n;
    // Tiles run down a band of kBandRows tile rows, column after column, then the next band: the
    // CTA pairs working at the same time cover a near-square patch of C (8 x 9 tiles on 74 pairs),
    // so a wave touches about 17 operand panels instead of 75 and a tall output (a weight
    // gradient of a wide layer) no longer re-reads its whole A operand once per tile column.
    const int band = tile / (kBandRows * tiles_n), first = band * kBandRows;
    const int rows = min(kBandRows, tiles_m - first), local = tile - band * kBandRows * tiles_n;
    const int m0 = (first + local % rows) * 256 + rank * 128;
    t.tile_n = local / rows;
    t.n0 = t.tile_n * 256;
    t.a_m = m0; t.a_k0 = 0; t.b_n = t.n0 + rank * 128; t.b_k0 = 0; t.num_kb = num_kb; t.c_row0 = m0; t.row_end = M;
    if (p.epilogue == kSwiGLU) {  // 128 gate rows for the leader, the matching up rows for its peer
      t.n0 = t.tile_n * 128;
      t.b_n = t.n0 + rank * (p.N >> 1);
    }
  } else if (p.grp.mode == kGroupRows) {
    int lo = 0, hi = p.grp.num_groups - 1;  // last e with tile_start[e] <= tile
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (p.grp.tile_start[mid] * tiles_n <= tile) lo = mid; else hi = mid - 1;
    }
    const int e = lo, s0 = p.grp.seg[e], s1 = p.grp.seg[e + 1];
    const int tm = (s1 - s0 + 255) >> 8, local = tile - p.grp.tile_start[e] * tiles_n;
    const int m0 = s0 + (local % tm) * 256 + rank * 128;
    t.tile_n = local / tm;
    t.n0 = t.tile_n * 256;
    t.a_m = m0; t.a_k0 = 0; t.num_kb = num_kb; t.c_row0 = m0; t.row_end = s1;
    t.b_n = (B_MN ? 0 : e * p.N) + t.n0 + rank * 128;
    t.b_k0 = B_MN ? e * p.K : 0;
    if (p.epilogue == kSwiGLU) {
      t.n0 = t.tile_n * 128;
      t.b_n = e * p.N + t.n0 + rank * (p.N >> 1);
    }
  } else {
    const int per = tiles_m * tiles_n, e = tile / per, local = tile % per;
    const int m0 = (local % tiles_m) * 256 + rank * 128, s0 = p.grp.seg[e];
    t.tile_n = local / tiles_m;
    t.n0 = t.tile_n * 256;
    t.a_m = m0; t.a_k0 = s0; t.b_n = t.n0 + rank * 128; t.b_k0 = s0; t.num_kb = (p.grp.seg[e + 1] - s0) >> 7;
    t.c_row0 = e * p.M + m0; t.row_end = e * p.M + p.M;
  }
  return t;
}

// 32-byte store (one full sector) of sixteen bf16; ptr must be 32-byte aligned.
__device__ __forceinline__ void st32(__nv_bfloat16* ptr, const bf16x8& a, const bf16x8& b) {
  const uint4 x = *reinterpret_cast<const uint4*>(&a), y = *reinterpret_cast<const uint4*>(&b);
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"l"(ptr), "r"(x.x), "r"(x.y), "r"(x.z), "r"(x.w), "r"(y.x), "r"(y.y), "r"(y.z), "r"(y.w)
               : "memory");
}

// Epilogue of one thread: TMEM lane `taddr` (its 256 fp32 columns) -> row `row`, columns
// n0 .. n0+255 of C, with the configured epilogue.
template <int W>
__device__ __forceinline__ void store_accumulator(const Params& p, const Scaling& sc, uint32_t taddr, int row, int n0, int z, int row_end, bool zero) {
  __nv_bfloat16* crow = c_chunk(p, row, n0, z);
  const __nv_bfloat16* rrow = p.residual ? p.residual + z * p.r_batch + (int64_t)row * p.ldr + n0 : nullptr;
  const bool vec_ok = ((p.ldc & 7) == 0) && ((reinterpret_cast<uintptr_t>(p.c) & 15) == 0) &&
                      (p.epilogue != kAddResidual || (((p.ldr & 7) == 0) && ((reinterpret_cast<uintptr_t>(p.residual) & 15) == 0)));
  const bool wide_ok = vec_ok && ((p.ldc & 15) == 0) && ((reinterpret_cast<uintptr_t>(p.c) & 31) == 0);
#pragma unroll 1
  for (int c = 0; c < W / 32; ++c) {
    uint32_t r[32];
    tmem_ld32(taddr + c * 32, r);
    tmem_ld_wait();
    if (zero) {  // no contraction step ran (an expert without rows): the accumulator holds nothing
#pragma unroll
      for (int j = 0; j < 32; ++j) r[j] = 0u;
    }
    if (row < row_end) {
      const int col0 = n0 + c * 32;
      if (vec_ok && col0 + 32 <= p.N) {
        bf16x8 packed[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          float f[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(r[v * 8 + j]);
          sc.product(f, row, col0 + v * 8);
          if (p.epilogue == kAccumulate) {
            float o[8];
            unpack8(ld8(crow + c * 32 + v * 8), o);
            sc.add(f, o);
          } else if (p.epilogue == kAddResidual) {
            float o[8];
            unpack8(ld8(rrow + c * 32 + v * 8), o);
            sc.add(f, o);
          }
          packed[v] = pack8(f);
        }
        if (wide_ok) {  // full 32-byte sectors per store
          st32(crow + c * 32, packed[0], packed[1]);
          st32(crow + c * 32 + 16, packed[2], packed[3]);
        } else {
#pragma unroll
          for (int v = 0; v < 4; ++v) st8(crow + c * 32 + v * 8, packed[v]);
        }
      } else {
        for (int j = 0; j < 32; ++j) {
          if (col0 + j < p.N) {
            float f[1] = {__uint_as_float(r[j])};
            sc.product(f, row, col0 + j);
            if (p.epilogue != kStore) {
              const float o[1] = {__bfloat162float((p.epilogue == kAccumulate ? crow : rrow)[c * 32 + j])};
              sc.add(f, o);
            }
            crow[c * 32 + j] = __float2bfloat16(f[0]);
          }
        }
      }
    }
  }
}

// ---- gated MLP: gate | up product with silu(gate) * up formed in the epilogue -------------------
// One thread = one row, one warp = 32 rows through its staging area; `tlane` = TMEM address of its lane at the first of the 64 gate columns it handles
// (the matching up columns sit 128 columns further), col0 = their column in [0, I).  The activation is
// taken from the bf16-rounded gate and up (what the backward pass reads back), in the element-wise
// kernel's order: silu(gate) rounded to bf16, times up.  Needs I % 128 == 0 and staged stores (checked on the host).
__device__ __forceinline__ void store_accumulator_swiglu(const Params& p, const CUtensorMap* map_c, const CUtensorMap* map_h, uint32_t stage, uint32_t tlane,
                                                         int row0, int col0, bool live, int lane) {
  const int I = p.N >> 1;
  stage_wait();
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    uint32_t g[32];
    tmem_ld32(tlane + c * 32, g);
    tmem_ld_wait();
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      float f[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(g[v * 8 + j]);
      stage_put8(stage, lane, c * 4 + v, pack8(f));
    }
  }
  stage_store(stage, map_c, col0, row0, 0, live);
  uint4 row[8];  // the lane's gate values, then its activated ones
#pragma unroll
  for (int v = 0; v < 8; ++v) row[v] = stage_get8(stage, lane, v);
  stage_wait();
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    uint32_t u[32];
    tmem_ld32(tlane + 128 + c * 32, u);
    tmem_ld_wait();
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      float gf[8], uf[8], o[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) uf[j] = __uint_as_float(u[v * 8 + j]);
      const bf16x8 up = pack8(uf);
      stage_put8(stage, lane, c * 4 + v, up);
      unpack8(up, uf);
      unpack8(*reinterpret_cast<const bf16x8*>(&row[c * 4 + v]), gf);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float sg = 1.f / (1.f + __expf(-gf[j]));
        o[j] = __bfloat162float(__float2bfloat16(gf[j] * sg)) * uf[j];
      }
      const bf16x8 act = pack8(o);
      row[c * 4 + v] = *reinterpret_cast<const uint4*>(&act);
    }
  }
  stage_store(stage, map_c, I + col0, row0, 0, live);
  stage_wait();
#pragma unroll
  for (int v = 0; v < 8; ++v) stage_put8(stage, lane, v, *reinterpret_cast<const bf16x8*>(&row[v]));
  stage_store(stage, map_h, col0, row0, 0, live);
}

// ---- epilogues that read memory (C += result, result + residual) ---------------------------
// The addend row (256 bf16 = 512 bytes per thread) is fetched into registers *before* the
// thread waits for the accumulator, so the loads' latency is spent while the tensor core still
// works on the tile.  With a short contraction (weight gradients: K = tokens of one step) the
// time per tile is otherwise set by eight dependent load round trips per thread.
template <int W>
struct RowPrefetch {
  uint4 v[W / 8];
  bool tile_ok;  // the same for every thread of the warp: selects the epilogue (its tcgen05.ld is warp-collective)
  bool valid;    // this thread's row exists (its loads were issued, its stores may be)
};

template <int W>
__device__ __forceinline__ bool tile_reads_vectorised(const Params& p, int n0) {
  if (p.epilogue == kStore || n0 + W > p.N || (p.ldc & 7) || (reinterpret_cast<uintptr_t>(p.c) & 15)) return false;
  if (p.epilogue == kAddResidual && ((p.ldr & 7) || (reinterpret_cast<uintptr_t>(p.residual) & 15))) return false;
  return true;
}

// Staged stores take every tile (N is a multiple of 8 then): a chunk past the edge reads as zeros.  The addend of a warp's 32
// rows comes in whole 128-byte lines, four rows of 64 columns a load (v[h * 8 + j]: row j * 4 + lane / 8, columns h * 64 +
// 8 * (lane % 8)), and meets its row in the staging area.  Loaded with a row per lane, 16 bytes each, every load touched 32
// lines and the addend's loads set the pace of a tile (us a wave of pair tiles, 4096 x 9472, at contractions of 128 and 1024: residual 8.7 and 9.9,
// now 5.4 and 8.3; accumulate 8.6 and 10.2, now 4.7 and 8.1; scaled by alpha and beta 10.8 and 11.0, now 6.5 and 8.8).
template <int W>
__device__ __forceinline__ void prefetch_addend_staged(const Params& p, int row0, int n0, int z, int row_end, int lane, int h, RowPrefetch<W>& pre) {
  const int row = row0 + (lane >> 3), col = n0 + h * 64 + (lane & 7) * 8;
  const int64_t ld = p.epilogue == kAccumulate ? p.ldc : p.ldr;
  const __nv_bfloat16* src = (p.epilogue == kAccumulate ? p.c + z * p.c_batch : p.residual + z * p.r_batch) + (int64_t)row * ld + col;
  if (row0 + 32 <= row_end && n0 + h * 64 + 64 <= p.N) {
#pragma unroll
    for (int j = 0; j < 8; ++j) pre.v[h * 8 + j] = __ldg(reinterpret_cast<const uint4*>(src + j * 4 * ld));
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j)
      pre.v[h * 8 + j] = row + j * 4 < row_end && col < p.N ? __ldg(reinterpret_cast<const uint4*>(src + j * 4 * ld)) : make_uint4(0u, 0u, 0u, 0u);
  }
}
template <int W>
__device__ __forceinline__ void prefetch_addend_staged(const Params& p, int row0, int n0, int z, int row_end, int lane, RowPrefetch<W>& pre) {
  pre.tile_ok = pre.valid = true;
  if (p.epilogue == kStore) return;
#pragma unroll
  for (int h = 0; h < W / 64; ++h) prefetch_addend_staged<W>(p, row0, n0, z, row_end, lane, h, pre);
}

template <int W>
__device__ __forceinline__ void prefetch_addend(const Params& p, int row, int n0, int z, int row_end, RowPrefetch<W>& pre) {
  pre.tile_ok = tile_reads_vectorised<W>(p, n0);
  pre.valid = pre.tile_ok && row < row_end;
  if (pre.valid) {
    const __nv_bfloat16* src = p.epilogue == kAccumulate ? p.c + z * p.c_batch + (int64_t)row * p.ldc + n0 : p.residual + z * p.r_batch + (int64_t)row * p.ldr + n0;
#pragma unroll
    for (int i = 0; i < W / 8; ++i) pre.v[i] = __ldg(reinterpret_cast<const uint4*>(src) + i);
  }
}

// Same result as store_accumulator for a tile whose addend rows are already in registers.  Called
// by whole warps (pre.tile_ok); a thread whose row does not exist takes part in the tensor-memory
// loads and stores nothing.
template <int W>
__device__ __forceinline__ void store_accumulator_prefetched(const Params& p, const Scaling& sc, uint32_t taddr, int row, int n0, int z, const RowPrefetch<W>& pre,
                                                             bool zero) {
  __nv_bfloat16* crow = p.c + z * p.c_batch + (int64_t)row * p.ldc + n0;
  const bool wide_ok = ((p.ldc & 15) == 0) && ((reinterpret_cast<uintptr_t>(p.c) & 31) == 0);
#pragma unroll
  for (int c = 0; c < W / 32; ++c) {
    uint32_t r[32];
    tmem_ld32(taddr + c * 32, r);
    tmem_ld_wait();
    bf16x8 packed[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      float f[8], o[8];
      unpack8(*reinterpret_cast<const bf16x8*>(&pre.v[c * 4 + v]), o);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = zero ? 0.f : __uint_as_float(r[v * 8 + j]);
      sc.product(f, row, n0 + c * 32 + v * 8);
      sc.add(f, o);
      packed[v] = pack8(f);
    }
    if (!pre.valid) continue;
    if (wide_ok) {
      st32(crow + c * 32, packed[0], packed[1]);
      st32(crow + c * 32 + 16, packed[2], packed[3]);
    } else {
#pragma unroll
      for (int v = 0; v < 4; ++v) st8(crow + c * 32 + v * 8, packed[v]);
    }
  }
}

// Four finished fp32 values -> row `row`, columns col0 .. col0 + 3 of C with the configured epilogue.
__device__ __forceinline__ void store_vec4(const Params& p, const Scaling& sc, const float4& t, int row, int col0, int z) {
  __nv_bfloat16* out = p.c + z * p.c_batch + (int64_t)row * p.ldc + col0;
  const __nv_bfloat16* add = p.epilogue == kAccumulate ? out : p.residual + z * p.r_batch + (int64_t)row * p.ldr + col0;
  float f[4] = {t.x, t.y, t.z, t.w}, o[4];
  sc.product(f, row, col0);
  const bool full = col0 + 4 <= p.N && (p.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(p.c) & 7) == 0;
  if (p.epilogue != kStore) {
    for (int j = 0; j < 4; ++j) o[j] = col0 + j < p.N ? __bfloat162float(add[j]) : 0.f;
    sc.add(f, o);
  }
  if (full) {
    __nv_bfloat162 lo = __floats2bfloat162_rn(f[0], f[1]), hi = __floats2bfloat162_rn(f[2], f[3]);
    *reinterpret_cast<uint2*>(out) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
  } else {
    for (int j = 0; j < 4; ++j)
      if (col0 + j < p.N) out[j] = __float2bfloat16(f[j]);
  }
}

// One warp's 32 rows x W columns through its 4 KB staging area, 64 columns at a time.  `row0`: C row of lane 0;
// `live`: the rows exist.  ADD: the epilogue reads, its addend is in `pre` (prefetch_addend_staged) and `ahead(h)` is called
// where the registers of the 64 columns h are free for the next tile's.  Instances of their own for what an epilogue does not
// do: with the tests in between a plain tile took 4.0 us where it takes 2.2 (contraction of 128; from 768 on the products are longer).
template <int W, bool ADD, bool SCALED, typename Ahead>
__device__ __forceinline__ void store_accumulator_staged_as(const Scaling& sc, const CUtensorMap* map_c, const CUtensorMap* map_t, uint32_t stage, uint32_t taddr,
                                                            int row0, int n0, int N, int z, RowPrefetch<W>& pre, bool live, bool mirror, bool zero, int lane,
                                                            const Ahead& ahead) {
#pragma unroll
  for (int h = 0; h < W / 64; ++h) {
    stage_wait();
    if (ADD) {
#pragma unroll
      for (int j = 0; j < 8; ++j) stage_put8(stage, j * 4 + (lane >> 3), lane & 7, *reinterpret_cast<const bf16x8*>(&pre.v[h * 8 + j]));
      __syncwarp();
      ahead(h);
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      uint32_t r[32];
      uint4 own[4];
      tmem_ld32(taddr + (h * 2 + q) * 32, r);
      if (ADD) {
#pragma unroll
        for (int v = 0; v < 4; ++v) own[v] = stage_get8(stage, lane, q * 4 + v);
      }
      tmem_ld_wait();
      if (zero) {
#pragma unroll
        for (int j = 0; j < 32; ++j) r[j] = 0u;
      }
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        float f[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(r[v * 8 + j]);
        if (SCALED) sc.product(f, row0 + lane, n0 + h * 64 + q * 32 + v * 8);
        if (ADD) {
          float o[8];
          unpack8(*reinterpret_cast<const bf16x8*>(&own[v]), o);
          if (SCALED) {
            sc.add(f, o);
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) f[j] += o[j];
          }
        }
        stage_put8(stage, lane, q * 4 + v, pack8(f));
      }
    }
    const bool inside = live && n0 + h * 64 < N;
    stage_store(stage, map_c, n0 + h * 64, row0, z, inside);
    if (mirror) {  // 64 rows (this half's columns) of 32 elements (the warp's rows); the lanes of a store are neighbours
      stage_wait();
      uint4 own[8];
#pragma unroll
      for (int v = 0; v < 8; ++v) own[v] = stage_get8(stage, lane, v);
      __syncwarp();
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        const uint32_t w[4] = {own[v].x, own[v].y, own[v].z, own[v].w};
#pragma unroll
        for (int j = 0; j < 8; ++j)
          asm volatile("st.shared.b16 [%0], %1;" ::"r"(stage + (v * 8 + j) * 64 + lane * 2), "h"((uint16_t)(w[j >> 1] >> (16 * (j & 1)))) : "memory");
      }
      stage_store(stage, map_t, row0, n0 + h * 64, z, inside);
    }
  }
}
struct NothingAhead {
  __device__ __forceinline__ void operator()(int) const {}
};
template <int W, typename Ahead = NothingAhead>
__device__ __forceinline__ void store_accumulator_staged(const Params& p, const Scaling& sc, const CUtensorMap* map_c, const CUtensorMap* map_t, uint32_t stage,
                                                         uint32_t taddr, int row0, int n0, int z, RowPrefetch<W>& pre, bool live, bool mirror, bool zero,
                                                         int lane, const Ahead& ahead = Ahead()) {
  const bool scaled = !sc.plain;
  if (p.epilogue == kStore && !scaled) store_accumulator_staged_as<W, false, false>(sc, map_c, map_t, stage, taddr, row0, n0, p.N, z, pre, live, mirror, zero, lane, ahead);
  else if (p.epilogue == kStore) store_accumulator_staged_as<W, false, true>(sc, map_c, map_t, stage, taddr, row0, n0, p.N, z, pre, live, mirror, zero, lane, ahead);
  else if (!scaled) store_accumulator_staged_as<W, true, false>(sc, map_c, map_t, stage, taddr, row0, n0, p.N, z, pre, live, mirror, zero, lane, ahead);
  else store_accumulator_staged_as<W, true, true>(sc, map_c, map_t, stage, taddr, row0, n0, p.N, z, pre, live, mirror, zero, lane, ahead);
}

// ---- logits tile + row statistics ------------------------------------------------------------
template <int W>
__device__ __forceinline__ void prefetch_targets(const Params& p, int row, int n0, RowPrefetch<W>& pre) {
  const int trow = row + p.rs.shift;
  pre.tile_ok = true;
  pre.valid = row < p.M && trow < p.rs.t_rows;
  const __nv_bfloat16* src = p.rs.targets + (int64_t)trow * p.rs.ldt + n0;
#pragma unroll
  for (int i = 0; i < W / 8; ++i) {
    if (pre.valid && n0 + i * 8 + 8 <= p.N) pre.v[i] = __ldg(reinterpret_cast<const uint4*>(src) + i);
    else pre.v[i] = make_uint4(0u, 0u, 0u, 0u);
  }
}

// Requires N % 8 == 0, ldc % 8 == 0 and 16-byte aligned C / target rows (checked on the host).
template <int W>
__device__ __forceinline__ void store_accumulator_with_stats(const Params& p, uint32_t taddr, int row, int n0, int record, int records_per_row,
                                                             const RowPrefetch<W>& pre) {
  __nv_bfloat16* crow = p.c + (int64_t)row * p.ldc + n0;
  RowStats sd{-INFINITY, 0.f, -INFINITY, 0x7fffffff}, st{-INFINITY, 0.f, -INFINITY, 0x7fffffff};
  float A = 0.f;
#pragma unroll
  for (int c = 0; c < W / 32; ++c) {
    uint32_t r[32];
    tmem_ld32(taddr + c * 32, r);
    tmem_ld_wait();
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int col0 = n0 + c * 32 + v * 8;
      float f[8], x[8], t[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(r[v * 8 + j]);
      const bf16x8 packed = pack8(f);
      if (col0 + 8 <= p.N) {
        unpack8(packed, x);
        unpack8(*reinterpret_cast<const bf16x8*>(&pre.v[c * 4 + v]), t);
        online_update(sd, x, col0);
        online_update_kl(st, A, t, x, col0);
        if (row < p.M) st8(crow + c * 32 + v * 8, packed);
      }
    }
  }
  if (pre.valid) {
    float4* out = reinterpret_cast<float4*>(p.rs.partial + ((int64_t)row * records_per_row + record) * kStatWords);
    out[0] = make_float4(sd.m, sd.z, sd.best, __int_as_float(sd.best_idx));
    out[1] = make_float4(st.m, st.z, A, st.best);
    out[2] = make_float4(__int_as_float(st.best_idx), 0.f, 0.f, 0.f);
  }
}

// ---- 128x64 tiles on single CTAs ---------------------------------------------------------------
// Products that leave most of the chip idle on 256x256 tiles (narrow drafts, short rows, weight gradients of
// small layers).  Such a launch is latency: load, a few dozen MMAs, one epilogue pass.  So a tile is small, the
// ring holds four 128-wide contraction steps (192 KB: a contraction of up to 512 is in flight as a whole), there
// is no persistence and no second accumulator, and where tiles are fewer than SMs a cluster of 2, 4 or 8 CTAs
// divides the contraction of one tile: every CTA pushes its fp32 partial sums, 128 / splits rows to each
// member, through distributed shared memory and finishes its own rows in member order (one launch, no
// workspace, the same bits on every run).  A step is 128 wide because waiting, announcing bytes and committing
// cost a single thread about 290 cycles each, whatever the step's width.
// 48 KB per step is three times the L2 traffic per FLOP of a pair tile: larger products do not come here
// (choose_variant).
constexpr int S_TILE_N = 64, S_STEP_K = 128, S_STAGES = 4, S_THREADS = 192, S_TMEM_COLS = 64;
constexpr int S_A_BYTES = BM * S_STEP_K * 2, S_B_BYTES = S_TILE_N * S_STEP_K * 2, S_STAGE_BYTES = S_A_BYTES + S_B_BYTES;
constexpr int S_RECV_BYTES = BM * S_TILE_N * 4;

__device__ __forceinline__ void st_cluster_f4(uint32_t addr, float a, float b, float c, float d) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__(S_THREADS, 1)
gemm_small_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                  const __grid_constant__ CUtensorMap map_c, const Params p, const int log_splits) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t bar_full[S_STAGES], bar_empty[S_STAGES], bar_acc_full;
  __shared__ uint32_t tmem_base_slot;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int splits = 1 << log_splits, split = blockIdx.x & (splits - 1);
  const int tiles_m = (p.M + BM - 1) / BM, tiles = tiles_m * ((p.N + S_TILE_N - 1) / S_TILE_N);
  const int z = (int)(blockIdx.x >> log_splits) / tiles, tile = (int)(blockIdx.x >> log_splits) - z * tiles;
  const int m0 = (tile % tiles_m) * BM, n0 = (tile / tiles_m) * S_TILE_N;
  int M = p.M, all_kb = (p.K + S_STEP_K - 1) / S_STEP_K;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S_STAGES; ++s) {
      mbar_init(smem_addr(&bar_full[s]), 1);
      mbar_init(smem_addr(&bar_empty[s]), 1);
    }
    mbar_init(smem_addr(&bar_acc_full), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base_slot)), "r"(S_TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem_base = tmem_base_slot;
  pdl_begin();
  constexpr bool kSumsRows = A_MN && B_MN;  // nothing to sum: zeros (a dead tile of the other layouts stores nothing)
  if (p.live != nullptr) {
    if (kSumsRows) all_kb = (live_rows(p.live, p.K) + S_STEP_K - 1) / S_STEP_K;
    else M = live_rows(p.live, p.M);
    if (m0 >= M) all_kb = 0;  // for the whole cluster: nothing is loaded, multiplied or stored
  }
  const int kb0 = (split * all_kb) >> log_splits, num_kb = (((split + 1) * all_kb) >> log_splits) - kb0;
  if (log_splits > 0) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");  // waited for before the first remote store

  bool ok = true;
  const Scaling sc(p);
  const int quarter = warp & 3, row = m0 + quarter * 32 + lane;
  if (warp == 0) {
    if (elect_one()) {
      uint32_t stage = 0, phase = 0;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (kb >= S_STAGES && !mbar_wait(smem_addr(&bar_empty[stage]), phase ^ 1, p.status, kTimeoutProducer)) break;
        const uint32_t full = smem_addr(&bar_full[stage]), sa = smem_addr(smem + stage * S_STAGE_BYTES), sb = sa + S_A_BYTES;
        const int k0 = (kb0 + kb) * S_STEP_K;
        mbar_expect_tx(full, S_STAGE_BYTES);
        // K-major: boxes of rows x 64 contraction columns; MN-major: boxes of 128 contraction rows x 64 MN-columns
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (A_MN) tma_load_3d(sa + u * (S_A_BYTES / 2), &map_a, full, m0 + u * 64, k0, z);
          else tma_load_3d(sa + u * (S_A_BYTES / 2), &map_a, full, k0 + u * 64, m0, z);
        }
        if (B_MN) {
          tma_load_3d(sb, &map_b, full, n0, k0, z);
        } else {
          tma_load_3d(sb, &map_b, full, k0, n0, z);
          tma_load_3d(sb + S_B_BYTES / 2, &map_b, full, k0 + 64, n0, z);
        }
        if (++stage == S_STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = instr_desc_ab(BM, S_TILE_N, A_MN, B_MN);
      uint32_t stage = 0, phase = 0;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!(ok = mbar_wait(smem_addr(&bar_full[stage]), phase, p.status, kTimeoutMma))) break;
        fence_after_sync();
        const uint32_t sa = smem_addr(smem + stage * S_STAGE_BYTES), sb = sa + S_A_BYTES;
        const uint64_t adesc = A_MN ? smem_desc_mnmajor_sw128(sa, S_A_BYTES / 2) : smem_desc_kmajor_sw128(sa);
        const uint64_t bdesc = B_MN ? smem_desc_mnmajor_sw128(sb, S_B_BYTES) : smem_desc_kmajor_sw128(sb);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t mn = k * (2048 >> 4), in_row = 2 * (k & 3);
          umma_bf16(tmem_base, adesc + (A_MN ? mn : (k >> 2) * (S_A_BYTES / 2 >> 4) + in_row),
                    bdesc + (B_MN ? mn : (k >> 2) * (S_B_BYTES / 2 >> 4) + in_row), idesc, (kb | k) != 0);
        }
        umma_commit(smem_addr(&bar_empty[stage]));
        if (++stage == S_STAGES) { stage = 0; phase ^= 1; }
      }
      if (ok) umma_commit(smem_addr(&bar_acc_full));
    }
  } else if (log_splits == 0) {
    RowPrefetch<S_TILE_N> pre;
    if (p.staged) prefetch_addend_staged<S_TILE_N>(p, m0 + quarter * 32, n0, z, M, lane, pre);
    else prefetch_addend<S_TILE_N>(p, row, n0, z, M, pre);
    ok = mbar_wait(smem_addr(&bar_acc_full), 0, p.status, kTimeoutEpilogue);
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      fence_after_sync();
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16);
      if (p.staged) {
        const uint32_t stage = smem_addr(smem + S_STAGES * S_STAGE_BYTES) + quarter * 4096;
        store_accumulator_staged<S_TILE_N>(p, sc, &map_c, &map_c, stage, taddr, m0 + quarter * 32, n0, z, pre, m0 + quarter * 32 < M, false, kSumsRows && num_kb == 0, lane);
        stage_wait();
      } else if (pre.tile_ok) {
        store_accumulator_prefetched<S_TILE_N>(p, sc, taddr, row, n0, z, pre, kSumsRows && num_kb == 0);
      } else {
        store_accumulator<S_TILE_N>(p, sc, taddr, row, n0, z, M, kSumsRows && num_kb == 0);
      }
    }
  } else {
    ok = mbar_wait(smem_addr(&bar_acc_full), 0, p.status, kTimeoutEpilogue);
    ok = __all_sync(0xffffffffu, ok);
    fence_after_sync();
  }
  __syncwarp();
  if (log_splits > 0) {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // every member's shared memory is live
    // Member j finishes rows j * 128 / splits .. of the tile: [source][own row][64 columns] fp32, 16-byte chunks
    // XOR-swizzled by the row, so that lanes (rows) that push the same columns do not share banks.
    const int log_rows = 7 - log_splits, tile_row = quarter * 32 + lane, own_rows = 1 << log_rows;
    const uint32_t recv = smem_addr(smem + S_STAGES * S_STAGE_BYTES);
    if (warp >= 2 && ok) {
      const int to = tile_row >> log_rows, r0 = tile_row & (own_rows - 1);
      const uint32_t dst = map_to_cta(recv, to) + ((split << log_rows) + r0) * 256;
      const bool empty = num_kb == 0;  // no contraction step ran here: the tensor memory holds nothing
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t r[32];
        tmem_ld32(tmem_base + ((uint32_t)(quarter * 32) << 16) + c * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int v = 0; v < 32; ++v)
          if (empty) r[v] = 0u;
#pragma unroll
        for (int v = 0; v < 8; ++v)
          st_cluster_f4(dst + (((c * 8 + v) ^ (r0 & 15)) << 4), __uint_as_float(r[v * 4]), __uint_as_float(r[v * 4 + 1]), __uint_as_float(r[v * 4 + 2]),
                        __uint_as_float(r[v * 4 + 3]));
      }
    }
    __syncwarp();
    cluster_sync_all();
    if (warp >= 2 && ok) {
      const float4* got = reinterpret_cast<const float4*>(smem + S_STAGES * S_STAGE_BYTES);
      for (int e = threadIdx.x - 64; e < own_rows * 16; e += 128) {  // 16 lanes per row: whole lines
        const int r0 = e >> 4, c = e & 15, orow = m0 + (split << log_rows) + r0;
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int src = 0; src < splits; ++src) {
          const float4 o = got[((src << log_rows) + r0) * 16 + (c ^ (r0 & 15))];
          t.x += o.x; t.y += o.y; t.z += o.z; t.w += o.w;
        }
        if (orow < M) store_vec4(p, sc, t, orow, n0 + c * 4, z);
      }
    }
  }

  // A role that gave up did so after seconds of polling, far beyond the lifetime of any
  // bulk copy it had issued, so no copy is still writing shared memory at this point.
  fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(S_TMEM_COLS) : "memory");
  }
}

// ---- 256x256 tiles on CTA pairs ----------------------------------------------------------
// A pipeline stage holds KSUB sub-tiles of 64 K-elements (KSUB x 32 KB per CTA); the ring
// always spans 192 KB.  KSUB = 2 halves the number of barrier waits / commits the MMA
// thread executes per unit of tensor work (its instruction stream, not the tensor pipe,
// is what paces the loop at KSUB = 1).
constexpr int P_HALF = 128;                                    // rows of A and of B staged per CTA
constexpr int P_A_BYTES = P_HALF * BK * 2, P_B_BYTES = P_HALF * BK * 2, P_SUB_BYTES = P_A_BYTES + P_B_BYTES;
constexpr int P_TILE_M = 2 * P_HALF, P_TILE_N = 2 * P_HALF;
constexpr int P_RING_BYTES = 6 * P_SUB_BYTES;
constexpr int P_STAGE_OUT_BYTES = 8 * 4096;  // one staging area per epilogue warp
// The pair kernel runs eight epilogue warps: warps w and w + 4 reach the same 32 TMEM lanes (rows) and take 128 of the
// tile's 256 columns each, so two warps per scheduler share the epilogue's instruction stream (with four warps the row
// statistics of the lm_head epilogue, and the addend of short-contraction weight gradients, set the pace of the tile).
constexpr int P_THREADS = 320, P_EPI_COLS = 128;

// A contraction in parts: the weight gradients of a weight that was used several times (training-time-test passes), each
// use with its own pair of operands.  As one product per use every product but the first read and wrote the gradient once
// more, and its tiles were short: at 736 rows the epilogue took longer than the products.  One tile loop over all parts
// accumulates them in tensor memory - in fp32, without the roundings in between.
//   24576 x 4096 x 736, three uses: 463 us as separate products, 286 as one; 16384 x 2048 x 1001: 191 and 133 us.
constexpr int kMoreParts = 3;
struct MoreParts {
  CUtensorMap a[kMoreParts], b[kMoreParts];
  const int* seg[kMoreParts];   // grouped contraction: the part's own segments
  const int* live[kMoreParts];  // as Params::live
  int rows[kMoreParts];
  int n;
};
struct NoParts {};
template <bool PARTS> struct PartsArg { typedef NoParts type; };
template <> struct PartsArg<true> { typedef MoreParts type; };
// 128-wide contraction steps of the parts of a plain product, read once per thread
template <bool PARTS> struct PartSteps {
  __device__ __forceinline__ explicit PartSteps(const NoParts&) {}
};
template <> struct PartSteps<true> {
  int kb[kMoreParts];
  __device__ __forceinline__ explicit PartSteps(const MoreParts& more) {
#pragma unroll
    for (int i = 0; i < kMoreParts; ++i) kb[i] = i < more.n ? (live_rows(more.live[i], more.rows[i]) + 127) >> 7 : 0;
  }
};
// ... of part i for this tile, and where they start
__device__ __forceinline__ int part_steps(const Params& p, const MoreParts& more, const PartSteps<true>& steps, int i, int tile, int per, int& k0) {
  k0 = 0;
  if (p.grp.mode != kGroupK) return i == 0 ? steps.kb[0] : i == 1 ? steps.kb[1] : steps.kb[2];
  const int e = tile / per;
  k0 = more.seg[i][e];
  return (more.seg[i][e + 1] - k0) >> 7;
}
__device__ __forceinline__ int more_steps(const Params& p, const MoreParts& more, const PartSteps<true>& steps, int tile, int per) {
  int sum = 0, k0;
  for (int i = 0; i < more.n; ++i) sum += part_steps(p, more, steps, i, tile, per, k0);
  return sum;
}
__device__ __forceinline__ int more_steps(const Params&, const NoParts&, const PartSteps<false>&, int, int) { return 0; }

// DIVIDE: the tiles of a part-filled last wave may be divided between pairs (an instance of its own: what that takes in registers
// cost undivided products 2 %).
template <int KSUB, bool A_MN = false, bool B_MN = false, bool PARTS = false, bool DIVIDE = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(P_THREADS, 1)
gemm_tn_2cta_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                    const __grid_constant__ CUtensorMap map_c, const __grid_constant__ CUtensorMap map_h, const Params p,
                    const __grid_constant__ typename PartsArg<PARTS>::type more) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  static_assert(!PARTS || (A_MN && B_MN), "parts are those of weight gradients");
  static_assert(!DIVIDE || !PARTS, "a contraction in parts is not divided");
  static_assert(KSUB == 2 || (!A_MN && !B_MN), "MN-major operands are staged as 128-row boxes: KSUB must be 2");
  constexpr int P_STAGES = 6 / KSUB;
  constexpr int P_STAGE_BYTES = KSUB * P_SUB_BYTES;
  constexpr int STAGE_K = KSUB * BK;
  __shared__ __align__(8) uint64_t bar_full[P_STAGES], bar_empty[P_STAGES], bar_acc_full[2], bar_acc_empty[2];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int ticket_slot;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int num_pairs = gridDim.x >> 1;
  if (threadIdx.x == 0) {
    for (int s = 0; s < P_STAGES; ++s) {
      mbar_init(smem_addr(&bar_full[s]), 1);   // the leader's expect_tx arrival; bytes come from both CTAs' copies
      mbar_init(smem_addr(&bar_empty[s]), 1);  // one multicast commit per use
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_addr(&bar_acc_full[a]), 1);
      mbar_init(smem_addr(&bar_acc_empty[a]), 512);  // the epilogue threads of both CTAs (used in the leader only)
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {  // collective over the pair: the same warp of both CTAs
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base_slot)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  fence_before_sync();
  cluster_sync_all();  // barriers of both CTAs are initialised before any remote signal
  fence_after_sync();
  const uint32_t tmem_base = tmem_base_slot;
  pdl_begin();
  constexpr bool kSumsRows = A_MN && B_MN;
  const int M = kSumsRows ? p.M : live_rows(p.live, p.M), K = kSumsRows ? live_rows(p.live, p.K) : p.K;
  const int tiles_m = (M + P_TILE_M - 1) / P_TILE_M, tiles_n = (p.N + P_TILE_N - 1) / P_TILE_N;
  const int num_kb = (K + STAGE_K - 1) / STAGE_K;
  [[maybe_unused]] const PartSteps<PARTS> part_kb(more);
  const int num_tiles = p.grp.mode == kGroupRows ? p.grp.tile_start[p.grp.num_groups] * tiles_n
                        : p.grp.mode == kGroupK  ? p.grp.num_groups * tiles_m * tiles_n
                                                 : p.batch * (p.symmetric ? tiles_m * (tiles_m + 1) / 2 : tiles_m * tiles_n);
  SplitPlan plan{num_tiles, {0, 0}, {1, 1}, 0, 0.f};
  if (DIVIDE) plan = split_plan(num_tiles, num_kb, num_pairs);
  int number = blockIdx.x >> 1;  // which pair this is; where tiles are divided in the order of starting
  if (DIVIDE && plan.left[0] > 0) {
    if (leader && threadIdx.x == 0) ticket_slot = atomicAdd(p.sync, 1);
    __syncwarp();
    cluster_sync_all();
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(number) : "r"(map_to_cta(smem_addr(&ticket_slot), 0)) : "memory");
  }

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    if (elect_one()) {
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      for (Pieces<DIVIDE> it(number); ok && it.advance(plan, num_kb, number, num_pairs);) {
        const int tile = it.tile;
        const TileInfo ti = decode_tile<B_MN>(p, M, tile, tiles_m, tiles_n, num_kb, (int)rank);
        auto load_steps = [&](const CUtensorMap* ma, const CUtensorMap* mb, int a_k0, int b_k0, int count) {
          for (int kb = 0; kb < count; ++kb) {
            if (!(ok = mbar_wait(smem_addr(&bar_empty[stage]), phase ^ 1, p.status, kTimeoutProducer))) break;
            const uint32_t full_local = smem_addr(&bar_full[stage]);
            if (leader) mbar_expect_tx(full_local, 2 * P_STAGE_BYTES);
            const uint32_t full_leader = map_to_cta(full_local, 0);
            const uint32_t sa = smem_addr(smem + stage * P_STAGE_BYTES);
            // Elements outside the matrices read as zeros (TMA fill).  K-major operand: sub-tile u =
            // 128 rows x 64 contraction columns.  MN-major operand: sub-tile u = 128 contraction rows x
            // 64 MN-columns (MN-elements 64u .. 64u+63 of this CTA's 128).  Either way 16 KB at the same place.
#pragma unroll
            for (int u = 0; u < KSUB; ++u) {
              if (A_MN) tma_load_3d_pair(sa + u * P_SUB_BYTES, ma, full_leader, ti.a_m + u * 64, a_k0 + kb * STAGE_K, ti.z);
              else tma_load_3d_pair(sa + u * P_SUB_BYTES, ma, full_leader, a_k0 + kb * STAGE_K + u * BK, ti.a_m, ti.z);
              if (B_MN) tma_load_3d_pair(sa + u * P_SUB_BYTES + P_A_BYTES, mb, full_leader, ti.b_n + u * 64, b_k0 + kb * STAGE_K, ti.z);
              else tma_load_3d_pair(sa + u * P_SUB_BYTES + P_A_BYTES, mb, full_leader, b_k0 + kb * STAGE_K + u * BK, ti.b_n, ti.z);
            }
            if (++stage == P_STAGES) { stage = 0; phase ^= 1; }
          }
        };
        load_steps(&map_a, &map_b, ti.a_k0 + it.k0 * STAGE_K, ti.b_k0 + it.k0 * STAGE_K, DIVIDE ? it.steps : ti.num_kb);
        if constexpr (PARTS) {
          for (int i = 0; i < more.n && ok; ++i) {
            int k0;
            const int count = part_steps(p, more, part_kb, i, tile, tiles_m * tiles_n, k0);
            load_steps(&more.a[i], &more.b[i], k0, k0, count);
          }
        }
      }
      // tail: stay until the MMAs that read this CTA's last slots have retired (their
      // completion is signalled into this CTA's shared memory)
      for (int s = 0; s < P_STAGES && ok; ++s) {
        ok = mbar_wait(smem_addr(&bar_empty[stage]), phase ^ 1, p.status, kTimeoutProducer);
        if (++stage == P_STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader CTA only)
    if (leader && elect_one()) {
      constexpr uint32_t idesc = instr_desc_ab(P_TILE_M, P_TILE_N, A_MN, B_MN);
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      int local = 0;
      for (Pieces<DIVIDE> it(number); ok && it.advance(plan, num_kb, number, num_pairs); ++local) {
        const int acc = local & 1;
        if (!(ok = mbar_wait(smem_addr(&bar_acc_empty[acc]), ((local >> 1) & 1) ^ 1, p.status, kTimeoutMma))) break;
        fence_after_sync();
        const uint32_t tmem_d = tmem_base + acc * BN;
        const int tile_kb = DIVIDE ? it.steps
                                    : decode_tile<B_MN>(p, M, it.tile, tiles_m, tiles_n, num_kb, 0).num_kb + more_steps(p, more, part_kb, it.tile, tiles_m * tiles_n);
        for (int kb = 0; kb < tile_kb; ++kb) {
          if (!(ok = mbar_wait(smem_addr(&bar_full[stage]), phase, p.status, kTimeoutMma))) break;
          fence_after_sync();
          const uint32_t sa = smem_addr(smem + stage * P_STAGE_BYTES);
          // MN-major: the two 64-element column blocks are P_SUB_BYTES apart (leading byte offset)
          const uint64_t adesc = A_MN ? smem_desc_mnmajor_sw128(sa, P_SUB_BYTES) : smem_desc_kmajor_sw128(sa);
          const uint64_t bdesc = B_MN ? smem_desc_mnmajor_sw128(sa + P_A_BYTES, P_SUB_BYTES) : smem_desc_kmajor_sw128(sa + P_A_BYTES);
#pragma unroll
          for (int u = 0; u < KSUB; ++u) {
#pragma unroll
            for (int k = 0; k < BK / 16; ++k) {
              // K-major: next sub-tile + P_SUB_BYTES, next 16 K-elements inside a 128-byte swizzled row + 32 bytes;
              // MN-major: 16 contraction rows of 128 bytes = 2048 bytes per step (all in 16-byte units)
              const uint32_t off_k = u * (P_SUB_BYTES >> 4) + 2 * k, off_mn = (u * (BK / 16) + k) * (2048 >> 4);
              umma_bf16_pair(tmem_d, adesc + (A_MN ? off_mn : off_k), bdesc + (B_MN ? off_mn : off_k), idesc, (kb | u | k) != 0);
            }
          }
          umma_commit_pair(smem_addr(&bar_empty[stage]));  // frees the slot in both CTAs
          if (++stage == P_STAGES) { stage = 0; phase ^= 1; }
        }
        if (ok) umma_commit_pair(smem_addr(&bar_acc_full[acc]));  // wakes the epilogues of both CTAs
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..9, both CTAs)
    const int quarter = warp & 3;         // TMEM lanes 32 * quarter .. + 31
    const int chalf = (warp - 2) >> 2;    // columns 128 * chalf .. + 127 of the tile
    const uint32_t acc_empty_leader[2] = {map_to_cta(smem_addr(&bar_acc_empty[0]), 0), map_to_cta(smem_addr(&bar_acc_empty[1]), 0)};
    const uint32_t stage = smem_addr(smem + P_RING_BYTES) + (warp - 2) * 4096;
    RowPrefetch<P_EPI_COLS> pre;
    bool ok = true;
    int local = 0;
    for (Pieces<DIVIDE> it(number); ok && it.advance(plan, num_kb, number, num_pairs); ++local) {
      const int acc = local & 1, tile = it.tile;
      const int parts = !DIVIDE || it.round < 0 ? 1 : it.round == 0 ? plan.parts[0] : plan.parts[1];
      const bool hands_over = DIVIDE && it.part + 1 < parts;  // another pair finishes the tile
      const TileInfo ti = decode_tile<B_MN>(p, M, tile, tiles_m, tiles_n, num_kb, (int)rank);
      const int row = ti.c_row0 + quarter * 32 + lane, n0 = ti.n0 + chalf * P_EPI_COLS;
      const bool zero = ti.num_kb + more_steps(p, more, part_kb, tile, tiles_m * tiles_n) == 0;
      const bool with_stats = p.rs.targets != nullptr, gated = p.epilogue == kSwiGLU;
      if (with_stats) prefetch_targets<P_EPI_COLS>(p, row, n0, pre);
      else if (hands_over) pre.tile_ok = pre.valid = false;
      else if (p.staged && !gated && (DIVIDE || local == 0)) prefetch_addend_staged<P_EPI_COLS>(p, ti.c_row0 + quarter * 32, n0, ti.z, ti.row_end, lane, pre);
      else if (!gated && !p.staged) prefetch_addend<P_EPI_COLS>(p, row, n0, ti.z, ti.row_end, pre);
      ok = mbar_wait(smem_addr(&bar_acc_full[acc]), (local >> 1) & 1, p.status, kTimeoutEpilogue);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      fence_after_sync();
      const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * BN, taddr = lane_base + chalf * P_EPI_COLS;
      if (DIVIDE && parts > 1) {
        auto slot = [&](int pair) { return ((it.round * num_pairs + pair) * 2 + (int)rank) * 8 + warp - 2; };
        if (hands_over) {
          split_put(p.partial + (int64_t)slot(number) * 1024, taddr, lane);
          __threadfence();
          __syncwarp();
          if (lane == 0) asm volatile("st.release.gpu.global.s32 [%0], 1;" ::"l"(p.sync + 1 + slot(number)) : "memory");
          fence_before_sync();
          mbar_arrive_cluster_relaxed(acc_empty_leader[acc]);
          continue;
        }
        const int n = it.round == 0 ? plan.left[0] : plan.left[1];
        for (int other = number - n * it.part; other < number && ok; other += n) {
          if (lane == 0) ok = flag_wait(p.sync + 1 + slot(other), p.status, kTimeoutPartial);
          ok = __shfl_sync(0xffffffffu, ok, 0);
          __syncwarp();
          if (ok) split_add(p.partial + (int64_t)slot(other) * 1024, taddr, lane);
        }
        if (!ok) break;
      }
      const int row0 = ti.c_row0 + quarter * 32;
      const Scaling sc(p);
      if (gated)  // this warp: gate columns 64 * chalf .. + 63 of the tile and the same up columns
        store_accumulator_swiglu(p, &map_c, &map_h, stage, lane_base + chalf * 64, row0, ti.n0 + chalf * 64,
                                 row0 < ti.row_end, lane);
      else if (with_stats) store_accumulator_with_stats<P_EPI_COLS>(p, taddr, row, n0, ti.tile_n * 2 + chalf, tiles_n * 2, pre);
      else if (p.staged) {
        const int following = tile + num_pairs;
        TileInfo tn{};
        auto ahead = [&](int h) {
          if (DIVIDE || following >= plan.whole) return;
          if (h == 0) tn = decode_tile<B_MN>(p, M, following, tiles_m, tiles_n, num_kb, (int)rank);
          prefetch_addend_staged<P_EPI_COLS>(p, tn.c_row0 + quarter * 32, tn.n0 + chalf * P_EPI_COLS, tn.z, tn.row_end, lane, h, pre);
        };
        store_accumulator_staged<P_EPI_COLS>(p, sc, &map_c, &map_h, stage, taddr, row0, n0, ti.z, pre, row0 < ti.row_end, ti.mirror, zero, lane, ahead);
      }
      else if (pre.tile_ok) store_accumulator_prefetched<P_EPI_COLS>(p, sc, taddr, row, n0, ti.z, pre, zero);
      else store_accumulator<P_EPI_COLS>(p, sc, taddr, row, n0, ti.z, ti.row_end, zero);
      fence_before_sync();
      mbar_arrive_cluster_relaxed(acc_empty_leader[acc]);
    }
    stage_wait();
  }

  // Both CTAs stay until the pair is done: the peer's copies signal the leader's barriers,
  // the leader's MMAs read the peer's shared memory and write its TMEM.
  fence_before_sync();
  __syncthreads();
  cluster_sync_relaxed();
  if (warp == 1) {
    fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// ---- 256x256 tiles with the contraction split over the CTA pairs of a cluster -----------------------
// A product with few tiles and a long contraction (short rows through a wide MLP, Gram-like weight gradients
// of narrow layers) occupies as many pairs as it has tiles.  Here a cluster of SPLITS pairs shares one tile:
// every pair runs its part of the contraction at the pair kernel's operand traffic (64 B per clock and SM,
// where smaller tiles would be bound by L2), then the partial accumulators are reduce-scattered through
// distributed shared memory: every CTA pushes 128 / SPLITS of its rows in fp32 to each member with its role,
// into the (now idle) operand ring, and the receiver sums its rows in pair order and stores whole lines.
// One launch, no workspace, the same bits on every run.
template <int SPLITS, bool A_MN, bool B_MN>
__global__ void __cluster_dims__(2 * SPLITS, 1, 1) __launch_bounds__(P_THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const Params p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int KSUB = 2, STAGES = 6 / KSUB, STAGE_BYTES = KSUB * P_SUB_BYTES, STAGE_K = KSUB * BK;
  constexpr int OWN_ROWS = P_HALF / SPLITS;  // rows of its 128 that this CTA finishes
  static_assert(P_HALF * P_TILE_N * 4 <= P_RING_BYTES, "the partial sums must fit the ring");
  __shared__ __align__(8) uint64_t bar_full[STAGES], bar_empty[STAGES], bar_acc_full;
  __shared__ uint32_t tmem_base_slot;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t crank = cluster_ctarank(), role = crank & 1, split = crank >> 1;
  const bool leader = role == 0;
  const int tiles_m = (p.M + P_TILE_M - 1) / P_TILE_M;
  const int tiles = tiles_m * ((p.N + P_TILE_N - 1) / P_TILE_N);
  const int z = (int)(blockIdx.x / (2 * SPLITS)) / tiles, tile = (int)(blockIdx.x / (2 * SPLITS)) - z * tiles;
  const int m0 = (tile % tiles_m) * P_TILE_M + role * P_HALF, n0 = (tile / tiles_m) * P_TILE_N;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_addr(&bar_full[s]), 1);
      mbar_init(smem_addr(&bar_empty[s]), 1);
    }
    mbar_init(smem_addr(&bar_acc_full), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base_slot)), "r"(P_TILE_N) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  fence_before_sync();
  cluster_sync_all();
  fence_after_sync();
  const uint32_t tmem_base = tmem_base_slot;
  pdl_begin();
  constexpr bool kSumsRows = A_MN && B_MN;
  const int M = kSumsRows ? p.M : live_rows(p.live, p.M), K = kSumsRows ? live_rows(p.live, p.K) : p.K;
  const bool dead = (tile % tiles_m) * P_TILE_M >= M;  // the whole cluster
  const int all_kb = dead ? 0 : (K + STAGE_K - 1) / STAGE_K, per_kb = (all_kb + SPLITS - 1) / SPLITS;
  const int kb0 = split * per_kb, num_kb = max(0, min(per_kb, all_kb - kb0));

  bool ok = true;
  const Scaling sc(p);
  const int quarter = warp & 3, chalf = (warp - 2) >> 2;
  if (warp == 0) {
    if (elect_one()) {
      uint32_t stage = 0, phase = 0;
      const int b0 = n0 + role * P_HALF;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!(ok = mbar_wait(smem_addr(&bar_empty[stage]), phase ^ 1, p.status, kTimeoutProducer))) break;
        const uint32_t full_local = smem_addr(&bar_full[stage]);
        if (leader) mbar_expect_tx(full_local, 2 * STAGE_BYTES);
        const uint32_t full_leader = map_to_cta(full_local, crank & ~1u);
        const uint32_t sa = smem_addr(smem + stage * STAGE_BYTES);
        const int k0 = (kb0 + kb) * STAGE_K;
#pragma unroll
        for (int u = 0; u < KSUB; ++u) {
          if (A_MN) tma_load_3d_pair(sa + u * P_SUB_BYTES, &map_a, full_leader, m0 + u * 64, k0, z);
          else tma_load_3d_pair(sa + u * P_SUB_BYTES, &map_a, full_leader, k0 + u * BK, m0, z);
          if (B_MN) tma_load_3d_pair(sa + u * P_SUB_BYTES + P_A_BYTES, &map_b, full_leader, b0 + u * 64, k0, z);
          else tma_load_3d_pair(sa + u * P_SUB_BYTES + P_A_BYTES, &map_b, full_leader, k0 + u * BK, b0, z);
        }
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      for (int s = 0; s < STAGES && ok; ++s) {  // every MMA that reads this CTA's ring has retired
        ok = mbar_wait(smem_addr(&bar_empty[stage]), phase ^ 1, p.status, kTimeoutProducer);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (leader && elect_one()) {
      constexpr uint32_t idesc = instr_desc_ab(P_TILE_M, P_TILE_N, A_MN, B_MN);
      const uint16_t mask = (uint16_t)(3u << (crank & ~1u));
      uint32_t stage = 0, phase = 0;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!(ok = mbar_wait(smem_addr(&bar_full[stage]), phase, p.status, kTimeoutMma))) break;
        fence_after_sync();
        const uint32_t sa = smem_addr(smem + stage * STAGE_BYTES);
        const uint64_t adesc = A_MN ? smem_desc_mnmajor_sw128(sa, P_SUB_BYTES) : smem_desc_kmajor_sw128(sa);
        const uint64_t bdesc = B_MN ? smem_desc_mnmajor_sw128(sa + P_A_BYTES, P_SUB_BYTES) : smem_desc_kmajor_sw128(sa + P_A_BYTES);
#pragma unroll
        for (int u = 0; u < KSUB; ++u) {
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            const uint32_t off_k = u * (P_SUB_BYTES >> 4) + 2 * k, off_mn = (u * (BK / 16) + k) * (2048 >> 4);
            umma_bf16_pair(tmem_base, adesc + (A_MN ? off_mn : off_k), bdesc + (B_MN ? off_mn : off_k), idesc, (kb | u | k) != 0);
          }
        }
        umma_commit_pair(smem_addr(&bar_empty[stage]), mask);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (ok) umma_commit_pair(smem_addr(&bar_acc_full), mask);
    }
  } else {
    ok = mbar_wait(smem_addr(&bar_acc_full), 0, p.status, kTimeoutEpilogue);
    ok = __all_sync(0xffffffffu, ok);
    fence_after_sync();
  }
  __syncwarp();
  // Every pair has finished its contraction: nothing reads or writes the rings any more, they can take partial sums.
  cluster_sync_relaxed();
  if (warp >= 2 && ok) {
    // [source pair][own row][256 columns] fp32, 16-byte chunks XOR-swizzled by the row (lanes are rows)
    const int tile_row = quarter * 32 + lane, to = tile_row / OWN_ROWS, r0 = tile_row % OWN_ROWS;
    const uint32_t dst = map_to_cta(smem_addr(smem), to * 2 + role) + (split * OWN_ROWS + r0) * (P_TILE_N * 4);
    const bool empty = num_kb == 0;  // this pair had no contraction step: its tensor memory holds nothing
#pragma unroll
    for (int c = 0; c < P_EPI_COLS / 32; ++c) {
      uint32_t r[32];
      tmem_ld32(tmem_base + ((uint32_t)(quarter * 32) << 16) + chalf * P_EPI_COLS + c * 32, r);
      tmem_ld_wait();
#pragma unroll
      for (int v = 0; v < 32; ++v)
        if (empty) r[v] = 0u;
#pragma unroll
      for (int v = 0; v < 8; ++v)
        st_cluster_f4(dst + (((chalf * 32 + c * 8 + v) ^ (r0 & 31)) << 4), __uint_as_float(r[v * 4]), __uint_as_float(r[v * 4 + 1]), __uint_as_float(r[v * 4 + 2]),
                      __uint_as_float(r[v * 4 + 3]));
    }
  }
  __syncwarp();
  cluster_sync_all();
  if (warp >= 2 && ok) {
    const float4* got = reinterpret_cast<const float4*>(smem);
#pragma unroll 4
    for (int e = threadIdx.x - 64; e < OWN_ROWS * (P_TILE_N / 4); e += 256) {  // 64 lanes per row: whole lines
      const int r0 = e / (P_TILE_N / 4), c = e % (P_TILE_N / 4), row = m0 + split * OWN_ROWS + r0;
      float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int src = 0; src < SPLITS; ++src) {  // in pair order on every pair
        const float4 o = got[(src * OWN_ROWS + r0) * (P_TILE_N / 4) + (c ^ (r0 & 31))];
        t.x += o.x; t.y += o.y; t.z += o.z; t.w += o.w;
      }
      if (row < M) store_vec4(p, sc, t, row, n0 + c * 4, z);
    }
  }
  fence_before_sync();
  __syncthreads();
  cluster_sync_relaxed();
  if (warp == 1) {
    fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(P_TILE_N) : "memory");
  }
}

// ---- host side ---------------------------------------------------------------------------
}  // namespace tc

template <typename Kernel>
static bool allow_smem(Kernel kernel, int bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
}

template <int SPLITS>
static void launch_split(int a_mn, int b_mn, int tiles, int smem, cudaStream_t stream, const CUtensorMap& map_a, const CUtensorMap& map_b, const tc::Params& p) {
  const int grid = tiles * 2 * SPLITS;
  if (a_mn && b_mn) launch_pdl(tc::gemm_split_kernel<SPLITS, true, true>, grid, tc::P_THREADS, smem, stream, map_a, map_b, p);
  else if (a_mn) launch_pdl(tc::gemm_split_kernel<SPLITS, true, false>, grid, tc::P_THREADS, smem, stream, map_a, map_b, p);
  else if (b_mn) launch_pdl(tc::gemm_split_kernel<SPLITS, false, true>, grid, tc::P_THREADS, smem, stream, map_a, map_b, p);
  else launch_pdl(tc::gemm_split_kernel<SPLITS, false, false>, grid, tc::P_THREADS, smem, stream, map_a, map_b, p);
}

static cudaError_t launch_small(int a_mn, int b_mn, int tiles, int log_splits, int smem, cudaStream_t stream, const CUtensorMap& map_a, const CUtensorMap& map_b,
                                const CUtensorMap& map_c, const tc::Params& p) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(tiles << log_splits);
  cfg.blockDim = dim3(tc::S_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2] = {};
  attr[0] = pdl_attribute();
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 1u << log_splits;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = log_splits > 0 ? 2 : 1;
  if (a_mn && b_mn) return cudaLaunchKernelEx(&cfg, tc::gemm_small_kernel<true, true>, map_a, map_b, map_c, p, log_splits);
  if (a_mn) return cudaLaunchKernelEx(&cfg, tc::gemm_small_kernel<true, false>, map_a, map_b, map_c, p, log_splits);
  if (b_mn) return cudaLaunchKernelEx(&cfg, tc::gemm_small_kernel<false, true>, map_a, map_b, map_c, p, log_splits);
  return cudaLaunchKernelEx(&cfg, tc::gemm_small_kernel<false, false>, map_a, map_b, map_c, p, log_splits);
}

enum Variant : int { kPairK64 = 2, kPair = 3, kSplit2 = 4, kSplit4 = 5, kPairDivided = 6, kSmall = 10, kSmall2 = 11, kSmall4 = 12, kSmall8 = 13 };
constexpr int kMaxPairs = kNumSM / 2;

// 256x256 tiles of a stack of products (of a symmetric one: the diagonal and what lies above it).
static int64_t pair_tile_count(int M, int N, int batch, int symmetric) {
  const int64_t m = (M + tc::P_TILE_M - 1) / tc::P_TILE_M, n = (N + tc::P_TILE_N - 1) / tc::P_TILE_N;
  return batch * (symmetric ? m * (m + 1) / 2 : m * n);
}

// How many clusters of `size` CTAs (one per SM) the device holds at a time: the GPCs do not divide evenly.  Where the runtime
// does not say, three quarters of the SMs; a call with more clusters than fit takes a second wave.
static int resident_clusters(int size) {
  static std::atomic<int> known[64][3];
  const int dev = PerDeviceOnce::device(), slot = size == 2 ? 0 : size == 4 ? 1 : 2;
  return remember(dev >= 0 ? &known[dev][slot] : nullptr, [size](int* n) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kNumSM / size * size);
    cfg.blockDim = dim3(tc::S_THREADS);
    cfg.dynamicSmemBytes = tc::S_STAGES * tc::S_STAGE_BYTES + tc::S_RECV_BYTES + 1024;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = size;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(n, tc::gemm_small_kernel<false, false>, &cfg) == cudaSuccess) return true;
    cudaGetLastError();
    return false;
  }, kNumSM / size * 3 / 4);
}

// The kernel for a plain product, by predicted time.  Each form costs a fixed part (launch, pipeline fill, epilogue,
// exchange of partial sums) plus its 128-wide contraction steps; the constants (us) are fits to launches inside CUDA
// graphs at 128 .. 3072 rows and columns and contractions of 128 .. 32000, all three layouts:
//   pair tiles     7.0 + 0.56 / step and wave     (2048 x 1024 x 1024: 10.9 us; 1000 x 2048 x 8192: 43.8)
//   the same with the tiles of a part-filled last wave divided: 8.0 + what split_plan says, 26.0 with no whole wave
//                                                  (1280 x 4096 x 4096: 43.9 -> 34.7; 768 x 2048 x 32000: 85.6 -> 78.5)
//   128 x 64 tiles 3.3 + 0.34 / step and wave     (1024 x 1024 x 1024: 6.7; 128 x 256 x 256: 4.0)
//   the same, contraction over 2, 4, 8 CTAs: 5.0 + 0.34 / step, one wave only   (128 x 512 x 2048: 6.1 at 8, 8.6 unsplit)
//   pair tiles over 2, 4 pairs: 10.8 + 0.66 / step, one wave only               (1000 x 2048 x 8192: 31.9 at 2)
// Several waves of small tiles are bound by L2-to-SM traffic, so they pay a full wave each; the model drops them
// quickly.  Products of more than about two waves of pair tiles always come out as pair tiles.
// Where the device's count bounds the rows, M is the most there can be: a captured launch serves any count, and
// so does the choice.  It stays the best form, or within 2 us of it, down to half the rows: 1001 x 2048 x 8192 with 1001, 768 and 512 rows in
// use: 2 pairs 41.0, 38.9 and 38.9, pair tiles 53.2, 53.2 and 51.2, 128 x 64 tiles 57.3, 56.2 and 36.9; 1001 x 3072 x 4096: pair tiles
// 34.8, 32.8 and 32.8, 128 x 64 tiles 49.2, 38.9 and 34.8.
// divide: tiles may be divided between pairs.  Gradients' products may; a forward product, whose rows give the same bits in a batch
// of any size (with all rows or only the needed ones), is not divided by what is left over of its tiles.
static int choose_variant(int M, int N, int K, int batch, int symmetric, bool divide) {
  using namespace tc;
  const int64_t small = (int64_t)((M + BM - 1) / BM) * ((N + S_TILE_N - 1) / S_TILE_N) * batch;
  const int64_t big = pair_tile_count(M, N, batch, 0);
  const int steps = (K + 127) / 128;
  int best = kPair;
  const int64_t pair_tiles = pair_tile_count(M, N, batch, symmetric);
  float t = 7.0f + 0.56f * steps * ((pair_tiles + kMaxPairs - 1) / kMaxPairs);
  auto consider = [&](int variant, float us) {
    if (us < t) { t = us; best = variant; }
  };
  if (divide && pair_tiles < (1 << 20)) {
    const SplitPlan s = split_plan((int)pair_tiles, steps, kMaxPairs);
    if (s.left[0] > 0) consider(kPairDivided, (s.whole > 0 ? 8.0f : 26.0f) + s.us);
  }
  if (small <= 4 * kNumSM) consider(kSmall, 2.0f + (1.3f + 0.34f * steps) * ((small + kNumSM - 1) / kNumSM));
  for (int log = 1; log <= 3; ++log)
    if (steps >= (2 << log) && small <= resident_clusters(1 << log)) consider(kSmall + log, 5.0f + 0.34f * ((steps + (1 << log) - 1) >> log));
  for (int log = 1; log <= 2; ++log)
    if (steps >= (4 << log) && big <= resident_clusters(2 << log)) consider(log == 1 ? kSplit2 : kSplit4, 10.8f + 0.66f * ((steps + (1 << log) - 1) >> log));
  return best;
}

// Space for the partial sums of divided tiles: what a product in this form may need, 0 if it never divides any.  rows_vary: M is
// only the most that the device may ask for.
static bool may_split(int M, int N, int K, int batch, int symmetric, bool rows_vary) {
  const int kb = (K + 127) / 128;
  for (int m = M; m > 0; m -= tc::P_TILE_M) {
    const int64_t tiles = pair_tile_count(m, N, batch, symmetric);
    if (tiles < (1 << 20) && tc::split_plan((int)tiles, kb, kMaxPairs).left[0] > 0) return true;
    if (!rows_vary) break;
  }
  return false;
}
int64_t gemm_split_floats() { return (int64_t)2 * kMaxPairs * 2 * 8 * 1024 * 4; }
int gemm_split_sync_ints() { return tc::kSplitSync; }
static_assert(kMaxPairs == 74, "kSplitSync counts the pairs");

// Further uses of a weight whose gradient is one product (see MoreParts); the first is the plain a, b, K.
struct PartsSpec {
  int n = 0;
  const void* a[tc::kMoreParts];
  const void* b[tc::kMoreParts];
  int K[tc::kMoreParts];
  int64_t lda[tc::kMoreParts], ldb[tc::kMoreParts];
  const int* seg[tc::kMoreParts];
  const int* live[tc::kMoreParts];
};

// What a stack of products adds to a single one; see Params.
struct BatchSpec {
  int batch = 1;
  int64_t a_stride = 0, b_stride = 0, c_stride = 0, r_stride = 0;
  float alpha = 1.f, beta = 1.f, diagonal = 0.f;
  bool once = false;
  bool symmetric = false;
};

// C[M,N] = op(A) * op(B)^T with epilogue (0 store, 1 C += result, 2 result + residual).
//   a_mn == 0: A is [M, K] row-major (K-major), lda = row stride;  a_mn == 1: A is [K, M] row-major (M contiguous)
//   b_mn == 0: B is [N, K] row-major (K-major), ldb = row stride;  b_mn == 1: B is [K, N] row-major (N contiguous)
// lda / ldb / ldc / ldr in elements; operand rows must be 16-byte aligned (ld multiple of 8).
// `status` is a device int the kernel writes a non-zero code to if a bounded wait ran out.
// variant: 0 = choose (choose_variant), 1 or 10 .. 13 = 128x64 tiles on one CTA or a cluster of 2, 4, 8 CTAs, 2 = CTA pairs with 64-wide K stages (K-major only),
// 3 = CTA pairs with 128-wide K stages (6 = the same, the tiles of a part-filled last wave divided; needs `space`), 4 / 5 = clusters of two / four pairs that split the contraction of a tile.
static int launch_gemm_impl(const void* a, const void* b, void* c, const void* residual, int M, int N, int K, int64_t lda,
                            int64_t ldb, int64_t ldc, int64_t ldr, int epilogue, int a_mn, int b_mn, int* status, int variant,
                            const void* stats_targets, int64_t stats_ldt, int stats_t_rows, int stats_shift, float* stats_partial,
                            const tc::Grouping* grp, cudaStream_t stream, const tc::Scatter* scatter = nullptr, void* gated_h = nullptr,
                            int64_t gated_ldh = 0, const BatchSpec* batched = nullptr, const PartsSpec* parts = nullptr, const int* live = nullptr, SplitSpace* space = nullptr) {
  using namespace tc;
  static const BatchSpec one{};
  const BatchSpec& bs = batched != nullptr ? *batched : one;
  const bool symmetric = bs.symmetric && M == N;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((lda & 7) || (ldb & 7) || (reinterpret_cast<uintptr_t>(a) & 15) || (reinterpret_cast<uintptr_t>(b) & 15)) return -1;
  constexpr int smem_pair = P_RING_BYTES + P_STAGE_OUT_BYTES + 1024, smem_small = S_STAGES * S_STAGE_BYTES + S_RECV_BYTES + 1024;
  static PerDeviceOnce configured;
  if (configured.needed()) {
    bool ok = allow_smem(gemm_tn_2cta_kernel<1>, smem_pair) && allow_smem(gemm_tn_2cta_kernel<2>, smem_pair) &&
              allow_smem(gemm_tn_2cta_kernel<2, false, true>, smem_pair) && allow_smem(gemm_tn_2cta_kernel<2, true, false>, smem_pair) &&
              allow_smem(gemm_tn_2cta_kernel<2, true, true>, smem_pair) && allow_smem(gemm_tn_2cta_kernel<2, true, true, true>, smem_pair);
    ok = ok && allow_smem(gemm_tn_2cta_kernel<2, false, false, false, true>, smem_pair) && allow_smem(gemm_tn_2cta_kernel<2, false, true, false, true>, smem_pair) &&
         allow_smem(gemm_tn_2cta_kernel<2, true, false, false, true>, smem_pair) && allow_smem(gemm_tn_2cta_kernel<2, true, true, false, true>, smem_pair);
    ok = ok && allow_smem(gemm_split_kernel<2, false, false>, smem_pair) && allow_smem(gemm_split_kernel<2, false, true>, smem_pair) &&
         allow_smem(gemm_split_kernel<2, true, false>, smem_pair) && allow_smem(gemm_split_kernel<2, true, true>, smem_pair);
    ok = ok && allow_smem(gemm_split_kernel<4, false, false>, smem_pair) && allow_smem(gemm_split_kernel<4, false, true>, smem_pair) &&
         allow_smem(gemm_split_kernel<4, true, false>, smem_pair) && allow_smem(gemm_split_kernel<4, true, true>, smem_pair);
    ok = ok && allow_smem(gemm_small_kernel<false, false>, smem_small) && allow_smem(gemm_small_kernel<false, true>, smem_small) &&
         allow_smem(gemm_small_kernel<true, false>, smem_small) && allow_smem(gemm_small_kernel<true, true>, smem_small);
    if (!ok) return -2;
    configured.mark();
  }
  const bool mn = a_mn || b_mn;
  const bool plain = stats_targets == nullptr && grp == nullptr && scatter == nullptr && epilogue != kSwiGLU;
  if (variant == 0) variant = plain ? choose_variant(M, N, K, bs.batch, symmetric, space != nullptr) : kPair;
  if (variant == 1) variant = kSmall;
  if (variant < kPairK64 || variant > kSmall8 || (variant > kPairDivided && variant < kSmall)) return -4;
  if (variant == kPairK64 && mn) return -4;
  if (variant > kPair && !plain) return -4;
  // How many rows there are is known on the device only: it decides whether there is anything to divide
  const bool divide = variant == kPairDivided || (variant == kPair && plain && live != nullptr && !(a_mn && b_mn));
  if (variant == kPairDivided) variant = kPair;
  const bool pairs = variant < kSmall;
  CUtensorMap map_a, map_b;
  constexpr int mn_rows = 2 * BK;  // contraction rows of a transposed operand's box
  int rc = a_mn ? make_map_bf16_stack(&map_a, a, K, M, lda, mn_rows, bs.batch, bs.a_stride) : make_map_bf16_stack(&map_a, a, M, K, lda, BM, bs.batch, bs.a_stride);
  if (rc) return rc;
  // grouped by rows: B is the stack of the experts' matrices
  const int64_t b_stack = (grp != nullptr && grp->mode == kGroupRows) ? grp->num_groups : 1;
  rc = b_mn ? make_map_bf16_stack(&map_b, b, b_stack * K, N, ldb, mn_rows, bs.batch, bs.b_stride)
            : make_map_bf16_stack(&map_b, b, b_stack * N, K, ldb, pairs ? P_HALF : S_TILE_N, bs.batch, bs.b_stride);
  if (rc) return rc;
  Params p{(__nv_bfloat16*)c, (const __nv_bfloat16*)residual, M, N, K, ldc, ldr, epilogue, status, RowStatsOut{nullptr, 0, 0, 0, nullptr},
           Grouping{kGroupNone, 0, nullptr, nullptr}, Scatter{}, (__nv_bfloat16*)gated_h, gated_ldh, 0, bs.alpha, bs.beta, bs.diagonal, bs.once ? 1 : 0, bs.batch,
           bs.c_stride, bs.r_stride, 0, live, nullptr, nullptr};
  if (live != nullptr && (grp != nullptr || scatter != nullptr || stats_targets != nullptr || bs.batch != 1 || (a_mn && !b_mn))) return -10;
  if (epilogue == kSwiGLU) {
    if (!pairs || a_mn || b_mn || (grp != nullptr && grp->mode != kGroupRows) || stats_targets != nullptr || scatter != nullptr || gated_h == nullptr || (N & 255) || (ldc & 7) ||
        (gated_ldh & 7) || (reinterpret_cast<uintptr_t>(c) & 15) || (reinterpret_cast<uintptr_t>(gated_h) & 15))
      return -8;
  }
  if (scatter != nullptr) {
    if (!pairs || grp != nullptr || stats_targets != nullptr || epilogue != kStore || scatter->world < 1 || scatter->world > kMaxScatterRanks ||
        scatter->cols * scatter->world != N || (scatter->cols & 255))
      return -7;
    p.sc = *scatter;
    p.c = scatter->stage[scatter->rank];  // alignment checks of the store path look at c / ldc
    p.ldc = scatter->cols;
    for (int q = 0; q < scatter->world; ++q)
      if (reinterpret_cast<uintptr_t>(scatter->stage[q]) & 31) return -7;
  }
  if (grp != nullptr) {
    if (variant != kPair || stats_targets != nullptr || residual != nullptr) return -6;
    if (grp->mode == kGroupRows && (a_mn || (K & 127) || (N & 255))) return -6;  // experts' matrices must not share a box
    if (grp->mode == kGroupK && !(a_mn && b_mn)) return -6;
    p.grp = *grp;
  }
  if (stats_targets != nullptr) {
    if (!pairs || a_mn || b_mn || epilogue != kStore || (N & 7) || (ldc & 7) || (stats_ldt & 7) || (reinterpret_cast<uintptr_t>(c) & 15) ||
        (reinterpret_cast<uintptr_t>(stats_targets) & 15))
      return -5;
    p.rs = RowStatsOut{(const __nv_bfloat16*)stats_targets, stats_ldt, stats_t_rows, stats_shift, stats_partial};
  }
  // Stores through staging: C must be a matrix that TMA can address, and a warp's 32 rows must not straddle an expert.
  CUtensorMap map_c = map_a, map_h = map_a;
  const bool reads_ok = epilogue != kAddResidual || ((ldr & 7) == 0 && (reinterpret_cast<uintptr_t>(residual) & 15) == 0);
  if (scatter == nullptr && stats_targets == nullptr && (N & 7) == 0 && (ldc & 7) == 0 && (reinterpret_cast<uintptr_t>(c) & 15) == 0 && reads_ok &&
      (grp == nullptr || grp->mode == kGroupRows || (M & 127) == 0)) {
    const int64_t rows = grp != nullptr && grp->mode == kGroupK ? (int64_t)grp->num_groups * M : M;
    rc = make_map_bf16_stack(&map_c, c, rows, N, ldc, 32, bs.batch, bs.c_stride);
    if (rc == 0 && epilogue == kSwiGLU) rc = make_map_bf16_stack(&map_h, gated_h, M, N / 2, gated_ldh, 32, 1, 0);
    if (rc == 0 && symmetric && variant == kPair) {  // transposed stores: 64 rows of 32 elements
      rc = make_map_bf16_stack(&map_h, c, M, N, ldc, 64, bs.batch, bs.c_stride, 32);
      p.symmetric = 1;
    }
    if (rc) return rc;
    p.staged = 1;
  }
  MoreParts more{};
  if (parts != nullptr) {
    if (!a_mn || !b_mn || variant != kPair || bs.batch != 1 || parts->n > kMoreParts) return -9;
    more.n = parts->n;
    for (int i = 0; i < parts->n; ++i) {
      if ((parts->lda[i] & 7) || (parts->ldb[i] & 7) || (reinterpret_cast<uintptr_t>(parts->a[i]) & 15) || (reinterpret_cast<uintptr_t>(parts->b[i]) & 15)) return -1;
      rc = make_map_bf16_stack(&more.a[i], parts->a[i], parts->K[i], M, parts->lda[i], mn_rows, 1, 0);
      if (rc == 0) rc = make_map_bf16_stack(&more.b[i], parts->b[i], parts->K[i], N, parts->ldb[i], mn_rows, 1, 0);
      if (rc) return rc;
      more.rows[i] = parts->K[i];
      more.seg[i] = parts->seg[i];
      more.live[i] = parts->live[i];
    }
  }
  const int pair_tiles = (int)pair_tile_count(M, N, bs.batch, p.symmetric);
  if (divide && space != nullptr && parts == nullptr &&
      may_split(M, N, K, bs.batch, p.symmetric, live != nullptr && !(a_mn && b_mn)) && space->get(reinterpret_cast<float**>(&p.partial), &p.sync)) {
    if (p.sync == nullptr || p.partial == nullptr) return -11;
  }
  count_launch(1);
  if (variant >= kSmall && variant <= kSmall8) {
    const int log_splits = variant - kSmall;
    const int tiles = ((M + BM - 1) / BM) * ((N + S_TILE_N - 1) / S_TILE_N) * bs.batch;
    if (launch_small(a_mn, b_mn, tiles, log_splits, smem_small, stream, map_a, map_b, map_c, p) != cudaSuccess) return -3;
  } else if (variant == kSplit2) {
    launch_split<2>(a_mn, b_mn, pair_tiles, smem_pair, stream, map_a, map_b, p);
  } else if (variant == kSplit4) {
    launch_split<4>(a_mn, b_mn, pair_tiles, smem_pair, stream, map_a, map_b, p);
  } else {
    // grouped: the number of tiles is known on the device only; every pair looks for work
    const int tiles = grp != nullptr || p.sync != nullptr ? kMaxPairs : pair_tiles;  // (divided tiles occupy every pair)
    const int grid = 2 * (tiles < kMaxPairs ? tiles : kMaxPairs);
    if (more.n > 0) launch_pdl(gemm_tn_2cta_kernel<2, true, true, true>, grid, P_THREADS, smem_pair, stream, map_a, map_b, map_c, map_h, p, more);
    else if (p.sync != nullptr && a_mn && b_mn) launch_pdl(gemm_tn_2cta_kernel<2, true, true, false, true>, grid, P_THREADS, smem_pair, stream, map_a, map_b, map_c, map_h, p, NoParts{});
    else if (p.sync != nullptr && a_mn) launch_pdl(gemm_tn_2cta_kernel<2, true, false, false, true>, grid, P_THREADS, smem_pair, stream, map_a, map_b, map_c, map_h, p, NoParts{});
    else if (p.sync != nullptr && b_mn) launch_pdl(gemm_tn_2cta_kernel<2, false, true, false, true>, grid, P_THREADS, smem_pair, stream, map_a, map_b, map_c, map_h, p, NoParts{});
    else if (p.sync != nullptr) launch_pdl(gemm_tn_2cta_kernel<2, false, false, false, true>, grid, P_THREADS, smem_pair, stream, map_a, map_b, map_c, map_h, p, NoParts{});
    else if (a_mn && b_mn) launch_pdl(gemm_tn_2cta_kernel<2, true, true>, grid, P_THREADS, smem_pair, stream, map_a, map_b, map_c, map_h, p, NoParts{});
    else if (a_mn) launch_pdl(gemm_tn_2cta_kernel<2, true, false>, grid, P_THREADS, smem_pair, stream, map_a, map_b, map_c, map_h, p, NoParts{});
    else if (b_mn) launch_pdl(gemm_tn_2cta_kernel<2, false, true>, grid, P_THREADS, smem_pair, stream, map_a, map_b, map_c, map_h, p, NoParts{});
    else if (variant == kPair) launch_pdl(gemm_tn_2cta_kernel<2>, grid, P_THREADS, smem_pair, stream, map_a, map_b, map_c, map_h, p, NoParts{});
    else launch_pdl(gemm_tn_2cta_kernel<1>, grid, P_THREADS, smem_pair, stream, map_a, map_b, map_c, map_h, p, NoParts{});
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

int launch_gemm_tcgen05(const void* a, const void* b, void* c, const void* residual, int M, int N, int K, int64_t lda,
                        int64_t ldb, int64_t ldc, int64_t ldr, int epilogue, int a_mn, int b_mn, int* status, int variant, const int* live,
                        SplitSpace* space, cudaStream_t stream) {
  return launch_gemm_impl(a, b, c, residual, M, N, K, lda, ldb, ldc, ldr, epilogue, a_mn, b_mn, status, variant, nullptr, 0, 0, 0, nullptr, nullptr, stream,
                          nullptr, nullptr, 0, nullptr, nullptr, live, space);
}

int launch_gemm_tn_tcgen05(const void* a, const void* b, void* c, const void* residual, int M, int N, int K, int64_t lda,
                           int64_t ldb, int64_t ldc, int64_t ldr, int epilogue, int* status, int variant, const int* live, SplitSpace* space,
                           cudaStream_t stream) {
  return launch_gemm_tcgen05(a, b, c, residual, M, N, K, lda, ldb, ldc, ldr, epilogue, 0, 0, status, variant, live, space, stream);
}

// c[M, N] (+)= sum_i a_i[K_i, M]^T . b_i[K_i, N]: one launch where pair tiles are the form for the whole contraction, else one each
// (small products are not bound by their epilogue, and have better forms).
int launch_gemm_parts(int n, const void* const* a, const void* const* b, const int* K, const int64_t* lda, const int64_t* ldb, const int* const* live,
                      void* c, int M, int N, int64_t ldc, int accumulate, int* status, SplitSpace* space, cudaStream_t stream) {
  if (n < 1 || n > tc::kMoreParts + 1) return -9;
  int total = 0;
  PartsSpec parts;
  for (int i = 0; i < n; ++i) {
    if (K[i] <= 0) return -9;
    total += (K[i] + 127) / 128 * 128;
    if (i == 0) continue;
    parts.a[i - 1] = a[i];
    parts.b[i - 1] = b[i];
    parts.K[i - 1] = K[i];
    parts.lda[i - 1] = lda[i];
    parts.ldb[i - 1] = ldb[i];
    parts.seg[i - 1] = nullptr;
    parts.live[i - 1] = live[i];
  }
  parts.n = n - 1;
  if (n > 1 && choose_variant(M, N, total, 1, 0, false) == kPair)
    return launch_gemm_impl(a[0], b[0], c, nullptr, M, N, K[0], lda[0], ldb[0], ldc, 0, accumulate ? 1 : 0, 1, 1, status, kPair, nullptr, 0, 0, 0, nullptr,
                            nullptr, stream, nullptr, nullptr, 0, nullptr, &parts, live[0]);
  for (int i = 0; i < n; ++i) {
    const int rc = launch_gemm_impl(a[i], b[i], c, nullptr, M, N, K[i], lda[i], ldb[i], ldc, 0, accumulate || i > 0 ? 1 : 0, 1, 1, status, 0, nullptr, 0, 0, 0,
                                    nullptr, nullptr, stream, nullptr, nullptr, 0, nullptr, nullptr, live[i], space);
    if (rc) return rc;
  }
  return 0;
}

// ---- stacks of products (Newton-Schulz iterations of equally shaped matrices) ----------------------
// c[z] = alpha * op(a[z]) * op(b[z])^T (+ beta * addend[z]), rounded as in Params; with `once` (+ diagonal * I) and rounded once.
// All stacks dense: [batch, rows, cols].  `symmetric`: the caller knows that the product is (a Gram matrix, a power of a
// symmetric matrix): only tiles on and above the diagonal are computed.
int launch_gemm_stack(const void* a, const void* b, void* c, const void* addend, int batch, int M, int N, int K, int a_mn, int b_mn, float alpha,
                      float beta, int once, float diagonal, int symmetric, int* status, SplitSpace* space, cudaStream_t stream) {
  BatchSpec bs;
  bs.batch = batch;
  bs.a_stride = (int64_t)M * K;
  bs.b_stride = (int64_t)N * K;
  bs.c_stride = bs.r_stride = (int64_t)M * N;
  bs.alpha = alpha;
  bs.beta = beta;
  bs.diagonal = diagonal;
  bs.once = once != 0;
  bs.symmetric = symmetric != 0;
  return launch_gemm_impl(a, b, c, addend, M, N, K, a_mn ? M : K, b_mn ? N : K, N, N, addend != nullptr ? tc::kAddResidual : tc::kStore, a_mn, b_mn, status, 0,
                          nullptr, 0, 0, 0, nullptr, nullptr, stream, nullptr, nullptr, 0, &bs, nullptr, nullptr, space);
}

// ---- row-parallel product with the reduce-scatter's transfer in the epilogue -----------------
// partial[M, N] = a[M, K] . b[N, K]^T, tile columns stored into slot `rank` of their owner's staging
// area stage[owner] = [world][M][N / world] (addresses valid on this device: peer-mapped for the
// other ranks).  N / world must be a multiple of 256.
int launch_gemm_scatter(const void* a, const void* b, void* const* stage, int world, int rank, int M, int N, int K, int64_t lda, int64_t ldb,
                        int* status, cudaStream_t stream) {
  if (world < 1 || world > tc::kMaxScatterRanks || rank < 0 || rank >= world || N % world) return -7;
  tc::Scatter sc{world, rank, N / world, {}};
  for (int q = 0; q < world; ++q) sc.stage[q] = static_cast<__nv_bfloat16*>(stage[q]);
  return launch_gemm_impl(a, b, stage[rank], nullptr, M, N, K, lda, ldb, N / world, 0, tc::kStore, 0, 0, status, 3, nullptr, 0, 0, 0, nullptr, nullptr,
                          stream, &sc);
}

// ---- gate | up product of a gated MLP with the activation in the epilogue ---------------------
// gate_up[M, 2 I] = x[M, K] . w[2 I, K]^T (gate rows first) and h[M, I] = silu(gate) * up.  I % 128 == 0.
int launch_gemm_swiglu(const void* x, const void* w, void* gate_up, void* h, int M, int I, int K, int64_t ldx, int64_t ldw, int64_t ldc, int64_t ldh,
                       int* status, const int* live, cudaStream_t stream) {
  return launch_gemm_impl(x, w, gate_up, nullptr, M, 2 * I, K, ldx, ldw, ldc, 0, tc::kSwiGLU, 0, 0, status, 3, nullptr, 0, 0, 0, nullptr, nullptr, stream,
                          nullptr, h, ldh, nullptr, nullptr, live);
}

// ---- grouped products for mixture-of-experts layers -----------------------------------------
// counts[e] rows belong to expert e.  seg[e] = offset of its (128-row aligned) segment in the padded
// row order, mtile_start[e] = prefix sum of ceil(segment rows / 256).  One block; E <= 4096.
__global__ void moe_group_plan_kernel(const int* __restrict__ counts, int num_groups, int* __restrict__ seg, int* __restrict__ mtile_start) {
  pdl_begin();
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  int off = 0, tiles = 0;
  for (int e = 0; e < num_groups; ++e) {
    seg[e] = off;
    mtile_start[e] = tiles;
    const int padded = (counts[e] + 127) & ~127;
    off += padded;
    tiles += (padded + 255) >> 8;
  }
  seg[num_groups] = off;
  mtile_start[num_groups] = tiles;
}

void launch_moe_group_plan(const int* counts, int num_groups, int* seg, int* mtile_start, cudaStream_t stream) {
  count_launch(1);
  launch_pdl(moe_group_plan_kernel, 1, 32, 0, stream, counts, num_groups, seg, mtile_start);
}

// mode 1 (rows grouped): c[R, N] = a[R, K] . b_e^T, b the stack [E, N, K] (b_mn 0) or, for the input
//   gradient, c[R, N] = a[R, K] . b_e with b = [E, K, N] (b_mn 1).  R = rows of the padded order.
// mode 2 (contraction grouped): c_e[M, N] (=, +=) a[seg_e, M]^T . b[seg_e, N], c the stack [E, M, N]; K = R.
int launch_gemm_grouped(const void* a, const void* b, void* c, int M, int N, int K, int64_t lda, int64_t ldb, int64_t ldc, int epilogue,
                        int mode, int b_mn, const int* seg, const int* mtile_start, int num_groups, int* status, cudaStream_t stream) {
  if (mode != tc::kGroupRows && mode != tc::kGroupK) return -6;
  const tc::Grouping grp{mode, num_groups, seg, mtile_start};
  const int a_mn = mode == tc::kGroupK ? 1 : 0;
  return launch_gemm_impl(a, b, c, nullptr, M, N, K, lda, ldb, ldc, 0, epilogue, a_mn, mode == tc::kGroupK ? 1 : b_mn, status, 3, nullptr, 0, 0, 0,
                          nullptr, &grp, stream);
}

// mode 2 over several uses, each with its own operands and segments: c_e (+)= sum_i a_i[seg_i,e, M]^T . b_i[seg_i,e, N]
int launch_gemm_grouped_parts(int n, const void* const* a, const void* const* b, const int* K, const int64_t* lda, const int64_t* ldb, const int* const* seg,
                              void* c, int M, int N, int accumulate, const int* mtile_start, int num_groups, int* status, cudaStream_t stream) {
  if (n < 1 || n > tc::kMoreParts + 1) return -9;
  PartsSpec parts;
  parts.n = n - 1;
  for (int i = 1; i < n; ++i) {
    parts.a[i - 1] = a[i];
    parts.b[i - 1] = b[i];
    parts.K[i - 1] = K[i];
    parts.lda[i - 1] = lda[i];
    parts.ldb[i - 1] = ldb[i];
    parts.seg[i - 1] = seg[i];
    parts.live[i - 1] = nullptr;
  }
  const tc::Grouping grp{tc::kGroupK, num_groups, seg[0], mtile_start};
  return launch_gemm_impl(a[0], b[0], c, nullptr, M, N, K[0], lda[0], ldb[0], N, 0, accumulate ? 1 : 0, 1, 1, status, kPair, nullptr, 0, 0, 0, nullptr, &grp,
                          stream, nullptr, nullptr, 0, nullptr, n > 1 ? &parts : nullptr);
}

// mode 1 with stacked [gate; up] experts [E, 2 I, K]: gate_up[R, 2 I] and h[R, I] = silu(gate) * up.
int launch_gemm_grouped_swiglu(const void* a, const void* b, void* gate_up, void* h, int M, int I, int K, int64_t lda, int64_t ldb, const int* seg,
                               const int* mtile_start, int num_groups, int* status, cudaStream_t stream) {
  const tc::Grouping grp{tc::kGroupRows, num_groups, seg, mtile_start};
  return launch_gemm_impl(a, b, gate_up, nullptr, M, 2 * I, K, lda, ldb, 2 * I, 0, tc::kSwiGLU, 0, 0, status, 3, nullptr, 0, 0, 0, nullptr, &grp, stream,
                          nullptr, h, I);
}

// ---- lm_head product fused with the row loss (KL divergence / cross-entropy on the argmax) -----
int lmhead_stat_words() { return tc::kStatWords; }
// records per logits row: two per 256-column tile (one per 128-column epilogue half)
int lmhead_tiles_n(int N) { return 2 * ((N + tc::P_TILE_N - 1) / tc::P_TILE_N); }

// logits[M,N] = x[M,K] * w[N,K]^T (stored, bf16) and, per (row, 256-column tile), the statistics of the logits
// row and of targets[row + shift] over those columns into partial[M, tiles_n, kStatWords].
int launch_lmhead_logits_stats(const void* x, const void* w, void* logits, const void* targets, int M, int N, int K, int64_t ldx,
                               int64_t ldw, int64_t ldc, int64_t ldt, int t_rows, int shift, float* partial, int* status,
                               cudaStream_t stream) {
  return launch_gemm_impl(x, w, logits, nullptr, M, N, K, ldx, ldw, ldc, 0, tc::kStore, 0, 0, status, 3, targets, ldt, t_rows, shift, partial, nullptr, stream);
}

// One warp per row: merge the row's tile records and write what the row-loss forward kernel writes
// (loss, the five saved statistics, both argmaxes); rows with active[r] == 0 get the same sentinels.
// op: 0 = KL(target || draft), 3 = cross-entropy against the target row's argmax.
__global__ void __launch_bounds__(128)
lmhead_combine_kernel(const float* __restrict__ partial, const __nv_bfloat16* __restrict__ logits, const uint8_t* __restrict__ active,
                      float* __restrict__ loss, float* __restrict__ stats, int* __restrict__ argmax_d, int* __restrict__ argmax_t,
                      int rows, int tiles_n, int64_t ld_logits, int op) {
  pdl_begin();
  const int r = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= rows) return;
  float* st = stats + r;
  if (active && !active[r]) {
    if (lane == 0) {
      loss[r] = 0.f;
      for (int k = 0; k < 5; ++k) st[(int64_t)k * rows] = 0.f;
      if (argmax_d) argmax_d[r] = -1;
      if (argmax_t) argmax_t[r] = -2;
    }
    return;
  }
  RowStats sd{-INFINITY, 0.f, -INFINITY, 0x7fffffff}, stt{-INFINITY, 0.f, -INFINITY, 0x7fffffff};
  float A = 0.f;
  for (int t = lane; t < tiles_n; t += 32) {
    const float4* rec = reinterpret_cast<const float4*>(partial + ((int64_t)r * tiles_n + t) * tc::kStatWords);
    const float4 a = rec[0], b = rec[1], c = rec[2];
    merge_stats(sd, RowStats{a.x, a.y, a.z, __float_as_int(a.w)});
    merge_stats_kl(stt, A, RowStats{b.x, b.y, b.w, __float_as_int(c.x)}, b.z);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    RowStats od{__shfl_xor_sync(0xffffffffu, sd.m, o), __shfl_xor_sync(0xffffffffu, sd.z, o), __shfl_xor_sync(0xffffffffu, sd.best, o),
                __shfl_xor_sync(0xffffffffu, sd.best_idx, o)};
    RowStats ot{__shfl_xor_sync(0xffffffffu, stt.m, o), __shfl_xor_sync(0xffffffffu, stt.z, o), __shfl_xor_sync(0xffffffffu, stt.best, o),
                __shfl_xor_sync(0xffffffffu, stt.best_idx, o)};
    const float oA = __shfl_xor_sync(0xffffffffu, A, o);
    merge_stats(sd, od);
    merge_stats_kl(stt, A, ot, oA);
  }
  if (lane == 0) {
    const float lse_d = sd.m + __logf(sd.z), lse_t = stt.m + __logf(stt.z);
    float L, extra;
    if (op == 3) {
      L = lse_d - __bfloat162float(logits[(int64_t)r * ld_logits + stt.best_idx]);
      extra = (float)stt.best_idx;
    } else {
      L = A / stt.z + lse_d - lse_t;
      extra = L;
    }
    loss[r] = L;
    st[0] = sd.m;
    st[(int64_t)rows] = sd.z;
    st[(int64_t)2 * rows] = stt.m;
    st[(int64_t)3 * rows] = stt.z;
    st[(int64_t)4 * rows] = extra;
    if (argmax_d) argmax_d[r] = sd.best_idx;
    if (argmax_t) argmax_t[r] = stt.best_idx;
  }
}

int launch_lmhead_combine(const float* partial, const void* logits, const uint8_t* active, float* loss, float* stats, int* argmax_d,
                          int* argmax_t, int rows, int tiles_n, int64_t ld_logits, int op, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (op != 0 && op != 3) return -1;
  count_launch(1);
  launch_pdl(lmhead_combine_kernel, (rows + 3) / 4, 128, 0, stream, partial, (const __nv_bfloat16*)logits, active, loss, stats, argmax_d, argmax_t, rows,
                                                          tiles_n, ld_logits, op);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace sb200
