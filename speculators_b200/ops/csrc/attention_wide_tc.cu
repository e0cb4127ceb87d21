// Masked attention at head dim 256 on the 5th-generation tensor cores: forward, dQ, dK and dV, one kernel template.
//
// All four products have the same shape.  128 rows (queries for the output and dQ, keys for dK and dV) stay in shared
// memory while tiles of 64 rows of the other side stream past, and one 128 x 256 accumulator fills half of the tensor
// memory:
//
//              resident R0  R1     streamed X0  X1    score tile          factor F in bf16       accumulator +=
//     forward           Q   -               K   V     S = Q K^T           online softmax of S    F V
//     dQ                Q   dO              K   V     S, dP = dO V^T      P (dP - delta)         F K
//     dK                K   V               Q   dO    S^T, dP^T           P^T (dP^T - delta)     F Q
//     dV                K   -               Q   dO    S^T                 P^T                    F dO
//
// A CTA that accumulated dK and dV together would need all 512 tensor memory columns for them and have none left for
// the scores, so the two are separate launches that recompute S^T: five products instead of four, against six if each
// CTA took half of the columns of both (and against the mma.sync kernels, which do exactly that).  Tiles of 64 streamed
// rows are what shared memory leaves room for beside 128 resident rows of one or two operands (64 KB each).
//
// Roles as in the narrower kernels: warp 0 loads by TMA, one thread of warp 1 issues the products, warps 2-9 do the
// element-wise work, two threads per TMEM lane with 32 of the 64 columns each.  Scores are double-buffered, so the
// products of tile t + 1 run during the element-wise work of tile t; F overwrites the first 16 of a thread's own 32
// score columns (bf16 pairs), from where the next product takes it as its A operand.
//
// The streamed tile's 64 columns bound the score products: their A operand is read from shared memory for only 64
// columns of results (6 KB per 32 cycles of work at 128 bytes per cycle), two thirds of the tensor rate at best.
// 16 query heads on 2 KV heads, one causal document, against the mma.sync kernels: 4096 tokens forward 674 -> 146 us
// (939 TFLOP/s), backward 2750 -> 744 us (462 TFLOP/s of the four products that are needed); 512 tokens 31 -> 20 and
// 103 -> 90 us.
//
// All waits are bounded: an expired one records a code in the status word, the element-wise threads keep walking their
// loops without waiting (no partner is left alone at a named barrier) and store nothing.
#include "attention_params.h"
#include "tcgen05_utils.cuh"

namespace sb200 {
namespace awtc {

using namespace tc;

enum Mode : int { kFwd = 0, kDq = 1, kDk = 2, kDv = 3 };
enum Status : int { kTimeoutProducer = 51, kTimeoutMma = 52, kTimeoutCompute = 53 };

constexpr int HD = 256, BM = 128, BX = 64, THREADS = 320;
constexpr int R_SUB = BM * 128, R_BYTES = 4 * R_SUB;  // [128 x 64] sub-tiles of a resident operand
constexpr int X_SUB = BX * 128, X_BYTES = 4 * X_SUB;  // [64 x 64] sub-tiles of a streamed one
constexpr uint32_t TMEM_COLS = 512;
constexpr uint32_t COL_S = 0, COL_DP = 128, COL_ACC = 256;  // S, dP: two buffers of 64 columns each
constexpr float kLog2e = 1.4426950408889634f;

template <int MODE> constexpr bool kDual = MODE == kDq || MODE == kDk;  // two resident operands, dP wanted
template <int MODE> constexpr bool kQueriesResident = MODE == kFwd || MODE == kDq;
template <int MODE> constexpr int kX1Stages = kDual<MODE> ? 1 : 2;  // X1 of a dual product is free again after dP
template <int MODE> constexpr int kSmem = (kDual<MODE> ? 2 : 1) * R_BYTES + (2 + kX1Stages<MODE>) * X_BYTES + 1024;

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 h2 = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h2);
}

template <int MODE>
__global__ void __launch_bounds__(THREADS, 1)
wide_kernel(const __grid_constant__ CUtensorMap map_r0, const __grid_constant__ CUtensorMap map_r1, const __grid_constant__ CUtensorMap map_x0,
            const __grid_constant__ CUtensorMap map_x1, const AttnParams p, int n_range_tiles, int* status) {
  constexpr bool DUAL = kDual<MODE>, QRES = kQueriesResident<MODE>;
  constexpr int NX1 = kX1Stages<MODE>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* r0_s = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* r1_s = r0_s + R_BYTES;
  unsigned char* x0_s = r0_s + (DUAL ? 2 : 1) * R_BYTES;  // 2 stages
  unsigned char* x1_s = x0_s + 2 * X_BYTES;               // NX1 stages
  __shared__ __align__(8) uint64_t bar_r, bar_x0_full[2], bar_x0_empty[2], bar_x1_full[2], bar_x1_empty[2], bar_s_full[2], bar_f_ready, bar_acc, bar_end;
  __shared__ uint32_t tmem_base_slot;
  __shared__ int s_range[2];
  __shared__ float s_xchg[MODE == kFwd ? 2 : 1][2][MODE == kFwd ? BM : 1];  // forward: what the two threads of a row hand each other
  __shared__ __align__(16) float st_lse[2][QRES ? 4 : BX], st_delta[2][QRES ? 4 : BX];  // dK / dV: statistics of the streamed queries
  __shared__ __align__(16) uint16_t st_iv[2][QRES ? 8 : BX];  // first | one-past-last resident row that the query sees, a byte each

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the tile with the most work under a causal mask first: the last queries, the first keys
  const int tile = QRES ? gridDim.y - 1 - blockIdx.y : blockIdx.y, h = blockIdx.x;
  const int group = p.nh / p.nkv, kvh = h / group;
  const int row0 = tile * BM;

  if (threadIdx.x == 0) {
    mbar_init(smem_addr(&bar_r), 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_addr(&bar_x0_full[s]), 1);
      mbar_init(smem_addr(&bar_x0_empty[s]), 1);
      mbar_init(smem_addr(&bar_x1_full[s]), 1);
      mbar_init(smem_addr(&bar_x1_empty[s]), 1);
      mbar_init(smem_addr(&bar_s_full[s]), 1);
    }
    mbar_init(smem_addr(&bar_f_ready), 8);  // one arrival per element-wise warp
    mbar_init(smem_addr(&bar_acc), 1);
    mbar_init(smem_addr(&bar_end), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_range[0] = 0x7fffffff;
    s_range[1] = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base_slot)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem_base = tmem_base_slot;
  pdl_begin();

  // streamed rows that the resident ones see
  int lo_all = 0x7fffffff, hi_all = 0;
  if (QRES) {
    if (threadIdx.x < BM && row0 + threadIdx.x < p.Tq) {
      const int l = p.lo[row0 + threadIdx.x], u = min(p.hi[row0 + threadIdx.x], p.Tc);
      if (l >= 0 && u > l) {
        lo_all = l;
        hi_all = u;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo_all = min(lo_all, __shfl_xor_sync(0xffffffffu, lo_all, o));
      hi_all = max(hi_all, __shfl_xor_sync(0xffffffffu, hi_all, o));
    }
    if (lane == 0) {
      atomicMin(&s_range[0], lo_all);
      atomicMax(&s_range[1], hi_all);
    }
    __syncthreads();
    lo_all = s_range[0];
    hi_all = s_range[1];
  } else {  // query ranges are kept per 64 keys
    for (int s = tile * (BM / kAttnKeyTile); s < min((tile + 1) * (BM / kAttnKeyTile), n_range_tiles); ++s) {
      lo_all = min(lo_all, p.tile_qmin[s]);
      hi_all = max(hi_all, p.tile_qmax[s]);
    }
  }
  const int j0 = hi_all > lo_all ? lo_all / BX : 0;
  const int n_tiles = hi_all > lo_all ? (hi_all + BX - 1) / BX - j0 : 0;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (n_tiles > 0 && elect_one()) {
      const int rcol = (QRES ? h : kvh) * HD, xcol = (QRES ? kvh : h) * HD;
      const uint32_t rb = smem_addr(&bar_r);
      mbar_expect_tx(rb, (DUAL ? 2 : 1) * R_BYTES);
#pragma unroll
      for (int c = 0; c < 4; ++c) tma_load_2d(smem_addr(r0_s) + c * R_SUB, &map_r0, rb, rcol + c * 64, row0);
      if (DUAL) {
#pragma unroll
        for (int c = 0; c < 4; ++c) tma_load_2d(smem_addr(r1_s) + c * R_SUB, &map_r1, rb, rcol + c * 64, row0);
      }
      auto load = [&](const CUtensorMap* map, unsigned char* dst, uint64_t* full, uint64_t* empty, int st, int round, int t) {
        if (!mbar_wait(smem_addr(&empty[st]), (round & 1) ^ 1, status, kTimeoutProducer)) return false;
        const uint32_t bar = smem_addr(&full[st]), d = smem_addr(dst + st * X_BYTES);
        mbar_expect_tx(bar, X_BYTES);
#pragma unroll
        for (int c = 0; c < 4; ++c) tma_load_2d(d + c * X_SUB, map, bar, xcol + c * 64, (j0 + t) * BX);
        return true;
      };
      // the operand that is released first goes first: dP of tile t - 1 precedes the accumulation of tile t - 2 in a
      // dual product, otherwise S of tile t - 2 precedes its accumulation
      for (int t = 0; t < n_tiles; ++t) {
        if (DUAL && !load(&map_x1, x1_s, bar_x1_full, bar_x1_empty, 0, t, t)) break;
        if (!load(&map_x0, x0_s, bar_x0_full, bar_x0_empty, t & 1, t >> 1, t)) break;
        if (!DUAL && !load(&map_x1, x1_s, bar_x1_full, bar_x1_empty, t & 1, t >> 1, t)) break;
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (n_tiles > 0 && elect_one()) {
      constexpr uint32_t idesc_s = instr_desc(BM, BX, false);
      constexpr uint32_t idesc_acc = instr_desc(BM, HD, true);
      auto scores = [&](uint32_t d, unsigned char* r, unsigned char* x) {
        const uint32_t ra = smem_addr(r), xa = smem_addr(x);
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk)
          umma_bf16(d, smem_desc_kmajor_sw128(ra + (kk >> 2) * R_SUB) + 2 * (kk & 3), smem_desc_kmajor_sw128(xa + (kk >> 2) * X_SUB) + 2 * (kk & 3), idesc_s,
                    kk != 0);
      };
      auto issue_scores = [&](int t) -> bool {
        if (!mbar_wait(smem_addr(&bar_x0_full[t & 1]), (t >> 1) & 1, status, kTimeoutMma)) return false;
        if (DUAL && !mbar_wait(smem_addr(&bar_x1_full[0]), t & 1, status, kTimeoutMma)) return false;
        fence_after_sync();
        scores(tmem_base + COL_S + (t & 1) * BX, r0_s, x0_s + (t & 1) * X_BYTES);
        if (DUAL) scores(tmem_base + COL_DP + (t & 1) * BX, r1_s, x1_s);
        umma_commit(smem_addr(&bar_s_full[t & 1]));
        umma_commit(smem_addr(DUAL ? &bar_x1_empty[0] : &bar_x0_empty[t & 1]));
        return true;
      };
      bool ok = mbar_wait(smem_addr(&bar_r), 0, status, kTimeoutMma) && issue_scores(0);
      for (int t = 0; t < n_tiles && ok; ++t) {
        // buffer (t + 1) & 1 held F of tile t - 1, whose product was issued before: products run in order
        if (t + 1 < n_tiles && !(ok = issue_scores(t + 1))) break;
        if (!DUAL && !(ok = mbar_wait(smem_addr(&bar_x1_full[t & 1]), (t >> 1) & 1, status, kTimeoutMma))) break;
        if (!(ok = mbar_wait(smem_addr(&bar_f_ready), t & 1, status, kTimeoutMma))) break;
        fence_after_sync();
        const uint32_t xa = smem_addr((DUAL ? x0_s : x1_s) + (t & 1) * X_BYTES);
        const uint32_t f = tmem_base + COL_S + (t & 1) * BX;
#pragma unroll
        for (int kk = 0; kk < BX / 16; ++kk)  // 16 streamed rows: 8 columns of pairs, in the 32-column block of the thread that wrote them
          umma_bf16_ts(tmem_base + COL_ACC, f + (kk >> 1) * 32 + (kk & 1) * 8, smem_desc_mnmajor_sw128(xa + kk * 2048, X_SUB), idesc_acc, (t | kk) != 0);
        if (MODE == kFwd) umma_commit(smem_addr(&bar_acc));
        umma_commit(smem_addr(DUAL ? &bar_x0_empty[t & 1] : &bar_x1_empty[t & 1]));
        if (t + 1 == n_tiles) umma_commit(smem_addr(&bar_end));
      }
    }
  } else {
    // ------------------------------------------------------------------ element-wise warps
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const int prow = quarter * 32 + lane, row = row0 + prow;
    const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const int colh = half * 32;
    const float sc = p.scale * kLog2e;
    const bool row_ok = row < (QRES ? p.Tq : p.Tc);
    const int lo = QRES && row_ok ? p.lo[row] : 0x7fffffff;
    const int hi = QRES && row_ok ? min(p.hi[row], p.Tc) : 0;
    const float lse = MODE == kDq && row_ok ? p.lse2[(int64_t)h * p.Tq + row] : INFINITY;
    const float delta = MODE == kDq && row_ok ? p.delta[(int64_t)h * p.Tq + row] : 0.f;
    bool ok = true;

    // forward: lazily moved reference maximum in the log2 domain and partial sum, as at head dim 128
    constexpr float kRescaleLog2 = 8.f;
    float m = -INFINITY, l = 0.f;
    int xc = 0;
    auto exchange = [&](float mine) -> float {
      float* slot = &s_xchg[MODE == kFwd ? (xc & 1) : 0][0][0];
      ++xc;
      slot[half * BM + prow] = mine;
      asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory");
      return slot[(half ^ 1) * BM + prow];
    };

    // dK / dV: statistics of 64 streamed queries through registers one tile ahead; two warps load log-sums and
    // deltas, two the intervals
    const int ct = (warp - 2) * 32 + lane;
    float ld_a = 0.f, ld_b = 0.f;
    uint32_t ld_full = 1;
    auto fetch_stats = [&](int t) {
      if (ct >= 2 * BX) return;
      const int r = (j0 + t) * BX + (ct & (BX - 1));
      const bool in = r < p.Tq;
      if (ct < BX) {
        ld_a = in ? p.lse2[(int64_t)h * p.Tq + r] : INFINITY;
        ld_b = in && MODE == kDk ? p.delta[(int64_t)h * p.Tq + r] : 0.f;
      } else {
        const int a = in ? p.lo[r] : 0x7fffffff, b = in ? min(p.hi[r], p.Tc) : 0;
        const int first = min(max(a - row0, 0), BM), end = min(max(b - row0, 0), BM);
        ld_a = __int_as_float(first | end << 8);
        ld_full = first == 0 && end == BM ? 1u : 0u;
      }
    };
    auto stash_stats = [&](int t) {
      if (ct >= 2 * BX) return;
      const int b = t & 1, c = ct & (BX - 1);
      if (ct < BX) {
        st_lse[b][c] = ld_a;
        st_delta[b][c] = ld_b;
      } else {
        st_iv[b][c] = (uint16_t)__float_as_int(ld_a);
      }
    };
    if (!QRES && n_tiles > 0) {
      fetch_stats(0);
      stash_stats(0);
    }

    for (int t = 0; t < n_tiles; ++t) {
      bool full;
      if (QRES) {
        const int key0 = (j0 + t) * BX + colh;
        full = __all_sync(0xffffffffu, lo <= key0 && hi >= key0 + 32);
      } else {
        // all 256 threads meet: the statistics of tile t are visible, and `full`: every query of it sees every key here
        uint32_t f;
        asm volatile(
            "{\n\t.reg .pred pi, po;\n\t"
            "setp.ne.u32 pi, %1, 0;\n\t"
            "bar.red.and.pred po, 9, 256, pi;\n\t"
            "selp.u32 %0, 1, 0, po;\n\t}"
            : "=r"(f)
            : "r"(ld_full)
            : "memory");
        full = f != 0;
        if (t + 1 < n_tiles) fetch_stats(t + 1);
      }
      if (ok) ok = mbar_wait(smem_addr(&bar_s_full[t & 1]), (t >> 1) & 1, status, kTimeoutCompute);
      ok = __all_sync(0xffffffffu, ok);
      fence_after_sync();
      const uint32_t tmem_s = lane_base + COL_S + (t & 1) * BX + colh;
      uint32_t s[32], d[DUAL ? 32 : 1], pk[16];
      tmem_ld32(tmem_s, s);
      if constexpr (DUAL) tmem_ld32(lane_base + COL_DP + (t & 1) * BX + colh, d);
      tmem_ld_wait();

      if constexpr (QRES) {
        const int key0 = (j0 + t) * BX + colh;
        if (!full) {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (key0 + i < lo || key0 + i >= hi) s[i] = 0xff800000u;  // -inf
        }
      }
      if constexpr (MODE == kFwd) {
        float cmax[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < 32; ++i) cmax[i & 3] = fmaxf(cmax[i & 3], __uint_as_float(s[i]));
        const float hmax = fmaxf(fmaxf(cmax[0], cmax[1]), fmaxf(cmax[2], cmax[3]));
        const float tmax = fmaxf(hmax, exchange(hmax)) * sc;  // sc > 0
        const bool move = tmax > m + kRescaleLog2 || (m == -INFINITY && tmax > -INFINITY);
        const float m_new = move ? tmax : m;
        const float alpha = move ? ex2(m - m_new) : 1.f;
        const float m_sub = m_new == -INFINITY ? 0.f : m_new;
        float csum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float p0 = ex2(fmaf(__uint_as_float(s[i]), sc, -m_sub)), p1 = ex2(fmaf(__uint_as_float(s[i + 1]), sc, -m_sub));
          csum[i & 3] += p0;
          csum[(i & 3) + 1] += p1;
          pk[i >> 1] = pack_bf16(p0, p1);
        }
        l = l * alpha + ((csum[0] + csum[1]) + (csum[2] + csum[3]));
        m = m_new;
        if (t > 0) {  // the accumulation of tile t - 1 has retired before the row may be rescaled
          if (ok) ok = mbar_wait(smem_addr(&bar_acc), (t - 1) & 1, status, kTimeoutCompute);
          ok = __all_sync(0xffffffffu, ok);
          fence_after_sync();
          if (__any_sync(0xffffffffu, move)) {
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
              uint32_t a[32];
              const uint32_t at = lane_base + COL_ACC + half * 128 + c * 32;
              tmem_ld32(at, a);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) a[i] = __float_as_uint(__uint_as_float(a[i]) * alpha);
              tmem_st32(at, a);
            }
          }
        }
      } else if constexpr (MODE == kDq) {
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float p0 = ex2(fmaf(__uint_as_float(s[i]), sc, -lse)), p1 = ex2(fmaf(__uint_as_float(s[i + 1]), sc, -lse));
          pk[i >> 1] = pack_bf16(p0 * (__uint_as_float(d[i]) - delta), p1 * (__uint_as_float(d[i + 1]) - delta));
        }
      } else {
        const int b = t & 1;
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          const float4 l4 = *reinterpret_cast<const float4*>(&st_lse[b][colh + i]);
          const float ls[4] = {l4.x, l4.y, l4.z, l4.w};
          float pr[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) pr[u] = ex2(fmaf(__uint_as_float(s[i + u]), sc, -ls[u]));
          if (!full) {
            const uint2 iv = *reinterpret_cast<const uint2*>(&st_iv[b][colh + i]);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int w = (int)((u < 2 ? iv.x : iv.y) >> (u & 1) * 16);
              if (prow < (w & 0xff) || prow >= (w >> 8 & 0xff)) pr[u] = 0.f;
            }
          }
          if constexpr (MODE == kDk) {
            const float4 d4 = *reinterpret_cast<const float4*>(&st_delta[b][colh + i]);
            pr[0] *= __uint_as_float(d[i]) - d4.x;
            pr[1] *= __uint_as_float(d[i + 1]) - d4.y;
            pr[2] *= __uint_as_float(d[i + 2]) - d4.z;
            pr[3] *= __uint_as_float(d[i + 3]) - d4.w;
          }
          pk[i >> 1] = pack_bf16(pr[0], pr[1]);
          pk[(i >> 1) + 1] = pack_bf16(pr[2], pr[3]);
        }
      }
      tmem_st16(tmem_s, pk);  // over the first half of this thread's own score columns
      tmem_st_wait();
      fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_addr(&bar_f_ready));
      if (!QRES && t + 1 < n_tiles) stash_stats(t + 1);
    }

    // results: this thread's row, 128 of its 256 columns, in two parts
    float mul = MODE == kDv ? 1.f : p.scale;
    if constexpr (MODE == kFwd) {
      const float l_all = l + exchange(l);
      mul = l_all > 0.f ? 1.f / l_all : 0.f;
      if (ok && row_ok && half == 0) p.lse2[(int64_t)h * p.Tq + row] = l_all > 0.f ? m + log2f(l_all) : INFINITY;
    }
    if (n_tiles > 0) {
      if (ok) ok = mbar_wait(smem_addr(&bar_end), 0, status, kTimeoutCompute);
      ok = __all_sync(0xffffffffu, ok);
      fence_after_sync();
    }
#pragma unroll 1
    for (int part = 0; part < 2; ++part) {
      const int col = half * 128 + part * 64;
      float acc[64];
#pragma unroll
      for (int i = 0; i < 64; ++i) acc[i] = 0.f;
      if (n_tiles > 0) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t a[32];
          tmem_ld32(lane_base + COL_ACC + col + c * 32, a);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) acc[c * 32 + i] = __uint_as_float(a[i]) * mul;
        }
      }
      if (!ok) continue;  // the same in the whole warp
      // whole rows through the warp's part of the streamed tiles' memory (idle by now): 8 x 8 KB
      unsigned char* stage = x0_s + (warp - 2) * 8192;
      const int warp_row0 = row0 + quarter * 32;
      if constexpr (QRES) {
        const int64_t rs = MODE == kFwd ? p.o_rs : p.dq_rs;
        store_rows_bf16(stage, acc, 1.f, (MODE == kFwd ? p.out : p.dq) + (int64_t)warp_row0 * rs + h * HD + col, rs, p.Tq - warp_row0, lane);
      } else {
        const int64_t rs = (int64_t)p.nkv * HD, off = (int64_t)warp_row0 * rs + kvh * HD + col, plane = (int64_t)p.Tc * rs;
        if (p.dkv_part != nullptr)
          store_rows_f32(stage, acc, p.dkv_part + ((int64_t)(h - kvh * group) * 2 + (MODE == kDv ? 1 : 0)) * plane + off, rs, p.Tc - warp_row0, lane);
        else
          store_rows_bf16(stage, acc, 1.f, (MODE == kDv ? p.dv : p.dk) + off, rs, p.Tc - warp_row0, lane);
      }
    }
    fence_before_sync();
  }

  fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

struct Maps {
  CUtensorMap q_r, do_r, k_r, v_r, q_x, do_x, k_x, v_x;  // resident (128-row boxes) and streamed (64-row boxes)
};

template <int MODE>
static int launch(const CUtensorMap& r0, const CUtensorMap& r1, const CUtensorMap& x0, const CUtensorMap& x1, const AttnParams& p, int* status,
                  cudaStream_t stream) {
  static PerDeviceOnce configured;
  if (configured.needed()) {
    if (cudaFuncSetAttribute(wide_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem<MODE>) != cudaSuccess) return -2;
    configured.mark();
  }
  dim3 grid(p.nh, ((kQueriesResident<MODE> ? p.Tq : p.Tc) + BM - 1) / BM);
  count_launch(1);
  launch_pdl(wide_kernel<MODE>, grid, THREADS, kSmem<MODE>, stream, r0, r1, x0, x1, p, (p.Tc + kAttnKeyTile - 1) / kAttnKeyTile, status);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace awtc

// Head dim 256 without extra keys.
int launch_attn_fwd_wide_tc(const AttnParams& p, int* status, cudaStream_t stream) {
  using namespace awtc;
  if (p.E > 0 || p.ext_block > 0) return -4;
  if (p.Tq <= 0) return 0;
  CUtensorMap q, k, v;
  int rc = tc::make_map_bf16(&q, p.q, p.Tq, (int64_t)p.nh * HD, p.q_rs, BM);
  if (rc == 0) rc = tc::make_map_bf16(&k, p.k, p.Tc, (int64_t)p.nkv * HD, p.k_rs, BX);
  if (rc == 0) rc = tc::make_map_bf16(&v, p.v, p.Tc, (int64_t)p.nkv * HD, p.v_rs, BX);
  return rc ? rc : launch<kFwd>(q, q, k, v, p, status, stream);
}

int launch_attn_bwd_wide_tc(const AttnParams& p, int* tile_qmin, int* tile_qmax, int* status, cudaStream_t stream) {
  using namespace awtc;
  if (p.E > 0 || p.ext_block > 0) return -4;
  if (p.Tq <= 0) return 0;
  Maps m;
  const int64_t qw = (int64_t)p.nh * HD, kw = (int64_t)p.nkv * HD;
  int rc = 0;
  auto map = [&](CUtensorMap* to, const void* base, int rows, int64_t width, int64_t rs, int box) { if (rc == 0) rc = tc::make_map_bf16(to, base, rows, width, rs, box); };
  map(&m.q_r, p.q, p.Tq, qw, p.q_rs, BM);
  map(&m.do_r, p.dout, p.Tq, qw, p.do_rs, BM);
  map(&m.k_r, p.k, p.Tc, kw, p.k_rs, BM);
  map(&m.v_r, p.v, p.Tc, kw, p.v_rs, BM);
  map(&m.q_x, p.q, p.Tq, qw, p.q_rs, BX);
  map(&m.do_x, p.dout, p.Tq, qw, p.do_rs, BX);
  map(&m.k_x, p.k, p.Tc, kw, p.k_rs, BX);
  map(&m.v_x, p.v, p.Tc, kw, p.v_rs, BX);
  if (rc) return rc;
  launch_attn_delta(p, HD, stream);
  rc = launch<kDq>(m.q_r, m.do_r, m.k_x, m.v_x, p, status, stream);
  if (rc == 0) rc = launch_kv_tile_range(p, tile_qmin, tile_qmax, stream);
  if (rc == 0) rc = launch<kDk>(m.k_r, m.v_r, m.q_x, m.do_x, p, status, stream);
  if (rc == 0) rc = launch<kDv>(m.k_r, m.k_r, m.q_x, m.do_x, p, status, stream);
  if (rc == 0 && p.dkv_part != nullptr) rc = launch_dkv_reduce(p, HD, stream);
  return rc;
}

}  // namespace sb200
