// SDPA backward for sm_100a (bf16, head size 128 or 64), mask from token positions: every score tile is formed ONCE.
//
// Given dO, the forward's O and log-sum-exp, computes dQ (B,H,T,D) bf16, and accumulates dK, dV into fp32 cache-shaped
// buffers (B,G,C,D).
//   dkv kernel : CTA = 128 KV slots, streams query tiles of 128 packed rows (npos positions x gs heads, head major)
//                S^T = K Q^T, dP^T = V dO^T  ->  P^T, dS^T  ->  dV += P^T dO, dK += dS^T Q;  dS (bf16) -> workspace
//   dq kernel  : CTA = 128 query rows, streams KV tiles: dQ += dS K, a product without any softmax in it
//
// Why this split. Forming S and dP in a launch for dQ and again in one for dK / dV (7 GEMM-equivalents, in units of 64
// columns whose M = 128, N = 64 MMAs re-read the 128-row A operand from shared memory for half the arithmetic) took
// 1.14 ms for 1024 queries x 32 heads over 16384 slots. Here S and dP are formed once, the five necessary products are
// all that is left, and S and dP have ONE buffer of 128 TMEM columns each beside dV and dK. Two chains, one issuer thread
// and one accumulator each, keep the tensor pipe busy:
//     thread A:  wait P(i)  -> dV += P(i) dO(i),  S(i+1)          thread B:  wait dS(i) -> dK += dS(i) Q(i),  dP(i+1)
// so that the exponentials of a tile run under dK / dP and the products P (dP − δ) under dV / S. S goes in two halves of
// 64 columns, so that the exponentials of one half overlap dV and the next S of the other. Measured: 0.81 ms back to back
// under the power cap, 0.69 ms in short runs (dkv 0.48, dq 0.18). dkv: 3220 cycles a tile, 2304 of them MMA, of which shared
// memory serves most. Marks of the first compute warp (kvb_sdpa_bwd_set_trace): stores of dS, wait and exponentials of the
// first half 1380, exponentials of the second half 770 (512 at the special-function rate), wait for dP and dS 960.
// dq: 1.1 GB of dS at 6.1 TB/s.
// dS passes through memory (32 KB written and read per tile) instead of being reduced into dQ by atomics: a coalesced
// red.add.f32 of the 64 KB dQ tile was measured at 5.9 TB/s over the chip, no faster than the two 32 KB passes, and its
// order is not fixed. Every output has one owner and a fixed order of sums: gradients are the same run to run.
// The workspace is bounded (BO_DS_LIMIT, or what the caller has): larger calls go in rounds over query tiles, then over
// (sequence, group) pairs.
//
// Replaces the blocked fp32 PyTorch backward of the reference
// (keys_values/attention/sdpa_op.py:31-251) and the library SDPA backward it otherwise uses.
#include <cuda.h>
#include <limits.h>
#include <stdlib.h>

#include "common.cuh"
#include "kvb200.h"

extern "C" int kvb_att_tile_minmax(const int32_t* token_pos, int32_t* tmin, int32_t* tmax, int B, int G, int L, long long tp_sb,
                                   long long tp_sg, int tile, void* stream);

namespace kvb {

constexpr int BO_TILE = 128 * 128 * 2;       // 32 KB: two 64-feature chunks of [128 rows x 128 B]
constexpr int BO_CHUNK = BO_TILE / 2;
constexpr int BO_QSTAGES = 3, BO_OSTAGES = 2;  // Q lives from S(i) to dK(i), dO from dP(i) to dV(i)
// Barriers of "thread A has issued S(i + 1)", used in turn. Nothing that A needs for tile i + 1 hangs on B having looked at the
// one of tile i (P(i + 1) comes after dS(i), whose dP(i) B issued a tile before), so a single barrier could move on by two
// phases and B would miss its own. Arrival i + 2 needs P(i + 2), hence dS(i + 1) and dP(i + 1), which B issues after its wait
// for tile i: two barriers are enough.
constexpr int BO_TURNS = 2;
constexpr int BO_THREADS = 384;              // producer, issuer A, issuer B, idle, 8 compute warps
constexpr int BO_QK_STAGES = 3;              // dq kernel: dS tile | K tile per stage
constexpr int BO_DQ_THREADS = 192;           // producer, issuer, 4 epilogue warps

struct BoSmem {
  static constexpr int K = 0;
  static constexpr int V = K + BO_TILE;
  static constexpr int Q = V + BO_TILE;
  static constexpr int O = Q + BO_QSTAGES * BO_TILE;
  static constexpr int STAT = O + BO_OSTAGES * BO_TILE;  // two slots of −lse·log2(e)[128] | −delta·scale[128]
  static constexpr int BAR = STAT + 2 * 1024;
  static constexpr int TOTAL = BAR + 256;
  static constexpr int ROW = 256 + 16;  // epilogue: padded half rows of 64 fp32, one buffer of 32 rows per compute warp
};
static_assert(BoSmem::TOTAL <= 232448, "shared memory of the dkv kernel exceeds the limit of a CTA");
static_assert(8 * 32 * BoSmem::ROW <= BO_QSTAGES * BO_TILE, "epilogue buffers alias the Q ring");

struct BoParams {
  const int32_t* token_pos;
  const int32_t* tile_min;   // (B,G,nT)
  const int32_t* tile_max;
  const float* stats;        // (B·G, nQT, 2, 128): −lse·log2(e) (−inf: no query), −delta·scale
  __nv_bfloat16* ds;         // workspace of the round: (pairs, nT, nq) tiles of [16 units of 8 rows][128 slots][8]
  __nv_bfloat16* dq;         // (B,H,T,D)
  float* dk;                 // (B,G,C,D) accumulated
  float* dv;
  int G, H, T, L, nT, nQT, gs, npos, rows_used;
  int bg0, q0, nq;           // this round: first (sequence, group) pair, query tiles [q0, q0 + nq)
  long long tp_sb, tp_sg, dk_sb, dk_sg;
  float scale, scale_log2;
  int input_pos;
  // Sliding window (0: none): a slot is visible to a query at position q iff q - window < token <= q.
  // Soft-capping (cap_pre = 0: none): s' = cap·tanh(scale·s / cap) with cap_pre = scale / cap, cap_l2 = cap·log2(e);
  // then P = exp2(cap_l2·t − lse·log2(e)) and dS = P (dP − δ) scale (1 − t²) with t = tanh(cap_pre·s).
  int window;
  float cap_pre, cap_l2;
  int* status;
  long long* trace;     // optional timeline of CTA 0: per role trace_cap (tag, clock) pairs
  int trace_cap;
};

// Timeline event of one role (1 MMA issuer, 2 first compute warp) of CTA 0; tr_n starts at BO_TRACE_OFF everywhere else.
#define BO_TRACE_OFF (1 << 30)
#define BO_TRACE(role, tag)                                               \
  do {                                                                    \
    if (tr_n < p.trace_cap) {                                             \
      p.trace[((role) * p.trace_cap + tr_n) * 2] = (long long)(tag);      \
      p.trace[((role) * p.trace_cap + tr_n) * 2 + 1] = clock64();         \
      ++tr_n;                                                             \
    }                                                                     \
  } while (0)

__device__ __forceinline__ int bo_qpos_max(const BoParams& p, int qt) { return p.input_pos + min((qt + 1) * p.npos, p.T) - 1; }
// some query of tile qt sees some slot of a KV tile whose token positions span [tmin, tmax]
template <bool GEN>
__device__ __forceinline__ bool bo_active(const BoParams& p, int qt, int tmin, int tmax) {
  return tmin <= bo_qpos_max(p, qt) && (!GEN || p.window <= 0 || tmax > p.input_pos + qt * p.npos - p.window);
}

// Statistics per packed query row and a head-major copy of dO, one warp per packed row:
// stats[bg][qt][0][row] = −lse·log2(e), stats[bg][qt][1][row] = −scale·sum_d dO·O; rows without a query: −inf, 0 (P = dS = 0).
template <int HD>
__global__ void bo_stats_kernel(const __nv_bfloat16* __restrict__ dO, const __nv_bfloat16* __restrict__ O, const float* __restrict__ lse,
                                float* __restrict__ stats, __nv_bfloat16* __restrict__ dOt, int B, int G, int H, int T, int gs,
                                int npos, int nQT, float scale) {
  const long long w = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int row = (int)(w & 127);
  const long long tile = w >> 7;  // (bg, qt)
  if (tile >= (long long)B * G * nQT) return;
  const int lane = threadIdx.x & 31;
  const int qt = (int)(tile % nQT);
  const int bg = (int)(tile / nQT);
  const int b = bg / G, g = bg % G;
  const int hq = row / npos, t = qt * npos + row % npos;
  float* st = stats + tile * 256 + row;
  if (hq >= gs || t >= T) {
    if (lane == 0) {
      st[0] = -INFINITY;
      st[128] = 0.f;
    }
    return;
  }
  const int h = g * gs + hq;
  constexpr int PER = HD / 32;  // features per lane: 4 (one 8-byte access) or 2 (one 4-byte access)
  const long long src = (((long long)b * T + t) * H + h) * HD + lane * PER;
  const long long hrow = ((long long)b * H + h) * T + t;
  uint2 a = make_uint2(0, 0), o = make_uint2(0, 0);
  if (PER == 4) {
    a = *reinterpret_cast<const uint2*>(dO + src);
    o = *reinterpret_cast<const uint2*>(O + src);
  } else {
    a.x = *reinterpret_cast<const uint32_t*>(dO + src);
    o.x = *reinterpret_cast<const uint32_t*>(O + src);
  }
  const __nv_bfloat162* ap = reinterpret_cast<const __nv_bfloat162*>(&a);
  const __nv_bfloat162* op = reinterpret_cast<const __nv_bfloat162*>(&o);
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < PER / 2; ++i) {
    const float2 x = __bfloat1622float2(ap[i]), y = __bfloat1622float2(op[i]);
    s += x.x * y.x + x.y * y.y;
  }
  s = warp_sum(s);
  if (PER == 4) *reinterpret_cast<uint2*>(dOt + hrow * HD + lane * 4) = a;
  else *reinterpret_cast<uint32_t*>(dOt + hrow * HD + lane * 2) = a.x;
  if (lane == 0) {
    st[0] = -lse[hrow] * 1.4426950408889634f;
    st[128] = -s * scale;
  }
}

__device__ __forceinline__ float bo_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// hardware tanh, as in the forward kernels (P must be recomputed from the same capped scores)
__device__ __forceinline__ float bo_tanh(float z) {
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(z));
  return t;
}

// Bits of the columns [c0, c0 + 32) whose position lies before `th` positions into the tile (columns are head major,
// npos per head): the queries that may not see a token `th` positions beyond the first one of the tile.
__device__ __forceinline__ uint32_t bo_hidden(int c0, int npos, int th) {
  uint32_t bits = 0;
  for (int lo = (c0 / npos) * npos - c0; lo < 32; lo += npos) {
    const int a = max(lo, 0), e = min(lo + th, 32);
    if (e > a) bits |= (0xffffffffu >> (32 - (e - a))) << a;
  }
  return bits;
}

// GEN: sliding window and / or soft-capping are in use (instantiations of their own, so that the plain kernels keep their
// registers). HD: head size, 128 or 64 (tiles of one 64-feature chunk, half as many K steps, accumulators of 64 columns).
template <bool GEN, int HD>
__global__ void __launch_bounds__(BO_THREADS, 1)
bwd_dkv_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
               const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmO, const BoParams p) {
  using S = BoSmem;
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023u) {  // swizzled tiles need a 1024-byte aligned window: report, do not run
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, STATUS_TIMEOUT_MISC);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::BAR);
  uint64_t* k_full = bars + 0;
  uint64_t* v_full = bars + 1;
  uint64_t* q_full = bars + 2;     // [3]
  uint64_t* q_empty = bars + 5;    // [3]
  uint64_t* o_full = bars + 8;     // [2]
  uint64_t* o_empty = bars + 10;   // [2] dV (thread A) and dP (thread B) have read dO
  uint64_t* st_full = bars + 12;   // [2]
  uint64_t* x_full = bars + 14;    // [2] halves of 64 columns
  uint64_t* p_full = bars + 16;    // [2]
  uint64_t* y_full = bars + 18;
  uint64_t* ds_full = bars + 19;
  uint64_t* acc_full = bars + 20;  // one commit per issuer
  uint64_t* a_issued = bars + 21;  // [BO_TURNS] thread A has issued S(i + 1)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 21 + BO_TURNS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kt = blockIdx.x % p.nT;
  const int lbg = blockIdx.x / p.nT;
  const int bg = p.bg0 + lbg;
  const int b = bg / p.G, g = bg % p.G;
  // Query tiles that see this KV tile: without a window all from one on (its oldest token), with one up to another (its newest).
  const int tmin = p.tile_min[(long long)bg * p.nT + kt], tmax = p.tile_max[(long long)bg * p.nT + kt];
  int q_first = p.q0, q_end = p.q0 + p.nq;
  while (q_first < q_end && !bo_active<GEN>(p, q_first, tmin, tmax)) ++q_first;
  if (GEN)
    while (q_end > q_first && !bo_active<GEN>(p, q_end - 1, tmin, tmax)) --q_end;
  const int n = q_end - q_first;
  if (n <= 0) return;

  if (p.rows_used < 128) {  // rows that no TMA box writes enter MMAs as operand rows: finite zeros
    const int n16 = (128 - p.rows_used) * 8;
    for (int i = threadIdx.x; i < (BO_QSTAGES + BO_OSTAGES) * 2 * n16; i += BO_THREADS)
      *reinterpret_cast<uint4*>(smem + S::Q + (i / n16) * BO_CHUNK + p.rows_used * 128 + (i % n16) * 16) = make_uint4(0, 0, 0, 0);
    fence_proxy_async_smem();
  }
  if (threadIdx.x == 0) {
    mbar_init(k_full, 1);
    mbar_init(v_full, 1);
    for (int s = 0; s < BO_QSTAGES; ++s) {
      mbar_init(&q_full[s], 1);
      mbar_init(&q_empty[s], 1);
    }
    for (int s = 0; s < BO_OSTAGES; ++s) {
      mbar_init(&o_full[s], 1);
      mbar_init(&o_empty[s], 2);
      mbar_init(&st_full[s], 1);
    }
    for (int h = 0; h < 2; ++h) {
      mbar_init(&x_full[h], 1);
      mbar_init(&p_full[h], 8);
    }
    mbar_init(y_full, 1);
    mbar_init(ds_full, 8);
    mbar_init(acc_full, 2);
    for (int u = 0; u < BO_TURNS; ++u) mbar_init(&a_issued[u], 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_X = tmem_base, tmem_Y = tmem_base + 128, tmem_dV = tmem_base + 256, tmem_dK = tmem_base + 384;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tma_prefetch_desc(&tmQ);
      tma_prefetch_desc(&tmO);
      mbar_expect_tx(k_full, 256 * HD);
      tma_load_4d(smem + S::K, &tmK, k_full, 0, kt * 128, g, b);
      if (HD == 128) tma_load_4d(smem + S::K + BO_CHUNK, &tmK, k_full, 64, kt * 128, g, b);
      bool ok = true;
      for (int i = 0; i < n && ok; ++i) {
        const int qs = i % BO_QSTAGES, os = i % BO_OSTAGES, t0 = (q_first + i) * p.npos;
        const uint32_t bytes = (uint32_t)(p.rows_used * HD * 2);
        if (!(ok = mbar_wait_bounded(&q_empty[qs], ((i / BO_QSTAGES) & 1) ^ 1, abort_flag, p.status, STATUS_TIMEOUT_EMPTY))) break;
        uint8_t* qd = smem + S::Q + qs * BO_TILE;
        mbar_expect_tx(&q_full[qs], bytes);
        tma_load_4d(qd, &tmQ, &q_full[qs], 0, t0, g * p.gs, b);
        if (HD == 128) tma_load_4d(qd + BO_CHUNK, &tmQ, &q_full[qs], 64, t0, g * p.gs, b);
        if (i == 0) {
          mbar_expect_tx(v_full, 256 * HD);
          tma_load_4d(smem + S::V, &tmV, v_full, 0, kt * 128, g, b);
          if (HD == 128) tma_load_4d(smem + S::V + BO_CHUNK, &tmV, v_full, 64, kt * 128, g, b);
        }
        if (!(ok = mbar_wait_bounded(&o_empty[os], ((i / BO_OSTAGES) & 1) ^ 1, abort_flag, p.status, STATUS_TIMEOUT_EMPTY))) break;
        uint8_t* od = smem + S::O + os * BO_TILE;
        mbar_expect_tx(&o_full[os], bytes);
        tma_load_4d(od, &tmO, &o_full[os], 0, t0, g * p.gs, b);
        if (HD == 128) tma_load_4d(od + BO_CHUNK, &tmO, &o_full[os], 64, t0, g * p.gs, b);
        // the slot of these statistics is free once dK(i − 2) has run, which the next Q tile waits for anyway
        if (i >= 2 && !(ok = mbar_wait_bounded(&q_empty[(i - 2) % BO_QSTAGES], ((i - 2) / BO_QSTAGES) & 1, abort_flag, p.status, STATUS_TIMEOUT_EMPTY))) break;
        mbar_expect_tx(&st_full[i & 1], 1024);
        bulk_load(smem + S::STAT + (i & 1) * 1024, p.stats + ((long long)bg * p.nQT + q_first + i) * 256, 1024, &st_full[i & 1]);
      }
      if (!ok) {  // let copies in flight land before the CTA's shared memory is released
        long long c0 = clock64();
        while (clock64() - c0 < 2000000LL) {
        }
      }
    }
  } else if (warp == 1 || warp == 2) {
    // ------------------------------------------------------------ MMA issuers
    if (elect_one()) {
      constexpr uint32_t idesc_acc = make_idesc_bf16(128, HD, 0, 1);  // A from TMEM, B MN-major
      constexpr uint32_t idesc_x = make_idesc_bf16(128, 64, 0, 0), idesc_y = make_idesc_bf16(128, 128, 0, 0);
      // scores from two K-major tiles in shared memory
      auto scores = [&](uint32_t d, uint32_t a, uint32_t bm, uint32_t idesc) {
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint32_t off = (uint32_t)((kk >> 2) * BO_CHUNK + (kk & 3) * 32);
          umma_f16_ss(d, make_smem_desc_sw128(a + off, 16, 1024), make_smem_desc_sw128(bm + off, 16, 1024), idesc, kk != 0);
        }
      };
      auto scores_half = [&](int h, uint32_t bm) {  // columns [64·h, +64) of S
        scores(tmem_X + (uint32_t)(64 * h), smem_u32(smem + S::K), bm + (uint32_t)(h * 64 * 128), idesc_x);
        umma_commit(&x_full[h]);
      };
      // D += A · B over the 64 query rows of half h, A (P or dS, packed bf16) in TMEM: the two compute warps of a lane
      // quarter keep their 32 columns as 16 packed ones at columns 0 and 32 of the half
      auto accumulate = [&](uint32_t d, uint32_t a, uint32_t bm, int h, bool first) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          umma_f16_ts(d, a + (uint32_t)(64 * h + 32 * (u >> 1) + 8 * (u & 1)),
                      make_smem_desc_sw128(bm + (uint32_t)((4 * h + u) * 16 * 128), BO_CHUNK, 1024), idesc_acc, (first && u == 0) ? 0u : 1u);
      };
      auto q_addr = [&](int i) { return smem_u32(smem + S::Q + (i % BO_QSTAGES) * BO_TILE); };
      auto o_addr = [&](int i) { return smem_u32(smem + S::O + (i % BO_OSTAGES) * BO_TILE); };
      auto wait_q = [&](int i) { return mbar_wait_bounded(&q_full[i % BO_QSTAGES], (i / BO_QSTAGES) & 1, abort_flag, p.status, STATUS_TIMEOUT_FULL); };
      auto wait_o = [&](int i) { return mbar_wait_bounded(&o_full[i % BO_OSTAGES], (i / BO_OSTAGES) & 1, abort_flag, p.status, STATUS_TIMEOUT_FULL); };
      bool ok;
      int tr_n = p.trace && blockIdx.x == 0 && warp == 1 ? 0 : BO_TRACE_OFF;
      if (warp == 1) {
        ok = mbar_wait_bounded(k_full, 0, abort_flag, p.status, STATUS_TIMEOUT_FULL) && wait_q(0);
        if (ok) {
          tc_fence_after();
          scores_half(0, q_addr(0));
          scores_half(1, q_addr(0));
        }
        for (int i = 0; i < n && ok; ++i) {
          const bool more = i + 1 < n;
          if (!(ok = wait_o(i) && (!more || wait_q(i + 1)))) break;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            BO_TRACE(1, 1000000 + 2 * i + h);
            if (!(ok = mbar_wait_bounded(&p_full[h], i & 1, abort_flag, p.status, STATUS_TIMEOUT_FULL))) break;
            BO_TRACE(1, 1100000 + 2 * i + h);
            tc_fence_after();
            accumulate(tmem_dV, tmem_X, o_addr(i), h, i == 0 && h == 0);
            if (h == 1) umma_commit(&o_empty[i % BO_OSTAGES]);
            if (more) scores_half(h, q_addr(i + 1));
            BO_TRACE(1, 1200000 + 2 * i + h);
          }
          if (!ok) break;
          mbar_arrive(&a_issued[i % BO_TURNS]);
        }
      } else {
        ok = mbar_wait_bounded(v_full, 0, abort_flag, p.status, STATUS_TIMEOUT_FULL) && wait_o(0);
        if (ok) {
          tc_fence_after();
          scores(tmem_Y, smem_u32(smem + S::V), o_addr(0), idesc_y);
          umma_commit(y_full);
          umma_commit(&o_empty[0]);
        }
        for (int i = 0; i < n && ok; ++i) {
          const bool more = i + 1 < n;
          if (!(ok = wait_q(i) && (!more || wait_o(i + 1)))) break;
          // The next scores go first: the exponentials hang on them, and the tensor pipe serves both threads in turn.
          if (!(ok = mbar_wait_bounded(&a_issued[i % BO_TURNS], (i / BO_TURNS) & 1, abort_flag, p.status, STATUS_TIMEOUT_FULL))) break;
          if (!(ok = mbar_wait_bounded(ds_full, i & 1, abort_flag, p.status, STATUS_TIMEOUT_FULL))) break;
          tc_fence_after();
          accumulate(tmem_dK, tmem_Y, q_addr(i), 0, i == 0);
          accumulate(tmem_dK, tmem_Y, q_addr(i), 1, false);
          umma_commit(&q_empty[i % BO_QSTAGES]);
          if (more) {
            scores(tmem_Y, smem_u32(smem + S::V), o_addr(i + 1), idesc_y);
            umma_commit(y_full);
            umma_commit(&o_empty[(i + 1) % BO_OSTAGES]);
          }
        }
      }
      if (ok) umma_commit(acc_full);
    }
  } else if (warp >= 4) {
    // ----------------------------------------------- compute + epilogue warps
    // two warps per TMEM lane quarter; thread (row, hh): KV slot `row`, columns [32·hh, +32) of both halves
    // of every query tile, columns [64·hh, +64) of the accumulators (head size 64: [32·hh, +32))
    const int quarter = warp & 3;
    const int hh = (warp - 4) >> 2;
    const int row = quarter * 32 + lane;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const int j = kt * 128 + row;
    const bool row_valid = j < p.L;
    int row_tp = INT_MAX;
    if (row_valid) row_tp = p.token_pos ? p.token_pos[b * p.tp_sb + g * p.tp_sg + j] : j;
    const uint32_t xaddr = tmem_X + lane_base + (uint32_t)(32 * hh), yaddr = tmem_Y + lane_base + (uint32_t)(32 * hh);
    const float2 c2 = make_float2(p.scale_log2, p.scale_log2), sc2 = make_float2(p.scale, p.scale);
    const bool soft = GEN && p.cap_pre != 0.f;
    bool ok = true;
    int tr_n = p.trace && blockIdx.x == 0 && warp == 4 && lane == 0 ? 0 : BO_TRACE_OFF;  // only the first compute warp records
    uint4* ds_dst = reinterpret_cast<uint4*>(p.ds + (((long long)lbg * p.nT + kt) * p.nq + (q_first - p.q0)) * 16384) + (4 * hh) * 128 + row;
    for (int i = 0; i < n && ok; ++i, ds_dst += 2048) {
      const float* nlse = reinterpret_cast<const float*>(smem + S::STAT + (i & 1) * 1024) + 32 * hh;
      const float* ndls = nlse + 128;
      const int qpos0 = p.input_pos + (q_first + i) * p.npos;
      uint32_t hide[2] = {0, 0};
      bool any_hidden = false;
      if (GEN && p.window > 0) {  // visible iff 0 <= position of the query − token < window
        const int th = (int)max(min((long long)row_tp - qpos0, (long long)p.npos), 0LL);
        const int te = (int)max(min((long long)row_tp + p.window - qpos0, (long long)p.npos), 0LL);
        any_hidden = __any_sync(0xffffffffu, th > 0 || te < p.npos);
        if (any_hidden) {
          hide[0] = bo_hidden(32 * hh, p.npos, th) | ~bo_hidden(32 * hh, p.npos, te);
          hide[1] = bo_hidden(64 + 32 * hh, p.npos, th) | ~bo_hidden(64 + 32 * hh, p.npos, te);
        }
      } else if (tmax > qpos0) {  // some slot of the tile is newer than the first query
        const int th = (int)min((long long)row_tp - qpos0, (long long)p.npos);
        any_hidden = __any_sync(0xffffffffu, th > 0);
        if (th >= p.npos) {  // newer than every query of the tile
          hide[0] = hide[1] = 0xffffffffu;
        } else if (th > 0) {
          hide[0] = bo_hidden(32 * hh, p.npos, th);
          hide[1] = bo_hidden(64 + 32 * hh, p.npos, th);
        }
      }
      if (!(ok = mbar_wait_bounded(&st_full[i & 1], (i >> 1) & 1, abort_flag, p.status, STATUS_TIMEOUT_FULL))) break;
      uint32_t xr[64];
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {  // the first half is on its way to dV while the second one is computed
        if (!(ok = mbar_wait_bounded(&x_full[hf], i & 1, abort_flag, p.status, STATUS_TIMEOUT_TMEM_FULL))) break;
        tc_fence_after();
        tmem_ld_32x32b_x32(xaddr + (uint32_t)(64 * hf), xr + 32 * hf);
        tmem_ld_wait();
        uint32_t pk[16];
        if (soft) {
          // capped scores: P for dV is packed here, what stays in registers is P (1 − tanh²), the factor of dS
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            float pp[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const float t = bo_tanh(__uint_as_float(xr[32 * hf + e + u]) * p.cap_pre);
              pp[u] = (hide[hf] & (1u << (e + u))) ? 0.f : bo_exp2(fmaf(t, p.cap_l2, nlse[64 * hf + e + u]));
              xr[32 * hf + e + u] = __float_as_uint(pp[u] * fmaf(-t, t, 1.f));
            }
            pk[e >> 1] = pack_bf16x2(pp[0], pp[1]);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 32; e += 4) {
            const float4 nl = *reinterpret_cast<const float4*>(nlse + 64 * hf + e);
            uint32_t* x = xr + 32 * hf + e;
            float2 a = ffma2(make_float2(__uint_as_float(x[0]), __uint_as_float(x[1])), c2, make_float2(nl.x, nl.y));
            float2 c = ffma2(make_float2(__uint_as_float(x[2]), __uint_as_float(x[3])), c2, make_float2(nl.z, nl.w));
            a = make_float2(bo_exp2(a.x), bo_exp2(a.y));
            c = make_float2(bo_exp2(c.x), bo_exp2(c.y));
            x[0] = __float_as_uint(a.x); x[1] = __float_as_uint(a.y); x[2] = __float_as_uint(c.x); x[3] = __float_as_uint(c.y);
          }
          if (any_hidden) {
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (hide[hf] & (1u << e)) xr[32 * hf + e] = 0;
          }
#pragma unroll
          for (int e = 0; e < 16; ++e) pk[e] = pack_bf16x2(__uint_as_float(xr[32 * hf + 2 * e]), __uint_as_float(xr[32 * hf + 2 * e + 1]));
        }
        tmem_st_32x32b_x16(xaddr + (uint32_t)(64 * hf), pk);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[hf]);
        BO_TRACE(2, 2200000 + 2 * i + hf);
      }
      if (!ok) break;
      if (!(ok = mbar_wait_bounded(y_full, i & 1, abort_flag, p.status, STATUS_TIMEOUT_TMEM_FULL))) break;
      tc_fence_after();
      uint32_t dk_[32];
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t yr[32];
        tmem_ld_32x32b_x32(yaddr + (uint32_t)(64 * hf), yr);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 32; e += 4) {
          const float4 nd = *reinterpret_cast<const float4*>(ndls + 64 * hf + e);
          const uint32_t* x = xr + 32 * hf + e;
          float2 a = ffma2(make_float2(__uint_as_float(yr[e]), __uint_as_float(yr[e + 1])), sc2, make_float2(nd.x, nd.y));
          float2 c = ffma2(make_float2(__uint_as_float(yr[e + 2]), __uint_as_float(yr[e + 3])), sc2, make_float2(nd.z, nd.w));
          a = fmul2(make_float2(__uint_as_float(x[0]), __uint_as_float(x[1])), a);
          c = fmul2(make_float2(__uint_as_float(x[2]), __uint_as_float(x[3])), c);
          dk_[16 * hf + (e >> 1)] = pack_bf16x2(a.x, a.y);
          dk_[16 * hf + (e >> 1) + 1] = pack_bf16x2(c.x, c.y);
        }
        tmem_st_32x32b_x16(yaddr + (uint32_t)(64 * hf), dk_ + 16 * hf);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full);
      BO_TRACE(2, 2300000 + 2 * i);
      // workspace: 8 query rows (16 bytes) of 32 consecutive slots per instruction, 512 contiguous bytes per warp. They hold
      // the warp ≈ 700 of 3220 cycles a tile (64 B/clk to L2); spread over the exponentials, or done by warps of their own
      // that read dS back from TMEM, they slow the exponentials down by more (both go through the queue of the LSU).
#pragma unroll
      for (int u = 0; u < 8; ++u)
        __stcs(ds_dst + (8 * (u >> 2) + (u & 3)) * 128, make_uint4(dk_[4 * u], dk_[4 * u + 1], dk_[4 * u + 2], dk_[4 * u + 3]));
    }
    // ---- epilogue: fp32 tiles -> padded rows in shared memory (the Q ring is free) -> coalesced vector reductions.
    // Every address is touched by this CTA only, so the sums do not depend on any order.
    if (ok) ok = mbar_wait_bounded(acc_full, 0, abort_flag, p.status, STATUS_TIMEOUT_TMEM_FULL);
    if (ok) {
      tc_fence_after();
      constexpr int W = HD / 2, LPR = W / 4;  // fp32 of a half row, lanes that add one
      uint8_t* buf = smem + S::Q + (warp - 4) * 32 * S::ROW;
      const long long off = b * p.dk_sb + g * p.dk_sg + (long long)(kt * 128 + quarter * 32) * HD + W * hh;
      const int rows = min(32, p.L - (kt * 128 + quarter * 32));
#pragma unroll 1
      for (int w = 0; w < 2; ++w) {
        uint32_t r[W];
        const uint32_t src = (w == 0 ? tmem_dV : tmem_dK) + lane_base + (uint32_t)(W * hh);
#pragma unroll
        for (int c = 0; c < W; c += 32) tmem_ld_32x32b_x32(src + (uint32_t)c, r + c);
        tmem_ld_wait();
#pragma unroll
        for (int u = 0; u < W / 4; ++u)
          *reinterpret_cast<uint4*>(buf + lane * S::ROW + u * 16) = make_uint4(r[4 * u], r[4 * u + 1], r[4 * u + 2], r[4 * u + 3]);
        __syncwarp();
        float* dst = (w == 0 ? p.dv : p.dk) + off + (lane % LPR) * 4;
#pragma unroll
        for (int u = 0; u < LPR; ++u) {
          const int rr = (32 / LPR) * u + lane / LPR;
          const float4 v = *reinterpret_cast<const float4*>(buf + rr * S::ROW + (lane % LPR) * 16);
          if (rr < rows)
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + rr * HD), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
        }
        __syncwarp();
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// Descriptor of an MN-major operand without swizzle: core matrices of 8 k-rows x 8 MN elements, 128 contiguous bytes;
// `k_bytes` / `mn_bytes` lie between core matrices along K (leading offset) and along MN (stride offset).
__device__ __forceinline__ uint64_t bo_desc_mn(uint32_t smem_addr, uint32_t k_bytes, uint32_t mn_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3FFF);
  d |= (uint64_t)((k_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((mn_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

// dQ of one query tile: dS tiles of the workspace (A operand, MN-major without swizzle: element (query row 8u + e, slot r) at
// 2048·u + 16·r + 2·e, so that the kernel above can write it coalesced) times K tiles (B operand, MN-major).
// Bound by reading dS: 64 KB per step into shared memory, 512 tensor cycles.
struct BoDqSmem {
  static constexpr int RING = 0;  // per stage: dS tile | K tile
  static constexpr int BAR = RING + BO_QK_STAGES * 2 * BO_TILE;
  static constexpr int TOTAL = BAR + 128;
};
template <bool GEN, int HD>
__global__ void __launch_bounds__(BO_DQ_THREADS, 1)
bwd_dq_kernel(const __grid_constant__ CUtensorMap tmK, const BoParams p) {
  using S = BoDqSmem;
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023u) {
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, STATUS_TIMEOUT_MISC);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::BAR);
  uint64_t* full = bars + 0;   // [3]
  uint64_t* empty = bars + 3;  // [3]
  uint64_t* acc_full = bars + 6;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 7);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lq = blockIdx.x % p.nq, lbg = blockIdx.x / p.nq;
  const int qt = p.q0 + lq, bg = p.bg0 + lbg;
  const int b = bg / p.G, g = bg % p.G;
  const int32_t* tmin = p.tile_min + (long long)bg * p.nT;
  const int32_t* tmax = p.tile_max + (long long)bg * p.nT;
  if (threadIdx.x == 0) {
    for (int s = 0; s < BO_QK_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 128);
    tmem_relinquish();
  }
  int n = 0;  // KV tiles that some query of this tile sees: those the kernel above wrote
  for (int t0 = 0; t0 < p.nT; t0 += BO_DQ_THREADS) {
    const int t = t0 + (int)threadIdx.x;
    n += __syncthreads_count(t < p.nT && bo_active<GEN>(p, qt, tmin[t], tmax[t]));
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    uint32_t s = 0;
    bool ok = true;
    for (int t0 = 0; t0 < p.nT && ok; t0 += 32) {
      const int tl = t0 + lane;
      uint32_t act = __ballot_sync(0xffffffffu, tl < p.nT && bo_active<GEN>(p, qt, tmin[tl], tmax[tl]));
      while (act && ok) {
        const int kt = t0 + __ffs(act) - 1;
        act &= act - 1;
        const uint32_t st = s % BO_QK_STAGES;
        if (lane == 0) {
          ok = mbar_wait_bounded(&empty[st], ((s / BO_QK_STAGES) & 1) ^ 1, abort_flag, p.status, STATUS_TIMEOUT_EMPTY);
          if (ok) {
            uint8_t* d = smem + S::RING + st * 2 * BO_TILE;
            mbar_expect_tx(&full[st], BO_TILE + 256 * HD);
            bulk_load(d, p.ds + (((long long)lbg * p.nT + kt) * p.nq + lq) * 16384, BO_TILE, &full[st]);
            tma_load_4d(d + BO_TILE, &tmK, &full[st], 0, kt * 128, g, b);
            if (HD == 128) tma_load_4d(d + BO_TILE + BO_CHUNK, &tmK, &full[st], 64, kt * 128, g, b);
          }
        }
        ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
        ++s;
      }
    }
    if (!ok && lane == 0) {  // let copies in flight land before the CTA's shared memory is released
      long long c0 = clock64();
      while (clock64() - c0 < 2000000LL) {
      }
    }
  } else if (warp == 1) {
    if (n > 0 && elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(128, HD, 1, 1);
      bool ok = true;
      int tr_n = p.trace && blockIdx.x == 0 ? 0 : BO_TRACE_OFF;
      for (int i = 0; i < n && ok; ++i) {
        const int st = i % BO_QK_STAGES;
        if (!(ok = mbar_wait_bounded(&full[st], (i / BO_QK_STAGES) & 1, abort_flag, p.status, STATUS_TIMEOUT_FULL))) break;
        tc_fence_after();
        const uint32_t a = smem_u32(smem + S::RING + st * 2 * BO_TILE), k = a + BO_TILE;
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)  // 16 slots per step
          umma_f16_ss(tmem_base, bo_desc_mn(a + (uint32_t)(kk * 256), 128, 2048),
                      make_smem_desc_sw128(k + (uint32_t)(kk * 16 * 128), BO_CHUNK, 1024), idesc, (i | kk) != 0);
        umma_commit(&empty[st]);
        BO_TRACE(1, 1000000 + i);
      }
      if (ok) umma_commit(acc_full);
    }
  } else {
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const int hq = row / p.npos, tq = qt * p.npos + row % p.npos;
    const bool row_valid = row < p.rows_used && tq < p.T;
    __nv_bfloat16* dst = p.dq + (((long long)b * p.H + g * p.gs + hq) * p.T + tq) * HD;
    bool ok = true;
    if (n > 0) ok = mbar_wait_bounded(acc_full, 0, abort_flag, p.status, STATUS_TIMEOUT_TMEM_FULL);
    tc_fence_after();
    if (ok) {
#pragma unroll 1
      for (int c0 = 0; c0 < HD; c0 += 32) {
        uint32_t r[32];
        if (n > 0) {
          tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0, r);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) r[e] = 0;
        }
        if (row_valid) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            uint4 o;
            o.x = pack_bf16x2(__uint_as_float(r[8 * u + 0]), __uint_as_float(r[8 * u + 1]));
            o.y = pack_bf16x2(__uint_as_float(r[8 * u + 2]), __uint_as_float(r[8 * u + 3]));
            o.z = pack_bf16x2(__uint_as_float(r[8 * u + 4]), __uint_as_float(r[8 * u + 5]));
            o.w = pack_bf16x2(__uint_as_float(r[8 * u + 6]), __uint_as_float(r[8 * u + 7]));
            *reinterpret_cast<uint4*>(dst + c0 + 8 * u) = o;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 128);
  }
}

// Rounds of one call. A round's workspace is pairs · nT · nq tiles of 32 KB; it is kept below a limit, by default 1 GiB, the dS of
// a chunk of 1024 queries x 32 heads over 16384 slots. Query tiles are divided first: every round then still has all (pair, KV
// tile) CTAs, so its last wave stays as full as that of one launch. Below 8 query tiles a round would mostly load and store its
// K, V, dK and dV tiles, and the pairs are divided as well. The least round is one query tile of one pair (32 KB per KV tile).
constexpr long long BO_DS_LIMIT = 1LL << 30;
struct BoRounds {
  int pairs, nq;
  BoRounds(long long bg, long long nT, long long nQT, long long limit) {
    const long long tiles = (limit > 0 ? limit : BO_DS_LIMIT) / BO_TILE;
    const long long least = nQT < 8 ? nQT : 8;
    long long pr = tiles / (nT * least);
    pr = pr < 1 ? 1 : (pr > bg ? bg : pr);
    long long q = tiles / (nT * pr);
    q = q < 1 ? 1 : (q > nQT ? nQT : q);
    const long long n = (nQT + q - 1) / q;
    pairs = (int)pr;
    nq = (int)((nQT + n - 1) / n);  // rounds of nearly equal length
  }
  long long bytes(long long nT) const { return (long long)pairs * nT * nq * BO_TILE; }
};

struct BoLayout {  // scratch: tile_min | tile_max | statistics | head-major copy of dO | dS
  long long stats, dot, ds, total;
  int npos, nT, nQT;
  BoRounds rounds;
  static long long round256(long long n) { return (n + 255) / 256 * 256; }
  BoLayout(int B, int H, int G, int T, int L, long long ds_limit)
      : npos(128 / (H / G)), nT((L + 127) / 128), nQT((T + npos - 1) / npos), rounds((long long)B * G, nT, nQT, ds_limit) {
    stats = round256(2LL * B * G * nT * 4);
    dot = stats + (long long)B * G * nQT * 1024;
    ds = dot + round256((long long)B * H * T * 256);
    total = ds + rounds.bytes(nT);
  }
};

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static int bw_make_tmap_4d(CUtensorMap* tm, const void* ptr, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t d3, uint64_t s1,
                           uint64_t s2, uint64_t s3, uint32_t b0, uint32_t b1, uint32_t b2) {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* pp = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &pp, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
      return KVB_ERR_DRIVER;
    fn = reinterpret_cast<EncodeTiledFn>(pp);
  }
  cuuint64_t dims[4] = {d0, d1, d2, d3};
  cuuint64_t strides[3] = {s1 * 2, s2 * 2, s3 * 2};
  cuuint32_t box[4] = {b0, b1, b2, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? KVB_OK : KVB_ERR_TMAP;
}

// all launches of one call for one (GEN, head size) instantiation; returns their number
template <bool GEN, int HD>
static int bo_launch(const CUtensorMap& tmQ, const CUtensorMap& tmO, const CUtensorMap& tmK, const CUtensorMap& tmV, BoParams p, int BG,
                      const BoRounds& rounds, long long* trace, int trace_mode, cudaStream_t s) {
  static kvb::PerDeviceOnce attr_once;
  if (attr_once.first()) {
    cudaFuncSetAttribute(bwd_dkv_kernel<GEN, HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, BoSmem::TOTAL);
    cudaFuncSetAttribute(bwd_dq_kernel<GEN, HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, BoDqSmem::TOTAL);
  }
  int launches = 0;
  for (int bg0 = 0; bg0 < BG; bg0 += rounds.pairs) {
    const int pairs = min(rounds.pairs, BG - bg0);
    for (int q0 = 0; q0 < p.nQT; q0 += rounds.nq) {
      p.bg0 = bg0; p.q0 = q0; p.nq = min(rounds.nq, p.nQT - q0);
      p.trace = trace_mode == 1 ? trace : nullptr;
      bwd_dkv_kernel<GEN, HD><<<pairs * p.nT, BO_THREADS, BoSmem::TOTAL, s>>>(tmK, tmV, tmQ, tmO, p);
      p.trace = trace_mode == 0 ? trace : nullptr;
      bwd_dq_kernel<GEN, HD><<<pairs * p.nq, BO_DQ_THREADS, BoDqSmem::TOTAL, s>>>(tmK, p);
      launches += 2;
    }
  }
  return launches;
}

}  // namespace kvb

// Optional timeline trace (diagnostics): `buf` holds 3 roles x `cap` events x 2 int64 (tag, SM clock),
// filled by CTA 0 of the dQ launch (mode 0) or the dK/dV launch (mode 1) of every later kvb_sdpa_bwd
// call of this process; buf = NULL switches tracing off. Tags: 1e6+ MMA issuer, 2e6+ compute warp;
// the digits below 1e5 count 64-column halves (dK/dV) or KV tiles (dQ).
static long long* g_bw_trace = nullptr;
static int g_bw_trace_cap = 0, g_bw_trace_mode = 0;
extern "C" int kvb_sdpa_bwd_set_trace(void* buf, int cap, int mode) {
  g_bw_trace = reinterpret_cast<long long*>(buf);
  g_bw_trace_cap = buf ? cap : 0;
  g_bw_trace_mode = mode;
  return KVB_OK;
}

extern "C" long long kvb_sdpa_bwd_scratch_bytes_within(int B, int H, int G, int q_len, int kv_len, long long ds_limit) {
  if (B <= 0 || G <= 0 || q_len <= 0 || kv_len <= 0 || H < G || H / G > 64) return 16;  // refused by the call
  return kvb::BoLayout(B, H, G, q_len, kv_len, ds_limit).total;
}
extern "C" long long kvb_sdpa_bwd_scratch_bytes(int B, int H, int G, int q_len, int kv_len) {
  return kvb_sdpa_bwd_scratch_bytes_within(B, H, G, q_len, kv_len, 0);
}

// head_size: 128 or 64; q_sb, q_sh: batch and head strides of q in elements (0, 0: contiguous (B,H,T,D)); window: sliding
// window in tokens (0: none); softcap: logit soft-capping threshold (0: none), as in the forward. ds_limit: bytes of dS in
// `scratch` (0: 1 GiB), the same as in the question for the scratch size; launches: their number, or NULL.
extern "C" int kvb_sdpa_bwd_ex(const void* q, const void* k, const void* v, const int32_t* token_pos, const void* out,
                               const void* dout, const float* lse, void* dq, float* dk, float* dv, void* scratch, int B, int H,
                               int G, int q_len, int kv_len, int head_size, long long q_sb, long long q_sh, long long k_sb,
                               long long k_sg, long long tp_sb, long long tp_sg, long long dk_sb, long long dk_sg, float scale,
                               int input_pos, int window, float softcap, int* status, void* stream) {
  return kvb_sdpa_bwd_within(q, k, v, token_pos, out, dout, lse, dq, dk, dv, scratch, B, H, G, q_len, kv_len, head_size, q_sb, q_sh,
                             k_sb, k_sg, tp_sb, tp_sg, dk_sb, dk_sg, scale, input_pos, window, softcap, 0, nullptr, status, stream);
}

extern "C" int kvb_sdpa_bwd(const void* q, const void* k, const void* v, const int32_t* token_pos, const void* out,
                            const void* dout, const float* lse, void* dq, float* dk, float* dv, void* scratch, int B, int H,
                            int G, int q_len, int kv_len, long long k_sb, long long k_sg, long long tp_sb, long long tp_sg,
                            long long dk_sb, long long dk_sg, float scale, int input_pos, int* status, void* stream) {
  return kvb_sdpa_bwd_ex(q, k, v, token_pos, out, dout, lse, dq, dk, dv, scratch, B, H, G, q_len, kv_len, 128, 0, 0, k_sb, k_sg,
                         tp_sb, tp_sg, dk_sb, dk_sg, scale, input_pos, 0, 0.f, status, stream);
}

extern "C" int kvb_sdpa_bwd_within(const void* q, const void* k, const void* v, const int32_t* token_pos, const void* out,
                                   const void* dout, const float* lse, void* dq, float* dk, float* dv, void* scratch, int B, int H,
                                   int G, int q_len, int kv_len, int head_size, long long q_sb, long long q_sh, long long k_sb,
                                   long long k_sg, long long tp_sb, long long tp_sg, long long dk_sb, long long dk_sg, float scale,
                                   int input_pos, int window, float softcap, long long ds_limit, int* launches, int* status,
                                   void* stream) {
  using namespace kvb;
  if (B <= 0 || H <= 0 || G <= 0 || q_len <= 0 || kv_len <= 0 || H % G) return KVB_ERR_ARG;
  if (window < 0 || softcap < 0.f || (softcap > 0.f && scale <= 0.f)) return KVB_ERR_ARG;
  if (head_size != 128 && head_size != 64) return KVB_ERR_UNSUPPORTED;
  if (q_sh == 0) q_sh = (long long)q_len * head_size;
  if (q_sb == 0) q_sb = (long long)H * q_sh;
  if ((q_sb % 8) || (q_sh % 8) || q_sh < (long long)q_len * head_size) return KVB_ERR_ALIGN;
  const int gs = H / G;
  if (gs > 64) return KVB_ERR_UNSUPPORTED;  // not tested beyond: such groups fill a tile with one position
  if ((k_sb % 8) || (k_sg % 8) || (dk_sb % 4) || (dk_sg % 4)) return KVB_ERR_ALIGN;
  cudaStream_t s = (cudaStream_t)stream;
  static const int dout_headmajor = [] {
    const char* e = getenv("KVB200_BWD_DOUT_T");  // "0": read dO in place (diagnostics)
    return (e && e[0] == '0') ? 0 : 1;
  }();
  const BoLayout lay(B, H, G, q_len, kv_len, ds_limit);
  uint8_t* sc = reinterpret_cast<uint8_t*>(scratch);
  BoParams p;
  p.G = G; p.H = H; p.T = q_len; p.L = kv_len; p.nT = lay.nT; p.nQT = lay.nQT;
  p.gs = gs; p.npos = lay.npos; p.rows_used = p.npos * gs;
  int32_t* tmin = reinterpret_cast<int32_t*>(sc);
  int32_t* tmax = tmin + (long long)B * G * p.nT;
  float* stats = reinterpret_cast<float*>(sc + lay.stats);
  __nv_bfloat16* dOt = reinterpret_cast<__nv_bfloat16*>(sc + lay.dot);
  p.token_pos = token_pos; p.tile_min = tmin; p.tile_max = tmax; p.stats = stats;
  p.ds = reinterpret_cast<__nv_bfloat16*>(sc + lay.ds);
  p.dq = (__nv_bfloat16*)dq; p.dk = dk; p.dv = dv;
  p.tp_sb = tp_sb; p.tp_sg = tp_sg; p.dk_sb = dk_sb; p.dk_sg = dk_sg;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.input_pos = input_pos; p.status = status;
  p.bg0 = p.q0 = p.nq = 0;
  p.window = window;
  p.cap_pre = softcap > 0.f ? scale / softcap : 0.f;
  p.cap_l2 = softcap * 1.4426950408889634f;
  p.trace = nullptr; p.trace_cap = g_bw_trace_cap;

  // boxes of npos positions x gs heads (Q, dO) or 128 slots (K, V)
  CUtensorMap tmQ, tmO, tmK, tmV;
  int rc;
  const uint64_t hd = (uint64_t)head_size, TD = (uint64_t)q_len * hd, HT = (uint64_t)H * q_len;
  if ((rc = bw_make_tmap_4d(&tmQ, q, hd, q_len, H, B, hd, (uint64_t)q_sh, (uint64_t)q_sb, 64, p.npos, gs))) return rc;
  if (dout_headmajor) {  // the head-major copy that the statistics kernel leaves: runs of positions of one head, as for Q
    if ((rc = bw_make_tmap_4d(&tmO, dOt, hd, q_len, H, B, hd, TD, H * TD, 64, p.npos, gs))) return rc;
  } else {               // dO (B,T,H,D) viewed with dims (D,T,H,B)
    if ((rc = bw_make_tmap_4d(&tmO, dout, hd, q_len, H, B, (uint64_t)H * hd, hd, HT * hd, 64, p.npos, gs))) return rc;
  }
  if ((rc = bw_make_tmap_4d(&tmK, k, hd, kv_len, G, B, hd, k_sg, k_sb, 64, 128, 1))) return rc;
  if ((rc = bw_make_tmap_4d(&tmV, v, hd, kv_len, G, B, hd, k_sg, k_sb, 64, 128, 1))) return rc;
  if ((rc = kvb_att_tile_minmax(token_pos, tmin, tmax, B, G, kv_len, tp_sb, tp_sg, 128, s))) return rc;
  const unsigned blocks = (unsigned)((long long)B * G * p.nQT * 16);  // a warp per packed row
  const __nv_bfloat16 *go = (const __nv_bfloat16*)dout, *o = (const __nv_bfloat16*)out;
  if (head_size == 128) bo_stats_kernel<128><<<blocks, 256, 0, s>>>(go, o, lse, stats, dOt, B, G, H, q_len, gs, p.npos, p.nQT, scale);
  else bo_stats_kernel<64><<<blocks, 256, 0, s>>>(go, o, lse, stats, dOt, B, G, H, q_len, gs, p.npos, p.nQT, scale);
  const bool gen = window > 0 || softcap > 0.f;
  auto launch = head_size == 128 ? (gen ? bo_launch<true, 128> : bo_launch<false, 128>) : (gen ? bo_launch<true, 64> : bo_launch<false, 64>);
  const int n = launch(tmQ, tmO, tmK, tmV, p, B * G, lay.rounds, g_bw_trace, g_bw_trace_mode, s);
  if (launches) *launches = 2 + n;
  return cudaGetLastError() == cudaSuccess ? KVB_OK : KVB_ERR_LAUNCH;
}
