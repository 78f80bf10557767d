// Dense flash attention forward on tcgen05 / TMEM, with an optional fused
// forward-mode tangent (JVP):
//
//   S = Q K^T * scale,  P = softmax(S),  O = P V
//   dS = (dQ K^T + Q dK^T) * scale,  T = P .* dS,
//   dO = (T V + P dV) / l - (rowsum(T) / l) O          (l = rowsum exp)
//
// i.e. the primal, its tangent and the log-sum-exp in ONE pass over K/V, with
// O(L) memory.  Replaces the reference's CuTeDSL mma.sync kernel and Triton
// flash-JVP kernel (reference models/flash_jvp_kernel.py:51-570,
// models/triton_block_jvp.py:228-346) and the FA/SDPA primal forward.
//
// The tangent is attn_jvp.cu's business except for some short problems of more query tiles than SMs,
// see tangent_pairs.  Work item = NT 128-row query tiles that share every 64-row K/V tile, of one (batch,
// head): four tiles in the primal kernel (three or two where rounding L up to 512 rows wastes more
// than that gains or SMs would stand idle, see primal_form), two in the tangent kernel; TMEM (512
// columns) holds no more.  Warps
// 4t .. 4t+3: softmax + O-correction + epilogue of tile t (one query row per thread, rows live
// in TMEM lanes); then one warp with the single-thread tcgen05.mma issuer, one TMA producer
// warp and two warps that only donate registers (setmaxnreg).  The tiles take turns: while
// one tile's softmax runs on the CUDA cores the tensor core works on another.
// The softmax warps are bound by dependency latency (0.4 instructions per cycle and scheduler,
// exponential unit some 70 % busy), so what counts is how many tiles are in flight: B 1, H 4,
// L 29,140 took 1.01 ms with four tiles and 1.08 to 1.16 with three when the row sum was of the
// exact exponentials; as it is now (below) four take 1.04 ms.  Pairs of scores go through packed
// fp32 instructions.  P (and T) are written back to TMEM as bf16 over
// the S (dS) columns and are the A operand of the second GEMM.  O is rescaled lazily (only
// when the running max grows by > 2^8).
//
// Scheduling: a persistent grid whose CTAs take equal shares of the flattened
// (item, K/V tile) space (attn_fwd_split.h); the partial results of split items go
// to a scratch buffer and a small second kernel merges them.
//
// Tensors are (B, L, H, 64) bf16 with arbitrary 16-byte-aligned strides;
// ragged L is handled by TMA zero fill + masking of the last K/V tile.
#include "attn_fwd128.h"
#include "attn_jvp.h"
#include "attn_fwd_split.h"
#include "common.cuh"
#include "host_util.h"

namespace imf {

constexpr int ATT_HD = 64;
constexpr int ATT_TILE_M = 128;

// Work item = NT query tiles of 128 rows that share every K/V tile (64 rows).
//   tangent kernel : NT 2, TMEM per tile S|dS|O|dO
//   primal kernel  : NT 2, 3 or 4, TMEM per tile S|O; or NT 2 with K/V tiles of 128 rows, for items
//                    that are not split (ATT_WIDE)
constexpr int ATT_WIDE = 1;
template <bool TANGENT, int NTP>
struct AttCfg {
  static constexpr bool WIDE = NTP == ATT_WIDE;
  static constexpr int NT = WIDE ? 2 : NTP;
  static constexpr int ITEM_M = NT * ATT_TILE_M;
  static constexpr int BN = WIDE ? 128 : 64;
  static constexpr int NQ = TANGENT ? 2 : 1;       // q + dq
  static constexpr int NKV = TANGENT ? 4 : 2;      // k, v (+ dk, dv)
  static constexpr int V = TANGENT ? 2 : 1;        // v's place: k, v  or  k, dk, v, dv
  static constexpr int STAGES = TANGENT ? 3 : 4;
  static constexpr int SOFT_WARPS = 4 * NT;
  static constexpr int WARP_MMA = SOFT_WARPS, WARP_TMA = SOFT_WARPS + 1;
  // softmax warps + one warpgroup holding the MMA warp, the TMA warp and two warps that
  // only donate registers (setmaxnreg is a warpgroup-wide instruction)
  static constexpr int THREADS = (SOFT_WARPS + 4) * 32;
  static constexpr int REG_SOFT = NT == 2 ? 216 : (NT == 3 ? 136 : 104);
  static constexpr int REG_OTHER = NT == 2 ? 72 : (NT == 3 ? 104 : 64);
  // setmaxnreg.inc draws from what the CTA was launched with (threads x registers per
  // thread as compiled: 168 / 128 / 96 for 384 / 512 / 640 threads); a request beyond
  // that pool blocks for ever
  static constexpr int REG_LAUNCH = NT == 2 ? 168 : (NT == 3 ? 128 : 96);
  static_assert(SOFT_WARPS * 32 * REG_SOFT + (THREADS - SOFT_WARPS * 32) * REG_OTHER <=
                    THREADS * REG_LAUNCH, "register pool exceeded");
  // TMEM columns per query tile
  static constexpr int COL_S = 0;
  static constexpr int COL_DS = BN;
  static constexpr int COL_O = TANGENT ? 2 * BN : BN;
  static constexpr int COL_DO = COL_O + ATT_HD;    // tangent only
  static constexpr int TILE_COLS = TANGENT || WIDE ? 256 : 128;
  static constexpr int TMEM_COLS = 512;
  static constexpr int ACC = TANGENT ? 2 * ATT_HD : ATT_HD;   // fp32 accumulators per row
  static_assert(COL_O + ACC <= TILE_COLS && NT * TILE_COLS <= 512, "");
  static constexpr float PART_COST = WIDE ? 1e9f : (TANGENT ? 0.65f : 0.3f);  // see fwd_share_cost
};

// scratch record of one part of a split item: [ACC][ITEM_M] accumulators (a column per row of the
// record: the softmax threads own a query row each, so a warp stores 128 consecutive bytes), then
// m, l, mu per query row (primal: in mu's place the row sum of the exact exponentials)
template <bool TANGENT, int NTP>
constexpr size_t att_part_floats() {
  return (size_t)AttCfg<TANGENT, NTP>::ITEM_M * (AttCfg<TANGENT, NTP>::ACC + 3);
}

template <bool TANGENT, int NTP>
struct AttSmem {
  using C = AttCfg<TANGENT, NTP>;
  alignas(1024) uint8_t q[C::NQ][C::NT][ATT_TILE_M * 128];           // [q|dq][tile]
  alignas(1024) uint8_t kv[C::STAGES][C::NKV][C::BN * 128];          // k, (dk,) v, (dv)
  uint64_t q_full, q_empty;
  uint64_t kv_full[C::STAGES];
  uint64_t kv_empty[C::STAGES];
  uint64_t s_full[C::NT];
  uint64_t p_full[C::NT];
  uint64_t o_done[C::NT];
  uint64_t o_free[C::NT];
  uint32_t tmem_base;
  int abort_flag;
};

struct AttParams {
  __nv_bfloat16* o;
  __nv_bfloat16* dout;     // tangent output (TANGENT only)
  float* lse;              // (B, H, L) natural-log LSE of scaled scores
  float* scratch;          // split-item partials: records of att_part_floats, two per CTA
  int B, H, L;
  int n_qblk;
  FwdShares sh;
  int64_t o_sb, o_sl, o_sh;   // output strides in elements
  float scale;
  int* status;
};

// The row sum that divides O is taken over P as the tensor core multiplies it, rounded to bf16: the
// rounding errors of a row's weights then cancel in part (with a sum of the exponentials themselves
// the error of O grows by 10 % where few keys carry the weight).  The log-sum-exp wants the exact
// sum; LSE instances of the primal kernel take both (B 1, H 4, L 29,140: 1.07 ms, without 1.04, with
// one exact sum for both 1.01; from the tensor core, three query tiles, 1.12).  The tangent kernel
// takes the exact sum only, as its T = P dS does.
template <bool TANGENT, int NTP, bool LSE>
__global__ void __launch_bounds__(AttCfg<TANGENT, NTP>::THREADS, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_dq,
                const __grid_constant__ CUtensorMap tm_dk,
                const __grid_constant__ CUtensorMap tm_dv, const AttParams p) {
  using C = AttCfg<TANGENT, NTP>;
  constexpr int BN = C::BN;
  extern __shared__ uint8_t smem_raw[];
  auto& s = *reinterpret_cast<AttSmem<TANGENT, NTP>*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cta = blockIdx.x, G = gridDim.x;

  if (threadIdx.x == 0) {
    mbar_init(&s.q_full, 1);
    mbar_init(&s.q_empty, 1);
    for (int i = 0; i < C::STAGES; ++i) {
      mbar_init(&s.kv_full[i], 1);
      mbar_init(&s.kv_empty[i], 1);
    }
    for (int t = 0; t < C::NT; ++t) {
      mbar_init(&s.s_full[t], 1);
      mbar_init(&s.p_full[t], 4);      // one arrival per softmax warp
      mbar_init(&s.o_done[t], 1);
      mbar_init(&s.o_free[t], 4);
    }
    s.abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == C::WARP_MMA) {
    tmem_alloc(&s.tmem_base, C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s.tmem_base;
  volatile int* abort_flag = &s.abort_flag;

  if (warp >= C::SOFT_WARPS) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::REG_OTHER));
    if (warp == C::WARP_TMA) {
      // ---------------------------------------------------- TMA producer --
      if (elect_one()) {
        prefetch_tmap(&tm_q);
        prefetch_tmap(&tm_k);
        prefetch_tmap(&tm_v);
        long kv_it = 0;
        Segment sg;
        bool ok = true;
        for (int si = 0; ok && get_segment(p.sh, cta, G, si, sg); ++si) {
          const int qb = sg.item % p.n_qblk, h = (sg.item / p.n_qblk) % p.H,
                    b = sg.item / (p.n_qblk * p.H);
          const int q0 = qb * C::ITEM_M;
          if (si > 0) ok = mbar_wait(&s.q_empty, (si - 1) & 1, abort_flag, p.status, STATUS_TIMEOUT_EMPTY);
          if (!ok) break;
          mbar_arrive_expect_tx(&s.q_full, C::NQ * C::NT * ATT_TILE_M * 128);
          for (int t = 0; t < C::NT; ++t) {
            tma_load_4d(s.q[0][t], &tm_q, &s.q_full, 0, h, q0 + t * ATT_TILE_M, b);
            if (TANGENT)
              tma_load_4d(s.q[C::NQ - 1][t], &tm_dq, &s.q_full, 0, h, q0 + t * ATT_TILE_M, b);
          }
          for (int j = sg.j0; j < sg.j1; ++j, ++kv_it) {
            const int st = (int)(kv_it % C::STAGES);
            if (kv_it >= C::STAGES) {
              ok = mbar_wait(&s.kv_empty[st], (uint32_t)((kv_it / C::STAGES) & 1) ^ 1, abort_flag,
                             p.status, STATUS_TIMEOUT_EMPTY);
              if (!ok) break;
            }
            mbar_arrive_expect_tx(&s.kv_full[st], C::NKV * BN * 128);
            tma_load_4d(s.kv[st][0], &tm_k, &s.kv_full[st], 0, h, j * BN, b);
            if (TANGENT) tma_load_4d(s.kv[st][1], &tm_dk, &s.kv_full[st], 0, h, j * BN, b);
            tma_load_4d(s.kv[st][C::V], &tm_v, &s.kv_full[st], 0, h, j * BN, b);
            if (TANGENT) tma_load_4d(s.kv[st][C::NKV - 1], &tm_dv, &s.kv_full[st], 0, h, j * BN, b);
          }
        }
      }
    } else if (warp == C::WARP_MMA) {
      // ------------------------------------------------------ MMA issuer --
      if (elect_one()) {
        // Tangent: k | dk and v | dv lie next to one another in shared memory, and S | dS and
        // O | dO in TMEM, so Q [K | dK]^T and P [V | dV] are one N = 128 product each.  An SM
        // reads 128 B of operands per clock: M = N = 128 with both operands in shared memory
        // needs 8 KB per 64 clocks, exactly that rate, where two N = 64 products need 6 KB per
        // 32 clocks each and wait for them.
        constexpr uint32_t idesc_qk = idesc_bf16(ATT_TILE_M, TANGENT ? 2 * BN : BN, 0, 0);
        constexpr uint32_t idesc_dqk = idesc_bf16(ATT_TILE_M, BN, 0, 0);
        constexpr uint32_t idesc_pv = idesc_bf16(ATT_TILE_M, C::ACC, 0, 1);
        constexpr uint32_t idesc_tv = idesc_bf16(ATT_TILE_M, ATT_HD, 0, 1);
        auto issue_qk = [&](int t, int st, uint64_t* done) {
          const uint32_t tb = tmem + t * C::TILE_COLS;
          const uint32_t qa = smem_u32(s.q[0][t]), ka = smem_u32(s.kv[st][0]);
#pragma unroll
          for (int ks = 0; ks < ATT_HD / 16; ++ks)
            mma_ss(tb + C::COL_S, sdesc_kmajor(qa + ks * 32), sdesc_kmajor(ka + ks * 32), idesc_qk,
                   ks != 0);
          if (TANGENT) {
            const uint32_t dqa = smem_u32(s.q[C::NQ - 1][t]);
#pragma unroll
            for (int ks = 0; ks < ATT_HD / 16; ++ks)
              mma_ss(tb + C::COL_DS, sdesc_kmajor(dqa + ks * 32), sdesc_kmajor(ka + ks * 32),
                     idesc_dqk, 1);
          }
          tc_commit(done);
        };
        auto issue_pv = [&](int t, int st, bool first) {
          const uint32_t tb = tmem + t * C::TILE_COLS;
          const uint32_t va = smem_u32(s.kv[st][C::V]);
#pragma unroll
          for (int ks = 0; ks < BN / 16; ++ks)
            mma_ts(tb + C::COL_O, tb + C::COL_S + ks * 8, sdesc_mnmajor(va + ks * 2048, BN * 128),
                   idesc_pv, !(first && ks == 0));
          if (TANGENT) {
#pragma unroll
            for (int ks = 0; ks < BN / 16; ++ks)
              mma_ts(tb + C::COL_DO, tb + C::COL_DS + ks * 8,
                     sdesc_mnmajor(va + ks * 2048, BN * 128), idesc_tv, 1);
          }
          tc_commit(&s.o_done[t]);
        };
        long kv_it = 0, it = 0;
        Segment sg;
        bool ok = true;
        for (int si = 0; ok && get_segment(p.sh, cta, G, si, sg); ++si) {
          const int n_j = sg.j1 - sg.j0;
          ok = mbar_wait(&s.q_full, si & 1, abort_flag, p.status, STATUS_TIMEOUT_TMA) &&
               mbar_wait(&s.kv_full[kv_it % C::STAGES], (uint32_t)((kv_it / C::STAGES) & 1),
                         abort_flag, p.status, STATUS_TIMEOUT_TMA);
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int t = 0; t < C::NT; ++t) issue_qk(t, (int)(kv_it % C::STAGES), &s.s_full[t]);
          if (n_j == 1) tc_commit(&s.q_empty);
          for (int jj = 0; jj < n_j && ok; ++jj, ++kv_it, ++it) {
            const int st = (int)(kv_it % C::STAGES), st1 = (int)((kv_it + 1) % C::STAGES);
            // the next K/V tile, loaded long ago: seen now, not between P V and the next Q K^T (a
            // wait costs some 200 clocks even when there is nothing to wait for)
            if (jj + 1 < n_j) {
              ok = mbar_wait(&s.kv_full[st1], (uint32_t)(((kv_it + 1) / C::STAGES) & 1), abort_flag,
                             p.status, STATUS_TIMEOUT_TMA);
              if (!ok) break;
            }
#pragma unroll
            for (int t = 0; t < C::NT; ++t) {
              if (!ok) break;
              ok = mbar_wait(&s.p_full[t], (uint32_t)(it & 1), abort_flag, p.status,
                             STATUS_TIMEOUT_SOFTMAX);
              if (ok && jj == 0 && si > 0)   // epilogue of the previous segment has drained O
                ok = mbar_wait(&s.o_free[t], (uint32_t)((si - 1) & 1), abort_flag, p.status,
                               STATUS_TIMEOUT_SOFTMAX);
              if (!ok) break;
              tc_fence_after();
              issue_pv(t, st, jj == 0);
              if (t == C::NT - 1) tc_commit(&s.kv_empty[st]);
              if (jj + 1 < n_j) {
                issue_qk(t, st1, &s.s_full[t]);
                if (t == C::NT - 1 && jj + 2 == n_j) tc_commit(&s.q_empty);   // last Q read of the item
              }
            }
          }
        }
      }
    }
  } else {
    // ------------------------------------- softmax / correction / epilogue --
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::REG_SOFT));
    const int t = warp >> 2;
    const int wl = warp & 3;
    const int row_in_item = t * ATT_TILE_M + wl * 32 + lane;
    const uint32_t tb = tmem_addr(tmem, wl * 32, t * C::TILE_COLS);
    const float scale_log2 = p.scale * 1.4426950408889634f;
    long it = 0;
    Segment sg;
    bool ok = true;
    for (int si = 0; ok && get_segment(p.sh, cta, G, si, sg); ++si) {
      const int qb = sg.item % p.n_qblk, h = (sg.item / p.n_qblk) % p.H,
                b = sg.item / (p.n_qblk * p.H);
      const int q_row = qb * C::ITEM_M + row_in_item;
      float m_used = -INFINITY, l_sum = 0.f, l_sum2 = 0.f, mu_sum = 0.f, mu_sum2 = 0.f;
      for (int j = sg.j0; j < sg.j1 && ok; ++j, ++it) {
        ok = __all_sync(0xffffffffu, mbar_wait(&s.s_full[t], (uint32_t)(it & 1), abort_flag,
                                               p.status, STATUS_TIMEOUT_MMA));
        if (!ok) break;
        tc_fence_after();
        const int kv_rem = p.L - j * BN;
        if constexpr (TANGENT) {
          // P = exp2(S scale - m) is computed against the reference maximum that the rows already
          // have while the maximum of the new scores is taken alongside: the chain S -> max -> exp
          // becomes S -> exp.  Only when a row has outgrown its reference by more than 2^8 (or has
          // none yet) is the reference moved, O rescaled and the tile, still in TMEM, done again.
          // (Measured where this form still took long problems, B 1, H 4, L 29,140: 2.23 -> 2.12 ms.  The
          // primal kernel, with four warps per scheduler to fill the gaps, gets slower this way:
          // 1.08 -> 1.31 ms.)
          const bool first = j == sg.j0;
          uint32_t pk[BN / 2];
          uint32_t tk[BN / 2];
          float alpha = 1.f;
          f32x2 l_new, mu_new;
          for (bool redo = false;; redo = true) {
            const f32x2 neg_m2 = dup2(-m_used * scale_log2);
            l_new = mu_new = dup2(0.f);
            float mx0 = -INFINITY, mx1 = -INFINITY;
            // 32-column chunks, the next one on its way from TMEM while one is worked on
            uint32_t sv[2][32], dsv[2][32];
            tmem_ld32(tb + C::COL_S, sv[0]);
            tmem_ld32(tb + C::COL_DS, dsv[0]);
            tc_wait_ld();
#pragma unroll
            for (int c = 0; c < BN; c += 32) {
              uint32_t* s_ = sv[(c / 32) & 1];
              const uint32_t* d_ = dsv[(c / 32) & 1];
              if (c + 32 < BN) {
                tmem_ld32(tb + C::COL_S + c + 32, sv[((c / 32) & 1) ^ 1]);
                tmem_ld32(tb + C::COL_DS + c + 32, dsv[((c / 32) & 1) ^ 1]);
              }
              if (kv_rem < c + 32) {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                  if (c + i >= kv_rem) s_[i] = 0xff800000u;  // -inf
              }
#pragma unroll
              for (int i = 0; i < 32; i += 2) {
                float& mx = (i & 2) ? mx1 : mx0;
                asm("max.f32 %0, %0, %1, %2;" : "+f"(mx) : "f"(__uint_as_float(s_[i])), "f"(__uint_as_float(s_[i + 1])));
                const f32x2 e = fma2(pair2(s_[i], s_[i + 1]), dup2(scale_log2), neg_m2);
                const float p0 = ex2(lo2(e)), p1 = ex2(hi2(e));
                pk[(c + i) / 2] = pack_bf16(p0, p1);
                const f32x2 pp = pair2(__float_as_uint(p0), __float_as_uint(p1));
                l_new = add2(l_new, pp);
                const f32x2 tt = mul2(mul2(pp, pair2(d_[i], d_[i + 1])), dup2(p.scale));
                mu_new = add2(mu_new, tt);
                tk[(c + i) / 2] = pack_bf16(lo2(tt), hi2(tt));
              }
              if (c + 32 < BN) tc_wait_ld();
            }
            if (redo) break;
            const float mx = fmaxf(mx0, mx1);
            const bool need = first || (mx - m_used) * scale_log2 > 8.0f;
            if (!__any_sync(0xffffffffu, need)) break;
            if (need) {
              if (!first) alpha = ex2((m_used - mx) * scale_log2);
              m_used = mx;
            }
            if (first) continue;               // nothing in O yet
            ok = __all_sync(0xffffffffu, mbar_wait(&s.o_done[t], (uint32_t)((it - 1) & 1),
                                                   abort_flag, p.status, STATUS_TIMEOUT_MMA));
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < C::ACC; c += 32) {
              uint32_t ov[32];
              tmem_ld32(tb + C::COL_O + c, ov);
              tc_wait_ld();
#pragma unroll
              for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
              tmem_st32(tb + C::COL_O + c, ov);
            }
            tc_wait_st();
          }
          if (!ok) break;
          l_sum = fmaf(l_sum, alpha, lo2(l_new));
          l_sum2 = fmaf(l_sum2, alpha, hi2(l_new));
          mu_sum = fmaf(mu_sum, alpha, lo2(mu_new));
          mu_sum2 = fmaf(mu_sum2, alpha, hi2(mu_new));
#pragma unroll
          for (int c = 0; c < BN; c += 64) {
            tmem_st32(tb + C::COL_S + c / 2, pk + c / 2);
            tmem_st32(tb + C::COL_DS + c / 2, tk + c / 2);
          }
        } else {
          // Maximum first, then the exponentials, with the scores read from TMEM again in between:
          // 64 scores held across the vote do not fit the registers of four tiles' warps.
          float mx0 = -INFINITY, mx1 = -INFINITY;
          auto load = [&](int c, uint32_t* x) {
            tmem_ld32(tb + C::COL_S + c, x);
          };
          auto mask = [&](int c, uint32_t* x) {
            if (kv_rem < c + 32) {
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (c + i >= kv_rem) x[i] = 0xff800000u;  // -inf
            }
          };
          {
            uint32_t sv[BN / 32][32];
#pragma unroll
            for (int c = 0; c < BN; c += 32) load(c, sv[c / 32]);
            tc_wait_ld();
#pragma unroll
            for (int c = 0; c < BN; c += 32) {
              const uint32_t* x = sv[c / 32];
              mask(c, sv[c / 32]);
#pragma unroll
              for (int i = 0; i < 32; i += 4) {
                asm("max.f32 %0, %0, %1, %2;" : "+f"(mx0) : "f"(__uint_as_float(x[i])), "f"(__uint_as_float(x[i + 1])));
                asm("max.f32 %0, %0, %1, %2;" : "+f"(mx1) : "f"(__uint_as_float(x[i + 2])), "f"(__uint_as_float(x[i + 3])));
              }
            }
          }
          const float mx = fmaxf(mx0, mx1);
          if (j == sg.j0) {
            m_used = mx;
          } else {
            const bool need = (mx - m_used) * scale_log2 > 8.0f;
            if (__any_sync(0xffffffffu, need)) {
              float alpha = 1.f;
              if (need) {
                alpha = ex2((m_used - mx) * scale_log2);
                m_used = mx;
              }
              l_sum *= alpha;
              l_sum2 *= alpha;
              mu_sum *= alpha;
              mu_sum2 *= alpha;
              ok = __all_sync(0xffffffffu, mbar_wait(&s.o_done[t], (uint32_t)((it - 1) & 1),
                                                     abort_flag, p.status, STATUS_TIMEOUT_MMA));
              if (!ok) break;
              tc_fence_after();
#pragma unroll
              for (int c = 0; c < C::ACC; c += 32) {
                uint32_t ov[32];
                tmem_ld32(tb + C::COL_O + c, ov);
                tc_wait_ld();
#pragma unroll
                for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
                tmem_st32(tb + C::COL_O + c, ov);
              }
              tc_wait_st();
            }
          }
          const f32x2 neg_m2 = dup2(-m_used * scale_log2);
          f32x2 exact2 = pair2(__float_as_uint(mu_sum), __float_as_uint(mu_sum2));
#pragma unroll
          for (int c = 0; c < BN; c += 32) {
            uint32_t x[32], pk[16];
            load(c, x);
            tc_wait_ld();
            mask(c, x);
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              const f32x2 e = fma2(pair2(x[i], x[i + 1]), dup2(scale_log2), neg_m2);
              const float p0 = ex2(lo2(e)), p1 = ex2(hi2(e));
              pk[i / 2] = pack_bf16(p0, p1);
              l_sum = add_bf16(pk[i / 2], l_sum);
              l_sum2 = add_bf16(pk[i / 2] >> 16, l_sum2);
              if (LSE) exact2 = add2(exact2, pair2(__float_as_uint(p0), __float_as_uint(p1)));
            }
            tmem_st16(tb + C::COL_S + c / 2, pk);
          }
          if (LSE) {
            mu_sum = lo2(exact2);
            mu_sum2 = hi2(exact2);
          }
        }
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s.p_full[t]);
      }
      // ---- epilogue of this segment ----
      if (ok)
        ok = mbar_wait(&s.o_done[t], (uint32_t)((it - 1) & 1), abort_flag, p.status,
                       STATUS_TIMEOUT_MMA);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const float l_tot = l_sum + l_sum2, mu_tot = mu_sum + mu_sum2;
      const bool live = q_row < p.L;
      if (sg.rec < 0) {
        const float inv_l = 1.f / l_tot;
        const int64_t off = (int64_t)b * p.o_sb + (int64_t)q_row * p.o_sl + (int64_t)h * p.o_sh;
#pragma unroll
        for (int c = 0; c < ATT_HD; c += 32) {
          uint32_t ov[32];
          tmem_ld32(tb + C::COL_O + c, ov);
          tc_wait_ld();
          uint32_t ob[16];
#pragma unroll
          for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * inv_l);
#pragma unroll
          for (int i = 0; i < 16; ++i)
            ob[i] = pack_bf16(__uint_as_float(ov[2 * i]), __uint_as_float(ov[2 * i + 1]));
          if (live) {
            uint4* dst = reinterpret_cast<uint4*>(p.o + off + c);
#pragma unroll
            for (int i = 0; i < 4; ++i)
              dst[i] = make_uint4(ob[4 * i], ob[4 * i + 1], ob[4 * i + 2], ob[4 * i + 3]);
          }
          if (TANGENT) {
            uint32_t dv_[32];
            tmem_ld32(tb + C::COL_DO + c, dv_);
            tc_wait_ld();
            const float mul = mu_tot * inv_l;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const float d0 = __uint_as_float(dv_[2 * i]) * inv_l - mul * __uint_as_float(ov[2 * i]);
              const float d1 =
                  __uint_as_float(dv_[2 * i + 1]) * inv_l - mul * __uint_as_float(ov[2 * i + 1]);
              ob[i] = pack_bf16(d0, d1);
            }
            if (live) {
              uint4* dst = reinterpret_cast<uint4*>(p.dout + off + c);
#pragma unroll
              for (int i = 0; i < 4; ++i)
                dst[i] = make_uint4(ob[4 * i], ob[4 * i + 1], ob[4 * i + 2], ob[4 * i + 3]);
            }
          }
        }
        if (LSE && live && p.lse)
          p.lse[((int64_t)b * p.H + h) * p.L + q_row] =
              m_used * p.scale + __logf(TANGENT ? l_tot : mu_tot);
      } else {
        // partial result of a split item: raw accumulators + (m, l, mu; primal: the exact row sum)
        float* part = p.scratch + (size_t)sg.rec * att_part_floats<TANGENT, NTP>();
#pragma unroll
        for (int c = 0; c < C::ACC; c += 32) {
          uint32_t ov[32];
          tmem_ld32(tb + C::COL_O + c, ov);
          tc_wait_ld();
          float* acc = part + (size_t)c * C::ITEM_M + row_in_item;
#pragma unroll
          for (int i = 0; i < 32; ++i) acc[i * C::ITEM_M] = __uint_as_float(ov[i]);
        }
        float* stats = part + (size_t)C::ITEM_M * C::ACC;
        stats[row_in_item] = m_used;
        stats[C::ITEM_M + row_in_item] = l_tot;
        stats[2 * C::ITEM_M + row_in_item] = mu_tot;
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s.o_free[t]);
    }
    tc_fence_before();
  }
  __syncthreads();
  if (warp == C::WARP_MMA) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, C::TMEM_COLS);
  }
}

template <bool TANGENT, int NTP>
__global__ void __launch_bounds__(32 * ATT_HD / COMBINE_COLS)
attn_fwd_combine_kernel(const AttParams p, int G) {
  combine_split_items<ATT_HD, AttCfg<TANGENT, NTP>::ITEM_M, TANGENT>(p, G);
}

static int make_qkv_map(CUtensorMap* m, const void* ptr, int B, int L, int H, int64_t sb,
                        int64_t sl, int64_t sh, int rows) {
  uint64_t dims[4] = {(uint64_t)ATT_HD, (uint64_t)H, (uint64_t)L, (uint64_t)B};
  uint64_t str[4] = {2, (uint64_t)sh * 2, (uint64_t)sl * 2, (uint64_t)sb * 2};
  uint32_t box[4] = {(uint32_t)ATT_HD, 1, (uint32_t)rows, 1};
  return make_tmap(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), dims, str, box);
}

template <bool TANGENT, int NTP>
static int launch_attn_fwd(const void* q, const void* k, const void* v, const void* dq,
                           const void* dk, const void* dv, const int64_t* strides, AttParams prm,
                           size_t scratch_bytes, cudaStream_t stream) {
  using C = AttCfg<TANGENT, NTP>;
  CUtensorMap mq, mk, mv, mdq, mdk, mdv;
  int rc;
  const int B = prm.B, L = prm.L, H = prm.H;
  prm.n_qblk = (L + C::ITEM_M - 1) / C::ITEM_M;
  prm.sh.n_items = prm.n_qblk * H * B;
  prm.sh.n_kv = (L + C::BN - 1) / C::BN;
  prm.sh.total = (long)prm.sh.n_items * prm.sh.n_kv;
  const int G = fwd_grid(prm.sh.n_items, prm.sh.n_kv, C::PART_COST, prm.scratch,
                         scratch_bytes / sizeof(float), att_part_floats<TANGENT, NTP>());
  if (G == 0) return IMF_ERR_ARG;
  // strides: [q_sb,q_sl,q_sh, k_sb,k_sl,k_sh, v_sb,v_sl,v_sh, dq.., dk.., dv..]
  if ((rc = make_qkv_map(&mq, q, B, L, H, strides[0], strides[1], strides[2], ATT_TILE_M))) return rc;
  if ((rc = make_qkv_map(&mk, k, B, L, H, strides[3], strides[4], strides[5], C::BN))) return rc;
  if ((rc = make_qkv_map(&mv, v, B, L, H, strides[6], strides[7], strides[8], C::BN))) return rc;
  if (TANGENT) {
    if ((rc = make_qkv_map(&mdq, dq, B, L, H, strides[9], strides[10], strides[11], ATT_TILE_M)))
      return rc;
    if ((rc = make_qkv_map(&mdk, dk, B, L, H, strides[12], strides[13], strides[14], C::BN)))
      return rc;
    if ((rc = make_qkv_map(&mdv, dv, B, L, H, strides[15], strides[16], strides[17], C::BN)))
      return rc;
  } else {
    mdq = mq;
    mdk = mk;
    mdv = mv;
  }
  const bool lse = TANGENT || prm.lse != nullptr;
  auto kern = lse ? attn_fwd_kernel<TANGENT, NTP, true> : attn_fwd_kernel<TANGENT, NTP, TANGENT>;
  const size_t smem = sizeof(AttSmem<TANGENT, NTP>) + 1024;
  static bool smem_set[2][HOST_MAX_DEVICES] = {{false}};
  if (!allow_smem((const void*)kern, smem, smem_set[lse])) return IMF_ERR_LAUNCH;
  kern<<<G, C::THREADS, smem, stream>>>(mq, mk, mv, mdq, mdk, mdv, prm);
  if (cudaGetLastError() != cudaSuccess) return IMF_ERR_LAUNCH;
  if (G != prm.sh.n_items) {
    const dim3 grid(G - 1, C::ITEM_M / COMBINE_ROWS);
    attn_fwd_combine_kernel<TANGENT, NTP><<<grid, 32 * ATT_HD / COMBINE_COLS, 0, stream>>>(prm, G);
    if (cudaGetLastError() != cudaSuccess) return IMF_ERR_LAUNCH;
  }
  return IMF_OK;
}

template <bool TANGENT, int NTP>
static size_t att_scratch_bytes(int B, int L, int H) {
  using C = AttCfg<TANGENT, NTP>;
  const long n_items = (long)((L + C::ITEM_M - 1) / C::ITEM_M) * H * B;
  const int G = fwd_grid(n_items, (L + C::BN - 1) / C::BN, C::PART_COST);
  return G == n_items ? 0 : (size_t)G * 2 * att_part_floats<TANGENT, NTP>() * sizeof(float);
}

// With tangent: one query tile per item (attn_jvp.cu) is 1.1 to 2 times faster than two, but a CTA's
// next item costs 5 us more than its K/V tiles.  So two where that counts:
//  - the tiles are more than the SMs, pairs are not, and walks are of nine K/V tiles at most: H 80, L 133
//    12.5 us against 16.0; B 3, H 40, L 205 14.8 and 16.9; H 48, L 576 24.0 and 24.6; B 3, H 16, L 955 32.9 and 32.8;
//  - walks of three K/V tiles in many rounds.  A round of tiles costs 6.3 us there, pairs 16.5 us and 8.1 us for
//    each of the SMs' number: B 8, H 128, L 145 (13.8 tiles an SM) 74.6 us against 82.5; B 6, H 80, L 143 (6.5)
//    44.5 and 48.3; B 16, H 32, L 137 (6.9) 45.2 and 43.2.  Of four K/V tiles pairs take 75 us and tiles 72
//    at 10.4 an SM, B 12, H 64, L 200.
static bool tangent_pairs(int B, int L, int H) {
  const long pairs = (long)((L + 2 * ATT_TILE_M - 1) / (2 * ATT_TILE_M)) * H * B;
  const long tiles = (long)((L + ATT_TILE_M - 1) / ATT_TILE_M) * H * B;
  const int sms = fwd_sm_count(), n_kv = (L + AttCfg<true, 2>::BN - 1) / AttCfg<true, 2>::BN;
  if (tiles <= sms) return false;
  if (pairs <= sms) return n_kv <= 9;
  const long rounds = (tiles + sms - 1) / sms;
  return n_kv == 3 && (float)rounds > 2.7f + 1.3f * (float)pairs / (float)sms;
}

static long primal_items(int B, int L, int H, int form) {
  const int item_m = (form == ATT_WIDE ? 2 : form) * ATT_TILE_M;
  return (long)((L + item_m - 1) / item_m) * H * B;
}

// Form of the primal kernel's work items: of two, three and four query tiles, and two with K/V tiles of
// 128 rows (never split), the one with the least time by the following account.  A K/V tile takes
// 1.13, 1.26 and 1.46 us (1.95 for the double one), so that with many items four are the best
// (B 1, H 4, L 29,140: 1.01 ms, three 1.16, both with exact row sums) unless rounding L up to 512 rows
// wastes more than that gains; with few items, SMs that would stand idle take smaller ones
// (H 4, L 532: two 15.7 us, three 17.3, four 20.5), and long walks the double tiles (H 24, L 1,000:
// 23.0 us against 25.5 and, three, 29.9).  A launch takes 5 to 7 us besides, and the merge of split
// items that are more than the SMs six tiles.  (165 shapes of 1 to 64 heads and 130 to 7,820 rows:
// 0.4 % from the best form on average.)
static int primal_form(int B, int L, int H) {
  constexpr int FORMS[4] = {2, 3, 4, ATT_WIDE};
  constexpr float TILE_US[4] = {1.13f, 1.26f, 1.46f, 1.95f}, BASE_US[4] = {5.1f, 6.5f, 7.0f, 5.7f};
  constexpr float PART_COST = AttCfg<false, 4>::PART_COST;
  const int sms = fwd_sm_count();
  int best = 4;
  if (B <= 0 || L <= 0 || H <= 0) return best;      // refused at the launch
  float best_us = 1e30f;
  for (int f = 0; f < 4; ++f) {
    const bool wide = FORMS[f] == ATT_WIDE;
    const long items = primal_items(B, L, H, FORMS[f]);
    const int bn = wide ? AttCfg<false, ATT_WIDE>::BN : AttCfg<false, 4>::BN, n_kv = (L + bn - 1) / bn;
    if (wide && items > sms) continue;
    const int g = wide ? (int)items : fwd_grid(items, n_kv, PART_COST);
    const float walk = (float)((items * n_kv + g - 1) / g);
    const float tiles = items > sms ? walk + 6.f
                        : g == items ? walk : walk + fwd_share_cost(items, n_kv, g, PART_COST);
    const float us = BASE_US[f] + TILE_US[f] * tiles;
    if (us < best_us) {
      best = FORMS[f];
      best_us = us;
    }
  }
  return best;
}

}  // namespace imf

// Bytes of scratch the forward takes for (B, L, H): 0 when no item is split.
extern "C" long imf_attn_fwd_scratch_bytes(int B, int L, int H, int tangent) {
  using namespace imf;
  if (B <= 0 || L <= 0 || H <= 0) return 0;       // refused at the launch
  if (tangent)
    return tangent_pairs(B, L, H) ? (long)att_scratch_bytes<true, 2>(B, L, H) : attn_jvp_scratch_bytes(B, L, H);
  switch (primal_form(B, L, H)) {
    case ATT_WIDE: return 0;
    case 2: return (long)att_scratch_bytes<false, 2>(B, L, H);
    case 3: return (long)att_scratch_bytes<false, 3>(B, L, H);
    default: return (long)att_scratch_bytes<false, 4>(B, L, H);
  }
}

// Same for either head_dim (64 or 128).
extern "C" long imf_attn_fwd_scratch_bytes_hd(int B, int L, int H, int tangent, int head_dim) {
  if (head_dim == 128) return imf::attn_fwd128_scratch_bytes(B, L, H, tangent);
  return imf_attn_fwd_scratch_bytes(B, L, H, tangent);
}

// Dense attention forward (+ optional tangent).  All tensors (B, L, H, head_dim)
// bf16, head_dim 64 or 128; `strides` holds (batch, row, head) element strides for q, k, v and,
// when tangents are given, dq, dk, dv.  o/dout contiguous-in-last-dim with
// strides (o_sb, o_sl, o_sh).  lse: (B, H, L) fp32 or null.  scratch: device
// buffer of imf_attn_fwd_scratch_bytes_hd() bytes.  With less (or null), problems that need some run
// without where their work items are no more than the SMs, one CTA per item, and are refused
// otherwise.  head_dim 64 with tangent: where pairs of 128-row query tiles, ceil(L / 256) H B, are no
// more than the SMs; the CTAs take whole items, tiles in rounds if need be.
extern "C" int imf_attn_fwd(const void* q, const void* k, const void* v, const void* dq,
                            const void* dk, const void* dv, void* o, void* dout, float* lse,
                            int B, int L, int H, int head_dim, const int64_t* strides,
                            int64_t o_sb, int64_t o_sl, int64_t o_sh, float scale, void* scratch,
                            long scratch_bytes, int* status, void* stream) {
  using namespace imf;
  if ((head_dim != ATT_HD && head_dim != 128) || B <= 0 || L <= 0 || H <= 0) return IMF_ERR_ARG;
  if ((o_sl & 7) || (o_sh & 7) || (o_sb & 7) || (reinterpret_cast<uintptr_t>(o) & 15))
    return IMF_ERR_ARG;
  if (dq != nullptr && (dout == nullptr || (reinterpret_cast<uintptr_t>(dout) & 15))) return IMF_ERR_ARG;
  if (head_dim == 128 || (dq != nullptr && !tangent_pairs(B, L, H))) {
    Fwd128Args a{q, k, v, dq, dk, dv, o, dout, lse, B, L, H, strides, o_sb, o_sl, o_sh, scale,
                 scratch, scratch_bytes, status, stream};
    return head_dim == 128 ? attn_fwd128_launch(a) : attn_jvp_launch(a);
  }
  AttParams prm;
  prm.o = static_cast<__nv_bfloat16*>(o);
  prm.dout = static_cast<__nv_bfloat16*>(dout);
  prm.lse = lse;
  prm.scratch = static_cast<float*>(scratch);
  prm.B = B;
  prm.H = H;
  prm.L = L;
  prm.o_sb = o_sb;
  prm.o_sl = o_sl;
  prm.o_sh = o_sh;
  prm.scale = scale;
  prm.status = status;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dq != nullptr) {
    return launch_attn_fwd<true, 2>(q, k, v, dq, dk, dv, strides, prm, (size_t)scratch_bytes, st);
  }
#define IMF_PRIMAL(NT)                                                                              \
  return launch_attn_fwd<false, NT>(q, k, v, nullptr, nullptr, nullptr, strides, prm,               \
                                    (size_t)scratch_bytes, st)
  switch (primal_form(B, L, H)) {
    case ATT_WIDE: IMF_PRIMAL(ATT_WIDE);
    case 2: IMF_PRIMAL(2);
    case 3: IMF_PRIMAL(3);
    default: IMF_PRIMAL(4);
  }
#undef IMF_PRIMAL
}

// ---------------------------------------------------------------------------
// Allocation-free entry point (see attn_noalloc.h for who needs it and why).
// ---------------------------------------------------------------------------
#include "attn_noalloc.h"

namespace imf {
constexpr size_t NOALLOC_FLOATS =
    (size_t)IMF_ATTN_NOALLOC_MAX_CTAS * 2 * ((size_t)AttCfg<false, 4>::ITEM_M * (ATT_HD + 3));
// Split-item partials of the primal forward.  In host code this name is only a
// stand-in for the symbol, not a device address: the address comes from
// cudaGetSymbolAddress below.
static __device__ __align__(256) float g_attn_noalloc_scratch[NOALLOC_FLOATS];
}  // namespace imf

extern "C" int imf_attn_fwd_noalloc(const void* q, const void* k, const void* v, void* o,
                                    float* lse, int B, int L, int H, int head_dim,
                                    const int64_t* strides, int64_t o_sb, int64_t o_sl,
                                    int64_t o_sh, float scale, int* status, void* stream) {
  using namespace imf;
  static_assert(NOALLOC_FLOATS == (size_t)IMF_ATTN_NOALLOC_MAX_CTAS * 2 * att_part_floats<false, 4>(),
                "scratch array and partial record size disagree");
  constexpr int MAX_DEVICES = 64;
  static float* scratch_of_device[MAX_DEVICES] = {nullptr};
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return IMF_ERR_DRIVER;
  if (scratch_of_device[dev] == nullptr) {
    // once per device, with that device current; do this outside stream capture
    void* ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, g_attn_noalloc_scratch) != cudaSuccess || ptr == nullptr) {
      fprintf(stderr, "imf_attn_fwd_noalloc: cudaGetSymbolAddress failed on device %d\n", dev);
      return IMF_ERR_DRIVER;
    }
    scratch_of_device[dev] = static_cast<float*>(ptr);
  }
  if (head_dim != ATT_HD) return IMF_ERR_ARG;     // the built-in scratch is sized for head_dim 64
  // problems of no more items than SMs leave the array alone (one CTA per item), so that short calls
  // on several streams share nothing
  const bool shares = B > 0 && L > 0 && H > 0 &&
                      primal_items(B, L, H, primal_form(B, L, H)) > fwd_sm_count();
  const long need = shares ? imf_attn_fwd_scratch_bytes(B, L, H, 0) : 0;
  if (need > (long)(NOALLOC_FLOATS * sizeof(float))) {
    fprintf(stderr,
            "imf_attn_fwd_noalloc: problem needs %ld bytes of partial-result scratch, the "
            "built-in array holds %zu (at most %d thread blocks)\n",
            need, NOALLOC_FLOATS * sizeof(float), IMF_ATTN_NOALLOC_MAX_CTAS);
    return IMF_ERR_TOO_LARGE;
  }
  return imf_attn_fwd(q, k, v, nullptr, nullptr, nullptr, o, nullptr, lse, B, L, H, head_dim,
                      strides, o_sb, o_sl, o_sh, scale, shares ? scratch_of_device[dev] : nullptr,
                      shares ? (long)(NOALLOC_FLOATS * sizeof(float)) : 0, status, stream);
}
