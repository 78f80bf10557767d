// Dense flash attention forward with its forward-mode tangent (JVP) on tcgen05 / TMEM, head_dim 64:
//
//   S = Q K^T * scale,  P = softmax(S),  O = P V
//   dS = (dQ K^T + Q dK^T) * scale,  T = P .* dS,
//   dO = (T V + P dV) / l - (rowsum(T) / l) O          (l = rowsum exp)
//
// i.e. value, tangent and log-sum-exp in ONE pass over K/V, with O(L) memory.  Replaces the
// reference's CuTeDSL mma.sync kernel and Triton flash-JVP kernel (reference
// models/flash_jvp_kernel.py:51-570, models/triton_block_jvp.py:228-346); the reference's are pinned
// to head_dim 64 (reference models/triton_mla_block_jvp.py:689).
//
// Work item = ONE 128-row query tile of one (batch, head).  TMEM (512 columns) holds its O | dO
// accumulators (128), two S | dS buffers (128 each) and two P | T buffers (bf16, 64 each).  Steps (64-row
// K/V tiles) alternate between two groups of four softmax warps, a query row per thread, each with
// buffers of its own: S | dS is free again as soon as a group has it in registers, so while one group
// is at its exponentials the tensor core is at the other's scores and at the products of the step
// before, and the two warps of a scheduler are half a step apart.
// Warps 0-3, 4-7: softmax / tangent math, O correction and epilogue of even and odd steps; warp 8 issues
// the score products, warp 10 the O products, warp 9 the TMA loads, warp 11 only donates registers.
// K | dK and V | dV travel in separate TMA rings: a K stage is free again as soon as its score products
// have run, long before the matching V stage.
//
// What bounds it.  The tensor core needs 832 clocks a step (Q [K | dK] 4 x 64, dQ K 4 x 48: 6 KB of
// operands at 128 B / clock, P [V | dV] 4 x 64, T V 4 x 32), the exponential unit 512.  B 1, H 4,
// L 29,140: 1.84 ms alone, 2.14 ms in a loop at the power cap, 1,030 clocks a step either way by the SM's
// own counter (2.05 and 2.40 ms in a form with two query tiles per item, one S | dS buffer per tile with P
// over it and one issuing thread).  What counted, alone, as measured when each was made:
//  - two issuing warps: an MMA costs its thread some 20 clocks, a commit or a satisfied wait 60 to 150,
//    so one thread with a step's 16 MMAs, 5 commits and 4 waits took 1,600 clocks (2.23 -> 2.09 ms);
//  - the reference maximum handed over as one tagged word in shared memory instead of named
//    barriers (2.09 -> 2.05 ms);
//  - dS loaded only after the maximum has been taken: with S and dS live at once the compiler moves
//    registers about, 558 -> 539 instructions a step (2.05 -> 1.92 ms);
//  - a scale that is a power of two multiplied into q and dq in shared memory, once per item, instead of
//    into every T (1.90 -> 1.81 ms).
// Exponentials against a stale reference with the tile done again where it was outgrown, and loads
// issued a step ahead, were slower (2.11 to 2.65 ms: registers moved).
//
// Scheduling: a persistent grid whose CTAs take whole items in rounds, or equal shares of the flattened
// (item, K/V tile) space (attn_fwd_split.h), whose partial results a second kernel merges.
// Tensors are (B, L, H, 64) bf16 with arbitrary 16-byte-aligned strides; ragged L is handled by
// TMA zero fill + masking of the last K/V tile.
#include "attn_fwd_split.h"
#include "attn_jvp.h"
#include "common.cuh"
#include "host_util.h"

#include <math.h>

namespace imf {
namespace jvp {

constexpr int HD = 64;
constexpr int TM = 128;                  // query rows per item
constexpr int BN = 64;                   // K/V rows per tile
constexpr int QTILE = TM * 128, KTILE = BN * 128;    // bytes
constexpr int SBUF = 2;                  // S | dS buffers, P | T buffers
constexpr int STAGES = 4;                // per ring
constexpr int GROUP_WARPS = 4;           // softmax warps of a step
constexpr int SOFT_WARPS = SBUF * GROUP_WARPS;
constexpr int WARP_QK = 8, WARP_TMA = 9, WARP_PV = 10;
// softmax warps + one warpgroup of the three single-thread warps and one that only donates registers
// (setmaxnreg is a warpgroup-wide instruction)
constexpr int THREADS = 12 * 32;
// setmaxnreg.inc draws from what the CTA was launched with (threads x registers per thread as
// compiled: 168); a request beyond that pool blocks for ever
constexpr int REG_SOFT = 216, REG_OTHER = 72, REG_LAUNCH = 168;
static_assert(SOFT_WARPS * 32 * REG_SOFT + (THREADS - SOFT_WARPS * 32) * REG_OTHER <= THREADS * REG_LAUNCH,
              "register pool exceeded");
// TMEM columns
constexpr int ACC = 2 * HD;              // fp32 accumulators per row: O, dO
constexpr int COL_O = 0, COL_DO = HD;
__host__ __device__ constexpr int col_s(int buf) { return ACC + buf * 2 * BN; }
__host__ __device__ constexpr int col_p(int buf) { return ACC + SBUF * 2 * BN + buf * BN; }
static_assert(col_p(SBUF) <= 512, "TMEM budget");

// scratch record of one part of a split item: [ACC][TM] accumulators (a column per row of the
// record, so that a warp stores 128 consecutive bytes), then m, l, mu per query row
constexpr size_t PART_FLOATS = (size_t)TM * (ACC + 3);

struct Smem {
  alignas(1024) uint8_t q[2][QTILE];               // q, dq
  alignas(1024) uint8_t k[STAGES][2 * KTILE];      // k, dk
  alignas(1024) uint8_t v[STAGES][2 * KTILE];      // v, dv
  uint64_t m_ref[TM];       // reference maximum of the row as of the last step decided | that step's number
  float xst[2][3][TM];      // l, mu and reference maximum of either group, at a segment's end
  uint64_t q_full, q_empty, q_ready;
  uint64_t k_full[STAGES], k_empty[STAGES];
  uint64_t v_full[STAGES], v_empty[STAGES];
  uint64_t s_full[SBUF], s_taken[SBUF], p_full[SBUF];
  uint64_t o_done[SBUF];    // every O product
  uint64_t o_final;         // the last one of a segment (one phase per segment, never skipped)
  uint64_t o_free, sums;
  uint32_t tmem_base;
  int abort_flag;
};

struct Params {
  __nv_bfloat16* o;
  __nv_bfloat16* dout;
  float* lse;              // (B, H, L) natural-log LSE of scaled scores, or null
  float* scratch;          // split-item partials: records of PART_FLOATS, two per CTA
  int B, H, L;
  int n_qblk;
  FwdShares sh;
  bool whole;              // no shares: CTA c takes items c, c + G, ... whole
  int64_t o_sb, o_sl, o_sh;   // output strides in elements
  float scale;             // of the scores as the kernel has them (UNIT: 1)
  float q_scale;           // UNIT: q and dq are multiplied by it in shared memory
  int* status;
};

// Segment `si` of CTA `c`
IMF_DEVICE bool next_segment(const Params& p, int c, int G, int si, Segment& sg) {
  if (!p.whole) return get_segment(p.sh, c, G, si, sg);
  sg.item = c + si * G;
  sg.j0 = 0;
  sg.j1 = p.sh.n_kv;
  sg.rec = -1;
  return sg.item < p.sh.n_items;
}

// q and dq times a power of two, in place, by the softmax warps
IMF_DEVICE void scale_queries(uint8_t (&q)[2][QTILE], float f) {
  uint4* qs = reinterpret_cast<uint4*>(q);
#pragma unroll 4
  for (int i = threadIdx.x; i < (int)(sizeof(q) / 16); i += SOFT_WARPS * 32) {
    uint4 x = qs[i];
    x.x = pack_bf16(bf16_lo(x.x) * f, bf16_hi(x.x) * f);
    x.y = pack_bf16(bf16_lo(x.y) * f, bf16_hi(x.y) * f);
    x.z = pack_bf16(bf16_lo(x.z) * f, bf16_hi(x.z) * f);
    x.w = pack_bf16(bf16_lo(x.w) * f, bf16_hi(x.w) * f);
    qs[i] = x;
  }
  fence_proxy_async_smem();
  __syncwarp();
}

// The row's reference maximum as step `n` left it goes to the warp of the other group in one 64-bit word,
// the step's number in its upper half.  One scalar access each way: a vector of two words is two accesses
// in no order, and the number could be seen before the maximum that it stands for.
IMF_DEVICE uint64_t ref_word(float m, int n) {
  return (uint64_t)(uint32_t)n << 32 | __float_as_uint(m);
}
IMF_DEVICE void publish_ref(uint64_t* addr, float m, int n) {
  asm volatile("st.volatile.shared.b64 [%0], %1;" ::"r"(smem_u32(addr)), "l"(ref_word(m, n)) : "memory");
}

// From the other group's warp, which decided long before as a rule.  Bounded; false: gave up.
IMF_DEVICE bool ref_of_step(const uint64_t* addr, int n, float& m, volatile int* abort_flag, int* status) {
  uint64_t t0 = 0;
  for (uint32_t spins = 1;; ++spins) {
    uint64_t word;
    asm volatile("ld.volatile.shared.b64 %0, [%1];" : "=l"(word) : "r"(smem_u32(addr)) : "memory");
    m = __uint_as_float((uint32_t)word);
    if (__all_sync(0xffffffffu, (int)(word >> 32) >= n)) return true;
    if ((spins & 63u) == 0) {
      if (__any_sync(0xffffffffu, *abort_flag)) return false;
      const uint64_t now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      if (__any_sync(0xffffffffu, now - t0 > IMF_WAIT_LIMIT_NS)) {
        *abort_flag = 1;
        if (status) atomicCAS(status, 0, STATUS_TIMEOUT_SOFTMAX);
        return false;
      }
    }
  }
}

template <bool UNIT>
__global__ void __launch_bounds__(THREADS, 1)
attn_jvp_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_dq,
                const __grid_constant__ CUtensorMap tm_dk, const __grid_constant__ CUtensorMap tm_dv,
                const Params p) {
  extern __shared__ uint8_t smem_raw[];
  auto& s = *reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cta = blockIdx.x, G = gridDim.x;

  if (threadIdx.x == 0) {
    mbar_init(&s.q_full, 1);
    mbar_init(&s.q_empty, 1);
    mbar_init(&s.q_ready, SOFT_WARPS);       // one arrival per softmax warp
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&s.k_full[i], 1);
      mbar_init(&s.k_empty[i], 1);
      mbar_init(&s.v_full[i], 1);
      mbar_init(&s.v_empty[i], 1);
    }
    for (int b = 0; b < SBUF; ++b) {
      mbar_init(&s.s_full[b], 1);
      mbar_init(&s.s_taken[b], GROUP_WARPS);
      mbar_init(&s.p_full[b], GROUP_WARPS);
      mbar_init(&s.o_done[b], 1);
    }
    mbar_init(&s.o_final, 1);
    mbar_init(&s.o_free, SOFT_WARPS);
    mbar_init(&s.sums, SOFT_WARPS);
    s.abort_flag = 0;
    fence_barrier_init();
  }
  if (threadIdx.x < TM) s.m_ref[threadIdx.x] = ref_word(0.f, -1);
  if (warp == WARP_QK) {
    tmem_alloc(&s.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s.tmem_base;
  volatile int* abort_flag = &s.abort_flag;

  if (warp >= SOFT_WARPS) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REG_OTHER));
    if (warp == WARP_TMA) {
      // ---------------------------------------------------- TMA producer --
      if (elect_one()) {
        prefetch_tmap(&tm_q);
        prefetch_tmap(&tm_k);
        prefetch_tmap(&tm_v);
        int st = 0;
        uint32_t par = 1;           // an "empty" wait passes in the first round of the ring
        Segment sg;
        bool ok = true;
        for (int si = 0; ok && next_segment(p, cta, G, si, sg); ++si) {
          const int qb = sg.item % p.n_qblk, h = (sg.item / p.n_qblk) % p.H,
                    b = sg.item / (p.n_qblk * p.H);
          const int q0 = qb * TM;
          if (si > 0) ok = mbar_wait(&s.q_empty, (si - 1) & 1, abort_flag, p.status, STATUS_TIMEOUT_EMPTY);
          if (!ok) break;
          mbar_arrive_expect_tx(&s.q_full, 2 * QTILE);
          tma_load_4d(s.q[0], &tm_q, &s.q_full, 0, h, q0, b);
          tma_load_4d(s.q[1], &tm_dq, &s.q_full, 0, h, q0, b);
          for (int j = sg.j0; j < sg.j1; ++j) {
            ok = mbar_wait(&s.k_empty[st], par, abort_flag, p.status, STATUS_TIMEOUT_EMPTY);
            if (!ok) break;
            mbar_arrive_expect_tx(&s.k_full[st], 2 * KTILE);
            tma_load_4d(s.k[st], &tm_k, &s.k_full[st], 0, h, j * BN, b);
            tma_load_4d(s.k[st] + KTILE, &tm_dk, &s.k_full[st], 0, h, j * BN, b);
            ok = mbar_wait(&s.v_empty[st], par, abort_flag, p.status, STATUS_TIMEOUT_EMPTY);
            if (!ok) break;
            mbar_arrive_expect_tx(&s.v_full[st], 2 * KTILE);
            tma_load_4d(s.v[st], &tm_v, &s.v_full[st], 0, h, j * BN, b);
            tma_load_4d(s.v[st] + KTILE, &tm_dv, &s.v_full[st], 0, h, j * BN, b);
            if (++st == STAGES) {
              st = 0;
              par ^= 1;
            }
          }
        }
      }
    } else if (warp == WARP_QK) {
      // -------------------------------------------- score product issuer --
      if (elect_one()) {
        // k | dk and v | dv lie next to one another in shared memory, and S | dS and O | dO in TMEM,
        // so Q [K | dK]^T and P [V | dV] are one product each.  An SM reads 128 B of operands per
        // clock: M = N = 128 with both operands in shared memory needs 8 KB per 64 clocks, exactly
        // that rate, where two N = 64 products need 6 KB per 32 clocks each and wait for them.
        constexpr uint32_t idesc_qk = idesc_bf16(TM, 2 * BN, 0, 0);
        constexpr uint32_t idesc_dqk = idesc_bf16(TM, BN, 0, 0);
        const uint64_t q_desc = sdesc_kmajor(smem_u32(s.q[0])), dq_desc = sdesc_kmajor(smem_u32(s.q[1]));
        const uint64_t k_desc = sdesc_kmajor(smem_u32(s.k[0]));
        int st = 0, buf = 0;
        uint32_t kpar = 0, tpar = 1;            // a "taken" wait passes in the first round
        Segment sg;
        bool ok = true;
        for (int si = 0; ok && next_segment(p, cta, G, si, sg); ++si) {
          ok = UNIT ? mbar_wait(&s.q_ready, si & 1, abort_flag, p.status, STATUS_TIMEOUT_SOFTMAX)
                    : mbar_wait(&s.q_full, si & 1, abort_flag, p.status, STATUS_TIMEOUT_TMA);
          for (int j = sg.j0; j < sg.j1 && ok; ++j) {
            ok = mbar_wait(&s.k_full[st], kpar, abort_flag, p.status, STATUS_TIMEOUT_TMA) &&
                 mbar_wait(&s.s_taken[buf], tpar, abort_flag, p.status, STATUS_TIMEOUT_SOFTMAX);
            if (!ok) break;
            tc_fence_after();
            const uint64_t kd = k_desc + (uint32_t)(st * (2 * KTILE >> 4));
            const uint32_t sc = tmem + col_s(buf);
#pragma unroll
            for (int ks = 0; ks < HD / 16; ++ks) mma_ss(sc, q_desc + 2 * ks, kd + 2 * ks, idesc_qk, ks != 0);
#pragma unroll
            for (int ks = 0; ks < HD / 16; ++ks) mma_ss(sc + BN, dq_desc + 2 * ks, kd + 2 * ks, idesc_dqk, 1);
            tc_commit(&s.s_full[buf]);
            tc_commit(&s.k_empty[st]);
            if (j + 1 == sg.j1) tc_commit(&s.q_empty);       // last Q read of the item
            if (++st == STAGES) {
              st = 0;
              kpar ^= 1;
            }
            if (++buf == SBUF) {
              buf = 0;
              tpar ^= 1;
            }
          }
        }
      }
    } else if (warp == WARP_PV) {
      // ------------------------------------------- O | dO product issuer --
      if (elect_one()) {
        constexpr uint32_t idesc_pv = idesc_bf16(TM, 2 * HD, 0, 1);
        constexpr uint32_t idesc_tv = idesc_bf16(TM, HD, 0, 1);
        const uint64_t v_desc = sdesc_mnmajor(smem_u32(s.v[0]), KTILE);
        int st = 0, buf = 0;
        uint32_t vpar = 0, ppar = 0;
        Segment sg;
        bool ok = true;
        for (int si = 0; ok && next_segment(p, cta, G, si, sg); ++si) {
          if (si > 0)      // epilogue of the previous segment has drained O
            ok = mbar_wait(&s.o_free, (uint32_t)((si - 1) & 1), abort_flag, p.status, STATUS_TIMEOUT_SOFTMAX);
          for (int j = sg.j0; j < sg.j1 && ok; ++j) {
            ok = mbar_wait(&s.v_full[st], vpar, abort_flag, p.status, STATUS_TIMEOUT_TMA) &&
                 mbar_wait(&s.p_full[buf], ppar, abort_flag, p.status, STATUS_TIMEOUT_SOFTMAX);
            if (!ok) break;
            tc_fence_after();
            const uint64_t vd = v_desc + (uint32_t)(st * (2 * KTILE >> 4));
            const uint32_t pc = tmem + col_p(buf);
#pragma unroll
            for (int ks = 0; ks < BN / 16; ++ks)
              mma_ts(tmem + COL_O, pc + ks * 8, vd + 128 * ks, idesc_pv, !(j == sg.j0 && ks == 0));
#pragma unroll
            for (int ks = 0; ks < BN / 16; ++ks)
              mma_ts(tmem + COL_DO, pc + BN / 2 + ks * 8, vd + 128 * ks, idesc_tv, 1);
            tc_commit(&s.o_done[buf]);
            tc_commit(&s.v_empty[st]);
            if (j + 1 == sg.j1) tc_commit(&s.o_final);
            if (++st == STAGES) {
              st = 0;
              vpar ^= 1;
            }
            if (++buf == SBUF) {
              buf = 0;
              ppar ^= 1;
            }
          }
        }
      }
    }
  } else {
    // ------------------------------------- softmax / correction / epilogue --
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REG_SOFT));
    // Group g takes the steps (K/V tiles) of parity g, with buffers g.  Either warp of a row pair needs
    // the row's reference maximum as the step before left it: it is handed from one to the other,
    // before the exponentials.
    const int g = warp >> 2, wl = warp & 3;
    const int row = wl * 32 + lane;
    const uint32_t tb = tmem_addr(tmem, wl * 32, 0);
    const uint32_t sc = tb + col_s(g), pc = tb + col_p(g);
    const float scale_log2 = p.scale * 1.4426950408889634f;
    uint32_t par = 0;                               // phase of this group's buffers
    int n0 = 0;                                     // number of the segment's first step
    Segment sg;
    bool ok = true;
    for (int si = 0; ok && next_segment(p, cta, G, si, sg); ++si) {
      const int qb = sg.item % p.n_qblk, h = (sg.item / p.n_qblk) % p.H,
                b = sg.item / (p.n_qblk * p.H);
      const int q_row = qb * TM + row;
      float m_used = -INFINITY, l_sum = 0.f, l_sum2 = 0.f, mu_sum = 0.f, mu_sum2 = 0.f;
      const int j_own = sg.j0 + ((n0 ^ g) & 1);     // this group's first step of the segment
      if (UNIT) {
        ok = __all_sync(0xffffffffu, mbar_wait(&s.q_full, si & 1, abort_flag, p.status, STATUS_TIMEOUT_TMA));
        if (!ok) break;
        scale_queries(s.q, p.q_scale);
        if (lane == 0) mbar_arrive(&s.q_ready);
      }
      for (int j = j_own; j < sg.j1; j += 2) {
        const int n = n0 + j - sg.j0;
        ok = __all_sync(0xffffffffu, mbar_wait(&s.s_full[g], par, abort_flag, p.status, STATUS_TIMEOUT_MMA));
        if (!ok) break;
        tc_fence_after();
        const int kv_rem = p.L - j * BN;
        // Scores of keys past the end: -inf, eight columns at a time (a column at a time: 65.1 us at
        // B 3, H 64, L 389, whose last tiles hold five keys; 60.8 this way)
        if (kv_rem < BN) {
          int c = kv_rem;
          for (; c & 7; ++c) tmem_st1(sc + c, 0xff800000u);
#pragma unroll 1
          for (; c < BN; c += 8) tmem_fill8(sc + c, 0xff800000u);
          tc_wait_st();
        }
        uint32_t sv[BN];
        tmem_ld32(sc, sv);
        tmem_ld32(sc + 32, sv + 32);
        // P of this group's step before has been read: probed here, long so as a rule
        const bool p_ok = mbar_test(&s.o_done[g], par ^ 1);
        tc_wait_ld();
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < BN; i += 2)
          asm("max.f32 %0, %0, %1, %2;" : "+f"(mx[(i / 2) & 3]) : "f"(__uint_as_float(sv[i])), "f"(__uint_as_float(sv[i + 1])));
        mx[0] = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
        // P V of this group's step before, n - 2, is seen to be over before the reference of step n is
        // published: whoever has that reference and asks o_done for P V of step n then finds the barrier
        // in that phase or one further.  (A wait by parity on a barrier still two phases back returns at
        // once: V late by two steps, and O would be rescaled under products that are still to run.)
        // P of step n may be written from here on, too.
        if (!__all_sync(0xffffffffu, p_ok)) {
          ok = __all_sync(0xffffffffu, mbar_wait(&s.o_done[g], par ^ 1, abort_flag, p.status, STATUS_TIMEOUT_MMA));
          if (!ok) break;
        }
        tc_fence_after();
        // The reference is moved only when a row has outgrown it by more than 2^8 (or has none yet)
        float m_prev;
        ok = ref_of_step(&s.m_ref[row], n - 1, m_prev, abort_flag, p.status);
        if (!ok) break;
        if (j == sg.j0) m_prev = mx[0];
        const bool need = (mx[0] - m_prev) * scale_log2 > 8.0f;
        const float m_new = need ? mx[0] : m_prev;
        publish_ref(&s.m_ref[row], m_new, n);
        if (__any_sync(0xffffffffu, m_new != m_used)) {
          if (__any_sync(0xffffffffu, need)) {      // O, as of the step before, to the new reference
            ok = __all_sync(0xffffffffu, mbar_wait(&s.o_done[g ^ 1], g == 0 ? par ^ 1 : par, abort_flag,
                                                   p.status, STATUS_TIMEOUT_MMA));
            if (!ok) break;
            tc_fence_after();
            const float alpha = ex2((m_prev - m_new) * scale_log2);
#pragma unroll 1
            for (int c = 0; c < ACC; c += 16) {
              uint32_t ov[16];
              tmem_ld16(tb + COL_O + c, ov);
              tc_wait_ld();
#pragma unroll
              for (int i = 0; i < 16; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
              tmem_st16(tb + COL_O + c, ov);
            }
          }
          if (j != j_own) {                         // the sums so far to the new reference
            const float alpha = ex2((m_used - m_new) * scale_log2);
            l_sum *= alpha;
            l_sum2 *= alpha;
            mu_sum *= alpha;
            mu_sum2 *= alpha;
          }
          m_used = m_new;
        }
        const f32x2 neg_m2 = dup2(-m_used * scale_log2);
        f32x2 l_new = dup2(0.f), mu_new = dup2(0.f);
        uint32_t dsv[2][32];
        tmem_ld32(sc + BN, dsv[0]);
        tmem_ld32(sc + BN + 32, dsv[1]);
        tc_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s.s_taken[g]);
#pragma unroll
        for (int c = 0; c < BN; c += 32) {
          uint32_t pk[16], tk[16];
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            const int i = c + e;
            const f32x2 x = fma2(pair2(sv[i], sv[i + 1]), dup2(scale_log2), neg_m2);
            const float p0 = ex2(lo2(x)), p1 = ex2(hi2(x));
            const f32x2 pp = pair2(__float_as_uint(p0), __float_as_uint(p1));
            pk[e / 2] = pack_bf16(p0, p1);
            l_new = add2(l_new, pp);
            f32x2 tt = mul2(pp, pair2(dsv[i >> 5][i & 31], dsv[i >> 5][(i & 31) + 1]));
            if (!UNIT) tt = mul2(tt, dup2(p.scale));
            mu_new = add2(mu_new, tt);
            tk[e / 2] = pack_bf16(lo2(tt), hi2(tt));
          }
          tmem_st16(pc + c / 2, pk);
          tmem_st16(pc + BN / 2 + c / 2, tk);
        }
        l_sum += lo2(l_new);
        l_sum2 += hi2(l_new);
        mu_sum += lo2(mu_new);
        mu_sum2 += hi2(mu_new);
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s.p_full[g]);
        par ^= 1;
      }
      // ---- epilogue of this segment ----
      if (ok) ok = mbar_wait(&s.o_final, (uint32_t)(si & 1), abort_flag, p.status, STATUS_TIMEOUT_MMA);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      s.xst[g][0][row] = l_sum + l_sum2;
      s.xst[g][1][row] = mu_sum + mu_sum2;
      s.xst[g][2][row] = m_used;
      __syncwarp();
      if (lane == 0) mbar_arrive(&s.sums);
      ok = __all_sync(0xffffffffu, mbar_wait(&s.sums, (uint32_t)(si & 1), abort_flag, p.status,
                                             STATUS_TIMEOUT_SOFTMAX));
      if (!ok) break;
      // the group of the last step has the final reference
      const int n_j = sg.j1 - sg.j0, gl = (n0 + n_j - 1) & 1;
      const float m_fin = s.xst[gl][2][row];
      float l_tot = s.xst[gl][0][row], mu_tot = s.xst[gl][1][row];
      if (n_j > 1) {
        const float alpha = ex2((s.xst[gl ^ 1][2][row] - m_fin) * scale_log2);
        l_tot += alpha * s.xst[gl ^ 1][0][row];
        mu_tot += alpha * s.xst[gl ^ 1][1][row];
      }
      n0 += n_j;
      const bool live = q_row < p.L;
      if (sg.rec < 0) {
        const float inv_l = 1.f / l_tot, mul = mu_tot * inv_l;
        const int64_t off = (int64_t)b * p.o_sb + (int64_t)q_row * p.o_sl + (int64_t)h * p.o_sh;
        // each group writes half the columns of o and of dout
        const int c = g * (HD / 2);
        uint32_t ov[32], dv_[32], ob[16], db[16];
        tmem_ld32(tb + COL_O + c, ov);
        tmem_ld32(tb + COL_DO + c, dv_);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float o0 = __uint_as_float(ov[2 * i]) * inv_l, o1 = __uint_as_float(ov[2 * i + 1]) * inv_l;
          ob[i] = pack_bf16(o0, o1);
          db[i] = pack_bf16(__uint_as_float(dv_[2 * i]) * inv_l - mul * o0,
                            __uint_as_float(dv_[2 * i + 1]) * inv_l - mul * o1);
        }
        if (live) {
          uint4* dst = reinterpret_cast<uint4*>(p.o + off + c);
          uint4* ddst = reinterpret_cast<uint4*>(p.dout + off + c);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            dst[i] = make_uint4(ob[4 * i], ob[4 * i + 1], ob[4 * i + 2], ob[4 * i + 3]);
            ddst[i] = make_uint4(db[4 * i], db[4 * i + 1], db[4 * i + 2], db[4 * i + 3]);
          }
        }
        if (live && p.lse && g == 0)
          p.lse[((int64_t)b * p.H + h) * p.L + q_row] = m_fin * p.scale + __logf(l_tot);
      } else {
        // partial result of a split item: raw accumulators + (m, l, mu); group 0 stores O, group 1 dO
        float* part = p.scratch + (size_t)sg.rec * PART_FLOATS;
#pragma unroll 1
        for (int c = g * HD; c < (g + 1) * HD; c += 32) {
          uint32_t ov[32];
          tmem_ld32(tb + COL_O + c, ov);
          tc_wait_ld();
          float* acc = part + (size_t)c * TM + row;
#pragma unroll
          for (int i = 0; i < 32; ++i) acc[i * TM] = __uint_as_float(ov[i]);
        }
        if (g == 0) {
          float* stats = part + (size_t)TM * ACC;
          stats[row] = m_fin;
          stats[TM + row] = l_tot;
          stats[2 * TM + row] = mu_tot;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s.o_free);
    }
    tc_fence_before();
  }
  __syncthreads();
  if (warp == WARP_QK) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

__global__ void __launch_bounds__(32 * HD / COMBINE_COLS)
attn_jvp_combine_kernel(const Params p, int G) {
  combine_split_items<HD, TM, true>(p, G);
}

// Whole items, CTA c taking items c, c + G, ..., or equal shares of the (item, K/V tile) space with a
// merge.  More items than SMs: walks of up to SHORT_WALK tiles always whole, since a share saves less than a
// walk and the two parts that each CTA stores and the merge cost some 18 tiles, 10 us (632 shapes of
// 1 to 128 heads, either way timed in turn, whole the faster in each: B 3, H 96, L 192, four rounds 30.6 us
// against 58.4; B 8, H 20, L 768 86.1 and 116.8).  Longer walks by an account in K/V tiles, of 0.57 to 0.7 us:
// a further round is charged 12 and shares 32 (H 4, L 29,140 2,173 us whole, 1,988 shared; H 16, L 7,820
// 642 and 617; 354 shapes, 4 % behind the better way on average: whole rounds are faster where the last is
// nearly full, and where K, V and tangents of all heads, which shares walk at once and rounds a few heads
// at a time, are beyond L2: B 4, H 4, L 29,140 8.3 ms whole, 11.4 shared).  Fewer items: fwd_share_cost
// with PART_COST (1 head, 6,500 rows 63.5 us whole, 41.8 shared; 8 heads, 2,068 rows 28.4 and 37.1).
constexpr float PART_COST = 2.2f, ROUND_COST = 12.f, ALL_SPLIT_COST = 32.f;
constexpr int SHORT_WALK = 16;
struct Plan {
  int G;
  bool whole;
};
static Plan plan(int B, int L, int H) {
  const long n = (long)((L + TM - 1) / TM) * H * B;
  const int n_kv = (L + BN - 1) / BN, sms = fwd_sm_count();
  const long total = n * n_kv, rounds = (n + sms - 1) / sms;
  const int one = (int)(n < sms ? n : sms);                       // CTAs that take whole items
  const int g = (int)(total / 2 < sms ? total / 2 : sms);         // .. shares of two tiles at least
  if (n > sms ? n_kv <= SHORT_WALK : g <= one) return {one, true};
  const float t_whole = (float)(rounds * n_kv) + ROUND_COST * (float)(rounds - 1);
  const float cost = n > sms ? ALL_SPLIT_COST : 1.f + fwd_share_cost(n, n_kv, g, PART_COST);
  return (float)((total + g - 1) / g) + cost < t_whole ? Plan{g, false} : Plan{one, true};
}

static int make_map(CUtensorMap* m, const void* ptr, const JvpArgs& a, const int64_t* st, int rows) {
  uint64_t dims[4] = {(uint64_t)HD, (uint64_t)a.H, (uint64_t)a.L, (uint64_t)a.B};
  uint64_t str[4] = {2, (uint64_t)st[2] * 2, (uint64_t)st[1] * 2, (uint64_t)st[0] * 2};
  uint32_t box[4] = {(uint32_t)HD, 1, (uint32_t)rows, 1};
  return make_tmap(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), dims, str, box);
}

template <bool UNIT>
static int launch(const JvpArgs& a) {
  Params prm;
  prm.o = static_cast<__nv_bfloat16*>(a.o);
  prm.dout = static_cast<__nv_bfloat16*>(a.dout);
  prm.lse = a.lse;
  prm.scratch = static_cast<float*>(a.scratch);
  prm.B = a.B; prm.H = a.H; prm.L = a.L;
  prm.o_sb = a.o_sb; prm.o_sl = a.o_sl; prm.o_sh = a.o_sh;
  prm.scale = UNIT ? 1.f : a.scale;
  prm.q_scale = a.scale;
  prm.status = a.status;
  prm.n_qblk = (a.L + TM - 1) / TM;
  prm.sh.n_items = prm.n_qblk * a.H * a.B;
  prm.sh.n_kv = (a.L + BN - 1) / BN;
  prm.sh.total = (long)prm.sh.n_items * prm.sh.n_kv;
  Plan pl = plan(a.B, a.L, a.H);
  if (!pl.whole && (a.scratch == nullptr || (size_t)a.scratch_bytes < (size_t)pl.G * 2 * PART_FLOATS * sizeof(float))) {
    // problems of no more pairs of query tiles than SMs do without, longer but as correct
    const int sms = fwd_sm_count();
    if ((long)((a.L + 2 * TM - 1) / (2 * TM)) * a.H * a.B > sms) return IMF_ERR_ARG;
    pl = Plan{prm.sh.n_items < sms ? prm.sh.n_items : sms, true};
  }
  prm.whole = pl.whole;
  CUtensorMap mq, mk, mv, mdq, mdk, mdv;
  int rc;
  const int64_t* st = a.strides;
  if ((rc = make_map(&mq, a.q, a, st, TM)) || (rc = make_map(&mk, a.k, a, st + 3, BN)) ||
      (rc = make_map(&mv, a.v, a, st + 6, BN)) || (rc = make_map(&mdq, a.dq, a, st + 9, TM)) ||
      (rc = make_map(&mdk, a.dk, a, st + 12, BN)) || (rc = make_map(&mdv, a.dv, a, st + 15, BN)))
    return rc;
  auto kern = attn_jvp_kernel<UNIT>;
  const size_t smem = sizeof(Smem) + 1024;
  static bool smem_set[HOST_MAX_DEVICES] = {false};
  if (!allow_smem((const void*)kern, smem, smem_set)) return IMF_ERR_LAUNCH;
  cudaStream_t stream = static_cast<cudaStream_t>(a.stream);
  kern<<<pl.G, THREADS, smem, stream>>>(mq, mk, mv, mdq, mdk, mdv, prm);
  if (cudaGetLastError() != cudaSuccess) return IMF_ERR_LAUNCH;
  if (!pl.whole) {
    const dim3 grid(pl.G - 1, TM / COMBINE_ROWS);
    attn_jvp_combine_kernel<<<grid, 32 * HD / COMBINE_COLS, 0, stream>>>(prm, pl.G);
    if (cudaGetLastError() != cudaSuccess) return IMF_ERR_LAUNCH;
  }
  return IMF_OK;
}

}  // namespace jvp

long attn_jvp_scratch_bytes(int B, int L, int H) {
  const jvp::Plan pl = jvp::plan(B, L, H);
  return pl.whole ? 0 : (long)((size_t)pl.G * 2 * jvp::PART_FLOATS * sizeof(float));
}

int attn_jvp_launch(const JvpArgs& a) {
  // Scales that are powers of two (head_dim 64: 1/8) go into q and dq, from 2^-8 to 1: nothing can
  // overflow, and only elements below 2^-118 lose bits.
  int e;
  const bool unit = a.scale > 0x1p-9f && a.scale <= 1.f && frexpf(a.scale, &e) == 0.5f;
  return unit ? jvp::launch<true>(a) : jvp::launch<false>(a);
}

}  // namespace imf
