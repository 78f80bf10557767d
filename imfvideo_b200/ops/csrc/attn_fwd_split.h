// How the work of the dense attention forward is shared out; used by the head_dim 64 and 128
// kernels.
//
// The flattened (item, K/V tile) iteration space is cut into G equal contiguous shares, one per
// CTA of a persistent grid, so the SMs finish together whatever the number of items (228 items
// on 148 SMs, B 1, H 4, L 29,140, would otherwise be two waves, the second half empty).  A share
// boundary inside an item leaves partial results (un-normalised accumulators, running maximum, sums), which a small
// second kernel merges.  With more items than SMs an item is cut at most once; with fewer (short
// sequences) an item's K/V tiles are spread over several CTAs.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace imf {

struct FwdShares {
  int n_items, n_kv;       // items, K/V tiles per item
  long total;              // n_items * n_kv
};

struct Segment {
  int item, j0, j1;        // K/V tile range [j0, j1)
  int rec;                 // scratch record when partial (< 0: complete item)
};

// Segment `s` of CTA `c` (its share is iterations [c*T/G, (c+1)*T/G)).  A CTA has at most two
// partial segments: record 2c continues an item begun by an earlier CTA, record 2c + 1 begins one.
__device__ __forceinline__ bool get_segment(const FwdShares& p, int c, int G, int s, Segment& sg) {
  const long it0 = (long)c * p.total / G, it1 = (long)(c + 1) * p.total / G;
  const int item = (int)(it0 / p.n_kv) + s;
  const long base = (long)item * p.n_kv;
  if (base >= it1 || item >= p.n_items) return false;
  sg.item = item;
  sg.j0 = (int)(it0 > base ? it0 - base : 0);
  sg.j1 = (int)(it1 < base + p.n_kv ? it1 - base : p.n_kv);
  if (sg.j0 >= sg.j1) return false;
  sg.rec = (sg.j0 == 0 && sg.j1 == p.n_kv) ? -1 : 2 * c + (sg.j0 == 0 ? 1 : 0);
  return true;
}

// The split item that begins in CTA `c`, and how many CTAs hold a part of it (records 2c + 1,
// 2(c + 1), 2(c + 2), ...); false if none does.  T: unsigned where (total + n_kv) * G fits 32 bits
// (a 64-bit division takes some 500 clocks, and this is on the merge kernel's critical path).
template <typename T>
__device__ __forceinline__ bool split_item_as(const FwdShares& p, int c, int G, int& item, int& parts) {
  const T total = (T)p.total, g = (T)G, n_kv = (T)p.n_kv;
  const T bound = (T)(c + 1) * total / g;
  const T it = bound / n_kv, base = it * n_kv;
  if (base == bound) return false;                          // the boundary falls on an item's start
  if (it >= (T)p.n_items || base < (T)c * total / g) return false;   // begun by an earlier CTA
  item = (int)it;
  parts = (int)(((base + n_kv) * g - 1) / total) - c + 1;   // .. up to the CTA of its last tile
  return true;
}
__device__ __forceinline__ bool split_item(const FwdShares& p, int c, int G, int& item, int& parts) {
  return (p.total + p.n_kv) * G < (1L << 32) ? split_item_as<unsigned>(p, c, G, item, parts)
                                             : split_item_as<long>(p, c, G, item, parts);
}

// Merge the parts of every split item.  A record is [ACC][ITEM_M] accumulators (o, then dout with
// a tangent), then m, l, mu per query row; without a tangent mu's place holds the row sum of the
// exact exponentials, for the log-sum-exp.  A CTA takes 32 query rows (a lane each), a warp 8 of
// the HD columns.  All of it is load latency, so the parts are merged in one pass (running maximum)
// whose loads are independent of one another.  147 split items of 384 to 512 rows took 16 us
// (head_dim 64, a warp per row) and 58 us (head_dim 128, a thread per row) before.
constexpr int COMBINE_ROWS = 32, COMBINE_COLS = 8;
template <int HD, int ITEM_M, bool TANGENT, typename P>
__device__ __forceinline__ void combine_split_items(const P& p, int G) {
  constexpr int ACC = TANGENT ? 2 * HD : HD;
  constexpr size_t REC = (size_t)ITEM_M * (ACC + 3);
  constexpr int STATS = ACC * ITEM_M;
  static_assert(ITEM_M % COMBINE_ROWS == 0 && HD % COMBINE_COLS == 0 && COMBINE_COLS == 8, "");
  const int c = blockIdx.x;
  int item, parts;
  if (!split_item(p.sh, c, G, item, parts)) return;
  const int qb = item % p.n_qblk, h = (item / p.n_qblk) % p.H, b = item / (p.n_qblk * p.H);
  const float scale_log2 = p.scale * 1.4426950408889634f;
  const int r = blockIdx.y * COMBINE_ROWS + (threadIdx.x & 31);
  const int col = (threadIdx.x >> 5) * COMBINE_COLS;
  const int q_row = qb * ITEM_M + r;
  if (q_row >= p.L) return;
  const float* x = p.scratch + (size_t)(2 * c + 1) * REC + r;     // then records 2c + 2, 2c + 4, ...
  // the first part's own maximum, not -inf: with a scale of zero or below, -inf has no finite weight
  float m = x[STATS], l = 0.f, mu = 0.f;
  float o[COMBINE_COLS], d[COMBINE_COLS];
#pragma unroll
  for (int i = 0; i < COMBINE_COLS; ++i) o[i] = d[i] = 0.f;
#pragma unroll 2
  for (int k = 0; k < parts; ++k, x += k == 1 ? REC : 2 * REC) {
    const float mk = x[STATS], mn = fmaxf(m, mk);
    const float w0 = ex2((m - mn) * scale_log2), w1 = ex2((mk - mn) * scale_log2);
    m = mn;
    l = l * w0 + x[STATS + ITEM_M] * w1;
    mu = mu * w0 + x[STATS + 2 * ITEM_M] * w1;
#pragma unroll
    for (int i = 0; i < COMBINE_COLS; ++i) {
      o[i] = o[i] * w0 + x[(col + i) * ITEM_M] * w1;
      if (TANGENT) d[i] = d[i] * w0 + x[(HD + col + i) * ITEM_M] * w1;
    }
  }
  const int64_t off = (int64_t)b * p.o_sb + (int64_t)q_row * p.o_sl + (int64_t)h * p.o_sh + col;
  const float inv_l = 1.f / l, mul = mu * inv_l;
  uint32_t ob[COMBINE_COLS / 2], db[COMBINE_COLS / 2];
#pragma unroll
  for (int i = 0; i < COMBINE_COLS / 2; ++i) {
    const float o0 = o[2 * i] * inv_l, o1 = o[2 * i + 1] * inv_l;
    ob[i] = pack_bf16(o0, o1);
    db[i] = pack_bf16(d[2 * i] * inv_l - mul * o0, d[2 * i + 1] * inv_l - mul * o1);
  }
  *reinterpret_cast<uint4*>(p.o + off) = make_uint4(ob[0], ob[1], ob[2], ob[3]);
  if (TANGENT) *reinterpret_cast<uint4*>(p.dout + off) = make_uint4(db[0], db[1], db[2], db[3]);
  if (p.lse && col == 0)
    p.lse[((int64_t)b * p.H + h) * p.L + q_row] = m * p.scale + __logf(TANGENT ? l : mu);
}

// SM count of the CURRENT device (cached per device index: a host may hold GPUs of
// different sizes, and a persistent grid larger than the device would not be co-resident).
inline int fwd_sm_count() {
  constexpr int MAX_DEVICES = 64;
  static int sms_of_device[MAX_DEVICES] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  int sms = (dev >= 0 && dev < MAX_DEVICES) ? sms_of_device[dev] : 0;
  if (!sms) {
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
      sms = 148;
    if (dev >= 0 && dev < MAX_DEVICES) sms_of_device[dev] = sms;   // same value from every thread
  }
  return sms;
}

// CTAs of the persistent grid.  Fewer items than SMs: shares of at least two K/V tiles, if that
// shortens a CTA's walk by more than it costs.  In K/V tiles (1 to 1.4 us) the second kernel and the
// extra stores cost three, `part_cost` for each part of an item, and seven parts' worth more where
// shares and items do not end together, so that a CTA begins and stores two.  Fitted to 375 shapes
// of the four kernels timed both ways (1 to 96 heads, 300 to 6,500 rows; 1.4 to 1.9 us rms):
// head_dim 128 with tangent, 8 heads, 532 rows 18 us without shares and 25 with; 1 head, 4,116 rows
// 80 and 42.
inline float fwd_share_cost(long n_items, int n_kv, long g, float part_cost) {
  const long total = n_items * n_kv, walk = (total + g - 1) / g;
  const bool uneven = total % g != 0 || n_kv % walk != 0;
  return 3.f + part_cost * ((float)g / (float)n_items + (uneven ? 7.f : 0.f));
}
inline int fwd_grid(long n_items, int n_kv, float part_cost) {
  const int sms = fwd_sm_count();
  if (n_items >= sms) return sms;
  const long total = n_items * n_kv;
  const long g = total / 2 < sms ? total / 2 : sms;
  if (g <= n_items) return (int)n_items;
  const float saved = (float)(n_kv - (total + g - 1) / g);
  return saved < 1.f + fwd_share_cost(n_items, n_kv, g, part_cost) ? (int)n_items : (int)g;
}

// The same for a launch whose caller gave `have` floats of scratch, at two records of `rec` floats
// per CTA.  Fewer items than SMs need none: one CTA takes each of them then, longer but as correct.
// 0: the scratch is too small for a problem that cannot do without.
inline int fwd_grid(long n_items, int n_kv, float part_cost, const float* scratch, size_t have,
                    size_t rec) {
  const int g = fwd_grid(n_items, n_kv, part_cost);
  if (g == n_items || (scratch != nullptr && have >= (size_t)g * 2 * rec)) return g;
  return n_items <= fwd_sm_count() ? (int)n_items : 0;
}

}  // namespace imf
