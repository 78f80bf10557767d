// How the K/V tiles (items) of the dense attention backward are spread over the SMs; shared by
// the head_dim 64 and 128 kernels.
//
// One CTA walks all query tiles of one 128-row K/V tile, one CTA per SM, so `items` equal walks
// take ceil(items / SMs) waves and the last wave may be nearly empty (912 items on 148 SMs, the
// shape B 1, H 4, L 29,140, is 6.16 waves).  Full waves keep one CTA per item; the items of the
// partial wave are cut into `parts` query ranges each, which then fill the chip for a
// correspondingly shorter time.  Only those items pay for fp32 partial dK / dV and their sum.
// Against splitting every item into two or three (forward + backward, ms): B 1, H 4, L 29,140,
// head_dim 64: 4.17 -> 3.96; B 1, H 12, L 7,820, head_dim 128: 2.07 -> 1.75.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace imf {

struct BwdSplit {
  int n_whole;     // items 0 .. n_whole - 1: one CTA each
  int parts;       // CTAs per remaining item
  int n_split;     // remaining items (0: nothing is split)
  int ctas() const { return n_whole + n_split * parts; }
};

// SM count of the current device, cached per device index (a host may hold GPUs of different
// sizes).
inline int bwd_sm_count() {
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

// `items` walks of `n_steps` query tiles; `cta_steps`: what starting a CTA, filling its pipeline
// and storing its results costs, in steps.  `parts` minimises the time of the partial wave; at
// most six waves of pieces, so the partials stay below 6 x SMs x 128 rows.
inline BwdSplit bwd_split(long items, int n_steps, int sms, float cta_steps) {
  BwdSplit r;
  const int rest = (int)(items % sms);
  r.n_whole = (int)(items - rest);
  r.parts = 1;
  r.n_split = 0;
  if (rest == 0) return r;
  // the kernel that adds the partials up is one launch more, some 2 (head_dim 64) to 4 us (128), which
  // short walks do not make up for (head_dim 64, 12 heads, 385 rows: 18.4 us whole, 20.1 split;
  // head_dim 128, 8 heads, 256 rows: 19.3 and 20.3)
  const float launch = 0.6f * cta_steps;
  float best = (float)n_steps + cta_steps;
  for (int p = 2; p <= n_steps && (long)rest * p <= 6L * sms; ++p) {
    const int waves = (rest * p + sms - 1) / sms;
    // the partials are written and summed on top: about half a CTA start per wave
    const float t = waves * ((float)((n_steps + p - 1) / p) + 1.5f * cta_steps) + launch;
    if (t < best - 0.01f) {
      best = t;
      r.parts = p;
    }
  }
  if (r.parts == 1)
    r.n_whole = (int)items;
  else
    r.n_split = rest;
  return r;
}

}  // namespace imf
