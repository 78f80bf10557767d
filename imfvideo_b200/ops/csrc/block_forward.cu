// Launch sequences of the transformer block's forward pass (ops/block.py): everything before the
// attention core in one call, everything after it in another.
//
// A block of a short clip (532 tokens) is some 14 launches of 3 to 10 us each; issued one by one
// from Python they cost 25 to 45 us of host time apiece, so the GPU waited (dual pass of a
// three-block model at 532 tokens: 3.4 ms, 2.2 ms this way).  Host code only: the kernels and their
// argument checks are those of the launchers called here.
#include <cuda_runtime.h>
#include <stdint.h>

#include "host_util.h"

extern "C" {
int imf_resnorm(void** ptrs, int nsnap, int rows, int D, float eps, int has_t, int bwd, void* stream);
int imf_rmsnorm_seg(void** ptrs, const int* dims, int nseg, int rows, float eps, int has_t, int bwd,
                    void* stream);
int imf_qkprep(void** p, int rows, int L, int H, int dn, int dr, int dv, int ld_kr, int ld_gkr,
               float eps, int has_t, int bwd, void* stream);
int imf_elementwise(int op, void** p, const int* dims, float beta, float lbeta, int has_lbeta,
                    int has_t, int bwd, void* stream);
int imf_gemm_bf16(const void* A, const void* B, void* C, const float* bias, int M, int N, int K,
                  int64_t lda, int64_t ldb, int64_t ldc, int a_mn, int b_mn, int out_fp32,
                  int bias_rows, float alpha, int accumulate_out, int* status, void* stream);
}

namespace imf {

constexpr int BLOCK_MAX_SNAPS = 16;

struct BlockDims {        // order of the `dims` argument
  int rows, L, d, T;      // rows = batch x tokens; T = 2 with a tangent, else 1
  int H, dq, dc, dn, dr, dv, na, fp;
  int nsnap, gate, has_lbeta;
  int ld_wa, ld_wqb, ld_wkvb, ld_wout, ld_w13, ld_w2;      // row pitches of the weights
};

static void* at(void* p, int64_t bytes) { return p ? static_cast<uint8_t*>(p) + bytes : nullptr; }

// y[T rows][n] = x[T rows][k] W^T, all rows contiguous
static int linear(void* x, void* w, void* y, int m, int n, int k, int ldw, void* status, void* stream) {
  return imf_gemm_bf16(x, w, y, nullptr, m, n, k, k, ldw, n, 0, 0, 0, m, 1.f, 0,
                       static_cast<int*>(status), stream);
}

static int resnorm(void* res, void* dres, void* y, void* dy, void* gate, void* w, void* gain,
                   void* pfx, void* dpfx, void* n, void* dn, void** snaps, int ns, bool has_t,
                   int rows, int d, float eps, void* stream) {
  void* p[16 + 3 * BLOCK_MAX_SNAPS] = {res, dres, y, dy, gate, w, gain, pfx, dpfx, n, dn};
  if (ns > BLOCK_MAX_SNAPS) return IMF_ERR_ARG;
  for (int i = 0; i < (has_t ? 2 : 1) * ns; ++i) p[16 + i] = snaps[i];
  return imf_resnorm(p, ns, rows, d, eps, has_t, 0, stream);
}

}  // namespace imf

#define IMF_STEP(call)          \
  {                             \
    const int rc_ = (call);     \
    if (rc_ != 0) return rc_;   \
  }

// n1 = norm1(remix(prefix, snaps)); a = n1 W_a^T; latent norms; q_b, kv_b; q / k preparation.
// ptrs: 0 prefix, 1 dprefix, 2 remix weight, 3 norm1 gain, 4 W_a, 5 q latent gain, 6 kv latent gain,
// 7 W_qb, 8 W_kvb, 9 cos, 10 sin, 11 q gain, 12 k gain, outputs 13 n1, 14 a, 15 q latent, 16 kv
// latent, 17 qb, 18 kvb, 19 q, 20 k (tangent rows behind the primal rows), 21 status word,
// 22.. snaps, then their tangents.
extern "C" int imf_block_pre(void** p, const int* dims, float eps, void* stream) {
  using namespace imf;
  const BlockDims& g = *reinterpret_cast<const BlockDims*>(dims);
  const bool t = g.T == 2;
  const int rows = g.rows, m = g.T * rows;
  const int64_t r = rows;
  IMF_STEP(resnorm(p[0], p[1], nullptr, nullptr, nullptr, p[2], p[3], nullptr, nullptr, p[13],
                   t ? at(p[13], r * g.d * 2) : nullptr, p + 22, g.nsnap, t, rows, g.d, eps, stream));
  IMF_STEP(linear(p[13], p[4], p[14], m, g.na, g.d, g.ld_wa, p[21], stream));
  void* a0 = p[14];
  void* a1 = t ? at(a0, r * g.na * 2) : nullptr;
  {
    void* q[16] = {a0, a1, p[5], p[15], t ? at(p[15], r * g.dq * 2) : nullptr, nullptr, nullptr, nullptr,
                   at(a0, g.dq * 2), at(a1, g.dq * 2), p[6], p[16],
                   t ? at(p[16], r * g.dc * 2) : nullptr, nullptr, nullptr, nullptr};
    const int sd[6] = {g.dq, g.na, g.dq, g.dc, g.na, g.dc};
    IMF_STEP(imf_rmsnorm_seg(q, sd, 2, rows, eps, t, 0, stream));
  }
  const int nq = g.H * (g.dn + g.dr), nkv = g.H * (g.dn + g.dv);
  IMF_STEP(linear(p[15], p[7], p[17], m, nq, g.dq, g.ld_wqb, p[21], stream));
  IMF_STEP(linear(p[16], p[8], p[18], m, nkv, g.dc, g.ld_wkvb, p[21], stream));
  const int64_t kr = (int64_t)(g.dq + g.dc) * 2;
  void* q[20] = {p[17], t ? at(p[17], r * nq * 2) : nullptr, p[18], t ? at(p[18], r * nkv * 2) : nullptr,
                 at(a0, kr), at(a1, kr), p[9], p[10], p[11], p[12],
                 p[19], t ? at(p[19], r * nq * 2) : nullptr, p[20], t ? at(p[20], r * nq * 2) : nullptr};
  return imf_qkprep(q, rows, g.L, g.H, g.dn, g.dr, g.dv, g.na, 0, eps, t, 0, stream);
}

// og = o * sigmoid(gate); a = og W_out^T; p2 = prefix + a * attn_scale; n2 = norm2(remix(p2, snaps));
// out = p2 + situ(n2 W13^T) W2^T * mlp_scale.
// ptrs: 0 o, 1 do, 2 a (projections of n1; the gate band starts at column dq + dc + dr), 3 og (given
// instead of computed when the block has no output gate), 4 W_out, 5 a_out, 6 attn_scale, 7 prefix
// and 8 dprefix (null when the residual restarts here), 9 p2, 10 n2, 11 remix weight, 12 norm2 gain,
// 13 W13, 14 gu, 15 act, 16 W2, 17 m, 18 mlp_scale, 19 out, 20 status word, 21.. snaps, then their
// tangents.
extern "C" int imf_block_post(void** p, const int* dims, float eps, float beta, float lbeta,
                              void* stream) {
  using namespace imf;
  const BlockDims& g = *reinterpret_cast<const BlockDims*>(dims);
  const bool t = g.T == 2;
  const int rows = g.rows, m = g.T * rows, hv = g.H * g.dv, d = g.d;
  const int64_t r = rows;
  if (g.gate) {
    const int64_t col = (int64_t)(g.dq + g.dc + g.dr) * 2;
    void* e[16] = {p[0], p[1], at(p[2], col), t ? at(p[2], r * g.na * 2 + col) : nullptr, nullptr, nullptr,
                   nullptr, p[3], t ? at(p[3], r * hv * 2) : nullptr};
    const int ed[7] = {rows, hv, hv, g.na, hv, 0, 0};
    IMF_STEP(imf_elementwise(0, e, ed, 0.f, 0.f, 0, t, 0, stream));
  }
  IMF_STEP(linear(p[3], p[4], p[5], m, d, hv, g.ld_wout, p[20], stream));
  void* dp2 = t ? at(p[9], r * d * 4) : nullptr;
  IMF_STEP(resnorm(p[7], p[8], p[5], t ? at(p[5], r * d * 2) : nullptr, p[6], p[11], p[12], p[9], dp2,
                   p[10], t ? at(p[10], r * d * 2) : nullptr, p + 21, g.nsnap, t, rows, d, eps, stream));
  IMF_STEP(linear(p[10], p[13], p[14], m, 2 * g.fp, d, g.ld_w13, p[20], stream));
  {
    void* gu1 = t ? at(p[14], r * 2 * g.fp * 2) : nullptr;
    void* e[16] = {p[14], gu1, at(p[14], (int64_t)g.fp * 2), at(gu1, (int64_t)g.fp * 2), nullptr, nullptr,
                   nullptr, p[15], t ? at(p[15], r * g.fp * 2) : nullptr};
    const int ed[7] = {rows, g.fp, 2 * g.fp, 2 * g.fp, g.fp, 0, 0};
    IMF_STEP(imf_elementwise(1, e, ed, beta, lbeta, g.has_lbeta, t, 0, stream));
  }
  IMF_STEP(linear(p[15], p[16], p[17], m, d, g.fp, g.ld_w2, p[20], stream));
  void* e[16] = {p[17], t ? at(p[17], r * d * 2) : nullptr, nullptr, nullptr, p[9], dp2, p[18], nullptr,
                 nullptr, p[19], t ? at(p[19], r * d * 4) : nullptr};
  const int ed[7] = {rows, d, d, d, d, 0, 0};
  return imf_elementwise(2, e, ed, 0.f, 0.f, 0, t, 0, stream);
}
#undef IMF_STEP
