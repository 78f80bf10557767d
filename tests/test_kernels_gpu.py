"""GPU: each sm_100a kernel against the plain-PyTorch fp32 formulas."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from imfvideo_b200.ops import cuda as cu

    assert cu.available(), "kernel library must load on a GPU box"
    from imfvideo_b200.ops import kernels

    return kernels


def _rel(a, b):
    a, b = a.float(), b.float()
    return ((a - b).norm() / (b.norm() + 1e-12)).item()


@pytest.mark.parametrize("M,N,Kd", [(128, 128, 64), (304, 200, 136), (1000, 528, 256), (77, 64, 8)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
def test_gemm(K, M, N, Kd, a_mn, b_mn):
    if (a_mn and M % 8) or (b_mn and N % 8):
        pytest.skip("MN-major operand needs a 16-byte-multiple row stride")
    torch.manual_seed(0)
    A = torch.randn(M, Kd, device="cuda").bfloat16()
    B = torch.randn(N, Kd, device="cuda").bfloat16()
    bias = torch.randn(N, device="cuda")
    out = K.gemm(A.t().contiguous() if a_mn else A, B.t().contiguous() if b_mn else B,
                 a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32, bias=bias, bias_rows=M // 2)
    ref = A.float() @ B.float().t()
    ref[: M // 2] += bias
    assert _rel(out, ref) < 1e-5
    out16 = K.gemm(A.t().contiguous() if a_mn else A, B.t().contiguous() if b_mn else B,
                   a_mn=a_mn, b_mn=b_mn)
    assert _rel(out16, A.float() @ B.float().t()) < 4e-3
    K.check_status()


@pytest.mark.parametrize("rows,M,N", [(29140, 528, 256), (1000, 144, 256), (4100, 256, 682),
                                      (333, 64, 72), (20000, 1364, 256)])
def test_gemm_weight_gradient_splitk(K, rows, M, N):
    """dY^T X over many token rows: split-K slices summed in a fixed order; strided operand
    views (a band of a wider dY, the first columns of a wider X); accumulation into an
    existing fp32 buffer; two runs give the same bits."""
    torch.manual_seed(rows)
    dy_full = torch.randn(rows, (M + 23) // 8 * 8, device="cuda").bfloat16()
    x_full = torch.randn(rows, (N + 15) // 8 * 8, device="cuda").bfloat16()   # 16-byte row pitch
    dy, x = dy_full[:, 8:8 + M], x_full[:, :N]
    ref = dy.float().t() @ x.float()
    out = K.gemm_wgrad(dy, x)
    assert out.dtype == torch.float32 and _rel(out, ref) < 1e-5
    base = torch.randn(M, N, device="cuda")
    acc = base.clone()
    K.gemm_wgrad(dy, x, out=acc, accumulate=True)
    assert _rel(acc, base + ref) < 1e-5
    assert torch.equal(K.gemm_wgrad(dy, x), out)
    K.check_status()


@pytest.mark.parametrize("M,N,Kd", [(256, 128, 128), (1000, 528, 256), (300, 200, 136), (4096, 768, 1024)])
def test_gemm_fp8(K, M, N, Kd):
    """e4m3 operands on the kind::f8f6f4 tensor path: exact against the same quantised values
    multiplied in fp32, and within the reference's fp8 envelope (4e-2) of the unquantised product."""
    torch.manual_seed(M)
    A = torch.randn(M, Kd, device="cuda").bfloat16()
    B = (torch.randn(N, Kd, device="cuda") * 0.05).bfloat16()
    bias = torch.randn(N, device="cuda")
    a8, sa = K.quantize_fp8(A)
    b8, sb = K.quantize_fp8(B)
    assert a8.shape == (M, (Kd + 15) // 16 * 16) and (a8[:, Kd:] == 0).all()
    deq = lambda t8, s_: t8.view(torch.float8_e4m3fn).float() * s_
    assert _rel(deq(a8, sa)[:, :Kd], A) < 4e-2 and float(sa) > 0
    out = K.gemm_fp8(a8, sa, b8, sb, out_dtype=torch.float32, bias=bias)
    exact = deq(a8, sa) @ deq(b8, sb).t() + bias
    assert _rel(out, exact) < 1e-5
    full = A.float() @ B.float().t() + bias
    assert _rel(out, full) < 4e-2
    y = K.linear_fp8(A, B, bias)
    assert y.dtype == torch.bfloat16 and _rel(y, full) < 4e-2
    K.check_status()


@pytest.mark.parametrize("b_mn", [False, True])
@pytest.mark.parametrize("M,N,Kd", [(1000, 1024, 1536), (300, 1400, 2736)])
def test_gemm_wide_tiles(K, M, N, Kd, b_mn):
    """Wide and deep products take the 128 x 256 tile instance (ragged M and N included)."""
    torch.manual_seed(N)
    A = torch.randn(M, Kd, device="cuda").bfloat16()
    B = (torch.randn(N, Kd, device="cuda") * 0.1).bfloat16()
    bias = torch.randn(N, device="cuda")
    out = K.gemm(A, B.t().contiguous() if b_mn else B, b_mn=b_mn, bias=bias, bias_rows=M // 2)
    ref = A.float() @ B.float().t()
    ref[: M // 2] += bias
    assert _rel(out, ref) < 4e-3
    K.check_status()


def test_gemm_rejects_bad_stride(K):
    A = torch.randn(64, 12, device="cuda").bfloat16()      # K = 12: stride not 16-byte multiple
    with pytest.raises(ValueError):
        K.gemm(A, A)


@pytest.mark.parametrize("B,L,H", [(1, 256, 1), (1, 300, 2), (2, 1000, 3), (1, 64, 1), (1, 2049, 2)])
def test_attention_forward(K, B, L, H):
    from imfvideo_b200.ops import reference as ref

    g = torch.Generator(device="cuda").manual_seed(L)
    q, k, v = (torch.randn(B, L, H, 64, device="cuda", generator=g).bfloat16() for _ in range(3))
    o, _, lse = K.attn_fwd(q, k, v)
    ro = ref.attention(q.float(), k.float(), v.float())
    assert (o.float() - ro).abs().max() < 2e-2 and _rel(o, ro) < 1e-2
    assert (lse - ref.attention_lse(q.float(), k.float())).abs().max() < 1e-3
    K.check_status()


@pytest.mark.parametrize("B,L,H", [(1, 256, 1), (1, 212, 2), (2, 1000, 3), (1, 2049, 2)])
def test_attention_forward_tangent(K, B, L, H):
    from imfvideo_b200.ops import reference as ref

    g = torch.Generator(device="cuda").manual_seed(L)
    mk = lambda s: (torch.randn(B, L, H, 64, device="cuda", generator=g) * s).bfloat16()
    q, k, v, dq, dk, dv = mk(1), mk(1), mk(1), mk(.5), mk(.5), mk(.5)
    o, do, lse = K.attn_fwd(q, k, v, dq, dk, dv)
    ro, rdo = ref.attention_jvp(*(t.float() for t in (q, k, v, dq, dk, dv)))
    assert (o.float() - ro).abs().max() < 2e-2 and _rel(o, ro) < 1e-2
    assert (do.float() - rdo).abs().max() < 2e-2 and _rel(do, rdo) < 1e-2
    o2, _, _ = K.attn_fwd(q, k, v)
    assert _rel(o2, o) < 5e-3            # primal-only and fused kernels agree
    K.check_status()


@pytest.mark.parametrize("B,L,H", [(1, 256, 1), (1, 300, 3), (2, 1000, 3), (1, 64, 1), (1, 2049, 2),
                                   (2, 2100, 12)])
def test_attention_forward_hd128(K, B, L, H):
    """head_dim 128, head counts that are not powers of two, ragged lengths, and (last case)
    more work items than SMs, so items are split between CTAs and merged."""
    from imfvideo_b200.ops import reference as ref

    g = torch.Generator(device="cuda").manual_seed(L)
    q, k, v = (torch.randn(B, L, H, 128, device="cuda", generator=g).bfloat16() for _ in range(3))
    o, _, lse = K.attn_fwd(q, k, v)
    for h in sorted({0, H // 2, H - 1}):
        sl = slice(h, h + 1)
        ro = ref.attention(q[:, :, sl].float(), k[:, :, sl].float(), v[:, :, sl].float())
        assert (o[:, :, sl].float() - ro).abs().max() < 2e-2 and _rel(o[:, :, sl], ro) < 1e-2
        rl = ref.attention_lse(q[:, :, sl].float(), k[:, :, sl].float())
        assert (lse[:, sl] - rl).abs().max() < 1e-3
    K.check_status()


@pytest.mark.parametrize("B,L,H", [(1, 128, 1), (1, 212, 3), (2, 1000, 3), (1, 2049, 2), (1, 2100, 12)])
def test_attention_forward_tangent_hd128(K, B, L, H):
    from imfvideo_b200.ops import reference as ref

    g = torch.Generator(device="cuda").manual_seed(L)
    mk = lambda s: (torch.randn(B, L, H, 128, device="cuda", generator=g) * s).bfloat16()
    q, k, v, dq, dk, dv = mk(1), mk(1), mk(1), mk(.5), mk(.5), mk(.5)
    o, do, lse = K.attn_fwd(q, k, v, dq, dk, dv)
    for h in sorted({0, H // 2, H - 1}):
        sl = slice(h, h + 1)
        ro, rdo = ref.attention_jvp(*(t[:, :, sl].float() for t in (q, k, v, dq, dk, dv)))
        assert (o[:, :, sl].float() - ro).abs().max() < 2e-2 and _rel(o[:, :, sl], ro) < 1e-2
        assert (do[:, :, sl].float() - rdo).abs().max() < 3e-2 and _rel(do[:, :, sl], rdo) < 1e-2
    o2, _, lse2 = K.attn_fwd(q, k, v)
    assert _rel(o2, o) < 5e-3            # primal-only and fused kernels agree
    assert (lse - lse2).abs().max() < 1e-3
    o3, do3, _ = K.attn_fwd(q, k, v, dq, dk, dv)
    assert torch.equal(o, o3) and torch.equal(do, do3)       # run twice: same bits
    K.check_status()


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("B,L,H,grow", [(1, 129, 1, False), (1, 532, 4, False), (1, 2049, 2, True),
                                        (2, 1300, 3, True), (1, 7000, 10, False), (1, 513, 1, True)])
def test_attention_forward_shares(K, hd, B, L, H, grow):
    """Few items (each spread over several CTAs), one more than fits evenly, more items than SMs,
    and every query-tile count of the last item.  ``grow``: the keys grow along the sequence, so
    rows outgrow their reference maximum again and again (tile redone, accumulators rescaled) and
    the parts of a split item have very different maxima.  P (and T) and the result are rounded to
    bf16, 2^-9 each, and the tangent is a difference of two such sums."""
    from imfvideo_b200.ops import reference as ref

    g = torch.Generator(device="cuda").manual_seed(L + hd)
    mk = lambda s=1.0: (torch.randn(B, L, H, hd, device="cuda", generator=g) * s).bfloat16()
    q, k, v, dq, dk, dv = mk(), mk(), mk(), mk(.5), mk(.5), mk(.5)
    if grow:
        k = (k * torch.linspace(0.05, 8.0, L, device="cuda").view(1, L, 1, 1)).bfloat16()
    ro, rdo = ref.attention_jvp(*(t.float() for t in (q, k, v, dq, dk, dv)))
    rl = ref.attention_lse(q.float(), k.float())
    o, _, lse = K.attn_fwd(q, k, v)
    o2, do, lse2 = K.attn_fwd(q, k, v, dq, dk, dv)
    for a in (o, o2):
        assert _rel(a, ro) < 6e-3
    assert _rel(do, rdo) < 1.2e-2
    # the row sum is taken in fp32 before P is rounded; 1e-3 is the envelope of every LSE here
    assert (lse - rl).abs().max() < 1e-3 and (lse2 - rl).abs().max() < 1e-3
    again = K.attn_fwd(q, k, v, dq, dk, dv)
    assert torch.equal(again[0], o2) and torch.equal(again[1], do) and torch.equal(again[2], lse2)
    K.check_status()


@pytest.mark.parametrize("L,H", [(130, 24), (2049, 8)])
@pytest.mark.parametrize("need_lse", [False, True])
def test_attention_forward_divides_by_the_sum_of_rounded_weights(K, L, H, need_lse):
    """Scores of standard deviation 16, few keys carry the weight: the error of o is that of weights
    rounded to bf16 and divided by their own sum (5 % for where a row's reference maximum lies and
    fp32 sums; the division by the sum of the exact weights costs 10 % and more); the log-sum-exp
    is that of the exact ones (1e-4: fp32 scores of up to 100)."""
    g = torch.Generator(device="cuda").manual_seed(L)
    q, k, v = ((torch.randn(1, L, H, 64, device="cuda", generator=g) * s).bfloat16() for s in (4, 4, 1))
    s = torch.einsum("blhd,bshd->bhls", q.double(), k.double()) / 8
    p = torch.exp(s - s[..., :64].amax(-1, keepdim=True))
    pr = p.float().bfloat16().double()
    mul = lambda w, d: (torch.einsum("bhls,bshd->bhld", w, v.double()) / d.sum(-1, keepdim=True)).transpose(1, 2)
    exact = mul(p, p)
    own = _rel(mul(pr, pr).bfloat16(), exact)
    o, _, lse = K.attn_fwd(q, k, v, need_lse=need_lse)
    assert _rel(o, exact) < 1.05 * own
    assert (lse is not None) == need_lse
    assert not need_lse or (lse - torch.logsumexp(s, -1)).abs().max() < 1e-4
    K.check_status()


@pytest.mark.parametrize("L,H", [(130, 3), (1000, 2), (850, 40), (2600, 8), (850, 64), (5200, 8), (200, 3),
                                 (1000, 24), (2068, 16)])
def test_attention_forward_items(K, L, H):
    """The primal kernel's work items of two, three and four query tiles, each whole and in shares, and
    of two with 128-row K/V tiles whose last one has 72, 104 and 20 rows (in this order two whole,
    two, three whole, three, four whole, four on 148 SMs); bounds as above."""
    from imfvideo_b200.ops import reference as ref

    g = torch.Generator(device="cuda").manual_seed(L + H)
    q, k, v = (torch.randn(1, L, H, 64, device="cuda", generator=g).bfloat16() for _ in range(3))
    o, _, lse = K.attn_fwd(q, k, v)
    assert _rel(o, ref.attention(q.float(), k.float(), v.float())) < 6e-3
    assert (lse - ref.attention_lse(q.float(), k.float())).abs().max() < 1e-3
    K.check_status()


@pytest.mark.parametrize("B,L,H,scale", [(1, 64, 1, 0.125), (1, 65, 1, 0.125), (1, 129, 2, 1.0), (1, 193, 1, 0.1),
                                         (1, 300, 2, 2.0 ** -8), (1, 300, 2, 2.0 ** -9), (3, 140, 60, 0.125),
                                         (1, 130, 80, 0.125), (1, 600, 40, 0.125), (1, 2600, 2, 0.125)])
def test_attention_forward_tangent_items(K, B, L, H, scale):
    """The tangent kernel's steps alternate between two groups of warps: one step, two, three and four
    of them; scales that are powers of two (multiplied into q and dq) and others; three rounds of whole
    items, items of two query tiles, two rounds, shares (in this order, on 148 SMs).  Bounds as above."""
    from imfvideo_b200.ops import reference as ref

    g = torch.Generator(device="cuda").manual_seed(L + H)
    q, k, v, dq, dk, dv = (torch.randn(B, L, H, 64, device="cuda", generator=g).bfloat16() for _ in range(6))
    f = lambda t: t.float()
    ro, rdo = ref.attention_jvp(*map(f, (q, k, v, dq, dk, dv)), scale=scale)
    o, do, lse = K.attn_fwd(q, k, v, dq, dk, dv, scale=scale)
    assert _rel(o, ro) < 6e-3 and _rel(do, rdo) < 1.2e-2
    assert (lse - ref.attention_lse(f(q), f(k), scale=scale)).abs().max() < 1e-3
    K.check_status()


@pytest.mark.parametrize("B,L,H,whole", [(3, 192, 96, True), (8, 128, 64, True), (8, 150, 60, False),
                                          (1, 2368, 16, False), (4, 1024, 40, True)])
def test_attention_forward_tangent_rounds(K, B, L, H, whole):
    """More query tiles than SMs: whole items in four rounds, of two K/V tiles, pairs of query tiles in shares,
    tiles in shares, nine rounds of sixteen K/V tiles (on 148 SMs).  Bounds as above, on the
    first and the last head of a batch."""
    from imfvideo_b200.ops import reference as ref

    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert (K._lib.imf_attn_fwd_scratch_bytes_hd(B, L, H, 1, 64) == 0) == whole
    g = torch.Generator(device="cuda").manual_seed(L + H)
    xs = [torch.randn(B, L, H, 64, device="cuda", generator=g).bfloat16() for _ in range(6)]
    o, do, lse = K.attn_fwd(*xs)
    for h in (slice(0, 1), slice(H - 1, H)):
        q, k, v, dq, dk, dv = (x[:, :, h].float() for x in xs)
        ro, rdo = ref.attention_jvp(q, k, v, dq, dk, dv, scale=0.125)
        assert _rel(o[:, :, h], ro) < 6e-3 and _rel(do[:, :, h], rdo) < 1.2e-2
        assert (lse[:, h] - ref.attention_lse(q, k, scale=0.125)).abs().max() < 1e-3
    K.check_status()


@pytest.mark.parametrize("rem", [1, 7, 8, 9, 31, 56, 57, 63])
@pytest.mark.parametrize("tiles,scale", [(0, 0.125), (2, 0.1)])
def test_attention_forward_tangent_ragged_tail(K, rem, tiles, scale):
    """Keys of a partial last K/V tile, their number around the groups of eight columns in which the rest
    is masked.  Bounds as above."""
    from imfvideo_b200.ops import reference as ref

    L = 64 * tiles + rem
    g = torch.Generator(device="cuda").manual_seed(L)
    q, k, v, dq, dk, dv = (torch.randn(1, L, 2, 64, device="cuda", generator=g).bfloat16() for _ in range(6))
    f = lambda t: t.float()
    ro, rdo = ref.attention_jvp(*map(f, (q, k, v, dq, dk, dv)), scale=scale)
    o, do, lse = K.attn_fwd(q, k, v, dq, dk, dv, scale=scale)
    assert _rel(o, ro) < 6e-3
    # one key: the tangent of o is dv, with whatever P dS V leaves of cancelled bf16 products beside it
    assert (do.float() - rdo).norm() < 1.2e-2 * max(rdo.norm(), v.float().norm())
    assert (lse - ref.attention_lse(f(q), f(k), scale=scale)).abs().max() < 1e-3
    K.check_status()


@pytest.mark.parametrize("B,L,H", [(1, 2049, 2), (2, 2600, 4), (1, 600, 58), (3, 140, 60)])
@pytest.mark.parametrize("scale", [0.125, 0.1])
def test_attention_forward_tangent_growing_keys(K, B, L, H, scale):
    """Keys that grow along the sequence: rows outgrow their reference maximum in step after step, which one
    group of warps finds and the other has to take over.  Shares of few items and of more than SMs, whole
    items in two and three rounds (on 148 SMs); either form of the scale.  Bounds as above; run twice: same
    bits."""
    from imfvideo_b200.ops import reference as ref

    g = torch.Generator(device="cuda").manual_seed(L + H)
    mk = lambda s=1.0: (torch.randn(B, L, H, 64, device="cuda", generator=g) * s).bfloat16()
    q, k, v, dq, dk, dv = mk(), mk(), mk(), mk(.5), mk(.5), mk(.5)
    k = (k * torch.linspace(0.05, 12.0, L, device="cuda").view(1, L, 1, 1)).bfloat16()
    f = lambda t: t.float()
    ro, rdo = ref.attention_jvp(*map(f, (q, k, v, dq, dk, dv)), scale=scale)
    o, do, lse = K.attn_fwd(q, k, v, dq, dk, dv, scale=scale)
    assert _rel(o, ro) < 6e-3 and _rel(do, rdo) < 1.2e-2
    assert (lse - ref.attention_lse(f(q), f(k), scale=scale)).abs().max() < 1e-3
    again = K.attn_fwd(q, k, v, dq, dk, dv, scale=scale)
    assert all(torch.equal(a, b) for a, b in zip((o, do, lse), again))
    K.check_status()


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("B,L,H", [(1, 576, 4), (1, 7040, 10)])
@pytest.mark.parametrize("scale", [0.0, -0.1])
def test_attention_forward_scale_of_zero_and_below(K, hd, B, L, H, scale):
    """Split items (few, and more than SMs) with every weight equal, and with the sign of the scores
    turned over.  Whole K/V tiles only: the keys past a ragged end are masked by a score of -inf
    before the scale is applied, which needs a scale above zero.  The rounding of P and of the
    result to bf16, 2^-9 each, bounds the error; the tangent is a difference of two such sums."""
    from imfvideo_b200.ops import reference as ref

    g = torch.Generator(device="cuda").manual_seed(L + hd)
    q, k, v, dq, dk, dv = (torch.randn(B, L, H, hd, device="cuda", generator=g).bfloat16() for _ in range(6))
    f = lambda t: t.float()
    ro, rdo = ref.attention_jvp(*map(f, (q, k, v, dq, dk, dv)), scale=scale)
    rl = ref.attention_lse(f(q), f(k), scale=scale)
    o, _, lse = K.attn_fwd(q, k, v, scale=scale)
    o2, do, lse2 = K.attn_fwd(q, k, v, dq, dk, dv, scale=scale)
    assert _rel(o, ro) < 6e-3 and _rel(o2, ro) < 6e-3 and _rel(do, rdo) < 1.2e-2
    assert (lse - rl).abs().max() < 1e-3 and (lse2 - rl).abs().max() < 1e-3
    K.check_status()


def test_attention_strided_views_and_run_twice(K):
    """v as a slice of a wider kv tensor (as in MLA); two runs are bit-equal."""
    torch.manual_seed(0)
    B, L, H = 1, 515, 4
    kv = torch.randn(B, L, H, 112, device="cuda").bfloat16()
    q = torch.randn(B, L, H, 64, device="cuda").bfloat16()
    k = torch.randn(B, L, H, 64, device="cuda").bfloat16()
    v = kv[..., 48:]
    o1, _, _ = K.attn_fwd(q, k, v)
    o2, _, _ = K.attn_fwd(q, k, v.contiguous())
    o3, _, _ = K.attn_fwd(q, k, v)
    assert torch.equal(o1, o2) and torch.equal(o1, o3)
    K.check_status()


def test_attention_autograd(K):
    from imfvideo_b200.ops import reference as ref
    from imfvideo_b200.ops.dual import Dual

    torch.manual_seed(0)
    B, L, H = 1, 333, 2
    q, k, v = (torch.randn(B, L, H, 64, device="cuda").bfloat16().requires_grad_(True)
               for _ in range(3))
    go = torch.randn(B, L, H, 64, device="cuda").bfloat16()
    out = K.attention_dual(Dual(q), Dual(k), Dual(v)).p
    out.backward(go)
    qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    ref.attention(qf, kf, vf).backward(go.float())
    for a, b in ((q, qf), (k, kf), (v, vf)):
        assert _rel(a.grad, b.grad) < 2e-2
    K.check_status()


@pytest.mark.parametrize("B,L,H,hd", [(1, 257, 1, 64), (1, 532, 4, 64), (2, 500, 3, 128),
                                      (1, 2500, 9, 64), (1, 2500, 9, 128)])
def test_attention_backward_split_tiles(K, B, L, H, hd):
    """K/V tiles whose query walk is cut into parts: all of them (few tiles), the ragged last one,
    and (2500 rows, 9 heads: 180 tiles) only those behind the last full wave.  Four roundings to
    bf16 (P, dS, operands, result) of at most 2^-9 each bound the relative error."""
    from imfvideo_b200.ops import reference as ref

    g = torch.Generator(device="cuda").manual_seed(L)
    q, k, v, go = (torch.randn(B, L, H, hd, device="cuda", generator=g).bfloat16() for _ in range(4))
    o, _, lse = K.attn_fwd(q, k, v)
    got = K.attn_bwd(q, k, v, o, lse, go)
    qf, kf, vf = (t.float().requires_grad_(True) for t in (q, k, v))
    ref.attention(qf, kf, vf).backward(go.float())
    for a, b in zip(got, (qf.grad, kf.grad, vf.grad)):
        assert _rel(a, b) < 8e-3
    again = K.attn_bwd(q, k, v, o, lse, go)
    assert torch.equal(got[1], again[1]) and torch.equal(got[2], again[2])   # parts: fixed order
    K.set_deterministic(True)
    try:
        first, second = (K.attn_bwd(q, k, v, o, lse, go)[0] for _ in range(2))
    finally:
        K.set_deterministic(False)
    assert torch.equal(first, second) and _rel(first, got[0]) < 1e-3
    K.check_status()


@pytest.mark.parametrize("hd", [64, 128])
def test_calls_on_two_streams(K, hd):
    """Forward (shares of few items), backward (split tiles), split-K weight gradients and
    Newton-Schulz (same shape, other values) issued on two streams in turn: what they compute one
    after the other.  Equal bits but for dQ, whose fp32 additions land in arrival order (bf16
    result: 2^-9)."""
    g = torch.Generator(device="cuda").manual_seed(hd)
    mk = lambda *shape: torch.randn(*shape, device="cuda", generator=g).bfloat16()
    sides = [([mk(1, L, H, hd) for _ in range(7)], mk(L, 256), mk(L, 136), mk(4, 256, 2 * hd))
             for L, H in ((2068, 4), (1300, 6))]

    def call(side):
        (q, k, v, go, *t), dy, x, G = side
        o, _, lse = K.attn_fwd(q, k, v)
        o2, do, _ = K.attn_fwd(q, k, v, *t)
        return (o, lse, o2, do, *K.attn_bwd(q, k, v, o, lse, go)[1:], K.gemm_wgrad(dy, x),
                K.newton_schulz(G, (3.4445, -4.7750, 2.0315)), K.attn_bwd(q, k, v, o, lse, go)[0])

    want = [call(side) for side in sides]
    streams = [torch.cuda.Stream() for _ in sides]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(6):
        for i, st in enumerate(streams):
            with torch.cuda.stream(st):
                got[i].append(call(sides[i]))
    torch.cuda.synchronize()
    K.check_status()
    for i in range(2):
        for res in got[i]:
            assert all(torch.equal(a, b) for a, b in zip(res[:-1], want[i][:-1]))
            assert _rel(res[-1], want[i][-1]) < 2e-3


@pytest.mark.parametrize("B,L,H", [(1, 128, 1), (1, 300, 2), (2, 1000, 3), (1, 2049, 2)])
def test_attention_backward(K, B, L, H):
    from imfvideo_b200.ops import reference as ref

    g = torch.Generator(device="cuda").manual_seed(L)
    q, k, v, go = (torch.randn(B, L, H, 64, device="cuda", generator=g).bfloat16() for _ in range(4))
    o, _, lse = K.attn_fwd(q, k, v)
    kvbuf = torch.zeros(B, L, H, 112, dtype=torch.bfloat16, device="cuda")
    dq, dk, dv = K.attn_bwd(q, k, v, o, lse, go, gv_out=kvbuf[..., 48:])
    qf, kf, vf = (t.float().requires_grad_(True) for t in (q, k, v))
    ref.attention(qf, kf, vf).backward(go.float())
    for name, a, b in (("dq", dq, qf.grad), ("dk", dk, kf.grad), ("dv", dv, vf.grad)):
        assert _rel(a, b) < 1.5e-2, (name, _rel(a, b))
    assert (kvbuf[..., :48] == 0).all()        # only the value band was written
    dq2, dk2, dv2 = K.attn_bwd(q, k, v, o, lse, go)
    assert torch.equal(dk, dk2) and torch.equal(dv2, dv.contiguous())
    assert _rel(dq2, dq) < 1e-3              # dQ tiles land in arrival order
    K.check_status()
    K.set_deterministic(True)                # fixed order: bit-identical dQ, same values
    try:
        dq3, dk3, dv3 = K.attn_bwd(q, k, v, o, lse, go)
        dq4, _, _ = K.attn_bwd(q, k, v, o, lse, go)
    finally:
        K.set_deterministic(False)
    assert torch.equal(dk3, dk) and torch.equal(dv3, dv.contiguous())
    assert torch.equal(dq3, dq4) and _rel(dq3, dq) < 1e-3
    K.check_status()


@pytest.mark.parametrize("B,L,H", [(1, 128, 1), (1, 300, 3), (2, 1000, 3), (1, 2049, 2), (1, 2100, 12)])
def test_attention_backward_hd128(K, B, L, H):
    """head_dim 128 reverse mode (64-row query steps, transposed dQ tiles); the last case
    splits the query range of each K/V tile over several CTAs."""
    from imfvideo_b200.ops import reference as ref

    g = torch.Generator(device="cuda").manual_seed(L)
    q, k, v, go = (torch.randn(B, L, H, 128, device="cuda", generator=g).bfloat16() for _ in range(4))
    o, _, lse = K.attn_fwd(q, k, v)
    kvbuf = torch.zeros(B, L, H, 224, dtype=torch.bfloat16, device="cuda")
    dq, dk, dv = K.attn_bwd(q, k, v, o, lse, go, gv_out=kvbuf[..., 96:])
    for h in sorted({0, H // 2, H - 1}):
        sl = slice(h, h + 1)
        qf, kf, vf = (t[:, :, sl].float().requires_grad_(True) for t in (q, k, v))
        ref.attention(qf, kf, vf).backward(go[:, :, sl].float())
        for name, a, b in (("dq", dq, qf.grad), ("dk", dk, kf.grad), ("dv", dv, vf.grad)):
            assert _rel(a[:, :, sl], b) < 1.5e-2, (name, h, _rel(a[:, :, sl], b))
    assert (kvbuf[..., :96] == 0).all()        # only the value band was written
    dq2, dk2, dv2 = K.attn_bwd(q, k, v, o, lse, go)
    assert torch.equal(dk, dk2) and torch.equal(dv2, dv.contiguous())
    assert _rel(dq2, dq) < 1e-3
    K.check_status()


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,Kd", [(264, 200, 800), (128, 328, 768), (136, 40, 760)])
def test_gemm_batched_additive_source(K, a_mn, b_mn, M, N, Kd):
    """Batched products around the K from which the deep ring is taken, with an additive source
    whose last 32-column group is whole, ragged or short; one rounding to bf16 of an fp32 sum."""
    torch.manual_seed(M + N)
    A = torch.randn(3, M, Kd, device="cuda").bfloat16()
    B = torch.randn(3, N, Kd, device="cuda").bfloat16()
    cin = (torch.randn(3, M, N, device="cuda") * 20).bfloat16()
    op = lambda t, mn: t.transpose(1, 2).contiguous() if mn else t
    out = K.gemm_batched(op(A, a_mn), op(B, b_mn), a_mn=a_mn, b_mn=b_mn, cin=cin, alpha=0.5, beta=-2.0)
    ref = 0.5 * A.float() @ B.float().transpose(1, 2) - 2.0 * cin.float()
    assert _rel(out, ref) < 2.5e-3              # rms of a bf16 rounding: 2^-9 / sqrt(3) at most
    if a_mn == b_mn and M % 8 == 0:
        full = K.gemm_batched(op(A, a_mn), op(A, a_mn), a_mn=a_mn, b_mn=a_mn)
        sym = K.gemm_batched(op(A, a_mn), op(A, a_mn), a_mn=a_mn, b_mn=a_mn, sym=True)
        assert torch.equal(sym.triu(), full.triu()) and torch.equal(sym, sym.transpose(1, 2))
    K.check_status()


@pytest.mark.parametrize("k,n,m", [(3, 128, 256), (2, 256, 128), (2, 256, 682), (2, 682, 256),
                                   (4, 1, 256), (1, 448, 128), (1, 520, 1024)])
def test_newton_schulz_kernel(K, k, n, m):
    from imfvideo_b200.ops import reference as ref

    torch.manual_seed(n + m)
    G = torch.randn(k, n, m, device="cuda")
    coeffs = (3.4445, -4.7750, 2.0315)
    X = K.newton_schulz(G, coeffs, steps=5)
    if n == 1:
        assert X is None            # vectors take the torch path
        return
    assert X.shape == (k, n, m)
    for i in range(k):
        R = ref.newton_schulz(G[i], coeffs, steps=5, dtype=torch.float32)
        assert _rel(X[i], R) < 4e-2, (i, _rel(X[i], R))
    K.check_status()


@pytest.mark.parametrize("n,m", [(128, 256), (256, 128), (256, 682)])
@pytest.mark.parametrize("given", [False, True])
def test_newton_schulz_without_steps(K, n, m, given):
    """No iteration: the normalised matrices, as on the torch path (one rounding to bf16, 2^-9, of
    G over a norm there taken in bf16), not memory that no product has written."""
    from imfvideo_b200.optim.moonlight import zeropower_via_newtonschulz5

    G = torch.randn(2, n, m, device="cuda")
    torch.empty(2, n, m, device="cuda").fill_(float("nan"))       # what the allocator hands out next
    out = torch.full((2, n, m), float("nan"), device="cuda").bfloat16() if given else None
    X = zeropower_via_newtonschulz5(G, steps=0, out=out)
    want = G / G.flatten(1).norm(dim=1).view(2, 1, 1)
    assert (X is out) == given and X.dtype == torch.bfloat16
    assert _rel(X, want) < 2.0 ** -8
    K.check_status()


@pytest.mark.parametrize("n,m,mp,shift", [(3, 13, 13, 0), (5, 12, 12, 0), (5, 16, 16, 0), (5, 16, 16, 1),
                                          (5, 16, 16, 2), (4, 13, 16, 0), (33, 24, 24, 0)])
def test_newton_schulz_prepare_forms(K, n, m, mp, shift):
    """The normalise-and-cast launcher takes any row length and address: widths that are no multiple
    of eight, and a source (shift 1) or destination (shift 2) off a 16-byte boundary, go value by
    value.  One rounding to bf16 (2^-9) of an fp32 quotient."""
    k = 3
    src = torch.randn(k * n * m + 1, device="cuda")[int(shift == 1):][:k * n * m].view(k, n, m)
    dst = torch.full((k * n * mp + 2,), 7.0, device="cuda").bfloat16()
    x = dst[int(shift == 2):][:k * n * mp].view(k, n, mp)
    part = torch.empty(k * 32, dtype=torch.float64, device="cuda")
    rc = K._lib.imf_ns_prepare(K._ptr(src), K._ptr(x), k, n, m, mp, K._ptr(part), 1e-7, K._stream())
    assert rc == 0
    want = src / src.flatten(1).norm(dim=1).view(k, 1, 1)
    assert _rel(x[..., :m], want) < 2.0 ** -9 and bool((x[..., m:] == 0).all())
    rest = torch.cat([dst[:int(shift == 2)], dst[int(shift == 2) + k * n * mp:]])
    assert bool((rest == 7.0).all())


def test_batched_gemm_with_additive_source(K):
    torch.manual_seed(0)
    a = torch.randn(3, 200, 136, device="cuda").bfloat16()
    b = torch.randn(3, 96, 136, device="cuda").bfloat16()
    cin = torch.randn(3, 200, 96, device="cuda").bfloat16()
    out = K.gemm_batched(a, b, cin=cin, alpha=0.5, beta=2.0)
    ref = 0.5 * torch.einsum("zmk,znk->zmn", a.float(), b.float()) + 2.0 * cin.float()
    assert _rel(out, ref) < 5e-3
    K.check_status()


@pytest.mark.parametrize("n,kdim,mn", [(200, 136, False), (264, 520, True), (1024, 256, False),
                                       (128, 64, False), (392, 1032, True)])
def test_batched_gemm_symmetric_products(K, n, kdim, mn):
    """X X^T / X^T X and b A + c A A with the symmetric mode (upper tiles + mirror image in
    the epilogue) against the full product: the upper triangle is bit-identical, the result
    exactly symmetric, and both agree with fp32."""
    torch.manual_seed(n)
    Z = 3
    x = (torch.randn(Z, kdim, n, device="cuda") if mn else
         torch.randn(Z, n, kdim, device="cuda")).bfloat16() * 0.1
    full = K.gemm_batched(x, x, a_mn=mn, b_mn=mn)
    sym = K.gemm_batched(x, x, a_mn=mn, b_mn=mn, sym=True)
    xf = x.float().transpose(1, 2) if mn else x.float()
    ref = torch.einsum("zik,zjk->zij", xf, xf)
    assert _rel(sym, ref) < 5e-3
    assert torch.equal(sym, sym.transpose(1, 2))
    iu = torch.triu_indices(n, n, device="cuda")
    # tiles on the diagonal are computed whole, tiles above it are the same launches' tiles
    assert torch.equal(sym[:, iu[0], iu[1]], full[:, iu[0], iu[1]])
    b2 = K.gemm_batched(sym, sym, cin=sym, alpha=2.0, beta=-4.75, sym=True)
    ref2 = 2.0 * torch.einsum("zik,zjk->zij", sym.float(), sym.float()) - 4.75 * sym.float()
    assert _rel(b2, ref2) < 5e-3
    assert torch.equal(b2, b2.transpose(1, 2))
    K.check_status()


@pytest.mark.parametrize("hd,B,L,H", [(64, 1, 9000, 4), (128, 1, 6000, 5)])
def test_attention_backward_bitwise_repeatable_over_several_waves(K, hd, B, L, H):
    """More K/V tiles than SMs (several waves of CTAs, split query ranges): the fixed-order dQ
    accumulation gives bit-identical gradients on every run."""
    g = torch.Generator(device="cuda").manual_seed(hd + L)
    q, k, v, go = (torch.randn(B, L, H, hd, device="cuda", generator=g).bfloat16() for _ in range(4))
    o, _, lse = K.attn_fwd(q, k, v)
    loose = K.attn_bwd(q, k, v, o, lse, go)
    K.set_deterministic(True)
    try:
        first = K.attn_bwd(q, k, v, o, lse, go)
        for _ in range(3):
            again = K.attn_bwd(q, k, v, o, lse, go)
            assert all(torch.equal(a, b) for a, b in zip(first, again))
    finally:
        K.set_deterministic(False)
    assert _rel(first[0], loose[0]) < 1e-3
    K.check_status()


@pytest.mark.parametrize("M,N,Kd", [(20480, 528, 256), (29140, 1000, 200), (58280, 264, 64),
                                    (19000, 768, 256)])
def test_gemm_short_k_many_tiles(K, M, N, Kd):
    """Short-K products with many tiles (the projections of a narrow model on a long sequence):
    ragged M, N and K, a strided A, bit-equal repeats."""
    g = torch.Generator(device="cuda").manual_seed(M + N + Kd)
    a_wide = torch.randn(M, Kd + 24, device="cuda", generator=g).bfloat16()
    a = a_wide[:, 8:8 + Kd]                                   # row pitch != K, 16-byte aligned
    b = torch.randn(N, Kd, device="cuda", generator=g).bfloat16()
    out = K.gemm(a, b, alpha=0.5)
    ref = 0.5 * (a.float() @ b.float().t())
    assert _rel(out, ref) < 4e-3
    idx = torch.tensor([0, 127, 128, M // 2, M - 1], device="cuda")
    assert torch.allclose(out[idx].float(), ref[idx], rtol=2e-2, atol=2e-2 * ref.abs().max().item())
    out2 = K.gemm(a, b, alpha=0.5)
    assert torch.equal(out, out2)
    K.check_status()
