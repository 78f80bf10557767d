"""GPU: the allocation-free attention entry point, called through its exported
C symbol exactly as an external caller would.

Who needs it: callers that cannot allocate device memory (no cudaMalloc where
they run, or no allocator of their own) and so cannot provide the scratch
buffer that the regular entry point takes.  The library keeps that scratch in
a built-in device array instead.  This test checks, on two calls in a row
(the array keeps the first call's contents), that the result equals the
regular entry point's and the plain fp32 formula, and that an oversized request
is refused with an error code rather than launched.  The file name sorts last so every other test has
already run if this one fails under ``-x``.
"""
import ctypes
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _call_noalloc(lib, q, k, v, status):
    B, L, H, hd = q.shape
    o = torch.empty_like(q)
    lse = torch.empty(B, H, L, dtype=torch.float32, device=q.device)
    strides = []
    for t in (q, k, v):
        strides += [t.stride(0), t.stride(1), t.stride(2)]
    arr = (ctypes.c_int64 * 9)(*strides)
    fn = lib.imf_attn_fwd_noalloc
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_void_p] * 5 + [ctypes.c_int] * 4 + [ctypes.c_void_p] + \
                  [ctypes.c_int64] * 3 + [ctypes.c_float, ctypes.c_void_p, ctypes.c_void_p]
    rc = fn(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr(), B, L, H, hd,
            ctypes.cast(arr, ctypes.c_void_p), o.stride(0), o.stride(1), o.stride(2),
            1.0 / math.sqrt(hd), status.data_ptr(), torch.cuda.current_stream().cuda_stream)
    return rc, o, lse


def test_noalloc_entry_matches_regular_entry_twice():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from imfvideo_b200.ops import cuda as cu

    assert cu.available()
    from imfvideo_b200.ops import kernels as K

    lib = ctypes.CDLL(cu.LIB_PATH)          # the exported symbol, not a Python wrapper
    status = K.status_word(torch.device("cuda", 0))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for seed, (B, L, H) in enumerate([(1, 2100, 40), (2, 4000, 24)]):
        assert B * H * math.ceil(L / 384) > sms       # items are split: the scratch is in use
        g = torch.Generator(device="cuda").manual_seed(seed)
        q, k, v = (torch.randn(B, L, H, 64, device="cuda", generator=g).bfloat16() for _ in range(3))
        o_ref, _, lse_ref = K.attn_fwd(q, k, v)
        rc, o, lse = _call_noalloc(lib, q, k, v, status)
        assert rc == 0
        torch.cuda.synchronize()
        K.check_status()
        assert (o.float() - o_ref.float()).abs().max() < 2e-2
        assert ((o.float() - o_ref.float()).norm() / o_ref.float().norm()) < 1e-2
        assert (lse - lse_ref).abs().max() < 1e-3
        if seed == 0:
            # and against the plain fp32 formula (one (batch, head) pair at a time: the score
            # matrix of the whole problem would not be small)
            from imfvideo_b200.ops import reference as ref

            for h in (0, H // 2, H - 1):
                ro = ref.attention(q[:, :, h:h + 1].float(), k[:, :, h:h + 1].float(),
                                   v[:, :, h:h + 1].float())
                assert (o[:, :, h:h + 1].float() - ro).abs().max() < 2e-2
                assert ((o[:, :, h:h + 1].float() - ro).norm() / ro.norm()) < 1e-2


def test_noalloc_entry_rejects_oversize_request():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from imfvideo_b200.ops import cuda as cu

    assert cu.available()
    from imfvideo_b200.ops import kernels as K

    lib = ctypes.CDLL(cu.LIB_PATH)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    q = torch.zeros(1, 64, 1, 64, dtype=torch.bfloat16, device="cuda")
    status = K.status_word(torch.device("cuda", 0))
    # wrong head_dim is refused before anything is launched
    bad = torch.zeros(1, 64, 1, 32, dtype=torch.bfloat16, device="cuda")
    rc, _, _ = _call_noalloc(lib, bad, bad, bad, status)
    assert rc == -1
    if sms <= 160:
        pytest.skip("this GPU never needs more partial slots than the built-in array holds")
    big = torch.zeros(1, 384 * (sms + 1), 1, 64, dtype=torch.bfloat16, device="cuda")
    rc, _, _ = _call_noalloc(lib, big, big, big, status)
    assert rc == -4


@pytest.mark.parametrize("sizes", [((1, 532, 4), (1, 130, 2)), ((2, 2068, 4), (1, 3000, 12))])
def test_short_calls_share_no_scratch(sizes):
    """Problems of fewer work items than SMs leave the built-in array alone: two calls on two
    streams at once give the bits of a call by itself.  Against the regular entry point, which
    spreads such items over several thread blocks, the results differ by the order of fp32 sums
    (rounded to bf16: 2^-9)."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from imfvideo_b200.ops import cuda as cu

    assert cu.available()
    from imfvideo_b200.ops import kernels as K

    lib = ctypes.CDLL(cu.LIB_PATH)
    status = K.status_word(torch.device("cuda", 0))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    xs, alone = [], []
    for seed, (B, L, H) in enumerate(sizes):
        assert B * H * math.ceil(L / 384) < sms
        g = torch.Generator(device="cuda").manual_seed(seed)
        xs.append([torch.randn(B, L, H, 64, device="cuda", generator=g).bfloat16() for _ in range(3)])
        rc, o, lse = _call_noalloc(lib, *xs[-1], status)
        assert rc == 0
        alone.append((o, lse))
        ref_o, _, ref_lse = K.attn_fwd(*xs[-1])
        assert ((o.float() - ref_o.float()).norm() / ref_o.float().norm()) < 4e-3
        assert (lse - ref_lse).abs().max() < 1e-4
    streams = [torch.cuda.Stream() for _ in sizes]
    torch.cuda.synchronize()
    got = []
    for _ in range(20):
        for i, st in enumerate(streams):
            with torch.cuda.stream(st):
                got.append((i, *_call_noalloc(lib, *xs[i], status)))
    torch.cuda.synchronize()
    K.check_status()
    for i, rc, o, lse in got:
        assert rc == 0 and torch.equal(o, alone[i][0]) and torch.equal(lse, alone[i][1])


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("tangent", [False, True])
def test_regular_entry_without_scratch(hd, tangent):
    """The regular C entry takes a null (or too small) scratch where items are fewer than SMs, and
    refuses it where they are more."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from imfvideo_b200.ops import cuda as cu

    assert cu.available()
    from imfvideo_b200.ops import kernels as K

    def call(L, H, nbytes):
        x = [torch.randn(1, L, H, hd, device="cuda", generator=g).bfloat16() for _ in range(6 if tangent else 3)]
        o, do = torch.empty_like(x[0]), torch.empty_like(x[0]) if tangent else None
        lse = torch.empty(1, H, L, device="cuda")
        scr = torch.empty(nbytes, dtype=torch.uint8, device="cuda") if nbytes else None
        rc = K._lib.imf_attn_fwd(*[t.data_ptr() for t in x], *([] if tangent else [None] * 3), o.data_ptr(),
                                 K._ptr(do), lse.data_ptr(), 1, L, H, hd, K._bls_array(x, 18), L * H * hd,
                                 H * hd, hd, 0.1, K._ptr(scr), nbytes,
                                 K.status_word(torch.device("cuda", 0)).data_ptr(), K._stream())
        return rc, x, o, do, lse

    g = torch.Generator(device="cuda").manual_seed(hd)
    for nbytes in (0, 4096):
        assert K._lib.imf_attn_fwd_scratch_bytes_hd(1, 2600, 2, int(tangent), hd) > nbytes
        rc, x, o, do, lse = call(2600, 2, nbytes)
        assert rc == 0
        want = K.attn_fwd(*x, scale=0.1)
        for a, b in zip((o, do), want):
            if a is not None:                      # order of fp32 sums, rounded to bf16 (2^-9)
                assert ((a.float() - b.float()).norm() / b.float().norm()) < 6e-3
        assert (lse - want[2]).abs().max() < 1e-4
        assert call(4000, 40, nbytes)[0] == -1
    K.check_status()


@pytest.mark.parametrize("L,H", [(2600, 8), (3000, 8)])
@pytest.mark.parametrize("nbytes", [0, 4096])
def test_tangent_in_rounds_without_scratch(L, H, nbytes):
    """head_dim 64 with tangent, a null (or too small) scratch, more query tiles than SMs but not more pairs of
    them: taken, whole items in two rounds in the place of shares, with the same results (bounds as above)."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from imfvideo_b200.ops import cuda as cu

    assert cu.available()
    from imfvideo_b200.ops import kernels as K

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("sizes are for 148 SMs")
    assert K._lib.imf_attn_fwd_scratch_bytes_hd(1, L, H, 1, 64) > nbytes
    g = torch.Generator(device="cuda").manual_seed(L)
    xs = [torch.randn(1, L, H, 64, device="cuda", generator=g).bfloat16() for _ in range(6)]
    o, do, lse = torch.empty_like(xs[0]), torch.empty_like(xs[0]), torch.empty(1, H, L, device="cuda")
    scr = torch.empty(nbytes, dtype=torch.uint8, device="cuda") if nbytes else None
    rc = K._lib.imf_attn_fwd(*[t.data_ptr() for t in xs], o.data_ptr(), do.data_ptr(), lse.data_ptr(), 1, L, H, 64,
                             K._bls_array(xs, 18), L * H * 64, H * 64, 64, 0.125, K._ptr(scr), nbytes,
                             K.status_word(torch.device("cuda", 0)).data_ptr(), K._stream())
    assert rc == 0
    for a, b in zip((o, do), K.attn_fwd(*xs)):
        assert ((a.float() - b.float()).norm() / b.float().norm()) < 6e-3
    assert (lse - K.attn_fwd(*xs)[2]).abs().max() < 1e-4
    K.check_status()
