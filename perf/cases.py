"""Benchmark cases: the work a user of this framework has it do, through the entry points a
program calls, with their sizes, inputs, algorithmic work, tolerances and a 64-bit oracle.

Kinds of case
  attn    dense attention on (B, L, H, head_dim) bf16 tensors through ``flash_jvp_attention``:
          "infer" (sampler and guidance passes), "jvp" (value and d/dt tangent, the pass behind
          the training target) and "train" (forward and reverse mode)
  sparse  the cube SLA2 INT8-QAT attention core on tile-major tensors: "jvp" and "train",
          routing included
  block   one transformer block on dual numbers, forward with tangent and reverse mode into
          attached fp32 gradient buffers, as a training step runs it
  ns      the Newton-Schulz orthogonalisation of a batch of equal matrices (optimizer step)
  model   a whole dual pass of a small model: u, du/dt and v
"""

import math

import torch
import torch.nn.functional as F

from imfvideo_b200.models import IMFDiTVideo, flash_jvp_attention
from imfvideo_b200.models.imf_dit_video import TransformerBlock, precompute_axial_rope_3d
from imfvideo_b200.models.sla2 import SLA2CubeQATAttentionImpl
from imfvideo_b200.ops.dual import Dual
from imfvideo_b200.optim.moonlight import zeropower_via_newtonschulz5

PREFIX = 20                    # conditioning tokens in front of the patches
EPS = 1e-5
SITU = (4.0, 25.0)
NS_COEFFS = (3.4445, -4.7750, 2.0315)
EPS_LINEAR = 1e-5


def listed():
    return [
        # sampling on the smallest clip the presets use in a smoke run (4 x 16 x 32 latents)
        dict(name="infer_short", kind="attn", mode="infer", B=1, L=532, H=4, hd=64),
        # guidance / sampler passes of the d=256 model: conditional and unconditional input as one batch
        dict(name="infer_d256", kind="attn", mode="infer", B=2, L=29140, H=4, hd=64),
        # the training target's value + tangent pass of the d=256 model
        dict(name="jvp_d256", kind="attn", mode="jvp", B=1, L=29140, H=4, hd=64),
        # forward and reverse mode of the d=256 model
        dict(name="train_d256", kind="attn", mode="train", B=1, L=29140, H=4, hd=64),
        # training on short clips, two of them per GPU (4 x 32 x 64 latents)
        dict(name="train_clip", kind="attn", mode="train", B=2, L=2068, H=4, hd=64),
        # the 16-head d=1024 model on a five-frame latent (5 x 60 x 104)
        dict(name="jvp_d1024_5f", kind="attn", mode="jvp", B=1, L=7820, H=16, hd=64),
        # twelve heads of 128 on the same latent: value + reverse mode
        dict(name="train_hd128_5f", kind="attn", mode="train", B=1, L=7820, H=12, hd=128),
        # cube attention of the d=256 model, top-k 10 %: forward and reverse mode
        dict(name="sparse_train_d256", kind="sparse", mode="train", B=1, gt=20, gh=28, gw=52, H=4,
             topk=0.1),
        # the same attention with tangent on an eight-frame clip
        dict(name="sparse_jvp_clip", kind="sparse", mode="jvp", B=1, gt=8, gh=16, gw=32, H=4,
             topk=0.1),
        # one block of the d=256 model: dual forward and reverse mode
        dict(name="block_d256", kind="block", B=1, gt=20, gh=28, gw=52, d=256, H=4, lora=128),
        # the optimizer's orthogonalisation of one shape of the d=1024 model
        dict(name="ns_d1024", kind="ns", k=24, n=1024, m=1024),
        # a whole dual pass of the smoke-run model: many small launches
        dict(name="model_smoke", kind="model", B=1, gt=4, gh=8, gw=16, d=256, H=4, lora=128, depth=3,
             aux=1),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: sequence lengths from some 130 to 32,780 tokens."""
    most = max(work(c)["flops"] for c in listed())
    while True:
        kind = rng.choice(["attn", "attn", "attn", "attn", "sparse", "block", "ns", "model"])
        if kind == "attn":
            c = dict(kind=kind, mode=rng.choice(["infer", "jvp", "train"]), B=rng.choice([1, 1, 2]),
                     L=_logint(rng, 130, 32780), H=rng.choice([2, 3, 4, 4, 6, 8, 12, 16]),
                     hd=rng.choice([64, 64, 128]))
        elif kind == "sparse":
            c = dict(kind=kind, mode=rng.choice(["jvp", "train"]), B=1, gt=4 * rng.randint(1, 5),
                     gh=4 * rng.randint(2, 7), gw=4 * rng.randint(2, 13), H=rng.choice([2, 4, 6]),
                     topk=round(rng.uniform(0.05, 0.2), 3))
        elif kind == "block":
            d, H, lora = rng.choice([(256, 4, 128), (384, 6, 96), (1024, 16, 512)])
            c = dict(kind=kind, B=rng.choice([1, 2]), gt=rng.randint(1, 20), gh=rng.randint(8, 30),
                     gw=rng.randint(8, 52), d=d, H=H, lora=lora)
        elif kind == "ns":
            c = dict(kind=kind, k=rng.randint(1, 30), n=8 * _logint(rng, 8, 192), m=8 * _logint(rng, 8, 192))
        else:
            c = dict(kind=kind, B=rng.choice([1, 2]), gt=rng.randint(1, 6), gh=rng.randint(4, 12),
                     gw=rng.randint(4, 16), d=256, H=4, lora=128, depth=rng.randint(2, 5), aux=1)
        if work(c)["flops"] <= most:
            return c


# ------------------------------------------------------------------ inputs ---
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, s=1.0, dtype=torch.float32):
    return (torch.randn(*shape, device="cuda", generator=g) * s).to(dtype)


def _length(c):
    return PREFIX + c["gt"] * c["gh"] * c["gw"]


def _qkv(c, g, s=1.0):
    """q, k of unit scale (they leave a per-head norm); v is a band of the wider kv projection."""
    B, L, H, hd = c["B"], c["L"], c["H"], c["hd"]
    q, k = (_randn(g, B, L, H, hd, s=s, dtype=torch.bfloat16) for _ in range(2))
    v = _randn(g, B, L, H, hd + hd // 2, s=s, dtype=torch.bfloat16)[..., hd // 2:]
    return q, k, v


def _cube_qkv(c, g, s=1.0):
    """Tile-major q, k, v: tokens of one 4 x 4 x 4 tile resemble one another, as in a video."""
    B, L, H = c["B"], _length(c), c["H"]
    nb = -(-L // 64)
    mk = lambda: (_randn(g, B, nb, 1, H, 64, s=0.6 * s).expand(B, nb, 64, H, 64)
                  .reshape(B, nb * 64, H, 64)[:, :L] + _randn(g, B, L, H, 64, s=0.8 * s)).bfloat16()
    return mk(), mk(), mk()


def _fill(module, g, bias):
    """Weights of a model some way into training: nothing is exactly zero or one."""
    with torch.no_grad():
        for p in module.parameters():
            p.copy_(p + _randn(g, *p.shape, s=bias))


def _block(c, g):
    hd = c["d"] // c["H"]
    rope = max(2, hd // 4)
    torch.manual_seed(0)
    blk = TransformerBlock(c["d"], c["H"], c["d"] // 2, c["lora"], hd - rope, rope, hd,
                           weight_init_constant=0.5, norm_eps=EPS, attn_impl=flash_jvp_attention,
                           situ_beta=SITU[0], situ_linear_beta=SITU[1]).cuda()
    _fill(blk, g, 0.02)
    with torch.no_grad():
        for gate in (blk.attn_scale, blk.mlp_scale):
            gate.add_(_randn(g, c["d"], s=0.3) + 0.5)
    cos, sin = precompute_axial_rope_3d(rope, (c["gt"], c["gh"], c["gw"]), PREFIX)
    return blk, cos.cuda(), sin.cuda()


def _model(c, g):
    torch.manual_seed(0)
    net = IMFDiTVideo(input_size=(2 * c["gh"], 2 * c["gw"]), num_frames=c["gt"], hidden_size=c["d"],
                      depth=c["depth"], aux_head_depth=c["aux"], num_heads=c["H"],
                      kv_lora_rank=c["lora"], weight_init_constant=0.5, rmsnorm_eps=EPS,
                      attn_impl=flash_jvp_attention, attn_res_block_size=2,
                      compute_dtype=torch.bfloat16).cuda()
    _fill(net, g, 0.02)
    return net


def prepare(case, seed):
    c, g = case, _gen(seed)
    if c["kind"] == "attn":
        q, k, v = _qkv(c, g)
        if c["mode"] == "jvp":
            return dict(c=c, x=(q, k, v), t=_qkv(c, g, 0.5))
        if c["mode"] == "train":
            go = _randn(g, c["B"], c["L"], c["H"], c["hd"], dtype=torch.bfloat16)
            return dict(c=c, x=tuple(z.requires_grad_() for z in (q, k, v)), go=go)
        return dict(c=c, x=(q, k, v))
    if c["kind"] == "sparse":
        L = _length(c)
        impl = SLA2CubeQATAttentionImpl(64, L, c["H"], (c["gt"], c["gh"], c["gw"]), topk=c["topk"],
                                        pre_permuted=True).cuda()
        with torch.no_grad():
            impl.proj_q.add_(_randn(g, 64, 64, s=0.05))
            impl.proj_k.add_(_randn(g, 64, 64, s=0.05))
            impl.alpha_logit.add_(_randn(g, *impl.alpha_logit.shape, s=0.5))
        x = _cube_qkv(c, g)
        if c["mode"] == "jvp":
            return dict(c=c, impl=impl, x=x, t=_cube_qkv(c, g, 0.5))
        return dict(c=c, impl=impl, x=x, go=_randn(g, c["B"], L, c["H"], 64, dtype=torch.bfloat16))
    if c["kind"] == "block":
        blk, cos, sin = _block(c, g)
        for p in blk.parameters():
            p.grad = torch.zeros_like(p)
        L = _length(c)
        return dict(c=c, blk=blk, rope=(cos, sin), x=_randn(g, c["B"], L, c["d"]).requires_grad_(),
                    dx=_randn(g, c["B"], L, c["d"], s=0.5), go=_randn(g, c["B"], L, c["d"]),
                    grads=[p.grad for p in blk.parameters()])
    if c["kind"] == "ns":
        return dict(c=c, G=_randn(g, c["k"], c["n"], c["m"], s=0.01))
    net = _model(c, g)
    B, shape = c["B"], (c["B"], 16, c["gt"], 2 * c["gh"], 2 * c["gw"])
    u = lambda: torch.rand(B, device="cuda", generator=g)
    return dict(c=c, net=net, x=_randn(g, *shape), dx=_randn(g, *shape), h=u(), w=1 + u(), lo=0.2 * u(),
                hi=1 - 0.2 * u(), y=torch.randint(0, 1000, (B,), device="cuda", generator=g))


# ------------------------------------------------------------------- a pass ---
def run(state):
    c = state["c"]
    if c["kind"] == "attn":
        q, k, v = state["x"]
        if c["mode"] == "train":
            o = flash_jvp_attention(q, k, v)
            return [o] + list(torch.autograd.grad(o, (q, k, v), state["go"]))
        with torch.no_grad():
            if c["mode"] == "jvp":
                out = flash_jvp_attention(*(Dual(a, b) for a, b in zip(state["x"], state["t"])))
                return [out.p, out.t]
            return [flash_jvp_attention(q, k, v)]
    if c["kind"] == "sparse":
        impl, (q, k, v) = state["impl"], state["x"]
        core = impl.fused_core
        with torch.no_grad():
            if c["mode"] == "jvp":
                o, do, _ = core.fwd(q, k, v, *state["t"], False)
                return [o, do]
            o, _, saved = core.fwd(q, k, v, None, None, None, True)
            impl.alpha_logit.grad = None
            grads = core.bwd(q, k, v, o, saved, state["go"])
            return [o, *grads, impl.alpha_logit.grad]
    if c["kind"] == "block":
        blk, x = state["blk"], state["x"]
        torch._foreach_zero_(state["grads"])
        x.grad = None
        out = blk(Dual(x, state["dx"]), *state["rope"], torch.bfloat16)
        out.p.backward(state["go"])
        return [out.p, out.t, x.grad] + state["grads"]
    if c["kind"] == "ns":
        return [zeropower_via_newtonschulz5(state["G"], steps=5, dtype=torch.bfloat16, coeffs=NS_COEFFS)]
    s = state
    with torch.no_grad():
        out = s["net"].forward_dual(Dual(s["x"], s["dx"]), Dual(s["h"], torch.ones_like(s["h"])), s["w"],
                                    s["lo"], s["hi"], s["y"])
    return [out["u"].p, out["u"].t, out["v"].p]


# ---------------------------------------------------------- what it has to do ---
def _block_gemm_flops(d, H, lora, rows):
    hv, f, dq, rope = d, int(d * 8 / 3), d // 2, max(2, d // H // 4)
    per_row = d * (dq + lora + rope + hv) + dq * d + lora * (2 * d - H * rope) + hv * d + 3 * d * f
    return 2.0 * rows * per_row


def work(case):
    c = case
    if c["kind"] == "attn":
        row = c["B"] * c["L"] * c["H"] * c["hd"] * 2
        pair = 4.0 * c["B"] * c["H"] * c["L"] ** 2 * c["hd"]
        mul, tensors = {"infer": (1, 4), "jvp": (3, 8), "train": (3.5, 8)}[c["mode"]]
        return {"bytes": tensors * row, "flops": mul * pair}
    if c["kind"] == "sparse":
        L = _length(c)
        row = c["B"] * L * c["H"] * 64 * 2
        live = c["topk"] + PREFIX / L
        sparse = 4.0 * c["B"] * c["H"] * L * L * 64 * live
        nb = -(-L // 64)
        linear = 4.0 * c["B"] * c["H"] * (L * 64 * 64 + nb * nb * 64 * 65 / 2)
        mul, tensors = (3, 8) if c["mode"] == "jvp" else (3.5, 8)
        return {"bytes": tensors * row, "flops": mul * (sparse + linear)}
    if c["kind"] == "block":
        rows = c["B"] * _length(c)
        gemm = _block_gemm_flops(c["d"], c["H"], c["lora"], rows)
        attn = 4.0 * c["B"] * _length(c) ** 2 * c["d"]
        return {"bytes": 6.0 * rows * c["d"] * 4, "flops": 4 * gemm + 5.5 * attn}
    if c["kind"] == "ns":
        g, r = min(c["n"], c["m"]), max(c["n"], c["m"])
        return {"bytes": c["k"] * c["n"] * c["m"] * 6, "flops": 5 * 2.0 * c["k"] * (2 * g * g * r + g ** 3)}
    rows = c["B"] * _length(c)
    trunk, v = c["depth"], c["aux"]
    gemm = _block_gemm_flops(c["d"], c["H"], c["lora"], rows)
    attn = 4.0 * c["B"] * _length(c) ** 2 * c["d"]
    return {"bytes": (3 * 2 + v) * 16 * 4.0 * rows + (trunk + v) * 900000.0 * 4,
            "flops": trunk * (2 * gemm + 3 * attn) + v * (gemm + attn)}


def tolerance(case):
    """About four times what two correct bf16 evaluations of the same formulas differ by (the
    error of the present code against the 64-bit oracle; fp32 sums, bf16 operands and results)."""
    c = case
    if c["kind"] == "attn":
        return {"rel": 1.2e-2, "max": 0.25}
    if c["kind"] == "sparse":
        return {"rel": 2e-2, "max": 0.5}
    if c["kind"] == "block":
        return {"rel": 2e-2, "max": 0.5}
    if c["kind"] == "ns":
        return {"rel": 3e-2, "max": 0.25}       # five bf16 iterations: 1e-2 off the 64-bit result
    return {"rel": 2e-2, "max": 0.5}


# ------------------------------------------------------------- 64-bit oracle ---
def _rows64(L, heads):
    return max(16, min(L, (1 << 28) // (L * heads)))       # query rows per chunk: 2 GiB of scores


def _attn64(q, k, v, dq=None, dk=None, dv=None, go=None):
    """(o, do, (gq, gk, gv)) of dense attention on (B, L, H, d) tensors, chunked over rows."""
    sc = q.shape[-1] ** -0.5
    q, k, v, dq, dk, dv, go = (None if z is None else z.detach().double().transpose(1, 2)
                               for z in (q, k, v, dq, dk, dv, go))
    B, H, L, _ = q.shape
    o = torch.empty_like(v)
    do = torch.empty_like(v) if dq is not None else None
    gq, gk, gv = (torch.zeros_like(z) for z in (q, k, v)) if go is not None else (None,) * 3
    step = _rows64(L, B * H)
    for i in range(0, L, step):
        r = slice(i, i + step)
        p = torch.softmax(q[:, :, r] @ k.transpose(-1, -2) * sc, -1)
        o[:, :, r] = p @ v
        if dq is not None:
            ds = (dq[:, :, r] @ k.transpose(-1, -2) + q[:, :, r] @ dk.transpose(-1, -2)) * sc
            ds = p * (ds - (p * ds).sum(-1, keepdim=True))
            do[:, :, r] = ds @ v + p @ dv
        if go is not None:
            gv += p.transpose(-1, -2) @ go[:, :, r]
            dp = go[:, :, r] @ v.transpose(-1, -2)
            ds = p * (dp - (go[:, :, r] * o[:, :, r]).sum(-1, keepdim=True)) * sc
            gq[:, :, r] = ds @ k
            gk += ds.transpose(-1, -2) @ q[:, :, r]
    back = lambda z: None if z is None else z.transpose(1, 2)
    return back(o), back(do), tuple(back(z) for z in (gq, gk, gv))


class _Attn64(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v):
        ctx.save_for_backward(q, k, v)
        return _attn64(q, k, v)[0]

    @staticmethod
    def backward(ctx, go):
        return _attn64(*ctx.saved_tensors, go=go)[2]


def _fake_quant64(x):
    """Per 64-row block and head, (B, L, H, 64): symmetric 8-bit grid, half away from zero."""
    B, L, H, D = x.shape
    nb = -(-L // 64)
    z = F.pad(x.double(), (0, 0, 0, 0, 0, nb * 64 - L)).view(B, nb, 64, H, D)
    s = z.abs().amax((2, 4), keepdim=True) / 127 + 1e-12
    y = torch.sign(z) * torch.floor((z / s).abs() + 0.5)
    return (y.clamp(-127, 127) * s).view(B, nb * 64, H, D)[:, :L]


def _block_mean64(x, n):
    B, L, H, D = x.shape
    pad = n * 64 - L
    z = F.pad(x.double(), (0, 0, 0, 0, 0, max(0, pad)))[:, :n * 64].view(B, n, 64, H, D).sum(2)
    cnt = torch.full((n,), 64.0, dtype=torch.double, device=x.device)
    if pad > 0:
        cnt[-1] = 64 - pad
    return (z / cnt.view(1, n, 1, 1)).permute(0, 2, 1, 3)


def _sparse64(s):
    """Cube attention: routed blocks + always-attended prefix in the softmax branch on the 8-bit
    grid of q, k, v (straight-through), complement in the linear branch, mixed by alpha."""
    c, impl = s["c"], s["impl"]
    x = [z.detach() for z in s["x"]]
    B, L, H, D = x[0].shape
    Np, rows = impl.Np, impl.a_index
    nb = -(-L // 64)
    T = max(1, min(Np, int(c["topk"] * Np)))
    qb = _block_mean64(x[0], impl.Mb) @ impl.proj_q.detach().double().t()
    kb = _block_mean64(x[1], Np) @ impl.proj_k.detach().double().t()
    top = torch.topk(qb @ kb.transpose(-1, -2), T, -1).indices
    sel = torch.zeros(B, H, impl.Mb, nb, device="cuda", dtype=torch.bool).scatter_(-1, top, True)
    sel[..., Np:] = True
    key_blk = torch.arange(L, device="cuda") // 64
    a = torch.sigmoid(impl.alpha_logit.detach().double())
    head = lambda z, b, h: z[b, :, h].detach().double()
    fq = [_fake_quant64(z) for z in x]
    jvp = c["mode"] == "jvp"
    o = torch.zeros(B, L, H, D, dtype=torch.double, device="cuda")
    do = torch.zeros_like(o) if jvp else None
    g = None if jvp else [torch.zeros_like(o) for _ in range(3)]
    ga = torch.zeros_like(a)
    sc = D ** -0.5
    step = _rows64(L, 2)
    phi = lambda z: torch.softmax(z, -1)
    dphi = lambda p, dz: p * (dz - (p * dz).sum(-1, keepdim=True))
    for b in range(B):
        for h in range(H):
            q, k, v = (head(z, b, h) for z in x)
            qs, ks, vs = (z[b, :, h] for z in fq)
            fk = phi(k)
            if jvp:
                dq, dk, dv = (head(z, b, h) for z in s["t"])
                dfk = dphi(fk, dk)
            else:
                go_, gfk = head(s["go"], b, h), torch.zeros_like(fk)
            for i in range(0, L, step):
                r = slice(i, min(L, i + step))
                m = sel[b, h, rows[r]][:, key_blk]
                p = torch.softmax((qs[r] @ ks.t() * sc).masked_fill(~m, -math.inf), -1)
                os_ = p @ vs
                fq_ = phi(q[r])
                wl = (fq_ @ fk.t()).masked_fill(m, 0.0)
                den = wl.sum(-1, keepdim=True) + EPS_LINEAR
                ol = wl @ v / den
                ar = a[h, rows[r]].unsqueeze(-1)
                o[b, r, h] = ar * os_ + (1 - ar) * ol
                if jvp:
                    ds = (dq[r] @ k.t() + q[r] @ dk.t()) * sc
                    ds = p * (ds - (p * ds).sum(-1, keepdim=True))
                    dos = ds @ v + p @ dv
                    dwl = (dphi(fq_, dq[r]) @ fk.t() + fq_ @ dfk.t()).masked_fill(m, 0.0)
                    dol = (dwl @ v + wl @ dv - dwl.sum(-1, keepdim=True) * ol) / den
                    do[b, r, h] = ar * dos + (1 - ar) * dol
                    continue
                gr = go_[r]
                ga[h].index_add_(0, rows[r], ((os_ - ol) * gr).sum(-1) * (ar * (1 - ar)).squeeze(-1))
                gos, gol = ar * gr, (1 - ar) * gr
                ds = p * (gos @ vs.t() - (gos * os_).sum(-1, keepdim=True)) * sc
                gnum = gol / den
                gw = (gnum @ v.t() - (gol * ol).sum(-1, keepdim=True) / den).masked_fill(m, 0.0)
                g[0][b, r, h] = ds @ ks + dphi(fq_, gw @ fk)
                g[1][b, :, h] += ds.t() @ qs[r]
                g[2][b, :, h] += p.t() @ gos + wl.t() @ gnum
                gfk += gw.t() @ fq_
            if not jvp:
                g[1][b, :, h] += dphi(fk, gfk)
    return [o, do] if jvp else [o, *g, ga]


def _rms64(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w


def _rope64(x, cos, sin):
    a, b, c, s = x[..., 0::2], x[..., 1::2], cos[None, :, None, :], sin[None, :, None, :]
    return torch.stack([a * c - b * s, a * s + b * c], -1).flatten(-2)


def _remix64(cands, w):
    v = torch.stack(cands, -2)
    s = ((v * torch.rsqrt(v.square().mean(-1, keepdim=True) + EPS)) * w).sum(-1)
    return (torch.softmax(s, -1).unsqueeze(-1) * v).sum(-2)


def _pre64(P, H, cos, sin, x):
    """Residual stream -> (q, k, v, gate) of a block; P: its parameters by name, 64 bits."""
    B, L, d = x.shape
    hd = d // H
    dr = 2 * cos.shape[-1]
    dn, dc = hd - dr, P["attn.kv_b_proj.weight"].shape[1]
    n = _rms64(x, P["norm1.weight"])
    kva = n @ P["attn.kv_a_proj.weight"].t()
    q = _rms64(n @ P["attn.q_a_proj.weight"].t(), P["attn.q_a_layernorm.weight"]) \
        @ P["attn.q_b_proj.weight"].t()
    kv = _rms64(kva[..., :dc], P["attn.kv_a_layernorm.weight"]) @ P["attn.kv_b_proj.weight"].t()
    q, kv = q.view(B, L, H, hd), kv.view(B, L, H, dn + hd)
    kr = _rope64(kva[..., dc:].unsqueeze(2), cos, sin).expand(B, L, H, dr)
    qf = torch.cat([_rms64(q[..., :dn], P["attn.q_norm.weight"]), _rope64(q[..., dn:], cos, sin)], -1)
    kf = torch.cat([_rms64(kv[..., :dn], P["attn.k_norm.weight"]), kr], -1)
    return qf, kf, kv[..., dn:], n @ P["attn.g_proj.weight"].t()


def _attn_out64(P, o, gate):
    return (o.flatten(2) * torch.sigmoid(gate)) @ P["attn.out_proj.weight"].t() * P["attn_scale"]


def _mlp64(P, h):
    n = _rms64(h, P["norm2.weight"])
    g, u = n @ P["mlp.w1.weight"].t(), n @ P["mlp.w3.weight"].t()
    act = SITU[0] * torch.tanh(g / SITU[0]) * torch.sigmoid(g) * SITU[1] * torch.tanh(u / SITU[1])
    return act @ P["mlp.w2.weight"].t() * P["mlp_scale"]


def _params64(module, grad=False):
    return {n: p.detach().double().requires_grad_(grad) for n, p in module.named_parameters()}


def _block64(s):
    c, blk = s["c"], s["blk"]
    P = _params64(blk, True)
    cos, sin = (z.double() for z in s["rope"])
    x = s["x"].detach().double().requires_grad_()
    pre = lambda z: _pre64(P, c["H"], cos, sin, z)

    def post(z, o, gate):
        z = z + _attn_out64(P, o, gate)
        return z + _mlp64(P, z)
    q, k, v, gate = pre(x)
    out = post(x, _Attn64.apply(q, k, v), gate)
    out.backward(s["go"].double())
    with torch.no_grad():
        dx = s["dx"].double()
        (q, k, v, gate), (dq, dk, dv, dgate) = torch.func.jvp(pre, (x.detach(),), (dx,))
        o, do, _ = _attn64(q, k, v, dq, dk, dv)
        _, dout = torch.func.jvp(post, (x.detach(), o, gate), (dx, do, dgate))
    return [out.detach(), dout, x.grad] + [P[n].grad for n, _ in blk.named_parameters()]


def _ns64(s):
    X = s["G"].double()
    X = X / (X.flatten(1).norm(dim=1).view(-1, 1, 1) + 1e-7)
    tall = X.shape[1] > X.shape[2]
    X = X.transpose(1, 2) if tall else X
    a, b, c = NS_COEFFS
    for _ in range(5):
        A = X @ X.transpose(1, 2)
        X = a * X + (b * A + c * (A @ A)) @ X
    return [X.transpose(1, 2) if tall else X]


def _model64(s):
    """The whole network as a function of (x, h), its value and derivative along (dx, 1)."""
    c, net = s["c"], s["net"]
    P = _params64(net)
    sub = lambda pre: {n[len(pre):]: p for n, p in P.items() if n.startswith(pre)}
    cos, sin = net.rope_cos.double(), net.rope_sin.double()
    H, bs = c["H"], net.attn_res_block_size
    half = 128
    freqs = torch.exp(-math.log(10000.0) * torch.arange(half, dtype=torch.double, device="cuda") / half)

    def time(pre, t):
        Q = sub(pre)
        e = t[:, None] * freqs
        e = torch.cat([torch.cos(e), torch.sin(e)], -1)
        return F.silu(e @ Q["mlp.0.weight"].t() + Q["mlp.0.bias"]) @ Q["mlp.2.weight"].t() + Q["mlp.2.bias"]

    def dense(q, k, v):
        q, k, v = (z.transpose(1, 2) for z in (q, k, v))
        return (torch.softmax(q @ k.transpose(-1, -2) * q.shape[-1] ** -0.5, -1) @ v).transpose(1, 2)

    def blocks(prefix, snaps, name, n, first):
        for j in range(n):
            Q = sub("%s.%d." % (name, j))
            fresh = (first + j) % bs == 0
            w1, w2 = (Q[m + "_norm.weight"] * Q[m + "_proj.weight"].reshape(-1) for m in ("attn_res", "mlp_res"))
            h = _remix64(snaps + [prefix], w1) if snaps else prefix
            q, k, v, gate = _pre64(Q, H, cos, sin, h)
            a = _attn_out64(Q, dense(q, k, v), gate)
            snaps, prefix = (snaps + [prefix], a) if fresh else (snaps, prefix + a)
            prefix = prefix + _mlp64(Q, _remix64(snaps + [prefix], w2))
        return prefix, snaps

    def net64(x, h):
        B = x.shape[0]
        gt, gh, gw = net.grid_size
        rows = x.view(B, 16, gt, gh, 2, gw, 2).permute(0, 2, 3, 5, 1, 4, 6).reshape(B, gt * gh * gw, 64)
        xe = rows @ P["x_embedder.proj.weight"].flatten(1).t() + P["x_embedder.proj.bias"]
        bank = lambda tok, e: P[tok] + e.unsqueeze(1)
        seq = torch.cat([bank("class_tokens", P["y_embedder.embedding_table.weight"][s["y"]]),
                         bank("omega_tokens", time("omega_embedder.", 1 - 1 / s["w"].double())),
                         bank("t_min_tokens", time("cfg_t_start_embedder.", s["lo"].double())),
                         bank("t_max_tokens", time("cfg_t_end_embedder.", s["hi"].double())),
                         bank("time_tokens", time("h_embedder.", h)), xe], 1)
        shared = c["depth"] - c["aux"]
        trunk, snaps = blocks(seq, [], "shared_blocks", shared, 0)
        out = []
        for b in ("u", "v"):
            z, sn = blocks(trunk, snaps, b + "_heads", c["aux"], shared)
            z = _remix64(sn + [z], P[b + "_out_res_norm.weight"] * P[b + "_out_res_proj.weight"].reshape(-1))
            z = _rms64(z[:, PREFIX:], P[b + "_final_layer.norm.weight"]) \
                @ P[b + "_final_layer.linear.weight"].t() + P[b + "_final_layer.linear.bias"]
            out.append(z.view(B, gt, gh, gw, 1, 2, 2, 16).permute(0, 7, 1, 4, 2, 5, 3, 6).reshape(x.shape))
        return tuple(out)
    (u, v), (du, _) = torch.func.jvp(net64, (s["x"].double(), s["h"].double()),
                                     (s["dx"].double(), torch.ones_like(s["h"]).double()))
    return [u, du, v]


def exact(case, seed):
    s = prepare(case, seed)
    if case["kind"] == "attn":
        if case["mode"] == "jvp":
            o, do, _ = _attn64(*s["x"], *s["t"])
            return [o, do]
        o, _, g = _attn64(*s["x"], go=s.get("go"))
        return [o, *g] if case["mode"] == "train" else [o]
    with torch.no_grad():
        if case["kind"] == "sparse":
            return _sparse64(s)
        if case["kind"] == "ns":
            return _ns64(s)
        if case["kind"] == "model":
            return _model64(s)
    return _block64(s)
