"""Performance cases: the calls that a diffusion transformer's attention blocks make through ``zdraw_b200.mattn``.

Four kinds of pass, each through the public entry points as a model's forward calls them:

* ``joint``  one joint text+image attention call on device tensors (q/k norm + RoPE, then attention):
             ``Context.joint_attention``
* ``block``  the attention sub-block: q/k/v projection of one activation, attention, output projection:
             ``Context.qkv_projection``, ``Context.run_on_handles``, ``Context.linear``
* ``wide``   the one-head attention of an image decoder's middle block: ``Context.wide_attention``
* ``host``   the joint call with q, k, v and the result in pinned host memory:
             ``Context.set_device_tables``, ``Context.joint_attention_host``

Shapes are those of ``zdraw_b200.workloads`` and of the benchmark, the same layers at smaller images, and
ragged ones. Values: activations N(0, 1), norm weights U(0.8, 1.2), projection weights N(0, 1/k), RoPE tables
of the token grid. Inputs are drawn on the GPU from the seed.
"""
from __future__ import annotations

import math

import torch

from zdraw_b200 import mattn
from zdraw_b200._lib import DTYPE_F16, DTYPE_F32, AttnParams, LinearParams

D = 128  # head_dim of the joint attention
DEVICE = "cuda"


def _joint(name, family, batch, heads, text, grid_h, grid_w, ref_h=0, ref_w=0, dtype="f16", masked=0, of_heads=0,
           kind="joint"):
    case = {"kind": kind, "family": family, "batch": batch, "heads": heads, "text": text, "grid_h": grid_h,
            "grid_w": grid_w, "ref_h": ref_h, "ref_w": ref_w, "dtype": dtype, "masked": masked, "of_heads": of_heads}
    return {"name": name, **case} if name else case


def _wide(name, tokens, channels):
    case = {"kind": "wide", "tokens": tokens, "channels": channels}
    return {"name": name, **case} if name else case


def listed():
    return [
        # The smallest call: 16 text + 8x8 image tokens, 2 heads, f32 tensors. Latency and launches.
        _joint("tiny_f32", "klein", 1, 2, 16, 8, 8, dtype="f32"),
        # One attention call of the 24-head model for a 256-pixel preview image (512 text + 16x16 tokens).
        _joint("klein_256", "klein", 1, 24, 512, 16, 16),
        # The same at 512 pixels.
        _joint("klein_512", "klein", 1, 24, 512, 32, 32),
        # The same at 1024 pixels: the model's default image, 100 such calls per picture.
        _joint("klein_1024", "klein", 1, 24, 512, 64, 64),
        # The 30-head single-stream model on an odd picture: 45x45 image tokens (padded to 2048), 77 caption
        # tokens, a token count that is no multiple of any tile.
        _joint("zimage_ragged", "zimage", 1, 30, 77, 45, 45),
        # Editing with a reference image: text + target + reference tokens, 128 of the text keys masked.
        _joint("klein_edit", "klein", 1, 24, 512, 64, 64, 64, 64, masked=128),
        # The largest image, two seeds in one call.
        _joint("klein_2048_x2", "klein", 2, 24, 512, 128, 128),
        # A whole attention sub-block (projections included) at 512 and at 1024 pixels.
        _joint("block_512", "klein", 1, 24, 512, 32, 32, kind="block"),
        _joint("block_1024", "klein", 1, 24, 512, 64, 64, kind="block"),
        # The decoder's middle-block attention for a 512-pixel and a 1024-pixel picture.
        _wide("wide_512", 4096, 512),
        _wide("wide_1024", 16384, 512),
        # The call of a program that keeps its activations on the host (the benchmark's end-to-end figure).
        _joint("host_1024", "klein", 1, 24, 512, 64, 64, kind="host"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["joint", "joint", "joint", "block", "wide", "host"])
    if kind == "wide":  # token counts are multiples of 32 (the entry point takes no others)
        return _wide("", 32 * _log_int(rng, 16, 512), rng.choice([256, 512, 512, 512]))
    family = rng.choice(["klein", "klein", "zimage"])
    most = {"joint": 128, "block": 80, "host": 64}[kind]
    grid_h, grid_w = _log_int(rng, 8, most), _log_int(rng, 8, most)
    text = _log_int(rng, 16, 512)
    ref_h = ref_w = masked = of_heads = 0
    heads = rng.choice([24, 30, rng.randint(2, 32)])
    batch, dtype = 1, "f16"
    if kind == "joint":
        option = rng.choice(["", "", "batch", "edit", "shard", "f32"])
        if option == "edit" and family == "klein":
            ref_h, ref_w, masked = grid_h, grid_w, rng.randint(1, text)
        elif option == "batch":
            batch = rng.randint(2, 8)
        elif option == "shard":  # a column slice of a wider tensor: the share of one GPU of several
            of_heads, heads = heads, rng.randint(1, heads)
        elif option == "f32":
            dtype = "f32"
    elif kind == "block":
        batch = rng.choice([1, 1, 2])
    case = _joint("", family, batch, heads, text, grid_h, grid_w, ref_h, ref_w, dtype, masked, of_heads, kind)
    while case["batch"] > 1 and work(case)["flops"] > 7.0e12:
        case["batch"] -= 1
    return case


# ------------------------------------------------------------------------------------------------ sizes
def _tokens(c):
    image = c["grid_h"] * c["grid_w"]
    if c["family"] == "zimage":
        image += mattn.zimage_pad_len(image)
    return c["text"] + image + c["ref_h"] * c["ref_w"]


def work(case):
    """What one pass cannot do without: each input read once, each output written once, the products' FLOPs
    over the keys that are not masked."""
    if case["kind"] == "wide":
        t, d = case["tokens"], case["channels"]
        return {"bytes": 4 * t * d * 4, "flops": 4 * t * t * d}
    s, h, b = _tokens(case), case["heads"], case["batch"]
    elem = 4 if case["dtype"] == "f32" else 2
    small = 2 * s * D * 4 + 4 * D * 4 + (4 * s if case["masked"] else 0)  # tables, norm weights, key mask
    attention = 4 * b * h * s * (s - case["masked"]) * D
    if case["kind"] == "block":
        n = h * D
        return {"bytes": 2 * b * s * n * 2 + 4 * n * n * 2 + small, "flops": 4 * 2 * b * s * n * n + attention}
    return {"bytes": 4 * b * s * h * D * elem + small, "flops": attention}


def tolerance(case):
    # Half operands and half probabilities (also behind f32 tensors), f32 sums. Against float64 from the same
    # inputs the listed cases differ by rel 3.9e-4 to 4.3e-4 and max 2.9e-3, the blocks by rel 4.7e-4 to 5.0e-4.
    return {"rel": 2e-3 if case["kind"] == "block" else 1.8e-3, "max": 1.2e-2}


# ------------------------------------------------------------------------------------------------ inputs
_context = None


def _ctx():
    """The program's one context of this GPU."""
    global _context
    if _context is None:
        _context = mattn.Context(torch.cuda.current_device())
    return _context


def _rope(ctx, c):
    if c["family"] == "klein":
        return ctx.klein_rope_table_device(c["text"], c["grid_h"], c["grid_w"], c["ref_h"], c["ref_w"], theta=2000.0)
    return ctx.zimage_rope_table_device(c["grid_h"], c["grid_w"], c["text"])


def prepare(case, seed):
    ctx = _ctx()
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)

    def normal(*shape, dtype=torch.float16, scale=1.0):
        return (torch.randn(shape, generator=g, device=DEVICE, dtype=torch.float32) * scale).to(dtype)

    if case["kind"] == "wide":
        t, d = case["tokens"], case["channels"]
        q, k, v = (normal(t, d, dtype=torch.float32) for _ in range(3))
        return {"kind": "wide", "ctx": ctx, "q": q, "k": k, "v": v, "out": torch.empty_like(q),
                "cfg": mattn.Config(t, 1, 1, d)}

    s, h, b = _tokens(case), case["heads"], case["batch"]
    klein = case["family"] == "klein"
    code, dtype = (DTYPE_F32, torch.float32) if case["dtype"] == "f32" else (DTYPE_F16, torch.float16)
    st = {"kind": case["kind"], "ctx": ctx}
    st["norm"] = [torch.rand(D, generator=g, device=DEVICE) * 0.4 + 0.8 for _ in range(4)]
    st["cos"], st["sin"] = _rope(ctx, case)
    txt_tokens = case["text"] if klein else 0
    eps = 1e-6 if klein else 1e-5
    st["p"] = AttnParams(batch=b, tokens=s, heads=h, head_dim=D, txt_tokens=txt_tokens, in_dtype=code, out_dtype=code,
                         out_layout=0, qk_layout=1, has_key_mask=1 if case["masked"] else 0, norm_eps=eps)
    st["mask"] = None
    if case["masked"]:
        st["mask"] = torch.zeros(s, dtype=torch.float32, device=DEVICE)
        st["mask"][case["text"] - case["masked"]:case["text"]] = -math.inf

    if case["kind"] == "block":
        n, m = h * D, b * s
        st["x"] = normal(m, n)
        st["w"] = [normal(n, n, scale=n ** -0.5) for _ in range(4)]
        st["q16"], st["k16"] = (torch.empty((b, h, s, D), dtype=torch.float16, device=DEVICE) for _ in range(2))
        st["v"], st["o"] = (torch.empty((b, s, h, D), dtype=torch.float16, device=DEVICE) for _ in range(2))
        st["out"] = torch.empty((m, n), dtype=torch.float16, device=DEVICE)
        st["lp_qkv"] = LinearParams(m=m, n=n, k=n, a_dtype=DTYPE_F16, w_dtype=DTYPE_F16, c_dtype=DTYPE_F16, epilogue=1,
                                    tokens=s, heads=h, txt_tokens=txt_tokens, norm_eps=eps)
        st["lp_out"] = LinearParams(m=m, n=n, k=n, a_dtype=DTYPE_F16, w_dtype=DTYPE_F16, c_dtype=DTYPE_F16)
        return st

    if case["of_heads"]:
        st["p"].ld_q = st["p"].ld_k = st["p"].ld_v = case["of_heads"] * D
    qkv = [normal(b, s, case["of_heads"] or h, D, dtype=dtype)[:, :, :h] for _ in range(3)]
    st["out"] = torch.empty((b, s, h, D), dtype=dtype, device=DEVICE)
    if case["kind"] == "host":
        def pinned(x):
            host = torch.empty(x.shape, dtype=x.dtype, pin_memory=True)
            return host.copy_(x)

        qkv = [pinned(x) for x in qkv]
        st["norm"] = [pinned(x) for x in st["norm"]]
        st["out"] = torch.empty((b, s, h, D), dtype=dtype, pin_memory=True)
    st["q"], st["k"], st["v"] = qkv
    return st


# ------------------------------------------------------------------------------------------------ one pass
def run(st):
    ctx, kind = st["ctx"], st["kind"]
    if kind == "wide":
        ctx.wide_attention(st["q"], st["k"], st["v"], st["out"], st["cfg"])
    elif kind == "joint":
        ctx.joint_attention(st["q"], st["k"], st["v"], *st["norm"], st["cos"], st["sin"], st["out"], st["p"],
                            key_mask=st["mask"])
    elif kind == "block":
        ctx.qkv_projection(st["x"], st["w"][0], st["w"][1], st["w"][2], st["q16"], st["k16"], st["v"], *st["norm"],
                           st["cos"], st["sin"], st["lp_qkv"])
        ctx.run_on_handles(st["q16"], st["k16"], st["v"], st["o"], st["p"])
        ctx.linear(st["o"], st["w"][3], st["out"], st["lp_out"])
    else:  # host: the tables of this forward stay on the device, every call copies q, k, v in and the result out
        ctx.set_device_tables(st["cos"], st["sin"])
        ctx.joint_attention_host(st["q"], st["k"], st["v"], *st["norm"], None, None, st["out"], st["p"])
    return st["out"]


# ------------------------------------------------------------------------------------------------ in 64 bits
def _norm_rope64(x, w_txt, w_img, cos, sin, txt, eps):
    """[batch, tokens, heads, D] in float64: RMS norm per head, weight of the token's segment, pair rotation."""
    x = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)
    x[:, :txt] *= w_txt.double()
    x[:, txt:] *= w_img.double()
    even, odd = x[..., 0::2], x[..., 1::2]
    c, s = cos.double()[None, :, None, :], sin.double()[None, :, None, :]
    out = torch.empty_like(x)
    out[..., 0::2] = even * c[..., 0::2] - odd * s[..., 0::2]
    out[..., 1::2] = odd * c[..., 1::2] + even * s[..., 1::2]
    return out


def _attention64(q, k, v, scale, mask=None):
    """One head: q, k, v [tokens, d] in float64, 2048 query rows at a time."""
    out = torch.empty_like(q)
    for r in range(0, q.shape[0], 2048):
        scores = (q[r:r + 2048] @ k.T) * scale
        if mask is not None:
            scores += mask
        out[r:r + 2048] = torch.softmax(scores, -1) @ v
    return out


def exact(case, seed):
    """What ``run`` gives for these inputs, in float64 with plain torch."""
    st = prepare(case, seed)
    if case["kind"] == "wide":
        return _attention64(st["q"].double(), st["k"].double(), st["v"].double(), case["channels"] ** -0.5)
    p = st["p"]
    b, s, h = p.batch, p.tokens, p.heads
    if case["kind"] == "block":
        x = st["x"].double()
        q, k, v = ((x @ w.double().T).view(b, s, h, D) for w in st["w"][:3])
    else:
        q, k, v = (t.to(DEVICE) for t in (st["q"], st["k"], st["v"]))
    norm = [w.to(DEVICE) for w in st["norm"]]
    mask = None if st["mask"] is None else st["mask"].double()
    out = torch.empty((b, s, h, D), dtype=torch.float64, device=DEVICE)
    for i in range(b):
        for j in range(h):
            one = (slice(i, i + 1), slice(None), slice(j, j + 1))
            qj = _norm_rope64(q[one].double(), norm[0], norm[1], st["cos"], st["sin"], p.txt_tokens, p.norm_eps)
            kj = _norm_rope64(k[one].double(), norm[2], norm[3], st["cos"], st["sin"], p.txt_tokens, p.norm_eps)
            out[i, :, j] = _attention64(qj[0, :, 0], kj[0, :, 0], v[one][0, :, 0].double(), D ** -0.5, mask)
    if case["kind"] == "block":
        return out.view(b * s, h * D) @ st["w"][3].double().T
    return out.cpu() if case["kind"] == "host" else out
