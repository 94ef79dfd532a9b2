"""The work that users of this library have it do, as measurable cases.

Five kinds, each through the library's public entry points:
  layer   moe_cuda_layer: one MoE layer, from one token to the largest batch, added into the fp32 residual
          streams (h) or followed by residual + RMSNorm (y16)
  stack   the teacher-forward stack: upstream projection (moe_cuda_mm) and layer, several times over
  steps   the reference's kernel sequence call by call (what moe_host_moe_rec does)
  mixer   the hyper-connection residual mixer in front of every layer (what moe_mix_res_rec does)
  head    the teacher's head on one chunk of rows: mixer, vocabulary product, distillation sink
Shapes are the configurations of r-mda_b200/synth.py and bench.py; values are drawn like theirs.
"""
import math

import numpy as np
import torch

import __graft_entry__ as entry

_pkg = entry.load_package()
mc = _pkg.moe_cuda

# (d, experts, topk, inter, shared) of the named configurations
FAMILIES = {"tiny": (256, 8, 2, 512, 0), "small": (512, 16, 4, 256, 0), "30B-A3B": (2048, 128, 8, 768, 0),
            "80B-A3B": (2048, 512, 10, 512, 512)}
PAD = 128            # columns of the projection beyond the router logits
HC, RANK, HC_PAD = 4, 320, 384  # residual streams of the teacher, its mixer's rank and padded width
VOCAB = 151936       # bench.py's byte-level vocabulary


def listed():
    a, b = "30B-A3B", "80B-A3B"
    return [
        # one token, the latency of a single decode step
        {"name": "decode-1", "kind": "layer", "family": a, "rows": 1, "skew": 0.0, "hc": 1, "norm": True},
        # small decode batches, one of them ragged
        {"name": "decode-16", "kind": "layer", "family": a, "rows": 16, "skew": 0.0, "hc": 1, "norm": True},
        {"name": "decode-129", "kind": "layer", "family": a, "rows": 129, "skew": 0.0, "hc": 1, "norm": False},
        # a small model's layer: launches and latency
        {"name": "tiny-512", "kind": "layer", "family": "tiny", "rows": 512, "skew": 0.0, "hc": 1, "norm": False},
        # the teacher's own layer on four windows of 384 tokens: shared expert, four residual streams
        {"name": "teacher-1536", "kind": "layer", "family": b, "rows": 1536, "skew": 0.0, "hc": HC, "norm": False},
        # the distillation batch, evenly routed and with popular experts
        {"name": "prefill-4096", "kind": "layer", "family": a, "rows": 4096, "skew": 0.0, "hc": 1, "norm": False},
        {"name": "skewed-4096", "kind": "layer", "family": a, "rows": 4096, "skew": 1.0, "hc": 1, "norm": False},
        # the largest batch of the largest layer
        {"name": "large-16384", "kind": "layer", "family": b, "rows": 16384, "skew": 0.0, "hc": 1, "norm": False},
        # projection and layer of consecutive layers on a medium batch
        {"name": "stack-2048", "kind": "stack", "family": a, "rows": 2048, "layers": 3},
        # a host that keeps the reference's sequence of calls, odd row count
        {"name": "steps-1003", "kind": "steps", "family": a, "rows": 1003},
        # the mixer between two layers, odd row count
        {"name": "mixer-3001", "kind": "mixer", "rows": 3001},
        # one window's rows through the head and the distillation sink
        {"name": "head-384", "kind": "head", "rows": 384, "vocab": VOCAB},
    ]


def _spread(rng, lo, hi):
    """A whole number from lo to hi, evenly over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["layer"] * 6 + ["stack", "steps", "mixer", "head"])
    if kind == "layer":
        family = rng.choice(["tiny", "small", "30B-A3B", "30B-A3B", "80B-A3B"])
        top = {"80B-A3B": 16384, "30B-A3B": 12288}.get(family, 16384)
        norm = rng.random() < 0.4
        return {"kind": kind, "family": family, "rows": _spread(rng, 1, top), "skew": rng.choice([0.0, 0.0, 0.55, 1.0]),
                "hc": 1 if norm else rng.choice([1, HC]), "norm": norm}
    if kind == "stack":
        return {"kind": kind, "family": rng.choice(["small", "30B-A3B"]), "rows": 128 * _spread(rng, 1, 32),
                "layers": rng.randint(2, 3)}
    if kind == "steps":
        return {"kind": kind, "family": rng.choice(["tiny", "small", "30B-A3B"]), "rows": _spread(rng, 16, 4096)}
    if kind == "mixer":
        return {"kind": kind, "rows": _spread(rng, 1, 12288)}
    return {"kind": kind, "rows": _spread(rng, 8, 1536), "vocab": 128 * _spread(rng, 24, VOCAB // 128)}


# ---- what a user's program has in hand ---------------------------------------------------------
_streams = {}


def _ctx():
    """A program's context: every state stands for a program of its own, all of them on one stream."""
    dev = torch.cuda.current_device()
    if dev not in _streams:
        _streams[dev] = torch.cuda.Stream()
    ctx = mc.Ctx(dev, _streams[dev].cuda_stream)
    ctx.check()
    return ctx


class _State(dict):
    def __del__(self):
        if "ctx" in self:
            self["ctx"].close()


class _Make:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.seed = int(seed)
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(self.seed)

    def f32(self, *shape, std=1.0):
        return torch.randn(shape, device="cuda", generator=self.gen) * std

    def f16(self, *shape, std=1.0):
        # in pieces, so that the fp32 draw of a large tensor is never whole
        out = torch.empty(shape, device="cuda", dtype=torch.float16)
        flat = out.view(-1)
        for lo in range(0, flat.numel(), 1 << 27):
            n = min(1 << 27, flat.numel() - lo)
            flat[lo:lo + n] = torch.randn(n, device="cuda", generator=self.gen) * std
        return out

    def bias(self, experts, beta):
        """Router bias of popular experts: beta * log of Zipf(1.2) weights in a random order."""
        rank = torch.randperm(experts, device="cuda", generator=self.gen).float() + 1.0
        return beta * torch.log_softmax(-1.2 * torch.log(rank), 0)


def _empty(*shape, dtype=torch.float32):
    return torch.empty(shape, device="cuda", dtype=dtype)


def _u32(*shape):
    return torch.zeros(shape, device="cuda", dtype=torch.int32)


def _layer(case, mk):
    d, e, k, i, s = FAMILIES[case["family"]]
    t, hc = case["rows"], case["hc"]
    keep = {"x16": mk.f16(t, d), "proj": mk.f32(t, e + PAD, std=0.9), "wgu": mk.f16(e, 2 * i, d, std=0.02),
            "wdown": mk.f16(e, d, i, std=0.02)}
    keep["proj"][:, :e] += mk.bias(e, case["skew"])
    if s:
        keep.update(wsgu=mk.f16(2 * s, d, std=0.02), wsdown=mk.f16(d, s, std=0.02))
    call = {}
    if hc > 1:
        keep["inj"] = mk.f32(t, HC_PAD)
        call.update(inj_stride=HC_PAD, inj_off=RANK)
    if case["norm"]:
        out = keep["y16"] = _empty(t, d, dtype=torch.float16)
        call["eps"] = 1e-6
    else:
        out = keep["h"] = mk.f32(t, hc, d)
    call.update({n: v.data_ptr() for n, v in keep.items()})
    call.update(rows=t, d=d, experts=e, topk=k, inter=i, shared=s, pstride=e + PAD, hc=hc)
    return {"call": call, "keep": keep, "out": out}


def _columns(experts):
    """Columns of the projection as a product: the dense kernels take multiples of 128."""
    return (experts + PAD + 127) // 128 * 128


def _stack(case, mk):
    d, e, k, i, _ = FAMILIES[case["family"]]
    t, cols = case["rows"], _columns(e)
    x, ya, yb = mk.f16(t, d), _empty(t, d, dtype=torch.float16), _empty(t, d, dtype=torch.float16)
    proj, tiles, keep, calls, src, dst = _empty(t, cols), _u32(t // 128), [], [], x, ya
    for _ in range(case["layers"]):
        wgu, wdown, wd = mk.f16(e, 2 * i, d, std=0.02), mk.f16(e, d, i, std=0.02), mk.f16(cols, d, std=0.02)
        wd[e + 1:] = 0
        keep.append((wgu, wdown, wd))
        calls.append(((src.data_ptr(), wd.data_ptr(), proj.data_ptr(), None, tiles.data_ptr(), t, cols, d),
                      dict(rows=t, d=d, experts=e, topk=k, inter=i, shared=0, pstride=cols, hc=1, proj=proj.data_ptr(),
                           x16=src.data_ptr(), wgu=wgu.data_ptr(), wdown=wdown.data_ptr(), y16=dst.data_ptr(), eps=1e-6)))
        src, dst = dst, yb if dst is ya else ya
    return {"calls": calls, "keep": (keep, x, ya, yb, proj, tiles), "out": src}


def _steps(case, mk):
    d, e, k, i, _ = FAMILIES[case["family"]]
    t = case["rows"]
    m = mc.moe_rows(t, k, e)
    b = {"proj": mk.f32(t, e + PAD, std=0.9), "x16": mk.f16(t, d), "wgu": mk.f16(e, 2 * i, d, std=0.02),
         "wdown": mk.f16(e, d, i, std=0.02), "h": mk.f32(t, d), "idx": _u32(t, k), "wt": _empty(t, k), "slot": _u32(t, k),
         "count": _u32(e), "off": _u32(e), "fill": _u32(e), "tiles": _u32(m // 128), "xp": _empty(m, d, dtype=torch.float16),
         "g": _empty(m, 2 * i), "hp": _empty(m, i), "hp16": _empty(m, i, dtype=torch.float16), "ye": _empty(m, d), "amax": _u32(256)}
    return {"b": b, "p": {n: v.data_ptr() for n, v in b.items()}, "size": (t, d, e, k, i, m)}


def _mixer(case, mk, vocab=0):
    d, rows = 2048, case["rows"]
    d4 = HC * d
    b = {"h": mk.f32(rows, d4), "norm": mk.f32(d4, std=0.1), "down": mk.f16(HC_PAD, d4, std=0.02), "up": mk.f16(d4, RANK, std=0.05),
         "hn": _empty(rows, d4), "a16": _empty(rows, d4, dtype=torch.float16), "t": _empty(rows, HC_PAD), "u": _empty(rows, RANK),
         "upo": _empty(rows, d4), "x": _empty(rows, d), "amax": _u32(256)}
    b["down"][RANK + HC:] = 0
    if vocab:
        b.update(_vocabulary(mk, rows, vocab), lm=mk.f16(vocab, d, std=0.1), logits=_empty(rows, vocab), outp=_u32(rows, 16, 8))
    return {"b": b, "p": {n: v.data_ptr() for n, v in b.items()}, "size": (rows, d, d4, vocab),
            "bytes": b["outp"].view(torch.int16)[..., 0::2] if vocab else None, "p16": b["outp"].view(torch.float16)[..., 1::2] if vocab else None}


def _vocabulary(mk, rows, vocab):
    """A byte-level vocabulary as sub-word tokenizers have it -- strings of 1 to 16 bytes, many of them words behind a
    space, some multi-byte characters, a few entries without a byte string -- and continuations spelled from its tokens."""
    rng = np.random.default_rng(mk.seed)
    letter = 1.0 / np.arange(1, 27)
    tb = (97 + rng.choice(26, (vocab, 16), p=letter / letter.sum())).astype(np.uint8)
    length = np.minimum(1 + rng.poisson(4.5, vocab), 16)
    kind = rng.random(vocab)
    tb[kind < 0.4, 0] = 32
    cjk = kind > 0.8
    tb[cjk, 0::3] = rng.integers(0xe4, 0xea, (int(cjk.sum()), 6))
    tb[cjk, 1::3] = rng.integers(0x80, 0xc0, (int(cjk.sum()), 5))
    tb[cjk, 2::3] = rng.integers(0x80, 0xc0, (int(cjk.sum()), 5))
    length[kind < 0.0005] = 0
    tb[np.arange(16)[None, :] >= length[:, None]] = 0
    toks = np.concatenate([tb.view(np.uint32).reshape(vocab, 4), length[:, None].astype(np.uint32)], 1)
    cont = np.zeros((rows, 5), np.uint32)
    for r in range(rows):
        s = b"".join(tb[t, :length[t]].tobytes() for t in rng.integers(0, vocab, 17))[:16]
        cont[r, :4] = np.frombuffer(s.ljust(16, b"\0"), np.uint32)
        cont[r, 4] = len(s)
    return {n: torch.from_numpy(np.ascontiguousarray(v).view(np.int32)).cuda() for n, v in (("toks", toks), ("cont", cont))}


def prepare(case, seed):
    mk = _Make(seed)
    kind = case["kind"]
    if kind == "layer":
        s = _layer(case, mk)
    elif kind == "stack":
        s = _stack(case, mk)
    elif kind == "steps":
        s = _steps(case, mk)
    else:
        s = _mixer(case, mk, case.get("vocab", 0))
    torch.cuda.synchronize()   # the tensors were made on another stream than the context's
    return _State(s, kind=kind, ctx=_ctx())


# ---- one pass ----------------------------------------------------------------------------------
def _cast(ctx, p, src, n, slot):
    ctx.absmax(p[src], p["amax"], n, slot)
    ctx.cast_f16(p[src], p["a16"], p["amax"], n, slot)


def _mix(s):
    ctx, p = s["ctx"], s["p"]
    rows, d, d4, _ = s["size"]
    mc.lib().moe_cuda_fill(ctx.p, p["amax"], 1024, 0)
    ctx.norm(p["h"], p["norm"], p["hn"], rows, HC, d, op=0, eps=1e-6)
    _cast(ctx, p, "hn", rows * d4, 0)
    ctx.dense(p["a16"], p["down"], p["t"], p["amax"], rows, HC_PAD, d4, sa=0)
    ctx.swiglu(p["t"], p["u"], rows, RANK, HC_PAD, 0, 0, op=1, scale=1.0 / HC)
    _cast(ctx, p, "u", rows * RANK, 1)
    ctx.dense(p["a16"], p["up"], p["upo"], p["amax"], rows, d4, RANK, sa=1)
    ctx.hc(p["upo"], p["hn"], p["x"], rows, d, HC, 0, HC_PAD, RANK)


def _steps_run(s):
    ctx, p = s["ctx"], s["p"]
    t, d, e, k, i, m = s["size"]
    fill = mc.lib().moe_cuda_fill
    fill(ctx.p, p["amax"], 1024, 0)
    fill(ctx.p, p["count"], e * 4, 0)
    fill(ctx.p, p["fill"], e * 4, 0)
    fill(ctx.p, p["tiles"], m // 128 * 4, 0xffffffff)
    fill(ctx.p, p["xp"], m * d * 2, 0)
    ctx.route(p["proj"], p["idx"], p["wt"], p["count"], t, e, k, e + PAD)
    ctx.scan(p["count"], p["off"], p["tiles"], e)
    ctx.scatter(p["idx"], p["off"], p["fill"], p["x16"], p["xp"], p["slot"], t, k, d // 8)
    fill(ctx.p, p["g"], m * 2 * i * 4, 0)
    ctx.mm(p["xp"], p["wgu"], p["g"], p["amax"], p["tiles"], m, 2 * i, d, experts_in_B=e)
    ctx.swiglu(p["g"], p["hp"], m, i, 2 * i, 0, i)
    ctx.absmax(p["hp"], p["amax"], m * i, 0)
    ctx.cast_f16(p["hp"], p["hp16"], p["amax"], m * i, 0)
    ctx.mm(p["hp16"], p["wdown"], p["ye"], p["amax"], p["tiles"], m, d, i, sa=0, experts_in_B=e)
    ctx.combine(p["wt"], p["slot"], p["ye"], p["proj"], None, None, p["h"], t, d, k, e + PAD, e)


def _pass(state):
    kind = state["kind"]
    ctx = state["ctx"]
    if kind == "layer":
        ctx.layer(**state["call"])
        return state["out"]
    if kind == "stack":
        for mm, layer in state["calls"]:
            ctx.mm(*mm, experts_in_B=1)
            ctx.layer(**layer)
        return state["out"]
    b = state["b"]
    if kind == "steps":
        _steps_run(state)
        return {n: b[n] for n in ("h", "idx", "wt", "slot", "count", "off")}
    _mix(state)
    if kind == "mixer":
        return {"x": b["x"], "t": b["t"]}
    p = state["p"]
    rows, d, _, vocab = state["size"]
    _cast(ctx, p, "x", rows * d, 2)
    ctx.dense(p["a16"], p["lm"], p["logits"], p["amax"], rows, vocab, d, sa=2)
    ctx.kd_bytes(p["logits"], p["toks"], p["cont"], p["outp"], rows, vocab)
    return {"logits": b["logits"], "bytes": state["bytes"], "p": state["p16"]}


def run(state):
    out = _pass(state)
    state["ctx"].check()   # a refused call shows here; nothing is waited for
    return out


# ---- what a pass cannot do without -------------------------------------------------------------
def _live(t, e, k, beta):
    """Experts that a batch of t tokens reaches on average."""
    if beta == 0.0:
        return e * (1.0 - (1.0 - k / e) ** t)
    rng = np.random.default_rng(0)
    bias = -1.2 * beta * np.log(np.arange(1, e + 1))
    top = np.argpartition(-(rng.standard_normal((4096, e)) * 0.9 + bias), k - 1, axis=1)[:, :k]
    return float((1.0 - (1.0 - np.bincount(top.ravel(), minlength=e) / 4096.0) ** t).sum())


def _layer_work(t, d, e, k, i, s, hc, norm, beta=0.0):
    live = _live(t, e, k, beta)
    res = 2 * t * d if norm else 8 * t * hc * d + (4 * t * hc if hc > 1 else 0)
    return {"bytes": live * 6 * i * d + 6 * s * d + 2 * t * d + 4 * t * e + res, "flops": 6.0 * t * d * (k * i + s)}


def work(case):
    kind = case["kind"]
    if kind in ("layer", "stack"):
        d, e, k, i, s = FAMILIES[case["family"]]
        w = _layer_work(case["rows"], d, e, k, i, s, case.get("hc", 1), case.get("norm", True), case.get("skew", 0.0))
        if kind == "layer":
            return w
        t, n, cols = case["rows"], case["layers"], _columns(e)
        return {"bytes": n * (w["bytes"] + 2 * cols * d + 2 * t * d + 4 * t * cols), "flops": n * (w["flops"] + 2.0 * t * cols * d)}
    if kind == "steps":
        # every call's own arguments: the caller holds xp, g, hp, hp16 and ye
        d, e, k, i, _ = FAMILIES[case["family"]]
        t = case["rows"]
        w, tk = _layer_work(t, d, e, k, i, 0, 1, False), t * k
        m = tk + e * 127
        return {"bytes": w["bytes"] + m * (2 * d + 8 * i + 22 * i) + tk * (2 * d + 2 * d + 8 * i + 2 * i + 4 * d + 4 * d), "flops": w["flops"]}
    rows, d = case["rows"], 2048
    d4, v = HC * d, case.get("vocab", 0)
    # norm, cast, down, gate, cast, up, read-out: arguments of each call, the reductions for the scale slots included
    b = rows * d4 * (4 + 4 + 4 + 4 + 2 + 2 + 4 + 8) + rows * (HC_PAD * 8 + RANK * 16 + d * 4) + 2 * d4 * (HC_PAD + RANK) + 4 * d4
    f = 2.0 * rows * d4 * (HC_PAD + RANK)
    if v:
        b += rows * d * 12 + 2 * v * d + rows * v * 8 + v * 20 + rows * 532
        f += 2.0 * rows * v * d
    return {"bytes": b, "flops": f}


def tolerance(case):
    # fp16 operands, intermediates and expert rows with fp32 sums: half a unit in the last place of fp16 (2^-11)
    # once or twice on the way.  Whole numbers are equal; in the sink's output two bytes of equal mass may swap.
    if case["kind"] == "head":
        return {"rel": 1e-3, "max": 0.02, "differ": 0.004}
    return {"rel": 1e-3, "max": 0.02}
