"""The work a user of this package has it do, as timed cases.

Compressed linears called one at a time the way a model's code calls them, the MLP of a decoder at
the token counts of interactive and of small-batch decoding, the projections of a decoder at batch
and at prompt sizes, the operator-level product on fp32 activations, dense weights back from
compressed ones, whole decode steps of a decoder, and the encoder that makes the weights.

Sizes are the Qwen2.5-7B / 14B projection shapes of the benchmark, their tensor-parallel shards, and
generic odd ones.  Weights are Student-t(5) at std 0.02 with a 256-entry codebook, most of them with
a group-128 scale / offset and the 0.1 % sidecar; activations are N(0, 1).
"""

from __future__ import annotations

import math

import torch

from helix_substrate_b200 import HelixLinear
from helix_substrate_b200.hxq_writer_gpu import assign_indices, compress_weight, student_t_weight
from helix_substrate_b200.qwen2_decode import Qwen2HxqDecoder, Qwen2Shape
from helix_substrate_b200.triton_affine_group_matmul import fused_affine_group_matmul

DEV = torch.device("cuda", 0)
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
GROUP = 128
SIDECAR = 0.001          # share of the weights kept exactly
VOCAB = 10864            # two layers' share of the 152064 rows a 28-layer decoder's head has
DECODE_LAYERS = 2
DECODE_MAX_LEN = 4160    # rows of the static cache


def listed():
    return [
        # the smallest product a decoder makes: a key / value projection of one token, called as a module
        dict(name="linear_kv_1", kind="linear", n_out=512, n_in=3584, tokens=1, x="bf16", group=GROUP, bias=True),
        # an odd linear in fp16 without a group affine: no size is a multiple of a tile
        dict(name="linear_odd_77", kind="linear", n_out=4619, n_in=1200, tokens=77, x="f16", group=0, bias=True),
        # gate, up and down of one layer, captured once and replayed for every token: one sequence ...
        dict(name="mlp_1", kind="mlp", hidden=3584, inter=18944, tokens=1, x="bf16"),
        # ... and four
        dict(name="mlp_4", kind="mlp", hidden=3584, inter=18944, tokens=4, x="bf16"),
        # the operator under the module, called with fp32 activations and fp16 scales (tight tolerance)
        dict(name="operator_f32_8", kind="operator", n_out=3584, n_in=3584, tokens=8, x="f32", st="f16"),
        # the four joint projections of a 14B layer at the batch of a busy server
        dict(name="projections_14b_64", kind="projections", hidden=5120, inter=13824, q=5120, kv=1024, joint=True, tokens=64, x="bf16"),
        # prompts: the seven projections of a 7B layer, one short prompt and a packed batch of long ones
        dict(name="projections_7b_512", kind="projections", hidden=3584, inter=18944, q=3584, kv=512, joint=False, tokens=512, x="bf16"),
        dict(name="projections_7b_8192", kind="projections", hidden=3584, inter=18944, q=3584, kv=512, joint=False, tokens=8192, x="bf16"),
        # the dense weight of a layer, for the buffered mode and for export
        dict(name="dense_gate", kind="dense", n_out=18944, n_in=3584, out="bf16", group=GROUP),
        # one token of a decoder behind a 2048-token context: one sequence, and a batch
        dict(name="decode_1", kind="decode", batch=1, context=2048),
        dict(name="decode_32", kind="decode", batch=32, context=2048),
        # compressing one attention projection of a checkpoint
        dict(name="encode_q", kind="encode", n_out=3584, n_in=3584),
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _log16(rng, lo, hi):
    return _log(rng, lo // 16, hi // 16) * 16


def draw(rng):
    kind = rng.choice(["linear", "linear", "mlp", "operator", "projections", "projections", "dense", "decode", "encode"])
    if kind == "linear":
        n_in = _log16(rng, 256, 19200)
        group = GROUP if n_in % GROUP == 0 or rng.random() < 0.5 else 0
        if group:
            n_in = max(GROUP, n_in // GROUP * GROUP)
        return dict(kind=kind, n_out=_log(rng, 128, 19200), n_in=n_in, tokens=_log(rng, 1, 1024),
                    x=rng.choice(["bf16", "bf16", "f16", "f32"]), group=group, bias=rng.random() < 0.5)
    if kind == "mlp":
        return dict(kind=kind, hidden=_log(rng, 16, 40) * GROUP, inter=_log(rng, 18, 148) * GROUP, tokens=_log(rng, 1, 16),
                    x=rng.choice(["bf16", "bf16", "f16"]))
    if kind == "operator":
        return dict(kind=kind, n_out=_log(rng, 256, 18944), n_in=_log(rng, 8, 148) * GROUP, tokens=_log(rng, 1, 16), x="f32",
                    st=rng.choice(["f16", "f32"]))
    if kind == "projections":
        kv = rng.choice([256, 512, 1024])
        hidden = rng.randint(16, 28) * GROUP
        return dict(kind=kind, hidden=hidden, inter=rng.randint(36, 148) * GROUP, q=hidden, kv=kv, joint=rng.random() < 0.5,
                    tokens=_log(rng, 5, 8192), x=rng.choice(["bf16", "bf16", "f16"]))
    if kind == "dense":
        return dict(kind=kind, n_out=_log(rng, 128, 18944), n_in=_log(rng, 2, 28) * GROUP, out=rng.choice(["bf16", "f16", "f32"]),
                    group=rng.choice([0, GROUP]))
    if kind == "decode":
        return dict(kind=kind, batch=_log(rng, 1, 64), context=_log(rng, 100, 4096))
    return dict(kind="encode", n_out=_log(rng, 128, 3584), n_in=_log(rng, 4, 28) * GROUP)


# ---- what a program has in hand before the call ---------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _compressed(n_out, n_in, group, seed, sidecar=True, st=torch.float32):
    """Constructor arguments of HelixLinear for a Student-t weight: quantile codebook, nearest codes,
    a group affine close to the identity, the largest 0.1 % kept."""
    w = student_t_weight((n_out, n_in), seed, DEV)
    g = _gen(seed + 1)
    flat = w.view(-1)
    sample = flat[torch.randint(0, flat.numel(), (1 << 18,), device=DEV, generator=g)].sort().values
    at = torch.linspace(0.5 / 256, 1 - 0.5 / 256, 256, device=DEV) * (sample.numel() - 1)
    cb = torch.unique(sample[at.long()])
    cb = torch.cat([cb, cb[-1:].expand(256 - cb.numel())]).contiguous()
    enc = dict(codebook=cb, indices=assign_indices(flat, cb).view(n_out, n_in))
    if sidecar:
        lim = sample.abs().sort().values[int((1 - SIDECAR) * sample.numel())]
        pos = torch.nonzero(flat.abs() > lim).reshape(-1)
        enc.update(sidecar_positions=pos, sidecar_values=flat[pos].half().float())
    if group:
        enc["group_scales"] = (1 + 0.05 * torch.randn(n_out, n_in // group, device=DEV, generator=g)).to(st)
        enc["group_offsets"] = (5e-4 * torch.randn(n_out, n_in // group, device=DEV, generator=g)).to(st)
        enc["group_size"] = group
    return enc


def _linear(n_out, n_in, group, seed, bias=False):
    b = 0.02 * torch.randn(n_out, device=DEV, generator=_gen(seed + 2)) if bias else None
    return HelixLinear(n_in, n_out, bias=b, **_compressed(n_out, n_in, group, seed))


def _x(tokens, n_in, dtype, seed):
    return torch.randn(tokens, n_in, device=DEV, generator=_gen(seed)).to(DTYPES[dtype])


def _captured(fn):
    """``fn``'s launches as a CUDA graph, warmed up on the stream they are captured on."""
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side), torch.no_grad():
        for _ in range(2):
            fn()
        side.synchronize()
        with torch.cuda.graph(graph, stream=side):
            out = fn()
    torch.cuda.current_stream().wait_stream(side)
    return graph, out


def _projection_shapes(case):
    h, i, q, kv = case["hidden"], case["inter"], case["q"], case["kv"]
    if case["joint"]:
        return [("qkv", q + 2 * kv, h, True), ("o", h, q, False), ("gate_up", 2 * i, h, False), ("down", h, i, False)]
    return [("q", q, h, True), ("k", kv, h, True), ("v", kv, h, True), ("o", h, q, False), ("gate", i, h, False),
            ("up", i, h, False), ("down", h, i, False)]


_decoder = None


def _the_decoder():
    """The decoder all decode cases step: loaded once per process, as a server loads it."""
    global _decoder
    if _decoder is None:
        shp = Qwen2Shape(layers=DECODE_LAYERS, vocab=VOCAB)
        _decoder = Qwen2HxqDecoder(shp, DEV, 1, DECODE_MAX_LEN)
    return _decoder


def _prepare_decode(case, seed):
    """Static caches holding ``context`` rows and the one-token step captured over them."""
    model = _the_decoder()
    shp, B, T = model.shp, case["batch"], case["context"]
    g = _gen(seed)
    shape = (shp.layers, B, shp.kv_heads, DECODE_MAX_LEN, shp.head_dim)
    caches = []
    for _ in range(2):
        c = torch.zeros(shape, device=DEV, dtype=torch.bfloat16)
        for li in range(shp.layers):
            c[li, :, :, :T] = 0.5 * torch.randn(B, shp.kv_heads, T, shp.head_dim, device=DEV, generator=g)
        caches.append(c)
    tok = torch.randint(0, shp.vocab, (B, 1), device=DEV, generator=g)
    pos = torch.full((1,), T, device=DEV, dtype=torch.long)
    model.k_cache, model.v_cache = caches
    graph, logits = _captured(lambda: model.step_fused(tok, pos))
    new_rows = [c[:, :, :, T] for c in caches]      # the rows the step appends
    return dict(kind="decode", graph=graph, keep=(caches, tok, pos, model._sb), out=[logits, *new_rows])


def prepare(case, seed):
    kind, seed = case["kind"], 1000 * seed
    if kind == "linear":
        return dict(kind=kind, mods=[_linear(case["n_out"], case["n_in"], case["group"], seed, case["bias"])],
                    xs=[_x(case["tokens"], case["n_in"], case["x"], seed + 9)])
    if kind == "projections":
        xs = {n: _x(case["tokens"], n, case["x"], seed + n) for n in {case["hidden"], case["q"], case["inter"]}}
        shapes = _projection_shapes(case)
        return dict(kind=kind, mods=[_linear(o, i, GROUP, seed + 10 * k, b) for k, (_, o, i, b) in enumerate(shapes)],
                    xs=[xs[i] for _, _, i, _ in shapes])
    if kind == "mlp":
        h, i = case["hidden"], case["inter"]
        mods = [_linear(i, h, GROUP, seed), _linear(i, h, GROUP, seed + 10), _linear(h, i, GROUP, seed + 20)]
        x, act = _x(case["tokens"], h, case["x"], seed + 30), _x(case["tokens"], i, case["x"], seed + 31)
        graph, out = _captured(lambda: [mods[0](x), mods[1](x), mods[2](act)])
        return dict(kind=kind, graph=graph, keep=(mods, x, act), out=out)
    if kind == "operator":
        enc = _compressed(case["n_out"], case["n_in"], GROUP, seed, sidecar=False)
        # the codes are the values 0..255: a step of 1/1500 and an offset that centres them at std ~0.02
        sc = (enc["group_scales"] * 8e-4).to(DTYPES[case["st"]])
        return dict(kind=kind, x=_x(case["tokens"], case["n_in"], case["x"], seed + 9), indices=enc["indices"], scales=sc,
                    offsets=(-127.5 * sc.float() + enc["group_offsets"]).to(sc.dtype))
    if kind == "dense":
        return dict(kind=kind, mod=_linear(case["n_out"], case["n_in"], case["group"], seed).packed(), dtype=DTYPES[case["out"]])
    if kind == "decode":
        return _prepare_decode(case, seed)
    return dict(kind=kind, w=student_t_weight((case["n_out"], case["n_in"]), seed, DEV))


# ---- one pass -------------------------------------------------------------------------------------

@torch.no_grad()
def run(state):
    kind = state["kind"]
    if kind in ("linear", "projections"):
        return [mod(x) for mod, x in zip(state["mods"], state["xs"])]
    if kind in ("mlp", "decode"):
        state["graph"].replay()
        return state["out"]
    if kind == "operator":
        return fused_affine_group_matmul(state["x"], state["indices"], state["scales"], state["offsets"], group_size=GROUP)
    if kind == "dense":
        return state["mod"].dequant(dtype=state["dtype"])
    return {k: v for k, v in compress_weight(state["w"], group_size=GROUP).items() if k != "group_size"}


# ---- what a pass cannot do without ----------------------------------------------------------------

def _matrix_bytes(n_out, n_in, group, sidecar=True, st_bytes=4):
    b = n_out * n_in + 1024
    if group:
        b += 2 * st_bytes * n_out * (n_in // group)
    if sidecar:
        b += int(SIDECAR * n_out * n_in) * 8 + (n_out + 1) * 4
    return b


def _product(n_out, n_in, tokens, group, x_bytes, y_bytes, sidecar=True, st_bytes=4, bias=False):
    return (_matrix_bytes(n_out, n_in, group, sidecar, st_bytes) + tokens * (n_in * x_bytes + n_out * y_bytes) + (4 * n_out if bias else 0),
            2 * tokens * n_out * n_in)


def _size(name):
    return 4 if name == "f32" else 2


def work(case):
    kind = case["kind"]
    if kind == "linear":
        parts = [_product(case["n_out"], case["n_in"], case["tokens"], case["group"], _size(case["x"]), _size(case["x"]), bias=case["bias"])]
    elif kind == "projections":
        parts = [_product(o, i, case["tokens"], GROUP, 2, 2, bias=b) for _, o, i, b in _projection_shapes(case)]
    elif kind == "mlp":
        h, i = case["hidden"], case["inter"]
        parts = [_product(o, k, case["tokens"], GROUP, 2, 2) for o, k in ((i, h), (i, h), (h, i))]
    elif kind == "operator":
        parts = [_product(case["n_out"], case["n_in"], case["tokens"], GROUP, 4, 4, sidecar=False, st_bytes=_size(case["st"]))]
    elif kind == "dense":
        parts = [(_matrix_bytes(case["n_out"], case["n_in"], case["group"]) + case["n_out"] * case["n_in"] * _size(case["out"]),
                  case["n_out"] * case["n_in"])]
    elif kind == "decode":
        s, B = Qwen2Shape(), case["batch"]
        layer = [_product(o, i, B, GROUP, 2, 2, bias=b) for _, o, i, b in
                 _projection_shapes(dict(hidden=s.hidden, inter=s.inter, q=s.heads * s.head_dim, kv=s.kv_heads * s.head_dim, joint=True))]
        layer.append((2 * B * s.kv_heads * (case["context"] + 1) * s.head_dim * 2, 4 * B * s.heads * s.head_dim * (case["context"] + 1)))
        head = (VOCAB * s.hidden * 2 + B * (s.hidden * 2 * 2 + VOCAB * 2), 2 * B * VOCAB * s.hidden)
        parts = layer * DECODE_LAYERS + [head]
    else:
        n = case["n_out"] * case["n_in"]
        parts = [(4 * n + _matrix_bytes(case["n_out"], case["n_in"], GROUP), 10 * n)]
    return dict(bytes=sum(b for b, _ in parts), flops=sum(f for _, f in parts))


def tolerance(case):
    kind = case["kind"]
    if kind == "operator":
        return dict(rel=1e-5, max=1e-4)               # fp32 weights, activations and sums
    if kind == "dense":
        return "exact"                                # one stated rounding per weight
    if kind == "encode":
        # fp32 centroid sums in any order: a code next to a midpoint falls to either side, and the (small) offset of its
        # group moves with it; two runs on the same weights differ by rel 0.0045, max 0.23 and 0.008 % of the codes
        return dict(rel=2e-2, max=0.9, differ=4e-4)
    if kind == "decode":
        return dict(rel=2e-2, max=0.2)                # two layers of bf16 activations
    return dict(rel=1e-2, max=0.1)                    # bf16 operands or bf16 / fp16 results
