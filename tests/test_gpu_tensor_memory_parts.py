"""hxq_gemm at 5 .. 128 tokens: every warp group owns a quarter of a CTA's K range.  Box counts that do not
divide by four, parts that start inside a block of scales, ragged ends, sidecar entries that meet in
one packed pair; and single-query attention at the edges of its steps, and of spans of one to four times
64 rows."""

import numpy as np
import pytest
import torch

from conftest import rel_l2
from test_gpu_parity import DEV, _make, _t, _weight

pytestmark = pytest.mark.gpu

# bf16 weights and activations (2^-9 each), bf16 result (2^-9): below 3 * 2^-9 in the 2-norm
TOL = 3 * 2.0 ** -9


@pytest.mark.parametrize("n_in,G", [(16, 0), (128, 128), (272, 0), (384, 64), (640, 128), (1168, 0), (1920, 128), (4480, 128)])
@pytest.mark.parametrize("M,n_out", [(5, 129), (17, 1), (64, 300), (65, 128), (128, 257)])
def test_parts_of_k(n_in, G, M, n_out):
    rng = np.random.default_rng(n_in + M)
    cb, idx, pos, vals, b, s, t = _make(rng, n_out, n_in, G, 0.004, np.float32 if M != 64 else np.float16)
    w = _weight(cb, idx, pos, vals, b, s, t, G)
    x = torch.randn(M, n_in, device=DEV, generator=torch.Generator(device=DEV).manual_seed(M)).bfloat16()
    y = w.matmul(x, torch.bfloat16, force="gemm")
    ref = x.double() @ w.dequant().double().t() + _t(b).double()
    assert w.gemm_status() == 0
    assert rel_l2(y.double().cpu().numpy(), ref.cpu().numpy()) < TOL
    assert torch.equal(y, w.matmul(x, torch.bfloat16, force="gemm"))


def test_dense_sidecar_rows():
    """Rows whose every weight is a sidecar entry, next to rows without any: both halves of each packed
    pair, more entries than a lane holds ahead, all lanes of a warp at once."""
    rng = np.random.default_rng(3)
    n_out, n_in = 160, 768
    cb, idx, _, _, b, s, t = _make(rng, n_out, n_in, 128, 0)
    rows = [0, 1, 31, 32, 33, 127, 128, 159]
    pos = np.sort(np.concatenate([r * n_in + np.arange(n_in) for r in rows]).astype(np.int64))
    vals = (0.1 * rng.standard_normal(len(pos))).astype(np.float16).astype(np.float32)
    w = _weight(cb, idx, pos, vals, b, s, t, 128)
    for M in (7, 100):
        x = torch.randn(M, n_in, device=DEV).bfloat16()
        y = w.matmul(x, torch.float32, force="gemm")
        ref = x.double() @ w.dequant().double().t() + _t(b).double()
        # the patched value is W^ rounded to bf16 plus delta, rounded again: two bf16 roundings on W^, not one
        assert rel_l2(y.double().cpu().numpy(), ref.cpu().numpy()) < 4 * 2.0 ** -9


@pytest.mark.parametrize("nq,nkv", [(1, 1), (6, 3), (9, 3), (8, 2), (5, 1), (12, 2), (7, 1), (16, 2)])
@pytest.mark.parametrize("D,max_len,pos", [(128, 64, 0), (128, 700, 63), (64, 700, 64), (8, 257, 256), (120, 2000, 1999)])
@pytest.mark.parametrize("B", [1, 40])
def test_attention_groups_and_edges(nq, nkv, D, max_len, pos, B):
    """Every group size, part-filled steps, head dimensions below 128 (idle lanes), rows past the
    position holding NaN (never read into the result); fp32 arithmetic on bf16 operands, bf16 result."""
    from helix_substrate_b200 import decode_ops
    g = torch.Generator(device=DEV).manual_seed(nq * D + pos)
    q = torch.randn(B, nq * D, device=DEV, generator=g).bfloat16()
    kc, vc = (torch.randn(B, nkv, max_len, D, device=DEV, generator=g).bfloat16() for _ in range(2))
    kc[:, :, pos + 1:] = float("nan")
    vc[:, :, pos + 1:] = float("nan")
    out = torch.empty_like(q)
    decode_ops.attn_decode(q, kc, vc, torch.tensor([pos], device=DEV), out, nq, D ** -0.5)
    k, v = (c[:, :, :pos + 1].double().repeat_interleave(nq // nkv, 1) for c in (kc, vc))
    p = torch.softmax(torch.einsum("bhd,bhtd->bht", q.double().view(B, nq, D), k) * D ** -0.5, -1)
    ref = torch.einsum("bht,bhtd->bhd", p, v).reshape(B, nq * D)
    assert rel_l2(out.double().cpu().numpy(), ref.cpu().numpy()) < 2.0 ** -8


@pytest.mark.parametrize("B,max_len,span", [(30, 4160, 192), (40, 4160, 256), (40, 2500, 128)])
@pytest.mark.parametrize("spans,rows", [(1, 0), (1, 1), (1, 32), (5, 34), (None, 0)])
@pytest.mark.parametrize("rising", [False, True])
def test_attention_spans(B, max_len, span, spans, rows, rising):
    """A block that walks several times 64 rows: its ring is filled again and again, its last span is short or whole,
    partial sums are found by the same span; scores that rise with the row, so that every step rescales what is
    there.  Rows past the position hold NaN."""
    from helix_substrate_b200 import _lib, decode_ops
    nq, nkv, D = 8, 4, 64
    assert _lib.lib().hxq_attn_decode_span(B, nkv, max_len) == span
    pos = max_len - 1 if spans is None else spans * span + rows - 1
    g = torch.Generator(device=DEV).manual_seed(pos)
    q = torch.randn(B, nq * D, device=DEV, generator=g).bfloat16()
    kc, vc = (torch.randn(B, nkv, max_len, D, device=DEV, generator=g).bfloat16() for _ in range(2))
    if rising:      # all heads look along the first dimension: scores from 0 to 16, 1 in a step of 260 rows or fewer
        q.view(B, nq, D)[:, :, 0] = 16.0
        kc[..., 0] = torch.linspace(0, 8, max_len, device=DEV).bfloat16()
    kc[:, :, pos + 1:] = float("nan")
    vc[:, :, pos + 1:] = float("nan")
    out = torch.empty_like(q)
    decode_ops.attn_decode(q, kc, vc, torch.tensor([pos], device=DEV), out, nq, D ** -0.5)
    k, v = (c[:, :, :pos + 1].double().repeat_interleave(nq // nkv, 1) for c in (kc, vc))
    p = torch.softmax(torch.einsum("bhd,bhtd->bht", q.double().view(B, nq, D), k) * D ** -0.5, -1)
    ref = torch.einsum("bht,bhtd->bhd", p, v).reshape(B, nq * D)
    assert rel_l2(out.double().cpu().numpy(), ref.cpu().numpy()) < 2.0 ** -8
