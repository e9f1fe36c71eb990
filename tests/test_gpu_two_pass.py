"""hxq_dequant's vector kernel and hxq_gemm in two passes (bf16 weight rows in scratch, then a dense
product), at the sizes where they can go wrong: against the oracle and the fp64 product."""

import ctypes as C

import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import hxq_oracle as O
from test_gpu_parity import DEV, _make, _t, _weight

pytestmark = pytest.mark.gpu

# bf16 weights and activations (2^-9 each), bf16 result (2^-9): below 3 * 2^-9 in the 2-norm
TOL = 3 * 2.0 ** -9


@pytest.mark.parametrize("n_out,n_in,G", [(1, 16, 16), (7, 16, 0), (65, 48, 48), (3, 16400, 0), (130, 1024, 128), (2, 18944, 128)])
@pytest.mark.parametrize("st", [np.float32, np.float16])
def test_dequant_runs_of_rows(n_out, n_in, G, st):
    """Runs of one row and of many, a last short run, rows of one piece; every output type; a row range
    that starts off a run; bit for bit."""
    rng = np.random.default_rng(n_out * 31 + n_in)
    cb, idx, pos, vals, _, s, t = _make(rng, n_out, n_in, G, 0.01, st, bias=False)
    w = _weight(cb, idx, pos, vals, None, s, t, G)
    ref = torch.from_numpy(O.reconstruct(cb, idx, pos, vals, s, t, G))
    for dt in (torch.float32, torch.bfloat16, torch.float16):
        assert torch.equal(w.dequant(dtype=dt).cpu(), ref.to(dt))
        lo = n_out // 3
        assert torch.equal(w.dequant(lo, n_out, dt).cpu(), ref[lo:].to(dt))
    # rows 16 but not 32 bytes apart: the narrower stores
    wide = torch.full((n_out, n_in + 8), 7.0, dtype=torch.bfloat16, device=DEV)
    w.dequant(dtype=torch.bfloat16, out=wide[:, :n_in])
    assert torch.equal(wide[:, :n_in].cpu(), ref.to(torch.bfloat16)) and bool((wide[:, n_in:] == 7.0).all())


def test_dequant_then_dense_product_on_one_stream():
    """hxq_dequant lets nothing start before it is done: a kernel that fetches its weights ahead (the dense
    product) finds the rows written, and not what the buffer held before."""
    from helix_substrate_b200 import decode_ops
    rng = np.random.default_rng(5)
    n_out, n_in = 18944, 3584
    cb, idx, pos, vals, _, s, t = _make(rng, n_out, n_in, 128, 0.001, bias=False)
    w = _weight(cb, idx, pos, vals, None, s, t, 128)
    x = torch.randn(1, n_in, device=DEV).bfloat16()
    dense = w.dequant(dtype=torch.bfloat16)
    torch.cuda.synchronize()
    want = decode_ops.dense_gemv(dense, x)
    for _ in range(5):
        dense.fill_(7.0)
        w.dequant(dtype=torch.bfloat16, out=dense)
        assert torch.equal(decode_ops.dense_gemv(dense, x), want)


def _check(M, n_out, n_in, G, xdt, ydt, bias=True, x=None, seed=0):
    rng = np.random.default_rng(M * 7 + n_out + n_in + seed)
    cb, idx, pos, vals, b, s, t = _make(rng, n_out, n_in, G, 0.001, bias=bias)
    w = _weight(cb, idx, pos, vals, b, s, t, G)
    if x is None:
        x = torch.randn(M, n_in, device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed)).to(xdt)
    ref = x.double() @ w.dequant().double().t() + (_t(b).double() if bias else 0)
    y = w.matmul(x, ydt)
    assert w.gemm_status() == 0
    assert rel_l2(y.double().cpu().numpy(), ref.cpu().numpy()) < TOL
    assert torch.equal(y, w.matmul(x, ydt)), "bit-identical from run to run"
    return w, x, y, ref


@pytest.mark.parametrize("M,n_out,n_in,G", [
    (1030, 64, 2064, 0),        # a K step mostly past the end, one narrow row tile
    (1025, 250, 592, 0),        # ragged in every direction, output rows not a multiple of a store
    (1200, 513, 1216, 64),      # a last token tile of 176, a last row tile of one row
    (3000, 4619, 1200, 0),      # more than one wave of tiles, odd output width
    (1030, 4100, 18944, 128),   # more rows than one run of scratch takes
    (520, 1000, 3584, 128),     # three token tiles, the last of 8 tokens
])
@pytest.mark.parametrize("xdt,ydt", [(torch.bfloat16, torch.bfloat16), (torch.float16, torch.float32), (torch.float32, torch.float16)])
def test_two_passes_against_fp64(M, n_out, n_in, G, xdt, ydt):
    w, *_ = _check(M, n_out, n_in, G, xdt, ydt)
    from helix_substrate_b200 import _lib
    assert _lib.lib().hxq_gemm_scratch_bytes(C.byref(w.desc), M, 1) > 0


@pytest.mark.parametrize("M,n_out,n_in,G,tile,rows", [
    (1030, 64, 2064, 0, 64, 64),            # less than a tile
    (300, 2573, 272, 0, 96, 2573),          # widths that divide neither the rows nor the accumulator
    (300, 3566, 272, 0, 128, 3566),
    (3000, 4619, 1200, 0, 224, 4619),       # three to four tiles per pair of CTAs: both accumulators, used again
    (2048, 18944, 3584, 128, 256, 9472),    # the widest tile, four per pair, and two runs of rows
])
def test_two_passes_tile_widths(M, n_out, n_in, G, tile, rows):
    """The widths and runs that the rule picks on 148 SMs, with more than one tile per pair where it does."""
    w, *_ = _check(M, n_out, n_in, G, torch.bfloat16, torch.bfloat16)
    from helix_substrate_b200 import _lib
    run = C.c_int32(-1)
    picked = _lib.lib().hxq_gemm_row_tile(C.byref(w.desc), M, C.byref(run))
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert (picked, run.value) == (tile, rows)
    assert _lib.lib().hxq_gemm_row_tile(C.byref(w.desc), 128, None) == 0, "one pass"


def test_out_of_memory_for_the_scratch_runs_in_one_pass(monkeypatch):
    """The caching allocator has no room for the bf16 rows: the call runs in one pass on the kept workspace."""
    from helix_substrate_b200 import _lib
    w, x, y, ref = _check(1024, 384, 1024, 128, torch.bfloat16, torch.bfloat16)
    need = _lib.lib().hxq_gemm_scratch_bytes(C.byref(w.desc), 1024, 1)
    real, refused = torch.empty, []

    def empty(*a, **kw):
        if kw.get("dtype") == torch.uint8 and a == (need,):
            refused.append(need)
            raise torch.OutOfMemoryError("no room")
        return real(*a, **kw)
    monkeypatch.setattr(torch, "empty", empty)
    out = w.matmul(x, torch.bfloat16)
    assert refused == [need] and w.gemm_status() == 0
    assert rel_l2(out.double().cpu().numpy(), ref.cpu().numpy()) < TOL


def test_two_passes_with_strided_activations_and_no_bias():
    """Rows of x inside a wider matrix: 16-byte aligned (read in place) and not (copied)."""
    for pad in (8, 3):
        base = torch.randn(1100, 512 + pad, device=DEV).bfloat16()
        _check(1100, 300, 512, 128, None, torch.bfloat16, bias=False, x=base[:, :512], seed=pad)


def test_two_passes_and_one_pass_agree_at_the_scratch_limit():
    """A workspace one byte short of the two-pass product's runs the one-pass kernel; both are within
    the tolerance of each other."""
    from helix_substrate_b200 import _lib
    w, x, y, ref = _check(1024, 384, 1024, 128, torch.bfloat16, torch.bfloat16)
    L = _lib.lib()
    need = L.hxq_gemm_scratch_bytes(C.byref(w.desc), 1024, 1)
    assert need > 0
    stream = torch.cuda.current_stream().cuda_stream
    for nb in (need, need - 1):
        ws = torch.empty(need, dtype=torch.uint8, device=DEV)
        out = torch.empty_like(y)
        st = L.hxq_gemm(C.byref(w.desc), x.data_ptr(), 2, 1024, x.stride(0), out.data_ptr(), 2, out.stride(0), ws.data_ptr(), nb,
                        None, stream)
        assert st == 0
        assert rel_l2(out.double().cpu().numpy(), ref.cpu().numpy()) < TOL
        if nb == need:
            assert torch.equal(out, y)


def test_two_passes_captured():
    """Inside a capture the scratch comes from the graph's pool; the replay follows new inputs."""
    w, x, y, _ = _check(1024, 384, 1024, 128, torch.bfloat16, torch.bfloat16)
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        w.matmul(x, torch.bfloat16)
        side.synchronize()
        with torch.cuda.graph(graph, stream=side):
            out = w.matmul(x, torch.bfloat16)
    torch.cuda.current_stream().wait_stream(side)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, y)
    x.neg_()
    want = w.matmul(x, torch.bfloat16)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
