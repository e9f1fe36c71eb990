"""hxq_set_weights_on_stream: products of weights that kernels in front of them on the same stream are still
writing, for every kernel that otherwise reads its weights before it waits."""

import ctypes as C

import numpy as np
import pytest
import torch

from test_gpu_parity import DEV, _make, _t, _weight

pytestmark = pytest.mark.gpu


def _rewritten(bufs, values, product):
    """``product`` behind the copies of new ``values`` into ``bufs`` and a kernel that lets its successor start
    early, none of them finished when it is enqueued; and once more with everything complete."""
    from helix_substrate_b200 import _lib, decode_ops
    small = torch.zeros(1, 64, device=DEV, dtype=torch.bfloat16)
    busy = torch.empty(1 << 28, dtype=torch.uint8, device=DEV)
    torch.cuda.synchronize()
    with _lib.weights_on_stream():
        busy.fill_(1)                       # ~80 us in front of the copies
        for b, v in zip(bufs, values):
            b.copy_(v)
        decode_ops.swiglu(small, small, torch.empty_like(small))
        got = product()
    torch.cuda.synchronize()
    return got, product()


@pytest.mark.parametrize("M,xdt", [(1, torch.bfloat16), (16, torch.float32), (5, torch.bfloat16), (40, torch.float16), (128, torch.bfloat16),
                                   (1030, torch.bfloat16)])
def test_products_of_weights_written_on_the_stream(M, xdt):
    from helix_substrate_b200 import _lib
    rng = np.random.default_rng(M)
    n_out, n_in = 2000, 1152
    cb, idx, pos, vals, b, s, t = _make(rng, n_out, n_in, 128, 0.002)
    w = _weight(cb, idx, pos, vals, b, s, t, 128)
    x = torch.randn(M, n_in, device=DEV).to(xdt)
    if M > 128:
        assert _lib.lib().hxq_gemm_scratch_bytes(C.byref(w.desc), M, 1) > 0, "two passes"
    before = w.matmul(x, torch.float32)
    bufs = [w.codebook, w.indices, w.scales, w.offsets, w.deltas, w.bias]
    new = [w.codebook.flip(0) * 1.5, 255 - w.indices, w.scales * 0.5, w.offsets + 0.01, w.deltas * 2, w.bias - 1]
    got, want = _rewritten(bufs, new, lambda: w.matmul(x, torch.float32))
    assert torch.equal(got, want) and not torch.equal(got, before) and w.gemm_status() == 0


@pytest.mark.parametrize("M", [1, 4])
def test_dense_product_of_a_weight_written_on_the_stream(M):
    from helix_substrate_b200 import decode_ops
    weight = torch.randn(5000, 2048, device=DEV).bfloat16()
    x = torch.randn(M, 2048, device=DEV).bfloat16()
    before = decode_ops.dense_gemv(weight, x)
    got, want = _rewritten([weight], [-2 * weight], lambda: decode_ops.dense_gemv(weight, x))
    assert torch.equal(got, want) and not torch.equal(got, before)
