"""The encoder's kernels against the same steps in torch ops on the CPU (the encoder's path for CPU
tensors) and against numpy."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _special(n, seed):
    """Ties, signed zeros, infinities and a NaN among normal values."""
    g = torch.Generator().manual_seed(seed)
    v = torch.randn(n, generator=g)
    v[torch.randint(0, n, (n // 3,), generator=g)] = 0.25
    for i, x in enumerate((0.0, -0.0, float("inf"), float("-inf"), 1e-42)):
        v[(7 * i + 3) % n] = x
    return v


@pytest.mark.parametrize("n,offset", [(1, 0), (2, 0), (5, 1), (1023, 0), (1025, 3), (300_001, 0)])
def test_two_order_statistics(n, offset):
    """Every rank pair at the ends and inside, from an address that is not 16-byte aligned too."""
    from helix_substrate_b200 import _lib
    L = _lib.lib()
    v = _special(n, n) if n > 40 else torch.randn(n)
    order = np.sort(v.numpy())
    d = torch.empty(n + offset, device=DEV)[offset:].copy_(v)
    ws = torch.empty(L.hxq_encode_select_workspace_bytes(), dtype=torch.uint8, device=DEV)
    out = torch.empty(2, device=DEV)
    for a, b in {(0, n - 1), (n // 2, n // 3), (n - 1, 0), (n // 7, n // 7)}:
        assert L.hxq_encode_select2(d.data_ptr(), n, a, b, out.data_ptr(), ws.data_ptr(), ws.numel(),
                                    torch.cuda.current_stream().cuda_stream) == 0
        assert np.array_equal(out.cpu().numpy(), order[[a, b]])
    assert L.hxq_encode_select2(d.data_ptr(), n, n, 0, out.data_ptr(), ws.data_ptr(), ws.numel(), None) == _lib.HXQ_E_SHAPE


@pytest.mark.parametrize("shape,pct", [((1, 7), 90.0), ((33, 31), 99.0), ((128, 1024), 99.95), ((300, 1000), 50.0)])
def test_outliers_match_the_torch_path(shape, pct):
    from helix_substrate_b200.hxq_writer_gpu import find_outliers_percentile
    w = _special(shape[0] * shape[1], 5).view(shape) if shape[0] > 1 else torch.randn(shape)
    pos, vals = find_outliers_percentile(w, pct)
    gp, gv = find_outliers_percentile(w.to(DEV), pct)
    assert torch.equal(gp.cpu(), pos) and torch.equal(gv.cpu(), vals)


@pytest.mark.parametrize("k", [1, 2, 200, 256])
@pytest.mark.parametrize("n", [1, 3, 4099])
def test_assignment_is_exact_at_midpoints(k, n):
    """fp32 separators give the fp64 midpoint rule: values on, just below and just above every midpoint."""
    from helix_substrate_b200.hxq_writer_gpu import assign_indices
    cb = torch.randn(k, generator=torch.Generator().manual_seed(k)).sort().values
    mids = ((cb[1:].double() + cb[:-1].double()) / 2).float()
    v = torch.cat([mids, torch.nextafter(mids, torch.tensor(9.0)), torch.nextafter(mids, torch.tensor(-9.0)), _special(64, 1), cb])
    v = v.repeat(-(-n // v.numel()))[:n] if n > v.numel() else v[:n]
    assert torch.equal(assign_indices(v.to(DEV), cb.to(DEV)).cpu(), assign_indices(v, cb))
    assert torch.equal(assign_indices(v.to(DEV).bfloat16(), cb.to(DEV)).cpu(), assign_indices(v.bfloat16(), cb))


@pytest.mark.parametrize("n,k", [(1, 1), (3, 8), (5000, 16), (200_000, 256), (600_000, 256)])
def test_kmeans_matches_the_cpu_path(n, k):
    """Same start, steps and stop, counts from the sorted sample; fp32 sums of n / k values of size up to 5 in
    another order differ by at most (n / k) * 2^-24 of a mean each step, ten steps."""
    from helix_substrate_b200.hxq_writer_gpu import kmeans_codebook
    v = torch.randn(n, generator=torch.Generator().manual_seed(n))
    a, b = kmeans_codebook(v.to(DEV), k).cpu(), kmeans_codebook(v, k)
    assert a.shape == b.shape and torch.equal(a, a.sort().values)
    assert float((a - b).abs().max()) <= 10 * 5 * max(1, n // k) * 2.0 ** -24
    assert torch.equal(kmeans_codebook(torch.full((100,), 0.5, device=DEV), 4).cpu(), torch.full((4,), 0.5))


def test_kmeans_roundings_do_not_line_up():
    """One cluster of half a million values: its fp32 sum reaches 2^20, where an addition rounds by up to 1/16.  Added
    in ascending order the roundings of neighbours agree, and every sample's mean is off by 2.2e-4 to 2.6e-4 to the
    same side.  Scattered additions mostly cancel, and how far depends on the hardware's order: twenty samples were off
    by between -1e-5 and 1.6e-4, one of them by -1.6e-4 in another process; mean 7e-5, deviation 5e-5.  So the bound is
    on the average of ten samples: 1.6e-4 is above five deviations of that from 7e-5, and far from what lines up."""
    from helix_substrate_b200.hxq_writer_gpu import kmeans_codebook
    off = []
    for seed in range(10):
        v = 1 + 3 * torch.rand(500_000, device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed))
        mean = float(v.double().mean())
        off.append((float(kmeans_codebook(v, 1, max_iters=1, rtol=0.0)) - mean) / mean)
    assert abs(sum(off) / len(off)) < 1.6e-4, off


@pytest.mark.parametrize("special", [float("-inf"), float("inf"), float("nan")])
def test_kmeans_of_a_special_value(special):
    """An infinity or a NaN reaches the same centroids as in the CPU path, and the others move as there; no steps:
    the percentile start."""
    from helix_substrate_b200.hxq_writer_gpu import kmeans_codebook
    v = torch.cat([torch.tensor([special]), torch.arange(1000.0)])
    for iters in (0, 1, 3):
        a, b = kmeans_codebook(v.to(DEV), 8, max_iters=iters).cpu(), kmeans_codebook(v, 8, max_iters=iters)
        torch.testing.assert_close(a, b, rtol=1e-6, atol=1e-6, equal_nan=True)


@pytest.mark.parametrize("n_out,n_in,G", [(1, 1, 1), (3, 96, 32), (5, 300, 100), (64, 1024, 128)])
@pytest.mark.parametrize("n_ex", [0, 1, 40])
def test_group_fit_matches_the_torch_path(n_out, n_in, G, n_ex):
    """fp64 sums in another order, rounded to fp32 once: equal to a few fp32 ulps; groups of one code,
    wholly excluded groups and unsorted positions included."""
    from helix_substrate_b200.hxq_writer_gpu import fit_group_affine
    g = torch.Generator().manual_seed(n_in)
    w = torch.randn(n_out, n_in, generator=g)
    cb = torch.randn(256, generator=g).sort().values
    idx = torch.randint(0, 256, (n_out, n_in), generator=g).to(torch.uint8)
    idx[0, :G] = 17
    ex = torch.randperm(n_out * n_in, generator=g)[:n_ex]
    if n_ex > 1:
        ex = torch.unique(torch.cat([ex, torch.arange(G)]))[torch.randperm(len(torch.unique(torch.cat([ex, torch.arange(G)]))), generator=g)]
    s, t = fit_group_affine(w, cb, idx, G, ex)
    gs, gt = fit_group_affine(w.to(DEV), cb.to(DEV), idx.to(DEV), G, ex.to(DEV))
    torch.testing.assert_close(gs.cpu(), s, rtol=1e-6, atol=1e-6)
    torch.testing.assert_close(gt.cpu(), t, rtol=1e-6, atol=1e-6)


@pytest.mark.parametrize("n_in,G", [(512, 256), (600, 200), (4096, 4096)])
@pytest.mark.parametrize("keep", [2, 3, 17])
def test_group_fit_with_most_positions_excluded(n_in, G, keep):
    """Lanes that skip runs of excluded positions, some of them given twice; a whole row in one group."""
    from helix_substrate_b200.hxq_writer_gpu import fit_group_affine
    g = torch.Generator().manual_seed(n_in + keep)
    w, cb = torch.randn(3, n_in, generator=g), torch.randn(256, generator=g).sort().values
    idx = torch.randint(0, 256, (3, n_in), generator=g).to(torch.uint8)
    ex = torch.arange(3 * n_in)
    ex = torch.cat([ex[ex % keep != 0], ex[1:7]])
    s, t = fit_group_affine(w, cb, idx, G, ex)
    gs, gt = fit_group_affine(w.to(DEV), cb.to(DEV), idx.to(DEV), G, ex.to(DEV))
    torch.testing.assert_close(gs.cpu(), s, rtol=1e-6, atol=1e-6)
    torch.testing.assert_close(gt.cpu(), t, rtol=1e-6, atol=1e-6)


@pytest.mark.parametrize("bad", [64, -65, 1 << 40])
def test_group_fit_refuses_what_lies_outside(bad):
    """An excluded position outside the matrix, a code outside the codebook: refused on both devices, the ends of
    the range taken."""
    from helix_substrate_b200.hxq_writer_gpu import fit_group_affine
    w, cb, idx = torch.randn(4, 16), torch.arange(8.0), torch.arange(64).view(4, 16).remainder(8).to(torch.uint8)
    for dev in ("cpu", DEV):
        a = [t.to(dev) for t in (w, cb, idx)]
        with pytest.raises(IndexError):
            fit_group_affine(*a, 16, torch.tensor([3, bad], device=dev))
        with pytest.raises(IndexError):
            fit_group_affine(a[0], a[1][:7], a[2], 16)
    ex = torch.tensor([-64, 63, -1])
    for x, y in zip(fit_group_affine(w.to(DEV), cb.to(DEV), idx.to(DEV), 16, ex.to(DEV)), fit_group_affine(w, cb, idx, 16, ex)):
        torch.testing.assert_close(x.cpu(), y, rtol=1e-6, atol=1e-6)


def test_compress_weight_round_trip():
    """The whole encoder on both devices: same outliers, codes that agree but for values next to a
    midpoint, the same reconstruction error."""
    from helix_substrate_b200.hxq_writer_gpu import compress_weight, student_t_weight
    w = student_t_weight((512, 1024), 3, DEV)
    a, b = compress_weight(w, group_size=128), compress_weight(w.cpu(), group_size=128)
    assert torch.equal(a["sidecar_positions"].cpu(), b["sidecar_positions"]) and torch.equal(a["sidecar_values"].cpu(), b["sidecar_values"])
    assert float((a["indices"].cpu() != b["indices"]).float().mean()) < 1e-3

    def err(e):
        e = {k: v.cpu() if torch.is_tensor(v) else v for k, v in e.items()}
        r = e["codebook"][e["indices"].long()].view(512, 8, 128) * e["group_scales"][..., None] + e["group_offsets"][..., None]
        r = r.reshape(-1)
        r[e["sidecar_positions"]] = e["sidecar_values"]
        return float((r - w.cpu().reshape(-1)).norm() / w.cpu().norm())
    assert abs(err(a) - err(b)) < 1e-3 * err(b)
