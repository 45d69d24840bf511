"""Kernel choices by size: every route of the search and of listed windows
gives the values of the all-windows kernels, bit for bit (the cells are the
same operations in the same order on every route)."""
import numpy as np
import pytest
import torch

import oracle
from cudadtw_b200 import Handle, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n,m,w", [
    ("ecg", 3000, 64, 6),        # a handful of LB_Kim survivors
    ("ecg", 33000, 512, 102),    # a warp per survivor in the stream-envelope pass
    ("ecg", 33000, 700, 100),    # few windows, W > 96: lane groups
    ("ecg", 70000, 300, 100),    # many windows, W > 96: register band
    ("ecg", 70000, 300, 30),     # a thread per survivor
    ("metal", 500000, 300, 15),  # a warp per survivor with its own envelope
    ("walk", 140000, 128, 12)])
@pytest.mark.parametrize("metric", ["euclidean", "manhattan"])
def test_search_routes_equal_the_unpruned_argmin(kind, n, m, w, metric):
    make = {"ecg": synth.ecg_like, "metal": synth.metal_like, "walk": synth.random_walk}[kind]
    x = make(n, seed=n + m)
    q, _ = synth.cut_query(x, m, seed=w, noise=0.3)
    dx = torch.from_numpy(x).cuda()
    with Handle(0) as h:
        avg, std = h.avg_std(dx, m)
        h.set_query(q, w)
        d = h.gpu_cdtw(dx, avg, std, metric=metric).cpu().numpy()
        loc, dist = h.prune_cdtw(dx, avg, std, metric)
    best = int(np.argmin(d))
    assert loc == best
    assert dist == (np.sqrt(d[best]) if metric == "euclidean" else d[best])


@pytest.mark.parametrize("w", [0, 1, 7, 8, 28, 29, 96, 97, 106, 107])
@pytest.mark.parametrize("m", [108, 127, 130])
def test_listed_windows_equal_all_windows(w, m):
    """One, two and three windows a thread, blocks of a warp and of four, both
    sides of the register band's limit; M mod 4 of 0, 3 and 2."""
    x = synth.metal_like(80000 + m, seed=m + w)
    q, _ = synth.cut_query(x, m, seed=w, noise=0.3)
    dx = torch.from_numpy(x).cuda()
    with Handle(0) as h:
        avg, std = h.avg_std(dx, m)
        h.set_query(q, w)
        d = h.gpu_cdtw(dx, avg, std)
        some = torch.tensor([0, d.numel() - 1, 17, 17, 40001], dtype=torch.int32, device="cuda")
        np.testing.assert_array_equal(h.gpu_cdtw(dx, avg, std, indices=some).cpu().numpy(),
                                      d[some.long()].cpu().numpy())
        g = torch.Generator().manual_seed(w)
        many = torch.randint(0, d.numel(), (78001,), generator=g).to(torch.int32).cuda()
        np.testing.assert_array_equal(h.gpu_cdtw(dx, avg, std, indices=many).cpu().numpy(),
                                      d[many.long()].cpu().numpy())
        idx = some.cpu().numpy()
        ref = np.array(oracle.cdtw_list(q, x, w, idx))
        got = d[some.long()].cpu().numpy().astype(np.float64)
        assert np.max(np.abs(got - ref) / np.maximum(ref, 1e-3)) < 1e-4
