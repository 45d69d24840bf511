"""Searches at W = 97..106, where the number of candidates picks the kernel on
the device: on both sides of it the result is the unpruned arg-min bit for bit,
and so are the top-k picks, which collect through the same kernels."""
import numpy as np
import pytest
import torch

from cudadtw_b200 import Handle, synth

pytestmark = pytest.mark.gpu

GATE = 1 << 15


@pytest.mark.parametrize("w", [96, 97, 106, 107])
@pytest.mark.parametrize("n,far,many", [(30000, True, False), (36000, True, True),
                                        (90000, True, True), (90000, False, False)])
@pytest.mark.parametrize("metric", [0, 1])
def test_both_sides_of_the_gate(w, n, far, many, metric):
    m = 300
    if far:  # noise against noise: few windows are pruned
        x = np.random.default_rng(3).standard_normal(n).astype(np.float32)
        q = np.random.default_rng(4).standard_normal(m).astype(np.float32)
    else:
        x = synth.metal_like(n, seed=5)
        q = synth.cut_query(x, m, seed=6, noise=0.1)[0]
    dx = torch.from_numpy(x).cuda()
    with Handle(0) as h:
        avg, std = h.avg_std(dx, m)
        h.set_query(q, w)
        full = h.gpu_cdtw(dx, avg, std, metric=metric)
        best = int(torch.argmin(full).item())
        loc, dist = h.prune_cdtw(dx, avg, std, metric)
        assert (h.search_counts()[2] > GATE) == many
        assert loc == best
        d = full[best].item()
        assert dist == (np.sqrt(np.float32(d)) if metric == 0 else np.float32(d))
        locs, dists = h.topk(dx, avg, std, 3, metric=metric)
        assert locs[0] == best and dists[0] == dist
