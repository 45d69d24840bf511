"""Top-k picks and distances, by either name of the call, against a greedy
selection on the host over the unpruned all-windows cDTW (the same cells, so
both are exact): few and many picks (the ordered rounds drop what is consumed
or covered), more picks than fit, equal distances, every kernel that collects
the candidates."""
import time

import numpy as np
import pytest
import torch

from cudadtw_b200 import Handle, synth

pytestmark = pytest.mark.gpu


def greedy(d, k, M):
    """As many as k windows at least M apart, by (distance, window)."""
    at = np.full(d.size // M + 3, -(1 << 40), np.int64)  # the accepted window of each M starts
    taken = []
    for w in np.argsort(d, kind="stable"):
        b = int(w) // M + 1
        if not np.isfinite(d[w]) or len(taken) == k:
            break
        if np.all(np.abs(at[b - 1:b + 2] - w) >= M):
            at[b] = w
            taken.append(int(w))
    return np.array(taken, np.int64)


def _check(x, q, W, k, metric, variant="auto"):
    M = q.size
    dx = torch.from_numpy(x).cuda()
    with Handle(0) as h:
        avg, std = h.avg_std(dx, M)
        h.set_band_variant(W, W, variant)
        h.set_query(q, W)
        full = h.gpu_cdtw(dx, avg, std, metric=metric).cpu().numpy()
        want = greedy(full, k, M)
        dist = np.sqrt(full[want]) if metric == 0 else full[want]
        for call in (h.topk, h.topk_device):
            locs, dists = call(dx, avg, std, k, metric=metric)
            np.testing.assert_array_equal(locs, want)
            np.testing.assert_array_equal(dists, dist)


@pytest.mark.parametrize("kind,n,M,P,k", [
    ("ecg", 4000, 64, 10, 1000), ("ecg", 1 << 16, 64, 10, 20), ("ecg", 1 << 18, 64, 10, 1000),
    ("ecg", 1 << 17, 64, 10, 1 << 20), ("walk", 1 << 17, 100, 5, 700), ("walk", 1 << 17, 33, 20, 3000),
    ("ties", 1 << 16, 64, 10, 1 << 20), ("ties", 1 << 16, 50, 10, 300), ("metal", 200001, 96, 5, 1500)])
@pytest.mark.parametrize("metric", [0, 1])
def test_picks_and_distances(kind, n, M, P, k, metric):
    if kind == "ties":  # an integer pattern of period 96 over and over
        x = np.tile(np.random.default_rng(1).integers(0, 6, 96), n // 96 + 1)[:n].astype(np.float32)
    else:
        x = {"ecg": synth.ecg_like, "metal": synth.metal_like, "walk": synth.random_walk}[kind](n, 7)
    q, _ = synth.cut_query(x, M, seed=9, noise=0.05)
    _check(x, q, synth.band_from_percent(M, P), k, metric)


@pytest.mark.parametrize("variant,W", [("register", 102), ("lane", 102), ("strip16", 102),
                                       ("strip32", 102), ("auto", 204)])
@pytest.mark.parametrize("k", [25, 5000])
def test_wide_bands(variant, W, k):
    x = synth.metal_like(1 << 16, seed=12)
    q, _ = synth.cut_query(x, 512, seed=13, noise=0.2)
    _check(x, q, W, k, 0, variant)


def test_many_picks_do_not_reread_the_whole_list():
    """As many picks as fit, every window a hit: about 20 times the call for 100
    picks on 2^20 windows, 400 times where each round reads all of them again."""
    n, M = 1 << 20, 64
    x = synth.ecg_like(n, seed=7)
    q, _ = synth.cut_query(x, M, seed=9, noise=0.05)
    dx = torch.from_numpy(x).cuda()
    took = []
    with Handle(0) as h:
        avg, std = h.avg_std(dx, M)
        h.set_query(q, 6)
        for k in (100, n // M):
            runs = []
            for _ in range(4):
                torch.cuda.synchronize()
                t = time.perf_counter()
                h.topk(dx, avg, std, k)
                runs.append(time.perf_counter() - t)
            took.append(min(runs))
    assert took[1] <= 100 * took[0]
