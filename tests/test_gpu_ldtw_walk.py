"""LDTW in the reference's FP32 arithmetic against the same steps taken with
numpy's correctly rounded float32 operations: equal bit for bit.  Sizes at
the block's edges (256 windows), the longest query, and inputs whose
quotients leave the range of the exact-residual division."""
import numpy as np
import pytest
import torch

from cudadtw_b200 import synth

pytestmark = pytest.mark.gpu

F = np.float32
INFTY = F(1e10)


def _walk(q, x, w, euclid, znorm):
    m, nw = q.size, x.size - q.size + 1
    if znorm:
        avg, sd = F(0), F(0)
        for v in q:
            avg, sd = F(avg + v), F(sd + F(v * v))
        avg = F(avg / F(m))
        q = (q - avg) / np.sqrt(F(F(sd / F(m)) - F(avg * avg)))
    win = np.lib.stride_tricks.sliding_window_view(x, m)
    if znorm:
        s1, s2 = np.zeros(nw), np.zeros(nw)
        for k in range(m):  # in sample order; the products are exact in FP64
            v = x[k:k + nw].astype(np.float64)
            s1 += v
            s2 += v * v
        a, ex2 = (s1 / m).astype(F), (s2 / m).astype(F)
        var = (ex2.astype(np.float64) - a.astype(np.float64) ** 2).astype(F)
        sd = np.where(var > 0, np.sqrt(np.maximum(var, F(0))), F(1))
        win = (win - a[:, None]) / sd[:, None]
    cost = (lambda d: d * d) if euclid else np.abs
    r = np.arange(nw)
    i, j = np.zeros(nw, int), np.zeros(nw, int)
    d = cost(q[0] - win[:, 0])
    for _ in range(2 * m - 2):
        vi, vj = i + 1 < m, j + 1 < m
        i1, j1 = np.minimum(i + 1, m - 1), np.minimum(j + 1, m - 1)
        diag = np.where(vi & vj, cost(q[i1] - win[r, j1]), INFTY)
        down = np.where(vi & (np.abs(i - j + 1) <= w), cost(q[i1] - win[r, j]), INFTY)
        rght = np.where(vj & (np.abs(j - i + 1) <= w), cost(q[i] - win[r, j1]), INFTY)
        md = (diag < down) & (diag < rght)
        mi = md | (~(diag < down) & (down < rght))
        step = np.where(md, diag, np.where(mi, down, rght))
        d = d + np.where(vi | vj, step, F(0))
        i, j = np.where(mi, i1, i), np.where(md | ~mi, j1, j)
    return d


@pytest.mark.parametrize("m,nw,w,euclid,znorm,scale", [
    (2, 257, 0, True, True, 1.0), (2, 256, 1, False, False, 1.0), (5, 1, 1, True, True, 1.0),
    (37, 255, 4, True, True, 1.0), (64, 1000, 0, False, True, 1.0), (97, 513, 30, True, True, 1.0),
    (128, 700, 12, True, False, 1.0), (64, 300, 6, True, True, 1e-24),
    (64, 300, 6, False, True, 1e22), (8192, 3, 40, True, True, 1.0)])
def test_ldtw_reference_arithmetic_steps(m, nw, w, euclid, znorm, scale):
    from cudadtw_b200 import Handle
    x = synth.metal_like(nw + m - 1, seed=m + nw)
    x[:m // 2] = x[0]  # a constant run (sigma 1 where it fills a window)
    x = (x * F(scale)).astype(F)
    q = (synth.random_walk(m, seed=w + 1) * F(scale)).astype(F)
    with np.errstate(all="ignore"):
        ref = _walk(q, x, w, euclid, znorm)
    with Handle(0) as h:
        h.set_query(q, w)
        got = h.ldtw_ref_all_windows(torch.from_numpy(x).cuda(), 0 if euclid else 1,
                                     znorm=znorm).cpu().numpy()
    np.testing.assert_array_equal(got, ref)
