"""LDTW quotients at the edges of the exact-residual division: deviations about
2^-60, 2^40 and 2^60, means about 2^-60, 2^-70 and 0, so that quotients come
near the subnormal numbers; equal bit for bit to numpy's float32 steps."""
import numpy as np
import pytest
import torch

from test_gpu_ldtw_walk import _walk

pytestmark = pytest.mark.gpu

F = np.float32


@pytest.mark.parametrize("sd_exp", [-61, -60, -59, 39, 40, 41, 60, 62])
@pytest.mark.parametrize("mean_exp", [-71, -62, -60, -58, None])
def test_quotients_at_the_edges(sd_exp, mean_exp):
    from cudadtw_b200 import Handle
    m, nw, w = 32, 300, 4
    rng = np.random.default_rng(sd_exp + 100)
    # +A and -A in turn: their sum over a window is 0 but for the small samples
    a = F(2.0) ** sd_exp
    x = np.where(np.arange(nw + m - 1) % 2, a, -a).astype(F)
    if mean_exp is not None:
        small = np.arange(0, x.size - 1, 8)  # pairs of small samples every 8
        x[small] = x[small + 1] = F(m * 2.0 ** mean_exp) * rng.uniform(0.5, 1.0, small.size)
    q = rng.standard_normal(m).astype(F)
    with np.errstate(all="ignore"):
        ref = _walk(q, x, w, True, True)
    with Handle(0) as h:
        h.set_query(q, w)
        got = h.ldtw_ref_all_windows(torch.from_numpy(x).cuda(), 0).cpu().numpy()
    np.testing.assert_array_equal(got, ref)
