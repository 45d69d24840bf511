"""Windowed statistics at the tile's edges (2048 windows, chunks of eight
samples), against two-pass FP64 sums: means to 1e-12 of the stream's range
(2^-52 times the square root of the 10^4 terms of a tile's prefix), sigmas to
one FP32 rounding (2^-24) plus 1e-9 of the FP64 ones."""
import numpy as np
import pytest
import torch

from cudadtw_b200 import synth

pytestmark = pytest.mark.gpu


def _ref(x, m):
    win = np.lib.stride_tricks.sliding_window_view(x.astype(np.float64), m)
    mu = np.empty(len(win))
    sd = np.empty(len(win))
    for a in range(0, len(win), 512):
        w = win[a:a + 512]
        mu[a:a + 512] = w[:, 0] + (w - w[:, :1]).mean(1)
        var = np.square(w - mu[a:a + 512, None]).mean(1)
        sd[a:a + 512] = np.sqrt(var)
    const = (win.max(1) == win.min(1))
    sd[const | (sd == 0)] = 1.0
    return mu, sd


def _check(x, m):
    from cudadtw_b200 import Handle
    with Handle(0) as h:
        mu, sd = h.avg_std(torch.from_numpy(x).cuda(), m)
        mu, sd = mu.cpu().numpy(), sd.cpu().numpy()
    rmu, rsd = _ref(x, m)
    ok = np.isfinite(rmu)
    assert np.all(np.isfinite(mu) == ok)
    assert np.max(np.abs(mu[ok] - rmu[ok])) <= 1e-12 * np.ptp(x[np.isfinite(x)]) + 1e-300
    assert np.max(np.abs(sd[ok] / rsd[ok] - 1.0)) <= 2.0 ** -24 + 1e-9


@pytest.mark.parametrize("m", [1, 2, 7, 8, 9, 63, 128, 2047, 2048, 2049, 8192, 8193])
@pytest.mark.parametrize("nw", [1, 2047, 2048, 2049, 6000])
def test_tile_edges(m, nw):
    _check(synth.metal_like(nw + m - 1, seed=m + nw), m)


def test_flat_runs_and_level_shift():
    x = synth.ecg_like(9000, seed=3)
    x[1000:2300] = np.float32(0.37)   # flat inside a tile and across its end
    x[5000:5100] = np.float32(-1.7)
    x[7000:] += np.float32(3.0e6)     # the tile's shift is far from these windows
    for m in (16, 100, 333):
        _check(x, m)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_bad_sample_spoils_its_own_windows_only(bad):
    x = synth.ecg_like(7000, seed=4)
    x[2048] = bad  # the first sample of a tile
    x[5000] = bad
    _check(x, 128)
