"""Windowed statistics and the ED's 1 / sigma on inputs that cancel: large
samples and level steps that enter and leave, flat runs, bad samples, at
lengths around the 16 windows a thread slides over.

Bounds: a window's sums are FP64 sums about one of its own samples (at most 16
slides and 13 joins, 2^-48 of its largest sample's square), taken again where
the variance is below 2^-22 (FP32 sigma) or 2^-10 (FP64) of the second moment:
means to 2^-47 of the window's largest sample, FP32 sigmas to their rounding
2^-24 and 1e-7, FP64 ones to 2^-37."""
import numpy as np
import pytest
import torch

from cudadtw_b200 import synth

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 8, 11, 14, 15, 16, 17, 31, 32, 100, 333, 1024]


def _windows(x, m):
    return np.lib.stride_tricks.sliding_window_view(x.astype(np.longdouble), m)


def _ref(x, m):
    win = _windows(x, m)
    mu, sd = np.empty(len(win), np.longdouble), np.empty(len(win), np.longdouble)
    for a in range(0, len(win), 1024):
        w = win[a:a + 1024]
        d = w - w[:, :1]
        mean = d.mean(1, keepdims=True)
        mu[a:a + 1024] = w[:, 0] + mean[:, 0]
        sd[a:a + 1024] = np.sqrt(np.square(d - mean).mean(1))
        sd[a:a + 1024][w.max(1) == w.min(1)] = 1.0
    return mu, sd


def _hard(kind, m):
    """9000 samples; tiles are 2048 windows, a thread's windows 16."""
    x = synth.ecg_like(9000, seed=m)
    if kind == "spikes":  # behind the first window of threads 0, 5 and 128 + 3
        for t, o in ((0, 0), (5, 1), (131, 3), (300, 2)):
            x[16 * t + m + o] = np.float32(3.0e6)
    elif kind == "steps":
        x[m:2000] = np.float32(1234.567)
        x[2048 + m:4000] = np.float32(-77.7)
        x[6000:] += np.float32(3.0e6)
    elif kind == "flat":
        x[1000:2300] = np.float32(0.37)
        x[5000:5000 + m + 9] = np.float32(-1.7)
    elif kind == "bad":
        x[[0, 2048, 5000, 5003, 7000 + m]] = np.float32(np.nan)
        x[3001] = np.float32(np.inf)
    return x


@pytest.mark.parametrize("m", LENGTHS)
@pytest.mark.parametrize("kind", ["spikes", "steps", "flat", "bad"])
def test_statistics(kind, m):
    from cudadtw_b200 import Handle
    x = _hard(kind, m)
    with Handle(0) as h:
        mu, sd = h.avg_std(torch.from_numpy(x).cuda(), m)
        mu, sd = mu.cpu().numpy(), sd.cpu().numpy()
    with np.errstate(invalid="ignore"):
        rmu, rsd = _ref(x, m)
        top = np.abs(_windows(x, m)).max(1)
    ok = np.isfinite(rmu)
    assert np.array_equal(np.isfinite(mu), ok)
    assert np.all(np.abs(mu[ok] - rmu[ok]) <= 2.0 ** -47 * top[ok])
    assert np.max(np.abs(sd[ok] / rsd[ok] - 1.0)) <= 2.0 ** -24 + 1e-7


@pytest.mark.parametrize("m", [2, 11, 15, 16, 33, 333])
@pytest.mark.parametrize("kind", ["spikes", "steps", "flat"])
def test_ed_on_the_same_inputs(kind, m):
    from cudadtw_b200 import Handle
    x = _hard(kind, m).astype(np.float64)
    q = np.cumsum(np.random.default_rng(m).standard_normal(m))
    with Handle(0) as h:
        got = h.ed_all_windows(torch.from_numpy(q).cuda(), torch.from_numpy(x).cuda())
        got = got.cpu().numpy()
    z = q.astype(np.longdouble) - q.astype(np.longdouble).mean()
    z /= np.sqrt(np.square(z).mean())
    _, sd = _ref(x, m)
    win = _windows(x, m)
    want = 2 * m - 2 * (win @ z) / sd
    size = 2 * m + 2 * (np.abs(win) @ np.abs(z)) / sd  # FP64 sums of m terms and sigma
    assert np.all(np.abs(got - want) <= (m * 2.0 ** -53 + 2.0 ** -37) * size)


def test_ed_precision_on_an_ordinary_stream():
    """FP64 sigmas from about 30 roundings of 2^-53: 3.4e-15 (sums that hold the
    whole tile lost a few more bits)."""
    from cudadtw_b200 import Handle
    n, m = 1 << 15, 64
    x = synth.ecg_like(n, seed=5).astype(np.float64)
    q = synth.cut_query(x.astype(np.float32), m, 3, 0.1)[0].astype(np.float64)
    with Handle(0) as h:
        got = h.ed_all_windows(torch.from_numpy(q).cuda(), torch.from_numpy(x).cuda())
        got = got.cpu().numpy()
    z = q.astype(np.longdouble) - q.astype(np.longdouble).mean()
    z /= np.sqrt(np.square(z).mean())
    want = 2 * m - 2 * (_windows(x, m) @ z) / _ref(x, m)[1]
    err = (got - want).astype(np.float64) / (2 * m)
    assert np.sqrt(np.square(err).mean()) <= 3.4e-15


def _time(h, x, m):
    d = torch.from_numpy(x).cuda()
    runs = []
    for _ in range(8):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        h.avg_std(d, m)
        b.record()
        torch.cuda.synchronize()
        runs.append(a.elapsed_time(b))
    return min(runs)


def test_bad_samples_do_not_serialise_the_pass():
    """A NaN every 3000 samples concerns a thread in 188: at most twice the time
    of a clean stream, with as much again for the clock."""
    from cudadtw_b200 import Handle
    x = synth.ecg_like(1 << 20, seed=3)
    y = x.copy()
    y[::3000] = np.float32(np.nan)
    with Handle(0) as h:
        assert _time(h, y, 2000) <= 4.0 * _time(h, x, 2000)


def test_single_samples_take_no_longer_than_short_windows():
    """Windows of one sample have no variance to lose (each taken again took 2.5
    times the pass)."""
    from cudadtw_b200 import Handle
    x = synth.metal_like(1 << 23, seed=3)
    with Handle(0) as h:
        assert _time(h, x, 1) <= 1.3 * _time(h, x, 32)
