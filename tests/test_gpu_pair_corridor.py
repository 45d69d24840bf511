"""The path from checkpoints (the library's choice, and the forced
recomputation) equals the one from stored directions byte for byte: at the
edges of the lane shapes (W + 1 a multiple of 32, of a lane's slots, just
inside and outside what the checkpoints' scratch holds), for segments that
start at the origin or hold one anti-diagonal, with ties everywhere (integer
series), and on series whose path hugs the band."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _series(kind, n, L, seed):
    g = torch.Generator().manual_seed(seed)
    q, s = torch.randn(n, L, generator=g), torch.randn(n, L, generator=g)
    if kind == "walk":
        q, s = q.cumsum(1), s.cumsum(1)
    elif kind == "ties":
        q, s = torch.round(q), torch.round(s)
    else:  # the path runs along one edge of the band
        t = torch.arange(L, dtype=torch.float32)
        q, s = (t + 0.01 * q), (0.5 * t + 0.01 * s)
    return q.cuda(), s.cuda()


@pytest.mark.parametrize("L,W,n", [
    (257, 3, 1), (260, 0, 9), (260, 1, 9), (261, 2, 9), (262, 15, 5), (300, 30, 7), (300, 31, 7),
    (700, 35, 33), (400, 59, 5), (400, 63, 5), (400, 127, 5), (400, 128, 5), (600, 239, 4),
    (600, 255, 4), (600, 256, 4), (2048, 409, 3), (700, 479, 3), (700, 480, 3), (1100, 511, 3),
    (300, 299, 3), (8192, 100, 2)])
@pytest.mark.parametrize("kind", ["walk", "ties", "edge"])
@pytest.mark.parametrize("metric", ["euclidean", "manhattan"])
def test_path_from_checkpoints_equals_stored_directions(L, W, n, kind, metric):
    from cudadtw_b200 import Handle
    q, s = _series(kind, n, L, L + W)
    got = {}
    with Handle(0) as h:
        for mode in (None, "recompute", "store"):
            path = torch.zeros(h.pair_path_bytes(n, L), dtype=torch.uint8, device="cuda")
            D = h.pair_fwd(q, s, W, metric=metric, znorm=kind == "walk", path=path, mode=mode)
            got[mode] = (D.cpu(), path.cpu())
    for mode in (None, "recompute"):
        assert torch.equal(got[mode][0], got["store"][0])
        assert torch.equal(got[mode][1], got["store"][1])


@pytest.mark.parametrize("W", [15, 31, 32])
@pytest.mark.parametrize("over", [0, 1])
def test_default_path_at_the_chip_filling_count(W, over):
    # narrow bands (W + 1 <= 32 slots) keep direction bits above 14 pairs an SM
    from cudadtw_b200 import Handle
    n = 14 * torch.cuda.get_device_properties(0).multi_processor_count + over
    q, s = _series("walk", n, 290, W)
    got = {}
    with Handle(0) as h:
        for mode in (None, "recompute", "store"):
            path = torch.zeros(h.pair_path_bytes(n, 290), dtype=torch.uint8, device="cuda")
            D = h.pair_fwd(q, s, W, path=path, mode=mode)
            got[mode] = (D.cpu(), path.cpu())
    for mode in (None, "recompute"):
        assert torch.equal(got[mode][0], got["store"][0])
        assert torch.equal(got[mode][1], got["store"][1])
