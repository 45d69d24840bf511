"""Few windows at the bands that both the register band and the lane groups
take (W = 97..106): the values at the edges of the rule are those of either
kernel bit for bit, and a handful of windows takes no longer than on the lane
groups (a thread's chain over the whole band took 1.3 to 1.6 times that)."""
import pytest
import torch

from cudadtw_b200 import Handle, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [96, 97, 104, 105, 106, 107])
@pytest.mark.parametrize("metric", ["euclidean", "manhattan"])
def test_values_at_the_edges(w, metric):
    m = 121
    block = 64 * torch.cuda.get_device_properties(0).multi_processor_count
    x = torch.from_numpy(synth.metal_like(2 * block + m + 1, seed=w)).cuda()
    q, _ = synth.cut_query(x.cpu().numpy(), m, seed=w, noise=0.3)
    with Handle(0) as h:
        avg, std = h.avg_std(x, m)
        h.set_band_variant(w, w, "auto" if w > 106 else "register")
        h.set_query(q, w)
        want = h.gpu_cdtw(x, avg, std, metric=metric)
        h.set_band_variant(w, w, "auto")
        h.set_query(q, w)
        for n in (1, 2, 63, block - 1, block, block + 1, 2 * block, 2 * block + 1):
            got = h.gpu_cdtw(x[:n + m - 1].contiguous(), avg[:n].contiguous(),
                             std[:n].contiguous(), metric=metric)
            assert torch.equal(got, want[:n])
            idx = torch.arange(n, dtype=torch.int32, device="cuda").flip(0).contiguous()
            got = h.gpu_cdtw(x, avg, std, indices=idx, metric=metric)
            assert torch.equal(got, want[:n].flip(0))


@pytest.mark.parametrize("w", [97, 102, 106])
@pytest.mark.parametrize("n", [64, 4096])
def test_no_slower_than_the_lane_groups(w, n):
    m = 1024
    x = torch.from_numpy(synth.metal_like(n + m - 1, seed=w)).cuda()
    q, _ = synth.cut_query(x.cpu().numpy(), m, seed=w, noise=0.3)
    took = {}
    with Handle(0) as h:
        avg, std = h.avg_std(x, m)
        for variant in ("lane", "auto"):
            h.set_band_variant(w, w, variant)
            h.set_query(q, w)
            runs = []
            for _ in range(8):
                a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                a.record()
                h.gpu_cdtw(x, avg, std)
                b.record()
                torch.cuda.synchronize()
                runs.append(a.elapsed_time(b))
            took[variant] = min(runs)
    assert took["auto"] <= 1.1 * took["lane"]
