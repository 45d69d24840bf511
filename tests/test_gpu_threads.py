"""Handles on several host threads (one handle a thread, as the header allows)
calling the same kernels with different lengths, hence different amounts of
shared memory: every call succeeds and gives what it gives alone, bit for bit."""
import threading

import numpy as np
import pytest
import torch

from cudadtw_b200 import synth

pytestmark = pytest.mark.gpu


def _ldtw(h, x, q, m):
    h.set_query(q[:m], 3)
    return h.ldtw_ref_all_windows(x, 0)


def _stats(h, x, q, m):
    return torch.cat([v.double() for v in h.avg_std(x, m)])


def _ed(h, x, q, m):
    return h.ed_all_windows(torch.from_numpy(q[:m].astype(np.float64)).cuda(), x.double())


def _pair(h, x, q, m):
    path = torch.zeros(h.pair_path_bytes(4, m), dtype=torch.uint8, device="cuda")
    s = x[:8 * m].reshape(2, 4, m).contiguous()
    h.pair_fwd(s[0], s[1], 20, path=path)
    return torch.cat([g.reshape(-1) for g in h.pair_bwd(s[0], s[1], path)])


@pytest.mark.parametrize("call,lengths", [(_ldtw, (4200, 8192, 5000)), (_stats, (5500, 8192, 7000)),
                                          (_ed, (3000, 8192, 5000)), (_pair, (600, 1000, 1024))])
def test_lengths_on_several_threads(call, lengths):
    from cudadtw_b200 import Handle
    x = torch.from_numpy(synth.ecg_like(8192 + 500, seed=2)).cuda()
    q = synth.ecg_like(8192, seed=3)
    want = {}
    for m in lengths:
        with Handle(0) as h:
            want[m] = call(h, x, q, m)
    torch.cuda.synchronize()
    wrong = []

    def work(m):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream), Handle(0) as h:
                for _ in range(200):
                    got = call(h, x, q, m)
                stream.synchronize()
                if not torch.equal(got, want[m]):
                    wrong.append((m, "differs"))
        except Exception as e:  # a launch that another thread's limit refused
            wrong.append((m, str(e)))

    threads = [threading.Thread(target=work, args=(m,)) for m in lengths]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
