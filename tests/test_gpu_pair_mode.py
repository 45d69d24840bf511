"""pair_last_mode names the scratch of the last pair_fwd with a path: "store"
for the default (whatever that scratch held), "recompute" where the smaller one
is forced or taken by the memory limit; other calls leave the answer alone."""
import numpy as np
import pytest
import torch

from cudadtw_b200 import Handle, synth

pytestmark = pytest.mark.gpu


def _pairs(n, L):
    g = torch.Generator().manual_seed(L)
    return [torch.randn(n, L, generator=g).cumsum(1).cuda() for _ in range(2)]


@pytest.mark.parametrize("L,W", [(300, 30), (700, 70), (2048, 409), (700, 480)])
def test_default_and_forced(L, W):
    q, s = _pairs(4, L)
    with Handle(0) as h:
        path = torch.zeros(h.pair_path_bytes(4, L), dtype=torch.uint8, device="cuda")
        for mode, want in ((None, "store"), ("recompute", "recompute"), (None, "store"),
                           ("store", "store")):
            h.pair_fwd(q, s, W, path=path, mode=mode)
            assert h.pair_last_mode() == want
    q, s = _pairs(400, L)  # (a work area has at least 1 MiB)
    with Handle(0) as h:  # half the limit is less than the direction bits take
        path = torch.zeros(h.pair_path_bytes(400, L), dtype=torch.uint8, device="cuda")
        h.set_memory_limit(h.pair_workspace_bytes(400, L, W, mode="store"))
        h.pair_fwd(q, s, W, path=path)
        assert h.pair_last_mode() == "recompute"


def test_a_refinement_leaves_the_answer_alone():
    L, W = 300, 30
    q, s = _pairs(4, L)
    x = synth.ecg_like(1 << 14, seed=5)
    t = synth.cut_query(x, L, seed=6, noise=0.2)[0]
    with Handle(0) as h:
        path = torch.zeros(h.pair_path_bytes(4, L), dtype=torch.uint8, device="cuda")
        h.pair_fwd(q, s, W, path=path, mode="store")
        h.refine_templates(torch.from_numpy(x).cuda(), [t], [W], np.arange(0, 8000, 400)[None], 1)
        assert h.pair_last_mode() == "store"
