"""The tuner's band limits are those of the kernels, and a tuned variant that
is the library's own choice leaves its rules by the number of windows on."""
import os
import re

from cudadtw_b200 import autotune as at

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cudadtw_b200",
                    "csrc")


def _constant(name, file):
    with open(os.path.join(CSRC, file)) as f:
        return int(re.search(rf"constexpr int {name} = (\d+);", f.read()).group(1))


def test_register_band_is_a_candidate_as_far_as_the_kernels_go():
    plain = _constant("kMaxRegW", "cdtw_reg.cuh")
    batched = _constant("kMaxBatchRegW", "batch_reg.cuh")
    assert plain > batched
    for w in (batched, batched + 1, plain, plain + 1):
        assert ("register" in at.variant_candidates(w)) == (w <= plain)
        assert any(r == 0 for r, _ in at.batched_candidates(w)) == (w <= batched)
        rows, _ = at.shapes_for([[0] * 512, [0] * 64], [w, 5],
                                {at.bucket(64, 5): {"rows": 0, "tiles": 512}})
        assert rows[0] == (0 if w <= batched else 16)


def test_apply_leaves_the_built_in_choice_on_auto():
    class Fake:
        def __init__(self):
            self.set = {}

        def set_band_variant(self, lo, hi, v):
            assert lo == hi
            self.set[lo] = v

    h = Fake()
    at.apply_variants(h, {"40": "register", "41": "lane", "102": "register", "103": "lane",
                          "204": "lane", "205": "strip32", "384": "strip16", "800": "strip16"})
    assert h.set == {40: "auto", 41: "lane", 102: "auto", 103: "lane", 204: "auto",
                     205: "strip32", 384: "auto", 800: "auto"}
