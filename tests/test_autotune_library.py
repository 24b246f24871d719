"""The tuner starts from, checks against and falls back to the untouched
library, whose cluster threshold and share are the rule for a call's members
(0); its space reaches the rule and the small thresholds the rule takes."""
import os
import re

import pytest

from asohf_b200 import autotune as at

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _context_member(name):
    s = open(os.path.join(ROOT, "asohf_b200", "csrc", "common.cuh")).read()
    return int(re.search(r"\b%s = (\d+)[,;]" % name, s).group(1))


def test_library_setting_is_the_untouched_state():
    assert at.LIBRARY == {"tier1": _context_member("tier1_k"), "tier2": _context_member("tier2_k"),
                          "cluster_min": _context_member("cluster_min"),
                          "cluster_share": _context_member("cluster_share")}
    assert at.valid(at.LIBRARY)
    assert not at.valid(dict(at.LIBRARY, cluster_min=1024))  # a threshold below tier2
    for f in ("cluster_min", "cluster_share"):
        assert 0 in at.SPACE[f] and min(v for v in at.SPACE[f] if v) == 2048


@pytest.mark.parametrize("faster,same,want", [(False, True, "LIBRARY"), (True, True, "chosen"),
                                              (True, False, "LIBRARY")])
def test_tune_plan_starts_from_and_returns_to_it(monkeypatch, faster, same, want):
    applied, checked = [], []

    class Lib:
        def set_group_tiers(self, a, b):
            applied.append([a, b])

        def set_cluster_threshold(self, a):
            applied[-1].append(a)

        def set_cluster_share(self, a):
            applied[-1].append(a)

    class Backend:
        a = Lib()
    timed = []

    def timer(p):
        timed.append(dict(p))
        return 1.0 if p == at.LIBRARY else (0.5 if faster and p["cluster_min"] == 8192 else 2.0)
    monkeypatch.setattr(at, "device_timer", lambda *a, **k: timer)
    monkeypatch.setattr(at, "catalogue_of", lambda plan, b, p, subs: checked.append(dict(p)) or dict(p))
    monkeypatch.setattr(at, "same_catalogue", lambda a, b: same)
    best, ms, trials = at.tune_plan(None, Backend(), rounds=1)
    chosen = dict(at.LIBRARY, cluster_min=8192)
    assert timed[0] == at.LIBRARY and checked[0] == at.LIBRARY
    assert best == (at.LIBRARY if want == "LIBRARY" else chosen)
    assert applied[-1] == [best["tier1"], best["tier2"], best["cluster_min"], best["cluster_share"]]
