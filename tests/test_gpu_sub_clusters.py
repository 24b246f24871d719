"""Subhaloes refined by thread-block clusters: the subhalo call takes clusters
from the smaller of the set threshold and max(tier2, 2048) members on, so small
sets reach them only where a small threshold is set.  1 sends every subhalo to a
cluster of 8 CTAs, 100 some of them; one and several particle masses (cumulative
masses by count and by scans), with and without energies, bars as in the halo
tests: integers and ID lists identical, floats to 1e-5."""
import numpy as np
import pytest

from asohf_b200 import api, driver, synth
from oracle import oracle as O
from tests.catalogue_compare import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["tiny", "small"])
@pytest.mark.parametrize("masses", ["equal", "unequal"])
@pytest.mark.parametrize("threshold", [1, 100])
def test_clusters_match_oracle(gpu_lib, name, masses, threshold):
    s = synth.generate(name)
    if masses == "unequal":
        rng = np.random.default_rng(7)
        s.m = (s.m * (1.0 + 0.5 * rng.random(s.m.shape[0]))).astype(np.float32)
    rg = driver.run(s, api.GpuBackend(cluster_threshold=threshold), with_subs=True)
    ro = driver.run(s, O.OracleBackend(), with_subs=True)
    assert np.array_equal(rg.subs_lev, ro.subs_lev)
    assert (ro.cat.realclus[ro.subs_lev[0]: ro.cat.nclus] > 0).sum() > 0
    compare(rg, ro)


@pytest.mark.parametrize("threshold", [1, 100])
def test_energies_match_oracle(gpu_lib, threshold):
    s = synth.generate("tiny")
    runs = []
    for b in (api.GpuBackend(cluster_threshold=threshold), O.OracleBackend()):
        p = driver.prepare(s)
        p.consts.do_compute_energies = 1
        p.consts.max_part_dsum = 1 << 30
        runs.append(driver.execute(p, b, with_subs=True))
    rg, ro = runs
    compare(rg, ro)
    n = ro.cat.nclus
    for f in ("kinetic_e", "potential_e"):
        a, b = (getattr(r.cat, f)[:n].astype(np.float64) for r in (rg, ro))
        assert np.all(np.abs(a - b) <= 1e-5 * np.maximum(np.abs(b), 1e-30)), f
