"""Catalogue fields below 256 KB cross to the device packed, larger ones by a
copy of their own: the calls give the same rows for a short catalogue and for
one whose fields are just below and just at that size (65536 rows of 4 bytes;
the wider fields are above it in both), filled up with dead rows that keep their
values.  Same kernels and groups in each: integers and IDs equal, floats to the
1e-5 of the reductions' order."""
from types import SimpleNamespace

import numpy as np
import pytest

from asohf_b200 import abi, api, driver, synth

pytestmark = pytest.mark.gpu


def chain(snap, plan, rows):
    """prune, halofind, cleaning and one level of substructure on the plan's
    candidates followed by dead rows up to `rows` (0: none)."""
    cfg, cand, cos = snap.cfg, plan.cand, plan.cos
    b = api.GpuBackend()
    b.upload(SimpleNamespace(**{f: getattr(snap, f) for f in ("x", "y", "z", "vx", "vy", "vz", "m", "id")}))
    b.species_sort(cfg.nx, plan.dx, cos["rodo"], cos["re0"])
    b.sort_x(cfg.nx, np.float32(cfg.lado0))
    n = len(cand.clusrx)
    total = max(rows, n)
    cat = abi.Catalogue(total + 4096)
    rng = np.random.default_rng(3)
    for f in cat.fields():
        a = getattr(cat, f)
        a[n:total] = rng.integers(1, 1000, a[n:total].shape)
    for f in ("clusrx", "clusry", "clusrz", "radio", "masa", "levhal", "patchclus"):
        getattr(cat, f)[:n] = getattr(cand, f)
    for f in ("clusrx", "clusry", "clusrz"):
        getattr(cat, f)[n:total] = rng.uniform(-0.25, 0.25, total - n) * cfg.lado0
    for f in ("radio", "patchclus", "realclus"):
        getattr(cat, f)[n:total] = 0
    cat.levhal[n:total] = plan.mesh.nl  # levels never decrease
    cat.realclus[:n] = -1
    cat.nclus = total
    dead = {f: getattr(cat, f)[n:total].copy() for f in cat.fields() if f not in ("dmpclus", "indcs")}
    b.prune_poor_haloes(plan.consts, cat, 1, total, np.float32(1.0), 1)
    b.halofind_particles(plan.consts, plan.mesh, cat, 1, total, None)
    b.check_rubish(cat, 1, total)
    b.accidental_substructure(cat)
    for f, a in dead.items():
        assert np.array_equal(getattr(cat, f)[n:total], a), f
    assert (cat.indcs[n:total] == -1).all() and (cat.dmpclus[n:total] == 0).all()
    slot = np.zeros(max(snap.halo_pos.shape[0], 1), np.int64)
    known = cand.truth >= 0
    slot[cand.truth[known]] = 1 + np.nonzero(known)[0]
    sx, sy, sz, srad, shost, _, slev = synth.build_sub_candidates(
        snap, slot, lambda s: cat.realclus[s - 1] == -1, float(plan.dx), plan.mesh.nl)
    ir = int(np.argmax(slev[1:])) + 1
    lo, ns = int(np.sum(slev[1:ir])), int(slev[ir])
    assert ns > 0
    at = slice(total, total + ns)
    cat.clusrx[at], cat.clusry[at], cat.clusrz[at] = sx[lo:lo + ns], sy[lo:lo + ns], sz[lo:lo + ns]
    cat.rsub[at], cat.realclus[at], cat.levhal[at] = srad[lo:lo + ns], shost[lo:lo + ns], ir
    cat.nclus = total + ns
    subs_lev = np.zeros(plan.mesh.nl + 1, np.int32)
    subs_lev[0], subs_lev[ir] = total, ns
    b.substructure_particles(plan.consts, plan.mesh, cat, ir, subs_lev, None)
    keep = np.r_[0:n, total:total + ns]
    return {f: getattr(cat, f)[keep].copy() for f in cat.fields()}, b.a.particles_per_halo().copy()


@pytest.mark.parametrize("rows", [65535, 65536])
def test_large_catalogues_give_the_rows_of_short_ones(gpu_lib, rows):
    snap = synth.generate("small")
    plan = driver.prepare(snap)
    want, ids = chain(snap, plan, 0)
    got, ids2 = chain(snap, plan, rows)
    assert (want["realclus"] != 0).sum() > 10 and np.array_equal(ids, ids2)
    for f, a in want.items():
        if a.dtype == np.int32:
            assert np.array_equal(got[f], a), f
        else:
            np.testing.assert_allclose(got[f], a, rtol=1e-5, atol=1e-30, err_msg=f)
