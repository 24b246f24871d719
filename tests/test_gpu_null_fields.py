"""A host catalogue with a missing array is refused with a status by every call
that would read or write it (the packed hand-over reads and writes the caller's
arrays on the host), and the context goes on working."""
import ctypes as C

import numpy as np
import pytest

from asohf_b200 import abi, api, driver, synth

pytestmark = pytest.mark.gpu
INVALID = 1
PRUNE = ["clusrx", "radio", "realclus", "dmpclus"]
CLEAN = ["clusry", "vx", "masa", "levhal", "realclus"]
OVERLAP = ["clusrz", "radio", "levhal", "realclus"]
ALL = ["clusrx", "masa", "vcmax", "dmpclus", "iplip", "profiles", "inertia_tensor", "indcs"]


@pytest.fixture(scope="module")
def case(gpu_lib):
    s = synth.generate("tiny")
    plan = driver.prepare(s)
    b = api.GpuBackend()
    b.upload(s)
    b.species_sort(s.cfg.nx, plan.dx, plan.cos["rodo"], plan.cos["re0"])
    b.sort_x(s.cfg.nx, np.float32(s.cfg.lado0))
    n = len(plan.cand.clusrx)
    cat = abi.Catalogue(n + 64)
    for f in ("clusrx", "clusry", "clusrz", "radio", "masa", "levhal", "patchclus"):
        getattr(cat, f)[:n] = getattr(plan.cand, f)
    cat.realclus[:n] = -1
    cat.nclus = n
    return s, plan, b, cat


def _call(case, name, cc):
    s, plan, b, cat = case
    L, h, n = b.a.L, b.a.h, cat.nclus
    mh = abi.MeshHolder(plan.mesh)
    k, out = C.byref(plan.consts), C.c_int32()
    if name == "prune":
        return L.asohf_prune_poor_haloes(h, k, C.byref(cc), 1, n, C.c_float(1.0), 1, 0)
    if name == "halofind":
        return L.asohf_halofind_particles(h, k, C.byref(mh.c), C.byref(cc), 1, n, 0)
    if name == "substructure":
        lev = np.zeros(plan.mesh.nl + 1, np.int32)
        lev[1] = n
        return L.asohf_substructure_particles(h, k, C.byref(mh.c), C.byref(cc), 1,
                                              lev.ctypes.data_as(C.POINTER(C.c_int32)), 0)
    if name == "rubish":
        return L.asohf_check_rubish(h, C.byref(cc), n, 1, n, 0, C.byref(out))
    if name == "accidental":
        return L.asohf_accidental_substructure(h, C.byref(cc), n, 0, C.byref(out))
    nh = np.array([n], np.int32)
    return L.asohf_overlapping(h, C.byref(cc), 0, nh.ctypes.data_as(C.c_void_p), C.c_float(0.2), 0, C.byref(out))


@pytest.mark.parametrize("name,fields", [("prune", PRUNE), ("halofind", ALL), ("substructure", ALL),
                                         ("rubish", CLEAN), ("accidental", CLEAN), ("overlapping", OVERLAP)])
def test_missing_arrays_are_refused(case, name, fields):
    for f in fields:
        cc = case[3].as_c()
        setattr(cc, f, None)
        assert _call(case, name, cc) == INVALID, f
    case[2].prune_poor_haloes(case[1].consts, case[3], 1, case[3].nclus, np.float32(1.0), 1)


def test_grid_finder_refuses_missing_columns(case):
    s, plan, b, cat = case
    cfg, cos = s.cfg, plan.cos
    npe = b.a.sort_dm_particles_localdensity(cfg.nx, plan.dx, cos["rodo"], cos["re0"])
    empty = synth.build_mesh(s, float(plan.dx), nl=0)
    u1 = np.empty(cfg.nx ** 3, np.float32)
    b.a.density(cfg.nx, np.float32(cfg.lado0), plan.dx, cos["rote"], cos["rete"], npe, empty, 2, u1, None)
    b.a.renorm_density(cfg.nx, empty, np.float32(cfg.fdm), u1, None)
    out = abi.Catalogue(20000)
    args = (cfg.nx, plan.dx, u1, plan.radx, cos["contrastec"], cos["rote"], cos["rete"], cos["rodo"], cos["re0"],
            np.float32(cfg.lado0 / 4), 0.2)
    as_c = out.as_c
    for f in ("levhal", "clusrx", "masa", "clusrzcm"):
        def broken():
            cc = as_c()
            setattr(cc, f, None)
            return cc
        out.as_c = broken
        with pytest.raises(api.AsohfError) as e:
            b.a.halofind_grid_base(*args, out)
        assert e.value.code == INVALID, f
    out.as_c = as_c
    assert b.a.halofind_grid_base(*args, out) > 0
