"""Work lists whose slices are the smallest, the largest and in between (their
size follows the work of a call): 1 to 130 patches over one crowded core,
in the patch deposits of one and of several masses, in the TSC and in the mesh
counts.  The deposits sum the same REAL*4 terms in float64 as the oracle and
round once: equal but at a rounding boundary, one float32 spacing; the counts
are whole numbers."""
from types import SimpleNamespace

import numpy as np
import pytest

from asohf_b200 import api, grid, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu
NX, LADO0 = 16, 16.0


def parts_of(n, masses):
    rng = np.random.default_rng(n)
    pos = np.clip(rng.normal(0.2, 1.0, (n, 3)), -7.9, 7.9).astype(np.float32)
    m = np.full(n, 0.5) if masses == 1 else rng.choice([0.5, 3.0], n)
    v = np.zeros(n, np.float32)
    return SimpleNamespace(x=pos[:, 0].copy(), y=pos[:, 1].copy(), z=pos[:, 2].copy(), vx=v, vy=v, vz=v,
                           m=m.astype(np.float32), id=np.arange(1, n + 1, dtype=np.int32))


def patches(k, dx):
    rng = np.random.default_rng(k)
    size = rng.integers(24, 33, (3, k)).astype(np.int32)
    size[:, 0] = 32
    corner = (NX // 2 - 8 + rng.integers(-1, 2, (3, k))).astype(np.int32)
    pr = [(np.float32(-LADO0 / 2) + corner[a] * dx + dx / 2).astype(np.float32) for a in range(3)]
    return synth.Mesh(1, np.array([0, k], np.int32), *size, *(corner + 1), *pr, np.zeros(k, np.int32))


# units of up to 512 (64 patches of 8, 128 of 4) and few enough slices: the list of one CTA, else the sorted one
CASES = [(600, 1), (9000, 1), (9000, 5), (120000, 12), (200000, 40), (3000, 64), (3000, 65), (200000, 64), (2000, 128),
         (2000, 129), (60000, 130)]


@pytest.mark.parametrize("n,k", CASES)
@pytest.mark.parametrize("masses", [1, 2])
def test_patch_deposit(gpu_lib, n, k, masses):
    _, dx = grid.malla(NX, LADO0)
    parts, mesh = parts_of(n, masses), patches(k, float(dx))
    npe = np.zeros(9, np.int32)
    npe[:3] = n // 8, n - n // 8 - n // 4, n // 4
    got = []
    for b in (api.GpuBackend(), O.OracleBackend()):
        b.upload(parts)
        args = (NX, np.float32(LADO0), dx, np.float32(1.0), np.float32(1.0), npe, mesh, 2)
        got.append(b.density(*args) if not got else b.density(*args, fp64=True))
    for a, b in zip(*got):
        assert np.allclose(a, b, rtol=2e-7, atol=0.0) and (b > 0).any()


@pytest.mark.parametrize("n,k", CASES)
def test_patch_tsc(gpu_lib, n, k):
    radx, dx = grid.malla(NX, LADO0)
    parts, mesh = parts_of(n, 2), patches(k, float(dx))
    got = []
    for b in (api.GpuBackend(), O.OracleBackend()):
        b.upload(parts)
        args = (NX, np.float32(LADO0), dx, radx, np.float32(1.0), np.float32(1.0), mesh)
        got.append(b.tsc_deposit(*args) if not got else b.tsc_deposit(*args, fp64=True))
    for a, b in zip(*got):
        assert np.allclose(a, b, rtol=2e-7, atol=0.0) and (b > 0).any()


@pytest.mark.parametrize("n,k", CASES)
def test_mesh_counts(gpu_lib, n, k):
    _, dx = grid.malla(NX, LADO0)
    parts, mesh = parts_of(n, 1), patches(k, float(dx))
    lib = api.Asohf(0)
    lib.upload_particles(parts.x, parts.y, parts.z, parts.vx, parts.vy, parts.vz, parts.m, parts.id)
    npe = np.zeros(9, np.int32)
    npe[:2] = n // 2, n - n // 2
    p = (mesh.patchnx, mesh.patchny, mesh.patchnz, mesh.patchrx, mesh.patchry, mesh.patchrz)
    got = np.asarray(lib.mesh_patch_counts(NX, np.float32(LADO0), dx, 1, 8, 1, npe, *p)).reshape(k, 32, 32, 32)
    lib.close()
    w = np.ones(n, np.int64)  # both species reach level 1
    d = np.float32(dx) / np.float32(2.0)
    for q in range(k):
        c = [np.floor((v - (r[q] - d)) / d) for v, r in zip((parts.x, parts.y, parts.z), p[3:])]
        s = [int(p[a][q]) for a in range(3)]
        inside = np.all([(c[a] >= 0) & (c[a] < s[a]) for a in range(3)], axis=0)
        ref = np.zeros((32, 32, 32), np.int64)
        np.add.at(ref, tuple(c[a][inside].astype(int) for a in (2, 1, 0)), w[inside])
        keep = np.zeros_like(ref, bool)
        keep[1:s[2] - 1, 1:s[1] - 1, 1:s[0] - 1] = True
        assert np.array_equal(got[q], np.where(keep, ref, 0)), q
