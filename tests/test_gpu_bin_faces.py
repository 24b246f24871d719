"""Particles a few float spacings from the faces of the work units' bins: the
host cell INT((z - corner) / cell) rounds up where the unit's own lower bound
does not, so such a particle lies below the bound and still deposits.  Every
axis, patches of several levels inside the box, by its lower face and a cell past
it, the cell the REAL*4 quotient of box and grid (RADX's own spacing, a little
smaller, keeps the bounds off the faces); the patch deposits of one and of two masses and
the TSC against the oracle (the same REAL*4 terms in float64 sums, rounded once:
equal but at a rounding boundary, one float32 spacing), the mesh counts against
a count in float32."""
from types import SimpleNamespace

import numpy as np
import pytest

from asohf_b200 import api, grid, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


MEET = {100: [41, 43, 45], 64: [15, 19, 22], 96: [29, 33], 128: [29, 31, 45]}  # corners whose bounds round past a face


def case(nx, lado0):
    """Patches at several corners, particles around every multiple of the cell near them."""
    dx = np.float32(lado0) / np.float32(nx)
    rng = np.random.default_rng(nx)
    rows = []
    for lev in (1, 2, 3):
        for c in [-1, 0, 1] + MEET.get(nx, []) + list(rng.integers(2, nx - 18, 6)):
            rows.append((lev, int(c)))
    lev = np.array([r[0] for r in rows], np.int32)
    corner = np.array([[r[1]] * 3 for r in rows], np.int32).T
    size = np.full(len(rows), 32, np.int32)
    pr = [(np.float64(np.float32(-lado0 / 2)) + corner[a] * np.float64(dx) + np.float64(dx) / 2.0 ** lev)
          .astype(np.float32) for a in range(3)]
    mesh = synth.Mesh(3, np.bincount(lev, minlength=4).astype(np.int32), size, size, size, *(corner + 1), *pr,
                      np.zeros(len(rows), np.int32))
    pts = []
    for q in range(len(rows)):
        for k in range(-3, 36):  # planes of the patch and around it
            z = np.float32(pr[2][q] + k * np.float64(dx) / 2.0 ** lev[q] - np.float64(dx) / 2.0 ** lev[q])
            up = down = z
            for _ in range(8):
                pts += [up, down]
                up, down = np.nextafter(up, np.float32(np.inf)), np.nextafter(down, np.float32(-np.inf))
    z = np.unique(np.array(pts, np.float32))
    z = z[np.abs(z) < np.float32(lado0) / 2]
    out = []
    for axis in range(3):  # the exact values on one axis, patch interiors on the others
        p = np.empty((z.size, 3), np.float32)
        p[:] = (z + 0.31 * np.float32(dx))[:, None]
        p[:, axis] = z
        out.append(p)
    pos = np.concatenate(out)
    pos = pos[(np.abs(pos) < np.float32(lado0) / 2).all(axis=1)]
    pos = pos[rng.permutation(len(pos))]
    return dx, mesh, pos


def parts_of(pos, masses):
    n = len(pos)
    m = np.full(n, 0.5) if masses == 1 else np.where(np.arange(n) % 2, 0.5, 3.0)
    v = np.zeros(n, np.float32)
    return SimpleNamespace(x=pos[:, 0].copy(), y=pos[:, 1].copy(), z=pos[:, 2].copy(), vx=v, vy=v, vz=v,
                           m=m.astype(np.float32), id=np.arange(1, n + 1, dtype=np.int32))


BOXES = [(100, 20.0), (64, 20.0 / 0.678), (96, 40.0 / 0.678), (128, 62.5 / 0.678), (40, 40.0)]


@pytest.mark.parametrize("nx,lado0", BOXES)
@pytest.mark.parametrize("masses", [1, 2])
def test_deposits(gpu_lib, nx, lado0, masses):
    dx, mesh, pos = case(nx, lado0)
    parts = parts_of(pos, masses)
    npe = np.zeros(9, np.int32)
    npe[:3] = len(pos) // 3, len(pos) // 3, len(pos) - 2 * (len(pos) // 3)
    radx, _ = grid.malla(nx, np.float32(lado0))
    one = np.float32(1.0)
    g, o = api.GpuBackend(), O.OracleBackend()
    for b in (g, o):
        b.upload(parts)
    for a, b in zip(g.density(nx, np.float32(lado0), dx, one, one, npe, mesh, 2),
                    o.density(nx, np.float32(lado0), dx, one, one, npe, mesh, 2, fp64=True)):
        assert np.allclose(a, b, rtol=2e-7, atol=0.0) and (b > 0).any()
    for a, b in zip(g.tsc_deposit(nx, np.float32(lado0), dx, radx, one, one, mesh),
                    o.tsc_deposit(nx, np.float32(lado0), dx, radx, one, one, mesh, fp64=True)):
        assert np.allclose(a, b, rtol=2e-7, atol=0.0) and (b > 0).any()


@pytest.mark.parametrize("nx,lado0", BOXES)
def test_mesh_counts(gpu_lib, nx, lado0):
    dx, mesh, pos = case(nx, lado0)
    parts = parts_of(pos, 1)
    lib = api.Asohf(0)
    lib.upload_particles(parts.x, parts.y, parts.z, parts.vx, parts.vy, parts.vz, parts.m, parts.id)
    npe = np.zeros(9, np.int32)
    npe[0] = len(pos)
    first = 0
    for lev in (1, 2, 3):
        sl = slice(first, first + int(mesh.npatch[lev]))
        first = sl.stop
        p = [a[sl] for a in (mesh.patchnx, mesh.patchny, mesh.patchnz, mesh.patchrx, mesh.patchry, mesh.patchrz)]
        got = np.asarray(lib.mesh_patch_counts(nx, np.float32(lado0), dx, lev, 8, 1, npe, *p)).reshape(-1, 32, 32, 32)
        d = np.float32(dx) / np.float32(2.0 ** lev)
        for q in range(got.shape[0]):
            c = [np.floor((v - (r[q] - d)) / d) for v, r in zip((parts.x, parts.y, parts.z), p[3:])]
            inside = np.all([(v >= 0) & (v < 32) for v in c], axis=0)
            ref = np.zeros((32, 32, 32), np.int64)
            np.add.at(ref, tuple(c[a][inside].astype(int) for a in (2, 1, 0)), 1)
            keep = np.zeros(ref.shape, bool)
            keep[1:-1, 1:-1, 1:-1] = True
            assert np.array_equal(got[q], np.where(keep, ref, 0)), (lev, q)
    lib.close()
