"""INTERPOLATE_DENSITY_TSC where its work units end: patches of 1 to 32 cells
(partial and empty plane slabs), dense cells (many particles of a warp on one
target), units cut into several slices, single particles, unequal masses and
particles on and beyond the box faces.

Both sides sum the same REAL*4 terms in float64 and round once, then divide
once in REAL*4: the sums differ by float64 rounding, so the results are equal
but where a sum sits at a rounding boundary, one float32 spacing (1.2e-7)."""
from types import SimpleNamespace

import numpy as np
import pytest

from asohf_b200 import api, grid, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def table(nx, lado0, dx, sizes):
    """Patches of the given (level, nx, ny, nz), corners near the box centre."""
    rows = sorted(sizes)
    nl = max(r[0] for r in rows)
    a = lambda k: np.array([r[k] for r in rows], np.int32)
    lev = a(0)
    rng = np.random.default_rng(len(rows))
    corner = np.array([[nx // 2 - 4 + rng.integers(0, 3) for _ in range(3)] for _ in rows], np.int32)
    pr = [(np.float32(-lado0 / 2) + corner[:, k] * dx + dx / 2.0 ** lev).astype(np.float32) for k in range(3)]
    z = np.zeros(len(rows), np.int32)
    return synth.Mesh(nl, np.bincount(lev, minlength=nl + 1).astype(np.int32), a(1), a(2), a(3),
                      corner[:, 0] + 1, corner[:, 1] + 1, corner[:, 2] + 1, *pr, z)


SIZES = [(1, 32, 32, 32), (1, 14, 9, 1), (2, 8, 32, 7), (2, 1, 1, 1), (3, 31, 17, 25), (3, 16, 8, 9)]


@pytest.mark.parametrize("n,core,spread", [(1, 0, 0.1), (33, 0, 0.2), (5000, 4000, 0.002), (40000, 30000, 0.05),
                                           (60000, 60000, 0.0005)])
def test_patch_and_base_tsc(gpu_lib, n, core, spread):
    nx, lado0 = 24, 24.0
    radx, dx = grid.malla(nx, lado0)
    rng = np.random.default_rng(n)
    pos = rng.uniform(-0.5 * lado0, 0.5 * lado0, (n, 3))
    pos[:core] = rng.normal(0, spread * lado0, (core, 3)) + 0.7
    if n > 100:
        pos[-1], pos[-2], pos[-3] = -0.5 * lado0, 0.5 * lado0, 0.53 * lado0
    pos = pos.astype(np.float32)
    v = np.zeros(n, np.float32)
    parts = SimpleNamespace(x=pos[:, 0].copy(), y=pos[:, 1].copy(), z=pos[:, 2].copy(), vx=v, vy=v, vz=v,
                            m=(1.0 + rng.random(n)).astype(np.float32), id=np.arange(1, n + 1, dtype=np.int32))
    mesh = table(nx, lado0, float(dx), SIZES)
    g, o = api.GpuBackend(), O.OracleBackend()
    g.upload(parts)
    o.upload(parts)
    args = (nx, np.float32(lado0), dx, radx, np.float32(1.0), np.float32(1.0), mesh)
    u1g, u11g = g.tsc_deposit(*args)
    u1o, u11o = o.tsc_deposit(*args, fp64=True)
    assert np.allclose(u1g, u1o, rtol=2e-7, atol=0)
    assert np.allclose(u11g, u11o, rtol=2e-7, atol=0)
    assert n < 100 or (u11o > 0).any()
