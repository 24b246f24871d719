"""DENSITY's patch deposit where its work units end: patches of 1 to 32 cells
at every level to 6 (clouds of 3 to 129 cells a side, so counted, tabulated and
listed hits), units cut into several slices, few and no particles, both kernels,
species ranges set by hand, equal masses, masses whose terms leave the normal
range, and unequal masses.

Both sides sum the same REAL*4 terms in float64, round once and divide once in
REAL*4: results differ by one float32 spacing (1.2e-7) at most where a sum sits
at a rounding boundary, and below the normal range by one spacing of it
(1.4e-45) over the cell volume."""
from types import SimpleNamespace

import numpy as np
import pytest

from asohf_b200 import api, grid, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [(1, 32, 32, 32), (1, 14, 9, 1), (2, 8, 32, 7), (2, 1, 1, 1), (3, 31, 17, 25), (4, 16, 8, 9), (5, 32, 32, 30),
         (6, 32, 5, 32)]


def table(nx, lado0, dx, sizes):
    rows = sorted(sizes)
    nl = max(r[0] for r in rows)
    col = lambda k: np.array([r[k] for r in rows], np.int32)
    lev = col(0)
    rng = np.random.default_rng(len(rows))
    corner = np.array([[nx // 2 - 4 + rng.integers(0, 5) for _ in range(3)] for _ in rows], np.int32)
    pr = [(np.float32(-lado0 / 2) + corner[:, k] * dx + dx / 2.0 ** lev).astype(np.float32) for k in range(3)]
    z = np.zeros(len(rows), np.int32)
    return synth.Mesh(nl, np.bincount(lev, minlength=nl + 1).astype(np.int32), col(1), col(2), col(3),
                      corner[:, 0] + 1, corner[:, 1] + 1, corner[:, 2] + 1, *pr, z)


@pytest.mark.parametrize("n,spread,split,degree,mass", [
    (1, 0.1, [1], 2, "equal"),
    (37, 0.2, [20, 10, 7], 1, "equal"),
    (3000, 0.3, [1000, 800, 600, 300, 200, 100], 2, "equal"),
    (20000, 0.1, [500, 1500, 6000, 12000], 1, "equal"),
    (70000, 0.03, [300, 700, 30000, 39000], 2, "equal"),   # slices, a dense core
    (9000, 0.1, [9000], 2, "equal"),                       # every hit listed: the list fills
    (5000, 0.1, [2000, 2000, 900], 2, "equal"),            # 100 particles past the species ranges
    (4000, 0.2, [1000, 1000, 2000], 2, "subnormal"),
    (4000, 0.2, [1000, 1000, 2000], 2, "unequal"),
])
def test_patch_deposit(gpu_lib, n, spread, split, degree, mass):
    nx, lado0 = 16, 16.0
    _, dx = grid.malla(nx, lado0)
    rng = np.random.default_rng(n)
    pos = np.clip(rng.normal(0, spread * lado0, (n, 3)) + 0.3, -7.9, 7.9).astype(np.float32)
    m = {"equal": np.full(n, 0.37), "subnormal": np.full(n, 1e-33), "unequal": 1.0 + rng.random(n)}[mass]
    v = np.zeros(n, np.float32)
    parts = SimpleNamespace(x=pos[:, 0].copy(), y=pos[:, 1].copy(), z=pos[:, 2].copy(), vx=v, vy=v, vz=v,
                            m=m.astype(np.float32), id=np.arange(1, n + 1, dtype=np.int32))
    mesh = table(nx, lado0, float(dx), SIZES)
    npe = np.zeros(9, np.int32)
    npe[:len(split)] = split
    g, o = api.GpuBackend(), O.OracleBackend()
    g.upload(parts)
    o.upload(parts)
    args = (nx, np.float32(lado0), dx, np.float32(1.0), np.float32(1.0), npe, mesh, degree)
    u1g, u11g = g.density(*args)
    u1o, u11o = o.density(*args, fp64=True)
    atol = 1.5e-45 * 2.0 ** 18 if mass == "subnormal" else 0.0
    assert np.allclose(u11g, u11o, rtol=2e-7, atol=atol)
    assert np.allclose(u1g, u1o, rtol=2e-7, atol=atol)
    assert (u11o > 0).any()
