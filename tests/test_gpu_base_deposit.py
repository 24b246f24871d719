"""DENSITY's base grid and the species sort in their branches: equal masses
(counts and stencil, in store order without patches and in binned order with
them) and unequal ones (atomics, or runs of a cell), particles outside the box
(the stencil's second pass), particles past the species ranges, cells with more
and fewer particles than a thread's chain, grids that are no multiple of a
block.

The base grid's float64 sums are rounded once on both sides: equal but for one
float32 spacing (1.2e-7) at a rounding boundary.  The species sort is exact."""
from types import SimpleNamespace

import numpy as np
import pytest

from asohf_b200 import api, grid, synth
from oracle import oracle as O
from tests.test_gpu_patch_units import table

pytestmark = pytest.mark.gpu


def particles(n, lado0, seed, mass, outside, cores=0.5):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(-0.5 * lado0, 0.5 * lado0, (n, 3))
    k = int(cores * n)
    pos[:k] = rng.uniform(-0.4, 0.4, (8, 3))[rng.integers(0, 8, k)] * lado0 + rng.normal(0, 0.004 * lado0, (k, 3))
    if outside:
        pos[::17] *= 1.25
        pos[1] = 0.5 * lado0
    pos = pos.astype(np.float32)
    m = {"equal": np.full(n, 0.37), "two": np.where(rng.random(n) < 0.3, 8.0, 1.0), "any": 1.0 + rng.random(n)}[mass]
    v = rng.normal(size=n).astype(np.float32)
    return SimpleNamespace(x=pos[:, 0].copy(), y=pos[:, 1].copy(), z=pos[:, 2].copy(), vx=v, vy=v + 1, vz=v - 1,
                           m=m.astype(np.float32), id=np.arange(1, n + 1, dtype=np.int32))


@pytest.mark.parametrize("nx,n,mass,outside,patches", [
    (5, 40, "equal", False, False), (17, 5000, "equal", True, False), (40, 60000, "equal", False, False),
    (17, 5000, "equal", True, True), (40, 60000, "equal", False, True), (33, 20000, "any", False, False),
    (17, 5000, "any", True, True), (40, 60000, "two", False, True), (16, 1, "two", False, True)])
def test_base_grid(gpu_lib, nx, n, mass, outside, patches):
    lado0 = float(nx)
    _, dx = grid.malla(nx, lado0)
    parts = particles(n, lado0, n + nx, mass, outside)
    mesh = table(nx, lado0, float(dx), [(1, 12, 9, 7), (2, 16, 16, 16)] if patches else [(1, 1, 1, 1)])
    if not patches:
        mesh = synth.Mesh(0, np.zeros(1, np.int32), *(np.zeros(0, np.int32) for _ in range(6)),
                          *(np.zeros(0, np.float32) for _ in range(3)), np.zeros(0, np.int32))
    npe = np.zeros(9, np.int32)
    npe[:3] = n // 3, n // 3, n - 2 * (n // 3) - (n > 1000) * 7  # some past the ranges
    g, o = api.GpuBackend(), O.OracleBackend()
    g.upload(parts)
    o.upload(parts)
    args = (nx, np.float32(lado0), dx, np.float32(1.0), np.float32(1.0), npe, mesh)
    u1g, u11g = g.density(*args)
    u1o, u11o = o.density(*args, fp64=True)
    assert np.allclose(u1g, u1o, rtol=2e-7, atol=0)
    assert np.allclose(u11g, u11o, rtol=2e-7, atol=0)


@pytest.mark.parametrize("nx,n,mass", [(3, 1, "two"), (8, 4095, "any"), (8, 4097, "equal"), (20, 50000, "two"),
                                       (64, 9000, "any"), (6, 30000, "equal")])
def test_species_sort(gpu_lib, nx, n, mass):
    lado0 = float(nx)
    _, dx = grid.malla(nx, lado0)
    parts = particles(n, lado0, n, mass, False, cores=0.8)
    g, o = api.GpuBackend(), O.OracleBackend()
    g.upload(parts)
    o.upload(parts)
    for _ in range(2):  # the second sort starts from the sorted store
        ng, no = g.species_sort(nx, dx, np.float32(0.01), np.float32(1.0)), \
            o.species_sort(nx, dx, np.float32(0.01), np.float32(1.0))
        assert np.array_equal(ng, no)
        pg, po = g.download(), o.download()
        for f in ["x", "y", "z", "vx", "vy", "vz", "m", "id"]:
            assert np.array_equal(getattr(pg, f), getattr(po, f)), f
    assert n < 1000 or np.count_nonzero(no) > 1
