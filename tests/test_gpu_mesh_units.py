"""CREATE_MESH patch counts where the work units end: dense patches cut into
several slices, partial plane slabs, one particle, no particles in a patch.
Integer counts: identical."""
from types import SimpleNamespace

import numpy as np
import pytest

from tests.test_gpu_mesh_counts import backends

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,spread,irpa", [(1, 0.1, 1), (70000, 0.01, 1), (70000, 0.003, 3), (30000, 0.2, 2)])
def test_units(gpu_lib, n, spread, irpa):
    nx, lado0 = 24, 24.0
    dx = lado0 / nx
    rng = np.random.default_rng(n + irpa)
    pos = np.clip(rng.normal(0.4, spread * lado0, (n, 3)), -11.9, 11.9).astype(np.float32)
    v = np.zeros(n, np.float32)
    g, o = backends(SimpleNamespace(x=pos[:, 0].copy(), y=pos[:, 1].copy(), z=pos[:, 2].copy(), vx=v, vy=v, vz=v,
                                    m=np.ones(n, np.float32), id=np.arange(1, n + 1, dtype=np.int32)))
    n3 = np.array([[32, 32, 32], [1, 1, 1], [9, 30, 8], [16, 7, 17], [32, 32, 25], [20, 20, 20]], np.int32)
    dpar = dx / 2.0 ** (irpa - 1)
    k = np.array([[-7, -7, -7], [0, 0, 0], [-2, -9, -1], [-5, -2, -4], [0, 0, 0], [-20, -20, -20]])
    pr = (0.5 * dpar + dpar * k).astype(np.float32)
    args = (n3[:, 0], n3[:, 1], n3[:, 2], pr[:, 0], pr[:, 1], pr[:, 2])
    esp = [n // 2, n // 4]
    cg = g.a.mesh_patch_counts(nx, lado0, dx, irpa, 8, 1, esp, *args)
    co = o.mesh_patch_counts(irpa, dx, 8, 1, esp, *args)
    assert np.array_equal(cg, co)
