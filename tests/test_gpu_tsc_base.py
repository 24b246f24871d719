"""INTERPOLATE_DENSITY_TSC without patches, on both sides of the sizes at which
its base grid changes path: in store order with one sum a cell, with 2 and 4,
and from the bins.  Uniform, crowded and on the faces, unequal masses.

Both sides sum the same REAL*4 terms in float64 and round once, then divide
once in REAL*4: equal but at a rounding boundary, one float32 spacing."""
from types import SimpleNamespace

import numpy as np
import pytest

from asohf_b200 import api, grid, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,n", [(8, 1), (24, 65536), (24, 65537), (81, 65537), (162, 65537), (32, 2 ** 21),
                                  (33, 2 ** 21 + 1)])
def test_base_grid(gpu_lib, nx, n):
    lado0 = np.float32(20.0)
    radx, dx = grid.malla(nx, lado0)
    rng = np.random.default_rng(n)
    pos = rng.uniform(-0.5, 0.5, (n, 3)) * float(lado0)
    k = n // 2
    pos[:k] = np.clip(rng.normal(0.2, 0.02, (k, 3)), -0.5, 0.5) * float(lado0)
    pos[k:k + n // 8, 0] = -0.5 * float(lado0)  # on a face
    pos = pos.astype(np.float32)
    v = np.zeros(n, np.float32)
    parts = SimpleNamespace(x=pos[:, 0].copy(), y=pos[:, 1].copy(), z=pos[:, 2].copy(), vx=v, vy=v, vz=v,
                            m=(1.0 + rng.random(n)).astype(np.float32), id=np.arange(1, n + 1, dtype=np.int32))
    z, zf = np.zeros(0, np.int32), np.zeros(0, np.float32)
    mesh = synth.Mesh(0, np.zeros(1, np.int32), z, z, z, z, z, z, zf, zf, zf, z)
    got = []
    for b in (api.GpuBackend(), O.OracleBackend()):
        b.upload(parts)
        args = (nx, lado0, dx, radx, np.float32(1.0), np.float32(1.0), mesh)
        got.append(b.tsc_deposit(*args)[0] if not got else b.tsc_deposit(*args, fp64=True)[0])
    assert np.allclose(*got, rtol=2e-7, atol=0)
