"""The layer's forward on crowded small sets (particles of a warp that share a
cell deposit together; sets of more than 65536 particles use 2 or 4 sums a
cell): all in one cell, in the corner cells around a wrapped vertex, in a blob
of a few cells, on both sides of the sizes at which the number of sums changes.

A REAL*4 weight is within 4 x 2^-24 of its float64 value and at most 0.75, the
mass and the three products add 4 roundings, so a term is within 8 x 2^-24 m;
the sums are float64.  At least one cell holds an eighth of a crowded set, so
the error is within 64 x 2^-24 = 3.8e-6 of the largest cell."""
import numpy as np
import pytest
import torch

from asohf_b200.autograd import DepositPoissonLayer
from tests.test_gpu_layer_paths import rho64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,batch,n", [(8, 1, 31), (24, 3, 1000), (24, 2, 65536), (24, 2, 65537), (80, 1, 70000),
                                        (81, 1, 70000), (160, 1, 163840)])
@pytest.mark.parametrize("kind", ["cell", "vertex", "blob"])
def test_crowded_sets(gpu_lib, nx, batch, n, kind):
    L = 10.0
    layer = DepositPoissonLayer(nx, L)
    rng = np.random.default_rng(n + nx)
    cell = L / nx
    if kind == "vertex":  # either side of the box's corner
        pos = rng.uniform(0.0, 0.4 * cell, (3, batch, n)) * rng.choice([-1.0, 1.0], (3, batch, n))
        pos = np.where(pos < 0, pos + L / 2, pos - L / 2)
    else:
        centre = -L / 2 + (nx // 3 + 0.5) * cell
        pos = centre + (rng.uniform(-0.2, 0.2, (3, batch, n)) if kind == "cell"
                        else np.clip(rng.normal(0, 0.4, (3, batch, n)), -2, 2)) * cell
    pos = np.clip(pos, -0.49999 * L, 0.49999 * L).astype(np.float32)
    m = (0.5 + rng.random((batch, n))).astype(np.float32)
    rho, _ = layer.forward(*(torch.tensor(a, device="cuda") for a in (*pos, m)))
    for b in range(batch):
        ref = rho64(layer, pos[:, b], m[b].astype(np.float64), L)
        assert np.abs(rho[b].cpu().numpy() - ref).max() <= 64 * 2.0 ** -24 * ref.max()
