"""The layer's forward on both sides of its size rule (small sets in input
order with float64 sums, larger ones sorted), with most particles in a few
cells, on grids of both transforms: rho and pot against float64.

rho: a float32 sum of n positive terms added in runs of 32 is within
(log2(32) + n/32) 2^-24 of the exact sum where every term of a cell is equal;
n <= 5100 in a cell here gives 1e-5.  pot: the Poisson solve's own bound 2e-6 of
the largest value, plus rho's error through a solve that averages it."""
import numpy as np
import pytest
import torch

from asohf_b200.autograd import DepositPoissonLayer
from tests.test_gpu_mesh import _solve64

pytestmark = pytest.mark.gpu


def rho64(layer, pos, m, L):
    nx, dx, radx = layer.nx, float(layer.dx), layer.radx.astype(np.float64)
    cells, ws = [], []
    for v in pos:
        i = np.clip(((v - np.float32(-np.float32(L) / 2)) / np.float32(dx)).astype(np.int64) + 1, 1, nx)
        d = [np.abs(v.astype(np.float64) - radx[i + o]) / dx for o in (-1, 0, 1)]
        ws.append([0.5 * (1.5 - d[0]) ** 2, 0.75 - d[1] ** 2, 0.5 * (1.5 - d[2]) ** 2])
        cells.append([(i - 1 + o) % nx for o in (-1, 0, 1)])
    out = np.zeros(nx ** 3)
    for k in range(3):
        for j in range(3):
            for i in range(3):
                np.add.at(out, (cells[2][k] * nx + cells[1][j]) * nx + cells[0][i],
                          m * ws[0][i] * ws[1][j] * ws[2][k])
    den = dx ** 3 * float(layer.rote) * float(layer.rete) ** 3
    return out.reshape(nx, nx, nx) / den


@pytest.mark.parametrize("nx,batch,n", [(16, 1, 1), (20, 3, 777), (64, 2, 81920), (64, 2, 81921), (48, 1, 163841)])
def test_forward_paths(gpu_lib, nx, batch, n):
    L = 10.0
    layer = DepositPoissonLayer(nx, L)
    rng = np.random.default_rng(n)
    pos = rng.uniform(-L / 2, L / 2, (3, batch, n))
    dense = rng.random((batch, n)) < 0.5
    blob = rng.uniform(-L / 2, L / 2, (3, 16))[:, rng.integers(0, 16, (batch, n))]
    pos = np.where(dense, blob + rng.normal(0, 0.02 * L / nx, (3, batch, n)), pos)
    pos = np.clip(pos, -0.4999 * L, 0.4999 * L).astype(np.float32)
    m = (0.5 + rng.random((batch, n))).astype(np.float32)
    t = [torch.tensor(a, device="cuda") for a in (*pos, m)]
    rho, pot = (a.cpu().numpy() for a in layer.forward(*t))
    for b in range(batch):
        ref = rho64(layer, pos[:, b], m[b].astype(np.float64), L)
        assert np.abs(rho[b] - ref).max() <= 1e-5 * np.abs(ref).max()
        phi = _solve64(ref, layer.dx)
        assert np.abs(pot[b] - phi).max() <= 4e-6 * np.abs(phi).max()
