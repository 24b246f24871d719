"""HALOFIND_GRID on wide haloes, whose shells are walked by the rows that can
meet them instead of by every cell of their box: centres at the middle, by the
faces and in a corner (clipped boxes), odd sizes, noise on the profile and a
shell box of one width on either side of the change.  The sums are the
reference's REAL*4 chains, so everything is identical."""
import numpy as np
import pytest

from asohf_b200 import grid
from tests.test_gpu_gridfind import _both, _same

pytestmark = pytest.mark.gpu


def field(nx, centres, r200, noise, contrast=200.0):
    """max over the centres of contrast r200^2/3 / (r+1)^2: mean contrast `contrast` near r200 cells."""
    q = np.arange(nx, dtype=np.float64)
    u = np.ones((nx, nx, nx))
    for (i, j, k), rad in zip(centres, r200):
        r = np.sqrt(((q - k) ** 2)[:, None, None] + ((q - j) ** 2)[None, :, None] + ((q - i) ** 2)[None, None, :])
        u = np.maximum(u, contrast * rad ** 2 / 3 / (r + 1) ** 2)
    rng = np.random.default_rng(nx)
    return (u * np.exp(noise * rng.standard_normal(u.shape))).astype(np.float32)


@pytest.mark.parametrize("nx,centres,r200,noise", [
    (41, [(20, 20, 20)], [9.5], 0.0),      # boxes to 15 cells
    (41, [(20, 20, 20)], [11.0], 0.0),     # and to 17
    (64, [(20, 22, 31), (52, 50, 12)], [13.0, 9.0], 0.02),
    (75, [(3, 40, 37), (70, 71, 72)], [22.0, 15.0], 0.05),
    (96, [(48, 47, 46)], [34.0], 0.0),
    (96, [(30, 90, 2), (60, 20, 60)], [30.0, 18.0], 0.1)])
def test_wide_haloes(gpu_lib, nx, centres, r200, noise):
    radx, dx = grid.malla(nx, float(nx))
    ng, cg, no, co = _both(nx, float(dx), field(nx, centres, r200, noise), radx,
                           (200.0, 1.0, 1.0, 1.0, 1.0, 0.5 * nx, 0.2))
    assert ng > 0 and cg.radio[:ng].max() > 5 * dx
    _same(ng, cg, no, co)
