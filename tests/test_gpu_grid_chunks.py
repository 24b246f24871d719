"""HALOFIND_GRID's ordered chunks: random fields with more peaks than a chunk
(1024), counts that are no multiple of a warp, shells that reach the faces, a
catalogue that fills and a growth past BOUND.  The sums are the reference's
REAL*4 chains, so everything is identical or the status is."""
import numpy as np
import pytest

from asohf_b200 import abi, api, grid
from tests.test_gpu_gridfind import _both, _same

pytestmark = pytest.mark.gpu


def field(nx, seed, sigma):
    rng = np.random.default_rng(seed)
    return np.exp(sigma * rng.standard_normal((nx, nx, nx))).astype(np.float32) * 40


@pytest.mark.parametrize("nx,seed,sigma,contrast", [(5, 1, 1.0, 150.0), (24, 2, 1.0, 150.0), (56, 3, 1.0, 150.0),
                                                    (48, 4, 2.0, 1200.0)])
def test_random_fields(gpu_lib, nx, seed, sigma, contrast):
    radx, dx = grid.malla(nx, float(nx))
    ng, cg, no, co = _both(nx, float(dx), field(nx, seed, sigma), radx, (contrast, 1.0, 1.0, 1.0, 1.0, 4.0 * nx, 0.2))
    assert ng > (1024 if nx >= 48 else 0)
    _same(ng, cg, no, co)


@pytest.mark.parametrize("cap,bound,contrast,code", [(7, 100.0, 150.0, 3), (20000, 1.0, 20.0, 9)])
def test_status(gpu_lib, cap, bound, contrast, code):
    nx = 32
    radx, dx = grid.malla(nx, float(nx))
    with pytest.raises(api.AsohfError) as e:
        api.GpuBackend().halofind_grid_base(nx, float(dx), field(nx, 9, 1.0), radx, contrast, 1.0, 1.0, 1.0, 1.0,
                                            bound, 0.2, abi.Catalogue(cap))
    assert e.value.code == code
