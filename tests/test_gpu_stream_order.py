"""The first calls of a context on a non-blocking stream give what a context on
the default stream gives: the tables a context keeps are in place before the
kernels that read them."""
import numpy as np
import pytest
import torch

from asohf_b200 import api, grid, synth

pytestmark = pytest.mark.gpu


def _density(s, mesh, degree, stream=None):
    cfg = s.cfg
    radx, dx = grid.malla(cfg.nx, np.float32(cfg.lado0))
    cos = grid.cosmology(cfg.h, cfg.omega_m, cfg.zeta)
    a = api.Asohf(0)
    if stream is not None:
        a.set_stream(stream.cuda_stream)
    a.upload_particles(s.x, s.y, s.z, s.vx, s.vy, s.vz, s.m, s.id)
    npe = a.sort_dm_particles_localdensity(cfg.nx, dx, cos["rodo"], cos["re0"])
    out = []
    for nl in range(mesh.nl + 1):  # more levels from call to call: the kept tables grow
        m = synth.build_mesh(s, float(dx), nl=nl)
        u1 = np.empty(cfg.nx ** 3, np.float32)
        u11 = np.empty((max(m.total, 1), 32 ** 3), np.float32)
        a.density(cfg.nx, np.float32(cfg.lado0), dx, cos["rote"], cos["rete"], npe, m, degree, u1, u11)
        out += [u1, u11[:m.total].copy()]
    a.close()
    return out


@pytest.mark.parametrize("degree", [1, 2])
def test_first_density_on_a_non_blocking_stream(gpu_lib, degree):
    s = synth.generate("tiny")
    _, dx = grid.malla(s.cfg.nx, np.float32(s.cfg.lado0))
    mesh = synth.build_mesh(s, float(dx))
    want = _density(s, mesh, degree)
    got = _density(s, mesh, degree, torch.cuda.Stream())
    for a, b in zip(got, want):  # float64 sums in any order, rounded once to REAL*4
        assert np.allclose(a, b, rtol=2.0 ** -23, atol=0.0)


@pytest.mark.parametrize("nx", [24, 64])
def test_first_solves_on_a_non_blocking_stream(gpu_lib, nx):
    g = torch.Generator(device="cuda").manual_seed(nx)
    L = np.float32(20.0)
    radx, dx = grid.malla(nx, L)
    cos = grid.cosmology(0.678, 0.31, 0.0)
    xyz = [((torch.rand(3000, generator=g, device="cuda") - 0.5) * 0.999 * float(L)) for _ in range(3)]
    m = torch.ones(3000, device="cuda")
    rho = torch.randn(nx ** 3, generator=g, device="cuda")
    got = []
    for st in (torch.cuda.default_stream(), torch.cuda.Stream()):
        st.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(st):
            pot, dep, phi = (torch.empty(nx ** 3, device="cuda") for _ in range(3))
            for fn in ("poisson", "forward"):  # each the first call of its context
                a = api.Asohf(0)
                a.set_stream(st.cuda_stream)
                if fn == "poisson":
                    a.poisson_fft(nx, dx, rho, pot)
                else:
                    a.tsc_poisson_forward(nx, L, dx, radx, cos["rote"], cos["rete"], *xyz, m, dep, phi, 1)
                st.synchronize()
                a.close()
            got.append([pot, dep, phi])
    torch.cuda.synchronize()
    for a, b in zip(*got):  # one plan on both streams; the deposit's float64 sums in any order
        assert float((a - b).abs().max()) <= 2.0 ** -20 * float(b.abs().max())
