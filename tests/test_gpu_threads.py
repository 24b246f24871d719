"""DENSITY from several threads at once, each with its own context, stream and
number of levels (so its own size of shared memory): every call succeeds and
gives what the same call gives alone."""
import threading

import numpy as np
import pytest
import torch

from asohf_b200 import api, grid, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("masses", ["equal", "unequal"])
def test_levels_by_thread(gpu_lib, masses):
    s = synth.generate("tiny")
    cfg = s.cfg
    _, dx = grid.malla(cfg.nx, np.float32(cfg.lado0))
    cos = grid.cosmology(cfg.h, cfg.omega_m, cfg.zeta)
    m = s.m if masses == "equal" else (s.m * np.where(np.arange(s.m.size) % 2, 1.0, 2.0)).astype(np.float32)
    full = synth.build_mesh(s, float(dx))
    levels = [0, 1, full.nl]

    class Work:
        def __init__(self, nl):
            self.mesh = synth.build_mesh(s, float(dx), nl=nl) if nl else synth.build_mesh(s, float(dx), nl=1)
            if nl > 1:  # the patches of level 1 named as the deepest level: the largest kernel table
                k = int(self.mesh.npatch[1])
                np_ = np.zeros(10, np.int32)
                np_[1], np_[9] = k - 1, 1
                self.mesh.nl, self.mesh.npatch = 9, np_
                for f in ("patchnx", "patchny", "patchnz", "patchrx", "patchry", "patchrz"):
                    setattr(self.mesh, f, getattr(self.mesh, f)[:k])
            self.stream = torch.cuda.Stream()
            self.lib = api.Asohf(0)
            self.lib.set_stream(self.stream.cuda_stream)
            self.lib.upload_particles(s.x, s.y, s.z, s.vx, s.vy, s.vz, m, s.id)
            self.npe = self.lib.sort_dm_particles_localdensity(cfg.nx, dx, cos["rodo"], cos["re0"])
            self.error = None

        def once(self):
            u1 = np.empty(cfg.nx ** 3, np.float32)
            u11 = np.empty((int(self.mesh.npatch.sum()), 32 ** 3), np.float32)
            self.lib.density(cfg.nx, np.float32(cfg.lado0), dx, cos["rote"], cos["rete"], self.npe, self.mesh, 2, u1,
                             u11)
            return u1, u11

        def loop(self, want):
            try:
                for _ in range(60):
                    for a, b in zip(self.once(), want):
                        assert np.allclose(a, b, rtol=2.0 ** -23, atol=0.0)
            except BaseException as e:  # noqa: B902 -- reported by the test
                self.error = e

    works = [Work(nl) for nl in levels]
    wants = [w.once() for w in works]
    threads = [threading.Thread(target=w.loop, args=(x,)) for w, x in zip(works, wants)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for w in works:
        w.lib.close()
        assert w.error is None, w.error
