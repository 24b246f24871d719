"""The work the framework is measured on, as calls a user's program makes.

Seven kinds of pass, each through the public entry points:

  catalogue  a snapshot to its halo catalogue: the driver's whole particle
             path (upload, species sort, deposit, x-slab sort, halo finder
             level by level, substructure, bound-particle IDs)
  density    the deposit stage alone: upload, species sort, DENSITY on the
             base grid and the AMR patches, RENORM_DENSITY
  tsc        INTERPOLATE_DENSITY_TSC of an uploaded snapshot
  mesh       the mesh builder's particle counts on the base grid and on the
             level-1 patches, and VEINSGRID_REDUCED on them
  grid       HALOFIND_GRID at the base level on a density grid
  poisson    MOMENTO + POFFT3D on device fields
  layer      the differentiable deposit + Poisson layer, forward and
             backward (the potential and every gradient)

Snapshots follow the generator's recipes: the 20, 62.5 and 100 Mpc/h
configurations and the same recipes at other particle counts.  A case fixes
its halo table (masses, so the number of patches and of candidates); the seed
turns the box, displaces every particle and shuffles their order.
"""
import dataclasses
import functools
import math

import numpy as np
import torch

from asohf_b200 import abi, api, driver, grid, synth
from asohf_b200.autograd import DepositPoissonLayer

NA = abi.NAMRX
H, OMEGA_M, FDM = 0.678, 0.31, 0.845
f32 = np.float32


def _snap(side, box, nx, nl, haloes, mlo, mhi, frac, subs, patches=4000):
    return dict(side=side, box=box, nx=nx, nl=nl, haloes=haloes, mlo=mlo, mhi=mhi, frac=frac, subs=subs,
                patches=patches)


def listed():
    return [
        # the smallest whole analysis: one 20 Mpc/h snapshot held in ordinary
        # host arrays, as the Fortran driver holds it; launches and latency
        dict(name="catalogue_64_host", kind="catalogue", host=True, drop=0,
             **_snap(64, 20.0, 64, 3, 40, 1e11, 1e13, 0.70, 0.0)),
        # an ordinary analysis: the benchmark recipe at 128^3, on the device
        dict(name="catalogue_128", kind="catalogue", host=False, drop=0,
             **_snap(128, 62.5, 128, 6, 3125, 1e10, 1e15, 0.70, 1e12)),
        # a large analysis: 256^3 particles in 100 Mpc/h, 5000 haloes with
        # subhaloes, 6 AMR levels
        dict(name="catalogue_256", kind="catalogue", host=False, drop=0,
             **_snap(256, 100.0, 256, 6, 5000, 1e10, 1e14, 0.65, 1e12)),
        # the deposit of a production snapshot: 56.6M particles, equal masses
        dict(name="density_384", kind="density", zoom=False, degree=2, drop=0,
             **_snap(384, 187.5, 384, 6, 84000, 1e10, 1e15, 0.70, 1e12)),
        # a zoom-in run: two particle masses, an odd count, the linear kernel
        dict(name="density_zoom", kind="density", zoom=True, degree=1, drop=1013,
             **_snap(112, 40.0, 96, 4, 600, 1e10, 1e14, 0.70, 1e12, 400)),
        # the TSC density of an ordinary snapshot with its patches
        dict(name="tsc_128", kind="tsc", zoom=False, drop=0,
             **_snap(128, 62.5, 128, 3, 3125, 1e10, 1e15, 0.70, 1e12, 1500)),
        # one level of mesh building on an ordinary snapshot
        dict(name="mesh_160", kind="mesh", drop=0, **_snap(160, 78.0, 160, 3, 6000, 1e10, 1e15, 0.70, 1e12, 2500)),
        # the candidates of an ordinary snapshot
        dict(name="grid_128", kind="grid", drop=0, **_snap(128, 62.5, 128, 0, 3125, 1e10, 1e15, 0.70, 1e12)),
        # one large potential
        dict(name="poisson_512", kind="poisson", nx=512, batch=1),
        # a training step on eight jittered copies of the 64^3 set
        dict(name="layer_256_b8", kind="layer", nx=256, batch=8, n_per=262144, grad_m=True),
        # ragged sets on a grid that is no power of two, positions only
        dict(name="layer_100_b3", kind="layer", nx=100, batch=3, n_per=50021, grad_m=False),
        # the smallest training step
        dict(name="layer_32", kind="layer", nx=32, batch=1, n_per=4096, grad_m=True),
    ]


FFT_SIZES = [24, 32, 40, 48, 60, 64, 75, 80, 96, 100, 120, 125, 128, 135, 144, 150, 160, 180, 192, 200, 216, 225,
             240, 243, 250, 256, 288, 300, 320, 360, 384, 400, 432, 448, 480, 500, 512]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _recipe(rng, side, patches=4000):
    """A snapshot of `side`^3 particles at the recipes' mean density."""
    nx = side if rng.random() < 0.6 else max(24, int(side * rng.uniform(0.5, 1.0)))
    haloes = max(6, int(side ** 3 / _log_int(rng, 700, 6000)))
    return _snap(side, round(side * rng.uniform(0.31, 0.49), 2), nx, rng.randint(1, 6), haloes, 1e10,
                 rng.choice([1e13, 1e14, 1e15]), round(rng.uniform(0.55, 0.75), 3), rng.choice([0.0, 1e12]), patches)


def draw(rng):
    kind = rng.choice(["catalogue", "catalogue", "density", "density", "tsc", "mesh", "grid", "poisson", "layer",
                       "layer"])
    if kind == "catalogue":
        side = _log_int(rng, 40, 200)
        return dict(kind=kind, host=side < 100 and rng.random() < 0.5, drop=rng.choice([0, rng.randint(1, 999)]),
                    **_recipe(rng, side))
    if kind == "density":
        zoom = rng.random() < 0.4
        side = _log_int(rng, 40, 140 if zoom else 320)
        return dict(kind=kind, zoom=zoom, degree=rng.choice([1, 2]), drop=rng.randint(0, 999),
                    **_recipe(rng, side, 600 if zoom else 3000))
    if kind == "tsc":
        return dict(kind=kind, zoom=rng.random() < 0.4, drop=rng.randint(0, 999),
                    **_recipe(rng, _log_int(rng, 40, 160), 1000))
    if kind == "mesh":
        return dict(kind=kind, drop=rng.randint(0, 999), **_recipe(rng, _log_int(rng, 48, 192), 3000))
    if kind == "grid":
        return dict(kind=kind, drop=rng.randint(0, 999), **dict(_recipe(rng, _log_int(rng, 40, 160)), nl=0))
    nx = rng.choice(FFT_SIZES if kind == "poisson" else [s for s in FFT_SIZES if s <= 256])
    most = (512 ** 3 if kind == "poisson" else 8 * 256 ** 3) // nx ** 3
    batch = min(rng.randint(1, 8), most)
    if kind == "poisson":
        return dict(kind=kind, nx=nx, batch=batch)
    return dict(kind=kind, nx=nx, batch=batch, n_per=_log_int(rng, 1000, 262144), grad_m=rng.random() < 0.5)


# ------------------------------------------------------------- inputs

def _config(case):
    return synth.SnapshotConfig("case", case["side"], case["box"], case["nx"], case["nl"], case["haloes"],
                                case["mlo"], case["mhi"], case["frac"], sub_host_min=case["subs"],
                                h=H, omega_m=OMEGA_M, fdm=FDM, max_patches_per_level=case["patches"])


def _snapshot(case, seed):
    """The snapshot on the device: axes permuted and mirrored, particles
    displaced by a twentieth of their mean spacing and shuffled, by the seed;
    `drop` particles fewer than side^3, and with `zoom` the particles outside
    a central sphere eight times heavier."""
    s = synth.generate_fast(_config(case), device="cuda", keep_on_device=True)
    rng = np.random.Generator(np.random.PCG64(int(seed)))
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    axes, signs = rng.permutation(3), rng.choice([-1.0, 1.0], 3)
    L, n = s.cfg.lado0, s.x.shape[0] - case.get("drop", 0)
    half = float(f32(L / 2))
    order = torch.randperm(s.x.shape[0], generator=g, device="cuda")[:n]
    pos, vel = [s.x, s.y, s.z], [s.vx, s.vy, s.vz]
    x, v = [], []
    for a, sign in zip(axes, signs):
        p = pos[a][order] * float(sign) + torch.randn(n, generator=g, device="cuda") * (0.05 * L / case["side"])
        p = torch.where(p >= half, p - 2 * half, p)
        x.append(torch.clamp(torch.where(p < -half, p + 2 * half, p), -half, half))
        x[-1][x[-1] >= half] = -half  # rounded up to the upper face
        v.append(vel[a][order] * float(sign))
    m = s.m[order]
    if case.get("zoom"):
        r = 0.3 * L
        m = torch.where(x[0] * x[0] + x[1] * x[1] + x[2] * x[2] > r * r, m * 8.0, m)
    return dataclasses.replace(s, x=x[0], y=x[1], z=x[2], vx=v[0], vy=v[1], vz=v[2], m=m,
                               id=torch.arange(1, n + 1, dtype=torch.int32, device="cuda"),
                               halo_pos=np.ascontiguousarray(s.halo_pos[:, axes] * signs))


def _field(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    return torch.randn((case["batch"], case["nx"], case["nx"], case["nx"]), generator=g, device="cuda")


def _layer_inputs(case, seed):
    """Positions (copies jittered by 0.01 cell), masses, and dL/dpot."""
    nx, batch, n = case["nx"], case["batch"], case["n_per"]
    side = 1
    while side ** 3 < n:
        side += 1
    c = _snap(side, 20.0, 64, 3, max(2, side ** 3 // 6500), 1e11, 1e13, 0.70, 0.0)
    s = _snapshot(c, seed)
    L = s.cfg.lado0
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
    pos = torch.stack([s.x[:n], s.y[:n], s.z[:n]])[:, None, :].double()
    pos = pos + torch.randn((3, batch, n), generator=g, device="cuda", dtype=torch.float64) * (0.01 * L / nx)
    pos = (torch.remainder(pos + L / 2, L) - L / 2).float()
    m = s.m[:n][None, :].repeat(batch, 1) * (0.5 + torch.rand((batch, n), generator=g, device="cuda"))
    return L, pos[0].contiguous(), pos[1].contiguous(), pos[2].contiguous(), m.contiguous(), _field(case, seed)


def _level1(mesh):
    n = int(mesh.npatch[1]) if mesh.nl >= 1 else 0
    return [a[:n] for a in (mesh.patchnx, mesh.patchny, mesh.patchnz, mesh.patchrx, mesh.patchry, mesh.patchrz)]


def _geometry(case):
    cfg = _config(case)
    radx, dx = grid.malla(cfg.nx, cfg.lado0)
    return cfg, radx, dx, grid.cosmology(cfg.h, cfg.omega_m, cfg.zeta)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "poisson":
        _, dx = grid.malla(case["nx"], f32(20.0 / H))
        rho = _field(case, seed)
        return dict(case=case, lib=api.Asohf(), dx=dx, rho=rho, pot=torch.empty_like(rho))
    if kind == "layer":
        L, x, y, z, m, w = _layer_inputs(case, seed)
        wanted = [a.requires_grad_() for a in ([x, y, z, m] if case["grad_m"] else [x, y, z])]
        return dict(case=case, layer=DepositPoissonLayer(case["nx"], L), args=(x, y, z, m), wanted=wanted, w=w)
    snap = _snapshot(case, seed)
    cfg, radx, dx, cos = _geometry(case)
    st = dict(case=case, cfg=cfg, radx=radx, dx=dx, cos=cos, snap=snap)
    if kind == "catalogue":
        if case["host"]:
            for f in ("x", "y", "z", "vx", "vy", "vz", "m", "id"):
                setattr(snap, f, getattr(snap, f).cpu().numpy())
        st["plan"] = driver.prepare(snap)
        st["ids"] = torch.zeros(snap.x.shape[0], dtype=torch.int32, device="cpu" if case["host"] else "cuda")
        st["backend"] = api.GpuBackend() if case["host"] else api.DeviceBackend()
        return st
    if kind == "density":
        st["mesh"] = synth.build_mesh(snap, float(dx))
        st["backend"] = api.DeviceBackend()
        return st
    lib = st["lib"] = api.Asohf()
    lib.upload_particles(snap.x, snap.y, snap.z, snap.vx, snap.vy, snap.vz, snap.m, snap.id)
    st["npe"] = lib.sort_dm_particles_localdensity(cfg.nx, dx, cos["rodo"], cos["re0"])
    if kind == "tsc":
        mesh = st["mesh"] = synth.build_mesh(snap, float(dx))
        st["u1"] = torch.empty(cfg.nx ** 3, device="cuda")
        st["u11"] = torch.empty((max(mesh.total, 1), NA ** 3), device="cuda")
    elif kind == "mesh":
        st["patches"] = _level1(synth.build_mesh(snap, float(dx), nl=1))
        n = st["patches"][0].shape[0]
        st["cr0"] = torch.empty(cfg.nx ** 3, dtype=torch.int32, device="cuda")
        st["cr01"] = torch.empty((n, NA ** 3), dtype=torch.int32, device="cuda")
    else:
        empty = synth.build_mesh(snap, float(dx), nl=0)
        u1 = st["u1"] = torch.empty(cfg.nx ** 3, device="cuda")
        lib.density(cfg.nx, f32(cfg.lado0), dx, cos["rote"], cos["rete"], st["npe"], empty, 2, u1, None)
        lib.renorm_density(cfg.nx, empty, f32(cfg.fdm), u1, None)
        st["cat"] = abi.Catalogue(cfg.nx ** 3 // 64 + 1024)
    torch.cuda.synchronize()
    return st


# ------------------------------------------------------------- the passes

CATALOGUE = (abi.CAT_SCALAR_FLOAT + abi.CAT_SCALAR_INT + list(abi.CAT_MULTI))
GRID_COLUMNS = ["realclus", "levhal", "patchclus", "clusrx", "clusry", "clusrz", "radio", "masa", "clusrxcm",
                "clusrycm", "clusrzcm"]


def run(st):
    kind = st["case"]["kind"]
    if kind == "poisson":
        st["lib"].poisson_fft(st["case"]["nx"], st["dx"], st["rho"], st["pot"], st["case"]["batch"])
        return st["pot"]
    if kind == "layer":
        pot = st["layer"](*st["args"])
        return [pot.detach(), *torch.autograd.grad(pot, st["wanted"], st["w"])]
    cfg, dx, cos = st["cfg"], st["dx"], st["cos"]
    nx, lado0 = cfg.nx, f32(cfg.lado0)
    if kind == "catalogue":
        s = st["snap"]
        r = driver.execute(st["plan"], st["backend"], with_subs=cfg.sub_host_min > 0, particles=s, download=False)
        # the program's own PARTICLES_PER_HALO, one entry per particle
        ids = st["ids"]
        ids[:r.pph.shape[0]] = torch.from_numpy(r.pph) if st["case"]["host"] else r.pph
        out = {f: getattr(r.cat, f) for f in CATALOGUE}
        out.update(nclus=r.cat.nclus, species=r.npart_esp, slabs=r.ndmpart_x, ids=ids, u1=r.u1,
                   u11=r.u11.reshape(-1)[:r.mesh.total * NA ** 3], nhallev=r.nhallev, subs_lev=r.subs_lev)
        return out
    if kind == "density":
        s, b = st["snap"], st["backend"]
        b.upload(s)
        npe = b.species_sort(nx, dx, cos["rodo"], cos["re0"])
        u1, u11 = b.density_renorm(nx, lado0, dx, cos["rote"], cos["rete"], npe, st["mesh"], st["case"]["degree"],
                                   f32(cfg.fdm))
        b.sync_outputs()
        return dict(species=npe, u1=u1, u11=u11[:st["mesh"].total * NA ** 3])
    lib = st["lib"]
    if kind == "tsc":
        lib.interpolate_density_tsc(nx, lado0, dx, st["radx"], cos["rote"], cos["rete"], st["mesh"], st["u1"],
                                    st["u11"])
        return dict(u1=st["u1"], u11=st["u11"][:st["mesh"].total])
    if kind == "mesh":
        p = st["patches"]
        cr0 = lib.mesh_base_counts(nx, dx, 8, 1, st["npe"], st["cr0"])
        cr01 = lib.mesh_patch_counts(nx, lado0, dx, 1, 8, 1, st["npe"], *p, out=st["cr01"])
        lib.veinsgrid_reduced(1, dx, st["radx"][1], *p, p[0].shape[0], cr01)
        return dict(cr0=cr0, cr01=cr01)
    n = lib.halofind_grid_base(nx, dx, st["u1"], st["radx"], cos["contrastec"], cos["rote"], cos["rete"],
                               cos["rodo"], cos["re0"], f32(cfg.lado0 / 4), 0.2, st["cat"])
    return dict({f: getattr(st["cat"], f) for f in GRID_COLUMNS}, nhal=n)


# ------------------------------------------------------------- the least work

@functools.lru_cache(maxsize=64)
def _patches(nl, items):
    """Patches of the recipe, from the halo table."""
    case = dict(items)
    cfg = _config(case)
    t = synth._halo_table(cfg, np.random.Generator(np.random.PCG64(cfg.seed)))
    return sum(min(int((t["npart"] >= 64 * 4 ** (ir - 1)).sum()), cfg.max_patches_per_level)
               for ir in range(1, nl + 1))


def _count_patches(case, nl):
    keys = ("side", "box", "nx", "nl", "haloes", "mlo", "mhi", "frac", "subs", "patches")
    return _patches(nl, tuple((k, case[k]) for k in keys))


def work(case):
    """Bytes: particles and fields in once, grids, lists and gradients out
    once.  Flops: the cloud and weight products and the transforms."""
    kind, nx = case["kind"], case["nx"]
    if kind in ("poisson", "layer"):
        g = case["batch"] * nx ** 3
        fft = 2 * 2.5 * g * math.log2(float(nx) ** 3)
        if kind == "poisson":
            return {"bytes": 8 * g, "flops": fft}
        n = case["batch"] * case["n_per"]
        return {"bytes": 16 * n + 8 * g + (16 if case["grad_m"] else 12) * n, "flops": 2 * fft + 27 * 14 * n}
    n, g = case["side"] ** 3 - case["drop"], nx ** 3
    if kind == "catalogue":
        cells = _count_patches(case, case["nl"]) * NA ** 3
        return {"bytes": 32 * n + 4 * g + 4 * cells + int(4 * case["frac"] * n), "flops": 27 * 3 * n + 20 * n}
    if kind == "density":
        return {"bytes": 16 * n + 4 * g + 4 * _count_patches(case, case["nl"]) * NA ** 3, "flops": 27 * 3 * n}
    if kind == "tsc":
        return {"bytes": 16 * n + 4 * g + 4 * _count_patches(case, case["nl"]) * NA ** 3, "flops": 27 * 4 * n}
    if kind == "mesh":
        return {"bytes": 12 * n + 4 * g + 4 * _count_patches(case, 1) * NA ** 3, "flops": 6 * n}
    return {"bytes": 4 * g, "flops": g}


# ------------------------------------------------------------- 64-bit values

D = torch.float64


def _malla32(nx, lado0):
    """RADX(0:NX+1) and DX in the driver's single precision."""
    lado = f32(f32(lado0) - f32(f32(lado0) / f32(nx)))
    a, b = f32(-lado / f32(2)), f32(lado / f32(2))
    c = f32(f32(b - a) / f32(nx - 1))
    r = np.zeros(nx + 2, f32)
    r[1:nx + 1] = a + np.arange(nx, dtype=f32) * c
    r[1] = a
    r[0], r[nx + 1] = f32(r[1] - c), f32(r[nx] + c)
    return r, f32(r[2] - r[1])


def _background32():
    ache = f32(float(f32(H)) * 3.66e-3)
    rodo = f32(float(f32(OMEGA_M)) * 3.0 * float(f32(ache * ache)))
    return rodo, f32(f32(1) / f32(10.98))  # RODO = ROTE and RE0 = RETE at redshift 0


def _cells32(v, low, d):
    """(v-low)/d of single-precision positions, correctly rounded (a division
    by a host scalar would be a product with its reciprocal)."""
    return (v - float(low)) / torch.tensor(float(d), dtype=torch.float32, device=v.device)


def _cell32(v, xl, d, nx):
    """INT((v-xl)/d)+1, clamped to the grid."""
    return torch.clamp(_cells32(v, xl, d).to(torch.int64) + 1, 1, nx)


def _tsc64(v, rm, r0, rp, d):
    """TSC weights and their derivatives, 64 bits."""
    v = v.double()
    a, b, c = v - rm, v - r0, v - rp
    ta, tc = 1.5 - a.abs() / d, 1.5 - c.abs() / d
    w = [0.5 * ta * ta, 0.75 - (b / d) ** 2, 0.5 * tc * tc]
    sign = lambda t: torch.copysign(torch.ones_like(t), t)
    return w, [-ta * sign(a) / d, -2 * b / (d * d), -tc * sign(c) / d]


def _tsc_base_parts(x, y, z, nx, lado0, radx, dx):
    xl = -f32(lado0) / f32(2)
    r = torch.from_numpy(radx.astype(np.float64)).to(x.device)
    cells, ws, dws = [], [], []
    for v in (x, y, z):
        i = _cell32(v, float(xl), float(dx), nx)
        w, dw = _tsc64(v, r[i - 1], r[i], r[i + 1], float(dx))
        cells.append([(i - 1 + o) % nx for o in (-1, 0, 1)])
        ws.append(w)
        dws.append(dw)
    return cells, ws, dws


def _tsc_base64(x, y, z, m, nx, lado0, radx, dx):
    cells, ws, _ = _tsc_base_parts(x, y, z, nx, lado0, radx, dx)
    out = torch.zeros(nx ** 3, dtype=D, device=x.device)
    for k in range(3):
        for j in range(3):
            for i in range(3):
                c = (cells[2][k] * nx + cells[1][j]) * nx + cells[0][i]
                out.index_add_(0, c, m.double() * ws[0][i] * ws[1][j] * ws[2][k])
    return out


def _green64(rho, nx, dx):
    """The periodic solve of POFFT3D of one (nx, nx, nx) field."""
    k = torch.arange(nx, dtype=D, device=rho.device)
    s2 = torch.sin(math.pi * k / nx) ** 2
    den = s2[:, None, None] + s2[None, :, None] + s2[None, None, :nx // 2 + 1]
    den[0, 0, 0] = 1e30
    return torch.fft.irfftn(torch.fft.rfftn(rho) * (-(float(dx) / 2) ** 2 / den), s=(nx, nx, nx))


def _exact_layer(case, seed):
    nx = case["nx"]
    L, x, y, z, m, w = _layer_inputs(case, seed)
    radx, dx = _malla32(nx, L)
    rote, rete = (float(v) for v in _background32())
    den = float(dx) ** 3 * rote * rete ** 3
    pot = torch.empty_like(w, dtype=D)
    grads = [torch.empty_like(x, dtype=D) for _ in range(4)]
    for b in range(case["batch"]):
        rho = _tsc_base64(x[b], y[b], z[b], m[b], nx, L, radx, dx).reshape(nx, nx, nx) / den
        pot[b] = _green64(rho, nx, dx)
        g = _green64(w[b].double(), nx, dx).reshape(-1)
        cells, ws, dws = _tsc_base_parts(x[b], y[b], z[b], nx, L, radx, dx)
        acc = [torch.zeros_like(x[b], dtype=D) for _ in range(4)]
        for k in range(3):
            for j in range(3):
                for i in range(3):
                    gv = g[(cells[2][k] * nx + cells[1][j]) * nx + cells[0][i]]
                    acc[0] += dws[0][i] * ws[1][j] * ws[2][k] * gv
                    acc[1] += ws[0][i] * dws[1][j] * ws[2][k] * gv
                    acc[2] += ws[0][i] * ws[1][j] * dws[2][k] * gv
                    acc[3] += ws[0][i] * ws[1][j] * ws[2][k] * gv
        for a in range(3):
            grads[a][b] = acc[a] * m[b].double() / den
        grads[3][b] = acc[3] / den
    return [pot, *grads[:4 if case["grad_m"] else 3]]


def _kernel64(level, degree):
    """COMPUTE_KERNELS in 64 bits: 2*2^level+1 weights of unit sum."""
    n = 1 << level
    i = np.abs(np.arange(-n, n + 1, dtype=np.float64))
    if degree == 2:
        b = i / (2.0 * (n + 0.5) / 3.0)
        k = np.where(b <= 0.5, 0.75 - b * b, 0.5 * (1.5 - b) ** 2)
    else:
        k = 1.0 - i / (n + 0.5)
    return k / k.sum()


def _species(x, y, z, m, nx, dx):
    """SORT_DM_PARTICLES_LOCALDENSITY: the cell's single-precision mass sum in
    input order, and the integer level of its density."""
    rodo, re0 = _background32()
    xmin = float(-(f32(nx) * dx) / f32(2))
    c = (_cell32(z, xmin, float(dx), nx) - 1) * nx + (_cell32(y, xmin, float(dx), nx) - 1)
    c = c * nx + (_cell32(x, xmin, float(dx), nx) - 1)
    order = torch.argsort(c, stable=True)
    cs, ms = c[order], m[order]
    count = torch.bincount(c, minlength=nx ** 3)
    start = torch.cumsum(count, 0) - count
    rank = torch.arange(c.shape[0], device=c.device) - start[cs]
    by_rank = torch.argsort(rank, stable=True)
    at = torch.cumsum(torch.bincount(rank), 0).tolist()
    dens = torch.zeros(nx ** 3, dtype=torch.float32, device=x.device)
    lo = 0
    for hi in at:  # the q-th particle of every cell that has one
        sel = by_rank[lo:hi]
        dens[cs[sel]] += ms[sel]
        lo = hi
    bas = f32(f32(f32(dx * dx) * dx) * rodo) * f32(f32(re0 * re0) * re0)
    lg = torch.log(_cells32(dens, 0.0, bas).double()).float()
    lg = _cells32(lg, 0.0, f32(math.log(8.0)))
    s = torch.clamp(torch.nan_to_num(lg, neginf=0.0), 0, abi.N_ESP - 1).to(torch.int64)
    return s[c]


def _toeplitz(n, level, degree, device):
    nk = 1 << level
    t = torch.zeros((n, n + 2 * nk), dtype=D, device=device)
    k = torch.from_numpy(_kernel64(level, degree)).to(device)
    for i in range(n):
        t[i, i:i + 2 * nk + 1] = k
    return t


def _exact_density(case, seed):
    snap = _snapshot(case, seed)
    cfg = snap.cfg
    nx, nl, degree, dev = cfg.nx, cfg.nl, case["degree"], snap.x.device
    radx, dx = _malla32(nx, cfg.lado0)
    rote, rete = (float(v) for v in _background32())
    spec = _species(snap.x, snap.y, snap.z, snap.m, nx, dx)
    species = torch.bincount(spec, minlength=abi.N_ESP)
    xl = float(-f32(cfg.lado0) / f32(2))
    host = [_cells32(v, xl, dx).to(torch.int64) % nx for v in (snap.x, snap.y, snap.z)]
    u1 = torch.zeros(nx ** 3, dtype=D, device=dev)
    u1.index_add_(0, (host[2] * nx + host[1]) * nx + host[0], snap.m.double())
    u1 = u1.reshape(nx, nx, nx)
    k0 = _kernel64(0, degree)
    for a in range(3):
        u1 = float(k0[1]) * u1 + float(k0[0]) * (torch.roll(u1, 1, a) + torch.roll(u1, -1, a))
    fdm = float(f32(FDM))
    out = {"species": species, "u1": (u1 / (float(dx) ** 3 * rote * rete ** 3) / fdm).reshape(-1), "u11": None}
    mesh = synth.build_mesh(snap, float(dx))
    if mesh.total > 2000:
        return out
    order = torch.argsort(snap.x)
    x, y, z, m, spec = (v[order] for v in (snap.x, snap.y, snap.z, snap.m, spec))
    level = np.repeat(np.arange(nl + 1), mesh.npatch)
    u11 = torch.zeros((mesh.total, NA, NA, NA), dtype=D, device=dev)
    for q in range(mesh.total):
        ir = int(level[q])
        dxpa = f32(dx / f32(2.0 ** ir))
        n = [int(a[q]) for a in (mesh.patchnx, mesh.patchny, mesh.patchnz)]
        low = [f32(a[q] - dxpa) for a in (mesh.patchrx, mesh.patchry, mesh.patchrz)]
        lo = [float(f32(v - dx)) for v in low]
        hi = [float(f32(f32(v + f32(f32(c) * dxpa)) + dx)) for v, c in zip(low, n)]
        a, b = (int(v) for v in torch.searchsorted(x, torch.tensor([lo[0], hi[0]], device=dev)))
        p = [v[a:b] for v in (x, y, z)]
        sel = torch.ones(b - a, dtype=torch.bool, device=dev)
        for v, l, h in zip(p, lo, hi):
            sel &= (v > l) & (v < h)
        at = sel.nonzero()[:, 0]
        cell = [torch.floor(_cells32(v[at], l, dxpa)).to(torch.int64) for v, l in zip(p, low)]
        mm = m[a:b][at].double()
        lev = torch.clamp(ir - spec[a:b][at], min=0)
        for l in torch.unique(lev).tolist():
            nk = 1 << l
            ext = [c + 2 * nk for c in n]
            ok = lev == l
            for c, e in zip(cell, ext):
                ok &= (c + nk >= 0) & (c + nk < e)
            cc = [c[ok] + nk for c in cell]
            hosts = torch.zeros(ext[0] * ext[1] * ext[2], dtype=D, device=dev)
            hosts.index_add_(0, (cc[2] * ext[1] + cc[1]) * ext[0] + cc[0], mm[ok])
            t = hosts.reshape(ext[2], ext[1], ext[0])
            t = torch.einsum("kji,ai->kja", t, _toeplitz(n[0], l, degree, dev))
            t = torch.einsum("kja,bj->kba", t, _toeplitz(n[1], l, degree, dev))
            u11[q, :n[2], :n[1], :n[0]] += torch.einsum("kba,ck->cba", t, _toeplitz(n[2], l, degree, dev))
        u11[q] /= float(dxpa) ** 3 * rote * rete ** 3 * fdm
    out["u11"] = u11.reshape(-1)
    return out


def _exact_tsc(case, seed):
    snap = _snapshot(case, seed)
    cfg = snap.cfg
    nx, dev = cfg.nx, snap.x.device
    radx, dx = _malla32(nx, cfg.lado0)
    rote, rete = (float(v) for v in _background32())
    order = torch.argsort(snap.x)
    x, y, z, m = (v[order] for v in (snap.x, snap.y, snap.z, snap.m))
    u1 = _tsc_base64(x, y, z, m, nx, cfg.lado0, radx, dx) / (float(dx) ** 3 * rote * rete ** 3)
    mesh = synth.build_mesh(snap, float(dx))
    level = np.repeat(np.arange(cfg.nl + 1), mesh.npatch)
    plev = torch.zeros(x.shape[0], dtype=torch.int64, device=dev)
    inside = []
    for q in range(mesh.total):  # the particles of each patch within its one-cell buffer
        dxpa = f32(dx / f32(2.0 ** int(level[q])))
        n = [int(a[q]) for a in (mesh.patchnx, mesh.patchny, mesh.patchnz)]
        lo = [f32(a[q] - f32(f32(2) * dxpa)) for a in (mesh.patchrx, mesh.patchry, mesh.patchrz)]
        hi = [f32(v + f32(f32(c + 2) * dxpa)) for v, c in zip(lo, n)]
        a, b = (int(v) for v in torch.searchsorted(x, torch.tensor([float(lo[0]), float(hi[0])], device=dev)))
        sel = torch.ones(b - a, dtype=torch.bool, device=dev)
        for v, l, h in zip((x[a:b], y[a:b], z[a:b]), lo, hi):
            sel &= (v > float(l)) & (v < float(h))
        at = sel.nonzero()[:, 0] + a
        plev[at] = torch.clamp(plev[at], min=int(level[q]))
        inside.append((at, dxpa, n, lo))
    u11 = torch.zeros((mesh.total, NA ** 3), dtype=D, device=dev)
    for q, (at, dxpa, n, lo) in enumerate(inside):
        at = at[plev[at] >= int(level[q])]
        cells, ws = [], []
        for v, l, r in zip((x, y, z), lo, (mesh.patchrx[q], mesh.patchry[q], mesh.patchrz[q])):
            i = _cells32(v[at], l, dxpa).to(torch.int64)
            c = [float(r) + (i.double() + o - 1.5) * float(dxpa) for o in (-1, 0, 1)]
            w, _ = _tsc64(v[at], *c, float(dxpa))
            cells.append([i + o - 1 for o in (-1, 0, 1)])
            ws.append(w)
        mm = m[at].double()
        for k in range(3):
            for j in range(3):
                for i in range(3):
                    ok = torch.ones(at.shape[0], dtype=torch.bool, device=dev)
                    for c, e in zip((cells[0][i], cells[1][j], cells[2][k]), n):
                        ok &= (c >= 0) & (c < e)
                    c = (cells[2][k] * NA + cells[1][j]) * NA + cells[0][i]
                    u11[q].index_add_(0, c[ok], (mm * ws[0][i] * ws[1][j] * ws[2][k])[ok])
        u11[q] /= float(dxpa) ** 3 * rote * rete ** 3
    return dict(u1=u1, u11=u11)


def exact(case, seed):
    """64-bit values of the deposits, potentials and gradients.  None for the
    catalogues (their numbers follow from the reference's single-precision
    decisions) and for whole-number grids; the patch deposit of very large
    tables is left out for its time."""
    kind = case["kind"]
    if kind == "poisson":
        _, dx = _malla32(case["nx"], f32(20.0 / H))
        rho = _field(case, seed)
        return torch.stack([_green64(r.double(), case["nx"], dx) for r in rho])
    if kind == "layer":
        return _exact_layer(case, seed)
    if kind == "density":
        return _exact_density(case, seed)
    if kind == "tsc":
        return _exact_tsc(case, seed)
    return None
