"""Performance cases: what a user of the library has it do, through its public entry points.

A case is one model and one kind of run:

* ``forward``: a batch of time steps of an elastic shot (ElasticSolver.run) followed by a field snapshot, as a
  run with snapshots does it; isotropic, anisotropic or 3-SLS viscoelastic, Newmark or LDDRK, flat or under
  topography, Stacey edges.
* ``ocean``: the same for a fluid-solid model (CoupledSolver) with CPML layers or Stacey edges.
* ``gradient``: one misfit gradient (FWIGradient: forward, adjoint sweep, kernels), of one model or of several
  models packed into one mesh.
* ``ocean_gradient``: the kernel run of a fluid-solid model (CoupledKernels).
* ``smooth``: Gaussian smoothing of sensitivity kernels.

Models are synthetic: 25 m quads, vp rising with depth with a 5 % random perturbation per GLL point.  A case's
model is fixed; the seed draws the shot (amplitudes, time function), the wavefield the run starts from and the
observed data, which is what changes between calls on one model.  `exact` restates the schemes in float64 torch.
"""
import copy
import math

import numpy as np
import torch

from specfem2d_b200 import batch
from specfem2d_b200.configs import gaussian_random_field
from specfem2d_b200.coupled import CoupledKernels, CoupledSolver
from specfem2d_b200.fwi import FWIGradient
from specfem2d_b200.runtime import ElasticSolver, smooth
from specfem2d_b200.setup.gll import GLL
from specfem2d_b200.setup.mesh import _interp_nodes, _shape_tables, internal_mesh
from specfem2d_b200.setup.solver_setup import ALPHA_LDDRK, BETA_LDDRK, Source, build_database

DX = 25.0


def listed():
    return [
        # a small 2-D shot (the 80 x 60 homogeneous example): launch and latency bound
        dict(name="shot_80x60", kind="forward", nx=80, nz=60, steps=200, nrec=20, topo=False, physics="iso",
             scheme=1),
        # an ordinary shot under topography, sizes that divide nothing
        dict(name="shot_topo_233x147", kind="forward", nx=233, nz=147, steps=200, nrec=31, topo=True, physics="iso",
             scheme=1),
        # the largest elastic shot: the 1000 x 400 model of the survey gradient
        dict(name="shot_1000x400", kind="forward", nx=1000, nz=400, steps=100, nrec=200, topo=False, physics="iso",
             scheme=1),
        # a homogeneous anisotropic body in an isotropic background
        dict(name="aniso_301x199", kind="forward", nx=301, nz=199, steps=100, nrec=40, topo=False, physics="aniso",
             scheme=1),
        # the viscoelastic model under topography at half scale, layered Q
        dict(name="visco_800x400", kind="forward", nx=800, nz=400, steps=60, nrec=100, topo=True, physics="visco",
             scheme=1),
        # the same physics with the low-storage Runge-Kutta scheme
        dict(name="visco_lddrk_301x150", kind="forward", nx=301, nz=150, steps=12, nrec=50, topo=True,
             physics="visco", scheme=2),
        # the marine model: water over rock, CPML sides and bottom
        dict(name="ocean_cpml_400x160", kind="ocean", nx=400, nz=160, steps=100, nrec=200, cpml=10),
        # a small marine model with absorbing edges
        dict(name="ocean_stacey_121x67", kind="ocean", nx=121, nz=67, steps=200, nrec=40, cpml=0),
        # one misfit gradient of a survey model
        dict(name="gradient_400x160", kind="gradient", nx=400, nz=160, members=1, steps=120, checkpoint_every=40,
             nrec=100, physics="iso"),
        # independent small models packed into one launch per step
        dict(name="gradient_batch_6", kind="gradient", nx=97, nz=49, members=6, steps=120, checkpoint_every=40,
             nrec=20, physics="iso"),
        # the kernel run of a marine model
        dict(name="ocean_gradient_250x100", kind="ocean_gradient", nx=250, nz=100, steps=100, checkpoint_every=50,
             nrec=60),
        # smoothing of the three kernels of a gradient
        dict(name="smooth_200x80", kind="smooth", nx=200, nz=80, nfields=3, sigma_h=100.0, sigma_v=60.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi, aspect=(0.35, 0.75)):
    nspec = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    nx = max(8, int(round(math.sqrt(nspec / rng.uniform(*aspect)))))
    return nx, max(8, int(round(nspec / nx)))


def draw(rng):
    kind = rng.choice(["forward", "forward", "forward", "ocean", "gradient", "gradient", "ocean_gradient", "smooth"])
    if kind == "forward":
        physics, scheme = rng.choice([("iso", 1), ("iso", 1), ("aniso", 1), ("visco", 1), ("visco", 2)])
        nx, nz = _grid(rng, 3e3, {("iso", 1): 3e5, ("aniso", 1): 6e4, ("visco", 1): 2e5, ("visco", 2): 4e4}[physics, scheme])
        return dict(kind=kind, nx=nx, nz=nz, steps=rng.randint(40, 100) if scheme == 1 else rng.randint(6, 12),
                    nrec=rng.randint(5, 100), topo=rng.random() < 0.5, physics=physics, scheme=scheme)
    if kind == "ocean":
        nx, nz = _grid(rng, 5e3, 6e4)
        return dict(kind=kind, nx=max(nx, 40), nz=max(nz, 40), steps=rng.randint(40, 100), nrec=rng.randint(5, 100),
                    cpml=rng.choice([0, 5, 8, 10]))
    if kind == "gradient":
        members = rng.choice([1, 1, 3, 5])
        nx, nz = _grid(rng, 2e3, 6e4 / members)
        steps = rng.randint(40, 100)
        return dict(kind=kind, nx=nx, nz=nz, members=members, steps=steps, checkpoint_every=rng.randint(15, steps),
                    nrec=rng.randint(5, 60), physics=rng.choice(["iso", "iso", "visco"]))
    if kind == "ocean_gradient":
        nx, nz = _grid(rng, 3e3, 2.5e4)
        steps = rng.randint(40, 90)
        return dict(kind=kind, nx=max(nx, 30), nz=max(nz, 30), steps=steps, checkpoint_every=rng.randint(15, steps),
                    nrec=rng.randint(5, 60))
    nx, nz = _grid(rng, 1e3, 1.5e4)
    return dict(kind=kind, nx=nx, nz=nz, nfields=rng.randint(1, 4), sigma_h=round(rng.uniform(50.0, 120.0), 1),
                sigma_v=round(rng.uniform(40.0, 90.0), 1))


# ---- models

_MODELS = {}


def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k not in ("name",)))


def _cached(key, build):
    """The model of a case, built once: several shots run on it."""
    if key not in _MODELS:
        while len(_MODELS) >= 2:
            _MODELS.pop(next(iter(_MODELS)))
        _MODELS[key] = build()
    return _MODELS[key]


def _perturbation(x, z, xmax, zmax, seed):
    gx, gz, f = gaussian_random_field(xmax, zmax, 200.0, seed=seed, spacing=50.0)
    h = gx[1] - gx[0]
    ix = np.clip((x / h).astype(np.int64), 0, len(gx) - 2)
    iz = np.clip((z / h).astype(np.int64), 0, len(gz) - 2)
    tx, tz = np.clip(x / h - ix, 0.0, 1.0), np.clip(z / h - iz, 0.0, 1.0)
    return ((1 - tx) * (1 - tz) * f[iz, ix] + tx * (1 - tz) * f[iz, ix + 1]
            + (1 - tx) * tz * f[iz + 1, ix] + tx * tz * f[iz + 1, ix + 1])


def _solid_model(nx, nz, nstep, nrec, topo, physics, scheme, seed=1, nsrc=1):
    xmax, zmax = nx * DX, nz * DX
    interfaces = [([0.0, xmax], [0.0, 0.0]), ([0.0, xmax], [zmax, zmax])]

    def top(x):
        return zmax + (0.02 * zmax * math.sin(2.0 * math.pi * x / (0.4 * xmax)) if topo else 0.0)

    mesh = internal_mesh(0.0, xmax, nx, interfaces, [nz], absorb=(True, True, False, True),
                         topography_fn=top if topo else None)
    sh, _, _ = _shape_tables(GLL(), mesh.ngnod)
    x, z = _interp_nodes(mesh, sh)
    depth = np.clip(zmax - z, 0.0, zmax)
    vp = (2500.0 + 2000.0 * depth / zmax) * (1.0 + 0.05 * _perturbation(x, z, xmax, zmax, seed))
    vs = vp / 1.73
    rho = 310.0 * vp ** 0.25
    q = {}
    if physics == "visco":
        # three layers of constant Q, as material tables define it
        layer = np.minimum(2, (3.0 * depth.mean(axis=(1, 2)) / zmax).astype(int))[:, None, None]
        q = dict(qkappa=np.choose(layer, [120.0, 200.0, 400.0]) + 0.0 * vp,
                 qmu=np.choose(layer, [50.0, 60.0, 150.0]) + 0.0 * vp)
    src = Source(x=0.47 * xmax, z=0.8 * zmax, source_type=2, f0=8.0, Mxx=0.6, Mzz=-0.4, Mxz=0.3, factor=1.0e12)
    if physics == "iso":
        src = Source(x=0.47 * xmax, z=0.8 * zmax, f0=8.0, anglesource_deg=30.0, factor=1.0e10)
    srcs, recs = [src], [(float(xr), top(float(xr)) - 0.1) for xr in np.linspace(0.05 * xmax, 0.95 * xmax, nrec)]
    if nsrc > 1:
        # simultaneous shots and a receiver line two elements above them
        srcs = [Source(x=float(xs), z=0.8 * zmax, f0=8.0, anglesource_deg=30.0, factor=1.0e10)
                for xs in np.linspace(0.1 * xmax, 0.9 * xmax, nsrc)]
        recs = [(float(xr), 0.8 * zmax + 2.0 * DX) for xr in np.linspace(0.05 * xmax, 0.95 * xmax, nrec)]
    dt = 4.0e-4 if scheme == 1 else 8.0e-4
    db = build_database(mesh, rho, vp, vs, srcs, recs, 1, dt, stacey=True, external_model=True, time_scheme=scheme,
                        **q)
    if physics == "aniso":
        f32 = np.float32
        body = ((np.abs(x - 0.5 * xmax) < 0.3 * xmax) & (np.abs(z - 0.5 * zmax) < 0.3 * zmax)).all(axis=(1, 2))
        lam = db.kappastore - db.mustore
        c = db.kappastore + db.mustore
        db.aniso = {"ispec": body, "c11": (1.15 * c).astype(f32), "c13": (0.9 * lam).astype(f32),
                    "c15": (0.03 * c).astype(f32), "c33": (0.95 * c).astype(f32), "c35": (-0.02 * c).astype(f32),
                    "c55": (1.05 * db.mustore).astype(f32)}
    db.nstep = nstep
    return db


def _ocean_model(nx, nz, nstep, nrec, cpml, seed=2, nsrc=1):
    xmax, zmax = nx * DX, nz * DX
    interfaces = [([0.0, xmax], [0.0, 0.0]), ([0.0, xmax], [zmax, zmax])]
    mesh = internal_mesh(0.0, xmax, nx, interfaces, [nz], absorb=(True, True, False, True))
    sh, _, _ = _shape_tables(GLL(), mesh.ngnod)
    x, z = _interp_nodes(mesh, sh)
    floor = DX * round(0.25 * nz)
    water = (zmax - z.mean(axis=(1, 2))) < floor
    vp = 2000.0 + 2500.0 * np.clip((zmax - z - floor) / (zmax - floor), 0.0, 1.0)
    vp = vp * (1.0 + 0.05 * _perturbation(x, z, xmax, zmax, seed))
    vs = vp / 1.73
    rho = 310.0 * vp ** 0.25
    vp[water], vs[water], rho[water] = 1500.0, 0.0, 1020.0
    # shots and receivers near the sea floor
    srcs = [Source(x=float(xs), z=zmax - floor + 1.4 * DX, f0=8.0, factor=1.0e10)
            for xs in (np.linspace(0.15 * xmax, 0.85 * xmax, nsrc) if nsrc > 1 else [0.5 * xmax])]
    recs = [(float(xr), zmax - floor + 0.6 * DX) for xr in np.linspace(0.12 * xmax, 0.88 * xmax, nrec)]
    pml = dict(pml=dict(nelem_thickness=cpml)) if cpml else {}
    db = build_database(mesh, rho, vp, vs, srcs, recs, 1, 5.0e-4, stacey=not cpml, external_model=True,
                        seismotype=4, **pml)
    db.nstep = nstep
    return db


def _nstep(case):
    # the trace buffer of a solver covers all the calls a program makes on it
    if case["kind"] in ("forward", "ocean"):
        return case["steps"] * (6000 if case["nx"] * case["nz"] < 20000 else 1000)
    return case["steps"]


def _model(case):
    def build():
        if case["kind"] in ("ocean", "ocean_gradient"):
            return _ocean_model(case["nx"], case["nz"], _nstep(case), case["nrec"], case.get("cpml", 0),
                                nsrc=1 if case["kind"] == "ocean" else 8)
        if case["kind"] == "smooth":
            return _solid_model(case["nx"], case["nz"], 1, 1, True, "iso", 1)
        if case["kind"] == "gradient":
            # members of a batch differ in size and material
            sizes = [(case["nx"] + 7 * m, case["nz"] + 3 * m) for m in range(case["members"])]
            dbs = [_solid_model(x, z, _nstep(case), case["nrec"], False, case["physics"], 1, seed=1 + m, nsrc=8)
                   for m, (x, z) in enumerate(sizes)]
            return dbs
        return _solid_model(case["nx"], case["nz"], _nstep(case), case["nrec"], case["topo"], case["physics"],
                            case["scheme"])
    return _cached(_key(case), build)


def _shot(db, case, rng):
    """A shot on the model: the seed sets its amplitude and the time function."""
    out = copy.copy(db)
    ns = 1 if db.time_scheme == 1 else 6
    nsrc, n = len(db.source_ispec), case["steps"]
    f0, amp = rng.uniform(6.0, 10.0, nsrc), rng.uniform(0.5, 1.5, nsrc)
    stage = np.array([0.0] if ns == 1 else [0.0, 0.0329, 0.2494, 0.4669, 0.5820, 0.8473])
    t = (np.arange(n)[:, None] + stage[None, :]) * float(db.dt)
    out.stf = np.zeros((nsrc, db.nstep, ns), dtype=np.float32)
    scale = 1.0e10 if db.acoustic is not None or case.get("physics") == "iso" else 1.0e12
    for s in range(nsrc):
        a = (math.pi * f0[s] * (t - 0.4 / f0[s])) ** 2
        out.stf[s, :n] = amp[s] * scale * (1.0 - 2.0 * a) * np.exp(-a)
    return out


def _wave(coord, rng, amp, omega, ncomp):
    """A smooth random wavefield (displacement or potential, and its rate) that fades towards the edges."""
    x, z = torch.from_numpy(coord[:, 0].copy()), torch.from_numpy(coord[:, 1].copy())
    lx, lz = float(x.max()), float(z.max())
    win = (torch.sin(math.pi * x / lx) * torch.sin(math.pi * (z / lz).clamp(0.0, 1.0))) ** 2
    u = torch.zeros(x.numel(), ncomp, dtype=torch.float64)
    v = torch.zeros_like(u)
    for c in range(ncomp):
        for _ in range(3):
            wl = rng.uniform(12.0, 24.0) * DX
            th, ph, a = rng.uniform(0.0, 2 * math.pi), rng.uniform(0.0, 2 * math.pi), rng.uniform(0.5, 1.0)
            arg = (2 * math.pi / wl) * (math.cos(th) * x + math.sin(th) * z) + ph
            u[:, c] += amp * a * torch.cos(arg)
            v[:, c] += amp * a * omega * torch.sin(arg)
    return [(f * win[:, None]).to(torch.float32).numpy() for f in (u, v)]


def _pinned(*shape):
    t = torch.empty(*shape, dtype=torch.float32)
    return (t.pin_memory() if torch.cuda.is_available() else t).numpy()


def _inputs(case, seed):
    """The model and what the seed draws: the same for `prepare` and `exact`."""
    rng = np.random.default_rng([int(seed), 77])
    base = _model(case)
    if case["kind"] == "smooth":
        k = np.arange(1, case["nfields"] + 1)[:, None, None, None]
        x, z = base.coord[base.ibool, 0], base.coord[base.ibool, 1]
        f = sum(rng.normal() * np.cos(rng.uniform(0.002, 0.02) * k * x + rng.uniform(0.002, 0.02) * z) for _ in range(3))
        return base, (f + 0.3 * rng.standard_normal(f.shape)).astype(np.float32)
    if case["kind"] == "gradient":
        shots = [_shot(d, case, rng) for d in base]
        db = shots[0] if len(shots) == 1 else batch.pack(shots)[0]
        return db, _observed(case, len(db.rec_ispec), float(db.dt), rng, 0.05)
    db = _shot(base, case, rng)
    if case["kind"] == "ocean_gradient":
        return db, _observed(case, len(db.rec_ispec), float(db.dt), rng, 1.0e3)
    f = {}
    if case["kind"] == "ocean":
        wet = np.zeros(db.nglob, dtype=bool)
        wet[db.ibool[np.asarray(db.acoustic["ispec"], dtype=bool)]] = True
        # free-surface points hold no potential, CPML layers start empty
        quiet = np.zeros(db.nglob, dtype=bool)
        quiet[db.acoustic["free_iglob"]] = True
        if db.pml is not None:
            quiet[db.ibool[np.asarray(db.pml["region"]) > 0]] = True
        dry = np.ones(db.nglob, dtype=bool)
        dry[db.ibool[np.asarray(db.acoustic["ispec"], dtype=bool)]] = False
        u, v = _wave(db.coord, rng, 0.02, 50.0, 2)
        p, pd = _wave(db.coord, rng, 1.0e3, 50.0, 1)
        keep_s, keep_f = (dry & ~quiet), (wet & ~quiet)
        f = dict(displ=u * keep_s[:, None], veloc=v * keep_s[:, None], pot=p[:, 0] * keep_f, pot_dot=pd[:, 0] * keep_f)
    else:
        u, v = _wave(db.coord, rng, 0.05, 50.0, 2)
        f = dict(displ=u, veloc=v)
    return db, f


def _observed(case, nrec, dt, rng, amp):
    t = np.arange(case["steps"]) * dt
    f0 = rng.uniform(5.0, 9.0, (nrec, 1, 2))
    a = (math.pi * f0 * (t[None, :, None] - rng.uniform(0.1, 0.9, (nrec, 1, 2)) * t[-1])) ** 2
    return amp * rng.uniform(0.5, 1.5, (nrec, 1, 2)) * (1.0 - 2.0 * a) * np.exp(-a)


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    db, data = _inputs(case, seed)
    kind = case["kind"]
    if kind == "forward":
        s.solver = ElasticSolver(db)
        s.solver.set_fields(data["displ"], data["veloc"])
        s.fields = [_pinned(db.nglob, 2) for _ in range(3)]
    elif kind == "ocean":
        s.solver = CoupledSolver(db)
        s.solver.set_fields(**data)
        s.fields = {k: _pinned(db.nglob, 2) for k in ("displ", "veloc", "accel")}
        s.fields.update({k: _pinned(db.nglob) for k in ("pot", "pot_dot", "pot_dot_dot")})
    elif kind == "gradient":
        s.solver, s.observed = FWIGradient(db, case["checkpoint_every"]), data
    elif kind == "ocean_gradient":
        s.solver, s.observed = CoupledKernels(db, case["checkpoint_every"]), data
    else:
        s.db, s.values = db, data
    if kind in ("forward", "ocean"):
        s.solver.prepare()
    return s


def run(state):
    case = state.case
    if case["kind"] in ("forward", "ocean"):
        seis = state.solver.run(case["steps"])
        return [seis, state.solver.get_fields(state.fields)]
    if case["kind"] in ("gradient", "ocean_gradient"):
        seis = state.solver.forward()
        return [seis, state.solver.backward(seis - state.observed)]
    return smooth(state.db, state.values, case["sigma_h"], case["sigma_v"])


def work(case):
    """Per step: the mapping and two moduli of every element point read (24 B), displacement and velocity of every
    global point read and written and its inverse mass read (a fluid point holds one component); 3 SLS add nine
    memory variables per element point read and written, a CPML point twelve (six in the fluid).  A gradient is the
    forward run, its recomputation and the adjoint run, which reads a forward frame and updates two kernel sums per
    element point.  Smoothing reads and writes the fields once and weighs every pair of points within six standard
    deviations."""
    nx, nz = case["nx"], case["nz"]
    if case["kind"] == "smooth":
        n = 25 * nx * nz
        pairs = n * min(n, 25 * math.pi * 36.0 * case["sigma_h"] * case["sigma_v"] / DX ** 2)
        return {"bytes": n * (16.0 + 8.0 * case["nfields"]), "flops": pairs * (8.0 + 2.0 * case["nfields"])}
    ocean = case["kind"].startswith("ocean")
    if case["kind"] == "gradient":
        nspec = sum((nx + 7 * m) * (nz + 3 * m) for m in range(case["members"]))
    else:
        nspec = nx * nz
    wet = nx * round(0.25 * nz) if ocean else 0
    dry = nspec - wet
    step = dry * (600.0 + 16 * 40.0) + wet * (500.0 + 16 * 20.0)
    flops = dry * 25 * 110.0 + wet * 25 * 56.0
    if case.get("physics") == "visco":
        step += dry * 1800.0
        flops += dry * 25 * 80.0
    if case.get("physics") == "aniso":
        step += 0.36 * dry * 25 * 16.0
        flops += 0.36 * dry * 25 * 10.0
    if case.get("cpml"):
        layer = 2 * nz * case["cpml"] + (nx - 2 * case["cpml"]) * case["cpml"]
        step += layer * 25 * 96.0
        flops += layer * 25 * 120.0
    if case.get("scheme") == 2:
        # six stages, each with the auxiliary fields and memory variables
        step = 6 * (step + dry * (16 * 32.0 + (1800.0 if case["physics"] == "visco" else 0.0)))
        flops *= 6
    n = case["steps"]
    if case["kind"] in ("gradient", "ocean_gradient"):
        adj = step + nspec * (25 * 16.0 + 16 * 16.0)
        return {"bytes": n * (2 * step + nspec * 16 * 8.0 + adj), "flops": n * (3 * flops + nspec * 25 * 50.0)}
    npts = 16 * nspec
    out = (24.0 if not ocean else 36.0) * npts
    return {"bytes": n * step + out, "flops": n * flops}


def tolerance(case):
    # four times the largest difference seen between two orders of the sums over a step (elements taken in another
    # order); the accelerations and pressures of a forward run, second derivatives of an FP32 field that is smooth on
    # the scale of the elements, carry the largest
    return {"forward": {"rel": 3.5e-3}, "ocean": {"rel": 1.4e-3}, "gradient": {"rel": 1e-4},
            "ocean_gradient": {"rel": 1e-4}, "smooth": {"rel": 2e-7, "max": 1e-5}}[case["kind"]]


# ---- the schemes in float64

def _t(a, dev, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), device=dev).to(dtype)


class _Lik:
    """Strain coefficients of a CPML point, per region (0 outside, 1 x, 2 z, 3 both)."""

    def __init__(self, kx, bx, ax, kz, bz, az, region, own, other):
        both, xo, zo = region == 3, region == own, region == other
        zero = np.zeros_like(kx)
        with np.errstate(divide="ignore", invalid="ignore"):
            gx = (ax * bz + ax * ax + 2 * bx * az - 2 * ax * (bx + az)) / (bz - ax)
            gz = (ax * bz + bz * bz + 2 * bx * az - 2 * bz * (bx + az)) / (ax - bz)
            self.A0 = np.where(both, kx / kz, np.where(xo, kx, np.where(zo, 1 / kz, zero)))
            self.A1 = np.where(both, kx / kz / 2 * (gx - ax), np.where(xo, -kx * (ax - bx), zero))
            self.A2 = np.where(both, kx / kz / 2 * (gz - bz), np.where(zo, -(bz - az) / kz, zero))


def _field_coefs(kx, bx, ax, kz, bz, az, region):
    both, xo, zo = region == 3, region == 1, region == 2
    zero = np.zeros_like(kx)
    with np.errstate(divide="ignore", invalid="ignore"):
        gx = (ax * az + ax * ax + 2 * bx * bz - 2 * ax * (bx + bz)) / (az - ax)
        gz = (ax * az + az * az + 2 * bx * bz - 2 * az * (bx + bz)) / (ax - az)
    k = kx * kz
    A0 = np.where(both, k, np.where(xo, kx, np.where(zo, kz, zero)))
    A1 = np.where(both, k / 2 * (gx - ax + gz - az), np.where(xo, kx * (bx - ax), np.where(zo, kz * (bz - az), zero)))
    A2 = np.where(both, k / 2 * (ax * ax - gx * ax + az * az - gz * az),
                  np.where(xo, -kx * ax * (bx - ax), np.where(zo, -kz * az * (bz - az), zero)))
    A3 = np.where(both, k / 2 * ax * ax * (gx - ax), np.where(xo, kx * ax * ax * (bx - ax), zero))
    A4 = np.where(both, k / 2 * az * az * (gz - az), np.where(zo, kz * az * az * (bz - az), zero))
    return A0, A1, A2, A3, A4


def _conv(b, dt):
    t = np.exp(-0.5 * b * dt)
    small = np.abs(b) <= 1e-5
    c1 = np.where(small, 0.5 * dt, (1 - t) / np.where(small, 1.0, b))
    return t * t, c1, np.where(small, c1, c1 * t)


class _Domain:
    """Elements of one domain: mapping, derivatives and the CPML layer among them."""

    def __init__(self, db, elems, dev):
        self.dev, self.e = dev, elems
        self.ib = torch.as_tensor(db.ibool[elems].astype(np.int64), device=dev)
        self.flat = self.ib.reshape(-1)
        self.xix, self.xiz, self.gx, self.gz = (_t(getattr(db, k)[elems].astype(np.float32), dev)
                                                for k in ("xix", "xiz", "gammax", "gammaz"))
        g = db.gll
        self.h = _t(np.asarray(g.hprime, np.float32).reshape(5, 5), dev)
        self.hw = _t(np.asarray(g.hprimewgll, np.float32).reshape(5, 5), dev)
        self.wx, self.wz = _t(np.asarray(g.wxgll, np.float32), dev), _t(np.asarray(g.wzgll, np.float32), dev)
        self.pml = None
        if db.pml is not None:
            reg = np.asarray(db.pml["region"])[elems]
            sel = np.flatnonzero(reg > 0)
            if sel.size:
                kx, kz, dx, dz, ax, az = (np.asarray(db.pml[k], np.float64)[elems][sel]
                                          for k in ("K_x", "K_z", "d_x", "d_z", "alpha_x", "alpha_z"))
                bx, bz = ax + dx / kx, az + dz / kz
                r = np.broadcast_to(reg[sel][:, None, None], kx.shape)
                zx, xz = _Lik(kz, bz, az, kx, bx, ax, r, 2, 1), _Lik(kx, bx, ax, kz, bz, az, r, 1, 2)
                dt = float(db.pml["dt"])
                t = lambda a: _t(a, dev)[..., None]  # noqa: E731
                self.pml = dict(sel=torch.as_tensor(sel, device=dev),
                                zx=[t(v) for v in (zx.A0, zx.A1, zx.A2)], xz=[t(v) for v in (xz.A0, xz.A1, xz.A2)],
                                L=[t(v) for v in _field_coefs(kx, bx, ax, kz, bz, az, r)],
                                **{n: [t(v) for v in _conv(b, dt)] for n, b in (("ax", ax), ("az", az), ("bx", bx), ("bz", bz))})

    def grad(self, f):
        """d/dx, d/dz of a field (points, ncomp) at the element points (ns, j, i, ncomp)."""
        fl = f[self.ib]
        dxi = torch.einsum("ejkc,ik->ejic", fl, self.h)
        dg = torch.einsum("ekic,jk->ejic", fl, self.h)
        return (dxi * self.xix[..., None] + dg * self.gx[..., None],
                dxi * self.xiz[..., None] + dg * self.gz[..., None])

    def weak(self, acc, t1, t2):
        """acc -= the weighted transposed derivatives of t1 (xi) and t2 (gamma)."""
        r = torch.einsum("ejkc,ki->ejic", t1, self.hw) * self.wz[None, :, None, None]
        r += torch.einsum("ekic,kj->ejic", t2, self.hw) * self.wx[None, None, :, None]
        acc.index_add_(0, self.flat, r.reshape(-1, r.shape[-1]), alpha=-1.0)

    @staticmethod
    def upd(r, c, f, fo):
        return c[0] * r + c[1] * f + c[2] * fo

    def layer(self, mem, gx, gz, gxo, gzo, f, fd, fo):
        """Advances the layer's memory variables; returns the modified gradients and the extra terms per unit of
        w_i w_j rho J (or J / kappa) at the layer's points."""
        P, s = self.pml, self.pml["sel"]
        a, b, ao, bo = gx[s], gz[s], gxo[s], gzo[s]
        q = self.ib[s]
        u, ud, uo = f[q], fd[q], fo[q]
        if not mem:
            mem.extend(torch.zeros_like(x) for x in (a, a, b, b, u, u))
        for n, (c, x, y) in enumerate(((P["az"], a, ao), (P["bx"], a, ao), (P["ax"], b, bo), (P["bz"], b, bo),
                                       (P["ax"], u, uo), (P["az"], u, uo))):
            mem[n] = self.upd(mem[n], c, x, y)
        ma = P["zx"][0] * a + P["zx"][1] * mem[0] + P["zx"][2] * mem[1]
        mb = P["xz"][0] * b + P["xz"][1] * mem[2] + P["xz"][2] * mem[3]
        extra = P["L"][1] * ud + P["L"][2] * u + P["L"][3] * mem[4] + P["L"][4] * mem[5]
        return ma, mb, extra * (self.wx[None, None, :, None] * self.wz[None, :, None, None])


class _Run64:
    """The Newmark or LDDRK time loop of a Database (solid, or fluid and solid) in float64."""

    def __init__(self, db, dev, adjoint=False):
        self.db, self.dev, self.adjoint = db, dev, adjoint
        t = lambda a: _t(a, dev)  # noqa: E731
        self.dt, self.dto2, self.dt2 = (float(np.float32(x)) for x in (db.deltat, db.deltatover2, db.deltatsquareover2))
        wet = np.zeros(db.nspec, bool) if db.acoustic is None else np.asarray(db.acoustic["ispec"], bool)
        self.wet = wet
        self.S, self.F = _Domain(db, np.flatnonzero(~wet), dev), None
        el = self.S.e
        f32 = np.float32
        rho = db.rhostore[el].astype(f32)
        cp = (db.rho_vpstore[el].astype(f32) / rho).astype(f32)
        mu = db.mustore[el].astype(f32)
        lam = ((rho * cp).astype(f32) * cp - f32(2.0) * mu).astype(f32)
        self.lam, self.mu = t(lam), t(mu)
        S = self.S
        self.J = 1.0 / (S.xix * S.gz - S.gx * S.xiz)
        self.rmass = t(db.rmass_inverse_elastic)
        self.st = torch.as_tensor(db.stacey_iglob.astype(np.int64), device=dev)
        self.stn = t(np.stack([db.stacey_nx, db.stacey_nz], -1).reshape(-1, 2))
        self.stw = t(db.stacey_weight)[:, None]
        self.srp, self.srs = t(db.stacey_rho_vp)[:, None], t(db.stacey_rho_vs)[:, None]
        z = lambda *s: torch.zeros(*s, dtype=torch.float64, device=dev)  # noqa: E731
        n = db.nglob
        self.u, self.v, self.a = z(n, 2), z(n, 2), z(n, 2)
        self.memS, self.memF, self.att = [], [], None
        if db.pml is not None:
            self.edge = torch.as_tensor(np.asarray(db.pml["bnd_el"], np.int64), device=dev)
            if S.pml is not None:
                s = S.pml["sel"].cpu().numpy()
                self.rhoj = t((rho[s] * db.jacobian[el][s].astype(f32)).astype(f32))[..., None]
        self.an = None
        if db.aniso is not None:
            self.an = torch.as_tensor(np.flatnonzero(np.asarray(db.aniso["ispec"], bool)[el]), device=dev)
            self.c = {k: t(db.aniso[k][el].astype(f32))[self.an] for k in ("c11", "c13", "c15", "c33", "c35", "c55")}
        if db.atten is not None:
            names = ("a1", "a2", "b1", "b2") if db.time_scheme == 1 else ("itau1", "itau2", "phi1", "phi2")
            self.att = [t(np.asarray(db.atten[k])[el].astype(f32)) for k in names]
            self.e = [torch.zeros_like(self.att[0]) for _ in range(6)]
            self.old = [torch.zeros_like(self.mu) for _ in range(3)]
        if db.time_scheme == 2:
            self.uL, self.vL = z(n, 2), z(n, 2)
        if db.acoustic is not None:
            self._fluid(t, z)
        self.rib = torch.as_tensor(db.ibool[db.rec_ispec].astype(np.int64), device=dev)
        self.rh = t(db.hxir.astype(f32)[:, None, :] * db.hgammar.astype(f32)[:, :, None])
        self.sib = torch.as_tensor(db.ibool[db.source_ispec].astype(np.int64), device=dev)
        self.sarr, self.swet = t(db.sourcearrays), wet[db.source_ispec]
        self.it = 0

    def _fluid(self, t, z):
        db, dev, ac, f32 = self.db, self.dev, self.db.acoustic, np.float32
        self.F = _Domain(db, np.flatnonzero(self.wet), dev)
        e = self.F.e
        jac, rho, kap = (getattr(db, k)[e].astype(f32) for k in ("jacobian", "rhostore", "kappastore"))
        self.fac, self.frho, self.fkap = t(jac / rho)[..., None], t(rho), t(kap)
        if self.F.pml is not None:
            s = self.F.pml["sel"].cpu().numpy()
            self.jk = t(jac[s] / kap[s])[..., None]
        self.p, self.pd, self.pdd = z(db.nglob, 1), z(db.nglob, 1), z(db.nglob, 1)
        self.frm = t(ac["rmass"])[:, None]
        i64 = lambda a: torch.as_tensor(np.asarray(a, np.int64), device=dev)  # noqa: E731
        self.free, self.fst = i64(ac["free_iglob"]), i64(ac["st_iglob"])
        self.fstw = (t(ac["st_w"]) / t(ac["st_rvp"]))[:, None]
        self.fedge = i64(db.pml["bnd_ac"]) if db.pml is not None else i64([])
        self.kappa_src = t(db.kappastore[db.source_ispec].astype(f32))
        self.ca, self.ce = i64(ac["cpl_ac_iglob"]), i64(ac["cpl_el_iglob"])
        self.can = t(np.stack([ac["cpl_ac_nx"], ac["cpl_ac_nz"]], -1))
        self.cen = t(np.stack([ac["cpl_el_nx"], ac["cpl_el_nz"]], -1))
        self.caw, self.cew = t(ac["cpl_ac_w"])[:, None], t(ac["cpl_el_w"])[:, None]
        self.cmem = None
        if db.pml is None:
            return
        # coupling points whose other side lies in a layer
        def at(q):
            q = np.asarray(q, np.int64)
            g = lambda k: np.asarray(db.pml[k], np.float64).reshape(-1)[q]  # noqa: E731
            kx, kz, ax, az = g("K_x"), g("K_z"), g("alpha_x"), g("alpha_z")
            return kx, ax + g("d_x") / kx, ax, kz, az + g("d_z") / kz, az, np.asarray(db.pml["region"])[q // 25]
        dt = float(db.pml["dt"])
        kx, bx, ax, kz, bz, az, r = at(ac["cpl_ac_elpt"])
        l13, l31 = _Lik(kx, bx, ax, kz, bz, az, r, 1, 2), _Lik(kz, bz, az, kx, bx, ax, r, 2, 1)
        pick = lambda a, b: t(np.where(r == 1, a, b))[:, None]  # noqa: E731
        self.ca_in = torch.as_tensor(r > 0, device=dev)[:, None]
        self.ca_c = [pick(l13.A0, l31.A0), pick(l13.A1, l31.A1)] + [t(x)[:, None] for x in _conv(np.where(r == 1, ax, az), dt)]
        kx, bx, ax, kz, bz, az, r = at(ac["cpl_el_acpt"])
        self.ce_in = torch.as_tensor(r > 0, device=dev)[:, None]
        self.ce_c = [t(x)[:, None] for x in _field_coefs(kx, bx, ax, kz, bz, az, r)[:4]] + [t(x)[:, None] for x in _conv(ax, dt)]
        self.cmem = [z(len(self.ca), 2), z(len(self.ce), 1)]

    def predicted(self, u, v, a):
        return u + self.dt * v + self.dt2 * a

    def sources(self, acc, wet, stage, override):
        db, n = self.db, self.it
        if override is not None:  # adjoint sources at the receivers: (nrec, 2)
            rw = torch.as_tensor(self.wet[db.rec_ispec] == wet, device=self.dev)
            s = override[:, None, None, :] * self.rh[..., None]
            s = s[..., :acc.shape[1]]
            acc.index_add_(0, self.rib[rw].reshape(-1), s[rw].reshape(-1, acc.shape[1]))
            return
        for k in range(len(db.source_ispec)):
            if bool(self.swet[k]) == wet and n < db.stf.shape[1]:
                f = float(db.stf[k, n, stage])
                s = self.sarr[k][..., :1] / self.kappa_src[k][..., None] if wet else self.sarr[k]
                acc.index_add_(0, self.sib[k].reshape(-1), (s * f).reshape(-1, acc.shape[1]))

    def attenuate(self, gx, gz, stage):
        xx, zz, xz = gx[..., 0], gz[..., 1], gz[..., 0] + gx[..., 1]
        th = (xx + zz)[..., None]
        q = self.att
        d, g = (xx[..., None] - th / 2), xz[..., None]
        if self.db.time_scheme == 1:
            o = [x[..., None] for x in self.old]
            tho = o[0] + o[1]
            self.e[0] = q[0] ** 2 * self.e[0] + q[2] * (th + q[0] * tho)
            self.e[1] = q[1] ** 2 * self.e[1] + q[3] * (d + q[1] * (o[0] - tho / 2))
            self.e[2] = q[1] ** 2 * self.e[2] + q[3] * (g + q[1] * o[2])
            self.old = [xx, zz, xz]
        else:
            al, be = float(ALPHA_LDDRK[stage]), float(BETA_LDDRK[stage])
            for k, (it, ph, x) in enumerate(((q[0], q[2], th), (q[1], q[3], d), (q[1], q[3], g))):
                self.e[3 + k] = al * self.e[3 + k] + self.dt * (ph * x - self.e[k] * it)
                self.e[k] = self.e[k] + be * self.e[3 + k]
        return [e.sum(-1) for e in self.e[:3]]

    def solid_forces(self, acc, uo, stage=0):
        S, lam, mu = self.S, self.lam, self.mu
        gx, gz = S.grad(self.u)
        if self.grads is not None:
            self.grads(gx, gz)
        xx, zx, xz, zz = gx[..., 0], gx[..., 1], gz[..., 0], gz[..., 1]  # ux,x uz,x ux,z uz,z
        sxx, szz, sxz = (lam + 2 * mu) * xx + lam * zz, (lam + 2 * mu) * zz + lam * xx, mu * (zx + xz)
        szx = sxz
        if self.an is not None:
            s, c = self.an, self.c
            a, b, g = xx[s], zz[s], (zx + xz)[s]
            sxx[s] = c["c11"] * a + c["c13"] * b + c["c15"] * g
            szz[s] = c["c13"] * a + c["c33"] * b + c["c35"] * g
            sxz[s] = c["c15"] * a + c["c35"] * b + c["c55"] * g
        if self.att is not None:
            e1, e11, e13 = self.attenuate(gx, gz, stage)
            sxx, szz = sxx + (lam + mu) * e1 + 2 * mu * e11, szz + (lam + mu) * e1 - 2 * mu * e11
            sxz = szx = sxz + mu * e13
        if S.pml is not None:
            s = S.pml["sel"]
            gxo, gzo = S.grad(uo)
            ma, mb, extra = S.layer(self.memS, gx, gz, gxo, gzo, self.u, self.v, uo)
            l, m = lam[s], mu[s]
            szx = sxz.clone()
            sxx[s] = (l + 2 * m) * ma[..., 0] + l * zz[s]
            szz[s] = (l + 2 * m) * mb[..., 1] + l * xx[s]
            szx[s] = m * (zx[s] + mb[..., 0])
            sxz[s] = m * (xz[s] + ma[..., 1])
            acc.index_add_(0, S.ib[s].reshape(-1), (extra * self.rhoj).reshape(-1, 2), alpha=-1.0)
        J = self.J
        st = lambda a, b: torch.stack((J * (sxx * a + szx * b), J * (sxz * a + szz * b)), -1)  # noqa: E731
        S.weak(acc, st(S.xix, S.xiz), st(S.gx, S.gz))

    def stacey(self, acc):
        v = self.v[self.st]
        vn = (v * self.stn).sum(-1, keepdim=True)
        acc.index_add_(0, self.st, (self.srp * vn * self.stn + self.srs * (v - vn * self.stn)) * self.stw, alpha=-1.0)

    def solid_step(self, adj=None):
        if len(self.S.e) == 0:
            return
        uo = self.u + 0.5 * self.dt2 * self.a if self.S.pml is not None else None
        self.u = self.predicted(self.u, self.v, self.a)
        self.v = self.v + self.dto2 * self.a
        if self.db.pml is not None:
            for f in (self.u, self.v, uo):
                f[self.edge] = 0.0
        acc = torch.zeros_like(self.u)
        self.stacey(acc)
        if self.F is not None:
            if self.adjoint:
                pr = self.predicted(self.p, self.pd, self.pdd)[self.ce]
            else:
                pr = -self.pdd[self.ce]
                if self.cmem is not None:
                    c = self.ce_c
                    self.cmem[1] = c[4] * self.cmem[1] + c[5] * self.p[self.ce] + c[6] * self.pold[self.ce]
                    lay = -(c[0] * self.pdd[self.ce] + c[1] * self.pd[self.ce] + c[2] * self.p[self.ce] + c[3] * self.cmem[1])
                    pr = torch.where(self.ce_in, lay, pr)
            acc.index_add_(0, self.ce, self.cew * self.cen * pr)
        self.sources(acc, False, 0, adj)
        self.solid_forces(acc, uo)
        self.a = acc * self.rmass
        self.v = self.v + self.dto2 * self.a

    def fluid_step(self, adj=None):
        if self.adjoint:
            un = -self.a[self.ca]
        else:
            un = self.predicted(self.u, self.v, self.a)[self.ca]
            if self.cmem is not None:
                c = self.ca_c
                uo = (self.u + 0.5 * self.dt2 * self.a)[self.ca]
                self.cmem[0] = c[2] * self.cmem[0] + c[3] * un + c[4] * uo
                un = torch.where(self.ca_in, c[0] * un + c[1] * self.cmem[0], un)
        self.pold = self.p + 0.5 * self.dt2 * self.pdd
        self.p = self.predicted(self.p, self.pd, self.pdd)
        self.pd = self.pd + self.dto2 * self.pdd
        zero = torch.cat((self.free, self.fedge))
        self.p[zero] = 0.0
        self.pd[zero] = 0.0
        self.pold[self.fedge] = 0.0
        acc = torch.zeros_like(self.p)
        acc.index_add_(0, self.fst, self.pd[self.fst] * self.fstw, alpha=-1.0)
        acc.index_add_(0, self.ca, self.caw * (un * self.can).sum(-1, keepdim=True))
        self.sources(acc, True, 0, adj)
        F = self.F
        gx, gz = F.grad(self.p)
        if F.pml is not None:
            s = F.pml["sel"]
            gxo, gzo = F.grad(self.pold)
            gx[s], gz[s], extra = F.layer(self.memF, gx, gz, gxo, gzo, self.p, self.pd, self.pold)
            acc.index_add_(0, F.ib[s].reshape(-1), (extra * self.jk).reshape(-1, 1), alpha=-1.0)
        F.weak(acc, self.fac * (F.xix[..., None] * gx + F.xiz[..., None] * gz),
               self.fac * (F.gx[..., None] * gx + F.gz[..., None] * gz))
        self.pdd = acc * self.frm
        self.pd = self.pd + self.dto2 * self.pdd
        for f in (self.p, self.pd, self.pdd):
            f[zero] = 0.0

    def step(self, adj=None, grads=None):
        self.grads = grads
        if self.db.time_scheme == 2:
            for k in range(6):
                acc = torch.zeros_like(self.u)
                self.stacey(acc)
                self.sources(acc, False, k, None)
                self.solid_forces(acc, None, k)
                self.a = acc * self.rmass
                al, be = float(ALPHA_LDDRK[k]), float(BETA_LDDRK[k])
                self.vL = al * self.vL + self.dt * self.a
                self.uL = al * self.uL + self.dt * self.v
                self.v = self.v + be * self.vL
                self.u = self.u + be * self.uL
        elif self.adjoint and self.F is not None:
            self.solid_step(adj)
            self.fluid_step(adj)
        else:
            if self.F is not None:
                self.fluid_step(adj)
            self.solid_step(adj)
        self.it += 1

    def record(self):
        """Displacement at the receivers, or the pressure of a marine run."""
        if self.F is not None:
            v = (-self.pdd[self.rib][..., 0] * self.rh).sum((1, 2))
            return torch.stack((v, torch.zeros_like(v)), -1)
        return (self.u[self.rib] * self.rh[..., None]).sum((1, 2))


def _exact_gradient(case, db, observed, dev):
    f, n = _Run64(db, dev), case["steps"]
    frames, seis = [], []
    for _ in range(n):
        f.step()
        frames.append((f.u, f.p if f.F is not None else None))
        seis.append(f.record())
    seis = torch.stack(seis, 1)
    adj = (seis - _t(observed, dev)).cpu().numpy().astype(np.float32)
    r = _Run64(db, dev, adjoint=True)
    S, F = r.S, r.F
    rho_s, kap_s, mu_s = (torch.zeros_like(r.mu) for _ in range(3))
    fl = [torch.zeros_like(r.fkap) for _ in range(2)] if F is not None else None
    for it in range(n):
        b, bp = frames[n - 1 - it]

        def kernels(gx, gz, b=b):
            bx, bz = S.grad(b)
            k = (gx[..., 0] + gz[..., 1]) * (bx[..., 0] + bz[..., 1])
            kap_s.add_(k)
            mu_s.add_(gx[..., 0] * bx[..., 0] + gz[..., 1] * bz[..., 1]
                      + 0.5 * (gx[..., 1] + gz[..., 0]) * (bx[..., 1] + bz[..., 0]) - k / 3)

        r.step(adj=_t(adj[:, n - 1 - it], dev), grads=kernels)
        rho_s += (r.a * b).sum(-1)[S.ib]
        if F is not None:
            (ax, az), (bx, bz) = F.grad(r.p), F.grad(bp)
            fl[0] += (ax * bx + az * bz)[..., 0] / r.frho * r.dt
            fl[1] += (r.pdd * bp)[:, 0][F.ib] / r.fkap * r.dt
    el = S.e
    rho, kap = (_t(getattr(db, k)[el].astype(np.float32), dev) for k in ("rhostore", "kappastore"))
    ker = [-rho * r.dt * rho_s, -kap * r.dt * kap_s, -2 * r.mu * r.dt * mu_s]
    if F is None:
        return [seis.cpu().numpy(), tuple(k.cpu().numpy() for k in ker)]
    out = {}
    for names, e, vals in ((("rho", "kappa", "mu"), el, ker), (("rho_ac", "kappa_ac"), F.e, fl)):
        for k, v in zip(names, vals):
            out[k] = np.zeros((db.nspec, 5, 5))
            out[k][e] = v.cpu().numpy()
    return [seis.cpu().numpy(), out]


def _exact_smooth(case, db, values, dev):
    x = _t((db.coord[db.ibool, 0].astype(np.float32) / np.float32(case["sigma_h"])).ravel(), dev)
    z = _t((db.coord[db.ibool, 1].astype(np.float32) / np.float32(case["sigma_v"])).ravel(), dev)
    w = db.gll.wgll_dble
    wj = _t((db.jacobian.astype(np.float32) * (w[None, :] * w[:, None]).astype(np.float32)[None]).ravel(), dev)
    f = _t(values.reshape(case["nfields"], -1), dev)
    order = torch.argsort(x)
    xs, zs, ws, fs = x[order], z[order], wj[order], f[:, order]
    out = torch.zeros_like(f)
    n, block = x.numel(), 256
    for b in range(0, n, block):
        tx, tz = xs[b:b + block], zs[b:b + block]
        lo = int(torch.searchsorted(xs, tx[0] - 6.0))
        hi = int(torch.searchsorted(xs, tx[-1] + 6.0, right=True))
        r2 = (tx[:, None] - xs[None, lo:hi]) ** 2 + (tz[:, None] - zs[None, lo:hi]) ** 2
        g = torch.exp(-0.5 * r2) * (r2 <= 36.0) * ws[None, lo:hi]
        out[:, order[b:b + block]] = (fs[:, lo:hi] @ g.T) / g.sum(1)[None]
    return out.reshape(values.shape).cpu().numpy()


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    db, data = _inputs(case, seed)
    if case["kind"] == "smooth":
        return _exact_smooth(case, db, data, dev)
    if case["kind"] in ("gradient", "ocean_gradient"):
        return _exact_gradient(case, db, data, dev)
    r = _Run64(db, dev)
    r.u, r.v = _t(data["displ"], dev), _t(data["veloc"], dev)
    if r.F is not None:
        r.p, r.pd = _t(data["pot"], dev)[:, None], _t(data["pot_dot"], dev)[:, None]
    seis = []
    for _ in range(case["steps"]):
        r.step()
        seis.append(r.record())
    seis = torch.stack(seis, 1).cpu().numpy()
    solid = [f.cpu().numpy() for f in (r.u, r.v, r.a)]
    if r.F is None:
        return [seis, solid]
    fluid = [f[:, 0].cpu().numpy() for f in (r.p, r.pd, r.pdd)]
    return [seis, dict(zip(("displ", "veloc", "accel", "pot", "pot_dot", "pot_dot_dot"), solid + fluid))]
