"""Performance cases of the MPM step: what a program that uses this framework has it do.

Every case goes through a public entry point: ``GpuSim`` (one scene: upload,
steps, read-back or frame rows), ``GpuBatch`` (scenes joining one batch) and
``mtr_p2g_noalloc`` (the transfer on device pointers).  Scenes are the
workloads of ``matter_tests_b200.scenes`` in mid-flow: the jittered lattice of
the builder with a smooth collapsing velocity field, the elastic strain of its
own weight with some noise, and a plastic history, as a restart from a
checkpoint uploads it.  A pass uploads that state, advances it and reads the
result back, so every pass does the same work.

``exact`` advances the same state with a plain FP64 torch restatement of the
step, which shares nothing with the package.
"""
import ctypes as C
import math

import torch

from matter_tests_b200 import abi
from matter_tests_b200.gpu import GpuBatch, GpuSim, load_library

DEV = "cuda"
F64 = torch.float64

# Material and boundary of each scene family (the builders of scenes.py).
FAMILIES = {
    # 2D plane-strain column of the FP64 reference workload, Drucker-Prager on a SlipFree floor
    "collapse2d": dict(dim=2, model="dp", E=1e6, nu=0.3, rho=1550.0, M=math.tan(math.radians(30.0)), aspect=2.0,
                       floor=("slipfree", 0.5)),
    # 3D mu(I) column, the headline workload: box 1 : 2 : 1 on a SlipStick floor
    "mui3d": dict(dim=3, model="mui", E=1e7, nu=0.3, rho=1500.0, mu_1=0.38, mu_2=0.64, aspect=2.0,
                  floor=("slipstick", 0.4)),
    # 3D Perzyna Cam-Clay block released on a 30 degree incline with Gaussian bumps
    "incline3d": dict(dim=3, model="mcc", E=5e6, nu=0.25, rho=1000.0, M=1.2, p0=1e4, visc=1e-3, aspect=0.3),
    # 3D Drucker-Prager column of the ensemble and serving workloads
    "dp3d": dict(dim=3, model="dp", E=2e6, nu=0.3, rho=1550.0, M=math.tan(math.radians(28.0)), aspect=1.5,
                 floor=("slipfree", 0.5)),
    # elastic block on a no-flow floor, frame rows written while it steps (Simulation::simulate's loop)
    "elastic3d": dict(dim=3, model="elastic", E=1e6, nu=0.3, rho=1000.0, aspect=1.0, floor=("slipstick", 0.3)),
}
# read back by a job: the whole state of an FP64 run (the plastic scalars of the mu(I) model come out of
# a cancelling closed form and feed nothing back, so its program reads x, v, F, B); a mixed run is read as
# the serving loop reads it, x and v, the latter in the FP32 it is kept in
FIELDS = {"dp": ("x", "v", "F", "B", "scalars"), "mcc": ("x", "v", "F", "B", "scalars"), "mui": ("x", "v", "F", "B"),
          "elastic": ("x", "v", "F", "B")}


def listed():
    return [
        # a real-time loop's transfer of a small particle set: launches and latency only
        dict(name="p2g_small", do="p2g", dim=3, deg=2, n=3993, seed_cells=0),
        # the same entry point at its documented capacity, cubic splines
        dict(name="p2g_full", do="p2g", dim=3, deg=3, n=261_003, seed_cells=0),
        # the ensemble's smallest scene on its own: 16 steps of 5k particles
        dict(name="tiny2d_fp64", do="job", family="collapse2d", deg=2, flip=-2.0, musl=False, mixed=False, n=4999,
             steps=16),
        # the FP64 2D column workload (51,200 particles)
        dict(name="collapse2d_fp64", do="job", family="collapse2d", deg=2, flip=-2.0, musl=False, mixed=False,
             n=51_200, steps=100),
        # a 2D serving request, cubic splines and PIC/FLIP, odd size
        dict(name="collapse2d_mixed", do="job", family="collapse2d", deg=3, flip=0.95, musl=False, mixed=True,
             n=211_777, steps=60),
        # the headline workload, FP64: MUSL, AFLIP, cubic
        dict(name="mui3d_fp64", do="job", family="mui3d", deg=3, flip=-0.95, musl=True, mixed=False, n=1_024_000,
             steps=96),
        # the same, mixed precision
        dict(name="mui3d_mixed", do="job", family="mui3d", deg=3, flip=-0.95, musl=True, mixed=True, n=1_024_000,
             steps=96),
        # the incline workload, FP64: USL, AFLIP, quadratic, Cam-Clay
        dict(name="incline3d_fp64", do="job", family="incline3d", deg=2, flip=-0.95, musl=False, mixed=False,
             n=1_200_000, steps=50),
        # the same, mixed precision
        dict(name="incline3d_mixed", do="job", family="incline3d", deg=2, flip=-0.95, musl=False, mixed=True,
             n=1_200_000, steps=50),
        # the largest serving request: 2M particles, mixed, APIC
        dict(name="dp3d_mixed_2m", do="job", family="dp3d", deg=2, flip=-2.0, musl=False, mixed=True, n=1_999_999,
             steps=50),
        # a frame loop: steps, a frame's rows copied out while the next steps run
        dict(name="frames3d_fp64", do="frames", family="elastic3d", deg=2, flip=0.9, musl=False, mixed=False,
             n=150_001, steps=40),
        # scenes joining a batch: 2D and 3D, 5k to 300k particles, log-spread
        dict(name="batch_mixed", do="batch", deg=2, flip=-2.0, mixed=True, scenes=16, n_min=5_000, n_max=300_000,
             steps=24),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    do = rng.choice(["p2g", "job", "job", "job", "job", "frames", "batch"])
    if do == "p2g":
        return dict(do="p2g", dim=rng.choice([2, 3, 3]), deg=rng.choice([2, 3]), n=size(3_000, 262_144),
                    seed_cells=rng.randint(0, 9))
    mixed = rng.random() < 0.5
    flip = rng.choice([-2.0, -0.95, 0.95])
    if do == "batch":
        lo = size(5_000, 20_000)
        return dict(do="batch", deg=rng.choice([2, 2, 3]), flip=flip, mixed=mixed, scenes=rng.randint(3, 16),
                    n_min=lo, n_max=size(2 * lo, 200_000), steps=rng.randint(8, 24))
    if do == "frames":
        return dict(do="frames", family="elastic3d", deg=rng.choice([2, 3]), flip=flip, musl=rng.random() < 0.3,
                    mixed=False, n=size(8_000, 300_000), steps=rng.randint(16, 48))
    family = rng.choice(["collapse2d", "mui3d", "incline3d", "dp3d"])
    n = size(5_000, 300_000 if family == "collapse2d" else 1_500_000)
    steps = max(8, min(100, int(3e7 / n) + rng.randint(0, 9)))
    return dict(do="job", family=family, deg=rng.choice([2, 3]), flip=flip, musl=family == "mui3d" or rng.random() < 0.2,
                mixed=mixed, n=n, steps=steps)


# ---------------------------------------------------------------------------
# scenes
# ---------------------------------------------------------------------------
def _lattice(lo, cells, dx, n, gen):
    """n particles of a jittered lattice, 2 per cell and axis, +-0.25 dx."""
    h = dx / 2
    axes = [lo[a] + (torch.arange(2 * cells[a], device=DEV, dtype=F64) + 0.5) * h for a in range(len(cells))]
    x = torch.stack([m.reshape(-1) for m in torch.meshgrid(*axes, indexing="ij")], dim=1)[:n]
    return x + (torch.rand(x.shape, generator=gen, device=DEV, dtype=F64) - 0.5) * (0.5 * dx)


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _scene(case, seed, family=None, n=None):
    """Parameters and the mid-flow particle state of one scene (device tensors, matrices [n, row, col])."""
    fam = dict(FAMILIES[family or case["family"]])
    n = n or case["n"]
    d, gen = fam["dim"], _gen(seed)
    base = 0.5 if family == "mui3d" or fam["model"] == "mui" else (1.0 if fam["model"] == "mcc" else 0.2)
    # cells per axis: width, height = aspect * width, depth = width (incline: 0.5 of the length)
    depth = 0.5 if fam["model"] == "mcc" else 1.0
    per = math.ceil(n / 2 ** d)
    nw = max(2, math.ceil((per / (fam["aspect"] * (depth if d == 3 else 1.0))) ** (1.0 / d)))
    cells = [nw, max(2, round(fam["aspect"] * nw))] + ([max(2, round(depth * nw))] if d == 3 else [])
    while cells[0] * cells[1] * (cells[2] if d == 3 else 1) < per:
        cells[0] += 1
    dx = base / nw
    y0 = 0.5 * dx if fam["model"] == "mcc" else 0.0
    lo = [0.0, y0] + ([0.0] if d == 3 else [])
    x = _lattice(lo, cells, dx, n, gen)
    size = [c * dx for c in cells]
    rnd = lambda *s: torch.rand(s, generator=gen, device=DEV, dtype=F64) * 2 - 1  # noqa: E731
    # collapsing flow: spreads sideways, sinks in proportion to height, slower near the floor
    u = 0.6
    rel = [(x[:, a] - lo[a]) / size[a] for a in range(d)]
    grad = torch.zeros(n, d, d, device=DEV, dtype=F64)
    v = torch.zeros(n, d, device=DEV, dtype=F64)
    for a in range(d):
        if a == 1:
            v[:, 1] = -u * rel[1]
            grad[:, 1, 1] = -u / size[1]
        else:
            v[:, a] = u * (rel[a] - 0.5) * (0.2 + rel[1])
            grad[:, a, a] = u / size[a] * (0.2 + rel[1])
            grad[:, a, 1] = u * (rel[a] - 0.5) / size[1]
    v += 0.01 * u * rnd(n, d)
    B = grad * (dx * dx / (3.0 if case["deg"] == 3 else 4.0)) * (1 + 0.05 * rnd(n, d, d))
    # elastic strain: own weight with a lateral share, some shear, 20% noise
    e = fam["rho"] * 9.81 * size[1] / fam["E"] * (1.0 - rel[1]).clamp(min=0.0) + 0.01 * fam["rho"] * 9.81 * dx / fam["E"]
    F = torch.zeros(n, d, d, device=DEV, dtype=F64)
    for a in range(d):
        F[:, a, a] = 1.0 - (0.74 if a == 1 else 0.25) * e
    F[:, 0, 1] = 0.3 * e
    F += 0.2 * e[:, None, None] * rnd(n, d, d)
    sc = torch.zeros(n, 6, device=DEV, dtype=F64)
    if fam["model"] != "elastic":
        sc[:, 0] = 0.05 * rnd(n).abs()
        sc[:, 1] = 0.001 * rnd(n)
    vol = dx ** d / 2 ** d
    g = [0.0, -9.81, 0.0]
    bumps = []
    if fam["model"] == "mcc":
        g = [9.81 * math.sin(math.pi / 6), -9.81 * math.cos(math.pi / 6), 0.0]
        r = _gen(seed + 1000)
        pos = torch.rand(3, 2, generator=r, device=DEV, dtype=F64).tolist()
        bumps = [(base * (0.2 + 1.2 * p[0]), size[2] * p[1] if d == 3 else 0.0, 0.04 * base, 0.15 * base) for p in pos]
    prm = dict(fam, dx=dx, mass=fam["rho"] * vol, vol=vol, gravity=g, bumps=bumps, deg=case["deg"], flip=case["flip"],
               musl=case.get("musl", False), mixed=case["mixed"], n=n)
    return prm, x, v, F, B, sc


def _batch_scenes(case, seed):
    """(family, n) of each scene of a batch: alternately 2D and 3D, sizes log-spread over the range."""
    k = case["scenes"]
    for i in range(k):
        f = i / max(1, k - 1)
        yield ("collapse2d", "dp3d")[i % 2], int(round(case["n_min"] * (case["n_max"] / case["n_min"]) ** f)), seed * 64 + i


def _params(prm):
    p = abi.default_params(prm["dim"], prm["deg"])
    p.precision = abi.PREC_MIXED if prm["mixed"] else abi.PREC_FP64
    p.flip_ratio, p.use_musl = prm["flip"], 1 if prm["musl"] else 0
    p.E, p.nu, p.rho = prm["E"], prm["nu"], prm["rho"]
    p.dx, p.particle_mass, p.particle_volume = prm["dx"], prm["mass"], prm["vol"]
    for a in range(3):
        p.gravity[a] = prm["gravity"][a]
    m = prm["model"]
    if m == "dp":
        p.plastic_model, p.M = abi.PlasticModel.DP, prm["M"]
    elif m == "mui":
        p.plastic_model, p.mu_1, p.mu_2, p.I_ref = abi.PlasticModel.DPMui, prm["mu_1"], prm["mu_2"], 0.279
        p.grain_diameter, p.rho_s = 1e-3, 2500.0
    elif m == "mcc":
        p.plastic_model, p.hardening_law = abi.PlasticModel.MCCVisc, abi.HardeningLaw.ExpoImpl
        p.M, p.beta, p.p0, p.perzyna_exp, p.perzyna_visc = prm["M"], 0.0, prm["p0"], 1.0, prm["visc"]
    return p


def _objects(prm):
    plates, objects = [], []
    if "floor" in prm:
        bc = abi.BC.SlipFree if prm["floor"][0] == "slipfree" else abi.BC.SlipStick
        plates = [abi.make_plate(0.0, abi.PlateType.bottom, bc, prm["floor"][1])]
    if prm["bumps"]:
        q = [0.0, float(len(prm["bumps"]))]
        for b in prm["bumps"]:
            q += list(b)
        objects = [abi.make_object(abi.ObjectKind.TerrainGauss, abi.BC.SlipFree, 0.45, q)]
    return plates, objects


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
_PD = C.POINTER(C.c_double)


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h


def _ptr(t):
    return C.cast(t.data_ptr(), _PD)


class _Job:
    """One scene: its context, the state to start from and the buffers it is read into, in pinned host memory."""

    def __init__(self, case, scene, fields=None):
        prm, x, v, F, B, sc = scene
        n, d = x.shape
        col = lambda m: m.transpose(1, 2).contiguous()  # noqa: E731  matrices are column-major at the boundary
        self.steps, self.mixed = case["steps"], prm["mixed"]
        self.host = [_pinned(t) for t in (x, v, col(F), col(B), sc)]
        self.fields = fields or (("x", "v") if prm["mixed"] else FIELDS[prm["model"]])
        shape = {"x": (n, d), "v": (n, d), "F": (n, d, d), "B": (n, d, d), "scalars": (n, 6)}
        self.out = {k: torch.empty(shape[k], dtype=F64, pin_memory=True) for k in self.fields}
        self.sim = GpuSim(_params(prm))
        self.upload()
        self.sim.set_objects(*_objects(prm))

    def upload(self):
        self.sim.upload(*(t.numpy() for t in self.host))

    def read(self):
        got = [_ptr(self.out[k]) if k in self.out else None for k in ("x", "v", "F", "B", "scalars")]
        if self.sim.lib.mtr_download(self.sim.h, *got):
            raise RuntimeError(self.sim.lib.mtr_last_error().decode())
        if self.mixed:  # the velocity as the mixed form keeps it
            return {"x": self.out["x"], "v": self.out["v"].float()}
        return dict(self.out)


def prepare(case, seed):
    if case["do"] == "p2g":
        return _prepare_p2g(case, seed)
    if case["do"] == "batch":
        jobs = [_Job(case, _scene(case, s, family=f, n=n), ("x", "v")) for f, n, s in _batch_scenes(case, seed)]
        return {"do": "batch", "jobs": jobs, "batch": GpuBatch([j.sim for j in jobs]), "steps": case["steps"]}
    return {"do": case["do"], "job": _Job(case, _scene(case, seed))}


def run(state):
    if state["do"] == "p2g":
        return _run_p2g(state)
    if state["do"] == "batch":
        jobs = state["jobs"]
        for j in jobs:
            j.upload()
        state["batch"].set_members([j.sim for j in jobs])
        state["batch"].step(state["steps"])
        return [j.read() for j in jobs]
    job = state["job"]
    job.upload()
    if state["do"] == "frames":  # the frame is copied and taken over while the second half steps
        half = job.steps // 2
        job.sim.step(half)
        job.sim.frame_begin()
        job.sim.step(job.steps - half)
        rows, _, _ = job.sim.frame_wait()
        return dict(job.read(), rows=rows)
    job.sim.step(job.steps)
    return job.read()


def _p2g_scene(case, seed):
    d, n = case["dim"], case["n"]
    gen = _gen(seed)
    per = math.ceil(n / 2 ** d)
    c0 = max(2, math.ceil(per ** (1.0 / d)))
    cells = [c0 + (case["seed_cells"] % 3 if a == 0 else 0) for a in range(d)]
    while math.prod(cells) < per:
        cells[0] += 1
    dx = 0.01
    x = _lattice([0.0] * d, cells, dx, n, gen)
    v = torch.randn(n, d, generator=gen, device=DEV, dtype=F64)
    B = torch.randn(n, d, d, generator=gen, device=DEV, dtype=F64) * (5.0 * dx * dx)
    axes = [torch.arange(-3, c + 5, device=DEV, dtype=F64) * dx for c in cells]
    return dx, x, v, B, axes


def _prepare_p2g(case, seed):
    dx, x, v, B, axes = _p2g_scene(case, seed)
    d, n = case["dim"], case["n"]
    p = abi.default_params(d, case["deg"])
    p.dx, p.flip_ratio, p.particle_mass = dx, -2.0, 1e-3
    dims = [a.numel() for a in axes]
    G = math.prod(dims)
    s = {"do": "p2g", "lib": load_library(), "p": p, "n": n, "x": x.t().contiguous(), "v": v.t().contiguous(),
         "B": B.reshape(n, d * d).t().contiguous(), "axes": axes + [axes[0]] * (3 - d),
         "dims": (C.c_uint32 * 3)(*(dims + [1] * (3 - d))), "mass": torch.empty(G, dtype=F64, device=DEV),
         "vel": torch.empty(d, G, dtype=F64, device=DEV), "status": torch.empty(1, dtype=torch.int32, device=DEV)}
    return s


def _run_p2g(s):
    q = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    rc = s["lib"].mtr_p2g_noalloc(C.byref(s["p"]), q(s["x"]), q(s["v"]), q(s["B"]), s["n"], *(q(a) for a in s["axes"]),
                                  s["dims"], q(s["mass"]), q(s["vel"]), q(s["status"]),
                                  C.c_void_p(torch.cuda.current_stream().cuda_stream))
    if rc:
        raise RuntimeError("mtr_p2g_noalloc returned %d" % rc)
    return {"mass": s["mass"], "v": s["vel"], "status": s["status"]}


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _step_work(dim, n, mixed, musl):
    """Bytes and flops of one step: the particle state read once and written once (positions 8 B, the rest in the
    storage type), and the multiply-adds of the sums over the 4^dim stencil nodes with their factors shared:
    scatter of mass, momentum and force, gather of velocity, flip, affine matrix and gradient."""
    r = 4 if mixed else 8
    state = 8 * dim + r * (dim + 2 * dim * dim + (6 if dim == 3 else 3))
    s = 4 ** dim
    fma = s * ((1 + 4 * dim) + 4 * dim) + (s * 2 * dim + s * dim if musl else 0)
    return n * (2 * state + 2 * r * 6 + 8), 2 * n * (fma + 300)


def work(case):
    if case["do"] == "p2g":
        d, n = case["dim"], case["n"]
        c = max(2, math.ceil(math.ceil(n / 2 ** d) ** (1.0 / d))) + 8
        return {"bytes": 8 * (n * (2 * d + d * d) + c ** d * (1 + d)), "flops": 2 * n * 4 ** d * (1 + 2 * d)}
    if case["do"] == "batch":
        per = [_step_work(2 if f == "collapse2d" else 3, n, case["mixed"], False) for f, n, _ in _batch_scenes(case, 0)]
        return {"bytes": case["steps"] * sum(b for b, _ in per), "flops": case["steps"] * sum(f for _, f in per)}
    b, f = _step_work(FAMILIES[case["family"]]["dim"], case["n"], case["mixed"], case["musl"])
    return {"bytes": case["steps"] * b, "flops": case["steps"] * f}


# ---------------------------------------------------------------------------
# the step in plain FP64 torch
# ---------------------------------------------------------------------------
def _spline(u, deg):
    a, s = u.abs(), torch.sign(u)
    if deg == 3:
        w = torch.where(a < 1, 0.5 * a ** 3 - a * a + 2.0 / 3.0, torch.where(a < 2, (2 - a) ** 3 / 6.0, 0.0 * a))
        g = torch.where(a < 1, u * (1.5 * a - 2.0), torch.where(a < 2, -0.5 * s * (2 - a) ** 2, 0.0 * a))
    else:
        w = torch.where(a < 0.5, 0.75 - a * a, torch.where(a < 1.5, 0.5 * (1.5 - a) ** 2, 0.0 * a))
        g = torch.where(a < 0.5, -2.0 * u, torch.where(a < 1.5, u - 1.5 * s, 0.0 * a))
    return w, g


def _stencil(x, org, dx, dims, deg):
    """Node index [n, S], weights [n, S], gradients [n, S, d] and offsets x_i - x_p [n, S, d] of each particle."""
    n, d = x.shape
    base = torch.floor((x - org) / dx).long() - 1
    o = torch.arange(4, device=DEV)
    node = base[:, :, None] + o  # [n, d, 4]
    pos = org[None, :, None] + node.to(F64) * dx
    w, g = _spline((x[:, :, None] - pos) / dx, deg)
    g = g / dx
    off = pos - x[:, :, None]
    lin, W, G, O = node[:, 0], w[:, 0], [g[:, 0]] + [w[:, 0]] * (d - 1), [off[:, 0]]
    for a in range(1, d):
        m = lin.shape[1]
        lin = (lin[:, :, None] * dims[a] + node[:, a][:, None, :]).reshape(n, -1)
        W = (W[:, :, None] * w[:, a][:, None, :]).reshape(n, -1)
        G = [(G[b][:, :, None] * (g if b == a else w)[:, a][:, None, :]).reshape(n, -1) for b in range(d)]
        O = [t[:, :, None].expand(n, m, 4).reshape(n, -1) for t in O] + [off[:, a][:, None, :].expand(n, m, 4).reshape(n, -1)]
    return lin, W, torch.stack(G, -1), torch.stack(O, -1)


def _eig(A):
    """Eigenvalues [n, d] and vectors [n, d, d] (columns) of symmetric matrices: cyclic Jacobi."""
    n, d, _ = A.shape
    A = A.clone()
    U = torch.eye(d, device=DEV, dtype=F64).repeat(n, 1, 1)
    for _ in range(8 if d == 3 else 2):
        for p in range(d):
            for q in range(p + 1, d):
                apq = A[:, p, q]
                tau = (A[:, q, q] - A[:, p, p]) / (2 * torch.where(apq == 0, torch.ones_like(apq), apq))
                t = torch.where(tau >= 0, 1.0, -1.0).to(F64) / (tau.abs() + torch.sqrt(1 + tau * tau))
                t = torch.where(apq == 0, torch.zeros_like(t), t)
                c = 1 / torch.sqrt(1 + t * t)
                s = t * c
                for M, right in ((A, True), (A, False), (U, True)):
                    a, b = (M[:, :, p], M[:, :, q]) if right else (M[:, p, :], M[:, q, :])
                    a, b = c[:, None] * a - s[:, None] * b, s[:, None] * a + c[:, None] * b
                    if right:
                        M[:, :, p], M[:, :, q] = a, b
                    else:
                        M[:, p, :], M[:, q, :] = a, b
    return torch.diagonal(A, dim1=1, dim2=2), U


def _camclay(p, q, M, p0, K, mu):
    """Implicit Cam-Clay projection (beta = 0, no hardening) of trial (p, q) outside the ellipse: Newton on the
    volumetric plastic strain with the limited step of the method, in stresses scaled by p0."""
    sc = 1.0 / p0
    pt, qt, K, mu = p * sc, q * sc, K * sc, mu * sc
    right = torch.where(pt > 0.5, 1, 0)
    epv, pc, qc = torch.zeros_like(pt), pt.clone(), qt.clone()
    live = torch.ones_like(pt, dtype=torch.bool)
    early = torch.zeros_like(live)
    mid = 0.5
    for it in range(30):
        hit = live & ((pc - mid).abs() < 1e-4)
        early |= hit
        live &= ~hit
        if not bool(live.any()):
            break
        pc = torch.where(live, epv * K + pt, pc)
        den = 2 * K * M * M * pc - M * M * K
        dg = (pt - pc) / den
        qd = 1 + 2 * mu * dg
        qc = torch.where(live, qt / qd, qc)
        y = M * M * (pc - 1) * pc + qc * qc
        if it > 5:
            live &= ~(y.abs() < 1e-4)
        ddg = -K / den - (pt - pc) * (2 * K * K * M * M) / (den * den)
        dq = -qt * 2 * mu * ddg / (qd * qd)
        dy = M * M * K * pc + M * M * (pc - 1) * K + 2 * qc * dq
        delta = y / dy
        new, todo, scale = epv.clone(), live.clone(), 1.0
        for _ in range(32):
            test = epv - scale * delta
            pp = K * test + pt
            val = 2 * pp - 1
            a = todo & ((pp - mid).abs() <= 1e-5)
            b = todo & ~a & (((right == 1) & ((pp < mid) | (pt < mid))) | ((right == 0) & ((pp > mid) | (pt > mid))))
            sg = torch.sign(-test)
            c = todo & ~a & ~b & ((sg == torch.sign(val)) | (sg == 0))
            new = torch.where(a | c, test, new)
            right = torch.where(b, torch.full_like(right, -1), right)
            todo &= ~(a | b | c)
            scale *= 0.5
            if not bool(todo.any()):
                break
        epv = torch.where(live, new, epv)
    pc = torch.where(early, pc, pc.clamp(min=0.0, max=1.0))
    return pc / sc, M * torch.sqrt(((1 - pc) * pc).clamp(min=0.0)) / sc


def _return_map(prm, dt, F, sc):
    """F (trial -> new), scalars and the Kirchhoff stress."""
    n, d, _ = F.shape
    lam = prm["nu"] * prm["E"] / ((1 + prm["nu"]) * (1 - 2 * prm["nu"]))
    mu = prm["E"] / (2 * (1 + prm["nu"]))
    K = lam + 2 * mu / d
    ev, U = _eig(F @ F.transpose(1, 2))
    S = torch.sqrt(ev)
    h = torch.log(S)
    model = prm["model"]
    if model != "elastic":
        qpre, dpre = 1 / math.sqrt(2.0), math.sqrt(2.0)
        emu, fmu = 2 * qpre * mu, 2 * qpre / dpre * mu
        tr = h.sum(1)
        dev = h - (tr / d)[:, None]
        hdn = dev.norm(dim=1)
        dev = dev / torch.where(hdn > 0, hdn, torch.ones_like(hdn))[:, None]
        p, q = -K * tr, emu * hdn
        new = h.clone()
        sc = sc.clone()
        sc[:, 3] = 0.0
        if model == "dp":
            qy = prm["M"] * p
            tip = qy < 1e-10
            dg = dpre * (hdn - qy / emu)
            sh = ~tip & (dg > 0)
            new = torch.where(tip[:, None], torch.zeros_like(h), new)
            new = torch.where(sh[:, None], h - (dg / dpre)[:, None] * dev, new)
            dg = torch.where(tip, dpre * hdn, torch.where(sh, dg, torch.zeros_like(dg)))
            sc[:, 3] = dg / dt
            sc[:, 0] += dg / dpre
            sc[:, 1] += torch.where(tip, -p / K, torch.zeros_like(p))
        elif model == "mui":
            m1, m2, tol = prm["mu_1"], prm["mu_2"], 1e-5
            fq = 0.279 / (1e-3 * math.sqrt(2500.0))
            ps = p - K * sc[:, 2]
            tip = ps < 0
            new = torch.where(tip[:, None], torch.zeros_like(h), new)
            sc[:, 0] += torch.where(tip, hdn, torch.zeros_like(hdn))
            sc[:, 1] += torch.where(tip, -p / K, torch.zeros_like(p))
            sc[:, 2] = torch.where(tip, sc[:, 2] - p / K, torch.zeros_like(p))
            qy = m1 * ps
            sh = (ps > 0) & (q > qy + tol)
            r = torch.sqrt((ps + tol).clamp(min=0.0))
            a = fmu * dt
            b = p * (m2 - m1) + a * fq * r - (q - qy)
            c = -(q - qy) * fq * r
            g = dt * (-b + torch.sqrt((b * b - 4 * a * c).clamp(min=0.0))) / (2 * a)
            g = torch.where(sh, g, torch.zeros_like(g))
            new = torch.where(sh[:, None], h - (g / dpre)[:, None] * dev, new)
            sc[:, 0] += g / dpre
        else:
            M, p0 = prm["M"], prm["p0"]
            out = M * M * (p * p - p0 * p) + q * q > 0
            pn, qy = p.clone(), q.clone()
            if bool(out.any()):
                pn[out], qy[out] = _camclay(p[out], q[out], M, p0, K, mu)
            dg = ((q - qy) / (fmu + qy * prm["visc"] / dt)).clamp(min=0.0)
            qn = torch.maximum(qy, q - fmu * dg)
            ep = pn / (K * d)
            new = torch.where(out[:, None], (qn / emu)[:, None] * dev - ep[:, None], h)
            sc[:, 1] += torch.where(out, tr + d * ep, torch.zeros_like(tr))
            dg = torch.where(out, (q - qn) / fmu, torch.zeros_like(q))
            sc[:, 0] += dg / dpre
            sc[:, 3] = dg / dt
        V = F.transpose(1, 2) @ U / S[:, None, :]
        F = (U * torch.exp(new)[:, None, :]) @ V.transpose(1, 2)
        h = new
    tau = (U * (2 * mu * h + lam * h.sum(1, keepdim=True))[:, None, :]) @ U.transpose(1, 2)
    return F, sc, tau


def _collide(prm, X, v):
    """The bumps (SlipFree 0.45) or the floor plate, on node velocities v at node positions X advanced by dt v."""
    d = v.shape[1]
    if prm["bumps"]:
        s, gx, gz = torch.zeros_like(X[:, 0]), torch.zeros_like(X[:, 0]), torch.zeros_like(X[:, 0])
        for bx, bz, hb, sb in prm["bumps"]:
            rx, rz = X[:, 0] - bx, X[:, 2] - bz
            e = hb * torch.exp(-(rx * rx + rz * rz) / (2 * sb * sb))
            s, gx, gz = s + e, gx - e * rx / (sb * sb), gz - e * rz / (sb * sb)
        nrm = torch.stack([-gx, torch.ones_like(gx), -gz], 1)
        nrm = nrm / nrm.norm(dim=1, keepdim=True)
        dot = (v * nrm).sum(1)
        vt = v - dot[:, None] * nrm
        nt = vt.norm(dim=1)
        slide = vt * (1 + dot * 0.45 / torch.where(nt > 0, nt, torch.ones_like(nt)))[:, None]
        slide = torch.where((-dot * 0.45 < nt)[:, None], slide, torch.zeros_like(v))
        return torch.where(((X[:, 1] < s) & (dot < 0))[:, None], slide, v)
    kind, mu = prm["floor"]
    hit = X[:, 1] <= 0
    if kind == "slipfree":
        hit &= v[:, 1] < 0
    tang = [a for a in range(d) if a != 1]
    vt = v[:, tang].norm(dim=1)
    lim = mu * v[:, 1].abs()
    f = torch.where(vt > lim, (vt - lim) / torch.where(vt > 0, vt, torch.ones_like(vt)), torch.zeros_like(vt))
    w = v * f[:, None]
    if d == 3:  # the plate's second tangential component is scaled with the first one's reduced value
        a, b = v[:, 0], v[:, 2]
        one = torch.ones_like(a)
        a2 = torch.sign(a) * (vt - lim) / torch.sqrt(1 + b * b / torch.where(a != 0, a * a, one))
        b2 = torch.sign(b) * (vt - lim) / torch.sqrt(1 + a2 * a2 / torch.where(b != 0, b * b, one))
        slip = vt > lim
        w[:, 0] = torch.where(slip, torch.where(a != 0, a2, 0 * a), 0 * a)
        w[:, 2] = torch.where(slip, torch.where(b != 0, b2, 0 * b), 0 * b)
    w[:, 1] = 0
    return torch.where(hit[:, None], w, v)


def _advance(prm, x, v, F, B, sc, steps, at=None):
    """`steps` steps of the scene; returns the state and, with `at`, the frame's rows after that many steps."""
    n, d = x.shape
    dx, deg, fr = prm["dx"], prm["deg"], prm["flip"]
    wave = math.sqrt(prm["E"] / prm["rho"])
    g = torch.tensor(prm["gravity"][:d], device=DEV, dtype=F64)
    dinv = (3.0 if deg == 3 else 4.0) / (dx * dx)
    time, rows = 0.0, None
    tau = _return_map(dict(prm, model="elastic"), 1.0, F, sc)[2]
    lo0, hi0 = x.min(0).values, x.max(0).values
    for step in range(steps):
        speed = float(v.norm(dim=1).max())
        dt = min(min(0.5 * dx / speed if speed > 1e-10 else 1e30, 0.5 * dx / wave), 1.0 - time)
        mn, mx = x.min(0).values, x.max(0).values
        f = lambda t: torch.floor((t / dx - 1e-8).clamp(min=0.0)) * dx  # noqa: E731
        low = lo0 - 2 * dx + torch.where(mn > lo0, f(mn - lo0), -f(lo0 - mn))
        high = hi0 + 2 * dx + torch.where(mx < hi0, -f(hi0 - mx), f(mx - hi0))
        dims = [int(c) + 3 for c in ((high - low) / dx).ceil().tolist()]
        lin, W, G, O = _stencil(x, low, dx, dims, deg)
        nodes = math.prod(dims)
        val = v[:, None, :]
        if fr < 0:
            val = val + dinv * torch.einsum("nab,nsb->nsa", B, O)
        flat = lin.reshape(-1)
        m = torch.zeros(nodes, device=DEV, dtype=F64).index_add_(0, flat, W.reshape(-1))
        mom = torch.zeros(nodes, d, device=DEV, dtype=F64).index_add_(0, flat, (W[:, :, None] * val).reshape(-1, d))
        force = torch.zeros(nodes, d, device=DEV, dtype=F64).index_add_(
            0, flat, torch.einsum("nab,nsb->nsa", tau, G).reshape(-1, d))
        live = m > 0
        ms = torch.where(live, m, torch.ones_like(m))[:, None]
        old = mom / ms
        vi = old - dt * prm["vol"] * force / (ms * prm["mass"]) + dt * g
        ax = torch.meshgrid(*[low[a] + torch.arange(dims[a], device=DEV, dtype=F64) * dx for a in range(d)], indexing="ij")
        X = torch.stack([t.reshape(-1) for t in ax], 1) + dt * vi
        vi = torch.where(live[:, None], _collide(prm, X, vi), torch.zeros_like(vi))
        flip = torch.where(live[:, None], vi - old, torch.zeros_like(vi))
        gi = vi[lin]
        pic = (W[:, :, None] * gi).sum(1)
        fl = (W[:, :, None] * flip[lin]).sum(1) if fr >= -1 else 0.0
        vn = pic if fr < -1 else (abs(fr) * (v + fl) + (1 - abs(fr)) * pic)
        Bn = torch.einsum("ns,nsa,nsb->nab", W, gi, O) if fr < 0 else torch.zeros_like(B)
        if prm["musl"]:
            val = vn[:, None, :] + (dinv * torch.einsum("nab,nsb->nsa", Bn, O) if fr < 0 else 0.0)
            v2 = torch.zeros(nodes, d, device=DEV, dtype=F64).index_add_(0, flat, (W[:, :, None] * val).reshape(-1, d))
            gi = (v2 / ms)[lin]
        gradv = torch.einsum("nsa,nsb->nab", gi, G)
        F, sc, tau = _return_map(prm, dt, F + dt * (gradv @ F), sc)
        x, v, B = x + dt * pic, vn, Bn
        time += dt
        if at is not None and step + 1 == at:
            p = -torch.diagonal(tau, dim1=1, dim2=2).sum(1) / d
            dv = tau + p[:, None, None] * torch.eye(d, device=DEV, dtype=F64)
            rows = torch.cat([x, v, p[:, None], torch.sqrt(0.5 * (dv * dv).sum((1, 2)))[:, None], torch.linalg.det(F)[:, None]], 1)
    return {"x": x, "v": v, "F": F.transpose(1, 2).contiguous(), "B": B.transpose(1, 2).contiguous(), "scalars": sc}, rows


def exact(case, seed):
    if case["do"] == "p2g":
        dx, x, v, B, axes = _p2g_scene(case, seed)
        d = case["dim"]
        dims = [a.numel() for a in axes]
        org = torch.stack([a[0] for a in axes])
        lin, W, _, O = _stencil(x, org, dx, dims, case["deg"])
        val = v[:, None, :] + (3.0 if case["deg"] == 3 else 4.0) / (dx * dx) * torch.einsum("nab,nsb->nsa", B, O)
        flat, G = lin.reshape(-1), math.prod(dims)
        m = torch.zeros(G, device=DEV, dtype=F64).index_add_(0, flat, W.reshape(-1))
        mom = torch.zeros(G, d, device=DEV, dtype=F64).index_add_(0, flat, (W[:, :, None] * val).reshape(-1, d))
        vel = torch.where((m > 0)[:, None], mom / torch.where(m > 0, m, torch.ones_like(m))[:, None], torch.zeros_like(mom))
        return {"mass": m * 1e-3, "v": vel.t().contiguous(), "status": None}
    if case["do"] == "batch":
        out = []
        for f, n, s in _batch_scenes(case, seed):
            got, _ = _advance(*_scene(case, s, family=f, n=n), case["steps"])
            out.append({"x": got["x"], "v": got["v"].float() if case["mixed"] else got["v"]})
        return out
    scene = _scene(case, seed)
    prm = scene[0]
    half = case["steps"] // 2 if case["do"] == "frames" else None
    got, rows = _advance(*scene, case["steps"], at=half)
    if case["mixed"]:
        return {"x": got["x"], "v": got["v"].float()}
    out = {k: got[k] for k in FIELDS[prm["model"]]}
    return dict(out, rows=rows) if rows is not None else out
