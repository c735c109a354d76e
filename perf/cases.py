"""Performance cases: the work a user of this package has it do, through its public entry points.

A case is one job: the state is uploaded from pinned host memory, the boundary
conditions are applied, a number of SSP-RK3 steps is taken, and the state is
downloaded again -- what a program does between two checkpoints.  How the steps
are taken differs: `run` (whole steps replayed from a CUDA graph), the
reference's own time loop call by call (`percall`), or many independent blocks
together (`batch`).  One kind is not a solve: `train`, a training step of the
learned sensor.

The FP64 path's state comes back as it is, in double precision; the FP32-flux
precisions (split, hybrid) come back in single precision, as a program keeps
fields whose fluxes were formed in FP32.

`exact` restates each job in plain torch, in double precision, with WENO5 on
every face: the values all three precisions approximate.
"""
import functools
import math
from pathlib import Path

import numpy as np
import torch

import cbns3d_cuda_b200 as cb
from cbns3d_cuda_b200 import CBNS_Q, Batch, Block, cases as grids, make_params, sensor

GAMMA = 1.4
NG = 2
PRECISION = {"fp64": cb.PREC_FP64, "split": cb.PREC_SPLIT, "hybrid": cb.PREC_HYBRID}
WEIGHTS = Path(cb.__file__).resolve().parent / "data" / "sensor_weights.npz"


def listed():
    return [
        # the small isentropic vortex on its own grid: few CTAs, short kernels, so launches and latency count
        dict(name="vortex_64x32x16_fp64", kind="run", flow="vortex", IM=64, JM=32, KM=16, precision="fp64",
             viscous=False, bc="reference", steps=100),
        # the reference's time loop call by call with dt read back every step, on an odd, ragged grid
        dict(name="percall_97x61x45_fp64", kind="percall", flow="vortex", IM=97, JM=61, KM=45, precision="fp64",
             viscous=False, bc="reference", steps=30),
        # the plain path at full size: the parity path of the shock/vortex configuration
        dict(name="shock_256x256x128_fp64", kind="run", flow="shock", IM=256, JM=256, KM=128, precision="fp64",
             viscous=False, bc="reference", steps=20),
        # the precision form: FP32 fluxes on every face, a blast on an uneven odd grid
        dict(name="blast_193x161x129_split", kind="run", flow="blast", IM=193, JM=161, KM=129, precision="split",
             viscous=False, bc="reference", steps=40),
        # the flagship: learned-sensor hybrid on the shock/vortex configuration, the largest job
        dict(name="shock_256x256x128_hybrid", kind="run", flow="shock", IM=256, JM=256, KM=128, precision="hybrid",
             viscous=False, bc="reference", steps=80),
        # a hybrid block of about a million points, odd in every direction
        dict(name="blast_129x113x97_hybrid", kind="run", flow="blast", IM=129, JM=113, KM=97, precision="hybrid",
             viscous=False, bc="reference", steps=60),
        # the host driver's loop over the hybrid path at a middle size
        dict(name="percall_192x192x96_hybrid", kind="percall", flow="shock", IM=192, JM=192, KM=96,
             precision="hybrid", viscous=False, bc="reference", steps=30),
        # the NACA 0012 O-grid, viscous: four points along the span, many short kernels per step
        dict(name="naca_384x128x4_fp64_viscous", kind="run", flow="naca", IM=392, JM=128, KM=4, precision="fp64",
             viscous=True, bc="ogrid", steps=200),
        # one viscous block of the largest batch size in double precision
        dict(name="vortex_128x64x64_fp64_viscous", kind="run", flow="vortex", IM=128, JM=64, KM=64,
             precision="fp64", viscous=True, bc="farfield", steps=40),
        # the batched-blocks configuration: 64 viscous blocks of uneven size, learned-sensor hybrid
        dict(name="batch_64_hybrid_viscous", kind="batch", flow="vortex", blocks=64, lo=32, precision="hybrid",
             viscous=True, bc="farfield", steps=20),
        # a smaller batch on the plain inviscid path
        dict(name="batch_12_fp64", kind="batch", flow="vortex", blocks=12, lo=32, precision="fp64", viscous=False,
             bc="farfield", steps=10),
        # one training step of the sensor at the training loop's default batch
        dict(name="train_16384", kind="train", samples=16384),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "percall", "percall", "batch", "train"])
    if kind == "train":
        return dict(kind="train", samples=_log_int(rng, 500, 2000000))
    if kind == "batch":
        precision = rng.choice(["fp64", "split", "hybrid", "hybrid"])
        return dict(kind="batch", flow="vortex", blocks=rng.randint(2, 24), lo=rng.randint(16, 40),
                    precision=precision, viscous=rng.random() < 0.6, bc="farfield", steps=rng.randint(5, 20))
    flow = rng.choice(["vortex", "vortex", "shock", "blast", "naca"])
    viscous, bc, precision = False, "reference", rng.choice(["fp64", "split", "hybrid"])
    if flow == "naca":
        IM, JM, KM, precision, viscous, bc = 8 + rng.randint(360, 400), rng.randint(120, 136), rng.randint(4, 6), \
            rng.choice(["fp64", "split"]), True, "ogrid"
    else:
        lo = 48 if flow == "shock" else 24
        IM, JM, KM = _log_int(rng, lo, 256), _log_int(rng, lo, 200), _log_int(rng, 16, 128)
        if flow == "vortex":
            bc = rng.choice(["reference", "farfield"])
            viscous = bc == "farfield" and rng.random() < 0.7
    steps = max(5, min(100, int(1.2e8 / (IM * JM * KM))))
    return dict(kind=kind, flow=flow, IM=IM, JM=JM, KM=KM, precision=precision, viscous=viscous, bc=bc, steps=steps)


# ---------------------------------------------------------------- inputs, from the seed alone
def _conservative(rho, u, v, p):
    E = p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)
    return torch.stack([rho, rho * u, rho * v, torch.zeros_like(rho), E], dim=-1)


def _ghosted(a):
    """A (KM, JM, IM) coordinate extended by NG layers on every side by odd reflection."""
    for dim in range(3):
        n = a.shape[dim]
        lo = 2 * a.narrow(dim, 0, 1) - a.narrow(dim, 1, NG).flip(dim)
        hi = 2 * a.narrow(dim, n - 1, 1) - a.narrow(dim, n - 1 - NG, NG).flip(dim)
        a = torch.cat([lo, a, hi], dim=dim)
    return a


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


@functools.lru_cache(maxsize=70)
def _grid(flow, *shape):
    """The grid of a flow, (x, y, z) of shape (KM, JM, IM); the O-grid as a whole case.  The same for every seed."""
    if flow == "naca":
        return grids.case_naca_ogrid(shape[0] - 8, shape[1], shape[2], grid="marched", start="potential")
    make = {"vortex": grids.perturbed_box, "blast": grids.stretched_skewed_box, "shock": grids.skewed_channel}[flow]
    return make(*shape)


def _block_inputs(c, rng):
    """Grid (numpy, (KM, JM, IM)), make_params keywords and ghosted initial state (torch) of one block."""
    shape = (c["IM"], c["JM"], c["KM"])
    dev = _device()
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    prm = dict(CFL=0.5, gamma=GAMMA, i_begin=1, i_end=0, T_inf=288.15, viscous=c["viscous"])
    if c["bc"] == "farfield":
        prm["bc_mode"] = cb.BC_FARFIELD
    if c["flow"] == "naca":
        case = _grid("naca", *shape)
        Q = to(case.Q0)
        # a seeded density disturbance of 1e-4, the same at every span station and across the seam
        w = rng.uniform(1, 4)
        Q = Q * (1.0 + 1e-4 * torch.sin(w * (to(_pad(case.x)) + to(_pad(case.y))))[..., None])
        return (case.x, case.y, case.z), dict(case.params), Q
    if c["flow"] == "vortex":
        x, y, z = _grid("vortex", *shape)
        xg, yg = _ghosted(to(x)), _ghosted(to(y))
        batch = c["kind"] == "batch"
        M = rng.uniform(0.3, 2.0) if batch else rng.uniform(0.45, 0.55)
        beta = rng.uniform(1.0, 5.0) if batch else rng.uniform(4.5, 5.0)
        xc, yc = rng.uniform(2.5, 7.5), rng.uniform(1.5, 3.5)
        dx, dy = xg - xc, yg - yc
        r2, U = dx * dx + dy * dy, M * math.sqrt(GAMMA)
        f = beta / (2 * math.pi) * torch.exp(0.5 * (1.0 - r2))
        T = 1.0 - (GAMMA - 1.0) * beta ** 2 / (8.0 * GAMMA * math.pi ** 2) * torch.exp(1.0 - r2)
        rho = T ** (1.0 / (GAMMA - 1.0))
        prm.update(Mach=M, Re=math.exp(rng.uniform(math.log(1e3), math.log(1e5))))
        return (x, y, z), prm, _conservative(rho, 1.0 - f * dy / U, f * dx / U, rho * T / (U * U))
    if c["flow"] == "blast":
        x, y, z = _grid("blast", *shape)
        xg, yg, zg = (_ghosted(to(a)) for a in (x, y, z))
        r = torch.sqrt(xg * xg + yg * yg + zg * zg)
        R, ratio = rng.uniform(0.18, 0.22), rng.uniform(60.0, 100.0)
        p = 0.1 * (1.0 + (ratio - 1.0) * 0.5 * (1.0 - torch.tanh((r - R) / 0.03)))
        prm.update(Mach=math.sqrt(1.0 / (GAMMA * 0.1)))
        zero = torch.zeros_like(p)
        return (x, y, z), prm, _conservative(torch.ones_like(p), zero, zero, p)
    # a stationary Mach 1.2 shock at x = 0.5 and a vortex moving into it
    x, y, z = _grid("shock", *shape)
    xg, yg = _ghosted(to(x)), _ghosted(to(y))
    g, Ms, eps, rc, a = GAMMA, 1.2, rng.uniform(0.25, 0.35), 0.075, 0.204
    xc, yc = rng.uniform(0.24, 0.32), rng.uniform(0.4, 0.6)
    p1 = 1.0 / (g * Ms * Ms)
    r21, p21 = (g + 1) * Ms * Ms / ((g - 1) * Ms * Ms + 2), 1 + 2 * g / (g + 1) * (Ms * Ms - 1)
    dx, dy = (xg - xc) / rc, (yg - yc) / rc
    t2, c1 = dx * dx + dy * dy, math.sqrt(g * p1)
    ut = eps * c1 * torch.exp(a * (1.0 - t2))
    T = 1.0 - (g - 1) * eps * eps * g / (4 * a * g) * torch.exp(2 * a * (1 - t2))
    up = xg < 0.5
    const = lambda v: torch.full_like(xg, v)  # noqa: E731
    rho = torch.where(up, T ** (1 / (g - 1)), const(r21))
    u = torch.where(up, 1.0 - ut * dy, const(1.0 / r21))
    v = torch.where(up, ut * dx, const(0.0))
    p = torch.where(up, p1 * T ** (g / (g - 1)), const(p1 * p21))
    prm.update(Mach=Ms)
    return (x, y, z), prm, _conservative(rho, u, v, p)


def _pad(a):
    return np.pad(a, NG, mode="edge")


def _blocks(case, seed):
    """The blocks of a case with their inputs."""
    rng = np.random.default_rng(seed)
    if case["kind"] != "batch":
        return [(case, *_block_inputs(case, rng))]
    # the sizes belong to the case, the flows to the seed
    sizes = np.random.default_rng(1000 + case["blocks"])
    lo, out = case["lo"], []
    for _ in range(case["blocks"]):
        c = dict(case, IM=int(sizes.integers(lo, 4 * lo + 1)), JM=int(sizes.integers(lo, 2 * lo + 1)),
                 KM=int(sizes.integers(lo, 2 * lo + 1)))
        out.append((c, *_block_inputs(c, rng)))
    return out


def _training_set(case, seed):
    """Sensor features (the log-compressed jumps, most of them small) and labels."""
    g = torch.Generator(device="cpu").manual_seed(int(seed))
    n = case["samples"]
    X = torch.randn(n, 15, generator=g) * torch.exp(torch.randn(n, 1, generator=g) - 1.0)
    Y = (X[:, 2].abs() + X[:, 7].abs() > 1.0).to(torch.uint8)
    return X, Y, torch.from_numpy(sensor.init_params(seed))


# ---------------------------------------------------------------- the jobs
class _Job:
    """One block with its pinned host buffers."""

    def __init__(self, c, grid, prm, Q):
        self.c = c
        self.block = Block(make_params(c["IM"], c["JM"], c["KM"], precision=PRECISION[c["precision"]], **prm))
        self.block.calc_metrics(*grid)
        if c["precision"] == "hybrid":
            w = np.load(WEIGHTS)
            self.block.sensor_load(w["params"], float(w["tau"]))
        self.hin = torch.empty(Q.numel(), dtype=torch.float64, pin_memory=True)
        self.hin.copy_(Q.reshape(-1))
        self.hout = torch.empty_like(self.hin, pin_memory=True)
        self.h32 = None if c["precision"] == "fp64" else torch.empty(Q.numel(), dtype=torch.float32)

    def start(self):
        b = self.block
        b.set_conservative(self.hin.numpy())
        if self.c["viscous"]:
            b.calc_primitive(CBNS_Q)
        b.set_bc_calc_primitive(CBNS_Q)
        if self.c["viscous"]:
            b.calc_viscous_terms()
        b.set_time(0.0)

    def result(self):
        self.block.get_conservative(CBNS_Q, self.hout.numpy())
        return self.hout if self.h32 is None else self.h32.copy_(self.hout)


def prepare(case, seed):
    if case["kind"] == "train":
        X, Y, P = _training_set(case, seed)
        return dict(case=case, X=X.cuda(), Y=Y.cuda(), P=P.cuda())
    jobs = [_Job(*b) for b in _blocks(case, seed)]
    state = dict(case=case, jobs=jobs)
    if case["kind"] == "batch":
        state["batch"] = Batch([j.block for j in jobs])
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "train":
        loss, grad = sensor.loss_and_grad(state["P"], state["X"], state["Y"], pos_weight=2.0)
        return {"loss": loss, "grad": grad}
    jobs, steps = state["jobs"], case["steps"]
    for j in jobs:
        j.start()
    if case["kind"] == "batch":
        state["batch"].run(steps)
        return {"Q": [j.result() for j in jobs]}
    block, t = jobs[0].block, 0.0
    if case["kind"] == "run":
        block.run(steps)
        t = block.get_time()[0]
    else:
        for _ in range(steps):
            t = block.step_like_reference(t, 1.0e30)
    return {"Q": jobs[0].result(), "t": t}


def _sizes(case):
    if case["kind"] != "batch":
        return [(case["IM"], case["JM"], case["KM"])]
    sizes, lo = np.random.default_rng(1000 + case["blocks"]), case["lo"]
    return [(int(sizes.integers(lo, 4 * lo + 1)), int(sizes.integers(lo, 2 * lo + 1)),
             int(sizes.integers(lo, 2 * lo + 1))) for _ in range(case["blocks"])]


def work(case):
    """Per cell update: the three stages' input, nine metrics and J, output and RK base (560 B).  Per face: about 950
    operations for the characteristic WENO5 flux, 200 for the linear one (a tenth of a hybrid's faces take WENO5)."""
    if case["kind"] == "train":
        n = case["samples"]
        return {"bytes": n * 61 + 2 * 6404, "flops": n * 6 * 1536}
    cells = sum((i - 2) * (j - 2) * (k - 2) for i, j, k in _sizes(case))
    nodes = sum((i + 4) * (j + 4) * (k + 4) for i, j, k in _sizes(case))
    face = 275 if case["precision"] == "hybrid" else 950
    per = 9 * face + (3 * 400 if case["viscous"] else 0)
    return {"bytes": case["steps"] * cells * 560 + 80 * nodes, "flops": case["steps"] * cells * per}


# ---------------------------------------------------------------- the same jobs in plain torch, FP64
def _sl(a, axis, off, n):
    """n entries from `off` along the axis of a (..., k, j, i) array (axis 0 = i, 1 = j, 2 = k)."""
    return a.narrow(a.dim() - 1 - axis, off, n)


def _axis_derivative(f, axis):
    dim = f.dim() - 1 - axis
    n = f.shape[dim]
    s = lambda a, b: f.narrow(dim, a, b - a)  # noqa: E731
    if n < 5:
        mid = 0.5 * (s(2, n) - s(0, n - 2))
        lo = 0.5 * (-3 * s(0, 1) + 4 * s(1, 2) - s(2, 3))
        hi = 0.5 * (3 * s(n - 1, n) - 4 * s(n - 2, n - 1) + s(n - 3, n - 2))
        return torch.cat([lo, mid, hi], dim)
    e = [s(k, k + 1) for k in range(5)]
    h = [s(n - 1 - k, n - k) for k in range(5)]
    d0 = -25 / 12 * e[0] + 4 * e[1] - 3 * e[2] + 4 / 3 * e[3] - 0.25 * e[4]
    d1 = -0.25 * e[0] - 5 / 6 * e[1] + 1.5 * e[2] - 0.5 * e[3] + 1 / 12 * e[4]
    h0 = 25 / 12 * h[0] - 4 * h[1] + 3 * h[2] - 4 / 3 * h[3] + 0.25 * h[4]
    h1 = 0.25 * h[0] + 5 / 6 * h[1] - 1.5 * h[2] + 0.5 * h[3] - 1 / 12 * h[4]
    mid = (s(0, n - 4) - s(4, n)) / 12 + (s(3, n - 1) - s(1, n - 3)) * (2 / 3)
    return torch.cat([d0, d1, mid, h1, h0], dim)


def _exact_metrics(grid, dev):
    """grad(xi), grad(eta), grad(zeta) and J on the ghosted box (ghosts take the nearest boundary node)."""
    d = [[_axis_derivative(torch.from_numpy(np.ascontiguousarray(a)).to(dev), ax) for ax in range(3)] for a in grid]
    (xx, xe, xz), (yx, ye, yz), (zx, ze, zz) = d
    J = xx * (ye * zz - yz * ze) - xe * (yx * zz - yz * zx) + xz * (yx * ze - ye * zx)
    m = [ye * zz - yz * ze, xz * ze - xe * zz, xe * yz - xz * ye, yz * zx - yx * zz, xx * zz - xz * zx,
         xz * yx - xx * yz, yx * ze - ye * zx, xe * zx - xx * ze, xx * ye - xe * yx]
    pad = torch.nn.functional.pad
    out = [pad((v / J)[None, None], (NG,) * 6, mode="replicate")[0, 0] for v in m]
    return out, pad(J[None, None], (NG,) * 6, mode="replicate")[0, 0]


def _weno5(a, b, c, d, e):
    s1 = 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2 + 1e-6
    s2 = 13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2 + 1e-6
    s3 = 13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2 + 1e-6
    a1, a2, a3 = 0.1 / (s1 * s1), 0.6 / (s2 * s2), 0.3 / (s3 * s3)
    n = a1 * (2 * a - 7 * b + 11 * c) + a2 * (5 * c - b + 2 * d) + a3 * (2 * c + 5 * d - e)
    return n / (6 * (a1 + a2 + a3))


def _prims(q):
    r = q[0]
    u, v, w = q[1] / r, q[2] / r, q[3] / r
    return r, u, v, w, (GAMMA - 1) * (q[4] - 0.5 * r * (u * u + v * v + w * w))


def _exact_flux(f, n):
    """Characteristic WENO5 with the local Lax-Friedrichs flux: f = six stencil states (each five fields), n = normal."""
    g1 = GAMMA - 1
    nx, ny, nz = n
    nn = torch.sqrt(nx * nx + ny * ny + nz * nz)
    ux, uy, uz = nx / nn, ny / nn, nz / nn
    use = ny * ny + nz * nz > 1e-16
    zero = torch.zeros_like(nx)
    lx, ly, lz = torch.where(use, zero, -nz), torch.where(use, nz, zero), torch.where(use, -ny, nx)
    mx = torch.where(use, -ny * ny - nz * nz, nx * ny)
    my = torch.where(use, nx * ny, -nx * nx - nz * nz)
    mz = torch.where(use, nx * nz, ny * nz)
    ln, mn = torch.sqrt(lx * lx + ly * ly + lz * lz), torch.sqrt(mx * mx + my * my + mz * mz)
    lx, ly, lz, mx, my, mz = lx / ln, ly / ln, lz / ln, mx / mn, my / mn, mz / mn
    ra, ua, va, wa, pa = _prims(f[2])
    rb, ub, vb, wb, pb = _prims(f[3])
    Ha, Hb = (f[2][4] + pa) / ra, (f[3][4] + pb) / rb
    sr = torch.sqrt(rb / ra)
    mean = lambda a, b: (a + sr * b) / (1 + sr)  # noqa: E731
    u, v, w, H = mean(ua, ub), mean(va, vb), mean(wa, wb), mean(Ha, Hb)
    q2 = u * u + v * v + w * w
    c2 = g1 * (H - 0.5 * q2)
    c = torch.sqrt(c2)
    qn, ql, qm = u * ux + v * uy + w * uz, u * lx + v * ly + w * lz, u * mx + v * my + w * mz
    W = []
    for s in f:
        A = g1 / (2 * c2) * (0.5 * q2 * s[0] - (u * s[1] + v * s[2] + w * s[3]) + s[4])
        B = (qn * s[0] - (ux * s[1] + uy * s[2] + uz * s[3])) / (2 * c)
        W.append([A + B, s[0] - 2 * A, A - B, lx * s[1] + ly * s[2] + lz * s[3] - ql * s[0],
                  mx * s[1] + my * s[2] + mz * s[3] - qm * s[0]])
    sides = []
    for order in ((0, 1, 2, 3, 4), (5, 4, 3, 2, 1)):
        a = [_weno5(*(W[p][m] for p in order)) for m in range(5)]
        s, d = a[0] + a[2], (a[2] - a[0]) * c
        r = s + a[1]
        sides.append([r, u * r + ux * d + lx * a[3] + mx * a[4], v * r + uy * d + ly * a[3] + my * a[4],
                      w * r + uz * d + lz * a[3] + mz * a[4], H * s + qn * d + 0.5 * q2 * a[1] + ql * a[3] + qm * a[4]])
    F, speed = [], []
    for q in sides:
        r, u, v, w, p = _prims(q)
        c = torch.sqrt(GAMMA * p / r)
        un = u * nx + v * ny + w * nz
        F.append([q[0] * un, q[1] * un + p * nx, q[2] * un + p * ny, q[3] * un + p * nz, (q[4] + p) * un])
        speed.append([u.abs() + c, v.abs() + c, w.abs() + c])
    ws = sum(torch.maximum(a, b) * m for a, b, m in zip(*speed, n)).abs()
    L, Hs = sides
    return [0.5 * (F[0][m] + F[1][m] - ws * (Hs[m] - L[m])) for m in range(5)]


class _Exact:
    """One block, inviscid (reference or far-field boundaries) or viscous (far field)."""

    def __init__(self, c, grid, prm, Q, dev):
        self.c, self.prm = c, prm
        self.met, self.J = _exact_metrics(grid, dev)
        self.area = [m * self.J for m in self.met]
        self.q = [Q.to(dev).reshape(c["KM"] + 4, c["JM"] + 4, c["IM"] + 4, 5)[..., m].clone() for m in range(5)]
        self.n = (c["IM"], c["JM"], c["KM"])
        self.p_inf = 1.0 / (GAMMA * prm["Mach"] ** 2)
        self.t = 0.0
        self.boundary(self.q)

    def boundary(self, q):
        if self.c["bc"] == "farfield":
            return
        IM, JM, KM = self.n
        js, ks = slice(3, JM + 1), slice(3, KM + 1)
        for src, to in ((3, (0, 1, 2)), (IM, (IM + 1, IM + 2, IM + 3))):
            s = [v[ks, js, src].clone() for v in q]
            s[4] = self.p_inf / (GAMMA - 1) + 0.5 * (s[1] ** 2 + s[2] ** 2 + s[3] ** 2) / s[0]
            for i in to:
                for m in range(5):
                    q[m][ks, js, i] = s[m]
        for src, to in ((3, (0, 1, 2)), (KM, (KM + 1, KM + 2, KM + 3))):
            for m in range(5):
                s = q[m][src, 2:JM + 2, 2:IM + 2].clone()
                for k in to:
                    q[m][k, 2:JM + 2, 2:IM + 2] = s

    def inner(self, a, axis=None, off=0, n=None):
        """Interior nodes of a ghosted array; along `axis` instead n entries from ghosted index `off`."""
        for ax in range(3):
            a = _sl(a, ax, off, n) if ax == axis else _sl(a, ax, 3, self.n[ax] - 2)
        return a

    def mu(self, q):
        T = GAMMA * self.prm["Mach"] ** 2 * _prims(q)[4] / q[0]
        CT = 110.5 / self.prm["T_inf"]
        return T, (1 + CT) / (T + CT) * torch.sqrt(T ** 3)

    def dt(self):
        r, u, v, w, p = _prims(self.q)
        c = torch.sqrt(GAMMA * p / r)
        fv = 0.0
        if self.c["viscous"]:
            Cv = max(4 / 3, GAMMA / 0.72) / self.prm["Re"]
            fv = 2 * self.mu(self.q)[1] * Cv * torch.sqrt(u * u + v * v + w * w) / c / r
        s = 0.0
        for d in range(3):
            mx, my, mz = self.met[3 * d:3 * d + 3]
            n2 = mx * mx + my * my + mz * mz
            s = s + (u * mx + v * my + w * mz).abs() + c * torch.sqrt(n2) + n2 * fv
        return self.prm["CFL"] / float(s[2:-2, 2:-2, 2:-2].max())

    def viscous_divergence(self, q):
        r, u, v, w, p = _prims(q)
        T, mu = self.mu(q)

        def grad(f, axis):  # ghosted nodes 1 .. n-2 of every axis: the inner rows of the 4th-order stencils
            d = _sl(_axis_derivative(f, axis), axis, 1, f.shape[2 - axis] - 2)
            for ax in range(3):
                if ax != axis:
                    d = _sl(d, ax, 1, d.shape[2 - ax] - 2)
            return d
        core = lambda a: a[1:-1, 1:-1, 1:-1]  # noqa: E731
        m = [core(a) for a in self.met]
        phys = []
        for f in (u, v, w, T):
            g = [grad(f, ax) for ax in range(3)]
            phys.append([sum(g[ax] * m[3 * ax + k] for ax in range(3)) for k in range(3)])
        (ux, uy, uz), (vx, vy, vz), (wx, wy, wz), gT = phys
        mr = core(mu) / self.prm["Re"]
        div = ux + vy + wz
        tau = [[2 * mr * (ux - div / 3), mr * (uy + vx), mr * (uz + wx)],
               [mr * (uy + vx), 2 * mr * (vy - div / 3), mr * (vz + wy)],
               [mr * (uz + wx), mr * (vz + wy), 2 * mr * (wz - div / 3)]]
        kq = mr / ((GAMMA - 1) * 0.72 * self.prm["Mach"] ** 2)
        vel = [core(a) for a in (u, v, w)]
        e = [sum(vel[b] * tau[a][b] for b in range(3)) + kq * gT[a] for a in range(3)]
        out = [0.0] * 4
        for ax in range(3):
            n = [core(a) for a in self.area[3 * ax:3 * ax + 3]]
            F = [sum(n[a] * tau[a][b] for a in range(3)) for b in range(3)] + [sum(n[a] * e[a] for a in range(3))]
            for b in range(4):
                # the derivative along ax, taken one node lower in the two other directions
                f = F[b]
                for o in range(3):
                    if o != ax:
                        f = _sl(f, o, 1, self.n[o] - 2)
                k = self.n[ax] - 2
                s = lambda off: _sl(f, ax, off, k)  # noqa: E731
                out[b] = out[b] + (s(0) - s(4)) / 12 + (s(3) - s(1)) * (2 / 3)
        return out

    def rhs(self, q):
        df = [0.0] * 5
        for ax in range(3):
            nf = self.n[ax] - 1
            f = [[self.inner(v, ax, p, nf) for v in q] for p in range(6)]
            n = [0.5 * (self.inner(a, ax, 2, nf) + self.inner(a, ax, 3, nf)) for a in self.area[3 * ax:3 * ax + 3]]
            F = _exact_flux(f, n)
            for m in range(5):
                df[m] = df[m] + _sl(F[m], ax, 1, nf - 1) - _sl(F[m], ax, 0, nf - 1)
        if self.c["viscous"]:
            for m, v in enumerate(self.viscous_divergence(q)):
                df[m + 1] = df[m + 1] - v
        iJ = 1.0 / self.inner(self.J)
        return [d * iJ for d in df]

    def step(self):
        dt = self.dt()
        q0 = [self.inner(v).clone() for v in self.q]
        q = [v.clone() for v in self.q]
        for a, b, c in ((0.0, 1.0, 1.0), (0.75, 0.25, 0.25), (1 / 3, 2 / 3, 2 / 3)):
            L = self.rhs(q)
            new = [a * o + b * self.inner(v) - c * dt * l for o, v, l in zip(q0, q, L)]
            for v, x in zip(q, new):
                self.inner(v).copy_(x)
            self.boundary(q)
        self.q = q
        self.t += dt


def exact(case, seed):
    if case["kind"] == "train":
        X, Y, P = (a.double() for a in _training_set(case, seed))
        P.requires_grad_(True)
        h = torch.relu(X @ P[:480].reshape(32, 15).T + P[480:512])
        h = torch.relu(h @ P[512:1536].reshape(32, 32).T + P[1536:1568])
        z = h @ P[1568:1600] + P[1600]
        w = torch.where(Y > 0, 2.0, 1.0).double()
        loss = (w * torch.nn.functional.binary_cross_entropy_with_logits(z, Y, reduction="none")).mean()
        loss.backward()
        return {"loss": loss.detach().reshape(1), "grad": P.grad}
    # the O-grid's seam, wall and characteristic boundaries are not restated; long jobs take too long
    cells = sum(i * j * k for i, j, k in _sizes(case))
    if case["bc"] == "ogrid" or case["steps"] * (len(_sizes(case)) * 0.05 + cells * 2.0e-8) > 18.0:
        return None
    out = []
    for b in _blocks(case, seed):
        e = _Exact(*b, _device())
        for _ in range(case["steps"]):
            e.step()
        out.append(torch.stack(e.q, dim=-1).reshape(-1).cpu())
        if case["kind"] != "batch":
            return {"Q": out[0], "t": e.t}
    return {"Q": out}
