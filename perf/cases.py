"""Timed cases of the framework's work, through its public entry points.

The framework solves the staggered-grid Stokes system of a time step
(gmres(...)): most cases are whole solves, over the grid sizes, dimensions,
boundary conditions, array layouts, methods and precisions that callers use,
from one 2D 64^2 problem (bound by launches and latency) to a 3D 256^3 one
(67 M unknowns).  One case is the operator alone and one the learned stage's
network (forward and backward).  Inputs follow lowmachmixtures_b200/synth.py:
a log-viscosity field of six Fourier modes with a given contrast, or the
four-species mixture rule, unit density and a normal right-hand side without
mean; they are made on the GPU from the seed alone.

Grids are given per direction, so drawn cases also have unequal extents and
sizes whose coarsest multigrid level has an odd cell count (96 -> 3,
80 -> 5).  Solves are returned as the velocity and pressure (and
norm_pre_rhs, which the reference's left-preconditioned method reports).
"""
import ctypes
import math

import numpy as np
import torch

from lowmachmixtures_b200 import _native, abi, learned
from lowmachmixtures_b200.gmres import StokesSolver

PERIODIC, NO_SLIP, SLIP = abi.LMM_BC_PERIODIC, abi.LMM_BC_NO_SLIP_WALL, abi.LMM_BC_SLIP_WALL
SPECIES_VISCOSITY = (1.0, 2.0, 5.0, 10.0)
LEVELS_PER_SWEEPS = 4  # two smoothing sweeps down, two up


def listed():
    return [
        # the smallest solve of the parity configuration: 2D 64^2, contrast 10, steady, FP32 V-cycles in FP64 FGMRES
        dict(name="mixed 2d 64", kind="solve", method="mixed", dm=2, nx=64, ny=64, nz=1, contrast=10.0, alpha=0.0, inner=5, walls="none"),
        # what the Fortran caller of a 2D run makes: BoxLib host arrays with ghost cells, the reference's GMRES and defaults
        dict(name="boxlib 2d 96x64 gmres", kind="boxlib", dm=2, nx=96, ny=64, nz=1, contrast=10.0, alpha=0.1),
        # a 2D channel (no-slip walls in y) with an odd coarsest level
        dict(name="mixed 2d channel 192x96", kind="solve", method="mixed", dm=2, nx=192, ny=96, nz=1, contrast=30.0, alpha=0.0, inner=5,
             walls="channel"),
        # an uneven ensemble of independent 2D problems on one device
        dict(name="ensemble 2d x96", kind="ensemble", count=96, sizes="64,96,128,192,256", contrast=1000.0),
        # 3D steady problem of the high-contrast family
        dict(name="mixed 3d 64", kind="solve", method="mixed", dm=3, nx=64, ny=64, nz=64, contrast=300.0, alpha=0.0, inner=5, walls="none"),
        # the same path between walls
        dict(name="mixed 3d channel 64x48x64", kind="solve", method="mixed", dm=3, nx=64, ny=48, nz=64, contrast=100.0, alpha=0.1, inner=5,
             walls="channel"),
        # the Fortran caller in 3D
        dict(name="boxlib 3d 64 gmres", kind="boxlib", dm=3, nx=64, ny=64, nz=64, contrast=100.0, alpha=0.1),
        # the headline workload: 3D 128^3, contrast 100, inertial
        dict(name="mixed 3d 128", kind="solve", method="mixed", dm=3, nx=128, ny=128, nz=128, contrast=100.0, alpha=0.1, inner=5, walls="none"),
        # the reference's method in FP64, device arrays, an odd coarsest level
        dict(name="gmres 3d 96 fp64", kind="solve", method="gmres", dm=3, nx=96, ny=96, nz=96, contrast=100.0, alpha=0.1, inner=5, walls="none"),
        # the largest: 3D 256^3 mixture viscosity, GMRES(20)
        dict(name="mixed 3d 256 mixture", kind="solve", method="mixed", dm=3, nx=256, ny=256, nz=256, contrast=0.0, alpha=0.0, inner=20,
             walls="none"),
        # the coupled operator alone on a ragged grid (a caller checking a residual)
        dict(name="apply_matrix 160x96x122", kind="operator", nx=160, ny=96, nz=122, contrast=100.0, alpha=0.1),
        # the learned stage's network, forward and backward: parameter gradients of a batch of two
        dict(name="net gradients 64x2", kind="net", nx=64, ny=64, nz=64, batch=2),
    ]


def draw(rng):
    kind = rng.choice(["2d", "2d", "walls2", "boxlib", "ensemble", "3d", "3d", "walls3", "gmres3", "operator", "net"])

    def log_size(lo, hi, step):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))

    contrast = round(10.0 ** rng.uniform(1.0, 2.5), 3)
    alpha = rng.choice([0.0, 0.1, round(10.0 ** rng.uniform(-2.0, 0.0), 4)])
    inner = rng.choice([5, 5, 10])
    if kind in ("2d", "walls2"):
        n = [log_size(32, 384, 16) for _ in range(2)]
        walls = "none" if kind == "2d" else rng.choice(["channel", "box", "slip"])
        return dict(kind="solve", method=rng.choice(["mixed", "mixed", "plain", "gmres"]), dm=2, nx=n[0], ny=n[1], nz=1,
                    contrast=contrast, alpha=alpha, inner=inner, walls=walls)
    if kind in ("3d", "walls3", "gmres3"):
        n = [log_size(32, 160, 16) for _ in range(3)]
        walls = rng.choice(["channel", "box", "slip"]) if kind == "walls3" else "none"
        return dict(kind="solve", method="gmres" if kind == "gmres3" else rng.choice(["mixed", "mixed", "plain"]), dm=3, nx=n[0],
                    ny=n[1], nz=n[2], contrast=contrast, alpha=alpha, inner=inner, walls=walls)
    if kind == "boxlib":
        dm = rng.choice([2, 3])
        n = [log_size(32, 256 if dm == 2 else 96, 16) for _ in range(dm)] + [1] * (3 - dm)
        return dict(kind="boxlib", dm=dm, nx=n[0], ny=n[1], nz=n[2], contrast=contrast, alpha=rng.choice([0.0, 0.1]))
    if kind == "ensemble":
        return dict(kind="ensemble", count=rng.randint(8, 160), sizes=rng.choice(["64", "64,96,128", "64,96,128,192,256", "48,80,160"]),
                    contrast=rng.choice([30.0, 100.0, 1000.0]))
    if kind == "operator":
        n = [rng.randint(33, 224) for _ in range(3)]
        return dict(kind="operator", nx=n[0], ny=n[1], nz=n[2], contrast=contrast, alpha=alpha)
    n = [rng.choice([32, 48, 64, 96]) for _ in range(3)]
    return dict(kind="net", nx=n[0], ny=n[1], nz=n[2], batch=rng.choice([1, 2, 4]))


# ------------------------------------------------------------ inputs
def _size(case):
    return (case["nx"], case["ny"], case["nz"])[: case.get("dm", 3)]


def _bc(case):
    """BC codes per direction: a channel has walls in y, a box in every direction, slip: a slip and a no-slip wall in x."""
    dm = case["dm"]
    w = case.get("walls", "none")
    if w == "channel":
        return ((PERIODIC, PERIODIC), (NO_SLIP, NO_SLIP), (PERIODIC, PERIODIC))[:dm]
    if w == "box":
        return ((NO_SLIP, NO_SLIP),) * dm
    if w == "slip":
        return ((SLIP, NO_SLIP),) + ((PERIODIC, PERIODIC),) * (dm - 1)
    return None


def _nodal_walls(n, bc, e):
    dm = len(n)
    return [n[d] + (1 if d in abi.edge_nodal(dm, e) and abi.walled(bc, d) else 0) for d in range(dm)]


def _wave(rng, dm):
    while True:
        k = rng.integers(-4, 5, size=dm)
        if 0 < int((k * k).sum()) <= 16:
            return [int(v) for v in k]


def _field(modes, ext, offs, n):
    """sum of cos(2 pi k.x + phase) on points (index + offset) / n[0], x fastest"""
    dm = len(ext)
    ax = [(torch.arange(ext[d], dtype=torch.float64, device="cuda") + offs[d]) / n[d] for d in range(dm)]
    g = torch.zeros(tuple(reversed(ext)), dtype=torch.float64, device="cuda")
    for k, ph in modes:
        arg = torch.full((1,) * dm, ph, dtype=torch.float64, device="cuda")
        for d in range(dm):
            shape = [1] * dm
            shape[dm - 1 - d] = ext[d]
            arg = arg + (2.0 * math.pi * k[d]) * ax[d].reshape(shape)
        g += torch.cos(arg)
    return g


def _places(dm):
    """offsets (x, y[, z]) of the cells and of each edge array"""
    edges = [(0.0, 0.0)] if dm == 2 else [(0.0, 0.0, 0.5), (0.0, 0.5, 0.0), (0.5, 0.0, 0.0)]
    return [(0.5,) * dm] + edges


def _viscosity(n, contrast, rng, bc=None):
    """beta at cells and edges; contrast 0: the mixture of four species"""
    dm = len(n)
    ext = [list(n)] + [_nodal_walls(n, bc, e) for e in range(1 if dm == 2 else 3)]

    def one():
        modes = [(_wave(rng, dm), float(rng.uniform(0.0, 2.0 * math.pi))) for _ in range(6)]
        f = [_field(modes, x, o, n) for x, o in zip(ext, _places(dm))]
        top = max(float(v.abs().max()) for v in f)
        return [v / top for v in f]

    if contrast > 0:
        f = [torch.exp(0.5 * math.log(contrast) * v) for v in one()]
    else:
        w = [[1.0 + 0.9 * v for v in one()] for _ in SPECIES_VISCOSITY]
        f = []
        for part in zip(*w):
            tot = sum(part)
            f.append(torch.exp(sum((wi / tot) * math.log(es) for wi, es in zip(part, SPECIES_VISCOSITY))))
    return f[0].contiguous(), [v.contiguous() for v in f[1:]]


def _problem(n, contrast, alpha, seed, bc=None):
    """the arrays of one problem on the GPU (compact layout): unit density, theta alpha dx^2 = alpha"""
    dm = len(n)
    rng = np.random.default_rng(seed)
    beta, bed = _viscosity(n, contrast, rng, bc)
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 7 + 1)
    shape = tuple(reversed(n))
    bu = []
    for d in range(dm):
        r = torch.randn(shape, dtype=torch.float64, device="cuda", generator=gen)
        r -= r.mean()
        if abi.walled(bc, d):  # face lo is the wall
            r.select(dm - 1 - d, 0).zero_()
        bu.append(r)
    z = torch.zeros(shape, dtype=torch.float64, device="cuda")
    return dict(dm=dm, n=n, dx=1.0 / n[0], theta=alpha * n[0] * n[0], bu=bu, bp=z, alpha=[torch.ones_like(z) for _ in range(dm)], beta=beta,
                bed=bed, gamma=torch.zeros_like(z), xu=[torch.zeros_like(z) for _ in range(dm)], xp=torch.zeros_like(z))


def _knobs(method, inner=5, tol=1e-9):
    kw = dict(visc_type=-2, gmres_max_inner=inner, gmres_rel_tol=tol, gmres_verbose=0, gmres_max_outer=40, gmres_max_iter=200)
    if method == "mixed":  # FP32 V-cycles inside FP64 flexible GMRES, classical Gram-Schmidt: the configuration of the benchmark
        return abi.make_knobs(precon_type=2, method=abi.LMM_METHOD_FGMRES, precision=abi.LMM_PRECISION_FP32, orthogonalization=1, **kw)
    if method == "plain":  # FGMRES all in FP64
        return abi.make_knobs(precon_type=2, method=abi.LMM_METHOD_FGMRES, precision=abi.LMM_PRECISION_FP64, **kw)
    if method == "gmres":  # the reference's algorithm
        return abi.make_knobs(precon_type=2, **kw)
    return abi.make_knobs(precon_type=1, **kw)  # its default preconditioner, the projection


def _boxlib(a, n, nodal, ng):
    """the BoxLib array (ghost cells, both copies of a periodic seam face) of a compact one"""
    idx = []
    for d in reversed(range(len(n))):
        idx.append((np.arange(n[d] + (1 if d in nodal else 0) + 2 * ng) - ng) % n[d])
    return np.ascontiguousarray(a.cpu().numpy()[np.ix_(*idx)])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "net":
        net = learned.Net(_size(case), case["batch"], 3)
        gen = torch.Generator(device="cuda").manual_seed(int(seed))
        shape = (case["batch"], case["nz"], case["ny"], case["nx"])
        x = torch.zeros(*shape, 8, device="cuda")
        x[..., :5] = torch.randn(*shape, 5, device="cuda", generator=gen)
        gy = torch.randn(*shape, 4, device="cuda", generator=gen) / float(np.prod(shape))
        s = dict(net=net, x=x.to(torch.bfloat16), gy=gy, y=torch.empty_like(gy), grads=np.zeros(net.num_params, np.float32))
    elif kind == "ensemble":
        rng = np.random.default_rng(seed + 17)
        sizes = [int(v) for v in case["sizes"].split(",")]
        probs = []
        for i in range(case["count"]):
            c = float(10.0 ** rng.uniform(1.0, math.log10(case["contrast"])))
            n = sizes[i % len(sizes)]
            probs.append(_problem((n, n), c, 0.0, seed * 1000 + i))
        items = (abi.EnsembleItem * len(probs))()
        for it, p in zip(items, probs):
            for d in range(3):
                it.n[d] = p["n"][d] if d < 2 else 1
            it.dx, it.theta_alpha = p["dx"], p["theta"]
            for d in range(2):
                it.b_u[d], it.alpha_fc[d], it.x_u[d] = abi.ptr(p["bu"][d]), abi.ptr(p["alpha"][d]), abi.ptr(p["xu"][d])
            it.beta_ed[0], it.b_p, it.beta = abi.ptr(p["bed"][0]), abi.ptr(p["bp"]), abi.ptr(p["beta"])
            it.gamma, it.x_p = abi.ptr(p["gamma"]), abi.ptr(p["xp"])
        s = dict(problems=probs, items=items, pool=_Pool(items, _knobs("mixed", 5, 1e-8)))
    elif kind == "operator":
        n = _size(case)
        p = _problem(n, case["contrast"], case["alpha"], seed)
        s = dict(p, solver=StokesSolver(3, n, p["dx"], knobs=_knobs("gmres")))
        s["solver"].load_coeffs(p["alpha"], p["beta"], p["bed"], p["gamma"], p["theta"])
        s["pin"] = torch.randn(p["bp"].shape, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(int(seed) + 5))
    elif kind == "boxlib":
        n, dm = _size(case), case["dm"]
        p = _problem(n, case["contrast"], case["alpha"], seed)
        ng = dict(b_u=0, b_p=0, alpha_fc=1, beta=1, beta_ed=0, gamma=1, x_u=1, x_p=1)
        face = [_boxlib(a, n, (d,), 0) for d, a in enumerate(p["bu"])]
        s = dict(dm=dm, theta=p["theta"], ng=ng, bu=face, bp=_boxlib(p["bp"], n, (), 0),
                 alpha=[_boxlib(a, n, (d,), 1) for d, a in enumerate(p["alpha"])], beta=_boxlib(p["beta"], n, (), 1),
                 bed=[_boxlib(a, n, abi.edge_nodal(dm, e), 0) for e, a in enumerate(p["bed"])], gamma=_boxlib(p["gamma"], n, (), 1),
                 xu=[_boxlib(a, n, (d,), 1) for d, a in enumerate(p["xu"])], xp=_boxlib(p["xp"], n, (), 1),
                 solver=StokesSolver(dm, n, p["dx"], knobs=_knobs("projection")))
    else:
        n, bc = _size(case), _bc(case)
        p = _problem(n, case["contrast"], case["alpha"], seed, bc)
        s = dict(p, solver=StokesSolver(case["dm"], n, p["dx"], knobs=_knobs(case["method"], case["inner"]), bc=bc))
    s["kind"] = kind
    torch.cuda.synchronize()
    return s


class _Pool:
    """an lmm_ensemble handle"""

    def __init__(self, items, knobs):
        self.lib = _native.load()
        self.h = ctypes.c_void_p()
        _native.check(self.lib.lmm_ensemble_create(2, ctypes.byref(knobs), 0, items, len(items), 4, ctypes.byref(self.h)), "lmm_ensemble_create")

    def run(self, items):
        _native.check(self.lib.lmm_ensemble_run(self.h, items, len(items)), "lmm_ensemble_run")

    def __del__(self):
        if self.h:
            self.lib.lmm_ensemble_destroy(self.h)
            self.h = None


# ------------------------------------------------------------ one pass
def run(s):
    """One call, as a time stepper makes it: zero initial guess in, solution out.  The library works on streams of its
    own, so a caller waits for what its own stream has written before the call."""
    kind = s["kind"]
    if kind == "net":
        lib = s["net"].lib
        _native.check(lib.lmm_net_gradients(s["net"].h, ctypes.c_void_p(s["x"].data_ptr()), ctypes.c_void_p(s["gy"].data_ptr()),
                                            s["grads"].ctypes.data_as(ctypes.c_void_p)), "lmm_net_gradients")
        _native.check(lib.lmm_net_forward(s["net"].h, ctypes.c_void_p(s["x"].data_ptr()), ctypes.c_void_p(s["y"].data_ptr())), "lmm_net_forward")
        return dict(grads=s["grads"], y=s["y"])
    if kind == "operator":
        out = [torch.empty_like(s["bp"]) for _ in range(4)]
        torch.cuda.current_stream().synchronize()
        s["solver"].apply_matrix(s["bu"], s["pin"], out[:3], out[3])
        return out
    if kind == "boxlib":
        for a in s["xu"]:
            a.fill(0.0)
        s["xp"].fill(0.0)
        _, npr, _ = s["solver"].solve(s["bu"], s["bp"], s["xu"], s["xp"], s["alpha"], s["beta"], s["bed"], s["gamma"], s["theta"],
                                      layout=abi.LMM_LAYOUT_BOXLIB, ng=s["ng"])
        return dict(u=s["xu"], p=s["xp"], norm_pre_rhs=npr)
    for p in s["problems"] if kind == "ensemble" else [s]:
        torch._foreach_zero_(p["xu"] + [p["xp"]])
    torch.cuda.current_stream().synchronize()
    if kind == "ensemble":
        s["pool"].run(s["items"])
        return dict(u=torch.cat([a.reshape(-1) for p in s["problems"] for a in p["xu"]]),
                    p=torch.cat([p["xp"].reshape(-1) for p in s["problems"]]))
    _, npr, _ = s["solver"].solve_device(s["bu"], s["bp"], s["xu"], s["xp"], s["alpha"], s["beta"], s["bed"], s["gamma"], s["theta"])
    return dict(u=s["xu"], p=s["xp"], norm_pre_rhs=npr)


# ------------------------------------------------------------ what a pass needs
def _solve_work(n, mixed, iters, m):
    """bytes and operations of `iters` iterations: per level of the V-cycle four smoothing sweeps, a residual, a restriction
    and a prolongation with every array passed once each, the pressure V-cycle's, then the coupled operator, the
    Gram-Schmidt passes (each basis vector read twice) and the normalisation in FP64"""
    dm = len(n)
    N = float(np.prod(n))
    w = 4.0 if mixed else 8.0
    ed = 1 if dm == 2 else 3
    levels = sum(0.5 ** (dm * l) for l in range(6))
    sweep = 3 * dm + 1 + ed                       # phi in and out, rhs, beta, beta_ed
    vcyc = levels * (LEVELS_PER_SWEEPS * sweep + (2 * dm + 1 + ed) + 3 * dm) + levels * (LEVELS_PER_SWEEPS * 3 + 2 + 3)
    vec = (dm + 1) * 8.0
    op = (dm + 1) * w + (2 * dm + 2 + ed) * 8.0 + vec
    j = (min(m, iters) + 1) / 2.0
    gs = 2 * (j + 1) * vec + vec + 2 * vec + (dm + 1) * w
    flops = levels * (LEVELS_PER_SWEEPS + 1.2) * dm * (55 if dm == 3 else 35) + dm * 60 + 4 * (dm + 1) * j
    return dict(bytes=iters * N * (vcyc * w + op + gs), flops=iters * N * flops)


def _iterations(case):
    c = case["contrast"] if case["contrast"] > 0 else 10.0
    return 10.0 + 6.0 * math.log10(max(c, 1.0) / 10.0)


def work(case):
    kind = case["kind"]
    if kind == "net":
        v = float(case["batch"] * case["nx"] * case["ny"] * case["nz"])
        grid = (1, 1, 8, 8, 64, 64, 8, 8, 1, 1, 1)
        fl = sum(2.0 * 27 * ci * co / g for (ci, co), g in zip(learned.LAYERS, grid))
        act = sum(2.0 * co / g for (_, co), g in zip(learned.LAYERS, grid))
        return dict(bytes=v * (2 * 16 + 4 * 4 + 4 * act), flops=4.0 * v * fl)  # two forward passes, data and weight gradients
    if kind == "operator":
        N = float(case["nx"] * case["ny"] * case["nz"])
        return dict(bytes=8.0 * N * (4 + 3 + 1 + 3 + 4), flops=N * 200.0)
    if kind == "ensemble":
        sizes = [int(v) for v in case["sizes"].split(",")]
        got = [_solve_work((n, n), True, 12.0 + 5.0 * math.log10(case["contrast"] / 10.0), 5)
               for n in (sizes[i % len(sizes)] for i in range(case["count"]))]
        return dict(bytes=sum(g["bytes"] for g in got), flops=sum(g["flops"] for g in got))
    if kind == "boxlib":
        return _solve_work(_size(case), False, _iterations(case), 5)
    return _solve_work(_size(case), case["method"] == "mixed", _iterations(case), case["inner"])


# ------------------------------------------------------------ in 64 bits
def _shift(a, d, s):
    """a at index + s along direction d (periodic)"""
    return torch.roll(a, -s, a.dim() - 1 - d)


def _operator(p, u, pr):
    """[A G; -D 0][u; pr] with A u = theta alpha u - div(beta (grad u + grad u^T))"""
    dx = p["dx"]
    edge = {(0, 1): 0, (0, 2): 1, (1, 2): 2}
    out = []
    for d in range(3):
        b, bm = p["beta"], _shift(p["beta"], d, -1)
        v = u[d]
        lap = 2 * b * (_shift(v, d, 1) - v) - 2 * bm * (v - _shift(v, d, -1))
        for t in range(3):
            if t == d:
                continue
            e = p["bed"][edge[(min(d, t), max(d, t))]]
            ep = _shift(e, t, 1)
            q = u[t]
            qm = _shift(q, d, -1)
            lap += ep * (_shift(v, t, 1) - v + _shift(q, t, 1) - _shift(qm, t, 1)) - e * (v - _shift(v, t, -1) + q - qm)
        out.append(p["theta"] * p["alpha"][d] * v - lap / dx ** 2 + (pr - _shift(pr, d, -1)) / dx)
    out.append(-sum((_shift(u[d], d, 1) - u[d]) / dx for d in range(3)))
    return out


def _network(params, x, batch, shape):
    """the learned stage's network in FP64: y and the parameters as leaves"""
    ws, o = [], 0
    for ci, co in learned.LAYERS:
        w = params[o: o + co * 27 * ci].reshape(co, 27, ci)
        o += co * 27 * ci
        ws.append((w, params[o: o + co]))
        o += co

    def conv(a, i):
        w, b = ws[i]
        a = torch.nn.functional.pad(a, (1,) * 6, mode="circular")
        n = [s - 2 for s in a.shape[2:]]
        y = b.reshape(1, -1, 1, 1, 1)
        for t in range(27):
            dz, dy, dx = t // 9, t // 3 % 3, t % 3
            y = y + torch.einsum("oc,bczyx->bozyx", w[:, t], a[:, :, dz: dz + n[0], dy: dy + n[1], dx: dx + n[2]])
        return y

    relu, pool = torch.relu, lambda a: torch.nn.functional.avg_pool3d(a, 2)  # noqa: E731

    def up(a):
        return a.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)

    s0 = relu(conv(relu(conv(x, 0)), 1))
    s1 = relu(conv(relu(conv(pool(s0), 2)), 3))
    b2 = relu(conv(relu(conv(pool(s1), 4)), 5))
    d1 = relu(conv(relu(conv(up(b2), 6) + s1), 7))
    d0 = relu(conv(relu(conv(up(d1), 8) + s0), 9))
    return conv(d0, 10)


def exact(case, seed):
    """The operator and the network have values of their own; a solve is an iterate that stopped at its tolerance."""
    if case["kind"] == "operator":
        p = _problem(_size(case), case["contrast"], case["alpha"], seed)
        pin = torch.randn(p["bp"].shape, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(int(seed) + 5))
        return _operator(p, p["bu"], pin)
    if case["kind"] == "net" and case["batch"] * case["nx"] * case["ny"] * case["nz"] <= 2 ** 20:
        s = prepare(case, seed)
        params = torch.from_numpy(s["net"].params()).double().cuda().requires_grad_(True)
        x = s["x"].double().permute(0, 4, 1, 2, 3)
        y = _network(params, x, case["batch"], x.shape[2:])
        gy = s["gy"].double().permute(0, 4, 1, 2, 3)
        g, = torch.autograd.grad((y * gy).sum(), params)
        return dict(grads=g, y=y.detach().permute(0, 2, 3, 4, 1).contiguous())
    return None
