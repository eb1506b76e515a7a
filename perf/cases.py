"""Measured work of the framework: what a user has it do, through its public
entry points, from the smallest dots to million-cell films.

The paths: one effective field (exact sum, FMM), one potential, fixed RK4
steps (exact sum, FMM, learned far field), the adaptive march, the batched
ensemble, and one training gradient of the learned far field.  Sizes are those
of the reference's run logs (16 x 16, 76 x 27 cells), of the tests (40 x 40
vortex disc, 64 .. 256 films), of the benchmark (256 x 256 x 3 dot lattice,
512 instances of 16 .. 64 cells a side) and one film of a million cells a
layer, with odd and ragged sizes among the drawn ones.

prepare() makes the inputs on the GPU from the seed and the context (plan,
weights) that a program keeps; run() is one pass; exact() is the same in 64
bits from plain torch: the potential as a zero-padded FFT convolution with
1/r, central differences, the classical RK4 step.
"""
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "mms-gpu_b200"))

import mmsb200  # noqa: E402
from mmsb200 import ensemble as mmsens  # noqa: E402

MS, AEX, ALPHA, GAMMA, MU0 = 8.6e5, 1.3e-11, 0.5, 2.21e5, 4e-7 * math.pi
HEXT_T, HEXT_B = [0.0, 1e-8], [[-0.05, 0.0, 0.0], [0.05, 0.0, 0.0]]  # the benchmark's ramp
DT = 1e-13
SIDES = (16, 24, 32, 40, 48, 56, 64)
STREAM = torch.cuda.Stream() if torch.cuda.is_available() else None  # a program steps one simulation at a time
WEIGHTS = os.path.join(ROOT, "mms-gpu_b200", "weights", "farnet_w24_d5.npz")


# ---- the cases -----------------------------------------------------------------
def _field(name, X, Y, Z, solver, P=4, leaf=0, d=5e-9, dz=5e-9, host=False):
    return {"name": name, "kind": "field", "X": X, "Y": Y, "Z": Z, "d": d, "dz": dz, "solver": solver, "P": P,
            "leaf": leaf, "host": host, "mask": "blocks", "ic": "sphere"}


def _steps(name, X, Y, Z, solver, n, P=4, leaf=0, mask="full", ic="sphere"):
    return {"name": name, "kind": "steps", "X": X, "Y": Y, "Z": Z, "d": 5e-9, "dz": 5e-9, "solver": solver, "P": P,
            "leaf": leaf, "n": n, "mask": mask, "ic": ic}


def listed():
    return [
        # the field of the smallest dot of the reference's logs: launches and latency
        _field("field exact 16x16x3", 16, 16, 3, "direct"),
        # the nanowires of the logs, odd and ragged: steps between two reads of the state
        _steps("steps exact 76x27x3", 76, 27, 3, "direct", 20, ic="plane"),
        # a vortex disc relaxed by the adaptive controller
        {"name": "march vortex 40x40x3", "kind": "march", "X": 40, "Y": 40, "Z": 3, "d": 5e-9, "dz": 5e-9,
         "solver": "direct", "P": 4, "leaf": 0, "mask": "disc", "ic": "vortex", "final": 1.5e-12},
        # a host program's Hfield call (the drop-in's boundary): host arrays in and out
        _field("field exact host 64x64x3", 64, 64, 3, "direct", host=True),
        # the exact field of a film: what every approximate solver is judged by
        _field("field exact 256x256x3", 256, 256, 3, "direct"),
        # the small film of the precision sweep, stepped with the FMM
        _steps("steps fmm 64x64x3", 64, 64, 3, "fmm", 20, P=5, mask="blocks"),
        # the benchmark: the 8 x 8 lattice of discs, FMM P = 4 on 8-cell leaves
        _steps("steps fmm 256x256x3", 256, 256, 3, "fmm", 20, P=4, leaf=8, mask="dots", ic="dots"),
        # a high-order potential on a ragged film (far-field training data, checks)
        {"name": "potential fmm P8 250x190x3", "kind": "potential", "X": 250, "Y": 190, "Z": 3, "d": 5e-9, "dz": 5e-9,
         "solver": "fmm", "P": 8, "leaf": 8, "mask": "blocks", "ic": "sphere"},
        # the field of a film of a million cells a layer
        _field("field fmm 1024x1024x3", 1024, 1024, 3, "fmm", P=4, leaf=8),
        # steps with the learned far field, checked against the FMM every 50
        _steps("steps network 256x256x3", 256, 256, 3, "net", 50, P=6, leaf=8, mask="dots", ic="dots"),
        # many independent dots at once, read back after 100 steps
        {"name": "ensemble 512", "kind": "ensemble", "count": 512, "n": 100},
        # one training gradient of the learned far field
        {"name": "gradient 8 of 256x256x3", "kind": "gradient", "X": 256, "Y": 256, "batch": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["field direct", "field direct", "field fmm", "potential", "steps direct", "steps fmm",
                       "steps fmm", "steps net", "march", "ensemble", "gradient"])
    Z = rng.choice([1, 2, 3, 3, 3, 3, 4])
    d = rng.choice([2e-9, 4e-9, 5e-9])
    if kind == "field direct":
        c = _field("", _log(rng, 12, 260), _log(rng, 12, 260), Z, "direct", d=d, dz=rng.choice([d, 3e-9]),
                   host=rng.random() < 0.25)
    elif kind == "field fmm":
        c = _field("", _log(rng, 40, 1000), _log(rng, 40, 1000), Z, "fmm", P=rng.randint(3, 6),
                   leaf=rng.choice([0, 4, 8]), d=d, dz=d, host=False)
    elif kind == "potential":
        c = _field("", _log(rng, 40, 400), _log(rng, 40, 400), 3, "fmm", P=rng.randint(4, 8), leaf=rng.choice([4, 8]),
                   d=d, dz=d)
        c["kind"] = "potential"
        del c["host"]
    elif kind == "steps direct":
        c = _steps("", _log(rng, 12, 160), _log(rng, 12, 160), Z, "direct", rng.randint(5, 25),
                   mask=rng.choice(["full", "disc", "blocks"]), ic=rng.choice(["sphere", "plane"]))
    elif kind == "steps fmm":
        c = _steps("", _log(rng, 48, 400), _log(rng, 48, 400), 3, "fmm", rng.randint(5, 25), P=rng.choice([3, 4, 4, 5, 6]),
                   leaf=rng.choice([0, 4, 8, 8]), mask=rng.choice(["full", "blocks", "disc"]),
                   ic=rng.choice(["sphere", "plane"]))
    elif kind == "steps net":
        c = _steps("", _log(rng, 64, 256), _log(rng, 64, 256), 3, "net", rng.randint(5, 60), P=6, leaf=8,
                   mask=rng.choice(["full", "blocks", "disc"]), ic=rng.choice(["sphere", "plane"]))
    elif kind == "march":
        s = _log(rng, 20, 72)
        c = {"kind": "march", "X": s, "Y": s, "Z": 3, "d": 5e-9, "dz": 5e-9, "solver": "direct", "P": 4, "leaf": 0,
             "mask": "disc", "ic": "vortex", "final": rng.choice([5e-13, 1e-12, 1.5e-12])}
    elif kind == "ensemble":
        c = {"kind": "ensemble", "count": _log(rng, 16, 512), "n": rng.randint(10, 100)}
    else:
        c = {"kind": "gradient", "X": rng.randint(40, 256), "Y": rng.randint(40, 256), "batch": rng.randint(1, 8)}
    c.pop("name", None)
    return c


def _ens_dims(case):
    r = random.Random(case["count"])
    return [(r.choice(SIDES), r.choice(SIDES), 3) for _ in range(case["count"])]


def _cells(case):
    if case["kind"] == "ensemble":
        return sum(x * y * z for x, y, z in _ens_dims(case))
    return case["X"] * case["Y"] * case.get("Z", 3)


# ---- inputs, plain torch -------------------------------------------------------
def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(1_000_003 * int(seed) + salt)


def _mask(kind, X, Y, Z, g):
    """(Z, Y, X) bool, material in the middle layers as the reference's driver places it, in all of a thinner film"""
    y, x = torch.meshgrid(torch.arange(Y, device="cuda"), torch.arange(X, device="cuda"), indexing="ij")
    if kind == "blocks":  # about 30 % of the cells taken out in 4 x 4 blocks
        keep = torch.rand(((Y + 3) // 4, (X + 3) // 4), device="cuda", generator=g) >= 0.3
        p = keep.repeat_interleave(4, 0).repeat_interleave(4, 1)[:Y, :X]
    elif kind == "disc":
        r = min(X, Y) / 2
        p = (x - (X - 1) / 2) ** 2 + (y - (Y - 1) / 2) ** 2 <= r * r
    elif kind == "dots":  # discs of radius 12 at a pitch of 32
        p = ((x % 32) - 15.5) ** 2 + ((y % 32) - 15.5) ** 2 <= 144
    else:
        p = torch.ones((Y, X), dtype=torch.bool, device="cuda")
    m = p[None].expand(Z, Y, X).clone()
    if Z >= 3:
        m[0] = False
        m[-1] = False
    return m


def _state(kind, m, g):
    """(Z, Y, X, 3) float32 of length Ms on the mask"""
    Z, Y, X = m.shape
    if kind == "sphere":
        v = torch.randn((Z, Y, X, 3), device="cuda", generator=g)
    elif kind == "vortex":
        y, x = torch.meshgrid(torch.arange(Y, device="cuda") - (Y - 1) / 2, torch.arange(X, device="cuda") - (X - 1) / 2,
                              indexing="ij")
        core = torch.where(torch.hypot(x, y) <= 2, 1.0, 0.0)
        r = torch.hypot(x, y).clamp(min=1e-3)
        v = torch.stack([-y / r * (1 - core), x / r * (1 - core), core], -1)[None].expand(Z, Y, X, 3)
        v = v + 0.0175 * torch.randn((Z, Y, X, 3), device="cuda", generator=g)  # about 1 degree
    elif kind == "dots":  # one in-plane direction per dot
        ny, nx = -(-Y // 32), -(-X // 32)
        ph = (2 * math.pi * torch.rand((ny, nx), device="cuda", generator=g))
        ph = ph.repeat_interleave(32, 0).repeat_interleave(32, 1)[:Y, :X]
        v = torch.stack([torch.cos(ph), torch.sin(ph), torch.zeros_like(ph)], -1)[None].expand(Z, Y, X, 3)
    else:  # in-plane film, a few degrees of disorder
        v = 0.05 * torch.randn((Z, Y, X, 3), device="cuda", generator=g)
        v = v + torch.tensor([1.0, 0.3, 0.0], device="cuda")
    v = v.double()
    v = v / v.norm(dim=-1, keepdim=True) * MS * m[..., None]
    return v.float().contiguous()


def _inputs(case, seed):
    g = _gen(seed)
    m = _mask(case["mask"], case["X"], case["Y"], case["Z"], g)
    return m, _state(case["ic"], m, g)


def _charge(case, M):
    """a charge density in float32, as a program hands it to the potential"""
    return _div(M.double(), case["d"], case["d"], case["dz"]).float().contiguous()


def _ens_inputs(case, seed):
    """masks, states and in-plane fields of all instances in one 64 x 64 x 3 canvas each, and the grids' extents"""
    g = _gen(seed)
    n = case["count"]
    dims = torch.tensor(_ens_dims(case), device="cuda")
    y, x = torch.meshgrid(torch.arange(64, device="cuda"), torch.arange(64, device="cuda"), indexing="ij")
    X, Y = dims[:, 0, None, None], dims[:, 1, None, None]
    inside = (x[None] < X) & (y[None] < Y)
    kind = torch.randint(0, 3, (n, 1, 1), device="cuda", generator=g)
    cx, cy = (X - 1) / 2, (Y - 1) / 2
    r = (torch.minimum(X, Y) - 2) / 2
    disc = (x - cx) ** 2 + (y - cy) ** 2 <= r * r
    ell = ((x - cx) / ((X - 2) / 2)) ** 2 + ((y - cy) / ((Y - 2) / 3)) ** 2 <= 1
    p = torch.where(kind == 0, inside, torch.where(kind == 1, disc, ell) & inside)
    m = torch.zeros((n, 3, 64, 64), dtype=torch.bool, device="cuda")
    m[:, 1] = p
    v = torch.randn((n, 3, 64, 64, 3), device="cuda", generator=g, dtype=torch.float64)
    v = (v / v.norm(dim=-1, keepdim=True) * MS * m[..., None]).float()
    b = 0.05 * torch.rand((n,), device="cuda", generator=g).sqrt()
    ph = 2 * math.pi * torch.rand((n,), device="cuda", generator=g)
    bext = torch.stack([b * torch.cos(ph), b * torch.sin(ph), torch.zeros_like(b)], -1).double()
    grid = inside[:, None].expand(n, 3, 64, 64)
    return m, v, bext, grid


def _net_inputs(case, seed):
    """dimensionless charges of block-masked films and far fields a tenth off theirs: a network away from its optimum"""
    B, X, Y = case["batch"], case["X"], case["Y"]
    g = _gen(seed)
    u = []
    for _ in range(B):
        m = _mask("blocks", X, Y, 3, g)
        u.append(_div(_state("sphere", m, g).double() / MS, 1.0, 1.0, 1.0))
    u = torch.stack(u).float().contiguous()
    far = _far_exact(u.double())
    far = (far + 0.1 * far.std() * torch.randn(far.shape, device="cuda", generator=g, dtype=torch.float64))
    nrm2 = (_potential(u.double(), 1.0, 1.0, 1.0) ** 2).sum((1, 2, 3))
    return u, far.float().contiguous(), nrm2.float().contiguous()


def _weights():
    with np.load(WEIGHTS) as f:
        return np.ascontiguousarray(f["weights"], np.float32)


# ---- what a program keeps, and one pass ----------------------------------------
def _params(external=True):
    return mmsb200.make_params(Ms=MS, Aexch=AEX, alpha=ALPHA, gamma=GAMMA, mu0=MU0, external=external,
                               hext_t=HEXT_T, hext_b=HEXT_B)


def _context(case):
    kind = {"direct": mmsb200.SOLVER_DIRECT, "fmm": mmsb200.SOLVER_FMM, "net": mmsb200.SOLVER_SURROGATE}[case["solver"]]
    grid = mmsb200.Grid(case["X"], case["Y"], case["Z"], case["d"], case["d"], case["dz"])
    ctx = mmsb200.Context(grid, _params(), mmsb200.make_solver(kind, case["P"], case["leaf"]),
                          stream=STREAM.cuda_stream)
    if case["solver"] == "net":
        ctx.set_surrogate(_weights(), check_every=50, tol=1e-3)
    return ctx


def prepare(case, seed):
    k = case["kind"]
    s = {"case": case}
    if k == "gradient":
        s["u"], s["far"], s["nrm2"] = _net_inputs(case, seed)
        s["net"] = mmsb200.FarNet(case["X"], case["Y"], case["batch"])
        s["net"].set_weights(_weights())
        return s
    if k == "ensemble":
        m, v, bext, grid = _ens_inputs(case, seed)
        sel = grid.cpu().numpy()
        mh, vh = m.cpu().numpy(), v.cpu().numpy()
        dims = _ens_dims(case)
        s["ens"] = mmsens.Ensemble(dims, (5e-9, 5e-9, 5e-9), _params(), bext=bext.cpu().numpy(),
                                   stream=STREAM.cuda_stream)
        s["ens"].state_set([mh[i][sel[i]] for i in range(len(dims))], [vh[i][sel[i]] for i in range(len(dims))])
        s["out"] = np.empty(3 * s["ens"].cells, np.float32)
        return s
    s["ctx"] = _context(case)
    with torch.cuda.stream(STREAM):
        return _prepare_grid(case, seed, s)


def _prepare_grid(case, seed, s):
    k = case["kind"]
    m, M = _inputs(case, seed)
    if k == "potential":
        s["rho"] = _charge(case, M)
        s["phi"] = torch.empty_like(s["rho"])
    elif k == "field" and case["host"]:
        s["M"] = M.cpu().numpy()
    elif k == "field":
        s["M"], s["H"] = M, torch.empty_like(M)
        s["q"] = torch.empty(M.shape[:3], device="cuda")
        s["phi"] = torch.empty_like(s["q"])
    else:
        s["mat"], s["M"], s["out"] = m.to(torch.uint8).contiguous(), M, torch.empty_like(M)
    return s


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "gradient":
        loss, g = s["net"].gradient(s["u"], s["far"], s["nrm2"], case["batch"])
        return {"loss": np.float32(loss), "grad": g}
    if k == "ensemble":  # advance, then read every instance in the reference's float32
        s["ens"].run_fixed(DT, case["n"])
        M, _ = s["ens"].state_get()
        np.concatenate([a.reshape(-1) for a in M], out=s["out"], casting="same_kind")
        return s["out"]
    ctx = s["ctx"]
    if k == "potential":
        ctx.potential_dev(s["rho"], s["phi"])
        return s["phi"]
    if k == "field" and case["host"]:
        H, q, phi = ctx.hfield_host(s["M"], 2e-9)
        return {"H": H, "q": q, "phi": phi}
    if k == "field":
        ctx.hfield_dev(s["M"], s["H"], s["q"], s["phi"], 2e-9)
        return {"H": s["H"], "q": s["q"], "phi": s["phi"]}
    ctx.state_set_f32_dev(s["mat"], s["M"])
    if k == "march":
        ctx.march(case["final"], DT, mode=1, rtol=1e-5, torque_stop=0.0, max_records=1000)
    else:
        ctx.run_fixed(DT, case["n"])
    ctx.state_get_f32_dev(s["out"])
    return s["out"]


def work(case):
    """each input read and each output written once; per cell and field evaluation the stencils, the LLG
    right-hand side (about 110 operations) and what an N log N sum of 1/r takes"""
    N = _cells(case)
    k = case["kind"]
    if k == "gradient":
        B = case["batch"]
        leaves = B * -(-case["X"] // 8) * -(-case["Y"] // 8)
        per_leaf = 2 * 2 * 192 * 24 + 1.34 * (27 + 2) * 320 * 2  # encoder, decoder; lateral, down, up over the levels
        return {"bytes": 8 * B * N + 8 * 97856, "flops": 3 * leaves * per_leaf}
    demag = 20 * math.log2(4 * N)
    if k == "potential":
        return {"bytes": 8 * N, "flops": N * demag}
    if k == "field":
        return {"bytes": 32 * N, "flops": N * (demag + 60)}
    evals = 4 * case["n"] if k != "march" else 12 * max(1, round(case["final"] / 2e-13))
    return {"bytes": 25 * N, "flops": evals * N * (demag + 110)}


# ---- the same in 64 bits -------------------------------------------------------
def _nb(a, dim, step):
    """the neighbour of every cell `step` along dim, zero outside"""
    out = torch.zeros_like(a)
    n = a.shape[dim]
    if step > 0:
        out.narrow(dim, 0, n - 1).copy_(a.narrow(dim, 1, n - 1))
    else:
        out.narrow(dim, 1, n - 1).copy_(a.narrow(dim, 0, n - 1))
    return out


def _cd(a, dim, h):
    return (_nb(a, dim, 1) - _nb(a, dim, -1)) / (2 * h)


def _div(M, dx, dy, dz):
    return _cd(M[..., 0], -1, dx) + _cd(M[..., 1], -2, dy) + _cd(M[..., 2], -3, dz)


_kernels = {}


def _kernel(X, Y, Z, dx, dy, dz):
    key = (X, Y, Z, dx, dy, dz)
    if key not in _kernels:
        _kernels.clear()
        ax = [torch.arange(2 * n, device="cuda", dtype=torch.float64) for n in (X, Y, Z)]
        x, y, z = (torch.minimum(a, 2 * n - a) for a, n in zip(ax, (X, Y, Z)))
        r = torch.sqrt((x * dx)[None, None] ** 2 + (y * dy)[None, :, None] ** 2 + (z * dz)[:, None, None] ** 2)
        r[0, 0, 0] = 1.0
        G = dx * dy * dz / r
        G[0, 0, 0] = 0.0
        _kernels[key] = torch.fft.rfftn(G).real.clone()
    return _kernels[key]


def _potential(rho, dx, dy, dz):
    Z, Y, X = rho.shape[-3:]
    f = torch.fft.rfftn(rho, s=(2 * Z, 2 * Y, 2 * X), dim=(-3, -2, -1))
    f *= _kernel(X, Y, Z, dx, dy, dz)
    return torch.fft.irfftn(f, s=(2 * Z, 2 * Y, 2 * X), dim=(-3, -2, -1))[..., :Z, :Y, :X].clone()


def _h_exact(M, h, bext, grid=None):
    """(H, charge, potential) of M (.., Z, Y, X, 3); grid: the cells that belong to a smaller grid in this canvas"""
    dx, dy, dz = h
    q = _div(M, dx, dy, dz)
    if grid is not None:
        q = q * grid
    phi = _potential(q, dx, dy, dz)
    if grid is not None:
        phi = phi * grid
    c = 1 / (4 * math.pi)
    H = torch.stack([c * _cd(phi, -1, dx), c * _cd(phi, -2, dy), c * _cd(phi, -3, dz)], -1)
    cm = 2 * AEX / (MU0 * MS * MS)
    for dim, d in ((-2, dx), (-3, dy), (-4, dz)):
        H += cm / (d * d) * (_nb(M, dim, 1) + _nb(M, dim, -1) - 2 * M)
    return H + bext / MU0, q, phi


def _bext(t):
    w = min(max(t / 1e-8, 0.0), 1.0)
    return torch.tensor([(1 - w) * HEXT_B[0][0] + w * HEXT_B[1][0], 0.0, 0.0], device="cuda", dtype=torch.float64)


def _rk4(M, m, t, dt, field):
    def k(S, ts):
        H = field(S, ts)
        c = torch.linalg.cross(S, H)
        return -GAMMA * c - ALPHA * GAMMA / MS * torch.linalg.cross(S, c)

    m = m[..., None]
    k1 = k(M, t) * m
    k2 = k(M + dt / 2 * k1, t + dt / 2) * m
    k3 = k(M + dt / 2 * k2, t + dt / 2) * m
    k4 = k(M + dt * k3, t + dt) * m
    N = M + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
    return N * (MS / N.norm(dim=-1, keepdim=True).clamp(min=1e-300)) * m


def _march_exact(M, m, final, field):
    t, dt = 0.0, DT
    while t < final:
        h = min(dt, final - t)
        if h <= 0:
            break
        full = _rk4(M, m, t, h, field)
        half = _rk4(_rk4(M, m, t, h / 2, field), m, t + h / 2, h / 2, field)
        err = float((full - half).abs().max()) / MS
        fac = 0.9 * (1e-5 / err) ** 0.2 if err > 0 else 5.0
        dt = min(h * min(5.0, max(0.2, fac)), 1e-11)
        if err <= 1e-5:
            M, t = half, t + h
    return M


# the learned far field: a linear quadtree network over 8 x 8 x 3 leaf boxes,
# 16 even + 8 odd channels, tables per depth below the leaves
_NE, _NO, _NR, _C, _OSZ, _DEPTHS = 16, 8, 24, 192, 320, 5


def _far_exact(u):
    """the far field of u (B, 3, Y, X): the whole 1/r sum less that of the 3 x 3 leaf boxes around each"""
    phi = _potential(u, 1.0, 1.0, 1.0)
    q = _boxes(u)
    nb = q.shape[1]
    i = torch.arange(_C, device="cuda")
    xyz = torch.stack([i % 8, i // 8 % 8, i // 64], -1).double()
    P = torch.nn.functional.pad(q, (0, 0, 1, 1, 1, 1))
    near = torch.zeros_like(q)
    for oy in (-1, 0, 1):
        for ox in (-1, 0, 1):
            r = torch.cdist(xyz, xyz + torch.tensor([8.0 * ox, 8.0 * oy, 0.0], device="cuda", dtype=torch.float64),
                            compute_mode="donot_use_mm_for_euclid_dist")
            G = torch.where(r > 0, 1 / r.clamp(min=0.5), torch.zeros_like(r))
            near += P[:, 1 + oy:1 + oy + nb, 1 + ox:1 + ox + nb] @ G.T
    return phi - _unboxes(near, u.shape[-2], u.shape[-1])


def _boxes(u):
    B, Z, Y, X = u.shape
    nb = 1
    while nb * 8 < max(X, Y):
        nb *= 2
    q = torch.zeros((B, Z, nb * 8, nb * 8), device=u.device, dtype=u.dtype)
    q[:, :, :Y, :X] = u
    return q.reshape(B, Z, nb, 8, nb, 8).permute(0, 2, 4, 1, 3, 5).reshape(B, nb, nb, _C)


def _unboxes(b, Y, X):
    B, nb = b.shape[:2]
    return b.reshape(B, nb, nb, 3, 8, 8).permute(0, 3, 1, 4, 2, 5).reshape(B, 3, nb * 8, nb * 8)[:, :, :Y, :X]


def _blocks(v):
    """packed [even | odd] operators -> full 24 x 24"""
    n = v.shape[0]
    top = torch.cat([v[:, :256].reshape(n, _NE, _NE), v.new_zeros(n, _NE, _NO)], 2)
    low = torch.cat([v.new_zeros(n, _NO, _NE), v[:, 256:].reshape(n, _NO, _NO)], 2)
    return torch.cat([top, low], 1)


def _net_exact(w, u):
    B, _, Y, X = u.shape
    at = [0]

    def take(n):
        at[0] += n
        return w[at[0] - n:at[0]]

    W, V = take(_C * _NR).reshape(_C, _NR), take(_NR * _C).reshape(_NR, _C)
    m2l = [_blocks(take(49 * _OSZ).reshape(49, _OSZ)) for _ in range(_DEPTHS)]
    m2m, l2l = [None], [None]
    for _ in range(1, _DEPTHS):
        m2m.append(_blocks(take(4 * _OSZ).reshape(4, _OSZ)))
        l2l.append(_blocks(take(4 * _OSZ).reshape(4, _OSZ)))
    q = _boxes(u)
    L = q.shape[1].bit_length() - 1
    M = {L: q @ W}
    kids = [(0, 0), (1, 0), (0, 1), (1, 1)]
    for lev in range(L - 1, 1, -1):
        M[lev] = sum(M[lev + 1][:, cy::2, cx::2] @ m2m[L - lev][c] for c, (cx, cy) in enumerate(kids))
    F = None
    for lev in range(2, L + 1):
        n = 1 << lev
        par = torch.arange(n, device="cuda") & 1
        P = torch.nn.functional.pad(M[lev], (0, 0, 3, 3, 3, 3))
        acc = torch.zeros_like(M[lev])
        for oy in range(-3, 4):
            for ox in range(-3, 4):
                if max(abs(ox), abs(oy)) < 2:
                    continue
                mx = ((par - 3 <= ox) & (ox <= par + 2)).double()
                my = ((par - 3 <= oy) & (oy <= par + 2)).double()
                src = P[:, 3 - oy:3 - oy + n, 3 - ox:3 - ox + n]
                acc = acc + (my[:, None] * mx[None])[None, :, :, None] * (src @ m2l[L - lev][(oy + 3) * 7 + ox + 3])
        if F is not None:
            up = torch.zeros_like(acc)
            for c, (cx, cy) in enumerate(kids):
                up[:, cy::2, cx::2] = F @ l2l[L - lev + 1][c]
            acc = acc + up
        F = acc
    return _unboxes(F @ V, Y, X)


def exact(case, seed):
    k = case["kind"]
    if k == "gradient":
        u, far, nrm2 = (a.double() for a in _net_inputs(case, seed))
        w = torch.tensor(_weights(), device="cuda", dtype=torch.float64, requires_grad=True)
        loss = (((_net_exact(w, u) - far) ** 2).sum((1, 2, 3)) / nrm2).mean()
        loss.backward()
        return {"loss": loss.detach(), "grad": w.grad}
    if k == "ensemble":
        m, v, bext, grid = _ens_inputs(case, seed)
        M, b = v.double(), bext[:, None, None, None, :]
        for i in range(case["n"]):
            M = _rk4(M, m, i * DT, DT, lambda S, t: _h_exact(S, (5e-9, 5e-9, 5e-9), b, grid)[0])
        return M[grid].reshape(-1)
    m, M = _inputs(case, seed)
    h = (case["d"], case["d"], case["dz"])
    if k == "potential":
        return _potential(_charge(case, M).double(), *h)
    M = M.double()
    if k == "field":
        H, q, phi = _h_exact(M, h, _bext(2e-9))
        return {"H": H, "q": q, "phi": phi}

    def field(S, t):
        return _h_exact(S, h, _bext(t))[0]

    if k == "march":
        return _march_exact(M, m, case["final"], field)
    for i in range(case["n"]):
        M = _rk4(M, m, i * DT, DT, field)
    return M
