"""What a program that uses quarz_b200 has it do, as cases that can be timed and checked.

A host code calls the library at three levels: single operations on device arrays (moment sums, beam deposit,
push with the next deposit), the quasi-static sweep of one time step, and whole jobs (a run of many time steps,
a parameter scan, the gradient of a run). The listed cases take each level at its smallest, ordinary and
largest use; draw() gives more of the same ranges. Everything is FP64, as the library is.

exact() restates the operations and the sweep in numpy: complex azimuthal modes, tridiagonal systems by cyclic
reduction in extended precision. Runs of several time steps, scans and gradients have no such restatement that
ends in seconds, so exact() is None for them.
"""
import math

import numpy as np
import torch

import quarz_b200 as qz
from quarz_b200 import deck

# components of the field store, the beam sources and the diagnostics (include/qz_b200.h): for modes = 0 the
# first 6 / 5 / 3
NF, NB, ND = (6, 18), (5, 15), (3, 9)


# ---------------------------------------------------------------------------------------- cases
def listed():
    return [
        # moment sums of a small bunch after each step of a host code: latency and launches
        dict(name="moments_small", kind="moments", n=20_000),
        # the first deposit of a driver into the paper box (512 nodes, 2400 slices), particles as sampled
        dict(name="deposit_driver", kind="deposit", n=1_000_000, modes=0, cells=511, slices=2400, ngp=False, axis=5e-4),
        # one time step of a host code that keeps its own loop: push with the fields and the next deposit
        dict(name="step_m0", kind="step", n=2_000_000, modes=0, cells=511, slices=2400, ngp=False, axis=5e-4),
        # the same with azimuthal modes 0 and 1 and an odd particle count
        dict(name="step_m1", kind="step", n=600_011, modes=1, cells=511, slices=1200, ngp=False, axis=5e-4),
        # one sweep on the uniform 256-cell grid of the plain blowout
        dict(name="sweep_blowout", kind="sweep", modes=0, cells=256, slices=1200, length=12.0, axis=0.0, ppc=1,
             ntheta=1, ab=3, ngp=False, smooth=0.0),
        # one sweep of a fine radial grid: more plasma particles per slice than one thread block has threads
        dict(name="sweep_fine", kind="sweep", modes=0, cells=1000, slices=400, length=8.0, axis=2e-3, ppc=1,
             ntheta=1, ab=3, ngp=False, smooth=0.0),
        # one sweep with modes 0 and 1 on the hosing grid, 8 azimuths per ring
        dict(name="sweep_hosing", kind="sweep", modes=1, cells=511, slices=200, length=4.0, axis=5e-4, ppc=1,
             ntheta=8, ab=3, ngp=False, smooth=0.0),
        # the plain blowout run: 10 time steps, one driver of 1e5 particles, host beams in and out
        dict(name="run_blowout", kind="run", modes=0, cells=256, slices=1200, length=12.0, axis=0.0, steps=10,
             n=100_000, witness=0, ngp=False, smooth=0.0),
        # the pinched-witness run: 100 time steps, driver and witness of 1e6 particles each
        dict(name="run_witness", kind="run", modes=0, cells=511, slices=2400, length=12.0, axis=5e-4, steps=100,
             n=1_000_000, witness=1_000_000, ngp=False, smooth=0.0),
        # a hosing run (modes 0 and 1) over some time steps
        dict(name="run_hosing", kind="run", modes=1, cells=511, slices=1200, length=12.0, axis=5e-4, steps=12,
             n=500_000, witness=500_000, ngp=False, smooth=0.0),
        # a parameter scan: independent runs with grids of 128 to 1024 cells in one call
        dict(name="scan", kind="scan", modes=0, runs=200, cells_min=128, cells_max=1024, slices_min=400, slices_max=800,
             steps=2, n=5_000),
        # the gradient of the witness gain with respect to every beam particle
        dict(name="gradient", kind="gradient", cells=511, slices=2400, length=12.0, axis=5e-4, steps=8, n=200_000,
             witness=200_000),
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    kind = rng.choice(["moments", "deposit", "step", "sweep", "sweep", "run", "run", "scan", "gradient"])
    modes = rng.choice([0, 0, 1])
    axis = rng.choice([0.0, _log(rng, 5e-4, 5e-3)])
    ngp = rng.random() < 0.2
    if kind == "moments":
        return dict(kind=kind, n=int(_log(rng, 1e3, 2e6)))
    if kind in ("deposit", "step"):
        return dict(kind=kind, n=int(_log(rng, 1e3, 1e6 if modes == 0 else 4e5)), modes=modes,
                    cells=int(_log(rng, 32, 1024)), slices=int(_log(rng, 100, 1200)), ngp=ngp, axis=axis)
    if kind == "sweep":
        cells = int(_log(rng, 32, 1024 if modes == 0 else 1023))
        slices = int(_log(rng, 60, 900 if modes == 0 else 200))
        return dict(kind=kind, modes=modes, cells=cells, slices=slices, length=slices * rng.choice([0.005, 0.01]),
                    axis=axis if cells >= 64 else 0.0, ppc=2 if cells < 400 and rng.random() < 0.3 else 1,
                    ntheta=1 if modes == 0 else rng.choice([4, 8]), ab=rng.choice([2, 3, 3, 3, 4, 5]), ngp=ngp,
                    smooth=0.005 if rng.random() < 0.25 else 0.0)
    if kind == "run":
        slices = int(_log(rng, 150, 1000 if modes == 0 else 300))
        return dict(kind=kind, modes=modes, cells=int(_log(rng, 64, 800 if modes == 0 else 511)), slices=slices,
                    length=slices * 0.01, axis=axis, steps=rng.randint(1, 20 if modes == 0 else 6),
                    n=int(_log(rng, 5e3, 3e5)), witness=rng.choice([0, int(_log(rng, 5e3, 3e5))]), ngp=ngp,
                    smooth=0.005 if rng.random() < 0.2 else 0.0)
    if kind == "scan":
        lo = int(_log(rng, 32, 400))
        return dict(kind=kind, modes=modes, runs=rng.randint(8, 180 if modes == 0 else 40), cells_min=lo,
                    cells_max=min(1023, lo + int(_log(rng, 8, 600))), slices_min=100, slices_max=rng.randint(120, 400),
                    steps=rng.randint(1, 3), n=int(_log(rng, 500, 5000)))
    slices = int(_log(rng, 150, 800))
    return dict(kind="gradient", cells=int(_log(rng, 64, 511)), slices=slices, length=slices * 0.01, axis=axis,
                steps=rng.randint(1, 8), n=int(_log(rng, 5e3, 1e5)), witness=int(_log(rng, 5e3, 1e5)))


# ---------------------------------------------------------------------------------------- inputs
def _nodes(cells, axis, R=6.0):
    """Uniform cells (axis = 0), or geometric ones from `axis` at the axis up to at most 0.05 at the wall."""
    if axis <= 0.0 or axis * cells >= R:
        return R * np.arange(cells + 1) / cells
    cap = max(0.05, 1.5 * R / cells)
    lo, hi = 1.0, 2.0
    for _ in range(200):
        q = 0.5 * (lo + hi)
        h = np.minimum(axis * q ** np.minimum(np.arange(cells), 600.0 / math.log(max(q, 1.0 + 1e-9))), cap)
        lo, hi = (q, hi) if h.sum() < R else (lo, q)
    r = np.concatenate([[0.0], np.cumsum(h)]) * (R / h.sum())
    r[-1] = R
    return r


def _bunch(g, n, n0, sr, sxi, xi0, x0=0.0):
    """A Gaussian bunch (n, 7): x y px py pz xi w, internal xi, cut at 3 sigma in xi; gamma 1000."""
    z = g.standard_normal((n, 6))
    t = z[:, 5]
    t = np.where(np.abs(t) < 3.0, t, 3.0 * (2.0 * g.random(n) - 1.0))
    p = np.empty((n, 7))
    p[:, 0] = np.clip(sr * z[:, 0], -4 * sr, 4 * sr) + x0
    p[:, 1] = np.clip(sr * z[:, 1], -4 * sr, 4 * sr)
    p[:, 2] = 0.1 * z[:, 2]
    p[:, 3] = 0.1 * z[:, 3]
    p[:, 4] = 1000.0 * (1.0 + 1e-3 * z[:, 4])
    p[:, 5] = xi0 + sxi * t
    p[:, 6] = n0 * (2.0 * math.pi) ** 1.5 * sr * sr * sxi / n
    return p


def _beams(g, case, length, n, witness, x0):
    """The driver (and the witness) of a box of that length: centres at a quarter and at 5/8 of it."""
    s = length / 12.0
    out = [_bunch(g, n, g.uniform(3.0, 6.0), 0.5, 1.0 * s, 0.25 * length, x0)]
    if witness:
        out.append(_bunch(g, witness, 20.0, 0.02, 0.1 * s, 0.625 * length, 0.2 * x0))
    return out


def _spec(case, nodes, beams=0, modes=None, slices=None, length=None):
    """The run set-up a deck gives (quarz_b200.deck), with this case's nodes."""
    modes = case["modes"] if modes is None else modes
    K = case["slices"] if slices is None else slices
    dxi = (case["length"] if length is None else length) / K
    names = ["driver", "witness"][:beams]
    text = "xi.convention = z-t\ngrid.type = uniform\ngrid.rmax = 6\ngrid.dr = 1\nxi.min = %r\nxi.max = 0\nxi.step = %r\n" % (
        -(K - 1) * dxi, dxi)
    text += "modes = %d\ntime.dt = 5\ntime.steps = %d\nplasma.species = electrons\nelectrons.ppc = %d\n" % (
        modes, case.get("steps", 1), case.get("ppc", 1))
    if modes:
        text += "electrons.ntheta = %d\nsolver.picard = 3\n" % case.get("ntheta", 8 if case["kind"] != "scan" else 4)
    text += "pusher.ab_order = %d\nplasma.smooth_length = %r\n" % (case.get("ab", 3), case.get("smooth", 0.0))
    if case.get("ngp"):
        text += "beams.xi_shape = ngp\n"
    if names:
        text += "beams = %s\n" % " ".join(names)
    for b in names:                                       # the particles are given; these are only required keys
        text += "%s.n0 = 1\n%s.sigma_r = 0.5\n%s.sigma_xi = 1\n%s.xi0 = -3\n%s.gamma = 1000\n" % (b, b, b, b, b)
    spec = deck.run_spec(deck.parse_deck(text))
    spec.nodes = nodes
    spec.K = K
    return spec


def _op_inputs(case, seed):
    """Particles, box and (for a step) fields of the single operations, on the host."""
    g = np.random.default_rng(seed)
    modes, K = case["modes"], case["slices"]
    nodes = _nodes(case["cells"], case["axis"])
    length = 12.0
    half = case["n"] // 2
    x0 = 0.1 if modes else 0.0
    p = np.concatenate(_beams(g, case, length, case["n"] - half, half, x0))
    fld = None
    if case["kind"] == "step":                            # smooth wake fields of both modes
        xi = (np.arange(K) * (length / K))[:, None]
        r = nodes[None, :]
        a = g.uniform(0.5, 1.0, 4)
        fld = np.zeros((K, case["cells"] + 1, NF[modes]))
        well = np.exp(-r * r / 8.0) * (1.0 - np.exp(-xi))
        fld[..., 0] = 0.5 * r * well
        fld[..., 1] = 0.02 * r * well * np.cos(a[0] * xi)
        fld[..., 2] = 0.01 * r * well
        fld[..., 3] = -0.25 * r * well * np.sin(a[1] * xi)
        fld[..., 4] = a[2] * np.sin(0.7 * xi) * np.exp(-r * r / 4.0)
        fld[..., 5] = 0.01 * a[3] * np.cos(0.7 * xi) * np.exp(-r * r / 4.0)
        for c in range(6, NF[modes]):
            fld[..., c] = 0.02 * math.cos(c) * (r if c > 13 else 1.0) * well * np.sin(a[c % 4] * xi + c)
    return nodes, length / K, p, fld


def _sweep_inputs(case, seed):
    """The beam sources (K, M, 5 or 15) of a Gaussian driver with particle noise, on the host."""
    g = np.random.default_rng(seed)
    K, modes = case["slices"], case["modes"]
    nodes = _nodes(case["cells"], case["axis"])
    L = case["length"]
    xi = (np.arange(K) * (L / K))[:, None]
    r = nodes[None, :]
    n0 = g.uniform(1.0, 4.0)
    rho = -n0 * np.exp(-0.5 * (r / 0.5) ** 2 - 0.5 * ((xi - 0.3 * L) / (0.09 * L)) ** 2)
    rho = rho * (1.0 + 0.01 * g.standard_normal(rho.shape))
    b = np.zeros((K, case["cells"] + 1, NB[modes]))
    b[..., 0], b[..., 1], b[..., 4] = 5e-7 * rho, rho, rho
    b[..., 2], b[..., 3] = 1e-5 * rho * r, 1e-5 * rho * r * g.standard_normal()
    if modes:
        d = 0.1 * r / 0.25 * 0.5                           # a driver displaced by 0.1
        for c, f in ((5, 5e-7), (7, 1.0), (13, 1.0)):
            b[..., c] = f * rho * d
            b[..., c + 1] = 0.1 * f * rho * d * g.uniform(0.5, 1.0)
        b[..., 9], b[..., 11] = 1e-5 * rho, 1e-6 * rho * r * r
    return nodes, b


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _zeros(*shape):
    return torch.zeros(shape, dtype=torch.float64, device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "moments":
        p = _bunch(np.random.default_rng(seed), case["n"], 5.0, 0.5, 1.0, 3.0)
        return dict(case=case, cols=_cuda(p.T), out=_zeros(17))
    if kind in ("deposit", "step"):
        nodes, dxi, p, fld = _op_inputs(case, seed)
        s = dict(case=case, grid=qz.RadialGrid(nodes), cols=_cuda(p.T), bsrc=_zeros(case["slices"], len(nodes), NB[case["modes"]]),
                 box=qz.BeamOps.box(0.0, dxi, case["slices"], case["ngp"], case["modes"]))
        if kind == "step":
            s.update(fld=_cuda(fld), old=s["cols"].clone())
        return s
    if kind == "sweep":
        nodes, b = _sweep_inputs(case, seed)
        spec = _spec(case, nodes)
        K, M = spec.K, len(nodes)
        sweep = qz.Sweep(qz.RadialGrid(nodes), qz.sweep_params(spec))
        return dict(case=case, sweep=sweep, bsrc=_cuda(b), fld=_zeros(K, M, NF[case["modes"]]), diag=_zeros(K, M, ND[case["modes"]]))
    g = np.random.default_rng(seed)
    if kind in ("run", "gradient"):
        modes = case.get("modes", 0)
        nodes = _nodes(case["cells"], case["axis"])
        beams = _beams(g, case, case["length"], case["n"], case["witness"], 0.1 if modes else 0.0)
        spec = _spec(case, nodes, len(beams), modes)
        sim = qz.Simulation(spec, beams=[(p, 1000.0, float(p[:, 5].mean())) for p in beams])
        if kind == "gradient":
            seeds = np.zeros((len(beams), 17))
            seeds[1, 1] = 1.0 / beams[1][:, 6].sum()      # the witness's mean gamma
            return dict(case=case, sim=sim, cols=[_cuda(p.T) for p in beams], seeds=seeds)
        cols = [torch.from_numpy(np.ascontiguousarray(p.T)).pin_memory() for p in beams]
        return dict(case=case, sim=sim, cols=cols, work=[torch.empty_like(c).pin_memory() for c in cols])
    batch = qz.Batch()
    kept = []
    for _ in range(case["runs"]):
        cells = int(g.integers(case["cells_min"], case["cells_max"] + 1))
        K = int(g.integers(case["slices_min"], case["slices_max"] + 1))
        nodes = _nodes(cells, float(np.exp(g.uniform(np.log(5e-4), np.log(5e-3)))))
        beams = _beams(g, case, 0.01 * K, case["n"], case["n"], 0.1 if case["modes"] else 0.0)
        rows = [(p, 1000.0, float(p[:, 5].mean())) for p in beams]
        batch.add(_spec(case, nodes, len(beams), slices=K, length=0.01 * K), rows)
        kept.append(rows)
    return dict(case=case, batch=batch, kept=kept)


# ---------------------------------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "moments":
        qz.BeamOps.sums(state["cols"], 1000.0, 3.0, state["out"])
        return state["out"]
    if kind == "deposit":
        state["bsrc"].zero_()
        qz.BeamOps.deposit(state["grid"], state["cols"], -1.0, 1.0, state["box"], state["bsrc"])
        return state["bsrc"]
    if kind == "step":                                    # the particles of the step before, pushed and deposited
        state["cols"].copy_(state["old"])
        state["bsrc"].zero_()
        qz.BeamOps.push_deposit(state["grid"], state["cols"], -1.0, 1.0, state["box"], state["fld"], 5.0, 5.0, 1, state["bsrc"])
        return dict(cols=state["cols"], bsrc=state["bsrc"])
    if kind == "sweep":
        state["sweep"].run(state["bsrc"], state["fld"], state["diag"])
        return dict(fld=state["fld"], diag=state["diag"])
    if kind == "run":                                     # host beams copied in, the run, and out again
        for w, c in zip(state["work"], state["cols"]):
            w.copy_(c)
        state["sim"].restart()
        mom = state["sim"].run_host(case["steps"], 5.0, state["work"])
        return dict(moments=mom, beams=state["work"])
    if kind == "gradient":
        state["sim"].restart()
        for b, c in enumerate(state["cols"]):
            state["sim"].set_beam(b, c)
        lam, mom, _ = state["sim"].adjoint(case["steps"], 5.0, state["seeds"])
        return dict(gradient=lam, moments=mom)
    # a batch goes on from where it stands (no entry point sets its beams back), so every pass takes the next
    # steps of all its runs
    return np.concatenate([m.reshape(-1) for m in state["batch"].run(case["steps"], 5.0)])


# ---------------------------------------------------------------------------------------- what a pass needs
def work(case):
    """Bytes: every input read and every output written once. Operations: counted from the update formulas,
    about 60 (deposit), 200 (push with the gather) and 45 (moments) per beam particle, 350 per plasma particle
    and slice and 120 per node and slice for m = 0; 2.5 to 4 times as many with mode 1."""
    kind, modes = case["kind"], case.get("modes", 0)
    if kind == "moments":
        return dict(bytes=56.0 * case["n"], flops=45.0 * case["n"])
    big = 1.0 + 2.0 * modes

    def sweep(cells, slices, ppc, ntheta, wide):
        nodes = (cells + 1.0) * slices
        read = (12 if modes else 3)                       # the source components a sweep reads
        w = 3.0 if modes else 1.0
        return (8.0 * nodes * ((read if wide else 0) + NF[modes] + ND[modes]),
                nodes * 120.0 * (4.0 if modes else 1.0) + cells * ppc * ntheta * slices * 350.0 * w)

    if kind in ("deposit", "step"):
        store = 8.0 * (case["cells"] + 1) * case["slices"]
        if kind == "deposit":
            return dict(bytes=56.0 * case["n"] + store * NB[modes], flops=60.0 * big * case["n"])
        return dict(bytes=112.0 * case["n"] + store * (NF[modes] + NB[modes]), flops=260.0 * big * case["n"])
    if kind == "sweep":
        b, f = sweep(case["cells"], case["slices"], case["ppc"], case["ntheta"], True)
        return dict(bytes=b, flops=f)
    if kind == "scan":
        cells = 0.5 * (case["cells_min"] + case["cells_max"])
        slices = 0.5 * (case["slices_min"] + case["slices_max"])
        b, f = sweep(cells, slices, 1, 4 if modes else 1, True)
        s, n = case["steps"], 2.0 * case["n"]
        return dict(bytes=case["runs"] * ((s + 1) * b + s * 112.0 * n), flops=case["runs"] * ((s + 1) * f + s * n * 305.0 * big))
    b, f = sweep(case["cells"], case["slices"], 1, 8 if modes else 1, True)
    s, n = case["steps"], float(case["n"] + case["witness"])
    k = 3.0 if kind == "gradient" else 1.0                # forward, its records, reverse
    return dict(bytes=k * ((s + 1) * b + s * 112.0 * n), flops=k * ((s + 1) * f + s * n * 305.0 * big))


def tolerance(case):
    """About four times what was seen against exact(), or between summation orders (FP64 reductions against exact
    integer sums, one launch against step by step). A sweep whose box reaches the closure of the blowout bubble
    amplifies rounding by some five orders there: 1.6e-8 was seen on 1000 cells, 3e-11 in shorter boxes."""
    kind = case["kind"]
    if kind in ("moments", "deposit", "step"):
        return {"rel": 1e-12}
    if kind == "sweep":
        return {"rel": 6e-8 if case["length"] > 6.0 else 2e-10}
    return {"rel": 1e-9 if kind == "gradient" else 1e-10}


# ---------------------------------------------------------------------------------------- plain restatement
def exact(case, seed):
    kind = case["kind"]
    if kind == "moments":
        p = _bunch(np.random.default_rng(seed), case["n"], 5.0, 0.5, 1.0, 3.0)
        x, y, px, py, pz, xi, w = p.T
        G = np.sqrt(1.0 + px * px + py * py + pz * pz) - 1000.0
        d = xi - 3.0
        one = np.ones_like(G)
        rows = [one, G, G * G, d, d * d, x * x + y * y, x, y, x * x, y * y, px, py, px * px, py * py, x * px, y * py]
        return torch.tensor([math.fsum(w * v) for v in rows] + [float(case["n"])], dtype=torch.float64)
    if kind in ("deposit", "step"):
        nodes, dxi, p, fld = _op_inputs(case, seed)
        if kind == "deposit":
            return torch.from_numpy(_deposit(case, nodes, dxi, p))
        p = _push(case, nodes, dxi, p, fld, 5.0)
        return dict(cols=torch.from_numpy(np.ascontiguousarray(p.T)), bsrc=torch.from_numpy(_deposit(case, nodes, dxi, p)))
    if kind == "sweep":
        nodes, b = _sweep_inputs(case, seed)
        fld, diag = _sweep(case, nodes, b)
        return dict(fld=torch.from_numpy(fld), diag=torch.from_numpy(diag))
    return None


def _volumes(r):
    h = np.diff(r)
    v = np.zeros(len(r))
    v[1:] += r[:-1] * h / 2 + h * h / 3
    v[:-1] += r[:-1] * h / 2 + h * h / 6
    return 2 * math.pi * v


def _cell(r, x):
    j = np.clip(np.searchsorted(r, x, side="right") - 1, 0, len(r) - 2)
    return j, np.clip((x - r[j]) / (r[j + 1] - r[j]), 0.0, 1.0)


def _deposit(case, r, dxi, p):
    """Linear (or nearest-slice) in xi, linear in r; the charge density's share rho - J_z, J_z, J_perp e^{-i k theta}."""
    modes, K, M = case["modes"], case["slices"], len(r)
    x, y, px, py, pz, xi, w = p[p[:, 6] != 0.0].T
    R2 = np.sqrt(x * x + y * y)
    s = xi / dxi
    k = np.floor(s + 0.5 if case["ngp"] else s).astype(np.int64)
    keep = (R2 <= r[-1]) & (k >= -1) & (k < K)
    x, y, px, py, pz, w, R2, s, k = (a[keep] for a in (x, y, px, py, pz, w, R2, s, k))
    th = (x + 1j * y) / np.where(R2 > 0, R2, 1.0)
    th[R2 == 0] = 1.0
    gam = np.sqrt(1.0 + px * px + py * py + pz * pz)
    om = (1.0 + px * px + py * py) / (gam * (gam + pz))
    vz, v = pz / gam, (px + 1j * py) / gam
    j, t = _cell(r, R2)
    V = _volumes(r)
    tk = np.zeros_like(s) if case["ngp"] else s - k
    out = np.zeros((K * M, NB[modes]))
    v0, v1, v2 = (v * np.conj(th) ** m for m in range(3))
    c, sn = th.real, th.imag
    comps = [om, vz, v1.real, v1.imag, np.ones_like(om)]
    if modes:
        comps += [om * c, -om * sn, vz * c, -vz * sn, v0.real, v0.imag, v2.real, v2.imag, c, -sn]
    for a in range(1 if case["ngp"] else 2):
        for b in range(2):
            kk, jj = k + a, j + b
            d = -w * (tk if a else 1.0 - tk) * (t if b else 1.0 - t) / V[jj] / dxi
            ok = (kk >= 0) & (kk < K)
            at = (kk * M + jj)[ok]
            for c, f in enumerate(comps):
                out[:, c] += np.bincount(at, (d * f)[ok], K * M)
    return out.reshape(K, M, NB[modes])


def _push(case, r, dxi, p, fld, dt):
    modes, K = case["modes"], case["slices"]
    x, y, px, py, pz, xi, w = p.T.copy()
    R2 = np.sqrt(x * x + y * y)
    th = (x + 1j * y) / np.where(R2 > 0, R2, 1.0)
    th[R2 == 0] = 1.0
    s = xi / dxi
    if case["ngp"]:
        k = np.clip(np.floor(s + 0.5).astype(np.int64), 0, K - 1)
        tk, k1 = np.zeros_like(s), k
    else:
        k = np.floor(s).astype(np.int64)
        s = np.where(k < 0, 0.0, np.where(k > K - 2, K - 1.0, s))
        k = np.clip(k, 0, K - 2)
        tk, k1 = s - k, k + 1
    j, t = _cell(r, R2)

    def at(c):
        return ((1 - tk) * ((1 - t) * fld[k, j, c] + t * fld[k, j + 1, c])
                + tk * ((1 - t) * fld[k1, j, c] + t * fld[k1, j + 1, c]))

    def vec(c1, c0, c2):
        v = (at(c1) + 1j * at(c1 + 1)) * th
        if modes:
            v = v + (at(c0) + 1j * at(c0 + 1)) + (at(c2) + 1j * at(c2 + 1)) * th * th
        return v

    E, B = vec(0, 6, 8), vec(2, 10, 12)
    Ez, Bz = at(4), at(5)
    if modes:
        Ez = Ez + 2.0 * ((at(14) + 1j * at(15)) * th).real
        Bz = Bz + 2.0 * ((at(16) + 1j * at(17)) * th).real
    E = np.stack([E.real, E.imag, Ez], 1)
    B = np.stack([B.real, B.imag, Bz], 1)
    u = np.stack([px, py, pz], 1)
    eps = -0.5 * dt
    g0 = np.sqrt(1.0 + (u * u).sum(1))[:, None]
    a = u + 2 * eps * E + (eps / g0) * np.cross(u, B)     # Vay (2008)
    b = eps * B
    b2, ab = (b * b).sum(1), (a * b).sum(1)
    h, c = 0.5 * (1.0 + (a * a).sum(1) - b2), b2 + ab * ab
    root = np.sqrt(h * h + c)
    g2 = np.where(h >= 0, h + root, c / np.where(root > h, root - h, 1.0))
    u = (g2[:, None] * a + np.sqrt(g2)[:, None] * np.cross(a, b) + ab[:, None] * b) / (g2 + b2)[:, None]
    p2 = u[:, 0] ** 2 + u[:, 1] ** 2
    gam = np.sqrt(1.0 + p2 + u[:, 2] ** 2)
    xn, yn = x + u[:, 0] / gam * dt, y + u[:, 1] / gam * dt
    xin = xi + (1.0 + p2) / (gam * (gam + u[:, 2])) * dt
    gone = (xn * xn + yn * yn >= r[-1] ** 2) | (xin < 0.0) | (xin > (K - 1) * dxi)
    return np.stack([xn, yn, u[:, 0], u[:, 1], u[:, 2], xin, np.where(gone, 0.0, w)], 1)


def _tri(a, b, c, d):
    """Tridiagonal systems by cyclic reduction in extended precision, rows last."""
    a, b, c, d = (np.array(v, dtype=np.longdouble) for v in (a, b, c, d))
    M = b.shape[-1]
    a[..., 0] = 0.0
    c[..., -1] = 0.0
    st = 1
    while st < M:
        al, ga = np.zeros_like(b), np.zeros_like(b)
        al[..., st:] = -a[..., st:] / b[..., :-st]
        ga[..., :-st] = -c[..., :-st] / b[..., st:]
        na, nc, nb, nd = np.zeros_like(b), np.zeros_like(b), b.copy(), d.copy()
        na[..., st:] = al[..., st:] * a[..., :-st]
        nb[..., st:] += al[..., st:] * c[..., :-st]
        nd[..., st:] += al[..., st:] * d[..., :-st]
        nc[..., :-st] = ga[..., :-st] * c[..., st:]
        nb[..., :-st] += ga[..., :-st] * a[..., st:]
        nd[..., :-st] += ga[..., :-st] * d[..., st:]
        a, b, c, d = na, nb, nc, nd
        st *= 2
    return (d / b).astype(np.float64)


def _rows(r, n, a2=None):
    """Finite-volume rows of the radial operator of angular number n (identity rows at both ends)."""
    h, mid = np.diff(r), 0.5 * (r[1:] + r[:-1])
    M = len(r)
    a, b, c = np.zeros(M), np.ones(M), np.zeros(M)
    i = slice(1, M - 1)
    dV = 0.5 * (h[1:] + h[:-1])
    pre = r[i] ** (n - 1) / dV
    kp = (1.0 if a2 is None else a2) / (h * mid ** (2 * n - 1))
    c[i] = pre * r[2:] ** n * kp[1:]
    a[i] = pre * r[:-2] ** n * kp[:-1]
    b[i] = -pre * r[i] ** n * (kp[1:] + kp[:-1])
    return a, b, c


def _sweep(case, r, bsrc):
    """The quasi-static slice loop: scalars f[0], f[1] (modes 0, 1) and vectors v[0..2] (V+ = sum v_k e^{i k theta})."""
    modes, K, M, N = case["modes"], case["slices"], len(r), len(r) - 1
    dxi = case["length"] / K
    R = r[-1]
    h, mid, V = np.diff(r), 0.5 * (r[1:] + r[:-1]), _volumes(r)
    ns, vk = (2, (1, 0, 2)) if modes else (1, (1,))
    # operators
    iV = 2 * math.pi / V
    L0 = [np.zeros(M), np.ones(M), np.zeros(M)]
    L0[0][1:N] = mid[:N - 1] / h[:N - 1] * iV[1:N]
    L0[2][:N] = mid / h * iV[:N]
    L0[1][:N] = -(L0[0][:N] + L0[2][:N])
    L1D, L2D = _rows(r, 1), _rows(r, 2)
    L1F = [v.copy() for v in L1D]
    fc = 1.0 / (0.5 * h[-1])
    L1F[0][N] = r[N - 1] * fc / (h[-1] * mid[-1])
    L1F[1][N] = -r[N] * fc / (h[-1] * mid[-1])
    a2 = case["smooth"] ** 2
    F = []
    if a2 > 0:
        am, cp = np.zeros(M), np.zeros(M)
        am[1:] = a2 * mid / h * iV[1:]
        cp[:N] = a2 * mid / h * iV[:N]
        F.append((-am, 1 + am + cp, -cp))
        for n in (1, 2):
            a, b, c = _rows(r, n, a2)
            b = 1.0 - b
            b[0] = b[N] = 1.0
            F.append((-a, b, -c))

    def filt(n, f):
        if not F:
            return f
        a, b, c = (np.broadcast_to(v, f.shape) for v in F[n])
        if np.iscomplexobj(f):
            return _tri(a, b, c, f.real) + 1j * _tri(a, b, c, f.imag)
        return _tri(a, b, c, f)

    hm, hp = h[:-1], h[1:]
    den = hm * hp * (hm + hp)

    def grad(f, odd):
        o = np.empty_like(f)
        o[0] = f[1] / r[1] if odd else 0.0
        o[1:N] = (-hp * hp * f[:-2] + (hp * hp - hm * hm) * f[1:N] + hm * hm * f[2:]) / den
        h1, h2 = h[-1], h[-2]
        o[N] = (2 * h1 + h2) / (h1 * (h1 + h2)) * f[N] - (h1 + h2) / (h1 * h2) * f[N - 1] + h1 / (h2 * (h1 + h2)) * f[N - 2]
        return o

    def over(f):
        o = f.copy()
        o[1:] = f[1:] / r[1:]
        o[0] = f[1] / r[1]
        return o

    def solve(op, rhs, chi=None, regular=False, wall=None):
        """rhs: one or more systems (.., M); Dirichlet rows hold 0."""
        a, b, c = (np.array(v) for v in op)
        d = np.array(rhs, dtype=np.float64)
        if chi is not None:
            lo, hi = (0 if regular else 1), (M if wall is not None else N)
            b[lo:hi] = b[lo:hi] - chi[lo:hi]
        if not regular:
            d[..., 0] = 0.0
        if wall is None:
            d[..., N] = 0.0
        else:
            d[..., N] -= fc * wall
        return _tri(*(np.broadcast_to(v, d.shape) for v in (a, b, c)), d)

    def csolve(op, rhs, **kw):
        o = solve(op, np.stack([rhs.real, rhs.imag]), **kw)
        return o[0] + 1j * o[1]

    # plasma
    ppc, nth = case["ppc"], case["ntheta"]
    e = (r[:-1, None] + np.arange(ppc + 1)[None, :] * (h[:, None] / ppc))
    ra, rb = e[:, :-1].ravel(), e[:, 1:].ravel()
    rr = (2.0 / 3.0) * (rb ** 3 - ra ** 3) / (rb ** 2 - ra ** 2)
    wr = math.pi * (rb ** 2 - ra ** 2) / nth
    off = (np.arange(len(rr)) % 2) * 0.5
    ang = 2 * math.pi * (np.arange(nth)[None, :] + off[:, None]) / nth
    X = (rr[:, None] * np.exp(1j * ang) if nth > 1 else rr[:, None] + 0j).ravel()
    w = np.repeat(wr, nth)
    P, D = np.zeros_like(X), np.ones(len(w))
    q = qm = -1.0
    AB = {2: [3 / 2, -1 / 2], 3: [23 / 12, -16 / 12, 5 / 12], 4: [55 / 24, -59 / 24, 37 / 24, -9 / 24],
          5: [1901 / 720, -2774 / 720, 2616 / 720, -1274 / 720, 251 / 720]}[case["ab"]]
    hist = []

    def geo(X):
        x = np.abs(X)
        th = np.where(x > 0, X / np.where(x > 0, x, 1.0), 1.0)
        j, t = _cell(r, x)
        ih = 1.0 / h[j]
        ir = np.where(x > 0, 1.0 / np.where(x > 0, x, 1.0), 0.0)
        Wor = (np.where(j == 0, 0.0, (1 - t) * ir), np.where(j == 0, ih, t * ir))
        return j, th, (1 - t, t), (-ih, ih), Wor

    def add(j, vals):
        """vals: pairs (left, right) of complex or real particle values -> nodes"""
        out = []
        for v in vals:
            f = 0
            for cc in range(2):
                if np.iscomplexobj(v[cc]):
                    f = f + np.bincount(j + cc, v[cc].real, M) + 1j * np.bincount(j + cc, v[cc].imag, M)
                else:
                    f = f + np.bincount(j + cc, v[cc], M)
            out.append(f / V)
        return out

    def at(f, g):
        j, W = g[0], g[2]
        return W[0] * f[j] + W[1] * f[j + 1]

    def vec(v, g):
        return sum(at(v[k], g) * g[1] ** k for k in vk)

    def scal(f, g):
        return at(f[0], g) + (2.0 * (at(f[1], g) * g[1]).real if modes else 0.0)

    live = w != 0
    g0 = geo(X)
    bg = add(g0[0], [[-q * w * g0[2][cc] * np.conj(g0[1]) ** m for cc in range(2)] for m in range(ns)])
    bg[0] = np.real(bg[0])
    bg = [filt(m, bg[m]) for m in range(ns)]
    col = [(0, 0), (5, 6)]

    def beam(k, c):
        return [bsrc[k, :, c[0]]] + ([bsrc[k, :, c[1]] + 1j * bsrc[k, :, c[1] + 1]] if modes else [])

    fld = np.zeros((K, M, NF[modes]))
    diag = np.zeros((K, M, ND[modes]))
    bp = {k: np.zeros(M, dtype=complex) for k in range(3)}
    idx = np.arange(len(w))
    for k in range(K):
        idx = np.nonzero(live)[0]
        x, p, d, ww = X[idx], P[idx], D[idx], w[idx]
        g = geo(x)
        j, th, W, dW, Wor = g
        gam = (1.0 + np.abs(p) ** 2 + d * d) / (2 * d)
        u = p / d
        ul = u * np.conj(th)                               # u_r + i u_theta
        wq = ww * q
        vals = []
        for m in range(ns):
            ph = np.conj(th) ** m if m else 1.0
            vals.append([wq * W[cc] * ph for cc in range(2)])
            vals.append([(wq * ul.real * dW[cc] - m * 1j * wq * ul.imag * Wor[cc]) * ph if m else wq * ul.real * dW[cc] for cc in range(2)])
            vals.append([wq * W[cc] * (gam - d) / d * ph for cc in range(2)])
            vals.append([wq * W[cc] * qm / d * ph for cc in range(2)])
            vals.append([ww * W[cc] * gam / d * ph for cc in range(2)])
        for m in vk:
            vals.append([wq * W[cc] * u * np.conj(th) ** m for cc in range(2)])
        vals = add(j, vals)
        rhot, drho, jz, chi, ne = ([filt(m, vals[5 * m + i]) for m in range(ns)] for i in range(5))
        jp = {m: filt(m, vals[5 * ns + i]) for i, m in enumerate(vk)}
        # beams: rho - J_z and its xi-derivative, J_z, J_perp
        brt, bjz = beam(k, (0, 5)), beam(k, (1, 7))
        if case["ngp"]:
            pr = beam(k - 1, (0, 5)) if k else [np.zeros(M)] * ns
            dr = [(brt[m] - pr[m]) / dxi for m in range(ns)]
        elif K == 1:
            dr = [np.zeros(M)] * ns
        else:
            lo, hi = beam(max(k - 1, 0), (0, 5)), beam(min(k + 1, K - 1), (0, 5))
            dr = [(hi[m] - lo[m]) / dxi * (0.5 if 0 < k < K - 1 else 1.0) for m in range(ns)]
        for m in range(ns):
            rhot[m] = rhot[m] + bg[m] + brt[m]
            drho[m] = drho[m] + dr[m]
            jz[m] = jz[m] + bjz[m]
        jp[1] = jp[1] + bsrc[k, :, 2] + 1j * bsrc[k, :, 3]
        if modes:
            jp[0] = jp[0] + bsrc[k, :, 9] + 1j * bsrc[k, :, 10]
            jp[2] = jp[2] + bsrc[k, :, 11] + 1j * bsrc[k, :, 12]
        ni = np.where(bg[0] > 0, bg[0], 0.0)
        # psi, E_z, B_z
        bz0 = -(grad(jp[1].imag, True) + over(jp[1].imag))
        s0 = solve(L0, np.stack([-rhot[0], -drho[0], bz0]), regular=True)
        psi, ez, bz = [s0[0]], [s0[1]], [s0[2]]
        if modes:
            D1 = grad(jp[2], True) + 2.0 * over(jp[2])
            Dm = grad(jp[0], False)
            b1 = -0.5 * (D1.imag + Dm.imag) + 0.5j * (D1.real - Dm.real)
            for lst, rhs in ((psi, -rhot[1]), (ez, -drho[1]), (bz, b1)):
                lst.append(csolve(L1D, rhs))
        wp = {1: -grad(psi[0], False) + 0j}
        if modes:
            gp, op = grad(psi[1], True), over(psi[1])
            wp[2] = -(gp - op)
            wp[0] = -np.conj(gp + op)
        # S+
        Wv, Ez, Bz = vec(wp, g), scal(ez, g), scal(bz, g)
        dD = qm * ((p * np.conj(Wv)).real / d - Ez)
        acc = qm * (gam * Wv - 1j * p * Bz) / d ** 2 - p * dD / d ** 2
        sv = []
        for m in vk:
            sv.append([wq * (acc * W[cc] + u * ul.real * dW[cc] - (m * 1j) * ul.imag * Wor[cc] * u) * np.conj(th) ** m for cc in range(2)])
        S = {m: filt(m, f) for m, f in zip(vk, add(j, sv))}
        # B+
        G = {1: grad(jz[0], False) + S[1]}
        if modes:
            gj, oj = grad(jz[1], True), over(jz[1])
            G[2] = (gj - oj) + S[2]
            G[0] = np.conj(gj + oj) + S[0]
        for _ in range(3 if modes else 1):
            rhs = {m: 1j * G[m] for m in vk}
            if modes:
                c1 = chi[1]
                rhs = {0: rhs[0] + np.conj(c1) * bp[1], 1: rhs[1] + c1 * bp[0] + np.conj(c1) * bp[2], 2: rhs[2] + c1 * bp[1]}
            bp[1] = solve(L1D, rhs[1].real, chi=chi[0]) + 1j * solve(L1F, rhs[1].imag, chi=chi[0], wall=jz[0][N])
            if modes:
                bp[0] = csolve(L0, rhs[0], chi=chi[0], regular=True)
                bp[2] = csolve(L2D, rhs[2], chi=chi[0])
        # store
        for m, (ce, cb) in {1: (0, 2), 0: (6, 10), 2: (8, 12)}.items():
            if m in vk:
                ep = wp[m] - 1j * bp[m]
                fld[k, :, ce], fld[k, :, ce + 1] = ep.real, ep.imag
                fld[k, :, cb], fld[k, :, cb + 1] = bp[m].real, bp[m].imag
        fld[k, :, 4], fld[k, :, 5] = ez[0], bz[0]
        diag[k, :, 0], diag[k, :, 1], diag[k, :, 2] = psi[0], ne[0], ni
        if modes:
            fld[k, :, 14], fld[k, :, 15], fld[k, :, 16], fld[k, :, 17] = ez[1].real, ez[1].imag, bz[1].real, bz[1].imag
            diag[k, :, 3], diag[k, :, 4], diag[k, :, 5], diag[k, :, 6] = psi[1].real, psi[1].imag, ne[1].real, ne[1].imag
        # push
        if k == K - 1:
            break
        Bv = vec(bp, g)
        f = np.zeros((3, len(w)), dtype=complex)
        f[0, idx] = u
        f[1, idx] = qm * (gam * Wv / d - 1j * Bv - 1j * p * Bz / d)
        f[2, idx] = dD
        hist = [f] + (hist[:len(AB) - 1] if hist else [f.copy() for _ in range(len(AB) - 1)])
        st = sum(c * f for c, f in zip(AB, hist))
        Xn, Pn, Dn = X + dxi * st[0], P + dxi * st[1], D + dxi * st[2].real
        with np.errstate(all="ignore"):
            gn = (1.0 + np.abs(Pn) ** 2 + Dn ** 2) / (2 * Dn)
            live = live & (Dn > 1e-3) & ~(gn > 35.0 * Dn)
            rn = np.abs(Xn)
            out = live & (rn > R)
            n = np.where(rn > 0, Xn / np.where(rn > 0, rn, 1.0), 1.0)
            live = live & ~(out & (2 * R - rn < 0))
            Xn = np.where(out, n * (2 * R - rn), Xn)
            Pn = np.where(out, Pn - 2 * (Pn * np.conj(n)).real * n, Pn)
            for f in hist:
                for c in range(2):
                    f[c] = np.where(out, f[c] - 2 * (f[c] * np.conj(n)).real * n, f[c])
        X, P, D = np.where(live, Xn, X), np.where(live, Pn, P), np.where(live, Dn, D)
    return fld, diag
