"""Sizes where the kernels' splits have their edges, against the CPU oracle on the same inputs:

- the solves by groups of warps (m = 0 up to 512 nodes: 3 x 5 and 2 x 8 warps; m = 1: 4 groups): node counts around
  whole numbers of rows per thread, and the block-wide solves of more than 512 nodes;
- every Adams-Bashforth order (the history is kept in shared memory up to order 3);
- the m = 1 sweep's particles over a cluster: particle counts around multiples of a CTA's threads;
- the beam kernels: counts around a warp and around the largest call whose lanes add their own values (m = 0: 16384,
  with the push 8192; m = 1: 4096 and 128), all particles in one cell, a field store off the 16-byte boundary.

- batches of every order.

Tolerances: fields and diagnostics after one sweep max(1e-10, 4 x the reference algorithm's own round-off floor, the
difference between its Thomas and partition solvers on the same input), per stored component; components that vanish in
the reference 1e-10 of the largest one; beam deposits 1e-12 and pushed particles 1e-13 as in test_gpu_parity.py, the
momenta plus the rounding of the kicks."""
import numpy as np
import pytest

import oracle as O
import quarz_b200 as Q
from helpers import rel_l2
from quarz_b200 import deck

pytestmark = pytest.mark.gpu

DECK = """
xi.convention = z-t
grid.type = uniform
grid.rmax = 6
grid.dr = 1
xi.min = -1.2
xi.max = 0
xi.step = 0.04
time.dt = 5
time.steps = 1
plasma.species = electrons
beams = driver
driver.n0 = 3
driver.sigma_r = 0.5
driver.sigma_xi = 0.3
driver.xi0 = -0.5
driver.gamma = 1000
driver.espread = 0.001
driver.emit_n = 0.05
driver.nparticles = 3000
"""


def _spec(nodes, extra=""):
    spec = deck.run_spec(deck.parse_deck(DECK + extra))
    spec.nodes = 6.0 * (np.arange(nodes) / (nodes - 1.0)) ** 1.2      # cells smaller at the axis
    return spec


def _check_sweep(spec):
    import torch

    beams = [Q.sample_beam(b) for b in spec.beams]
    a = O.OracleSim(spec, beams=beams, tridiag="thomas")
    a.step_fields(0.0)
    b = O.OracleSim(spec, beams=beams, tridiag="partition")
    b.step_fields(0.0)
    K, M = spec.K, spec.M
    nf, nd = (18, 9) if spec.modes else (6, 3)
    bsrc = torch.from_numpy(np.ascontiguousarray(a.bsrc())).cuda()
    fld = torch.zeros((K, M, nf), dtype=torch.float64, device="cuda")
    diag = torch.zeros((K, M, nd), dtype=torch.float64, device="cuda")
    Q.Sweep(Q.RadialGrid(spec.nodes), Q.sweep_params(spec)).run(bsrc, fld, diag)
    bad = {}
    for name, got, ra, rb in (("fld", fld.cpu().numpy(), a.fld(), b.fld()), ("diag", diag.cpu().numpy(), a.diag(), b.diag())):
        top = np.max(np.abs(ra))
        for c in range(got.shape[-1]):
            if not np.any(ra[..., c]) and not np.max(np.abs(got[..., c])) <= 1e-10 * top:
                bad[f"{name}{c}"] = (np.max(np.abs(got[..., c])), top)
            if np.any(ra[..., c]):
                e, floor = rel_l2(got[..., c], ra[..., c]), rel_l2(rb[..., c], ra[..., c])
                if not e < max(1e-10, 4.0 * floor):
                    bad[f"{name}{c}"] = (e, floor)
    assert not bad, bad


@pytest.mark.parametrize("nodes", [17, 160, 161, 256, 257, 480, 481, 511, 512, 513, 769, 1025])
def test_sweep_m0_nodes(nodes):
    _check_sweep(_spec(nodes, "electrons.ppc = 1\n"))


@pytest.mark.parametrize("order", [1, 2, 4, 5])
@pytest.mark.parametrize("ppc", [1, 3])
def test_sweep_m0_orders(order, ppc):
    _check_sweep(_spec(257, f"electrons.ppc = {ppc}\npusher.ab_order = {order}\n"))


@pytest.mark.parametrize("nodes,ntheta", [(17, 4), (128, 4), (129, 4), (130, 4), (257, 8), (512, 8), (513, 4), (641, 8)])
def test_sweep_m1_particles_over_a_cluster(nodes, ntheta):
    _check_sweep(_spec(nodes, f"modes = 1\nelectrons.ppc = 1\nelectrons.ntheta = {ntheta}\ndriver.x0 = 0.1\n"))


def _teams(steps):
    # 2056 particles per slice: as many CTAs per sweep (8, 4, 2) as let every sweep have them at once, else one
    spec = _spec(258, "modes = 1\nelectrons.ppc = 1\nelectrons.ntheta = 8\ndriver.x0 = 0.1\n")
    return spec, [Q.sample_beam(b) for b in spec.beams]


@pytest.mark.parametrize("steps,team", [(1, 8), (12, 4), (25, 2), (46, 1)])
def test_run_m1_teams(steps, team):
    spec, beams = _teams(steps)
    sim = Q.Simulation(spec, beams=beams)
    mom = sim.run(steps, spec.dt)
    assert sim.schedule()["sweep_ctas"] == (steps + 1) * team
    ref = O.OracleSim(spec, beams=beams).run(steps, spec.dt)
    assert rel_l2(mom, np.asarray(ref).reshape(mom.shape)) < 1e-12


def test_run_m1_team_gives_up_together():
    # a wait of the team's first CTA that runs out (its limit is 100 ns) ends every CTA of the cluster, and the run with
    # an error; the device is as usable as before
    spec, beams = _teams(1)
    sim = Q.Simulation(spec, beams=beams)
    sim.set_schedule(True, timeout_s=1e-7)
    with pytest.raises(Q.QZError, match="timed out"):
        sim.run(1, spec.dt)
    test_run_m1_teams(1, 8)


@pytest.mark.parametrize("order", [1, 2, 4, 5])
def test_batch_orders(order):
    # plasma in registers and in global memory, up to and beyond 512 nodes, both modes
    extra = f"pusher.ab_order = {order}\n"
    specs = [_spec(65, extra), _spec(257, "electrons.ppc = 3\n" + extra), _spec(600, extra),
             _spec(65, "modes = 1\nelectrons.ntheta = 4\ndriver.x0 = 0.1\n" + extra)]
    beams = [[Q.sample_beam(b) for b in s.beams] for s in specs]
    batch = Q.Batch()
    for s, bm in zip(specs, beams):
        batch.add(s, bm)
    for s, bm, mom in zip(specs, beams, batch.run(2, specs[0].dt)):
        ref = O.OracleSim(s, beams=bm).run(2, s.dt)
        assert rel_l2(mom, np.asarray(ref).reshape(mom.shape)) < 1e-12


@pytest.mark.parametrize("modes", [0, 1])
@pytest.mark.parametrize("n,one_cell", [(1, False), (31, False), (32, True), (33, True), (257, False), (4000, True),
                                        (128, False), (129, True), (160, False), (4096, False), (4097, True),
                                        (8192, False), (8193, True), (16384, False), (16417, True)])
def test_beam_push_deposit(n, one_cell, modes):
    import torch

    spec = _spec(65, "modes = 1\nelectrons.ntheta = 4\n" if modes else "")
    spec.beams[0].nparticles = n
    parts, gref, xiref = Q.sample_beam(spec.beams[0])
    if one_cell:
        parts[:, 5] = 0.5 + 0.01 * (parts[:, 5] - 0.5) / 0.9
        parts[:, :2] *= 0.004
    K, M = spec.K, spec.M
    nf, nb = (18, 15) if modes else (6, 5)
    o = O.OracleSim(spec, beams=[(parts, gref, xiref)])
    o.step_fields(0.0)
    F = np.ascontiguousarray(o.fld())
    o.push_beams(5.0, 5.0)
    o.deposit_beams()
    grid = Q.RadialGrid(spec.nodes)
    box = Q.BeamOps.box(spec.xi_min, spec.dxi, K, spec.ngp, modes)
    want, wantb = o.beam(0), o.bsrc()
    for shift in (0, 1):                               # the second field store starts 8 bytes off a 16-byte boundary
        store = torch.zeros(K * M * nf + 1, dtype=torch.float64, device="cuda")
        fld = store[shift:shift + K * M * nf]
        fld.copy_(torch.from_numpy(F.reshape(-1)))
        cols = torch.from_numpy(np.ascontiguousarray(parts.T)).cuda()
        bsrc = torch.zeros((K, M, nb), dtype=torch.float64, device="cuda")
        Q.BeamOps.push_deposit(grid, cols, -1.0, 1.0, box, fld, 5.0, 5.0, 0, bsrc)
        got = cols.cpu().numpy().T
        # momenta: the kicks of E and of v x B, each up to 5 max|F| (here up to 2000), nearly cancel; a gather rounds
        # each of them in about four operations
        kick = 4 * np.finfo(float).eps * 5.0 * np.max(np.abs(F))
        for c in range(7):
            tol = 1e-13 * max(np.max(np.abs(want[:, c])), 1.0) + (kick if 2 <= c <= 4 else 0.0)
            assert np.max(np.abs(got[:, c] - want[:, c])) <= tol, c
        B = bsrc.cpu().numpy()
        assert rel_l2(B, wantb) < 1e-12
        bsrc.zero_()                                   # and the deposit by itself, of the pushed particles
        Q.BeamOps.deposit(grid, cols, -1.0, 1.0, box, bsrc)
        assert rel_l2(bsrc.cpu().numpy(), wantb) < 1e-12
