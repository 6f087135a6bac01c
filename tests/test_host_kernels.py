"""Kernels run on the host (host_kernels.py): what must hold whatever the inputs and the order of the warps, and what a
GPU must not be given to find out."""
import contextlib
import ctypes as C

import numpy as np
import pytest

import host_kernels as H
import quarz_b200 as Q

if not H.available():
    pytest.skip("needs g++ on x86-64", allow_module_level=True)


def _grid(nodes):
    g = C.c_void_p()
    nodes = np.ascontiguousarray(nodes, dtype=np.float64)
    H.check(H.library().qz_grid_create(nodes.ctypes.data_as(C.POINTER(C.c_double)), len(nodes), C.byref(g)))
    return g


def _view(cols, q=-1.0, m=1.0):
    from quarz_b200 import _lib as L

    n = cols.shape[1]
    return L.BeamView(*[cols[c].ctypes.data for c in range(7)], n, q, m, 0)


@pytest.mark.parametrize("bad", [None, "momentum", "weight"])
@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("ngp", [0, 1])
def test_compact_deposit_stays_in_its_rows(ngp, exact, bad):
    # Particles in every xi cell, among them -1 (just ahead of the box: row 0 only) and K - 1 (behind it: row K - 1
    # only). A row outside the box belongs to another ring slot or to nobody: nothing is added there, not by a particle
    # whose momentum or weight is not finite either (0 x NaN is not 0).
    lib = H.library()
    K, dxi, xi_min = 6, 0.25, -1.5
    nodes = 3.0 * (np.arange(17) / 16.0) ** 1.2
    M = len(nodes)
    rng = np.random.default_rng(5)
    n = 200
    cols = np.empty((7, n))
    r, th = rng.uniform(0.0, 2.9, n), rng.uniform(0.0, 2 * np.pi, n)
    cols[0], cols[1] = r * np.cos(th), r * np.sin(th)
    cols[2:4] = rng.normal(size=(2, n))
    cols[4] = rng.uniform(50.0, 100.0, n)
    cell = rng.integers(-1, K, n)
    cell[:40], cell[40:80] = -1, K - 1
    cols[5] = xi_min + dxi * (cell + rng.uniform(0.1, 0.9, n))
    cols[6] = rng.uniform(0.5, 1.0, n)
    finite = cols.copy()
    if bad:
        cols[4 if bad == "momentum" else 6, ::7] = np.nan
    g = _grid(nodes)
    V = np.empty(M)
    H.check(lib.qz_grid_volumes(g, V.ctypes.data_as(C.POINTER(C.c_double))))
    inv_h, inv_V = np.append(1.0 / np.diff(nodes), 0.0), 1.0 / V
    # exact: quanta of 2^-40, limbs of 20 bits
    nc, scale = (6, np.full(M, 2.0 ** 40)) if exact else (3, None)
    store = np.zeros((K + 4, M, nc))                  # two guard rows on either side
    rc = lib.emu_deposit_compact(M, H.ptr(nodes), H.ptr(inv_h), H.ptr(inv_V), C.c_double(xi_min), C.c_double(dxi), K,
                                 ngp, H.ptr(cols), C.c_long(n), C.c_double(-1.0), H.ptr(scale) if exact else None, 20,
                                 H.ptr(store[2:]))
    assert rc == 0
    assert not np.any(store[:2]) and not np.any(store[K + 2:])
    if bad:
        return
    want = np.zeros((K, M, 5))
    box = Q.BeamOps.box(xi_min, dxi, K, ngp, 0)
    v = _view(finite)
    H.check(lib.qz_beam_deposit(g, C.byref(v), C.byref(box), H.ptr(want), None))
    got = store[2:K + 2]
    if exact:
        got = (got[..., :3] * 2.0 ** 20 + got[..., 3:]) * 2.0 ** -40
    # FP64: the same sums in another order; exact: half a quantum per particle and value
    tol = n * 2.0 ** -41 if exact else 1e-13 * np.max(np.abs(want))
    assert np.max(np.abs(got - want[..., [0, 1, 3]])) <= tol


DECK = """
xi.convention = z-t
grid.type = uniform
grid.rmax = 6
grid.dr = 1
xi.min = -0.36
xi.max = 0
xi.step = 0.04
time.dt = 5
time.steps = 1
plasma.species = electrons
electrons.ppc = 1
beams = driver
driver.n0 = 3
driver.sigma_r = 0.5
driver.sigma_xi = 0.1
driver.xi0 = -0.2
driver.gamma = 1000
driver.espread = 0.001
driver.emit_n = 0.05
driver.nparticles = 3000
"""


def _spec(nodes, extra=""):
    from quarz_b200 import deck

    spec = deck.run_spec(deck.parse_deck(DECK + extra))
    spec.nodes = 6.0 * (np.arange(nodes) / (nodes - 1.0)) ** 1.2
    return spec


@contextlib.contextmanager
def _sweep(spec, change=lambda p: None):
    lib, s, g = H.library(), C.c_void_p(), _grid(spec.nodes)
    p = Q.sweep_params(spec)
    change(p)
    try:
        H.check(lib.qz_sweep_create(g, C.byref(p), C.byref(s)))
        yield s
    finally:                                          # (freeing looks at the words around every allocation)
        if s:
            lib.qz_sweep_destroy(s)
        lib.qz_grid_destroy(g)


def _fields(spec):
    nf, nd = (18, 9) if spec.modes else (6, 3)
    return np.zeros((spec.K, spec.M, nf)), np.zeros((spec.K, spec.M, nd))


# the warps that run ahead of the others (each as far as it can): none, all in turn, the last or one half, the first
ORDERS = [((), False), (range(16), True), (range(15, -1, -1), True), (range(8, 16), True), (range(4), True)]


@pytest.mark.parametrize("nodes,extra", [
    (3, ""), (33, "beams.xi_shape = ngp\n"), (33, "electrons.ppc = 20\n"), (513, ""), (550, "electrons.ppc = 2\n"),
    (300, "electrons.ppc = 3\npusher.ab_order = 5\n"),
    (140, "plasma.smooth_length = 0.05\n"), (550, "plasma.smooth_length = 0.05\n"),
    (65, "pusher.max_cells_per_step = 0.3\n"), (65, "pusher.max_cells_per_step = 0.3\nelectrons.ppc = 12\n"),
    (9, "modes = 1\nelectrons.ntheta = 4\n"),
    (130, "modes = 1\nelectrons.ntheta = 4\ndriver.x0 = 0.1\nbeams.xi_shape = ngp\n"),
    (140, "modes = 1\nelectrons.ntheta = 4\ndriver.x0 = 0.1\n"),
    (140, "modes = 1\nelectrons.ntheta = 4\ndriver.x0 = 0.1\nplasma.smooth_length = 0.05\n"),
])
def test_sweep_in_every_order_of_the_warps(nodes, extra):
    # a barrier too few shows when a warp lags behind; tolerance as on the GPU: max(1e-10, 4 x the reference algorithm's
    # round-off floor, the difference between its Thomas and partition solvers)
    import oracle as O
    from helpers import rel_l2

    spec = _spec(nodes, extra)
    beams = [Q.sample_beam(b) for b in spec.beams]
    a, b = (O.OracleSim(spec, beams=beams, tridiag=t) for t in ("thomas", "partition"))
    a.step_fields(0.0)
    b.step_fields(0.0)
    bsrc = np.ascontiguousarray(a.bsrc())
    for first, keep in ORDERS:
        H.schedule(first, keep)
        fld, diag = _fields(spec)
        with _sweep(spec) as s:
            H.check(H.library().qz_sweep_run(s, H.ptr(bsrc), H.ptr(fld), H.ptr(diag), None, None))
        for got, ra, rb in ((fld, a.fld(), b.fld()), (diag, a.diag(), b.diag())):
            for c in range(got.shape[-1]):
                if np.any(ra[..., c]):
                    assert rel_l2(got[..., c], ra[..., c]) < max(1e-10, 4.0 * rel_l2(rb[..., c], ra[..., c])), (list(first), c)


@pytest.mark.parametrize("extra,most", [("", 1439), ("plasma.smooth_length = 0.05\n", 1180)])
def test_largest_grid(extra, most):
    # the widest grid that a CTA's shared memory holds: 160 bytes per node (192 with the filter) beside 2128 (5712) in
    # 232448; one node more is refused
    with pytest.raises(RuntimeError, match=f"M = {most + 1} is too large"), _sweep(_spec(most + 1, extra)):
        pass
    test_sweep_in_every_order_of_the_warps(most, extra)


def test_gamma_beyond_the_range():
    # momenta whose squares overflow: 1 / gamma = 0 and v = 0 in the beam's deposit (m = 0 and 1), as a division gives
    import oracle as O

    for extra in ("", "modes = 1\nelectrons.ntheta = 4\n"):
        spec = _spec(17, extra)
        parts = np.array([[0.3, 0.1, 0.2, 0.1, 1e200, 0.1, 1.0]])
        o = O.OracleSim(spec, beams=[(parts, 1.0, 0.0)])
        o.deposit_beams()
        want = o.bsrc()
        got = np.zeros_like(want)
        v, box = _view(np.ascontiguousarray(parts.T)), Q.BeamOps.box(spec.xi_min, spec.dxi, spec.K, spec.ngp, spec.modes)
        H.check(H.library().qz_beam_deposit(_grid(spec.nodes), C.byref(v), C.byref(box), H.ptr(got), None))
        assert np.any(want) and np.max(np.abs(got - want)) <= 1e-13 * np.max(np.abs(want))


@pytest.mark.parametrize("ppc", [1, 20])
@pytest.mark.parametrize("n0", ["3e155", "1e200"])
def test_plasma_beyond_the_range(n0, ppc):
    # a driver so strong that the plasma's gamma overflows in its first push: every particle is removed as trapped and
    # the fields stay the driver's own
    import oracle as O
    from quarz_b200 import _lib as L

    spec = _spec(33, f"driver.n0 = {n0}\nelectrons.ppc = {ppc}\n")
    spec.beams[0].q = 1.0
    a = O.OracleSim(spec, beams=[Q.sample_beam(b) for b in spec.beams])
    a.step_fields(0.0)
    bsrc, want, (fld, diag), cnt = np.ascontiguousarray(a.bsrc()), a.fld(), _fields(spec), L.Counters()
    H.schedule()
    with _sweep(spec) as s:
        H.check(H.library().qz_sweep_run(s, H.ptr(bsrc), H.ptr(fld), H.ptr(diag), C.byref(cnt), None))
    assert (cnt.lost, cnt.trapped, cnt.nonfinite) == (a.lost(), a.lost(), 0) and cnt.lost > 0
    top = np.max(np.abs(want))
    assert np.max(np.abs(fld / top - want / top)) < 1e-12


@pytest.mark.parametrize("ppc", [1, 20])
@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_removed_particles_keep_their_state(order, ppc):
    # a slab hands its plasma on with every particle's history; a removed particle's is that of the push that removed it,
    # however many slices follow (history in shared memory, in registers and in global memory)
    from quarz_b200 import _lib as L

    lib = H.library()
    spec = _spec(33, f"beams.xi_shape = ngp\ndriver.n0 = 60\nelectrons.ppc = {ppc}\npusher.ab_order = {order}\n")
    bsrc = np.zeros((spec.K, spec.M, 5))
    parts, _, _ = Q.sample_beam(spec.beams[0])
    v, box = _view(np.ascontiguousarray(parts.T)), Q.BeamOps.box(spec.xi_min, spec.dxi, spec.K, spec.ngp, 0)
    H.check(lib.qz_beam_deposit(_grid(spec.nodes), C.byref(v), C.byref(box), H.ptr(bsrc), None))
    H.schedule()
    states = {}
    for K in range(3, spec.K + 1):
        def change(p):
            p.K, p.max_qsa = K, 1.0 + 1e-3

        n, npad, ord_ = C.c_int(), C.c_int(), C.c_int()
        with _sweep(spec, change) as s:
            H.check(lib.qz_sweep_state_shape(s, C.byref(n), C.byref(npad), C.byref(ord_)))
            out = np.zeros((6 + 5 * order, npad.value))
            fld, diag = np.zeros((K, spec.M, 6)), np.zeros((K, spec.M, 3))
            st = L.PlasmaState(out.ctypes.data, n.value, npad.value, order, 0)
            H.check(lib.qz_sweep_run_stage(s, H.ptr(bsrc), None, None, H.ptr(fld), H.ptr(diag), C.byref(st), None, None))
        states[K] = out[:, :n.value]
    seen = 0
    for K in range(3, spec.K):
        gone = states[K][5] == 0.0
        seen += bool(np.any(gone)) and not np.all(gone)
        assert np.array_equal(states[K + 1][:, gone], states[K][:, gone]), K
    assert seen >= 3


def test_grid_set_up_is_one_copy():
    # a scan makes a grid per instance: its arrays reach the device in one allocation and one blocking copy
    lib, n = H.library(), [C.c_long() for _ in range(4)]
    lib.emu_counts(C.byref(n[0]), C.byref(n[1]))
    _grid(_spec(257).nodes)
    lib.emu_counts(C.byref(n[2]), C.byref(n[3]))
    assert (n[2].value - n[0].value, n[3].value - n[1].value) == (1, 1)


@pytest.mark.parametrize("with_filter", [False, True])
@pytest.mark.parametrize("nodes,ppc,order", [(65, 1, 3), (512, 1, 1), (512, 1, 4), (513, 1, 3), (257, 4, 3), (600, 1, 3)])
def test_batch_layouts_are_the_kernels(nodes, ppc, order, with_filter):
    # qz_batch_tuning gives the layout the kernel uses, and the autotuner's candidates are different kernels: each reads
    # back as it was set, and every layout as one of them
    from quarz_b200 import tune

    lib, b, n = H.library(), C.c_void_p(), C.c_int()
    H.check(lib.qz_batch_create(C.byref(b)))

    def add(spec):
        p = Q.sweep_params(spec)
        a = np.ascontiguousarray(spec.nodes)
        H.check(lib.qz_batch_add(b, a.ctypes.data_as(C.POINTER(C.c_double)), len(a), C.byref(p), 0, None, None, None,
                                 None, None, None, None, C.byref(n)))
        return n.value

    def read(i):
        lay, cost = C.c_int(), C.c_double()
        H.check(lib.qz_batch_tuning(b, i, C.byref(lay), C.byref(cost)))
        return lay.value

    extra = f"pusher.ab_order = {order}\n"
    spec = _spec(nodes, f"electrons.ppc = {ppc}\n" + extra)
    i = add(spec)
    if with_filter:
        add(_spec(33, "plasma.smooth_length = 0.05\n" + extra))
    cands = tune.candidate_layouts(spec, with_filter)
    assert read(i) in cands
    glob = tune.plasma_per_slice(spec) > tune.REG_PARTICLES
    for lay in range(8):
        rc = lib.qz_batch_set_tuning(b, i, lay, 0.0)
        if lay & 4 and not glob:
            assert rc != 0
        elif rc == 0:
            assert read(i) == tune.used_layout(spec, lay, with_filter) and read(i) in cands
        else:
            assert glob or nodes > 512               # does not fit
    H.check(lib.qz_batch_destroy(b))


def _sim(spec, beams):
    lib, sim = H.library(), C.c_void_p()
    p = Q.sweep_params(spec)
    H.check(lib.qz_sim_create(_grid(spec.nodes), C.byref(p), C.byref(sim)))
    for b, (parts, gref, xiref) in zip(spec.beams, beams):
        a = np.ascontiguousarray(parts)
        H.check(lib.qz_sim_add_beam(sim, a.ctypes.data_as(C.POINTER(C.c_double)), len(a), b.q, b.m, 0, gref, xiref))
    H.check(lib.qz_sim_set_schedule(sim, 0, 0, 0, 0, 0.0))
    return sim


@pytest.mark.parametrize("nodes,extra", [(33, ""), (200, "pusher.ab_order = 2\n"), (65, "plasma.smooth_length = 0.05\n"),
                                         (65, "beams.xi_shape = ngp\n"), (512, "pusher.ab_order = 5\n")])
def test_adjoint_in_every_order_of_the_warps(nodes, extra):
    # the reverse sweep like the forward, against the oracle's adjoint: 1e-8 per component as on the GPU
    import oracle as O

    lib, dp = H.library(), C.POINTER(C.c_double)
    spec = _spec(nodes, "driver.nparticles = 300\n" + extra)
    beams, T, dt = [Q.sample_beam(b) for b in spec.beams], 2, 5.0
    mom0 = O.OracleSim(spec, beams=beams).run(T, dt)
    seeds = np.random.default_rng(5).normal(size=(1, 17)) / (np.abs(mom0[-1]) + 1e-30)
    seeds[:, 16] = 0.0
    ref, _ = O.OracleSim(spec, beams=beams).adjoint(T, dt, seeds)
    for first, keep in ORDERS:
        H.schedule(first, keep)
        sim = _sim(spec, beams)
        lam, mom, ms = np.zeros((7, len(beams[0][0]))), np.zeros((T + 1, 1, 17)), np.zeros(2)
        out = (C.c_void_p * 1)(lam.ctypes.data)
        H.check(lib.qz_sim_adjoint(sim, T, dt, seeds.ctypes.data_as(dp), out, mom.ctypes.data_as(dp),
                                   ms.ctypes.data_as(dp), None))
        H.check(lib.qz_sim_destroy(sim))
        for c in range(7):
            want = ref[0][:, c]
            assert np.linalg.norm(lam[c] - want) <= 1e-8 * np.linalg.norm(want), (list(first), c)
