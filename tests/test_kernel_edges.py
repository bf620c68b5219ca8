"""Kernels at the sizes where their split can go wrong: one particle, one
tile more or less, both sides of each rule that picks a variant, lists longer
than one pass of a cluster.  The references are the FP64 CPU oracle, numpy
restatements of the fixed-point rules (csrc/pgb_physics.cuh), or another
route to the same state through the public entry points.

Tolerances: none, unless a test states one.  Charge sums, record positions
and FP64 multigrid sweeps are exact by design, and two routes to one state
run the same arithmetic per particle.
"""
import ctypes as C

import numpy as np
import pytest

from conftest import load_golden
import orc
import picgb

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(lib):
    return lib


def pos_shift(n):
    return max(8, min(23, 29 - int(np.ceil(np.log2(n - 1)))))


def fixed(x, d, ps):
    """A record's position in units of 2^-ps of a cell (pos_from_m); NaN is INT_MIN + 1."""
    with np.errstate(invalid="ignore", over="ignore"):
        v = np.clip(np.rint(np.ldexp(x / d, ps)), -2.0**30, 2.0**30)
    return np.where(np.isnan(v), -2.0**31 + 1, v).astype(np.int64)


def plasma(p, n, seed, temp_e=2.0, temp_i=0.5, lo=0.02, hi=0.98):
    rng = np.random.default_rng(seed)
    out = []
    for m, t in ((picgb.ELECTRON_MASS, temp_e), (p.ion_mass, temp_i)):
        a = np.empty((n, 6))
        a[:, :2] = rng.uniform(lo * p.xlength, hi * p.xlength, (n, 2))
        a[:, 2:5] = rng.normal(0.0, np.sqrt(t * picgb.CHARGE / m), (n, 3))
        a[:, 5] = 1.0
        out.append(a)
    return out


def loaded(p, state):
    r = picgb.Run(p)
    for s in (0, 1):
        r.load_particles(s, state[s])
    return r


def end_state(r):
    return r.get_particles(0), r.get_particles(1), r.get_grid("q_e"), r.get_grid("q_i"), r.get_grid("phi")


def assert_same(a, b, what):
    for k, (x, y) in enumerate(zip(a, b)):
        assert np.array_equal(x, y, equal_nan=True), (what, k)


# ------------------------------------------------------------------ deposit
def deposit_reference(a, n, d, qc):
    ps = pos_shift(n)
    x, y = fixed(a[:, 0], d, ps), fixed(a[:, 1], d, ps)
    ok = (x > 0) & (y > 0) & (x >> ps < n - 1) & (y >> ps < n - 1)
    x, y, w = x[ok], y[ok], a[ok, 5].astype(np.float32)
    one = np.float32(1.0)
    f = [((v & ((1 << ps) - 1)) * 2.0**-ps).astype(np.float32) for v in (x, y)]
    node = (y >> ps) * n + (x >> ps)
    acc = np.zeros(n * n, dtype=np.int64)
    for share, k in (((one - f[0]) * (one - f[1]), 0), (f[0] * (one - f[1]), 1), (f[1] * (one - f[0]), n),
                     (f[0] * f[1], n + 1)):
        np.add.at(acc, node + k, np.rint(share * w * np.float32(2.0**19)).astype(np.int64))
    edge = np.ones((n, n))
    edge[[0, -1], :] *= 2.0
    edge[:, [0, -1]] *= 2.0
    edge[np.ix_([0, -1], [0, -1])] *= 2.0
    return acc * 2.0**-19 * (qc / (d * d)) * edge.ravel()


@pytest.mark.parametrize("nodes,n,order", [
    (17, 1, "random"), (17, 8191, "random"), (17, 8192, "random"), (33, 17423, "random"), (33, 17424, "random"),
    (65, 2048 * 33 + 1, "binned"), (129, 266255, "random"), (129, 266256, "random"), (257, 1056784, "binned"),
    (257, 1056785, "random"), (513, 200003, "binned"), (513, 200003, "random"),
    (17, 2000003, "one node")])
def test_deposit_windows_add_the_exact_integers(lib, nodes, n, order):
    """pgb_deposit_static and pgb_deposit on both sides of the rule that picks
    the windows, with weights that a window's word may not take (>= 1.99 and
    negative ones), positions on and beyond the walls, and sums that wrap a
    32-bit word at one node."""
    torch = pytest.importorskip("torch")
    p = picgb.make_params(X_NO_OF_CELLS=nodes, STEADYSTATE="NO")
    d = p.xlength / (nodes - 1)
    rng = np.random.default_rng(nodes + n)
    a = np.zeros((n, 6))
    a[:, :2] = rng.uniform(-0.02, 1.02, (n, 2)) * p.xlength
    a[:, 5] = rng.choice([1.0, 1.0, 1.0, 0.37, 1.98, 1.99, 2.5, 0.0, -0.0, -0.5], n)
    if order == "binned":
        a = a[np.lexsort((np.floor(a[:, 0] / (8 * d)), np.floor(a[:, 1] / (8 * d))))]
    if order == "one node":
        a[:, :2] = (nodes // 2 + rng.uniform(0.0, 0.01, (n, 2))) * d
        a[:, 5] = 1.98
    want = deposit_reference(a, nodes, d, p.qce)
    with picgb.Run(p) as r:
        r.load_particles(0, a)
        r.deposit(0)
        run = r.get_grid("q_e").ravel()
    recs = torch.from_numpy(a).cuda()
    q = torch.full((nodes * nodes,), float("nan"), dtype=torch.float64, device="cuda")
    st = torch.cuda.current_stream()
    assert lib.pgb_deposit_static(C.c_void_p(recs.data_ptr()), n, nodes, nodes, d, d, p.qce, C.c_void_p(q.data_ptr()),
                                  C.c_void_p(st.cuda_stream)) == 0
    st.synchronize()
    assert np.array_equal(run, want)
    assert np.array_equal(q.cpu().numpy(), want)


# ------------------------------------------------------------------ records
@pytest.mark.parametrize("nodes,n", [(5, 1), (33, 255), (65, 4097), (513, 100003)])
def test_records_round_as_the_division_does(nodes, n):
    """Load and dump: x/DX 2^ps rounded to nearest even and clipped, also at
    halves, their neighbours, zero, infinity and NaN; the dump is that number
    times DX 2^-ps, and weights are the nearest float."""
    p = picgb.make_params(X_NO_OF_CELLS=nodes, STEADYSTATE="NO")
    ps, d = pos_shift(nodes), p.xlength / (nodes - 1)
    rng = np.random.default_rng(n)
    a = np.zeros((n, 6))
    a[:, 0] = rng.uniform(-0.5, 1.5, n) * p.xlength
    half = (rng.integers(-(1 << 22), 1 << 28, n) + 0.5) * (d * 2.0**-ps)
    a[:, 1] = half
    a[1::3, 1] = np.nextafter(half[1::3], np.inf)
    a[2::3, 1] = np.nextafter(half[2::3], -np.inf)
    a[:, 5] = rng.choice([1.0, 0.5, 1.0 / 3.0, 1e-42, 3e38, 0.0, -0.0, -1.7, 1.0 + 2.0**-25], n)
    odd = np.array([0.0, -0.0, np.nan, np.inf, -np.inf, 1e300, -1e300, 5e-324, 1e-310, d * 2.0**(30 - ps), -d * 2.0**(30 - ps),
                    d * 2.0**-ps / 2, d * 2.0**-ps * 1.5, -d * 2.0**-ps / 2])
    k = min(n, odd.size)
    a[:k, 0] = odd[:k]
    with picgb.Run(p) as r:
        r.load_particles(0, a)
        got = r.get_particles(0)
    assert got.shape == a.shape
    for c in (0, 1):
        v = fixed(a[:, c], d, ps)
        want = np.where(v == -2**31 + 1, np.nan, v * (d * 2.0**-ps))
        assert np.array_equal(got[:, c], want, equal_nan=True), c
    assert np.array_equal(got[:, 5], a[:, 5].astype(np.float32).astype(np.float64))


# ------------------------------------------------------------------- fields
@pytest.mark.parametrize("n", [5, 9, 17, 33, 65, 129, 1025])
def test_multigrid_of_every_depth_equals_oracle(n):
    """The reference's FP64 schedule with the levels in one CTA (to 9), on a
    cluster (to 65) and in tiles (above)."""
    p = picgb.make_params(X_NO_OF_CELLS=n, PHI_RIGHT=1.5, PHI_LEFT=-0.5, PHI_TOP=0.25, PHI_BOTTOM=0.1, PHI_PERIOD=0.02)
    rho = 1e-6 * np.random.default_rng(n).standard_normal((n, n))
    o = orc.Oracle(p)
    with picgb.Run(p) as r:
        for t in (3, 4):
            for x in (o, r):
                x.set_rho(rho * t)
                x.poisson(t)
                x.efield()
            for grid in ("phi", "ex", "ey"):
                assert np.array_equal(r.get_grid(grid), o.get_grid(grid)), (t, grid)


@pytest.mark.parametrize("mode,n,bound", [(m, n, b) for m, b in (("FP32_DC", 1e-9), ("DST_DC", 1e-9))
                                          for n in (5, 9, 17, 33, 129)] + [("FP32_DC", 513, 1e-9)])
def test_converged_modes_at_every_depth(mode, n, bound):
    """The FP32 multigrid's levels and the fused corrections, walls at
    different potentials.  Bound: a V-cycle divides the error by at least
    three, so 27 corrections leave 1.3e-13 of it and a transform pass by 1e4,
    so three leave 1e-12; E, a difference over a cell, may show n / 2 times
    that."""
    passes = 28 if mode == "FP32_DC" else 3
    p = picgb.make_params(X_NO_OF_CELLS=n, POISSON=mode, DC_MAX_ITERS=passes, DC_TOLERANCE=0.0, PHI_RIGHT=1.5,
                          PHI_LEFT=-0.5, PHI_TOP=0.25)
    rho = 1e-6 * np.random.default_rng(n + 2).standard_normal((n, n))
    o = orc.Oracle(p)
    o.set_rho(rho)
    o.poisson_converged(0, 30)
    o.efield()
    with picgb.Run(p) as r:
        r.set_rho(rho)
        r.poisson(0)
        r.efield()
        for grid in ("phi", "ex", "ey"):
            a, b = r.get_grid(grid), o.get_grid(grid)
            assert np.max(np.abs(a - b)) <= bound * np.max(np.abs(b)), grid


@pytest.mark.parametrize("n", [513, 1025])
def test_two_converged_solvers_agree_on_large_grids(n):
    """The sine transforms against the multigrid's tiles (1025 nodes are the
    most that a run takes): both are the discrete solution, up to FP64
    rounding of the residual, 2e-16 n^2 / pi^2 of phi = 2e-11 at 1025; bound
    1e-9."""
    rho = 1e-6 * np.random.default_rng(n).standard_normal((n, n))
    phi = []
    for mode, passes in (("DST_DC", 3), ("FP32_DC", 28)):
        p = picgb.make_params(X_NO_OF_CELLS=n, POISSON=mode, DC_MAX_ITERS=passes, DC_TOLERANCE=0.0, PHI_RIGHT=1.5)
        with picgb.Run(p) as r:
            r.set_rho(rho)
            r.poisson(0)
            phi.append(r.get_grid("phi"))
    assert np.max(np.abs(phi[0] - phi[1])) <= 1e-9 * np.max(np.abs(phi[1]))


# -------------------------------------------------------------------- steps
@pytest.mark.parametrize("inject,ratio,n", [(0, 1.0, 1), (1, 2.0, 257), (40, 1.0, 5000), (256, 2.0, 3000), (257, 1.0, 3000), (4500, 2.0, 3000)])
def test_absorbing_push_equals_the_calls(inject, ratio, n):
    """pgb_step removes particles at absorbing walls in the push; the same
    step call by call builds lists for the walls.  Injection on both sides of
    its one-block size."""
    p = picgb.make_params(X_NO_OF_CELLS=33, STEADYSTATE="NO", NUMBER_TO_INJECT=inject, DTI_RATIO=ratio, RAND_SEED=7)
    state = plasma(p, n, 11, temp_e=20.0, temp_i=2000.0, lo=0.0, hi=1.0)
    with loaded(p, state) as a, loaded(p, state) as b:
        a.initial_boundary()
        b.initial_boundary()
        for t in range(5):
            a.step(1)
            b.set_time_step(t)
            b.inject()
            b.gather_push(0)
            if t % int(ratio) == 0:
                b.gather_push(1)
                b.boundary(picgb.PGB_BOUNDARY_IONS)
            b.boundary(picgb.PGB_BOUNDARY_ELECTRONS)
            b.deposit(1)
            b.deposit(0)
            b.grid_rho()
            b.poisson(t)
            b.efield()
            assert_same(end_state(a), end_state(b), t)
        ca, cb = a.counters(), b.counters()
        assert {k: ca[k] for k in ca if k != "step"} == {k: cb[k] for k in cb if k != "step"}
        assert n < 3000 or ca["absorbed_e"] > 0


@pytest.mark.parametrize("nodes,n,steady,magnetic", [
    (5, 400, "NO", 0.0), (17, 16 * 289 - 1, "NO", 0.0), (17, 16 * 289, "YES", 0.02), (17, 1500001, "NO", 0.0),
    (65, 16 * 4225, "NO", 0.02), (129, 16 * 16641, "YES", 0.0), (129, 400003, "NO", 0.0), (257, 1100003, "NO", 0.0)])
def test_unsorted_push_through_the_whole_grid_equals_the_calls(nodes, n, steady, magnetic):
    """A run without sort deposits through windows of the whole grid up to 65
    nodes a side and from 16 particles a node, else two lanes to a particle;
    gather_push and deposit, call by call, take other kernels.  Weights of every kind, sums that wrap 32 bits on the smallest
    grids, injection on the way."""
    p = picgb.make_params(X_NO_OF_CELLS=nodes, STEADYSTATE=steady, MAGNETIC_FIELD=magnetic, RAND_SEED=2, POISSON="DST_DC",
                          DC_MAX_ITERS=2, NUMBER_TO_INJECT=0 if steady == "YES" else 17)
    state = plasma(p, n, nodes + n, lo=0.0, hi=1.0)
    for a in state:
        a[:, 5] = np.random.default_rng(n).choice([1.0, 1.0, 1.98, 0.25, 2.5, 0.0, -0.5], n)
    with loaded(p, state) as a, loaded(p, state) as b:
        a.initial_boundary()
        b.initial_boundary()
        for t in range(3):
            a.step(1)
            b.set_time_step(t)
            b.inject()
            b.gather_push(0)
            b.gather_push(1)
            b.boundary(picgb.PGB_BOUNDARY_IONS)
            b.boundary(picgb.PGB_BOUNDARY_ELECTRONS)
            if steady == "NO":
                b.contain_growth(0)
                b.contain_growth(1)
            b.deposit(1)
            b.deposit(0)
            b.grid_rho()
            b.poisson(t)
            b.efield()
            assert_same(end_state(a), end_state(b), t)


@pytest.mark.parametrize("nodes,n", [(33, 6001), (129, 300007)])
def test_push_items_do_not_depend_on_the_launch(nodes, n):
    """More items than blocks, and blocks without an item: any grid of the
    push gives the same particles and charge."""
    p = picgb.make_params(X_NO_OF_CELLS=nodes, STEADYSTATE="NO", SORT_INTERVAL=2, POISSON="DST_DC", DC_MAX_ITERS=2)
    state = plasma(p, n, 3)
    ends = []
    for shape in (None, (1, 140), (2, 0), (16, 32)):
        with loaded(p, state) as r:
            if shape:
                r.set_launch_config(*shape)
            r.initial_boundary()
            r.step(5)
            ends.append(end_state(r))
    for k, e in enumerate(ends[1:]):
        assert_same(ends[0], e, k)


def test_sorts_of_different_grids_in_turn():
    """The sort's tables and shared memory belong to a run: a run of 513^2
    nodes and one of 17^2 that sort in turn end as each alone."""
    ps = [picgb.make_params(X_NO_OF_CELLS=n, STEADYSTATE="NO", SORT_INTERVAL=1, POISSON="FMG32") for n in (513, 17)]
    states = [plasma(p, n, 5) for p, n in zip(ps, (4096 * 3 + 1, 4095))]
    alone = []
    for p, s in zip(ps, states):
        with loaded(p, s) as r:
            r.initial_boundary()
            r.step(6)
            alone.append(end_state(r))
    runs = [loaded(p, s) for p, s in zip(ps, states)]
    for r in runs:
        r.initial_boundary()
    for _ in range(3):
        for r in runs:
            r.step(1)
    picgb.step_batch(runs, 3)
    for r, want in zip(runs, alone):
        assert_same(end_state(r), want, "in turn")
        r.close()


@pytest.mark.parametrize("inject", [256, 257, 4096, 6000])
def test_injected_electrons_join_the_wall_list_in_order(inject):
    """Walls that emit take the new electrons that left from the list's end, in
    slot order, and give the secondaries slots and ids by that order: one
    step against the same step call by call, on both sides of the injection's
    one-block size.  A time step of several cells puts many outside."""
    p = picgb.make_params(X_NO_OF_CELLS=17, STEADYSTATE="NO", NUMBER_TO_INJECT=inject, DT_SCALE=40.0, TEMPERATURE=30.0,
                          E_IMPACT_SEE="YES", REFLECTION="YES", BACKSCATTER="YES", RAND_SEED=9)
    state = plasma(p, 2000, 4, temp_e=200.0)
    with loaded(p, state) as a, loaded(p, state) as b:
        a.initial_boundary()
        b.initial_boundary()
        for t in range(2):
            a.step(1)
            b.set_time_step(t)
            b.inject()
            b.gather_push(0)
            b.gather_push(1)
            b.boundary(picgb.PGB_BOUNDARY_IONS)
            b.boundary(picgb.PGB_BOUNDARY_ELECTRONS)
            b.deposit(1)
            b.deposit(0)
            b.grid_rho()
            b.poisson(t)
            b.efield()
            assert_same(end_state(a), end_state(b), t)
        ca, cb = a.counters(), b.counters()
        assert {k: ca[k] for k in ca if k != "step"} == {k: cb[k] for k in cb if k != "step"}
        assert ca["absorbed_e"] > 50


# -------------------------------------------------------------------- walls
@pytest.mark.parametrize("ne,ni", [(1, 1), (3, 0), (8191, 8193), (20011, 9000), (500, 30000)])
def test_steady_walls_with_long_lists(ne, ni):
    """Pairs across both axes from lists longer than one pass of the cluster.
    Positions are quarters of a cell, so the classes are exact and the
    particle counts equal the oracle's; new positions agree to FP32 rounding
    (2e-4 cell), new velocities to 1e-4 vt."""
    p = picgb.make_params(X_NO_OF_CELLS=65, STEADYSTATE="YES", RAND_SEED=3)
    d = p.xlength / 64
    rng = np.random.default_rng(ne + ni)
    state = []
    for n in (ne, ni):
        a = np.zeros((n, 6))
        a[:, :2] = (rng.integers(-8, 4 * 64 + 9, (n, 2)) * 0.25 + 0.125) * d
        side = rng.integers(0, 2, n)
        a[np.arange(n), rng.integers(0, 2, n)] = np.where(side == 1, 65.375, -1.625) * d
        a[:, 5] = 1.0
        state.append(a)
    o = orc.Oracle(p, rng=orc.ORC_RNG_PHILOX, order=orc.ORC_ORDER_STABLE)
    with loaded(p, state) as r:
        for s in (0, 1):
            o.load_particles(s, state[s])
        for x in (o, r):
            x.boundary(picgb.PGB_BOUNDARY_IONS)
            x.boundary(picgb.PGB_BOUNDARY_ELECTRONS)
        co, cr = o.counters(), r.counters()
        for k in ("n_e", "n_i", "plopped"):
            assert cr[k] == co[k], (k, cr[k], co[k])
        assert co["plopped"] > 0 or ni == 0
        for s, vt in ((0, p.vte), (1, p.vti)):
            a, b = r.get_particles(s), o.get_particles(s)
            assert a.shape == b.shape
            if a.size:
                assert np.max(np.abs(a[:, :2] - b[:, :2])) <= 2e-4 * d
                assert np.max(np.abs(a[:, 2:5] - b[:, 2:5])) <= 1e-4 * vt


@pytest.mark.parametrize("species,see,inject", [("ARGON", "NO", 33), ("ARGON", "NO", 300), ("ARGON", "YES", 300),
                                                ("HYDROGEN", "YES", 33)])
def test_collisions_and_walls_in_full_queues(species, see, inject):
    """A gas so dense that most electrons collide each step, and hot particles
    that reach the walls in long lists: event counts agree with the oracle to
    1% + 2 (decisions within FP32 rounding of their threshold)."""
    p = picgb.make_params(X_NO_OF_CELLS=33, STEADYSTATE="NO", HAVE_COLLISIONS=True, GAS_PRESSURE_TORR=200.0, RAND_SEED=4,
                          SPECIES=species, ION_MASS_AMU=1.0 if species == "HYDROGEN" else 39.948, THRESHOLD=15.75 if
                          species == "ARGON" else 13.6, SIGMA="ENERGY_DEPENDENT", SIGMA_ELASTIC="ENERGY_DEPENDENT",
                          SIGMA_IONIZATION="ENERGY_DEPENDENT", E_IMPACT_SEE=see, REFLECTION=see, BACKSCATTER=see,
                          NUMBER_TO_INJECT=inject, DTI_RATIO=2.0, SORT_INTERVAL=2)
    state = plasma(p, 30011, 8, temp_e=60.0, temp_i=30.0, lo=0.0, hi=1.0)
    o = orc.Oracle(p, rng=orc.ORC_RNG_PHILOX, order=orc.ORC_ORDER_STABLE)
    with loaded(p, state) as r:
        for s in (0, 1):
            o.load_particles(s, state[s])
        for x in (o, r):
            x.initial_boundary()
            x.step(3)
        co, cr = o.counters(), r.counters()
        assert co["elastic"] > 3000 and co["absorbed_e"] > 100
        assert co["charge_exchange"] > 1000 or species == "HYDROGEN"   # whose fit is below 1e-113
        for k in ("n_e", "n_i", "absorbed_e", "absorbed_i", "reflected", "backscattered", "see_events", "see_emitted",
                  "elastic", "ionization", "charge_exchange", "injected_e", "injected_i"):
            assert abs(cr[k] - co[k]) <= 0.01 * co[k] + 2, (k, cr[k], co[k])


# -------------------------------------------------------------------- plots
@pytest.mark.parametrize("size", [(1, 1), (33, 7), (1280, 1280), (1280, 1281)])
def test_plots_on_both_sides_of_the_layer_in_shared_memory(size):
    """An image's layer of one bit per pixel fits in shared memory up to
    1280 x 1280; both routes and ragged widths equal the oracle."""
    g = load_golden("core65")
    o = orc.Oracle(g["p"], rng=orc.ORC_RNG_PHILOX, order=orc.ORC_ORDER_STABLE)
    with picgb.Run(g["p"]) as r:
        for x in (o, r):
            x.load_particles(0, g["e_in"])
            x.load_particles(1, g["i_in"])
        for plot in ("particle_xy", "electron_vx_vy"):
            assert np.array_equal(r.render(plot, *size, 300, 7), o.render(plot, *size, 300, 7)), plot
