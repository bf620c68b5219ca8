"""A run that injects as many particles as leave keeps within its capacity: the
counts by which the host decides to compact, or to grow the storage before a
sort, are fresh enough for a caller that queues a step at a time and waits for
the run's stream."""
import numpy as np
import pytest

import picgb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sort,inject", [(0, 9000), (0, 20000), (1, 9000), (2, 4000)])
def test_steady_injection_stays_within_the_capacity(sort, inject):
    torch = pytest.importorskip("torch")
    # a step takes a thermal particle of either species across the box, so most leave within one
    p = picgb.make_params(X_NO_OF_CELLS=33, STEADYSTATE="NO", SPECIES="HYDROGEN", ION_MASS_AMU=5.486e-4, DT_SCALE=64.0,
                          NUMBER_TO_INJECT=inject, SIZE_TO_CHECK=2**31 - 1, RAND_SEED=2, SORT_INTERVAL=sort)
    rng = np.random.default_rng(3)
    with picgb.Run(p) as r:
        for s in (0, 1):
            a = np.zeros((1000, 6))
            a[:, :2] = rng.uniform(0.1, 0.9, (1000, 2)) * p.xlength
            r.load_particles(s, a)
        stream = torch.cuda.ExternalStream(r.stream())
        for _ in range(40):   # 160 K and more injected, room for about 70 K slots
            assert r.lib.pgb_step_async(r.h, 1) == 0
            stream.synchronize()
        r.sync()
        c = r.counters()
    assert c["injected_e"] == c["injected_i"] == 40 * inject
    assert 0 < c["n_e"] < 4 * inject and 0 < c["n_i"] < 6 * inject


@pytest.mark.parametrize("nodes,sort,inject,n,collisions,poisson", [
    (129, 1, 4000, 30000, False, "FP32_DC"), (65, 1, 8000, 30000, True, "FMG_REF"), (129, 3, 5000, 1025, False, "DST_DC"),
    (129, 3, 8000, 30000, True, "FMG32")])
def test_storage_grows_in_time_for_steps_queued_ahead(nodes, sort, inject, n, collisions, poisson):
    """Steps queued without a wait, many ahead of the GPU: the growth before a
    sort counts the injection of the steps that the counts do not show yet."""
    p = picgb.make_params(X_NO_OF_CELLS=nodes, STEADYSTATE="NO", HAVE_COLLISIONS=collisions, GAS_PRESSURE_TORR=1.0,
                          SIGMA_ELASTIC="ENERGY_DEPENDENT", SIGMA_IONIZATION="ENERGY_DEPENDENT", POISSON=poisson,
                          DC_MAX_ITERS=2, NUMBER_TO_INJECT=inject, SIZE_TO_CHECK=2**31 - 1, SORT_INTERVAL=sort, RAND_SEED=6)
    rng = np.random.default_rng(8)
    state = []
    for m, t in ((picgb.ELECTRON_MASS, 3.0), (p.ion_mass, 0.03)):
        a = np.ones((n, 6))
        a[:, :2] = rng.uniform(0.02, 0.98, (n, 2)) * p.xlength
        a[:, 2:5] = rng.normal(0.0, np.sqrt(t * picgb.CHARGE / m), (n, 3))
        state.append(a)
    ends = []
    for queued in (True, False):
        with picgb.Run(p) as r:
            for s in (0, 1):
                r.load_particles(s, state[s])
            for _ in range(17):
                if queued:
                    assert r.lib.pgb_step_async(r.h, 1) == 0
                else:
                    r.step(1)
            r.sync()
            ends.append([r.get_particles(s) for s in (0, 1)] + [r.get_grid("phi")])
    for k, (a, b) in enumerate(zip(*ends)):
        assert np.array_equal(a, b, equal_nan=True), k
