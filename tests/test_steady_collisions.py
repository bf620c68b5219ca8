"""Steady-state walls together with collisions, pipelined against in order.

Steady walls keep the ionization products of every step, so on an ion step
the electrons' kernels append ions while the charge exchange of the ions that
were there before runs on the ions' stream.  The exchange must see the ions
before the products join, whatever the kernels' lengths: few electrons beside
many ions, and the other way round.  With THRESHOLD 0 the products have finite
velocities and take part in the later passes.

Tolerance: none; the same steps in order, and one call per step, are the
reference.
"""
import numpy as np
import pytest

import picgb

pytestmark = pytest.mark.gpu


def _state(p, ne, ni, seed):
    rng = np.random.default_rng(seed)
    out = []
    for n, m, t in ((ne, picgb.ELECTRON_MASS, 40.0), (ni, p.ion_mass, 5.0)):
        a = np.empty((n, 6))
        a[:, :2] = rng.uniform(0.02, 0.98, (n, 2)) * p.xlength
        a[:, 2:5] = rng.normal(0.0, np.sqrt(t * picgb.CHARGE / m), (n, 3))
        a[:, 5] = 1.0
        out.append(a)
    return out


def _run(p, state, n, mode):
    with picgb.Run(p) as r:
        for s in (0, 1):
            r.load_particles(s, state[s])
        r.initial_boundary()
        if mode == "in order":
            r.set_profiling(True)
        if mode == "one call per step":
            for _ in range(n):
                r.step(1)
        else:
            r.step(n)
        return ([r.get_particles(s) for s in (0, 1)] + [r.get_ids(s) for s in (0, 1)]
                + [r.get_grid(k) for k in ("q_e", "q_i", "phi")], r.counters())


@pytest.mark.parametrize("threshold", [15.75, 0.0])
@pytest.mark.parametrize("ne,ni,dti,sort,inject", [(30011, 30011, 1.0, 0, 0), (30011, 9001, 2.0, 4, 0),
                                                   (1500, 600007, 1.0, 0, 0), (1500, 600007, 1.0, 5, 7)])
def test_products_join_after_the_charge_exchange(ne, ni, dti, sort, inject, threshold):
    p = picgb.make_params(X_NO_OF_CELLS=65, STEADYSTATE="YES", HAVE_COLLISIONS=True, GAS_PRESSURE_TORR=60.0, RAND_SEED=9,
                          SIGMA="ENERGY_DEPENDENT", SIGMA_ELASTIC="ENERGY_DEPENDENT",
                          SIGMA_IONIZATION="ENERGY_DEPENDENT", THRESHOLD=threshold, DTI_RATIO=dti, SORT_INTERVAL=sort,
                          NUMBER_TO_INJECT=inject)
    state = _state(p, ne, ni, ne + ni)
    want, count = _run(p, state, 9, "in order")
    assert count["ionization"] > 20 and count["charge_exchange"] > 100
    for mode in ("pipelined", "one call per step"):
        got, c = _run(p, state, 9, mode)
        assert c == count, mode
        for k, (a, b) in enumerate(zip(want, got)):
            assert np.array_equal(a, b, equal_nan=True), (mode, k)
