"""A step that ends in a capacity error leaves nothing to the next one.

In a run that may reduce its species the error comes back in the middle of a
step, with charge in the accumulators and ionization events counted.  A handle
that is loaded again after it must step exactly as a new one.
"""
import numpy as np
import pytest

import picgb

pytestmark = pytest.mark.gpu


def _state(p, n, seed):
    rng = np.random.default_rng(seed)
    out = []
    for m, t in ((picgb.ELECTRON_MASS, 30.0), (p.ion_mass, 1.0)):
        a = np.empty((n, 6))
        a[:, :2] = rng.uniform(0.1, 0.9, (n, 2)) * p.xlength
        a[:, 2:5] = rng.normal(0.0, np.sqrt(t * picgb.CHARGE / m), (n, 3))
        a[:, 5] = 1.0
        out.append(a)
    return out


def _step(r, state):
    """one step from `state` at time 0 without a field: the end state and what it counted"""
    for s in (0, 1):
        r.load_particles(s, state[s])
    r.set_time_step(0)
    r.set_rho(np.zeros((33, 33)))
    r.poisson(0)
    r.efield()
    before = r.counters()
    r.step(1)
    after = r.counters()
    return ([r.get_particles(s) for s in (0, 1)] + [r.get_ids(s) for s in (0, 1)]
            + [r.get_grid(k) for k in ("q_e", "q_i", "rho", "phi")],
            {k: after[k] - before[k] for k in after if k not in ("n_e", "n_i", "step")})


@pytest.mark.parametrize("collisions", [False, True])
def test_a_handle_steps_as_new_after_a_capacity_error(collisions):
    n, inject = 30000, 40000
    # room for two injections; the reduction limit lies just below it
    p = picgb.make_params(X_NO_OF_CELLS=33, STEADYSTATE="NO", HAVE_COLLISIONS=collisions, GAS_PRESSURE_TORR=60.0,
                          SIGMA_ELASTIC="ENERGY_DEPENDENT", SIGMA_IONIZATION="ENERGY_DEPENDENT", NUMBER_TO_INJECT=inject,
                          SIZE_TO_CHECK=2 * n + 65000, RAND_SEED=5)
    later = _state(p, 20000, 2)
    with picgb.Run(p) as r:
        for s, a in enumerate(_state(p, n, 1)):
            r.load_particles(s, a)
        r.step(2)
        with pytest.raises(picgb.PicError, match="capacity exceeded") as e:
            r.step(1)
        assert e.value.code == picgb.PGB_ERR_CAPACITY
        got, counted = _step(r, later)
    with picgb.Run(p) as r:
        want, expected = _step(r, later)
    assert counted == expected
    assert not collisions or expected["ionization"] > 20
    for k, (a, b) in enumerate(zip(got, want)):
        assert np.array_equal(a, b, equal_nan=True), k
