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
