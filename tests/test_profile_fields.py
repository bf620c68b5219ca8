"""The profile's fields hold times of work or 0, not gaps between records."""
import pytest

import picgb
from conftest import load_golden

pytestmark = pytest.mark.gpu


def test_no_time_is_reported_for_a_kernel_that_is_not_launched():
    """The electron scatterings are part of the collision kernel."""
    g = load_golden("arcoll33")
    with picgb.Run(g["p"]) as r:
        r.load_particles(0, g["e_in"])
        r.load_particles(1, g["i_in"])
        r.set_profiling(True)
        r.step(4)
        t = r.profile()
    assert t["steps"] == 4 and t["ms_collide_e"] > 0.0 and t["ms_push_e_kernel"] > 0.0
    assert t["ms_scatter_e"] == 0.0
