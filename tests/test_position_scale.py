"""Record positions in cells of extreme size.

The integer form of x / DX must leave to the division what it does not
represent: a position of 0 (or a subnormal one) has no leading 1 in its
mantissa.  A particle at x = 0 deposits nothing (particle.cpp:491-510), in
cells of any size that pgb_deposit_static accepts.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes", [17, 33, 65])
@pytest.mark.parametrize("exponent", [-1003, -1000, -990, -900, -40, 900])
def test_a_particle_at_zero_deposits_nothing(lib, nodes, exponent):
    torch = pytest.importorskip("torch")
    dx = 2.0**exponent
    a = np.zeros((3, 6))
    a[:, 5] = 1.0
    a[:, 1] = 2.5           # dy is 1
    a[0, 0] = 0.0
    a[1, 0] = -0.0
    a[2, 0] = 3.0 * dx      # on node 3: half its charge on each of rows 2 and 3
    recs, st = torch.from_numpy(a).cuda(), torch.cuda.current_stream()
    q = torch.full((nodes, nodes), float("nan"), dtype=torch.float64, device="cuda")
    assert lib.pgb_deposit_static(C.c_void_p(recs.data_ptr()), 3, nodes, nodes, dx, 1.0, dx, C.c_void_p(q.data_ptr()),
                                  C.c_void_p(st.cuda_stream)) == 0
    want = np.zeros((nodes, nodes))
    want[2:4, 3] = 0.5
    assert np.array_equal(q.cpu().numpy(), want)
