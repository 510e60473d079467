"""Staged stepping takes the wave speed of its own last stage (B200): what a
call between two steps left in the handle's wave-speed word (a right-hand side
of a faster state, apollo_dg_init_dt) does not reach dt."""
import ctypes as C

import numpy as np
import pytest

from apollo_b200 import NodalDG2d, problems
from apollo_b200.dg import PREC

pytestmark = pytest.mark.gpu


def _step(s, prec):
    for stage in range(5):
        s._check(s.lib.apollo_dg_stage_begin(s.h, stage, PREC[prec]))
        s._check(s.lib.apollo_dg_stage_end(s.h, stage, PREC[prec]))
    s._check(s.lib.apollo_dg_step_end(s.h))


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("fields,N", [(4, 4), (4, 2), (5, 3)])  # both mixed stage kernels
def test_calls_between_steps(fields, N, prec):
    p = problems.euler_vortex(n=12, N=N, fields=fields)
    got = []
    for interrupted in (False, True):
        # one part: staged calls without peers
        s = NodalDG2d(p.N, p.cfl, p.equation, p.eq_params, p.mesh, part=np.zeros(p.mesh.K, np.int32), rank=0)
        x, y = s.node_coords()
        U = np.ascontiguousarray(p.ic(x, y))
        fast = U.copy()
        fast[..., -1] *= 100.0  # nine times the sound speed and more
        s.set_state(U)
        dt0 = s.init_dt()
        s._check(s.lib.apollo_dg_dist_start(s.h, 0.0, dt0, PREC[prec]))
        _step(s, prec)
        if interrupted:
            s.init_dt()
            assert s.step(0.0, 0.0, fast)[1] < 0.5 * dt0
        _step(s, prec)
        t, dt = C.c_double(), C.c_double()
        s._check(s.lib.apollo_dg_get_time(s.h, C.byref(t), C.byref(dt)))
        got.append((t.value, dt.value, s.get_state()))
    assert got[0][:2] == got[1][:2]
    np.testing.assert_array_equal(got[0][2], got[1][2])
