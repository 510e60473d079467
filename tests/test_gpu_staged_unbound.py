"""Staged calls of a partition with peers whose halo buffers are not bound are
refused on the host (B200)."""
import numpy as np
import pytest

from apollo_b200 import ApolloError, NodalDG2d, problems
from apollo_b200.distributed import partition

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
def test_refused(prec):
    p = problems.euler_vortex(n=9, N=3)
    s = NodalDG2d(p.N, p.cfl, p.equation, p.eq_params, p.mesh, part=partition(p.mesh, 2), rank=0)
    x, y = s.node_coords()
    s.set_state(np.ascontiguousarray(p.ic(x, y)))
    for call in (s.lib.apollo_dg_stage_begin, s.lib.apollo_dg_stage_end):
        with pytest.raises(ApolloError) as e:
            s._check(call(s.h, 0, prec))
        assert e.value.code == 7  # APOLLO_ERR_STATE
    s.close()
