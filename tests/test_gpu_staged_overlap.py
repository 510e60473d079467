"""What is queued behind apollo_dg_stage_begin runs beside the stage of the
elements without a cut face (B200): a small copy on the handle's stream, queued
when that stage already runs, ends well before it does."""
import time

import numpy as np
import pytest

from apollo_b200 import problems
from apollo_b200.distributed import DistNodalDG2d, partition

pytestmark = pytest.mark.gpu


def test_copy_beside_the_interior_stage():
    torch = pytest.importorskip("torch")

    class OneRank:  # one rank of two, its exchange a local copy
        rank, size = 0, 2

        def allreduce_min(self, x):
            return x

    p = problems.euler_vortex(n=320, N=5)  # some 0.3 ms of interior work
    d = DistNodalDG2d(p.N, p.cfl, p.equation, p.eq_params, p.mesh, partition(p.mesh, 2), OneRank(), bcs=p.bcs)
    x, y = d.node_coords()
    d.set_state(np.ascontiguousarray(p.ic(x, y)))
    chk, lib, h, st = d.solver._check, d.lib, d.h, d.torch_stream
    dt = d.init_dt()
    chk(lib.apollo_dg_dist_start(h, 0.0, dt, 0))
    a = torch.zeros(1 << 16, device="cuda")
    b = torch.zeros_like(a)
    ratio = []
    for stage in [0, 1, 2, 3] * 3:
        torch.cuda.synchronize()
        begun, copied, done = (torch.cuda.Event(enable_timing=True) for _ in range(3))
        with torch.cuda.stream(st):
            begun.record(st)
            chk(lib.apollo_dg_stage_begin(h, stage, 0))
            end = time.perf_counter() + 40e-6
            while time.perf_counter() < end:
                pass
            b.copy_(a)
            copied.record(st)
            d.recv.copy_(d.send)
            chk(lib.apollo_dg_stage_end(h, stage, 0))
            done.record(st)
        torch.cuda.synchronize()
        ratio.append(begun.elapsed_time(copied) / begun.elapsed_time(done))
    d.close()
    # a launch on every SM lets the copy start at its end, some 0.85 of the way
    assert np.median(ratio) < 0.5
