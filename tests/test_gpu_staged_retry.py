"""A partitioned step whose exchange fails (B200): the error reaches the caller,
the state is still the one the step started from, and the step taken again
gives, bit for bit, what an undisturbed run gives.  The ranks are host threads
on one device whose kernels never wait on one another; the failure is a message
that the communicator drops, on every rank in the same stage."""
import numpy as np
import pytest

from apollo_b200 import problems
from apollo_b200.distributed import DistNodalDG2d, partition
from thread_comm import ThreadComm, run_ranks

pytestmark = pytest.mark.gpu


class Dropped(Exception):
    pass


class DroppingComm(ThreadComm):
    """Drops the exchange number `at` (counted from the first call)."""

    def __init__(self, comm, at):
        super().__init__(comm.g, comm.rank)
        self.at, self.calls = at, 0

    def exchange(self, *args):
        self.calls += 1
        if self.calls - 1 == self.at:
            raise Dropped
        super().exchange(*args)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("stage", [0, 1, 3, 4])
def test_dropped_exchange(stage, precision):
    p = problems.euler_vortex(n=21, N=3)
    part = partition(p.mesh, 2)

    def run(drop):
        def fn(rank, comm):
            c = DroppingComm(comm, 5 + stage if drop else -1)
            d = DistNodalDG2d(p.N, p.cfl, p.equation, p.eq_params, p.mesh, part, c, bcs=p.bcs)
            x, y = d.node_coords()
            d.set_state(np.ascontiguousarray(p.ic(x, y)))
            t, dt = d.advance(1, 0.0, d.init_dt(), precision=precision)
            before = d.get_state()
            if drop:
                with pytest.raises(Dropped):
                    d.advance(2, t, dt, precision=precision)
                np.testing.assert_array_equal(d.get_state(), before)
            t, dt = d.advance(2, t, dt, precision=precision)
            out = d.get_state(), t, dt
            d.close()
            return out

        return run_ranks(2, fn)

    for (U, t, dt), (Ur, tr, dtr) in zip(run(True), run(False)):
        np.testing.assert_array_equal(U, Ur)
        assert (t, dt) == (tr, dtr)


def test_stage_begun_again():
    """apollo_dg_stage_begin twice in a row (a retried exchange) changes nothing."""
    p = problems.euler_vortex(n=21, N=2)
    part = partition(p.mesh, 2)

    class Again(ThreadComm):
        again = None

        def exchange(self, *args):
            if self.again:
                self.again()
            super().exchange(*args)

    def run(twice):
        def fn(rank, comm):
            c = Again(comm.g, comm.rank)
            d = DistNodalDG2d(p.N, p.cfl, p.equation, p.eq_params, p.mesh, part, c, bcs=p.bcs)
            x, y = d.node_coords()
            d.set_state(np.ascontiguousarray(p.ic(x, y)))
            stage = [0]

            def begin():
                d.solver._check(d.lib.apollo_dg_stage_begin(d.h, stage[0] % 5, 0))
                stage[0] += 1

            if twice:
                c.again = begin
            t, dt = d.advance(2, 0.0, d.init_dt())
            out = d.get_state(), t, dt
            d.close()
            return out

        return run_ranks(2, fn)

    for (U, t, dt), (Ur, tr, dtr) in zip(run(True), run(False)):
        np.testing.assert_array_equal(U, Ur)
        assert (t, dt) == (tr, dtr)
