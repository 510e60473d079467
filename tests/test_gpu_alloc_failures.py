"""A device allocation that fails in a call on a ready handle (B200; the test
hook makes the n-th one fail on the host): the call reports it, and later calls
find every buffer they use, or say that there is no trajectory."""
import numpy as np
import pytest

from apollo_b200 import ApolloError, NodalDG2d, problems
from apollo_b200.mesh import jittered_square

pytestmark = pytest.mark.gpu

ERR_STATE, ERR_ALLOC = 7, 9


def _fails(s, nth, call):
    s.lib.apollo_dg_debug_fail_alloc(nth)
    try:
        with pytest.raises(ApolloError) as e:
            call()
    finally:
        s.lib.apollo_dg_debug_fail_alloc(-1)
    assert e.value.code == ERR_ALLOC


def _vortex(N=2):
    p = problems.euler_vortex(n=7, N=N)
    s = NodalDG2d(p.N, p.cfl, p.equation, p.eq_params, p.mesh)
    x, y = s.node_coords()
    return s, np.ascontiguousarray(p.ic(x, y))


@pytest.mark.parametrize("nth", range(9))
def test_derivative_buffers(nth):
    rng = np.random.default_rng(nth)
    s, U = _vortex()
    v = rng.standard_normal(U.shape)
    ref = _vortex()[0]
    _fails(s, nth, lambda: s.rhs_jvp(0.0, U, v))
    np.testing.assert_array_equal(s.rhs_vjp(0.0, U, v), ref.rhs_vjp(0.0, U, v))
    np.testing.assert_array_equal(s.rhs_jvp(0.0, U, v), ref.rhs_jvp(0.0, U, v))
    for h in (s, ref):
        h.set_state(U)
    np.testing.assert_array_equal(s.tangent(1, 0.0, 1e-3, v), ref.tangent(1, 0.0, 1e-3, v))


@pytest.mark.parametrize("again", ["fixed", "revolve"])
def test_trajectory_ends_before_its_buffers_are_resized(again):
    s, U = _vortex()
    s.set_state(U)
    s.forward_fixed(4, 0.0, 1e-3, 1)  # four checkpoints, a segment of one step
    if again == "fixed":
        _fails(s, 0, lambda: s.forward_fixed(4, 0.0, 1e-3, 4))  # one checkpoint, a segment of four
    else:
        _fails(s, 0, lambda: s.forward_revolve(6, 0.0, 1e-3, 6))  # six slots
    with pytest.raises(ApolloError) as e:
        s.backward(U)
    assert e.value.code == ERR_STATE
    s.set_state(U)
    s.forward_fixed(2, 0.0, 1e-3, 1)
    assert np.isfinite(s.backward(U)).all()


@pytest.mark.parametrize("nth", range(3))
def test_limiter_buffers(nth):
    args = ("eulerLimiterHW", (1.4, 1e-4, 1e-4))
    s, U = _vortex()
    ref = _vortex()[0]
    _fails(s, nth, lambda: s.set_limiter(*args))
    np.testing.assert_array_equal(s.step(0.0, 0.0, U)[0], ref.step(0.0, 0.0, U)[0])  # still without one
    for h in (s, ref):
        h.set_limiter(*args)
    np.testing.assert_array_equal(s.step(0.0, 0.0, U)[0], ref.step(0.0, 0.0, U)[0])


def test_source_buffer():
    src = ("tranverseMagneticSrc", (2,), ())
    m = jittered_square(7, seed=1, periodic=False)

    def make(sources):
        return NodalDG2d(3, 0.5, "maxwellTM", (1.0,), m, bcs=(("maxwellTransverseMagneticBC", ()),), sources=sources)

    def add(s):
        out = np.asarray(src[1], dtype=np.int32)
        import ctypes as C
        s._check(s.lib.apollo_dg_add_source(s.h, src[0].encode(), out.ctypes.data_as(C.POINTER(C.c_int)), 1, None, 0))

    s, bare, full = make(()), make(()), make((src,))
    U = np.random.default_rng(0).standard_normal(s.shape)
    _fails(s, 0, lambda: add(s))
    for prec in ("fp64", "mixed"):  # the source that could not be held is not there
        np.testing.assert_array_equal(s.step(0.3, 0.0, U, precision=prec)[0], bare.step(0.3, 0.0, U, precision=prec)[0])
    add(s)
    for prec in ("fp64", "mixed"):
        np.testing.assert_array_equal(s.step(0.3, 0.0, U, precision=prec)[0], full.step(0.3, 0.0, U, precision=prec)[0])
