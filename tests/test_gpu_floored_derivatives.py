"""Tangent and adjoint of Euler states below the density floor (B200), where both
leave their fast derivatives for those of the equation's own code: the tangent
against central differences, the adjoint as its transpose."""
import numpy as np
import pytest

from apollo_b200 import NodalDG2d
from apollo_b200.mesh import jittered_square
from golden_cases import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("N", [2, 3, 4, 5])
@pytest.mark.parametrize("fields", [4, 5])
def test_below_the_density_floor(fields, N, walls):
    """Central differences with a step of 1e-6, densities from 0.1: truncation 1e-10
    of the third derivative, rounding 1e-16 / 1e-6 of terms a hundred times the
    result, so 1e-7 relative; no state within a step of the floor."""
    m = jittered_square(6, seed=N, periodic=not walls)  # K = 50: a partial tile
    s = NodalDG2d(N, 0.5, {4: "eulerEqn2d", 5: "eulerEqn"}[fields], (1.4, 1e-3, 0.2), m,
                  bcs=(("eulerWallBC", ()),) if walls else ())
    rng = np.random.default_rng(10 * N + fields)
    x = rng.uniform(-0.02, 0.02, s.shape)
    x[..., 0] += 1.0
    x[..., 1] += 0.3
    x[6, :, 0] = 0.15
    x[33, :, :-1] *= 0.12
    x[49, :, 0] = 0.17
    x[..., -1] = 0.5 * (x[..., 1:-1] ** 2).sum(-1) / x[..., 0] + rng.uniform(2.4, 2.6, s.shape[:2])
    v, w = rng.standard_normal(s.shape), rng.standard_normal(s.shape)
    jv = s.rhs_jvp(0.0, x, v)
    h = 1e-6
    fd = (s.step(0.0, 0.0, x + h * v)[0] - s.step(0.0, 0.0, x - h * v)[0]) / (2 * h)
    assert rel_l2(jv, fd) <= 1e-7
    # the transpose, also with points of one element on both sides of the floor
    for crossing in (False, True):
        if crossing:
            x[20, :, 0] = 0.21  # the interpolant stays positive
            x[20, : s.Np // 2, 0] = 0.19
            x[20, :, -1] += 1.0
        jv, jtw = s.rhs_jvp(0.0, x, v), s.rhs_vjp(0.0, x, w)
        scale = np.linalg.norm(jv) * np.linalg.norm(w)
        assert abs(np.vdot(jv, w) - np.vdot(v, jtw)) <= 1e-12 * scale
