"""The float64 stage kernel of each Euler flux (B200) against the volume, face
and LIFT kernels, which take every state through the equation's own code:
pressures on either side of the floor (Apollo's Wave flux floors them itself),
walls and inflow beside sound neighbours, non-physical states, and no flux,
order, field count or mesh size where it is the slower of the two."""
import numpy as np
import pytest

from apollo_b200 import ApolloError, NodalDG2d, problems
from apollo_b200.mesh import jittered_square
from golden_cases import rel_l2

pytestmark = pytest.mark.gpu

KIND = {4: "eulerEqn2d", 5: "eulerEqn"}
FLUXES = ["LF", "HLL", "Roe", "Wave"]


def _state(s, rng):
    U = rng.uniform(-0.05, 0.05, s.shape)
    U[..., 0] += 1.0
    U[..., 1] += 0.37  # off the integers of the truncated HLL bound
    U[..., 2] += 0.21
    U[..., -1] = 0.5 * (U[..., 1:-1] ** 2).sum(-1) / U[..., 0] + rng.uniform(2.4, 2.6, s.shape[:2])
    return U


def _both(s, U):
    got = {}
    for form in (1, 0):
        s.set_fp64_kernels(form)
        got[form] = s.step(0.1, 0.0, np.ascontiguousarray(U))
    return got


@pytest.mark.parametrize("N", [2, 3, 4, 5])
@pytest.mark.parametrize("fields", [4, 5])
@pytest.mark.parametrize("flux", FLUXES)
def test_pressure_floor_and_boundaries(flux, fields, N):
    """Elements whose pressure lies below, within rounding of and above the
    floor, in a mesh with a wall.  1e-12 as for the kernels' other comparisons."""
    floor = 0.75
    m = jittered_square(6, seed=2, periodic=False)  # K = 50: a partial tile
    s = NodalDG2d(N, 0.5, KIND[fields], (1.4, floor, 1e-3), m, bcs=(("eulerWallBC", ()),), numerical_flux=flux)
    rng = np.random.default_rng(10 * N + fields)
    U = _state(s, rng)
    kinetic = 0.5 * (U[..., 1:-1] ** 2).sum(-1) / U[..., 0]
    for k, p in ((3, 0.5), (11, floor), (12, floor * (1 + 1e-13)), (24, 0.76), (41, 1e-3)):
        U[k, :, -1] = kinetic[k] + p / 0.4
    got = _both(s, U)
    assert rel_l2(got[1][0], got[0][0]) <= 1e-12
    assert got[1][1] == pytest.approx(got[0][1], rel=1e-13)


@pytest.mark.parametrize("fields", [4, 5])
@pytest.mark.parametrize("flux", FLUXES)
def test_nonphysical_states_are_refused(flux, fields):
    s = NodalDG2d(3, 0.5, KIND[fields], (1.4, 0.0, 0.0), jittered_square(6, seed=2), numerical_flux=flux)
    rng = np.random.default_rng(fields)
    for sign in (0, -1):  # the density, the energy
        U = _state(s, rng)
        U[7, :, sign] *= -1.0
        for form in (1, 0):
            s.set_fp64_kernels(form)
            with pytest.raises(ApolloError) as e:
                s.step(0.0, 0.0, np.ascontiguousarray(U))
            assert e.value.code == 3  # APOLLO_ERR_NONPHYSICAL


@pytest.mark.parametrize("n", [17, 33, 91])
@pytest.mark.parametrize("N", [2, 3, 4, 5])
@pytest.mark.parametrize("fields", [4, 5])
@pytest.mark.parametrize("flux", FLUXES)
def test_not_slower_than_the_three_kernels(flux, fields, N, n):
    """K = 512, 2,048 and 16,200; measured 0.84 of the three kernels' time at most."""
    p = problems.euler_vortex(n=n, N=N, fields=fields)
    s = NodalDG2d(p.N, p.cfl, p.equation, p.eq_params, p.mesh, bcs=p.bcs, numerical_flux=flux)
    x, y = s.node_coords()
    s.set_state(np.ascontiguousarray(p.ic(x, y)))
    us = {0: [], 1: []}
    for _ in range(8):  # in turn, so that a slow spell meets both
        for form in (0, 1):
            s.set_fp64_kernels(form)
            s.kernel_times(3)
            us[form].append(sum(s.kernel_times(10)) * 1e3)
    s.close()
    assert min(us[1]) <= min(us[0])
