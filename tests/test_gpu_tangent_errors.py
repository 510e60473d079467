"""What the tangent calls report (B200): a non-physical state at a cubature
point and a NaN in the result end rhs_jvp and tangent with an error, for the
fluxes of every tangent kernel; sound inputs do not."""
import numpy as np
import pytest

from apollo_b200 import ApolloError, NodalDG2d
from apollo_b200.mesh import jittered_square

pytestmark = pytest.mark.gpu

NONPHYSICAL, NAN = 3, 4
KINDS = [("advectionEqn", (0.7, -1.2, 0.0), "LF"), ("maxwellTM", (1.3,), "LF"), ("phMaxwellEqn", (1.3, 0.2, 0.7), "LF"),
         ("eulerEqn", (1.4, 0.0, 0.0), "LF"), ("eulerEqn2d", (1.4, 0.0, 0.0), "LF"),
         ("eulerEqn2d", (1.4, 0.0, 0.0), "Roe")]


def _setup(kind, params, flux, N):
    s = NodalDG2d(N, 0.5, kind, params, jittered_square(4, seed=N), numerical_flux=flux)  # K = 18: a partial tile
    rng = np.random.default_rng(N)
    U = rng.uniform(-0.1, 0.1, s.shape)
    if kind.startswith("euler"):
        U[..., 0] += 1.0
        U[..., -1] += 3.0
    return s, U, rng.standard_normal(s.shape)


def _code(call):
    with pytest.raises(ApolloError) as e:
        call()
    return e.value.code


@pytest.mark.parametrize("N", [2, 3, 5])
@pytest.mark.parametrize("kind,params,flux", KINDS)
def test_nan_is_reported(kind, params, flux, N):
    s, U, v = _setup(kind, params, flux, N)
    s.rhs_jvp(0.0, U, v)
    for k, node in ((0, 0), (s.K - 1, s.Np - 1)):  # the first and the last node of the mesh
        bad = v.copy()
        bad[k, node, 0] = np.nan
        assert _code(lambda: s.rhs_jvp(0.0, U, bad)) == NAN
        s.set_state(U)
        assert _code(lambda: s.tangent(1, 0.0, 1e-4, bad)) == NAN
    assert np.isfinite(s.rhs_jvp(0.0, U, v)).all()


@pytest.mark.parametrize("N", [2, 3, 5])
@pytest.mark.parametrize("kind,params,flux", [k for k in KINDS if k[0].startswith("euler")])
def test_nonphysical_state_is_reported(kind, params, flux, N):
    s, U, v = _setup(kind, params, flux, N)
    bad = U.copy()
    bad[s.K - 1, :, -1] = -1.0
    assert _code(lambda: s.rhs_jvp(0.0, bad, v)) == NONPHYSICAL
    assert np.isfinite(s.rhs_jvp(0.0, U, v)).all()
