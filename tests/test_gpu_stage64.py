"""The fused float64 stage kernel where its tiling can go wrong (B200): meshes
whose element count is below, at and above its tiles of eight, states that take
the equations' own flux code (floors, non-physical), and inputs it must not
take (an output over its input, arrays off a 16-byte boundary), against the
volume, face and LIFT kernels.  Tolerance: both forms evaluate the same sums of
some hundred float64 terms in different orders, 1e-12 relative L2 as in the
parity tests (1e-11 where the terms cancel)."""
import numpy as np
import pytest

from apollo_b200 import ApolloError, NodalDG2d
from apollo_b200.mesh import Mesh, jittered_square
from golden_cases import rel_l2

pytestmark = pytest.mark.gpu

CASES = {
    "advectionEqn": ((0.7, -1.2, 0.0), ("gridFixedBC", (0.25,)), "LF", 1),
    "maxwellTM": ((1.3,), ("phmConductingWallBC", ()), "upwind", 3),
    "phMaxwellEqn": ((1.3, 0.2, 0.7), ("phmConductingWallBC", ()), "LF", 8),
    "eulerEqn": ((1.4, 0.0, 0.0), ("eulerWallBC", ()), "LF", 5),
    "eulerEqn2d": ((1.4, 0.0, 0.0), ("isentropicVortexBC", (1.0, 0.3, 1.0, 0.5, 1.4, 2.0)), "HLL", 4),
}


def _mesh(K, seed):
    """The first K triangles of a walled square; faces left without a partner
    are boundary faces of condition 1."""
    m = jittered_square(7, (0.0, 0.0), (2.0, 1.0), seed=seed, periodic=False)
    return Mesh(vx=m.vx, vy=m.vy, etov=np.ascontiguousarray(m.etov[:K]), face_tag=np.ascontiguousarray(m.face_tag[:K]),
                vert_canon=m.vert_canon, n=0, lo=m.lo, hi=m.hi, periodic=False)


def _state(kind, shape, rng):
    U = rng.uniform(-1, 1, shape)
    if kind.startswith("euler"):
        U *= 0.1
        U[..., 0] += 1.0
        U[..., 1] += 0.5
        U[..., -1] += 0.5 * (U[..., 1:-1] ** 2).sum(-1) / U[..., 0] + 2.0
    return np.ascontiguousarray(U)


def _solver(kind, N, mesh, params=None):
    p, bc, flux, _ = CASES[kind]
    return NodalDG2d(N, 0.5, kind, params or p, mesh, bcs=(bc,), numerical_flux=flux)


@pytest.mark.parametrize("K", [1, 7, 8, 9, 25])
@pytest.mark.parametrize("N", [2, 3, 4, 5])
@pytest.mark.parametrize("kind", list(CASES))
def test_partial_tiles(kind, N, K):
    s = _solver(kind, N, _mesh(K, seed=N))
    U = _state(kind, s.shape, np.random.default_rng(10 * K + N))
    got = {}
    for form in (1, 0):
        s.set_fp64_kernels(form)
        r, sugg = s.step(0.3, 0.01, U)
        s.set_state(U)
        t, dt = s.advance(2, 0.0, 1e-3)
        got[form] = (r, sugg, s.get_state(), dt)
    assert rel_l2(got[1][0], got[0][0]) <= 1e-12
    assert got[1][1] == pytest.approx(got[0][1], rel=1e-14)
    assert rel_l2(got[1][2], got[0][2]) <= 1e-12
    assert got[1][3] == pytest.approx(got[0][3], rel=1e-13)


@pytest.mark.parametrize("kind", ["eulerEqn", "eulerEqn2d"])
def test_floored_states(kind):
    """Densities and pressures below the floors take the equation's own code,
    beside points of the same element that do not."""
    s = _solver(kind, 3, _mesh(25, seed=1), params=(1.4, 1e-3, 0.05))
    U = _state(kind, s.shape, np.random.default_rng(3))
    U[2, :, 0] = 0.01                # below minDensity
    U[5, 3, -1] = 0.05               # negative pressure at one node
    U[9, :, 0] = 0.05                # at the floor
    got = {}
    for form in (1, 0):
        s.set_fp64_kernels(form)
        got[form] = s.step(0.0, 0.0, U)
    assert rel_l2(got[1][0], got[0][0]) <= 1e-12
    assert got[1][1] == pytest.approx(got[0][1], rel=1e-13)
    bad = _solver(kind, 3, _mesh(25, seed=1))  # no floors
    for form in (1, 0):
        bad.set_fp64_kernels(form)
        with pytest.raises(ApolloError) as e:
            bad.step(0.0, 0.0, np.where(np.arange(25)[:, None, None] == 4, -U, U))
        assert e.value.code == 3     # APOLLO_ERR_NONPHYSICAL


@pytest.mark.parametrize("kind", ["maxwellTM", "eulerEqn2d"])
def test_overlapping_and_misaligned_arrays(kind):
    torch = pytest.importorskip("torch")
    s = _solver(kind, 4, _mesh(25, seed=2))
    U = _state(kind, s.shape, np.random.default_rng(5))
    ref, sugg = s.step(0.1, 0.01, U)
    n = U.size
    buf = torch.zeros(2 * n + 3, dtype=torch.float64, device="cuda")
    views = {
        "in place": (buf[:n], buf[:n]),
        "shifted": (buf[2:2 + n], buf[4:4 + n]),
        "odd input": (buf[1:1 + n], buf[n + 2:2 * n + 2]),
        "odd output": (buf[:n], buf[n + 1 + n % 2:2 * n + 1 + n % 2][:n]),
    }
    for name, (x, out) in views.items():
        x, out = x.view(s.shape), out.view(s.shape)
        x.copy_(torch.from_numpy(U))
        _, got = s.step(0.1, 0.01, x, out)
        assert rel_l2(out.cpu().numpy(), ref) <= 1e-12, name
        assert got == pytest.approx(sugg, rel=1e-14), name
