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


@pytest.mark.parametrize("K", [7, 25])
@pytest.mark.parametrize("N", [2, 3, 4, 5])
@pytest.mark.parametrize("kind,flux", [(k, CASES[k][2]) for k in CASES] + [("eulerEqn2d", "LF")])
def test_derivatives_on_partial_tiles(kind, flux, N, K):
    """The tangent against central differences of the right-hand side (step
    1e-5 of the state: truncation 1e-10 of the third derivative, rounding 1e-16
    / 1e-5 of the terms, so 1e-7 relative), the adjoint as its transpose."""
    p, bc, _, _ = CASES[kind]
    s = NodalDG2d(N, 0.5, kind, p, _mesh(K, seed=N + 3), bcs=(bc,), numerical_flux=flux)
    rng = np.random.default_rng(K + N)
    x, v, w = _state(kind, s.shape, rng), rng.standard_normal(s.shape), rng.standard_normal(s.shape)
    if kind.startswith("euler") and flux != "LF":
        x[..., 1:-1] *= 1.01  # off the integers of the truncated HLL bound
    jv, jtw = s.rhs_jvp(0.2, x, v), s.rhs_vjp(0.2, x, w)
    h = 1e-5
    fd = (s.step(0.2, 0.0, x + h * v)[0] - s.step(0.2, 0.0, x - h * v)[0]) / (2 * h)
    if flux != "HLL":
        assert rel_l2(jv, fd) <= 1e-7
    scale = np.linalg.norm(jv) * np.linalg.norm(w)
    assert abs(np.vdot(jv, w) - np.vdot(v, jtw)) <= 1e-12 * scale


def test_derivatives_with_overlapping_and_misaligned_arrays():
    """Such arrays go through the handle's own buffers: the same bits."""
    torch = pytest.importorskip("torch")
    p, bc, _, _ = CASES["eulerEqn2d"]
    s = NodalDG2d(3, 0.5, "eulerEqn2d", p, _mesh(25, seed=2), bcs=(bc,))
    rng = np.random.default_rng(1)
    x, v = _state("eulerEqn2d", s.shape, rng), rng.standard_normal(s.shape)
    n, sh = x.size, s.shape
    xd, vd = torch.from_numpy(x).cuda(), torch.from_numpy(v).cuda()
    jv, jtv = s.rhs_jvp(0.0, xd, vd).cpu(), s.rhs_vjp(0.0, xd, vd).cpu()
    buf = torch.zeros(3 * n + 6, dtype=torch.float64, device="cuda")
    x1, v1, o1 = buf[1:1 + n].view(sh), buf[n + 1:2 * n + 1].view(sh), buf[2 * n + 3:3 * n + 3].view(sh)
    x1.copy_(xd)
    v1.copy_(vd)
    s.rhs_jvp(0.0, x1, v1, o1)
    assert torch.equal(o1.cpu(), jv)
    s.rhs_vjp(0.0, x1, v1, o1)
    assert torch.equal(o1.cpu(), jtv)
    x2, v2 = xd.clone(), vd.clone()
    s.rhs_jvp(0.0, x2, v2, v2)
    assert torch.equal(v2.cpu(), jv)


@pytest.mark.parametrize("kind", ["maxwellTM", "eulerEqn2d"])
def test_tangent_trajectory_is_the_transpose_of_the_adjoint(kind):
    """Two steps each way on a partial tile: the tangent's stage buffers."""
    p, bc, _, _ = CASES[kind]
    s = NodalDG2d(3, 0.5, kind, p, _mesh(25, seed=4), bcs=(bc,), numerical_flux="LF")
    rng = np.random.default_rng(7)
    x, v, w = _state(kind, s.shape, rng), rng.standard_normal(s.shape), rng.standard_normal(s.shape)
    s.set_state(x)
    du = s.tangent(2, 0.0, 1e-3, v)
    s.set_state(x)
    s.forward_fixed(2, 0.0, 1e-3, 1)
    g = s.backward(w)
    assert abs(np.vdot(du, w) - np.vdot(v, g)) <= 1e-12 * np.linalg.norm(du) * np.linalg.norm(w)
