"""Which states the float64 Euler kernels send to the equation's own flux code
(B200): densities on either side of the floor give what the volume, face and
LIFT kernels give, for every flux, order and field count, and sound states stay
on the fast fluxes (a right-hand side with the HLL flux then costs at most half
as much again as with Lax-Friedrichs; with sound states on the general code it
cost 1.9 times as much)."""
import time

import numpy as np
import pytest

from apollo_b200 import NodalDG2d, problems
from apollo_b200.mesh import jittered_square
from golden_cases import rel_l2

pytestmark = pytest.mark.gpu

KIND = {4: "eulerEqn2d", 5: "eulerEqn"}


@pytest.mark.parametrize("floor", [0.0, 0.05, 2.0 ** -4, 1e-3])
@pytest.mark.parametrize("N", [2, 3, 4, 5])
@pytest.mark.parametrize("fields", [4, 5])
@pytest.mark.parametrize("flux", ["LF", "HLL", "Roe", "Wave"])
def test_densities_at_the_floor(flux, fields, N, floor):
    """Whole elements just below, at and just above the floor (also within its
    high word).  1e-12 as for the kernels' other comparisons; velocities off the
    integers of the truncated HLL bound."""
    s = NodalDG2d(N, 0.5, KIND[fields], (1.4, 1e-3, floor), jittered_square(6, seed=1), numerical_flux=flux)
    rng = np.random.default_rng(N)
    U = rng.uniform(-0.01, 0.01, s.shape)
    U[..., 0] += 1.0
    base = floor or 1e-3
    for k, r in ((1, 1 - 1e-9), (4, 1.0), (8, 1 + 1e-12), (13, 1 + 2.0 ** -22), (21, 1 + 1e-3), (30, 1.7)):
        U[k, :, 0] = base * r
        U[k, :, 1:-1] *= base
    U[..., -1] = 0.5 * (U[..., 1:-1] ** 2).sum(-1) / U[..., 0] + 2.345 * U[..., 0] + rng.uniform(0, 0.01, s.shape[:2])
    U = np.ascontiguousarray(U)
    got = {}
    for form in (1, 0):
        s.set_fp64_kernels(form)
        got[form] = s.step(0.0, 0.0, U)
    assert rel_l2(got[1][0], got[0][0]) <= 1e-12
    assert got[1][1] == pytest.approx(got[0][1], rel=1e-13)


@pytest.mark.parametrize("N", [2, 3, 4, 5])
@pytest.mark.parametrize("fields", [4, 5])
def test_sound_states_take_the_fast_flux(fields, N):
    p = problems.euler_vortex(n=91, N=N, fields=fields)
    s = {f: NodalDG2d(p.N, p.cfl, p.equation, p.eq_params, p.mesh, bcs=p.bcs, numerical_flux=f) for f in ("LF", "HLL")}
    us = {"LF": [], "HLL": []}
    for h in s.values():
        x, y = h.node_coords()
        h.set_state(np.ascontiguousarray(p.ic(x, y)))
    for _ in range(8):  # in turn, so that a slow spell meets both
        for f, h in s.items():
            h.kernel_times(3)
            us[f].append(sum(h.kernel_times(10)) * 1e3)
    assert min(us["HLL"]) <= 1.5 * min(us["LF"])


@pytest.mark.parametrize("N", [4, 5])
def test_sound_states_take_the_fast_tangent(N):
    """The tangent of 5 fields against that of 4 (1.3 and 1.6 times as long; with
    sound states differentiated through the equation's own code 2.6 and 3.2)."""
    torch = pytest.importorskip("torch")
    us = {}
    for fields in (4, 5):
        p = problems.euler_vortex(n=181, N=N, fields=fields)
        s = NodalDG2d(p.N, p.cfl, p.equation, p.eq_params, p.mesh)
        x, y = s.node_coords()
        U = torch.from_numpy(np.ascontiguousarray(p.ic(x, y))).cuda()
        v, out = torch.ones_like(U), torch.empty_like(U)
        times = []
        for _ in range(25):
            t = time.perf_counter()
            s.rhs_jvp(0.0, U, v, out)
            times.append(time.perf_counter() - t)
        us[fields] = np.median(times[5:])
        s.close()
    assert us[5] <= 2.0 * us[4]
