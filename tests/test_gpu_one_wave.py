"""Form 2 of apollo_dg_set_fp64_kernels (B200): the fused kernel up to the tiles
that its resident warps hold, the volume, face and LIFT kernels from one element
more, told apart by their bits."""
import numpy as np
import pytest

from apollo_b200 import NodalDG2d
from apollo_b200.mesh import Mesh, jittered_square

pytestmark = pytest.mark.gpu


def _mesh(K):
    m = jittered_square(int(np.ceil((K / 2) ** 0.5)) + 1, seed=1, periodic=False)
    return Mesh(vx=m.vx, vy=m.vy, etov=np.ascontiguousarray(m.etov[:K]), face_tag=np.ascontiguousarray(m.face_tag[:K]),
                vert_canon=m.vert_canon, n=0, lo=m.lo, hi=m.hi, periodic=False)


# the planar Maxwell system at order 5 has shared memory for fifteen warps
@pytest.mark.parametrize("kind,params,bc,flux,N,warps", [
    ("maxwellTM", (1.0,), "phmConductingWallBC", "LF", 5, 15),
    ("maxwellTM", (1.0,), "phmConductingWallBC", "LF", 3, 16),
    ("phMaxwellEqn", (1.0, 0.8, 0.6), "phmConductingWallBC", "LF", 4, 8),
    ("eulerEqn2d", (1.4, 0.0, 0.0), "eulerWallBC", "LF", 3, 16),
    ("eulerEqn", (1.4, 0.0, 0.0), "eulerWallBC", "HLL", 3, 8),
    ("eulerEqn2d", (1.4, 0.0, 0.0), "eulerWallBC", "Roe", 5, 8),
])
def test_one_wave(kind, params, bc, flux, N, warps):
    torch = pytest.importorskip("torch")
    one_wave = 8 * warps * torch.cuda.get_device_properties(0).multi_processor_count
    for K, form in ((one_wave, 1), (one_wave + 1, 0)):
        s = NodalDG2d(N, 0.5, kind, params, _mesh(K), bcs=((bc, ()),), numerical_flux=flux)
        U = np.random.default_rng(N).uniform(-0.1, 0.1, s.shape)
        if kind.startswith("euler"):
            U[..., 0] += 1.0
            U[..., -1] += 3.0
        got = {}
        for f in (0, 1, 2):
            s.set_fp64_kernels(f)
            got[f] = s.step(0.0, 0.0, U)[0]
        assert not np.array_equal(got[0], got[1])
        np.testing.assert_array_equal(got[2], got[form])
        s.close()
