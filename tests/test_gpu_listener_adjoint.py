"""S^H pbar and D^H pbar (bem_boundary2potential_adjoint) against the FP64
potential matrices: listeners around the edges of the kernel's split (one lane
per quadrature point below 16, up to 32 lanes, remainders), equal weights at a
low wavenumber, so that every sum grows from its first term to its last.

Tolerance, with u = 2^-24: an addition to a growing sum is off by about 0.4 u of
its value, n of them by 0.4 u sqrt(n / 3) of the result.  A vertex takes 6
additions per triangle (36 here: 1.4 u), a lane's chain at most 64 listeners
(1.9 u, independent between the points: less), the kernel's own values 2 u,
independent as well.  4 u in all, as the 2-norm over the vertices.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level", [0, 2])
@pytest.mark.parametrize("points", [1, 8, 15, 16, 17, 63, 64, 615, 2000])
def test_listener_adjoint(level, points):
    import torch

    from neuralat_b200 import _lib as L
    from neuralat_b200.bem import BEM_Solver
    from neuralat_b200.bem import meshes as M

    O.build()
    v, t = M.icosphere(level, 0.1)
    v, t = (v * [1.2, 0.8, 1.0]).astype(np.float32), t.astype(np.int32)
    x = M.sphere_points(points, 0.5, seed=points).astype(np.float32)
    k = 2.0
    s = BEM_Solver(v, t)
    X, pbar = torch.from_numpy(x).cuda(), torch.ones(points, dtype=torch.complex64, device="cuda")
    out = [torch.empty(len(v), dtype=torch.complex64, device="cuda") for _ in range(2)]
    L.check(L.lib().bem_boundary2potential_adjoint(s.geometry.ptr, X.data_ptr(), points, k, pbar.data_ptr(),
                                                   out[0].data_ptr(), out[1].data_ptr(),
                                                   torch.cuda.current_stream().cuda_stream))
    for layer, got in zip(("single", "double"), out):
        P = O.potential_matrix(layer, v.astype(np.float64), t, x.astype(np.float64), np.float32(k))
        ref = P.conj().T @ np.ones(points)
        err = np.linalg.norm(got.cpu().numpy() - ref) / np.linalg.norm(ref)
        assert err < 4 * 2.0 ** -24, (layer, err)
