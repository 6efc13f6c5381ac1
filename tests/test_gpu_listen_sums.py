"""Accuracy of the listeners' FP32 sums where they are longest: few listeners on
many triangles (hundreds of runs are added to an output), many listeners (long
runs), either kernel, at a wavenumber that leaves the summation as the main
error; against the FP64 potential matrices.

Tolerance, with u = 2^-24: n additions to a sum that grows are off by about
0.4 u sqrt(n / 3) of it.  An output takes at most 148 runs' sums (2.8 u), a chain
within a run at most 80 FMAs (2.1 u); the hardware's sine, cosine and inverse
root contribute 2.5 u.  Together 4.3 u; times 1.4, since parts of a field that
changes sign cancel in the result: 6 u as the 2-norm over the listeners, worst
right-hand side.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def body():
    from neuralat_b200.bem import BEM_Solver
    from neuralat_b200.bem import meshes as M

    O.build()
    v, t = M.icosphere(5, 0.15)
    v = (v * [1.2, 0.8, 1.0]).astype(np.float32)
    return BEM_Solver(v, t.astype(np.int32)), v.astype(np.float64), t.astype(np.int32)


@pytest.mark.parametrize("points,rhs", [(20, 1), (33, 2), (20, 4), (30, 5), (128, 9), (129, 17), (4000, 33), (2625, 58)])
def test_listen_sums(body, points, rhs):
    import torch

    from neuralat_b200.bem import meshes as M

    s, v, t = body
    k = 4.0
    x = M.sphere_points(points, 0.5, seed=points).astype(np.float32)
    g, u = (M.smoothed_gaussian_field(len(v), t, rhs, seed=rhs + i).astype(np.complex64) for i in (0, 7))
    got = s.boundary2potential(k, *(torch.from_numpy(y).cuda() for y in (g, u, x))).cpu().numpy()
    some = np.linspace(0, points - 1, min(points, 40)).astype(int)
    ref = [O.potential_matrix(layer, v, t, x[some].astype(np.float64), np.float32(k)) @ f.astype(complex)
           for layer, f in (("single", g), ("double", u))]
    ref = ref[1] - ref[0]
    err = np.linalg.norm(got[some] - ref, axis=0) / np.linalg.norm(ref, axis=0)
    assert err.max() < 6 * 2.0 ** -24, err.max()
