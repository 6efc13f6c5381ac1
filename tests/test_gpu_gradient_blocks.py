"""Vertex gradient of the listener pressures on meshes around the 32-triangle
blocks of the pair walk: fewer triangles than a block (20), two full blocks and
a half (80), two bodies with a short last block (100), against central
differences of the FP64 oracle.

Tolerance: 1e-3 relative to the largest gradient entry, the bar of the
differentiation workload (FP32 kernels, differences with a step of 1e-6).
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _mesh(name):
    from neuralat_b200.bem import meshes as M

    v0, t0 = M.icosphere(0, 0.1)
    v1, t1 = M.icosphere(1, 0.12)
    if name == "20":
        v, t = v0 * [1.1, 0.9, 1.0], t0
    elif name == "80":
        v, t = v1 * [1.1, 0.9, 1.2], t1
    else:
        v, t = np.concatenate([v1, v0 * 0.8 + [0.28, 0.02, 0.0]]), np.concatenate([t1, t0 + len(v1)])
    return v.astype(np.float32), t.astype(np.int32)


@pytest.mark.parametrize("name", ["20", "80", "100"])
def test_gradient_blocks(name):
    import torch

    from neuralat_b200.bem import meshes as M
    from neuralat_b200.bem.adjoint import listener_pressure

    O.build()
    v, t = _mesh(name)
    rng = np.random.default_rng(len(t))
    g = (rng.standard_normal(len(v)) + 1j * rng.standard_normal(len(v))).astype(np.complex64)
    pts, k = M.sphere_points(19, 0.6, seed=1).astype(np.float32), 9.0

    def loss(x):
        V, K = (O.boundary_matrix(layer, x, t, k) for layer in ("single", "double"))
        u = np.linalg.solve(0.5 * O.identity_matrix(x, t) - K, -V @ g.astype(complex))
        return (np.abs(O.boundary2potential(x, t, k, g.astype(complex), u, pts.astype(float))) ** 2).sum()

    vt = torch.from_numpy(v).cuda().requires_grad_(True)
    p = listener_pressure(vt, torch.from_numpy(g).cuda(), torch.from_numpy(t).cuda(), torch.from_numpy(pts).cuda(), k)
    (gx,) = torch.autograd.grad((p.real ** 2 + p.imag ** 2).sum(), vt)
    gx, h = gx.double().cpu().numpy(), 1e-6
    for i in range(0, len(v), max(1, len(v) // 5)):
        for c in range(3):
            a, b = v.astype(float), v.astype(float)
            a[i, c] += h
            b[i, c] -= h
            assert abs((loss(a) - loss(b)) / (2 * h) - gx[i, c]) < 1e-3 * np.abs(gx).max()
