"""Strip walk of the regular pairs (V/K and Burton-Miller) at the edges of its
32-triangle blocks: meshes smaller than a block, one triangle more or less
than a block, blocks of disjoint triangles (96 vertices), vertices with more
corners in one block than a lane keeps in registers, against the FP64 oracle.

Tolerance: 1e-5 relative Frobenius norm, the bar of every assembled matrix.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-5


def patch(count, seed):
    """The first `count` triangles of a bumpy grid, vertices renumbered."""
    n = 9
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    v = np.stack([0.05 * i, 0.05 * j, 0.01 * np.sin(1.3 * i + 0.7 * j)], -1).reshape(-1, 3)
    t = []
    for a in range(n - 1):
        for b in range(n - 1):
            p = a * n + b
            t += [(p, p + n, p + 1), (p + 1, p + n, p + n + 1)]
    t = np.array(t)[:count]
    used, t = np.unique(t, return_inverse=True)
    return v[used], t.reshape(-1, 3)


def fan(count):
    """A cone of `count` triangles around one vertex."""
    a = 2 * np.pi * np.arange(count) / count
    v = np.concatenate([[[0.0, 0.0, 0.05]], np.stack([0.2 * np.cos(a), 0.2 * np.sin(a), 0 * a], 1)])
    k = np.arange(count)
    return v, np.stack([0 * k, 1 + k, 1 + (k + 1) % count], 1)


def soup(count, seed):
    """Disjoint triangles."""
    rng = np.random.default_rng(seed)
    c = rng.uniform(-0.3, 0.3, (count, 1, 3))
    v = (c + rng.uniform(-0.02, 0.02, (count, 3, 3))).reshape(-1, 3)
    return v, np.arange(3 * count).reshape(-1, 3)


MESHES = {
    "one triangle": lambda: patch(1, 0), "two triangles": lambda: patch(2, 0), "31": lambda: patch(31, 1),
    "32": lambda: patch(32, 2), "33": lambda: patch(33, 3), "65": lambda: patch(65, 4), "fan 40": lambda: fan(40),
    "disjoint 33": lambda: soup(33, 5),
}


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("name", list(MESHES))
def test_block_edges(name):
    import torch

    from neuralat_b200.bem import BEM_Solver
    from neuralat_b200.bem.batch import assemble_batch, assemble_batch_bm

    O.build()
    v, t = MESHES[name]()
    v, t, k = v.astype(np.float32), t.astype(np.int32), 21.7
    s = BEM_Solver(torch.from_numpy(v).cuda(), torch.from_numpy(t).cuda())
    v64, M = v.astype(np.float64), O.identity_matrix(v.astype(np.float64), t)
    refs = (O.boundary_matrix("single", v64, t, k), 0.5 * M - O.boundary_matrix("double", v64, t, k))
    for pair in (s.assemble_vk(k), assemble_batch([s], [k])[0]):  # one problem, and the same through the queue
        assert all(rel(x.cpu().numpy(), y) < TOL for x, y in zip(pair, refs))
    for approx, order in ((True, "_approx"), (False, "")):
        refs = (O.boundary_matrix("bm_lhs", v64, t, k, order) + 0.5 * M,
                O.boundary_matrix("bm_rhs", v64, t, k, order) - 0.5j / k * M)
        for pair in (s.assemble_bm(k, approx=approx), assemble_batch_bm([s], [k], approx=approx)[0]):
            assert all(rel(x.cpu().numpy(), y) < TOL for x, y in zip(pair, refs))
    for layer in ("hypersingular", "bm_lhs"):  # the sorted records' curls in the general kernel
        got = s.assemble_boundary_matrix(k, layer, approx=True).cpu().numpy()
        assert rel(got, O.boundary_matrix(layer, v64, t, k, "_approx")) < TOL


def sheet(count):
    """The first `count` triangles of a long bumpy sheet."""
    n, m = 60, 56
    i, j = np.meshgrid(np.arange(n), np.arange(m), indexing="ij")
    v = np.stack([0.01 * i, 0.01 * j, 0.01 * np.sin(0.3 * i + 0.2 * j)], -1).reshape(-1, 3)
    a = (np.arange(n - 1)[:, None] * m + np.arange(m - 1)).reshape(-1)
    t = np.stack([a, a + m, a + 1, a + 1, a + m, a + m + 1], 1).reshape(-1, 3)[:count]
    used, t = np.unique(t, return_inverse=True)
    return v[used], t.reshape(-1, 3)


@pytest.mark.parametrize("count", [3072, 3073, 4321, 6300])
def test_rounds(count):
    """Items in one round, in two (97 blocks) and more, and the Burton-Miller
    panels with an uneven last one: one problem against the queue's items.
    Tolerance: both within 1e-5 of the exact matrices, so within 2e-5."""
    from neuralat_b200.bem import BEM_Solver
    from neuralat_b200.bem.batch import assemble_batch, assemble_batch_bm

    v, t = sheet(count)
    s, k = BEM_Solver(v.astype(np.float32), t.astype(np.int32)), 17.0
    pairs = [(s.assemble_vk(k), assemble_batch([s], [k])[0])]
    pairs += [(s.assemble_bm(k, approx=a), assemble_batch_bm([s], [k], approx=a)[0]) for a in (True, False)]
    for one, many in pairs:
        for x, y in zip(one, many):
            assert float((x - y).norm() / y.norm()) < 2 * TOL
