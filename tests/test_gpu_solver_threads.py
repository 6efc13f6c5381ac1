"""Solves with one right-hand side from several host threads, of sizes whose
launches need different shared memory: none may fail, whatever the order.

Tolerance: the solver's own bound on the FP64 residual of its FP64 solution,
rtol = 1e-6, plus 1e-6 for the complex64 solution (condition < 10).
"""
import concurrent.futures as cf

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def system(n):
    rng = np.random.default_rng(n)
    A = np.eye(n) + 0.3 / np.sqrt(2 * n) * (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))
    b = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    return torch.from_numpy(A.astype(np.complex64)).cuda(), torch.from_numpy(b.astype(np.complex64)).cuda()


def test_alternating_sizes():
    from neuralat_b200.bem.solver import gmres

    systems = [system(n) for n in (150, 1100, 150, 5000)]
    torch.cuda.synchronize()

    def run(i):
        worst = 0.0
        with torch.cuda.stream(torch.cuda.Stream()):
            for j in range(150):
                A, b = systems[(i + j) % 4]
                x = gmres(A, b, rtol=1e-6)
                if j >= 146:
                    A, b, x = (y.to(torch.complex128) for y in (A, b, x))
                    worst = max(worst, float((A @ x - b).norm() / b.norm()))
        return worst

    with cf.ThreadPoolExecutor(4) as ex:
        for r in ex.map(run, range(4)):
            assert r < 2e-6


def test_batches_of_uneven_meshes():
    from neuralat_b200.bem import meshes as M
    from neuralat_b200.bem.batch import BatchRunner

    meshes = [M.icosphere(s, 0.1) for s in (1, 2, 3, 4)]
    points = np.array([[0.5, 0.1, 0.0], [0.0, 0.4, 0.3]], np.float32)
    ks = [[10.0, 12.0, 14.0, 16.0] for _ in meshes]
    fields = [np.ones(len(v), np.complex64) for v, _ in meshes]
    with BatchRunner(memory_budget_bytes=1 << 30, rtol=1e-6) as runner:
        first = runner.run(meshes, ks, fields, points)
        for _ in range(15):
            again = runner.run(meshes, ks, fields, points)
            for p, q in zip(first.pressure, again.pressure):
                assert float((p - q).norm() / p.norm()) < 2e-5
