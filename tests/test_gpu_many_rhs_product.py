"""Complex product with more than eight right-hand sides at the edges of its
tiles: 16, 32 and 64 right-hand sides and remainders, rows around multiples of
64 and 128, the smallest size it takes, odd column counts (8-byte copies) and an
A that is not 16-byte aligned, against NumPy in complex128.

Tolerance: an entry is a sum of at most 32 + 64 + 8 roundings in a row, errors
that add like a random walk: sqrt(104) * 2^-24 = 6e-7 relative to the norm;
2e-6 allows for the worst column.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 2e-6


@pytest.mark.parametrize("n,m", [(1, 9), (512, 64), (513, 9), (514, 64), (575, 16), (576, 17), (577, 33), (640, 32),
                                 (641, 24), (642, 65), (1000, 96), (1001, 70), (1025, 97), (2500, 9), (2500, 130)])
@pytest.mark.parametrize("shift", [0, 1])
def test_product(n, m, shift):
    import torch

    from neuralat_b200.bem.solver import cmatmul

    rng = np.random.default_rng(n * 1000 + m)
    a, x = ((rng.standard_normal((n, c)) + 1j * rng.standard_normal((n, c))).astype(np.complex64) for c in (n, m))
    A = torch.empty(n * n + 1, dtype=torch.complex64, device="cuda")[shift:shift + n * n].view(n, n)
    A.copy_(torch.from_numpy(a))
    y = cmatmul(A, torch.from_numpy(x).cuda()).cpu().numpy()
    ref = a.astype(complex) @ x.astype(complex)
    err = np.linalg.norm(y - ref, axis=0) / np.linalg.norm(ref, axis=0)
    assert err.max() < TOL, err.max()
