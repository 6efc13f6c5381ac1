"""One right-hand side in one launch (whole GMRES solve): sizes around the 15
unknowns of a CTA and the rows of a sweep, odd sizes, restarts, a start
vector, the iteration cap, a breakdown (b an eigenvector), zero and non-finite
right-hand sides; against the FP64 residual of the returned solution and the
cluster kernel's iteration count.

Tolerances: the reported status promises the FP64 residual of the FP64 solution
<= rtol |b|; the returned complex64 solution adds |A| |x| 2^-24 to it, below
1e-6 |b| for these matrices (condition < 10), hence rtol + 1e-6.
"""
import numpy as np
import pytest

from neuralat_b200 import _lib as L

pytestmark = pytest.mark.gpu


def system(n, seed=0):
    rng = np.random.default_rng(1000 * seed + n)
    A = np.eye(n) + 0.3 / np.sqrt(2 * n) * (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))
    b = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    return A.astype(np.complex64), b.astype(np.complex64)


def solve(A, b, **kw):
    import torch

    from neuralat_b200.bem.solver import gmres

    info = {}
    x = gmres(torch.from_numpy(A).cuda(), torch.from_numpy(b).cuda(), info=info, **kw)
    x = x.cpu().numpy().astype(complex)
    with np.errstate(invalid="ignore"):
        res = np.linalg.norm(A.astype(complex) @ x - b) / max(np.linalg.norm(b), 1e-300)
    return x, res, info


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 16, 17, 31, 33, 127, 480, 481, 1000, 2220, 2221, 2367, 2369, 3001, 4441, 6661, 7400, 7401])
def test_sizes(n):
    A, b = system(n)
    for precision in ("fp32", "fp16x3"):
        _, res, info = solve(A, b, rtol=1e-6, precision=precision)
        assert info["status"] == L.BEM_OK and res < 2e-6, (precision, res, info)
    L.check(L.lib().bem_set_tuning(L.TUNE_ARNOLDI_MODE, 1))
    try:
        _, _, ref = solve(A, b, rtol=1e-6)
    finally:
        L.check(L.lib().bem_set_tuning(L.TUNE_ARNOLDI_MODE, 0))
    assert abs(info["iterations"] - ref["iterations"]) <= 1 and info["refinements"] == ref["refinements"]


@pytest.mark.parametrize("restart", [1, 2, 3, 5, 255])
def test_restarts(restart):
    A, b = system(300, 1)
    _, res, info = solve(A, b, rtol=1e-6, restart=restart, max_refine=4)
    assert info["status"] == L.BEM_OK and res < 2e-6, (res, info)
    assert info["iterations"] >= (restart < 5) * 8


def test_start_vector_cap_and_breakdown():
    import torch

    A, b = system(257, 2)
    x, _, full = solve(A, b, rtol=1e-6)
    x0 = torch.from_numpy(x.astype(np.complex64)).cuda()
    _, res, info = solve(A, b, x=x0, rtol=1e-6)
    assert info["status"] == L.BEM_OK and info["iterations"] == 0 and res < 2e-6
    _, res, info = solve(A, b, x=0.9 * x0, rtol=1e-6)
    assert info["status"] == L.BEM_OK and 0 < info["iterations"] < full["iterations"] and res < 2e-6
    _, res, info = solve(A, b, rtol=1e-6, max_iters=3)
    assert info["status"] == L.BEM_ERR_NOT_CONVERGED and info["iterations"] == 3 and res < 0.5
    D = np.diag(np.linspace(1, 2, 40)).astype(np.complex64)  # one step ends the Krylov space
    _, res, info = solve(D, D[3] + 0, rtol=1e-6)
    assert info["status"] == L.BEM_OK and info["iterations"] == 1 and res < 2e-6


def test_zero_and_nonfinite():
    A, b = system(100, 3)
    x, _, info = solve(A, 0 * b, rtol=1e-6)
    assert info["status"] == L.BEM_OK and info["iterations"] == 0 and not x.any()
    b[5] = np.nan
    with pytest.raises(L.BEMError) as e:
        solve(A, b, rtol=1e-6)
    assert e.value.status == L.BEM_ERR_NONFINITE


def test_solves_side_by_side():
    """Cooperative launches of several host threads and streams."""
    import concurrent.futures as cf

    import torch

    systems = [system(n, 4) for n in (150, 400, 700, 1100)]

    def run(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            return [solve(*systems[i], rtol=1e-6)[1] for _ in range(5)]

    with cf.ThreadPoolExecutor(4) as ex:
        for r in ex.map(run, range(4)):
            assert max(r) < 2e-6
