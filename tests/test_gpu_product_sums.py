"""Complex product with more than eight right-hand sides on either side of the
size from which it is tiled (8193 unknowns): tiles of 16 and 64 right-hand sides
and remainders, odd sizes, an A that is not 16-byte aligned; a single layer's
kernel times smooth fields, against complex128.

Tolerance, with u = 2^-24: the result's own rounding 0.4 u, runs of at most 32
terms 0.4 u sqrt(32 / 3) = 1.3 u of a run, independent over the runs (0.1 u of
the result, times 4 for fields whose parts cancel), and at most 10 additions of
1024 columns each, 0.4 u sqrt(10 / 3) = 0.7 u: 0.9 u as the 2-norm; 1.5 u leaves
room for the distribution of the roundings.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(2500, 16), (8192, 9), (8193, 9), (8194, 16), (8195, 17), (8200, 48), (8200, 49),
                                 (8201, 65), (8256, 64), (8256, 130), (10242, 64)])
@pytest.mark.parametrize("shift", [0, 1])
def test_smooth_product(n, m, shift):
    from neuralat_b200.bem.solver import cmatmul

    # points along a spiral on a sphere: neighbours in number lie together, as the vertices of a mesh do
    z = 1.0 - (2.0 * torch.arange(n, device="cuda", dtype=torch.float64) + 1.0) / n
    turn, r = (torch.pi * n) ** 0.5 * torch.arccos(z), (1.0 - z * z).sqrt()
    x = 0.15 * torch.stack([r * torch.cos(turn), r * torch.sin(turn), z], 1)
    k = 4.0
    A = torch.empty(n * n + 1, dtype=torch.complex64, device="cuda")[shift:shift + n * n].view(n, n)
    s = torch.arange(1, m + 1, device="cuda", dtype=torch.float64)
    X = torch.exp(1j * (3.0 * x @ x.new_tensor([7.0, 3.0, 5.0]))[:, None] * (1 + s / m)).to(torch.complex64)
    ref = torch.empty(n, m, dtype=torch.complex128, device="cuda")
    for r in range(0, n, 2048):
        d = (x[r:r + 2048, None] - x[None]).norm(dim=2).clamp_min(0.15 / n ** 0.5)
        A[r:r + 2048] = (torch.exp(1j * k * d) / d).to(torch.complex64)
        ref[r:r + 2048] = A[r:r + 2048].to(torch.complex128) @ X.to(torch.complex128)
    err = (cmatmul(A, X) - ref).norm(dim=0) / ref.norm(dim=0)
    assert float(err.max()) < 1.5 * 2.0 ** -24, float(err.max())
