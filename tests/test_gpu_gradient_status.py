"""A bounded wait of the vertex gradient's kernels that expired: the status word
it raises on the geometry ends the backward pass with an error.  The word is
raised by the test (int32 number 7 of the geometry's header)."""
import numpy as np
import pytest
import torch

from neuralat_b200 import _lib as L

pytestmark = pytest.mark.gpu


def test_backward_reads_the_status_word():
    from neuralat_b200.bem import meshes as M
    from neuralat_b200.bem.adjoint import listener_pressure

    v, t = M.icosphere(1, 0.1)
    v = torch.from_numpy(v.astype(np.float32)).cuda().requires_grad_(True)
    t = torch.from_numpy(t.astype(np.int32)).cuda()
    g = torch.ones(len(v), dtype=torch.complex64, device="cuda", requires_grad=True)
    p = listener_pressure(v, g, t, torch.tensor([[0.4, 0.1, 0.2]], device="cuda"), 9.0)
    loss = (p.abs() ** 2).sum()
    geometry = p.grad_fn.solver.geometry
    loss.backward(retain_graph=True)
    first = v.grad.clone()
    geometry.buffer.view(torch.int32)[7] = 1
    with pytest.raises(L.BEMError) as e:
        loss.backward(retain_graph=True)
    assert e.value.status == L.BEM_ERR_CUDA
    v.grad = None
    loss.backward()  # the word was cleared with the report
    assert float((v.grad - first).norm() / first.norm()) < 1e-5
