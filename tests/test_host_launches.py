"""What the host code asks of the CUDA runtime, on a runtime that runs no
kernel and refuses what the real one refuses (fake_cudart.cpp)."""
import ctypes

import numpy as np
import pytest

from fake_cuda import FakeCuda, array, at
from neuralat_b200 import _lib as L


@pytest.fixture(scope="module")
def linked(tmp_path_factory):
    return FakeCuda(tmp_path_factory.mktemp("host"))


@pytest.fixture
def cuda(linked):
    linked.on = None
    linked.launched.clear()
    linked.refused.clear()
    linked.device(0)
    yield linked
    linked.on = None
    linked.device(0)


@pytest.mark.parametrize("large,small,restart", [(5000, 150, 200), (1100, 150, 200), (2487, 2486, 255), (150, 150, 3)])
def test_solves_of_different_sizes_at_once(cuda, large, small, restart):
    """A smaller solve of another thread that runs wholly between a solve's
    look at the device and its launch leaves it the shared memory it asks for."""
    inner = []

    def on(event, name, pointer, value):
        if event == "occupancy" and "gm_single_kernel" in name and not inner:
            inner.append(None)
            inner[0] = cuda.solve(small, restart=1)

    cuda.on = on
    assert cuda.solve(large, restart=restart) == L.BEM_OK
    assert inner == [L.BEM_OK] and not cuda.refused
    assert len([k for k in cuda.launched if "gm_single_kernel" in k]) == 2


# ---- every entry point with kernels above the default shared memory, by name ----
def one_problem(kind, g, first, second):
    p = kind()
    p.geom, p.k = at(g), 1.0
    for (name, _), value in zip(kind._fields_[2:], (first, second)):
        setattr(p, name, at(value))
    return p


def mesh_calls(cuda):
    from neuralat_b200.bem import meshes as M

    lib = cuda.lib
    v, t = M.icosphere(2, 0.1)
    n = len(v)
    g = cuda.geometry(v, t)
    X, Y, f, u, p, out = array((n, n)), array((n, n)), array((n, 64)), array((n, 64)), array((300, 64)), array((300, 64))
    x, grad = array((300, 3), np.float32), array((n, 3), np.float64)
    ws = array(1 << 20, np.uint8)
    for a, b in ((X, Y), (X, None), (None, Y)):
        yield "vk", lib.bem_boundary_matrices_vk(at(g), 1.0, at(a) if a is not None else None,
                                                 at(b) if b is not None else None, 0.5, -1.0, None)
    for order in range(3):
        yield "bm", lib.bem_boundary_matrices_bm(at(g), order, 1.0, at(X), at(Y), None)
        one = one_problem(L.BmProblem, g, X, Y)
        yield "bm batch", lib.bem_batch_matrices_bm(ctypes.byref(one), 1, order, at(ws), ws.nbytes, None)
        for layer in range(6):
            yield "matrix", lib.bem_boundary_matrix(at(g), layer, order, 1.0, None, None, at(X), None)
    one = one_problem(L.BatchProblem, g, X, Y)
    yield "vk batch", lib.bem_batch_matrices_vk(ctypes.byref(one), 1, 0.5, -1.0, at(ws), ws.nbytes, None)
    for m in (1, 2, 4, 8, 16, 32, 64):
        yield "listen", lib.bem_boundary2potential_noalloc(at(g), at(x), 300, 1.0, at(f), at(u), m, at(out), None)
    yield "gradient", lib.bem_vertex_gradient(at(g), 1.0, at(f), at(f), at(u), at(x), 300, at(p), at(grad), None)


def linear_calls(cuda):
    lib = cuda.lib
    for n, m in ((600, 1), (600, 2), (600, 4), (600, 8), (8194, 9), (8194, 64), (8193, 9), (8193, 64)):
        A, X, Y = array((n, n)), array((n, m)), array((n, m))
        yield "product", lib.bem_cmatmul(at(A), n, at(X), m, at(Y), None)
    n = 200
    for precision in (L.PREC_BF16X3, L.PREC_BF16, L.PREC_FP16X3):
        for m in (4, 16, 32, 64, 128):
            A, X, Y = array((n, n)), array((n, m)), array((n, m))
            ws = array(int(lib.bem_tc_operator_bytes(n, m, precision)), np.uint8)
            yield "split", lib.bem_tc_operator_prepare(at(A), n, precision, at(ws), ws.nbytes, None)
            yield "tensor product", lib.bem_tc_matmul(at(ws), ws.nbytes, n, precision, at(X), m, at(Y), None)
    yield "one side", cuda.solve(2487)
    for m in (4, 8, 16, 40):
        yield "residual", cuda.solve(600, m, use_x0=1)
    # past the first test of convergence: |b| and |r| read as 1
    cuda.on = lambda event, name, pointer, value: (ctypes.memset(pointer, 0x3f, value) and 0
                                                   if event == "copy" and name == "to host" and value == 8 * m else 0)
    for mode in range(4):
        L.check(lib.bem_set_tuning(L.TUNE_ARNOLDI_MODE, mode))
        for m in (2, 4, 8, 16, 40):
            yield "steps", cuda.solve(600, m, restart=3) in (L.BEM_OK, L.BEM_ERR_NOT_CONVERGED) and L.BEM_OK
    L.check(lib.bem_set_tuning(L.TUNE_ARNOLDI_MODE, 0))
    cuda.on = None


@pytest.mark.parametrize("calls", [mesh_calls, linear_calls])
def test_second_device(cuda, calls):
    """What a kernel needs before its first launch is done on each device."""
    for device in (0, 1, 70):
        cuda.device(device)
        for what, status in calls(cuda):
            assert status == L.BEM_OK and not cuda.refused, (device, what, status, cuda.refused)
        large = {k for k in cuda.launched}
        cuda.launched.clear()
    assert any("strip_vk" in k for k in large) or any("cgemm" in k for k in large)


@pytest.mark.parametrize("event", ["launch", "copy", "occupancy"])
def test_a_reported_error_is_gone(cuda, event):
    """An error of the runtime ends the call that met it and no later one."""
    A, X, Y = array((600, 600)), array((600, 8)), array((600, 8))
    calls = [lambda: cuda.solve(600), lambda: cuda.solve(600, 8, use_x0=1),
             lambda: cuda.lib.bem_cmatmul(at(A), 600, at(X), 8, at(Y), None)]
    for first in calls:
        failed = []

        def on(name, kernel, pointer, value):
            if name == event and not failed:
                failed.append(kernel)
                return 1  # cudaErrorInvalidValue
            return 0

        cuda.on = on
        status = first()
        cuda.on = None
        assert status in (L.BEM_OK, L.BEM_ERR_CUDA)  # where there is another way, it is taken
        for call in calls:
            assert call() == L.BEM_OK, failed


@pytest.mark.parametrize("blocks", [1, 3, 4, 100, (1 << 31) - 1])
def test_chunk_knob_means_blocks(cuda, blocks):
    """The chunk knob counts 32-triangle trial blocks in every V and K assembly:
    chunk is argument 6 of the one-operator kernel, in 16-triangle tiles, and
    number 2 (behind two 64-bit counts) of the strip kernel's items, in steps of a
    triangle."""
    from neuralat_b200.bem import meshes as M

    v, t = M.icosphere(3, 0.1)
    g, X, Y = cuda.geometry(v, t), array((len(v), len(v))), array((len(v), len(v)))
    seen = {}

    def on(event, name, pointer, value):
        if event == "launch" and "regular" in name:
            argument = ctypes.cast(pointer, ctypes.POINTER(ctypes.POINTER(ctypes.c_int)))[6]
            seen["strip" if "strip" in name else "tiles"] = argument[4] if "strip" in name else 16 * argument[0]
        return 0

    L.check(cuda.lib.bem_set_tuning(L.TUNE_ASSEMBLY_CHUNK, blocks))
    try:
        cuda.on = on
        for a, b in ((at(X), at(Y)), (at(X), None), (None, at(Y))):
            assert cuda.lib.bem_boundary_matrices_vk(at(g), 1.0, a, b, 0.5, -1.0, None) == L.BEM_OK
            if len(seen) == 2:
                assert min(seen["strip"], len(t)) == min(seen["tiles"], len(t)) == min(32 * blocks, len(t))
                del seen["tiles"]
        assert "strip" in seen
    finally:
        cuda.on = None
        L.check(cuda.lib.bem_set_tuning(L.TUNE_ASSEMBLY_CHUNK, 0))
