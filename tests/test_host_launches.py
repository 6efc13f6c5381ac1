"""What the host code asks of the CUDA runtime, on a runtime that runs no
kernel and refuses what the real one refuses (fake_cudart.cpp)."""
import pytest

from fake_cuda import FakeCuda
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
