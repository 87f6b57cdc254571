"""What the library's host code launches, without a GPU: the objects of the
library run over a fake CUDA runtime (tests/fake_cuda.py) that refuses what a
device would refuse and logs every launch."""
import ctypes as C
import shutil

import numpy as np
import pytest

import fake_cuda as F

M32, M64 = "cuda_multigrid32f_gpu", "cuda_multigrid64_gpu"


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None or shutil.which("nvcc") is None:
        pytest.skip("no compiler")
    return F.Fake(str(tmp_path_factory.mktemp("fake") / "libpsum_fake.so"))


@pytest.fixture
def fake(lib):
    lib.reset()
    yield lib
    lib.reset()


@pytest.mark.parametrize("kind,nodes,options,blocks", [
    (M64, (64, 64), "", 1), (M32, (96, 96), "", 16), (M32, (400, 410), "", "sms"), (M64, (48, 48, 48), "", "sms"),
    (M32, (32, 32, 32), "tma_min_rows 1000", None), (M64, (32, 32, 32), "tma_min_rows 1000", None)])
def test_a_second_device_of_the_process(fake, kind, nodes, options, blocks):
    """Kernel attributes and SM counts belong to a device: what ran on the first runs on the second, with its SMs."""
    for device, sms in ((0, 148), (1, 100)):
        fake.lib.fake_device(device, sms)
        s = F.Solver(fake, kind, nodes, options)
        fake.lib.fake_clear_log()
        s.check(s.solve_async(fake.stream()))
        if blocks:
            (k,) = fake.kernels("k_mg_persist")
            assert (k.device, k.grid) == (device, sms if blocks == "sms" else blocks)
        else:
            assert fake.kernels("k_level_op_tma")
        s.close()
