"""GPU: a bounded wait that runs out is reported in the caller's status word, whichever warp it belongs to and however
long before it the reporting thread was done."""
import ctypes as C
import os
import subprocess
import time

import pytest
import torch

from evoformer_triton_b200 import build

pytestmark = pytest.mark.gpu

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "wait_limit.cu")


@pytest.fixture(scope="module")
def wait_kernel(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("wait") / "wait_limit.so")
    subprocess.check_call([build._nvcc(), *build.NVCC_FLAGS, "-shared", "-o", so, SRC])
    fn = C.CDLL(so).run_wait_kernel
    fn.argtypes = [C.c_int, C.c_int, C.c_void_p]
    return fn


@pytest.mark.parametrize("warp", [0, 1, 3])
def test_wait_that_runs_out_is_reported(wait_kernel, warp):
    status = torch.zeros(1, dtype=torch.int32, device="cuda:0")
    torch.cuda.synchronize()
    assert wait_kernel(warp, 1, status.data_ptr()) == 0
    torch.cuda.synchronize()
    assert status.item() == 0
    t0 = time.monotonic()
    assert wait_kernel(warp, 0, status.data_ptr()) == 0
    torch.cuda.synchronize()
    assert status.item() == 2  # the code of the wait that ran out, not of those that then fell through
    assert 0.5 < time.monotonic() - t0 < 4  # (2e9 cycles, once)
    torch.ones(4, device="cuda:0").sum().item()  # the context goes on
