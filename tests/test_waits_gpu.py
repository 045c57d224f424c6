"""The bounded wait: whoever shares a warp or a named barrier with a thread that gives up leaves with it."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_bounded_wait_gives_one_answer_to_the_warp(cuda):
    torch = cuda
    src = os.path.join(ROOT, "tests", "wait_check.cu")
    lib = os.path.join(ROOT, "tests", "build", "libwait_check.so")
    os.makedirs(os.path.dirname(lib), exist_ok=True)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-o", lib, src])
    L = C.CDLL(lib)
    L.wait_check.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.full((128,), -1, dtype=torch.int32, device="cuda")
    assert L.wait_check(status.data_ptr(), out.data_ptr(), None) == 0
    torch.cuda.synchronize()
    o = out.cpu().numpy()
    assert int(status) == 32
    assert (o[:32] == 0).all(), "the lanes of a warp have to agree when one of them gives up"
    assert (o[32:64] == 1).all()
    assert (o[64:] == 1).all()
