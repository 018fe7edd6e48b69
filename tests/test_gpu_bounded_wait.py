"""GPU: a bounded wait of the grouped GEMM that runs out does so soon. How long a try suspends its thread is the hardware's choice, so it is
measured: a thousand tries of a barrier that nobody arrives at. 2.0 us a try was seen (the limit of tries then is half a second); up to
8 us, two seconds a wait, is what the launches around it can bear."""
import ctypes
import os
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
LIB = os.path.join(HERE, "_build", "wait_kernel.so")


def test_a_wait_ends_in_time():
    if not os.path.isfile(LIB):
        os.makedirs(os.path.dirname(LIB), exist_ok=True)
        subprocess.run(["nvcc", "-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-gencode", "arch=compute_100a,code=sm_100a",
                        os.path.join(HERE, "wait_kernel.cu"), "-o", LIB], check=True)
    lib = ctypes.CDLL(LIB)
    lib.run_wait.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
    lib.wait_limit.restype = ctypes.c_uint
    out = torch.zeros(2, dtype=torch.int64, device="cuda")
    assert lib.run_wait(1000, out.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    ns, passed = out.tolist()
    assert passed == 0 and ns < 1000 * 8000
    assert ns / 1000 * lib.wait_limit() < 2.1e9
