"""The weight stream's bounded waits are for its own copies: a kernel in front of it that takes far longer than their bound is waited for.
The kernel is built with a bound of some microseconds (the library's is a fraction of a second) and stands behind a launch of 30 ms."""
import ctypes as C
import os
import shutil
import subprocess

import pytest
import torch

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "blok_b200", "csrc")


@pytest.mark.gpu
@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not on PATH")
def test_a_slow_launch_in_front(cuda, tmp_path):
    out = str(tmp_path / "slow_front.so")
    cmd = ["nvcc", "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
           "-DBLOK_SPIN_LIMIT=2000", "-I", CSRC, "-shared", "-o", out, os.path.join(HERE, "slow_front.cu")]
    cmd += [os.path.join(CSRC, n + ".cu") for n in ("wgemm_stream", "gemm_tma", "gemm_pair", "abi")]
    p = subprocess.run(cmd, capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stderr[-2000:]
    lib = C.CDLL(out)
    g = torch.Generator(device=cuda).manual_seed(1)
    R, K, T = 256, 1024, 8
    w, x = ((torch.randn((n, K), generator=g, device=cuda) / 32).bfloat16() for n in (R, T))
    to, y, err = torch.zeros_like(x), torch.zeros((T, R), device=cuda), torch.zeros(1, dtype=torch.int32, device=cuda)
    p = [C.c_void_p(t.data_ptr()) for t in (w, x, to, y)]
    for us in (0, 30000):
        y.zero_()
        assert lib.slow_front_product(*p, R, K, T, us, C.c_void_p(err.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        torch.cuda.synchronize()
        assert int(err) == 0, us
        torch.testing.assert_close(y.double(), x.double() @ w.double().T, rtol=0, atol=1e-4)  # 1,024 fp32 products of about 1e-3
