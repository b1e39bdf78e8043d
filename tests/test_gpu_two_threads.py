"""Two host threads with handles, buffers and streams of their own, over launches of the same kernels that want different amounts of
shared memory: a function's limit is the program's, so neither may lower it under the other."""
import ctypes as C
import os
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu


class MlpCall(C.Structure):
    _fields_ = [(n, C.c_void_p) for n in ("gate", "up", "down", "x", "y")] + [(n, C.c_int) for n in ("hidden", "ffn", "T")] + [
        ("ws", C.c_void_p), ("ws_bytes", C.c_size_t), ("stream", C.c_void_p)]


def test_launches_of_different_shared_memory(cuda, tmp_path):
    from blok_b200 import lib
    so = str(tmp_path / "two_threads.so")
    source = os.path.join(os.path.dirname(os.path.abspath(__file__)), "two_threads.cpp")
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-pthread", source, "-o", so], check=True)
    native, library = C.CDLL(so), lib.load()
    g = torch.Generator(device=cuda).manual_seed(1)
    hidden, ffn = 512, 512
    w = [(torch.randn(s, generator=g, device=cuda) * 0.03).bfloat16() for s in ((ffn, hidden), (ffn, hidden), (hidden, ffn))]
    calls, want, keep = [], [], []
    for T in (9, 48):  # 108 and 88 KB of the weight stream
        x = torch.randn((T, hidden), generator=g, device=cuda).bfloat16()
        y, ws, stream = torch.empty_like(x), torch.empty(1 << 20, device=cuda, dtype=torch.uint8), torch.cuda.Stream()
        want.append(lib.bf16_mlp(*w, x))
        keep.append((x, y, ws, stream))
        calls.append(MlpCall(*(t.data_ptr() for t in (*w, x, y)), hidden, ffn, T, ws.data_ptr(), ws.numel(), stream.cuda_stream))
    torch.cuda.synchronize()
    failed = native.two_threads(C.cast(library.blok_bf16_mlp, C.c_void_p), C.cast(library.blok_last_error, C.c_void_p), C.byref(calls[0]), C.byref(calls[1]), 10000)
    torch.cuda.synchronize()
    assert failed == 0
    for (x, y, _, _), z in zip(keep, want):
        assert torch.equal(y, z)
