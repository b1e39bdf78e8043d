"""Two host threads with handles, buffers and streams of their own, over launches of the same kernels that want different amounts of
shared memory: a function's limit is the program's, so neither may lower it under the other."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_launches_of_different_shared_memory(cuda):
    from blok_b200 import lib
    g = torch.Generator(device=cuda).manual_seed(1)
    hidden, ffn = 512, 512
    w = [(torch.randn(s, generator=g, device=cuda) * 0.03).bfloat16() for s in ((ffn, hidden), (ffn, hidden), (hidden, ffn))]
    xs = {T: torch.randn((T, hidden), generator=g, device=cuda).bfloat16() for T in (9, 48)}  # 108 and 88 KB of the weight stream
    want = {T: lib.bf16_mlp(*w, x) for T, x in xs.items()}
    torch.cuda.synchronize()
    errors, last = [], {}

    def work(T):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(4000):
                    last[T] = lib.bf16_mlp(*w, xs[T])
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(T,)) for T in xs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for T in xs:
        assert torch.equal(last[T], want[T]), T
