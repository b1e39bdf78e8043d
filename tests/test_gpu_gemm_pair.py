"""bf16 products over more than 128 rows, which pairs of CTAs take from 512 columns on: against 64 bits at the edges of their tiles (256 rows
of x by 128 or 256 weight rows, 64-column steps) and on both sides of the lines to the one-CTA kernel."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,R,K", [(128, 256, 128), (129, 4, 8), (129, 256, 64), (255, 260, 72), (256, 128, 1000), (257, 36, 520), (513, 516, 200),
                                   (300, 18944, 64), (1000, 2048, 8192), (2047, 8512, 2048)])
def test_plain(cuda, T, R, K):
    from blok_b200 import lib
    g = torch.Generator(device=cuda).manual_seed(T)
    x, w = ((torch.randn(s, generator=g, device=cuda) / K ** 0.25).bfloat16() for s in ((T, K), (R, K)))
    want = x.double() @ w.double().T
    # fp32 sums of up to 8,192 products; with one rounding to bf16 of the squared result 2^-9 / sqrt(3) of it, rms
    for relu2, f32, ref, bar in ((False, True, want, 3e-5), (True, True, want.clamp(min=0) ** 2, 6e-5), (False, False, want, 3e-3),
                                 (True, False, want.clamp(min=0) ** 2, 3e-3)):
        got = lib.gemm_bf16(x, w, relu2, f32)
        assert float((got.double() - ref).norm() / ref.norm()) < bar, (relu2, f32)
        assert torch.equal(got, lib.gemm_bf16(x, w, relu2, f32))


@pytest.mark.parametrize("T,R,K", [(128, 128, 64), (129, 4, 64), (256, 132, 264), (300, 200, 1000), (1025, 8192, 512)])
def test_gated(cuda, T, R, K):
    from blok_b200 import lib
    g = torch.Generator(device=cuda).manual_seed(R)
    x, w = ((torch.randn(s, generator=g, device=cuda) / K ** 0.25).bfloat16() for s in ((T, K), (2 * R, K)))
    gate, up = x.double() @ w[:R].double().T, x.double() @ w[R:].double().T
    want = gate * torch.sigmoid(gate) * up
    got = lib.gemm_swiglu(x, w)
    assert float((got.double() - want).norm() / want.norm()) < 3e-3


# from 512 columns on pairs take a product, with exceptions below 2,048 columns where most of a half tile is empty: every edge of a pair's
# tile, and both sides of the lines
@pytest.mark.parametrize("T,R,K", [(129, 4, 512), (129, 256, 520), (255, 260, 584), (256, 128, 1000), (257, 36, 520), (513, 516, 712), (300, 18944, 512),
                                   (384, 8192, 512), (385, 8192, 512), (513, 4096, 2040), (513, 4096, 2048), (640, 4096, 1024), (641, 4096, 1024),
                                   (300, 2048, 504), (300, 2048, 512)])
def test_lines_between_the_kernels(cuda, T, R, K):
    test_plain(cuda, T, R, K)


@pytest.mark.parametrize("T,R,K", [(128, 128, 512), (129, 4, 512), (256, 132, 584), (300, 200, 1000), (300, 4736, 512), (300, 4864, 512), (385, 4864, 520),
                                   (1025, 8192, 504)])
def test_gated_lines_between_the_kernels(cuda, T, R, K):
    test_gated(cuda, T, R, K)
