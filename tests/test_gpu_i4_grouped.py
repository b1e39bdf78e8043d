"""The batched layer's products on tcgen05 at the edges of their tiles (csrc/wgemm_tc.cu, csrc/gemm_tma.cu), and the INT4
dequantisation on the CPU."""
import numpy as np
import pytest
import torch

import util


def _bf16(a):
    """Round to nearest even to 8 significant bits (normal numbers)."""
    m, e = np.frexp(np.asarray(a, dtype=np.float64))
    return np.ldexp(np.rint(m * 256) / 256, e)


def test_dequantisation_by_one_rounding():
    """fma(n 2^-129, s 2^100, -s 2^-26) and fma(n 2^-133, s 2^104, -s 2^-26), rounded once, are 2^-29 bf16(q s) for every nibble
    and every scale mantissa, over the exponents the kernel claims; the bit patterns are the numbers the kernel takes them for."""
    n = np.arange(16)
    for shift, power in ((0, -133), (4, -129)):
        bits = (n << shift).astype(np.uint32) << 16
        assert np.array_equal(bits.view(np.float32).astype(np.float64), np.ldexp(n.astype(np.float64), power))
    mant = 1 + np.arange(128) / 128
    for e in (-97, -40, -9, 0, 23):
        s = np.ldexp(mant, e)[:, None] * np.array([[1.0], [-1.0]])[:, None]
        want = np.ldexp(_bf16((n - 8) * s), -29)
        for power, scale in ((-129, 100), (-133, 104)):
            got = _bf16(np.ldexp(n * 1.0, power) * np.ldexp(s, scale) - np.ldexp(s, -26))
            assert np.array_equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("hidden,inter,counts,scale_octaves", [
    (512, 512, [1, 15, 16, 17, 0, 31, 33, 48], 0),      # two weight stages per product; the token steps of the MMA
    (1024, 512, [63, 64, 65, 2], 0),                    # a full tile, and one token of a second
    (512, 1536, [130, 1, 1, 7], 12),                    # three tiles of one expert; scales over 24 octaves
    (7168, 2048, [5, 20], 0),                           # more stages than the rings hold
])
def test_grouped_experts_at_tile_edges(cuda, monkeypatch, hidden, inter, counts, scale_octaves):
    """Against the mma.sync kernel, which dequantises to the same values: the fp32 sums differ in order only (below 1e-5 of the
    sum of magnitudes), so a bf16 rounding of gate, up, mid or y moves by at most one place of 2^-8."""
    from blok_b200 import lib, synth
    w = synth.moe_layer_weights(cuda, seed=5, hidden=hidden, inter=inter, experts=128, shared_inter=0)
    g = torch.Generator(device=cuda)
    g.manual_seed(7)
    for k in ("gate_s", "up_s", "down_s"):
        s = w[k].float() * 8
        if scale_octaves:
            s = s * torch.exp2(torch.randint(-scale_octaves, scale_octaves + 1, (s.shape[0], s.shape[1], 1), generator=g, device=cuda).float())
        w[k] = s.bfloat16()
    N = sum(counts)
    layer = lib.MoeLayer(w, max_tokens=max(2, (N + 7) // 8))
    x = synth.activations(N, hidden, cuda, 6)
    e = torch.cat([torch.full((c,), 3 + 5 * i, dtype=torch.int32, device=cuda) for i, c in enumerate(counts)])
    e = e[torch.randperm(N, generator=g, device=cuda)].contiguous()
    rows = torch.randint(0, N, (N,), generator=g, device=cuda).to(torch.int32)
    out = {}
    for impl in ("mma", "tc"):
        monkeypatch.setenv("BLOK_WGEMM_IMPL", impl)
        out[impl] = layer.experts_grouped(x, e, rows).float()
        layer.check()
    ref = out["mma"]
    err = (out["tc"] - ref).abs()
    top = ref.abs().amax(dim=1, keepdim=True)
    assert bool(torch.isfinite(ref).all()) and float((err / top).max()) <= 2.0 ** -7
    assert torch.equal(out["tc"], layer.experts_grouped(x, e, rows).float())
    # without a row index the rows are taken as they come
    assert torch.equal(out["tc"], layer.experts_grouped(x[rows.long()].contiguous(), e).float())
    layer.close()


@pytest.mark.gpu
@pytest.mark.parametrize("T,hidden,shared", [(65, 1024, 512), (128, 2048, 1024), (129, 7168, 2048), (1153, 1024, 1024)])
def test_dense_products_of_a_batch(cuda, monkeypatch, T, hidden, shared):
    """The router and the shared expert over more than 64 tokens (TMA-fed GEMM, K split where its tiles are few) against the
    mma.sync kernel: the same operands and rounding points, fp32 sums in another order (as above)."""
    from blok_b200 import lib, synth
    w = synth.moe_layer_weights(cuda, seed=9, hidden=hidden, inter=512, experts=128, shared_inter=shared)
    x = synth.activations(T, hidden, cuda, 10)
    layer = lib.MoeLayer(w, max_tokens=T)
    out = {}
    for impl in ("mma", ""):
        monkeypatch.setenv("BLOK_WGEMM_IMPL", impl)
        y, ids, wts = layer.batched(x, return_routing=True)
        out[impl] = y.float(), layer.shared(x).float(), ids.view(torch.int16).clone(), wts.clone()
        layer.check()
    (y0, s0, i0, w0), (y1, s1, i1, w1) = out["mma"], out[""]
    assert float(((s1 - s0).abs() / s0.abs().amax(dim=1, keepdim=True)).max()) <= 2.0 ** -7
    same = (i0 == i1).all(dim=1)  # two scores closer than the sums' noise may change places
    assert float(same.float().mean()) > 0.98 and torch.allclose(w0[same], w1[same], rtol=1e-4)
    assert float(((y1 - y0).abs() / y0.abs().amax(dim=1, keepdim=True))[same].max()) <= 2.0 ** -6
    layer.close()
