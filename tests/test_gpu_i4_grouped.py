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
    """fma(n 2^-129, s 2^117, -s 2^-9) and fma(n 2^-133, s 2^121, -s 2^-9), rounded once, are 2^-12 bf16(q s) for every nibble
    and every scale mantissa, over the exponents the kernel claims; the bit patterns are the numbers the kernel takes them for."""
    n = np.arange(16)
    for shift, power in ((0, -133), (4, -129)):
        bits = (n << shift).astype(np.uint32) << 16
        assert np.array_equal(bits.view(np.float32).astype(np.float64), np.ldexp(n.astype(np.float64), power))
    mant = 1 + np.arange(128) / 128
    for e in (-114, -40, -9, 0, 6):
        s = np.ldexp(mant, e)[:, None] * np.array([[1.0], [-1.0]])[:, None]
        want = np.ldexp(_bf16((n - 8) * s), -12)
        for power, scale in ((-129, 117), (-133, 121)):
            got = _bf16(np.ldexp(n * 1.0, power) * np.ldexp(s, scale) - np.ldexp(s, -9))
            assert np.array_equal(got, want)


def test_range_of_scales_by_their_bits():
    """The kernel's two integer tests over every bf16 bit pattern: the exact one says whether s = 0 or 2^-114 <= |s| < 2^7, and what
    the quick one lets by (exponent bits 01......) is inside."""
    bits = np.arange(1 << 16, dtype=np.uint32)
    with np.errstate(invalid="ignore"):
        s = np.abs((bits << 16).view(np.float32).astype(np.float64))
    inside = (s == 0) | ((s >= 2.0 ** -114) & (s < 2.0 ** 7))
    v = ((bits | 0x8000) - 1).astype(np.uint16)
    outside = (v > np.uint16(0xc2fe)) | (v.view(np.int16) < np.array(0x867f, dtype=np.uint16).view(np.int16))
    assert np.array_equal(~outside, inside)
    assert inside[((bits ^ 0x2000) & 0x6000) == 0].all()


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
@pytest.mark.parametrize("gate,up,down,act", [
    (0, 40, -112, 0),      # every up scale above the range of the one-instruction dequantisation, every down scale below it
    (0, -112, 60, 0),      # and the other way round
    (-112, 112, 0, 0),
    (None, None, None, 0),  # single blocks of 32 columns in a few rows: 2^25, 2^-116 and 2^-133 (the smallest there is), and zeros
    (0, 0, 0, -59),        # activations whose results lie near the smallest normal numbers
])
def test_grouped_experts_take_any_scale(cuda, monkeypatch, gate, up, down, act):
    """Scales outside 2^-114 .. 2^7: the tcgen05 kernel against the mma.sync kernel, which multiplies every nibble by its scale.
    The same weights, fp32 sums in another order: tolerance as above."""
    from blok_b200 import lib, synth
    hidden, inter, N = 1024, 512, 75
    w = synth.moe_layer_weights(cuda, seed=8, hidden=hidden, inter=inter, experts=128, shared_inter=0)
    for k, octaves in (("gate_s", gate), ("up_s", up), ("down_s", down)):
        s = w[k].float() * 8
        if octaves is None:
            s[:, 5::64, 3] = 2.0 ** 25
            s[:, 6::64, 7] = 2.0 ** -116
            s[:, 7::64, :] = 2.0 ** -133
            s[:, 8::64, ::2] = 0.0
        else:
            s = s * 2.0 ** octaves
        w[k] = s.bfloat16()
    layer = lib.MoeLayer(w, max_tokens=16)
    x = (synth.activations(N, hidden, cuda, 6).float() * 2.0 ** act).bfloat16()
    e = torch.tensor([3] * 66 + [4, 4, 4] + [90] * 6, dtype=torch.int32, device=cuda)
    out = {}
    for impl in ("mma", "tc", ""):
        monkeypatch.setenv("BLOK_WGEMM_IMPL", impl)
        out[impl] = layer.experts_grouped(x, e).double()  # squares of the largest results overflow fp32
        layer.check()
    ref = out["mma"]
    assert bool(torch.isfinite(ref).all()) and bool((ref.abs().amax(dim=1) > 0).all())
    for impl in ("tc", ""):
        assert float(((out[impl] - ref).abs() / ref.abs().amax(dim=1, keepdim=True)).max()) <= 2.0 ** -7
        # rows of small weights beside rows of large ones
        rows = ref.abs().amax(dim=0)
        assert float(((out[impl] - ref).abs().amax(dim=0) / rows.clamp_min(1e-300)).max()) <= 2.0 ** -6
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


@pytest.mark.gpu
@pytest.mark.parametrize("T,experts,topk", [(1, 32, 8), (5, 128, 8), (33, 384, 8), (9, 385, 6), (4, 1024, 16)])
def test_router_ties_and_special_scores(cuda, T, experts, topk):
    """Selection by the reference's rule (strict '>' over ascending indices): equal scores by index, +0 and -0 alike, -inf and
    NaN never, +inf first.  Scores are set through the bias; a zero router matrix makes every sigmoid 0.5."""
    from blok_b200 import lib
    g = torch.Generator().manual_seed(experts)
    bias = torch.randint(-3, 4, (experts,), generator=g).float() * 0.25 - 0.5  # sel = 0.5 + bias: many ties, zeros among them
    bias[3], bias[7], bias[11] = float("nan"), -float("inf"), float("inf")
    bias[13] = -0.5
    x = torch.randn(T, 256, generator=g).to(cuda, torch.bfloat16)
    ids, wts = lib.router(torch.zeros(experts, 256, dtype=torch.bfloat16, device=cuda), bias.to(cuda), x, topk=topk)
    sel = (bias + 0.5).numpy()
    want = []
    for _ in range(topk):
        best, at = -np.inf, 0
        for i, v in enumerate(sel):
            if v > best:
                best, at = v, i
        want.append(at)
        sel[at] = -np.inf
    assert all(r == want for r in util.ids_np(ids).reshape(T, topk).tolist())
    assert torch.allclose(wts.float(), torch.full_like(wts.float(), 2.827 / topk), rtol=1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("N", [1023, 1024, 1025, 4096])
def test_order_of_assignments(cuda, monkeypatch, N):
    """Up to 1,024 assignments are sorted by the plan kernel, more by a kernel of their own: each row's result does not depend on
    which, nor on the rows around it."""
    from blok_b200 import lib, synth
    monkeypatch.setenv("BLOK_WGEMM_IMPL", "tc")
    w = synth.moe_layer_weights(cuda, seed=3, hidden=512, inter=512, experts=128, shared_inter=0)
    layer = lib.MoeLayer(w, max_tokens=512)
    g = torch.Generator(device=cuda)
    g.manual_seed(N)
    x = synth.activations(N, 512, cuda, 4)
    e = torch.randint(0, 128, (N,), generator=g, device=cuda).to(torch.int32)
    y = layer.experts_grouped(x, e)
    for lo in (0, N // 2):
        part = slice(lo, lo + 300)
        assert torch.equal(y[part], layer.experts_grouped(x[part].contiguous(), e[part].contiguous()))
    layer.close()


@pytest.mark.gpu
@pytest.mark.parametrize("hidden,topk,offset", [(512, 8, 0), (514, 8, 0), (512, 3, 2), (1032, 12, 0)])
def test_combine_by_16_and_by_4_bytes(cuda, hidden, topk, offset):
    """bf16(bf16(sum_k w y) + shared) with the sum in slot order, whatever the rows' length and alignment."""
    from blok_b200 import lib
    g = torch.Generator(device=cuda)
    g.manual_seed(hidden)
    T = 5

    def rand(n):
        return torch.randn(n + offset, generator=g, device=cuda).bfloat16()[offset:]

    y, s = rand(T * topk * hidden).view(T * topk, hidden), rand(T * hidden).view(T, hidden)
    wts = torch.rand(T, topk, generator=g, device=cuda)
    got = lib.moe_combine(y, wts, s)
    acc = torch.zeros(T, hidden, device=cuda, dtype=torch.float64)
    for k in range(topk):
        acc = (acc + y.view(T, topk, hidden)[:, k].double() * wts[:, k:k + 1].double()).float().double()
    want = (acc.float().bfloat16().float() + s.float()).bfloat16()
    # one rounding per fused multiply-add; where the emulation's double rounding of the product differs, by one place of bf16
    assert float((got.float() - want.float()).abs().max() / want.float().abs().max()) <= 2.0 ** -8
    assert float((got == want).float().mean()) > 0.99
