"""GPU parity of the batched routed-MoE layer (config 2) against the oracle and against the batch-1 path."""
import numpy as np
import pytest
import torch

import util
from test_gpu_moe_decode import _host_layer

pytestmark = pytest.mark.gpu
MARGIN = 2e-6


def _oracle_layer(oracle, w, x, ids_needed, topk=8):
    slot_of, packs, scs, shared = _host_layer(w, ids_needed)
    return oracle.moe_layer(util.t2np_bf16(w["router_w"]), util.t2np_f32(w["router_bias"]), slot_of, packs["gate_w"],
                            scs["gate_s"], packs["up_w"], scs["up_s"], packs["down_w"], scs["down_s"], shared[0], shared[1],
                            shared[2], util.t2np_f32(x), topk=topk, mode=0)


# the mma.sync kernel and the tcgen05 kernels, whatever the size; "auto": the library's own choice, which takes the mat-vec-style
# kernel (wgemv_small.cu) up to 40 assignments (T = 5) and the tcgen05 kernel from there
@pytest.mark.parametrize("impl", ["mma", "tc", "auto"])
@pytest.mark.parametrize("T,hidden,inter,experts,shared,seed", [(40, 1024, 512, 128, 512, 31), (1, 1024, 512, 128, 512, 32),
                                                                (64, 7168, 2048, 384, 2048, 2), (130, 512, 512, 128, 0, 33),
                                                                (7, 1024, 512, 128, 512, 34), (2, 2048, 1024, 128, 512, 35),
                                                                (5, 1536, 512, 128, 0, 36)])
def test_moe_batched_vs_oracle(cuda, oracle, monkeypatch, impl, T, hidden, inter, experts, shared, seed):
    from blok_b200 import lib, synth
    if impl == "auto":
        monkeypatch.delenv("BLOK_WGEMM_IMPL", raising=False)
    else:
        monkeypatch.setenv("BLOK_WGEMM_IMPL", impl)
    w = synth.moe_layer_weights(cuda, seed=seed, hidden=hidden, inter=inter, experts=experts, shared_inter=shared)
    if hidden < 7168:
        for k in ("gate_s", "up_s", "down_s"):
            w[k] = (w[k].float() * 8).bfloat16()
        w["router_w"] = (w["router_w"].float() * 20).bfloat16()
    layer = lib.MoeLayer(w, max_tokens=max(T, 2))
    x = synth.activations(T, hidden, cuda, seed)
    y, ids, wts = layer.batched(x, return_routing=True)
    layer.check()  # no tensor-core tile gave up on a barrier
    ids_h = util.ids_np(ids)
    oid, owt, margin, _ = oracle.router(util.t2np_bf16(w["router_w"]), util.t2np_f32(w["router_bias"]), util.t2np_f32(x), mode=0)
    clear = margin > MARGIN
    assert clear.mean() > 0.95
    for t in np.nonzero(clear)[0]:
        assert set(ids_h[t].tolist()) == set(oid[t].tolist()), "token %d" % t
    out, _, _ = _oracle_layer(oracle, w, x, list(ids_h.ravel()) + list(oid.ravel()))
    yh = util.t2np_f32(y)
    same = np.all(ids_h == oid, axis=1)
    for t in np.nonzero(same)[0]:
        util.assert_close(yh[t], out[t], "batched token %d" % t)
    assert same.mean() > 0.9
    assert torch.equal(y, layer.batched(x)), "deterministic"
    layer.close()


def test_moe_batched_agrees_with_decode_path_at_2048_tokens(cuda):
    """T = 2048 (config 2's large case): every token of the batch must match the batch-1 kernel on the same token."""
    from blok_b200 import lib, synth
    w = synth.moe_layer_weights(cuda, seed=2)
    layer = lib.MoeLayer(w, max_tokens=2048)
    x = synth.activations(2048, 7168, cuda, 2)
    y, ids, wts = layer.batched(x, return_routing=True)
    counts = torch.bincount(ids.view(torch.int16).long().ravel() & 0xFFFF, minlength=384)
    assert int(counts.sum()) == 2048 * 8 and int((counts > 0).sum()) > 350
    for t in (0, 1, 777, 2047):
        y1, i1, w1 = layer.decode(x[t].contiguous(), return_routing=True)
        if torch.equal(i1, ids[t]):
            assert util.max_abs_rel(util.t2np_f32(y[t]), util.t2np_f32(y1)) < 1e-2
            assert util.cosine(util.t2np_f32(y[t]), util.t2np_f32(y1)) > 0.9999
    np.testing.assert_allclose(util.t2np_f32(wts).sum(axis=1), 2.827, rtol=1e-5)
    layer.close()


def test_moe_batched_2048_tokens_against_the_oracle(cuda, oracle):
    """Config 2's large case at full size (T = 2048, 384 experts): the routing of EVERY token against the oracle, in
    selection order, and the layer output of 64 tokens spread over the batch against the oracle's layer."""
    from blok_b200 import lib, synth
    w = synth.moe_layer_weights(cuda, seed=2)
    layer = lib.MoeLayer(w, max_tokens=2048)
    x = synth.activations(2048, 7168, cuda, 2)
    y, ids, wts = layer.batched(x, return_routing=True)
    layer.check()
    ids_h, wts_h = util.ids_np(ids), util.t2np_f32(wts)
    oid, owt, margin, _ = oracle.router(util.t2np_bf16(w["router_w"]), util.t2np_f32(w["router_bias"]), util.t2np_f32(x), mode=0)
    # a token's selection is beyond doubt when the 8th and 9th candidates are apart (margin) and so are the selected ones
    # among themselves (their weights are the scores, normalised: distinct weights, distinct scores)
    gaps = np.abs(np.diff(np.sort(owt, axis=1), axis=1)).min(axis=1)
    clear = (margin > MARGIN) & (gaps > 1e-6)
    assert clear.mean() > 0.9
    assert np.array_equal(ids_h[clear], oid[clear]), "top-k ids, in selection order"
    np.testing.assert_allclose(wts_h[clear], owt[clear], rtol=2e-5)
    sample = np.nonzero(clear)[0][:: max(1, int(clear.sum()) // 64)][:64]
    assert len(sample) == 64
    xs = x[torch.from_numpy(sample).to(cuda)]
    out, _, _ = _oracle_layer(oracle, w, xs, list(oid[sample].ravel()))
    yh = util.t2np_f32(y)
    worst = 0.0
    for i, t in enumerate(sample):
        r, c = util.assert_close(yh[t], out[i], "T=2048 token %d" % t)
        worst = max(worst, r)
    print("T=2048: %d tokens routed as the oracle routes them, 64 outputs checked, worst max-abs-rel %.2e" % (int(clear.sum()), worst))
    layer.close()


@pytest.mark.parametrize("impl", ["mma", "tc", "auto"])
def test_experts_grouped_handles_empty_and_ragged_groups(cuda, oracle, monkeypatch, impl):
    """Assignments concentrated on few experts (others get zero tokens), more than one 64-token tile for one expert.
    Left to itself ("auto") the library takes the tcgen05 kernel: there are more than 40 assignments."""
    from blok_b200 import lib, synth
    monkeypatch.setenv("BLOK_WGEMM_IMPL", impl)
    hidden, inter, experts = 512, 512, 128
    w = synth.moe_layer_weights(cuda, seed=41, hidden=hidden, inter=inter, experts=experts, shared_inter=0)
    for k in ("gate_s", "up_s", "down_s"):
        w[k] = (w[k].float() * 8).bfloat16()
    layer = lib.MoeLayer(w, max_tokens=64)
    x = synth.activations(30, hidden, cuda, 41)
    e = torch.tensor([5] * 70 + [127] * 3 + [0] + [64] * 9, dtype=torch.int32, device=cuda)
    rows = torch.arange(e.numel(), dtype=torch.int32, device=cuda) % 30
    y = util.t2np_f32(layer.experts_grouped(x, e, rows))
    xh = util.t2np_f32(x)
    for a in (0, 69, 70, 72, 73, 82):
        ex = int(e[a])
        ref = oracle.expert_ffn(util.t2np_u32(w["gate_w"][ex]), util.t2np_bf16(w["gate_s"][ex]), util.t2np_u32(w["up_w"][ex]),
                                util.t2np_bf16(w["up_s"][ex]), util.t2np_u32(w["down_w"][ex]), util.t2np_bf16(w["down_s"][ex]),
                                xh[int(rows[a])], mode=0, round_out=True)
        util.assert_close(y[a], ref, "assignment %d" % a)
    layer.check()
    assert layer.experts_grouped(x, e[:0].contiguous(), rows[:0].contiguous()).shape == (0, hidden)
    with pytest.raises(lib.BlokError):
        layer.experts_grouped(x, torch.zeros(64 * 8 + 1, dtype=torch.int32, device=cuda))
    layer.close()


# blocks of 512 assignments sort (mb_sort_kernel): one short of a block, one block, one more, several with a remainder; ids that are no
# expert of the layer's (-1, the count itself) lie between the others
@pytest.mark.parametrize("N,only", [(511, None), (512, None), (513, None), (1025, None), (4136, None), (1500, 9)])
def test_sort_of_the_assignments(cuda, N, only):
    """A row of the result holds its own assignment's value: the same, bit for bit, as a call for that (expert, row) pair gives.  A
    row's arithmetic in the tcgen05 kernel does not depend on the tile it lies in, so there is no tolerance."""
    from blok_b200 import lib, synth
    hidden, inter, experts, nrows = 512, 512, 40, 3
    w = synth.moe_layer_weights(cuda, seed=47, hidden=hidden, inter=inter, experts=experts, shared_inter=0)
    layer = lib.MoeLayer(w, max_tokens=600)
    x = synth.activations(nrows, hidden, cuda, 47)
    g = torch.Generator().manual_seed(N)
    e = torch.full((N,), only) if only is not None else torch.randint(-1, experts + 1, (N,), generator=g)
    rows = torch.randint(0, nrows, (N,), generator=g)
    pairs_e = torch.arange(experts).repeat_interleave(nrows)
    each = layer.experts_grouped(x, pairs_e.int().to(cuda), torch.arange(nrows).repeat(experts).int().to(cuda))
    got = layer.experts_grouped(x, e.int().to(cuda), rows.int().to(cuda))
    layer.check()
    ours = (e >= 0) & (e < experts)
    want = each[(e.clamp(0, experts - 1) * nrows + rows).to(cuda)]
    assert len(torch.unique(each.view(torch.int16), dim=0)) == experts * nrows, "every pair has a value of its own"
    assert torch.equal(got[ours.to(cuda)], want[ours.to(cuda)])
    layer.close()


@pytest.mark.parametrize("hidden,inter,groups,small", [
    (512, 512, {7: 40}, True),                               # ten passes of four tokens over one expert
    (2048, 1024, {0: 2, 5: 3, 64: 4, 90: 9, 127: 5}, True),  # passes of 1 to 4 tokens; scales staged in chunks of 16 k-blocks
    (1536, 512, {3: 9, 4: 5, 126: 26}, True),                # 40 assignments; chunks of 14
    (7168, 512, {2: 1, 3: 2, 383: 6}, True),                 # rows of full length, four whole chunks of 14
    (1024, 512, {0: 1, 1: 40}, False),                       # one more than the mat-vec-style kernel takes
])
def test_few_assignments(cuda, oracle, monkeypatch, hidden, inter, groups, small):
    """The library's own choice up to 40 assignments, the mat-vec-style kernel (wgemv_small.cu), in passes of up to four tokens of
    one expert, every assignment against the oracle; the tcgen05 kernel gives other bits below the limit and the same above."""
    from blok_b200 import lib, synth
    monkeypatch.delenv("BLOK_WGEMM_IMPL", raising=False)
    w = synth.moe_layer_weights(cuda, seed=43, hidden=hidden, inter=inter, experts=384, shared_inter=0)
    if hidden < 7168:
        for k in ("gate_s", "up_s", "down_s"):
            w[k] = (w[k].float() * 8).bfloat16()
    N = sum(groups.values())
    layer = lib.MoeLayer(w, max_tokens=8)
    x = synth.activations(N, hidden, cuda, 44)
    e = torch.tensor([k for k, n in groups.items() for _ in range(n)], dtype=torch.int32, device=cuda)
    e = e[torch.randperm(N, generator=torch.Generator().manual_seed(N)).to(cuda)].contiguous()
    got = layer.experts_grouped(x, e)
    assert torch.equal(got, layer.experts_grouped(x, e))
    y, xh = util.t2np_f32(got), util.t2np_f32(x)
    host = {k: [util.t2np_u32(w[n][k]) if n.endswith("_w") else util.t2np_bf16(w[n][k])
                for n in ("gate_w", "gate_s", "up_w", "up_s", "down_w", "down_s")] for k in groups}
    for a in range(N):
        util.assert_close(y[a], oracle.expert_ffn(*host[int(e[a])], xh[a], mode=0, round_out=True), "assignment %d" % a)
    monkeypatch.setenv("BLOK_WGEMM_IMPL", "tc")
    assert torch.equal(got, layer.experts_grouped(x, e)) != small
    layer.check()
    layer.close()


def test_a_product_that_gave_up_is_reported_by_its_own_handle(cuda):
    """The error word of the products over several tokens belongs to the handle: another layer's check neither reports nor clears
    it.  The word is set from the host (blok_moe_layer_debug_set_error): no wait is made to run out on the device."""
    import ctypes as C
    from blok_b200 import lib, synth
    w = synth.moe_layer_weights(cuda, seed=41, hidden=512, inter=512, experts=128, shared_inter=0)
    a, b, one = lib.MoeLayer(w, max_tokens=4), lib.MoeLayer(w, max_tokens=4), lib.MoeLayer(w)
    assert lib.load().blok_moe_layer_debug_set_error(a._handle, C.c_uint(256), None) == 0
    b.check()
    one.check()
    with pytest.raises(lib.BlokError) as e:
        a.check()
    assert e.value.code == -5 and "blok_moe_batched" in str(e.value)
    a.check()                                   # reported once; the handle stays usable
    x = synth.activations(4, 512, cuda, 1)
    assert torch.equal(a.batched(x), b.batched(x))
    assert lib.load().blok_moe_layer_debug_set_error(one._handle, C.c_uint(256), None) == -4  # no such products on this handle
    for layer in (a, b, one):
        layer.close()


@pytest.mark.parametrize("T,experts,topk,hidden,inter,shared", [
    (1, 128, 8, 512, 512, 512), (2, 384, 8, 1024, 512, 0), (31, 128, 1, 1536, 512, 1024), (32, 256, 6, 512, 1024, 512),
    (33, 384, 16, 512, 512, 512), (63, 128, 16, 2048, 512, 2048), (64, 384, 8, 1024, 512, 512), (64, 128, 7, 512, 512, 0)])
def test_front_of_a_small_batch(cuda, monkeypatch, T, experts, topk, hidden, inter, shared):
    """Up to 64 tokens the router and the shared expert's first half are one launch and what follows them another (routing, sorted
    order, tile table, gated vector): against the separate launches that BLOK_WGEMM_IMPL=tc takes, at the edges of warps and tiles."""
    from blok_b200 import lib, synth
    w = synth.moe_layer_weights(cuda, seed=T + experts, hidden=hidden, inter=inter, experts=experts, shared_inter=shared)
    for k in ("gate_s", "up_s", "down_s"):
        w[k] = (w[k].float() * 8).bfloat16()
    w["router_w"] = (w["router_w"].float() * 20).bfloat16()
    layer = lib.MoeLayer(w, topk=topk, max_tokens=T + 1)
    x = synth.activations(T, hidden, cuda, T)
    monkeypatch.delenv("BLOK_WGEMM_IMPL", raising=False)
    y, ids, wts = layer.batched(x, return_routing=True)
    assert torch.equal(y, layer.batched(x))
    monkeypatch.setenv("BLOK_WGEMM_IMPL", "tc")
    want, wid, wwt = layer.batched(x, return_routing=True)
    assert torch.equal(ids, wid)                       # fp32 logits, summed in another order
    assert float(((wts - wwt).abs() / wwt.abs().clamp(min=1e-6)).max()) < 1e-4
    # eight roundings to bf16 on each side, the intermediate vectors' and the outputs' among them (2^-9 / sqrt(3) each, rms)
    assert float((y.float() - want.float()).norm() / want.float().norm()) < 1e-2
    layer.check()
    layer.close()


def test_a_wide_layer_has_room_for_its_sums(cuda, monkeypatch):
    """The shared expert's down projection leaves its sums also where K is not split: hidden / 128 tiles for all SMs, and a front (twice the
    shared expert and the router) of fewer columns than hidden.  Against the separate launches, as above."""
    from blok_b200 import lib, synth
    T, hidden, shared = 64, 20480, 9728
    w = synth.moe_layer_weights(cuda, seed=9, hidden=hidden, inter=512, experts=128, shared_inter=shared)
    layer = lib.MoeLayer(w, max_tokens=T)
    x = synth.activations(T, hidden, cuda, 9)
    monkeypatch.delenv("BLOK_WGEMM_IMPL", raising=False)
    y, ids, _ = layer.batched(x, return_routing=True)
    monkeypatch.setenv("BLOK_WGEMM_IMPL", "tc")
    want, wid, _ = layer.batched(x, return_routing=True)
    layer.check()
    assert torch.equal(ids, wid)
    assert float((y.float() - want.float()).norm() / want.float().norm()) < 1e-2
    layer.close()


def test_a_refused_launch_is_reported_once(cuda):
    """A launch that CUDA refuses (more tokens than a grid has rows) is the call's error and nobody else's."""
    from blok_b200 import lib
    T = 65536
    y, wts = torch.zeros((T, 2), device=cuda, dtype=torch.bfloat16), torch.ones((T, 1), device=cuda)
    with pytest.raises(lib.BlokError):
        lib.moe_combine(y, wts)
    assert int(torch.ones(3, device=cuda).sum()) == 3
    assert lib.moe_combine(y[:4].contiguous(), wts[:4].contiguous()).shape == (4, 2)


@pytest.mark.parametrize("T,experts,topk,hidden,inter,shared", [(1, 512, 8, 1024, 512, 512), (33, 512, 16, 512, 512, 0), (64, 512, 16, 512, 512, 1024),
                                                                (7, 640, 8, 512, 512, 512)])
def test_front_of_a_small_batch_with_many_experts(cuda, monkeypatch, T, experts, topk, hidden, inter, shared):
    test_front_of_a_small_batch(cuda, monkeypatch, T, experts, topk, hidden, inter, shared)


# one block that counts its own, part of it empty; up to 40 assignments through the tcgen05 kernel as well, whose bits the comparison has
@pytest.mark.parametrize("N,only", [(1, 39), (2, None), (41, None), (100, None)])
def test_sort_of_few_assignments(cuda, monkeypatch, N, only):
    monkeypatch.setenv("BLOK_WGEMM_SMALL", "0")
    test_sort_of_the_assignments(cuda, N, only)
