"""Kernels that become resident while the kernel before them runs (launch_pdl in csrc/common.cuh): a chain of calls without a
synchronisation between them, started behind a long wait, must give the bits of the same chain synchronised after every call."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _chain(step, x, n, sync):
    torch.cuda._sleep(20_000_000)  # the first input is still to be written when the chain is enqueued
    y = x.clone()
    outs = []
    for _ in range(n):
        y = step(y)
        outs.append(y)
        if sync:
            torch.cuda.synchronize()
    torch.cuda.synchronize()
    return outs


def _same(step, x, n=12):
    want, got = _chain(step, x, n, True), _chain(step, x, n, False)
    assert bool(torch.isfinite(want[-1].float()).all()) and float(want[-1].float().abs().max()) > 0
    for i, (a, b) in enumerate(zip(want, got)):
        assert torch.equal(a, b), "call %d" % i


@pytest.mark.parametrize("T,n", [(1, 7168), (148, 1536), (1700, 7168), (300, 1030)])  # one block, a wave, several; rows of odd length
def test_norms(cuda, T, n):
    from blok_b200 import lib, synth
    x, w = synth.activations(T, n, cuda, 1), synth.activations(1, n, cuda, 2)[0]
    _same(lambda y: lib.rmsnorm(lib.rmsnorm(y, w), w), x)

    def residual(y):  # both rows are results of the launches just before
        t = lib.rmsnorm(y, w)
        return lib.add_rmsnorm(t, y, w)
    _same(residual, x)


@pytest.mark.parametrize("T", [9, 33, 64])
def test_streaming_products(cuda, T):
    """Both products of a dense layer with their K-split reductions, a norm between the layers."""
    from blok_b200 import lib, synth
    g = torch.Generator(device=cuda)
    g.manual_seed(T)
    hidden, inter = 2048, 3072
    w = [(torch.randn(s, generator=g, device=cuda) * 0.02).bfloat16() for s in ((inter, hidden), (inter, hidden), (hidden, inter))]
    ln = torch.ones(hidden, device=cuda, dtype=torch.bfloat16)
    _same(lambda y: lib.bf16_mlp(*w, lib.rmsnorm(y, ln)), synth.activations(T, hidden, cuda, T))


@pytest.mark.parametrize("B,paged", [(1, False), (8, False), (33, False), (5, True)])
def test_attention_block(cuda, B, paged):
    """The MLA block: every call appends a cache row that the next one reads, and its input is the output before, normalised."""
    from blok_b200 import lib, synth
    ctx, rows = 300, 384
    layer = lib.MlaLayer(synth.mla_weights(cuda), max_batch=B, max_ctx=rows)
    ln = torch.ones(7168, device=cuda, dtype=torch.bfloat16)
    cache0 = synth.latent_cache(B, rows, cuda)
    table = torch.randperm(B * rows // 64, generator=torch.Generator().manual_seed(3)).int().view(B, -1).to(cuda)
    state = {}

    def step(y):
        y = lib.rmsnorm(y, ln)
        pos = torch.full((B,), ctx + state["n"], dtype=torch.int32, device=cuda)
        state["n"] += 1
        if paged:
            return layer.decode_paged(y, state["cache"].view(-1, 64, 576), table, pos)
        return layer.decode(y, state["cache"], pos)

    outs = {}
    for sync in (True, False):
        state.update(n=0, cache=cache0.clone())
        outs[sync] = _chain(step, synth.activations(B, 7168, cuda, 4), 12, sync) + [state["cache"]]
    layer.check()
    for i, (a, b) in enumerate(zip(outs[True], outs[False])):
        assert torch.equal(a, b), "call %d" % i
    layer.close()
