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


@pytest.mark.parametrize("what,rows", [("expert", 1), ("mla", 1), ("mla", 20), ("moe", 5), ("moe", 60)])
def test_weights_written_just_before(cuda, what, rows):
    """Kernels that fetch their weights before the launches in front of them have finished: weights that an ordinary launch wrote
    just before the call are the ones that count."""
    from blok_b200 import lib, synth
    if what == "mla":
        names = ("q_a", "q_b", "kv_a", "o")
        w, other = synth.mla_weights(cuda, seed=1), synth.mla_weights(cuda, seed=2)
        layer = lib.MlaLayer(w, max_batch=rows, max_ctx=128)
        hidden, cache0 = 7168, synth.latent_cache(rows, 128, cuda)
        pos = torch.full((rows,), 90, dtype=torch.int32, device=cuda)
        call = lambda y: layer.decode(y, cache0.clone(), pos)  # noqa: E731
    else:
        hidden = 2048
        w, other = (synth.moe_layer_weights(cuda, seed=s, hidden=hidden, inter=1024, experts=128, shared_inter=1024) for s in (1, 2))
        if what == "moe":
            names = ("router_w", "shared_gate", "shared_up", "shared_down")
            layer = lib.MoeLayer(w, max_tokens=rows)
            call = layer.batched
        else:
            w, other = ({k: v[3].contiguous() for k, v in t.items() if v.dim() == 3} for t in (w, other))
            names = ("gate_w", "gate_s", "up_w", "up_s", "down_w", "down_s")
            call = lambda y: lib.expert_ffn(*(w[k] for k in names), y[0])[None]  # noqa: E731
    sets = [{k: t[k].clone() for k in names} for t in (w, other)]
    ln = torch.ones(hidden, device=cuda, dtype=torch.bfloat16)
    turn = [0]

    def step(y):
        y = lib.rmsnorm(y, ln)
        turn[0] += 1
        for k in names:
            w[k].copy_(sets[turn[0] % 2][k])
        return call(y)

    _same(step, synth.activations(rows, hidden, cuda, 4))
