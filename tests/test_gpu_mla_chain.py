"""The MLA block's chain of launches at the edges of its tiles: columns that end inside a 64-column step, heads of 16 to 144 values,
query parts around the 128-column piece, entries around the 16-token groups, splits of the context from one to many."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

HEADS, ROPE, RANK = 64, 64, 512


def _weights(cuda, hidden, q_rank, nope, v_head, seed):
    g = torch.Generator(device=cuda).manual_seed(seed)

    def mat(r, c):
        return (torch.randn((r, c), generator=g, device=cuda) / math.sqrt(c)).bfloat16()

    w = dict(q_a=mat(q_rank, hidden), q_b=mat(HEADS * (nope + ROPE), q_rank), kv_a=mat(RANK + ROPE, hidden),
             kv_b=mat(HEADS * (nope + v_head), RANK), o=mat(hidden, HEADS * v_head))
    for k, n in (("q_a_ln", q_rank), ("kv_a_ln", RANK)):
        w[k] = (1 + 0.2 * torch.randn((n,), generator=g, device=cuda)).bfloat16()
    return w, g


def _rms(x, w):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w


def _rotate(x, pos, factor):
    def place(r):
        return ROPE * math.log(4096.0 / (r * 2 * math.pi)) / (2 * math.log(50000.0))
    low, high = max(math.floor(place(32.0)), 0), min(math.ceil(place(1.0)), ROPE - 1)
    p = torch.arange(ROPE // 2, device=x.device, dtype=torch.float64)
    fast, ramp = 50000.0 ** (-2 * p / ROPE), ((p - low) / (high - low)).clamp(0, 1)
    ang = (pos.double()[:, None] * (fast / factor * ramp + fast * (1 - ramp))).reshape((len(pos),) + (1,) * (x.dim() - 2) + (ROPE // 2,))
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()], dim=-1)


def _plain(w, n, pos, nope, v_head, rows_of, factor=32.0):
    """The block in 64 bits; rows_of(b, new rows) -> the cached rows entry b sees."""
    w = {k: t.double() for k, t in w.items()}
    q = (_rms(n @ w["q_a"].T, w["q_a_ln"]) @ w["q_b"].T).reshape(len(n), HEADS, nope + ROPE)
    kv = n @ w["kv_a"].T
    new = torch.cat([_rms(kv[:, :RANK], w["kv_a_ln"]), _rotate(kv[:, RANK:], pos, factor)], dim=1)
    kvb = w["kv_b"].reshape(HEADS, nope + v_head, RANK)
    qf = torch.cat([torch.einsum("bhd,hdj->bhj", q[..., :nope], kvb[:, :nope]), _rotate(q[..., nope:], pos, factor)], dim=-1)
    scale = (0.1 * math.log(factor) + 1) ** 2 / math.sqrt(nope + ROPE)
    o = torch.stack([torch.softmax(qf[b] @ r.T * scale, dim=-1) @ r[:, :RANK] for b in range(len(n)) for r in [rows_of(b, new)]])
    return torch.einsum("bhj,hvj->bhv", o, kvb[:, nope:]).reshape(len(n), -1) @ w["o"].T, new


def _check(got, want, what):
    # nine roundings to bf16 (2^-9 / sqrt(3) each, rms) and the softmax between them: 0.004; twice that and a margin
    err = float((got.double() - want).norm() / want.norm())
    assert err < 1e-2, (what, err)


@pytest.mark.parametrize("hidden,q_rank,nope,v_head,B", [
    (288, 96, 32, 16, 1), (288, 96, 96, 48, 2), (512, 160, 160, 144, 3), (7168, 1536, 128, 128, 8), (800, 96, 128, 128, 9),
    (512, 1536, 288, 32, 16), (1056, 1536, 128, 112, 17), (288, 512, 64, 128, 32), (512, 96, 128, 128, 33), (288, 224, 160, 16, 49),
    (2048, 1536, 128, 128, 64)])
def test_chain(cuda, hidden, q_rank, nope, v_head, B):
    from blok_b200 import lib
    w, g = _weights(cuda, hidden, q_rank, nope, v_head, B)
    layer = lib.MlaLayer(w, yarn_factor=32.0, max_batch=64, max_ctx=700, qk_nope=nope, v_head=v_head)
    n = torch.randn((B, hidden), generator=g, device=cuda).bfloat16()
    # a batch of sequences of different lengths
    ctx = 700
    pos = torch.randint(0, ctx, (B,), generator=g, device=cuda).to(torch.int32)
    pos[0], pos[-1] = 0, ctx - 1
    cache = torch.randn((B, ctx, RANK + ROPE), generator=g, device=cuda).bfloat16()
    before = cache.clone()
    out = layer.decode(n, cache, pos)
    want, new = _plain(w, n.double(), pos, nope, v_head, lambda b, new: torch.cat([before[b, :int(pos[b])].double(), new[b:b + 1]]))
    _check(out, want, "decode")
    at = torch.arange(B, device=cuda), pos.long()
    _check(cache[at], new, "rows")
    cache[at] = before[at]
    assert torch.equal(cache, before)
    assert torch.equal(layer.decode(n, cache, pos), out)  # repeats bit for bit
    # the same entries as a chunk of one sequence
    first, rows = 70, torch.randn((70 + B, RANK + ROPE), generator=g, device=cuda).bfloat16()
    head = rows[:first].double()
    out = layer.prefill(n, rows, torch.tensor([first], dtype=torch.int32, device=cuda))
    want, new = _plain(w, n.double(), first + torch.arange(B, device=cuda), nope, v_head, lambda b, new: torch.cat([head, new[:b + 1]]))
    _check(out, want, "chunk")
    _check(rows[first:], new, "chunk rows")
    layer.check()
    layer.close()


# around 48 KB of a norm's shared memory (12,160 to 12,288 values leave no room for its static arrays), and rows longer than an SM's
@pytest.mark.parametrize("q_rank", [11264, 11296, 12160, 12288, 61440])
def test_long_query_rows(cuda, q_rank):
    from blok_b200 import lib
    hidden, nope, v_head, B = 288, 32, 16, 2
    w, g = _weights(cuda, hidden, q_rank, nope, v_head, q_rank)
    layer = lib.MlaLayer(w, yarn_factor=32.0, max_batch=B, max_ctx=100, qk_nope=nope, v_head=v_head)
    n = torch.randn((B, hidden), generator=g, device=cuda).bfloat16()
    pos = torch.tensor([7, 99], dtype=torch.int32, device=cuda)
    cache = torch.randn((B, 100, RANK + ROPE), generator=g, device=cuda).bfloat16()
    before = cache.clone()
    out = layer.decode(n, cache, pos)
    want, _ = _plain(w, n.double(), pos, nope, v_head, lambda b, new: torch.cat([before[b, :int(pos[b])].double(), new[b:b + 1]]))
    _check(out, want, "decode")
    layer.check()
    layer.close()


@pytest.mark.parametrize("lens", [
    [1] * 60 + [900, 64, 65, 3000],                    # pieces over the sequences' borders, several sequences to a CTA
    [0, 5, 0, 700, 128, 0],                            # empty sequences: zeros
    [1300] * 50, [64 * 37] * 4, list(range(1, 65))])
def test_core_over_lengths(cuda, lens):
    """The attention core alone over batches of sequences whose tiles fall on the CTAs in every way."""
    from blok_b200 import lib
    w, g = _weights(cuda, 288, 96, 32, 16, len(lens))
    layer = lib.MlaLayer(w, yarn_factor=32.0, max_batch=64, max_ctx=64, qk_nope=32, v_head=16)
    B, ctx = len(lens), max(lens) + 3
    cache = torch.randn((B, ctx, RANK + ROPE), generator=g, device=cuda).bfloat16()
    for b, n in enumerate(lens):
        cache[b, n:] = float("nan")                    # rows past a sequence's end are nobody's business
    q = (torch.randn((B, HEADS, RANK + ROPE), generator=g, device=cuda) * 0.3).bfloat16()
    o = layer.attend(q, cache, torch.tensor(lens, dtype=torch.int32, device=cuda))
    layer.check()
    for b, n in enumerate(lens):
        rows = cache[b, :n].double()
        want = torch.softmax(q[b].double() @ rows.T * layer.scale, dim=-1) @ rows[:, :RANK]
        if n == 0:
            assert not o[b].any(), b
        else:                                          # probabilities and results to bf16: 2^-9 each
            err = float((o[b].double() - want).norm() / want.norm())
            assert err < 6e-3, (b, n, err)
    layer.close()


# one sequence has a plan without a search; parts from one to all CTAs', around the sixteen that the merge has in flight, and (320 blocks)
# around its eight
@pytest.mark.parametrize("lens", [[1], [64 * 15], [64 * 16 + 1], [64 * 17], [3000], [64 * 148], [64 * 149 - 1], [64 * 300 + 5], [20000] * 5])
def test_core_over_few_long_sequences(cuda, lens):
    test_core_over_lengths(cuda, lens)
