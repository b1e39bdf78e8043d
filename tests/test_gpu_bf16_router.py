"""GPU parity of the bf16 mat-vec / MLP / RMSNorm kernels and of the router."""
import ctypes as C

import numpy as np
import pytest
import torch

import util

pytestmark = pytest.mark.gpu


def _w(rng, rows, cols, std=0.006):
    return util.f32_to_bf16_np(rng.normal(0, std, (rows, cols)).astype(np.float32))


@pytest.mark.parametrize("rows,cols,T", [(384, 7168, 1), (2048, 7168, 1), (7168, 2048, 1), (576, 7168, 8),
                                         (1536, 7168, 3), (12288, 1536, 8), (48, 512, 2), (10, 64, 1)])
def test_bf16_gemv(cuda, oracle, rows, cols, T):
    from blok_b200 import lib
    rng = np.random.default_rng(rows + cols + T)
    w = _w(rng, rows, cols)
    x = oracle.bf16_round(rng.normal(size=(T, cols)).astype(np.float32))
    dw, dx = util.np_bf16_to_torch(w, cuda), torch.from_numpy(x).to(cuda).bfloat16()
    y16 = util.t2np_f32(lib.bf16_gemv(dw, dx))
    y32 = util.t2np_f32(lib.bf16_gemv(dw, dx, out_f32=True))
    for t in range(T):
        wide = oracle.bf16_gemv(w, x[t], mode=0, round_out=False)
        assert util.max_abs_rel(y32[t], wide) < 1e-5, "fp32 logits path"
        util.assert_close(y16[t], oracle.bf16_round(wide), "bf16_gemv")


# more than 8 rows: each matrix streamed once for all rows (wgemm_stream.cu), K split for the down projection
@pytest.mark.parametrize("hidden,ffn,T", [(7168, 2048, 1), (7168, 2048, 8), (256, 128, 2), (7168, 2048, 9), (7168, 2048, 33),
                                         (512, 256, 64), (1024, 4608, 17)])
def test_bf16_mlp(cuda, oracle, hidden, ffn, T):
    from blok_b200 import lib
    rng = np.random.default_rng(hidden + ffn + T)
    g, u, d = _w(rng, ffn, hidden, 0.02), _w(rng, ffn, hidden, 0.02), _w(rng, hidden, ffn, 0.02)
    x = oracle.bf16_round(rng.normal(size=(T, hidden)).astype(np.float32))
    y = util.t2np_f32(lib.bf16_mlp(util.np_bf16_to_torch(g, cuda), util.np_bf16_to_torch(u, cuda),
                                   util.np_bf16_to_torch(d, cuda), torch.from_numpy(x).to(cuda).bfloat16()))
    for t in range(T):
        util.assert_close(y[t], oracle.bf16_mlp(g, u, d, x[t], mode=0, round_out=True), "bf16_mlp")
        util.assert_close(y[t], oracle.bf16_mlp(g, u, d, x[t], mode=1, round_out=True), "bf16_mlp vs ref_exact")


# up to 8 rows with room behind the vector: K in parts (wgemm_stream_takes_parts) for down only (gate and up below 32 MB, or 64 with
# one row), for both, and for neither (columns no multiple of 256); more: launches that add the parts
@pytest.mark.parametrize("hidden,ffn,T,more", [(1024, 4096, 1, 1), (1024, 4096, 8, 1), (2048, 4096, 2, 2), (4096, 4096, 1, 2), (2048, 2112, 3, 0),
                                               (288, 4128, 4, 0)])
def test_bf16_mlp_with_room_for_a_split(cuda, oracle, hidden, ffn, T, more):
    """With too little room, or where neither product takes parts, the bits are those of a workspace without room.  Nothing behind the
    workspace is touched.  The bars are those of the other forms: only the order of the fp32 sums differs."""
    from blok_b200 import lib
    rng = np.random.default_rng(hidden + ffn + T)
    g, u, d = _w(rng, ffn, hidden, 0.02), _w(rng, ffn, hidden, 0.02), _w(rng, hidden, ffn, 0.02)
    x = oracle.bf16_round(rng.normal(size=(T, hidden)).astype(np.float32))
    dg, du, dd, dx = (util.np_bf16_to_torch(g, cuda), util.np_bf16_to_torch(u, cuda), util.np_bf16_to_torch(d, cuda),
                      torch.from_numpy(x).to(cuda).bfloat16())
    vector = (ffn * T * 2 + 255) // 256 * 256

    def run(nbytes):
        ws = torch.full((nbytes + 4096,), 0x5A, dtype=torch.uint8, device=cuda)
        y = torch.empty((T, hidden), dtype=torch.bfloat16, device=cuda)
        lib._check(lib.load().blok_bf16_mlp(lib._ptr(dg), lib._ptr(du), lib._ptr(dd), lib._ptr(dx), lib._ptr(y), C.c_int(hidden), C.c_int(ffn),
                                            C.c_int(T), lib._ptr(ws), C.c_size_t(nbytes), lib._stream()))
        assert bool((ws[nbytes:] == 0x5A).all())
        return y

    def launches(nbytes):
        before = lib.kernel_launch_count()
        y = run(nbytes)
        return y, lib.kernel_launch_count() - before

    room = vector + 4 * T * 65536
    (plain, few), (split, many) = launches(ffn * T * 2), launches(room)
    assert many - few == more
    assert torch.equal(plain, lib.bf16_mlp(dg, du, dd, dx))
    yh = util.t2np_f32(split)
    for t in range(T):
        util.assert_close(yh[t], oracle.bf16_mlp(g, u, d, x[t], mode=0, round_out=True), "bf16_mlp")
    assert torch.equal(split, plain if more == 0 else run(room))
    assert torch.equal(plain, run(vector + 16))


@pytest.mark.parametrize("n,T", [(7168, 1), (1536, 4), (512, 8)])
def test_rmsnorm(cuda, oracle, n, T):
    from blok_b200 import lib
    rng = np.random.default_rng(n)
    x = oracle.bf16_round(rng.normal(0, 2.0, (T, n)).astype(np.float32))
    w = util.f32_to_bf16_np(rng.normal(1, 0.2, n).astype(np.float32))
    y = util.t2np_f32(lib.rmsnorm(torch.from_numpy(x).to(cuda).bfloat16(), util.np_bf16_to_torch(w, cuda), 1e-5))
    for t in range(T):
        exact = oracle.rmsnorm(x[t], w, 1e-5, mode=1)
        assert np.mean(y[t] == exact) > 0.98 and util.max_abs_rel(y[t], exact) < 1e-2


def test_add_round(cuda, oracle):
    from blok_b200 import lib
    rng = np.random.default_rng(0)
    a = oracle.bf16_round(rng.normal(size=7168).astype(np.float32))
    b = oracle.bf16_round(rng.normal(size=7168).astype(np.float32))
    da = torch.from_numpy(a).to(cuda).bfloat16()
    lib.add_(da, torch.from_numpy(b).to(cuda).bfloat16())
    assert np.array_equal(util.t2np_f32(da), oracle.add_round(a, b))


# A token is "ambiguous" when its 8th and 9th selection scores are closer than fp32
# summation-order noise of the logits; index parity is required on every other token.
MARGIN = 2e-6


@pytest.mark.parametrize("T,experts,hidden,topk,seed", [(1, 384, 7168, 8, 1), (64, 384, 7168, 8, 2), (300, 384, 7168, 8, 3),
                                                        (5, 48, 64, 8, 4), (9, 16, 256, 4, 5)])
def test_router_ids_bit_exact(cuda, oracle, T, experts, hidden, topk, seed):
    from blok_b200 import lib
    rng = np.random.default_rng(seed)
    wr = _w(rng, experts, hidden)
    bias = rng.normal(0, 0.01, experts).astype(np.float32)
    x = oracle.bf16_round(rng.normal(size=(T, hidden)).astype(np.float32))
    ids, wts = lib.router(util.np_bf16_to_torch(wr, cuda), torch.from_numpy(bias).to(cuda),
                          torch.from_numpy(x).to(cuda).bfloat16(), topk=topk, routed_scale=2.827)
    ids, wts = util.ids_np(ids), util.t2np_f32(wts)
    oid, owt, margin, _ = oracle.router(wr, bias, x, topk=topk, routed_scale=2.827, mode=0)
    clear = margin > MARGIN
    assert clear.mean() > 0.98
    # order inside the top-k can also flip on near-ties between selected experts: compare sets, then order where gaps are clear
    for t in np.nonzero(clear)[0]:
        assert set(ids[t].tolist()) == set(oid[t].tolist()), "token %d" % t
    same_order = np.all(ids == oid, axis=1)
    assert same_order[clear].mean() > 0.98
    sel = same_order & clear
    np.testing.assert_allclose(wts[sel], owt[sel], rtol=2e-5)
    np.testing.assert_allclose(wts.sum(axis=1), 2.827, rtol=1e-5)


def test_router_tie_rule_on_device(cuda):
    """All logits equal: the selection must be by bias, ties to the lowest index, output in descending order."""
    from blok_b200 import lib
    experts, hidden = 384, 256
    wr = torch.zeros((experts, hidden), dtype=torch.bfloat16, device=cuda)
    bias = torch.zeros(experts, dtype=torch.float32, device=cuda)
    bias[[300, 17, 200]] = 0.25
    bias[5] = 0.5
    x = torch.ones((2, hidden), dtype=torch.bfloat16, device=cuda)
    ids, wts = lib.router(wr, bias, x, topk=8, routed_scale=2.827)
    for t in range(2):
        assert util.ids_np(ids)[t].tolist() == [5, 17, 200, 300, 0, 1, 2, 3]
    np.testing.assert_allclose(util.t2np_f32(wts), 2.827 / 8, rtol=1e-6)


@pytest.mark.parametrize("vocab,hidden,T", [(163840, 7168, 1), (4096, 512, 3), (4096, 512, 40), (163840, 7168, 64)])
def test_lm_head_argmax_and_embed(cuda, oracle, vocab, hidden, T):
    from blok_b200 import lib
    g = torch.Generator(device=cuda).manual_seed(vocab)
    w = (torch.randn((vocab, hidden), generator=g, device=cuda) * 0.006).bfloat16()
    ids_in = torch.randint(0, vocab, (T,), generator=g, device=cuda, dtype=torch.int32)
    x = lib.embed(w, ids_in)
    assert torch.equal(x, w[ids_in.long()])
    # a query aligned with its own row must select that row; identical rows resolve to the lowest id
    w[vocab - 5] = w[17]
    n = (w[torch.tensor([17] + [int(i) for i in ids_in[1:]], device=cuda)].float() * 50).bfloat16()
    got = lib.lm_head_argmax(w, n).cpu().numpy()
    assert got[0] == 17
    if T > 8:  # the rows of a large call and the same rows 8 at a time select the same ids
        by8 = torch.cat([lib.lm_head_argmax(w, n[b:b + 8]) for b in range(0, T, 8)]).cpu().numpy()
        assert (got == by8).all()
    if vocab <= 4096:
        wh, nh = util.t2np_bf16(w), util.t2np_f32(n)
        for t in range(T):
            tok, _ = oracle.lm_head_argmax(wh, nh[t], mode=0)
            assert got[t] == tok


@pytest.mark.parametrize("T,n", [(1, 7168), (8, 7168), (3, 1536), (2, 100)])
def test_add_rmsnorm_is_add_then_rmsnorm(cuda, T, n):
    """The fused residual add + norm equals the two separate calls bit for bit (rows in registers or the element loop)."""
    from blok_b200 import lib, synth
    x = synth.activations(T, n, cuda, 61)
    t = synth.activations(T, n, cuda, 62)
    w = (synth.activations(1, n, cuda, 63)[0].float() * 0.1 + 1).bfloat16()
    x_ref = x.clone()
    lib.add_(x_ref, t)
    y_ref = lib.rmsnorm(x_ref, w, eps=1e-5)
    x_got = x.clone()
    y = lib.add_rmsnorm(x_got, t, w, eps=1e-5)
    assert torch.equal(x_got, x_ref) and torch.equal(y, y_ref)
    assert torch.equal(x_ref, (x.float() + t.float()).bfloat16())


@pytest.mark.parametrize("cols,T", [(6784, 3), (7168, 3), (8000, 3), (5056, 4), (2560, 8), (24576, 1)])
def test_staged_rows_around_the_shared_memory_limit(cuda, cols, T):
    """Rows of x that fill 40 to 48 KB of shared memory: with the kernels' static arrays more than a launch gets without asking."""
    from blok_b200 import lib, synth
    g = torch.Generator(device=cuda).manual_seed(cols)
    w = (torch.randn((64, cols), generator=g, device=cuda) / cols ** 0.5).bfloat16()
    x = synth.activations(T, cols, cuda, 5)
    want = x.double() @ w.double().T
    got = lib.bf16_gemv(w, x, out_f32=True)
    assert float((got.double() - want).norm() / want.norm()) < 1e-5  # fp32 sums
    y = lib.bf16_mlp(w, w, w.T.contiguous(), x)
    mid = want * torch.sigmoid(want) * want
    ref = mid @ w.double()
    assert float((y.double() - ref).norm() / ref.norm()) < 1e-2      # five roundings to bf16
