"""The work that programs built on this library have it do, as cases that can be timed and checked.

A case is a dict of plain values with a "kind":

  expert   one INT4 expert over one token (lib.expert_ffn)
  decode   the routed-MoE layer over one token (MoeLayer.decode)
  layer    the same layer over T tokens (MoeLayer.batched)
  attend   the MLA block of one layer for a batch of sequences, dense latent cache (MlaLayer.decode)
  paged    the same over a page pool with a block table (MlaLayer.decode_paged)
  chunk    the MLA block over a chunk of a prompt (MlaLayer.prefill)
  step     decode steps of a Kimi model of a dense and a MoE layer (Model.step)
  prompt   a prompt through a Pamopel model opened from a folder, logits at four places (Model.extend)

Sizes are Kimi K2's ("kimi") and those of the benchmark's small models ("small"); weights and activations have the
distributions of the benchmark's configurations.
"""
import json
import math
import os
import struct
import tempfile

import numpy as np
import torch

from blok_b200 import lib

SIZES = {"kimi": dict(hidden=7168, inter=2048, experts=384, shared=2048), "small": dict(hidden=2048, inter=1024, experts=128, shared=1024)}
TOPK, ROUTED_SCALE = 8, 2.827
HEADS, NOPE, ROPE, VHEAD, QRANK, KVRANK = 64, 128, 64, 128, 1536, 512
LAT = KVRANK + ROPE
THETA, YARN, EPS = 50000.0, 32.0, 1e-5
MODEL_YARN = 64.0  # the Kimi model's own default
PAGE = 64
STEP_VOCAB, DENSE_INTER = 32768, 18432

# the benchmark's small Pamopel model: state space, attention, attention that borrows its keys and values, state space
PW, PV, PFF, PBUCKETS, PBIAS = 2048, 32768, 8192, 8191, 32


def listed():
    return [
        # one routed expert for one token: the smallest call, a building block of other executors
        dict(name="expert_one", kind="expert", size="kimi"),
        # the layer a token passes 60 times per decode step
        dict(name="decode_one", kind="decode", size="kimi"),
        # a handful of sequences, or the tokens of a speculative step
        dict(name="layer_6", kind="layer", size="kimi", tokens=6),
        # a serving batch
        dict(name="layer_64", kind="layer", size="kimi", tokens=64),
        # an odd mixture of prompt tokens and decoding sequences
        dict(name="layer_517", kind="layer", size="kimi", tokens=517),
        # a prompt's chunk, or several prompts together
        dict(name="layer_2048", kind="layer", size="kimi", tokens=2048),
        # one interactive sequence
        dict(name="attend_1", kind="attend", batch=1, ctx=4001, ragged=False),
        # long documents
        dict(name="attend_8_long", kind="attend", batch=8, ctx=32768, ragged=False),
        # continuous batching: sequences of different lengths in a page pool
        dict(name="paged_33", kind="paged", batch=33, ctx=6000, ragged=True),
        # the largest chunk of a prompt the block takes, in the middle of the prompt
        dict(name="chunk_64", kind="chunk", tokens=64, first=1987),
        # greedy decoding of one sequence: embedding, dense layer, MoE layer, norms, vocabulary, graph replay
        dict(name="step_one", kind="step", batch=1, steps=4),
        # scoring a prompt
        dict(name="prompt_1000", kind="prompt", tokens=1000),
    ]


def log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["expert", "decode", "layer", "layer", "layer", "layer", "layer", "attend", "attend", "attend", "paged", "paged", "chunk", "step", "prompt"])
    size = rng.choice(["kimi", "kimi", "small"])
    if kind == "expert":  # other experts' sizes as well: multiples of 256
        return dict(kind=kind, size="", hidden=256 * rng.randint(4, 28), inter=256 * rng.randint(2, 12))
    if kind == "decode":
        return dict(kind=kind, size=size, topk=rng.choice([4, 6, 8]))
    if kind == "layer":
        return dict(kind=kind, size=size, tokens=log_uniform(rng, 2, 2040))
    if kind in ("attend", "paged"):
        batch = log_uniform(rng, 1, 64)
        return dict(kind=kind, batch=batch, ctx=log_uniform(rng, 100, min(32000, 250000 // batch)), ragged=rng.random() < 0.5)
    if kind == "chunk":
        return dict(kind=kind, tokens=log_uniform(rng, 2, 63), first=log_uniform(rng, 1, 12000))
    if kind == "step":
        return dict(kind=kind, batch=log_uniform(rng, 1, 48), steps=rng.randint(2, 4))
    return dict(kind=kind, tokens=log_uniform(rng, 40, 2040))


# ---- inputs --------------------------------------------------------------------------------------------------------------

DEV = "cuda"


def source(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(1000003 * int(seed) + 17)
    return g


def normal(g, shape, std=1.0, dtype=torch.bfloat16):
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.float32).mul_(std).to(dtype)


def words(g, shape):
    """Eight uniform nibbles per word."""
    return torch.randint(-(1 << 31), 1 << 31, shape, generator=g, device=DEV, dtype=torch.int32)


def quantised(g, n, rows, cols):
    lead = (n,) if n else ()
    return words(g, lead + (rows, cols // 8)), normal(g, lead + (rows, cols // 32), 0.003).abs()


def expert_inputs(c, seed):
    s = SIZES.get(c["size"]) or c
    H, I, g = s["hidden"], s["inter"], source(seed)
    w = [*quantised(g, 0, I, H), *quantised(g, 0, I, H), *quantised(g, 0, H, I)]
    return w, normal(g, (H,))


def moe_inputs(c, seed, tokens):
    s, g = SIZES[c["size"]], source(seed)
    H, I, E, S = s["hidden"], s["inter"], s["experts"], s["shared"]
    w = dict(router_w=normal(g, (E, H), 0.006), router_bias=normal(g, (E,), 0.01, torch.float32))
    for name, r, k in (("gate", I, H), ("up", I, H), ("down", H, I)):
        w[name + "_w"], w[name + "_s"] = quantised(g, E, r, k)
    w.update(shared_gate=normal(g, (S, H), 0.006), shared_up=normal(g, (S, H), 0.006), shared_down=normal(g, (H, S), 0.006))
    return w, normal(g, (tokens, H) if tokens else (H,))


def mla_inputs(c, seed, entries):
    g, H = source(seed), SIZES["kimi"]["hidden"]
    w = dict(q_a=normal(g, (QRANK, H), 0.006), q_b=normal(g, (HEADS * (NOPE + ROPE), QRANK), 0.006), kv_a=normal(g, (LAT, H), 0.006),
             kv_b=normal(g, (HEADS * (NOPE + VHEAD), KVRANK), 0.006), o=normal(g, (H, HEADS * VHEAD), 0.006),
             q_a_ln=torch.ones(QRANK, device=DEV, dtype=torch.bfloat16), kv_a_ln=torch.ones(KVRANK, device=DEV, dtype=torch.bfloat16))
    return w, normal(g, (entries, H)), g


def lengths(c, g):
    """Tokens cached per sequence; the step's own token comes on top."""
    B, ctx = c["batch"], c["ctx"]
    if not c["ragged"]:
        return torch.full((B,), ctx - 1, device=DEV, dtype=torch.int32)
    return torch.randint(ctx // 4, ctx, (B,), generator=g, device=DEV, dtype=torch.int64).to(torch.int32)


def page_numbers(c, g):
    stride = (c["ctx"] + PAGE - 1) // PAGE
    return torch.randperm(c["batch"] * stride, generator=g, device=DEV).to(torch.int32).reshape(c["batch"], stride)


def pamopel_config():
    mlp = {"kind": "dense", "ff": PFF}
    state = {"heads": 64, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1}
    attn = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "bias_max": 128}
    return {"architecture": "Pamopel", "width": PW, "vocab": PV, "norm": {"eps": EPS}, "residual_mult": 0.5, "logit_scale": 1.0,
            "embedding": {"scale": 1.0, "bigram": {"buckets": PBUCKETS, "mul_prev": 1009, "mul_cur": 17}},
            "layers": [{"type": "mamba2", "mixer": state, "mlp": mlp}, {"type": "attention", "mixer": attn, "mlp": mlp},
                       {"type": "attention", "mixer": dict(attn, kv_from=1), "mlp": mlp}, {"type": "mamba2", "mixer": state, "mlp": mlp}]}


def pamopel_weights(seed):
    g, t = source(seed), {}

    def mat(name, r, k, gain=1.0):
        t[name] = normal(g, (r, k), gain / math.sqrt(k))

    def vec(name, n, mean=1.0, dev=0.1):
        t[name] = (mean + dev * torch.randn((n,), generator=g, device=DEV)).to(torch.bfloat16)

    mat("embed", PV, PW, math.sqrt(PW))
    mat("bigram", PBUCKETS + 1, PW, math.sqrt(PW))
    for i, L in enumerate(pamopel_config()["layers"]):
        p, m = "l%d." % i, L["mixer"]
        for n in ("norm1", "norm1b", "norm2", "norm2b"):
            vec(p + n, PW)
        if L["type"] == "mamba2":
            inner, bc = m["heads"] * m["vdim"], m["groups"] * m["state"]
            mat(p + "mix.in", 2 * inner + 2 * bc + m["heads"], PW)
            mat(p + "mix.conv", inner + 2 * bc, m["conv"])
            vec(p + "mix.conv.b", inner + 2 * bc, 0.1)
            vec(p + "mix.dt_bias", m["heads"], -2.0, 1.0)
            vec(p + "mix.A_log", m["heads"], 0.3, 0.5)
            vec(p + "mix.D", m["heads"], 0.8, 0.3)
            vec(p + "mix.norm", inner)
            mat(p + "mix.o", PW, inner)
        else:
            hd, kd = m["heads"] * m["dim"], m["kv_heads"] * m["dim"]
            mat(p + "mix.q", hd, PW)
            vec(p + "mix.q.norm", hd)
            if "kv_from" not in m:
                mat(p + "mix.k", kd, PW)
                vec(p + "mix.k.norm", kd)
                mat(p + "mix.v", m["kv_heads"] * m["vdim"], PW)
            t[p + "mix.rel"] = normal(g, (PBIAS, m["heads"]))
            mat(p + "mix.g", m["heads"], PW)
            mat(p + "mix.o", PW, m["heads"] * m["vdim"])
        mat(p + "mlp.gate", PFF, PW)
        mat(p + "mlp.up", PFF, PW)
        mat(p + "mlp.down", PW, PFF)
    vec("final.norm", PW)
    mat("head", PV, PW)
    return t


def prompt_tokens(c, seed):
    return np.random.RandomState(seed % (1 << 31)).randint(0, PV, c["tokens"]), sorted({0, c["tokens"] // 3, c["tokens"] // 2, c["tokens"] - 1})


def write_model(folder, tensors):
    head, at = {}, 0
    for name, a in tensors.items():
        n = 2 * a.numel()
        head[name] = {"dtype": "BF16", "shape": list(a.shape), "data_offsets": [at, at + n]}
        at += n
    h = json.dumps(head).encode()
    h += b" " * (-len(h) % 8)
    with open(os.path.join(folder, "config.json"), "w") as f:
        json.dump(pamopel_config(), f)
    with open(os.path.join(folder, "model.safetensors"), "wb") as f:
        f.write(struct.pack("<Q", len(h)) + h)
        for a in tensors.values():
            a.contiguous().view(torch.int16).cpu().numpy().tofile(f)


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = dict(case=c)
    if kind == "expert":
        s["w"], s["x"] = expert_inputs(c, seed)
    elif kind in ("decode", "layer"):
        w, s["x"] = moe_inputs(c, seed, c.get("tokens", 0))
        s["layer"] = lib.MoeLayer(w, topk=c.get("topk", TOPK), routed_scale=ROUTED_SCALE, max_tokens=c.get("tokens", 1))
    elif kind in ("attend", "paged"):
        w, s["x"], g = mla_inputs(c, seed, c["batch"])
        s["layer"] = lib.MlaLayer(w, yarn_factor=YARN, rope_theta=THETA, rms_eps=EPS, max_batch=c["batch"], max_ctx=c["ctx"])
        s["len"] = lengths(c, g)
        if kind == "paged":
            s["table"] = page_numbers(c, g)
            s["cache"] = normal(g, (s["table"].numel(), PAGE, LAT))
        else:
            s["cache"] = normal(g, (c["batch"], c["ctx"], LAT))
    elif kind == "chunk":
        w, s["x"], g = mla_inputs(c, seed, c["tokens"])
        s["layer"] = lib.MlaLayer(w, yarn_factor=YARN, rope_theta=THETA, rms_eps=EPS, max_batch=c["tokens"], max_ctx=c["first"] + c["tokens"])
        s["cache"] = normal(g, (c["first"] + c["tokens"], LAT))
        s["first"] = torch.tensor([c["first"]], device=DEV, dtype=torch.int32)
    elif kind == "step":
        s["model"] = lib.Model(seed=seed, layers=2, first_dense=1, vocab=STEP_VOCAB, dense_inter=DENSE_INTER, max_batch=c["batch"], max_ctx=64)
        s["ids"] = step_ids(c, seed)
        s["stream"] = torch.cuda.Stream()
    else:
        with tempfile.TemporaryDirectory(dir="/dev/shm" if os.path.isdir("/dev/shm") else None) as folder:
            write_model(folder, pamopel_weights(seed))
            s["model"] = lib.Model.open(folder, max_batch=1, max_ctx=2048, prefill_chunk=2048)
        s["ids"], s["want"] = prompt_tokens(c, seed)
        s["stream"] = torch.cuda.Stream()
    return s


def step_ids(c, seed):
    g = source(seed)
    return [torch.randint(0, STEP_VOCAB, (c["batch"],), generator=g, device=DEV).to(torch.int32) for _ in range(c["steps"])]


def run(state):
    s, kind = state, state["case"]["kind"]
    if kind == "expert":
        return lib.expert_ffn(*s["w"], s["x"])
    if kind == "decode":
        return s["layer"].decode(s["x"])
    if kind == "layer":
        return s["layer"].batched(s["x"])
    if kind == "attend":
        return s["layer"].decode(s["x"], s["cache"], s["len"]), s["cache"]
    if kind == "paged":
        return s["layer"].decode_paged(s["x"], s["cache"], s["table"], s["len"]), s["cache"]
    if kind == "chunk":
        return s["layer"].prefill(s["x"], s["cache"], s["first"]), s["cache"]
    with torch.cuda.stream(s["stream"]):
        m = s["model"]
        if kind == "step":  # a new sequence in every slot; the tokens are the program's own
            for b in range(s["case"]["batch"]):
                m.release_slot(b)
            for ids in s["ids"]:
                m.step(ids)
            return m.hidden(s["case"]["batch"])
        m.release_slot(0)
        return m.extend(0, s["ids"], s["want"])


# ---- what a pass cannot do without -----------------------------------------------------------------------------------------

def expert_bytes(H, I):
    return 3 * (H * I // 2 + H * I // 32 * 2)


def mla_work(B, rows):
    H = SIZES["kimi"]["hidden"]
    w = QRANK * H + HEADS * (NOPE + ROPE) * QRANK + LAT * H + HEADS * (NOPE + VHEAD) * KVRANK + H * HEADS * VHEAD
    return w, 2 * (w + 4 * H * B) + 2 * LAT * rows[0], 2 * B * w + 2 * rows[1] * HEADS * (LAT + KVRANK)


def moe_work(s, T, topk=TOPK):
    H, I, E, S = s["hidden"], s["inter"], s["experts"], s["shared"]
    touched = E * (1 - (1 - topk / E) ** T)
    return (touched * expert_bytes(H, I) + 2 * E * H + 4 * E + 6 * S * H + 4 * T * H, 2 * T * (3 * topk * H * I + 3 * H * S + E * H))


def work(case):
    c, kind = case, case["kind"]
    if kind == "expert":
        s = SIZES.get(c["size"]) or c
        return dict(bytes=expert_bytes(s["hidden"], s["inter"]) + 4 * s["hidden"], flops=6 * s["hidden"] * s["inter"])
    if kind in ("decode", "layer"):
        b, f = moe_work(SIZES[c["size"]], c.get("tokens", 1), c.get("topk", TOPK))
    elif kind in ("attend", "paged"):
        rows = c["batch"] * c["ctx"] * (0.625 if c["ragged"] else 1.0)
        _, b, f = mla_work(c["batch"], (rows, rows))
    elif kind == "chunk":
        _, b, f = mla_work(c["tokens"], (c["first"] + c["tokens"], c["tokens"] * (c["first"] + c["tokens"] / 2)))
    elif kind == "step":
        B, H = c["batch"], SIZES["kimi"]["hidden"]
        w, ab, af = mla_work(B, (B * 4, B * 4))
        mb, mf = moe_work(SIZES["kimi"], B)
        b, f = 2 * ab + mb + 6 * H * DENSE_INTER + 2 * STEP_VOCAB * H, 2 * af + mf + 6 * B * H * DENSE_INTER + 2 * B * STEP_VOCAB * H
        b, f = b * c["steps"], f * c["steps"]
    else:
        T, inner, bc = c["tokens"], 4096, 256
        dense = 2 * (PW * (3 * inner + bc + 64)) + 2 * 2 * PW * 2048 + 2 * PW * 512 + 2 * PW * 16 + 4 * 3 * PW * PFF
        b = 2 * dense + 2 * PV * PW + 4 * T * PW + 4 * 4 * PV
        f = 2 * T * dense + 2 * 2 * 2 * T * inner * 128 + 2 * T * T // 2 * 16 * 256 * 2 + 2 * 4 * PV * PW
    return dict(bytes=b, flops=f)


def tolerance(case):
    # against 64 bits: 0.0045 to 0.0055 for an expert or a layer (bf16 at every rounding point of the reference), 0.01 after
    # two layers' residuals, 0.0035 for the attention block and a prompt; two correct implementations differ by up to 1.4 times that
    return {"rel": {"expert": 1.5e-2, "decode": 1.5e-2, "layer": 1.5e-2, "step": 3e-2}.get(case["kind"], 1e-2)}


# ---- the same in 64 bits -----------------------------------------------------------------------------------------------------

def dequantised(w, s):
    """The weight the layout stands for, bf16(q * scale), in 64 bits."""
    q = torch.stack([((w >> (4 * k)) & 15) - 8 for k in range(8)], dim=-1).reshape(w.shape[0], -1).float()
    return (q * s.float().repeat_interleave(32, dim=1)).to(torch.bfloat16).double()


def silu(z):
    return z * torch.sigmoid(z)


def swiglu(gate, up, down, x):
    return (silu(x @ gate.T) * (x @ up.T)) @ down.T


def moe_exact(w, x, topk=TOPK):
    score = torch.sigmoid(x @ w["router_w"].double().T)
    ids = torch.topk(score + w["router_bias"].double(), topk, dim=-1).indices
    wt = score.gather(1, ids)
    wt = wt / wt.sum(1, keepdim=True) * ROUTED_SCALE
    y = swiglu(*(w[k].double() for k in ("shared_gate", "shared_up", "shared_down")), x)
    for e in ids.unique().tolist():
        t, k = (ids == e).nonzero(as_tuple=True)
        m = [dequantised(w[n + "_w"][e], w[n + "_s"][e]) for n in ("gate", "up", "down")]
        y.index_add_(0, t, swiglu(*m, x[t]) * wt[t, k][:, None])
    return y


def rms(x, w, eps=EPS):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w.double()


def rotate(x, pos, factor):
    """x [..., ROPE] with pairs (2p, 2p + 1), its first axis over pos -> the rotated halves."""
    half = ROPE // 2

    def place(rotations):
        return ROPE * math.log(4096.0 / (rotations * 2 * math.pi)) / (2 * math.log(THETA))

    low, high = max(math.floor(place(32.0)), 0), min(math.ceil(place(1.0)), ROPE - 1)
    p = torch.arange(half, device=x.device, dtype=torch.float64)
    fast = THETA ** (-2 * p / ROPE)
    ramp = ((p - low) / (high - low)).clamp(0, 1)
    ang = pos.double()[:, None] * (fast / factor * ramp + fast * (1 - ramp))
    shape = (len(pos),) + (1,) * (x.dim() - 2) + (half,)
    co, si = ang.cos().reshape(shape), ang.sin().reshape(shape)
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.cat([a * co - b * si, b * co + a * si], dim=-1)


def mla_exact(w, n, pos, rows_of, factor=YARN):
    """n [B, hidden] at positions pos; rows_of(b, new rows) -> the cached rows entry b sees; returns (out, new rows)."""
    w = {k: v.double() for k, v in w.items()}
    B = n.shape[0]
    q = (rms(n @ w["q_a"].T, w["q_a_ln"]) @ w["q_b"].T).reshape(B, HEADS, NOPE + ROPE)
    kv = n @ w["kv_a"].T
    new = torch.cat([rms(kv[:, :KVRANK], w["kv_a_ln"]), rotate(kv[:, KVRANK:], pos, factor)], dim=1)
    kvb = w["kv_b"].reshape(HEADS, NOPE + VHEAD, KVRANK)
    qf = torch.cat([torch.einsum("bhd,hdj->bhj", q[..., :NOPE], kvb[:, :NOPE]), rotate(q[..., NOPE:], pos, factor)], dim=-1)
    scale = (0.1 * math.log(factor) + 1) ** 2 / math.sqrt(NOPE + ROPE)
    o = torch.stack([torch.softmax(qf[b] @ r.T * scale, dim=-1) @ r[:, :KVRANK] for b in range(B) for r in [rows_of(b, new)]])
    return torch.einsum("bhj,hvj->bhv", o, kvb[:, NOPE:]).reshape(B, -1) @ w["o"].T, new


def attend_exact(c, seed):
    w, x, g = mla_inputs(c, seed, c["batch"])
    pos = lengths(c, g)
    if c["kind"] == "paged":
        table = page_numbers(c, g).long()
        cache = normal(g, (table.numel(), PAGE, LAT))
        at = torch.gather(table, 1, (pos.long() // PAGE)[:, None])[:, 0], pos.long() % PAGE
        rows = lambda b: cache[table[b]].reshape(-1, LAT)[: int(pos[b])].double()  # noqa: E731
    else:
        cache = normal(g, (c["batch"], c["ctx"], LAT))
        at = torch.arange(c["batch"], device=DEV), pos.long()
        rows = lambda b: cache[b, : int(pos[b])].double()  # noqa: E731
    out, new = mla_exact(w, x.double(), pos, lambda b, new: torch.cat([rows(b), new[b:b + 1]]))
    full = cache.double()
    full[at] = new
    return out, full


def chunk_exact(c, seed):
    w, x, g = mla_inputs(c, seed, c["tokens"])
    cache = normal(g, (c["first"] + c["tokens"], LAT)).double()
    pos = c["first"] + torch.arange(c["tokens"], device=DEV)
    out, new = mla_exact(w, x.double(), pos, lambda b, new: torch.cat([cache[: c["first"]], new[: b + 1]]))
    cache[c["first"]:] = new
    return out, cache


def step_exact(c, seed):
    m = lib.Model(seed=seed, layers=2, first_dense=1, vocab=STEP_VOCAB, dense_inter=DENSE_INTER, max_batch=c["batch"], max_ctx=64)
    H, s = SIZES["kimi"]["hidden"], SIZES["kimi"]

    def get(layer, name, shape, dtype=torch.bfloat16):
        return torch.from_numpy(m.tensor(layer, name, np.int16 if dtype == torch.bfloat16 else np.int32)).to(DEV).view(dtype).reshape(shape)

    def block(l):
        return dict(q_a=get(l, "q_a_proj", (QRANK, H)), q_a_ln=get(l, "q_a_layernorm", (QRANK,)), q_b=get(l, "q_b_proj", (-1, QRANK)),
                    kv_a=get(l, "kv_a_proj_with_mqa", (LAT, H)), kv_a_ln=get(l, "kv_a_layernorm", (KVRANK,)), kv_b=get(l, "kv_b_proj", (-1, KVRANK)),
                    o=get(l, "o_proj", (H, -1)))

    ids = torch.stack(step_ids(c, seed), dim=1).long()  # [B, steps]
    B, S = ids.shape
    embed = get(-1, "embed_tokens", (STEP_VOCAB, H))
    x = embed[ids].double().reshape(B * S, H)
    pos = torch.arange(S, device=DEV).repeat(B)
    for l in range(2):
        n = rms(x, get(l, "input_layernorm", (H,)))
        x = x + mla_exact(block(l), n, pos, lambda b, new: new[b - b % S: b + 1], MODEL_YARN)[0]
        n = rms(x, get(l, "post_attention_layernorm", (H,)))
        if l == 0:
            x = x + swiglu(*(get(0, k, sh).double() for k, sh in (("gate_proj", (-1, H)), ("up_proj", (-1, H)), ("down_proj", (H, -1)))), n)
        else:
            w = dict(router_w=get(1, "router", (-1, H)), router_bias=get(1, "router_bias", (-1,), torch.float32))
            for k, sh in (("shared_gate", (-1, H)), ("shared_up", (-1, H)), ("shared_down", (H, -1))):
                w[k] = get(1, k, sh)
            for k, r, cols in (("gate", s["inter"], H), ("up", s["inter"], H), ("down", H, s["inter"])):
                w[k + "_w"], w[k + "_s"] = get(1, k + "_w", (-1, r, cols // 8), torch.int32), get(1, k + "_s", (-1, r, cols // 32))
            x = x + moe_exact(w, n)
    out = rms(x, get(-1, "norm", (H,)))
    m.close()
    return out.reshape(B, S, H)[:, -1]


def layer_norm(x, w):
    d = x - x.mean(-1, keepdim=True)
    return d / torch.sqrt((d * d).mean(-1, keepdim=True) + EPS) * w


def mamba_exact(h, w, m):
    T, H, dv, N = len(h), m["heads"], m["vdim"], m["state"]
    inner = H * dv
    p = h @ w["in"].T
    z, xbc, dt = p[:, :inner], p[:, inner: 2 * inner + 2 * N], p[:, 2 * inner + 2 * N:]
    taps = w["conv"].shape[1]
    padded = torch.cat([xbc.new_zeros(taps - 1, xbc.shape[1]), xbc])
    xbc = silu(sum(padded[j: j + T] * w["conv"][:, j] for j in range(taps)) + w["conv.b"])
    x, Bm, Cm = xbc[:, :inner].reshape(T, H, dv), xbc[:, inner: inner + N], xbc[:, inner + N:]
    dt = torch.nn.functional.softplus(dt + w["dt_bias"])
    keep = torch.exp(-torch.exp(w["A_log"]) * dt)
    S, y = x.new_zeros(H, N, dv), torch.empty_like(x)
    for t in range(T):
        S = keep[t][:, None, None] * S + Bm[t][None, :, None] * (dt[t][:, None] * x[t])[:, None, :]
        y[t] = torch.einsum("hnv,n->hv", S, Cm[t])
    y = (y + w["D"][:, None] * x).reshape(T, inner)
    return (rms(y * silu(z), torch.ones(inner, device=DEV)) * w["norm"]) @ w["o"].T


def bucket(n, rows, top):
    half = rows // 2
    return n if n < half else min(rows - 1, half + math.floor(math.log(n / half) / math.log(top / half) * (rows - half)))


def grouped_exact(h, w, m, kv):
    T, H, G, d, dv = len(h), m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q = rms(h @ w["q"].T, w["q.norm"]).reshape(T, H, d)
    if kv is None:
        kv = rms(h @ w["k"].T, w["k.norm"]).reshape(T, G, d), (h @ w["v"].T).reshape(T, G, dv)
    of = torch.arange(H, device=DEV) // (H // G)
    by_distance = w["rel"][torch.tensor([bucket(n, len(w["rel"]), m["bias_max"]) for n in range(T)], device=DEV)]
    dist = torch.arange(T, device=DEV)[:, None] - torch.arange(T, device=DEV)[None]
    o = torch.empty(T, H, dv, device=DEV, dtype=torch.float64)
    for k in range(H):
        s = q[:, k] @ kv[0][:, of[k]].T * m["scale"] + by_distance[:, k][dist.clamp(min=0)]
        o[:, k] = torch.softmax(s.masked_fill(dist < 0, -math.inf), dim=-1) @ kv[1][:, of[k]]
    return (o * torch.sigmoid(h @ w["g"].T)[:, :, None]).reshape(T, H * dv) @ w["o"].T, kv


def prompt_exact(c, seed):
    cfg, t = pamopel_config(), {k: v.double() for k, v in pamopel_weights(seed).items()}
    ids, want = prompt_tokens(c, seed)
    b = cfg["embedding"]["bigram"]
    pair = [b["buckets"]] + [(int(ids[i - 1]) * b["mul_prev"] + int(ids[i]) * b["mul_cur"]) % b["buckets"] for i in range(1, len(ids))]
    i = torch.arange(PW, device=DEV)
    ang = torch.arange(len(ids), device=DEV, dtype=torch.float64)[:, None] * 10000.0 ** (-(i - i % 2).double() / PW)
    x = t["embed"][torch.as_tensor(ids, device=DEV)] + t["bigram"][torch.tensor(pair, device=DEV)] + torch.where(i % 2 == 1, ang.cos(), ang.sin())
    kept = {}
    for j, L in enumerate(cfg["layers"]):
        p = "l%d." % j
        w = {k[len(p) + 4:]: v for k, v in t.items() if k.startswith(p + "mix.")}
        h = layer_norm(x, t[p + "norm1"])
        if L["type"] == "mamba2":
            y = mamba_exact(h, w, L["mixer"])
        else:
            y, kept[j] = grouped_exact(h, w, L["mixer"], kept.get(L["mixer"].get("kv_from")))
        x = x + cfg["residual_mult"] * layer_norm(y, t[p + "norm1b"])
        y = swiglu(t[p + "mlp.gate"], t[p + "mlp.up"], t[p + "mlp.down"], layer_norm(x, t[p + "norm2"]))
        x = x + cfg["residual_mult"] * layer_norm(y, t[p + "norm2b"])
    return (layer_norm(x[want], t["final.norm"]) @ t["head"].T).cpu().numpy()


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "expert":
        w, x = expert_inputs(c, seed)
        return swiglu(dequantised(w[0], w[1]), dequantised(w[2], w[3]), dequantised(w[4], w[5]), x.double())
    if kind in ("decode", "layer"):
        w, x = moe_inputs(c, seed, c.get("tokens", 0))
        y = moe_exact(w, x.double().reshape(-1, x.shape[-1]), c.get("topk", TOPK))
        return y.reshape(x.shape)
    if kind in ("attend", "paged"):
        return attend_exact(c, seed)
    if kind == "chunk":
        return chunk_exact(c, seed)
    return step_exact(c, seed) if kind == "step" else prompt_exact(c, seed)
