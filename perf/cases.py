"""The work that a user of this framework has it do, as cases that can be timed and compared.

Every case is one pass through public entry points (`ops`, `engine.ModelRunner`, `models.build_runner`), with random
inputs and weights of the sizes that `synthetic.SHAPES`, the benches and the tests of this repository use.  `kind`:

  linears           the four quantised projections of one decoder layer (qkv, o, gate|up with SiLU, down)
  mlp               the fp16 feed-forward of one decoder layer over prompt rows
  decode_attention  paged attention of decoded tokens over a fp16, bf16 or e4m3 cache
  prefill_attention causal attention of prompt rows over the paged cache
  llama_step        a decode step of a whole quantised decoder (a few layers, full vocabulary): logits
  window_attention  windowed grouped-head attention of the hybrid decoders, prompts and decoded tokens
  latent_attention  compressed-KV attention of the hybrid decoders
  experts           routed experts of the hybrid decoders
  recurrence        gated delta rule / decayed linear attention of the hybrid decoders
  hybrid_step       a step of a whole hybrid decoder (Zalalix: windowed attention, decayed linear attention, dense
                    feed-forwards, four layers): logits

Sequences of a ragged case get their lengths from the case alone; values come from the seed.
"""
import math

import numpy as np
import torch

from vllm_rs_b200 import models, ops, synthetic
from vllm_rs_b200.engine import ModelRunner, QuantLinear

DEV = "cuda"
PAGE = 64
GROUP = 128


def listed():
    return [
        # one user chatting: the projections of a layer for a single token, where launches and latency count
        dict(name="linears_1_token", kind="linears", model="llama3-8b", fmt="awq", bits=4, rows=1),
        # the headline batch of the benchmark: 32 sequences decode together
        dict(name="linears_32_tokens", kind="linears", model="llama3-8b", fmt="awq", bits=4, rows=32),
        # an unquantised checkpoint reads a long prompt: most of the time to the first token goes here
        dict(name="mlp_prompt_4096", kind="mlp", model="llama3-8b", rows=4096),
        # the headline batch reads its caches
        dict(name="decode_attention_32x4096", kind="decode_attention", heads=32, kv_heads=8, dim=128, seqs=32, ctx=4096,
             cache="f16"),
        # three prompts of unlike lengths in one prefill step, one of them in a later portion
        dict(name="prefill_attention_8192", kind="prefill_attention", heads=32, kv_heads=8, dim=128, seqs=3, rows=8192,
             past=512, dtype="f16"),
        # the whole decode step behind the headline number, on four of the layers
        dict(name="llama_step_32x4096", kind="llama_step", model="llama3-8b", layers=4, seqs=32, ctx=4096),
        # a long prompt through windowed attention with kept first tokens, capped scores, sink and head gate
        dict(name="window_prompt_4096", kind="window_attention", heads=16, kv_heads=4, dim=128, vdim=128, seqs=1, rows=4096,
             past=0, window=1024, keep_first=4, softcap=30.0, gate=True),
        # a batch that decodes through the same attention at the larger of the bench's widths
        dict(name="window_decode_32x2048", kind="window_attention", heads=32, kv_heads=8, dim=128, vdim=128, seqs=32,
             rows=32, past=2047, window=2048, keep_first=4, softcap=50.0, gate=False),
        # two prompts through latent attention at the larger width
        dict(name="latent_prompt_4096", kind="latent_attention", heads=32, kv_rank=512, rot_dim=32, seqs=2, rows=4096,
             past=0, window=2048, gate=False),
        # the tokens of a long prompt spread over routed experts
        dict(name="experts_prompt_4096", kind="experts", width=2048, ff=512, experts=16, top=4, rows=4096, act="silu_gate"),
        # a long prompt through the gated delta rule
        dict(name="delta_prompt_4096", kind="recurrence", rule="delta", heads=16, kv_heads=8, dim=128, vdim=128, seqs=1,
             rows=4096, past=0),
        # three prompts of unlike lengths through a whole hybrid decoder
        dict(name="hybrid_step_3001", kind="hybrid_step", seqs=3, rows=3001, past=0),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["linears", "mlp", "decode_attention", "prefill_attention", "llama_step", "window_attention",
                       "latent_attention", "experts", "recurrence", "hybrid_step"])
    c = dict(kind=kind)
    llama_heads = [(32, 8, 128), (32, 4, 64), (64, 8, 128)]
    if kind == "linears":
        fmt, bits = rng.choice([("awq", 4), ("awq", 4), ("gptq", 4), ("gptq", 8)])
        c.update(model=rng.choice(["tinyllama-1.1b", "llama3-8b", "llama3-70b"]), fmt=fmt, bits=bits,
                 rows=_log_int(rng, 1, 64))
    elif kind == "mlp":
        c.update(model=rng.choice(["tinyllama-1.1b", "llama3-8b"]), rows=_log_int(rng, 128, 4096))
    elif kind == "decode_attention":
        H, G, D = rng.choice(llama_heads)
        c.update(heads=H, kv_heads=G, dim=D, seqs=_log_int(rng, 1, 32), ctx=_log_int(rng, 64, 4096),
                 cache=rng.choice(["f16", "bf16", "fp8"]) if D == 128 else "f16")
    elif kind == "prefill_attention":
        H, G, D = rng.choice(llama_heads)
        rows = _log_int(rng, 256, 8192 if H == 32 else 5000)
        c.update(heads=H, kv_heads=G, dim=D, seqs=rng.randint(1, 4), rows=rows, past=rng.choice([0, 0, rng.randint(1, 512)]),
                 dtype=rng.choice(["f16", "bf16"]))
    elif kind == "llama_step":
        c.update(model=rng.choice(["tinyllama-1.1b", "llama3-8b"]), layers=rng.randint(2, 4), seqs=_log_int(rng, 1, 32),
                 ctx=_log_int(rng, 64, 4096))
    elif kind == "window_attention":
        H = rng.choice([16, 32])
        c.update(heads=H, kv_heads=H // 4, dim=128, vdim=128, window=rng.choice([0, 1024, 2048]),
                 keep_first=rng.choice([0, 4]), softcap=rng.choice([0.0, 30.0, 50.0]), gate=rng.random() < 0.5)
        if rng.random() < 0.5:
            c.update(seqs=rng.randint(1, 4), rows=_log_int(rng, 80, 4096), past=rng.choice([0, 0, rng.randint(1, 500)]))
        else:
            n = _log_int(rng, 1, 64)
            c.update(seqs=n, rows=n, past=_log_int(rng, 64, 2047))
    elif kind == "latent_attention":
        H, r = rng.choice([(16, 256), (32, 512)])
        c.update(heads=H, kv_rank=r, rot_dim=32, window=rng.choice([0, 1024, 2048]), gate=rng.random() < 0.5)
        if rng.random() < 0.5:
            c.update(seqs=rng.randint(1, 4), rows=_log_int(rng, 80, 3000), past=rng.choice([0, 0, rng.randint(1, 300)]))
        else:
            n = _log_int(rng, 1, 64)
            c.update(seqs=n, rows=n, past=_log_int(rng, 64, 2047))
    elif kind == "experts":
        D, F, E = rng.choice([(2048, 512, 16), (4096, 1024, 32)])
        c.update(width=D, ff=F, experts=E, top=4, rows=_log_int(rng, 1, 4096), act=rng.choice(["silu_gate", "relu2", "clamped"]))
    elif kind == "recurrence":
        rule = rng.choice(["delta", "decay"])
        H = rng.choice([16, 32]) if rule == "delta" else rng.choice([8, 16])
        c.update(rule=rule, heads=H, kv_heads=H // 2 if rule == "delta" else H, dim=128, vdim=128 if rule == "delta" else 256)
        if rng.random() < 0.6:
            c.update(seqs=rng.randint(1, 4), rows=_log_int(rng, 64, 4096), past=0)
        else:
            n = _log_int(rng, 1, 32)
            c.update(seqs=n, rows=n, past=rng.randint(1, 2000))
    else:
        if rng.random() < 0.5:
            c.update(seqs=rng.randint(1, 4), rows=_log_int(rng, 100, 3001), past=0)
        else:
            n = _log_int(rng, 1, 32)
            c.update(seqs=n, rows=n, past=_log_int(rng, 64, 2047))
    return c


# ------------------------------------------------------------------------------------------ shared pieces
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 13)


def _randn(g, *shape, dtype=torch.float32):
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float32).to(dtype)


def _i32(a):
    return torch.tensor(np.asarray(a).tolist(), dtype=torch.int32, device=DEV)


def _lens(c):
    """Rows that each sequence brings: 1 each for a batch that decodes, otherwise unlike lengths that sum to `rows`."""
    n, rows = c["seqs"], c["rows"]
    if rows == n:
        return [1] * n
    part = [rows * (i + 1) * 2 // (n * (n + 1)) for i in range(n)]
    part[-1] += rows - sum(part)
    return [max(1, p) for p in part]


def _pasts(c):
    """Tokens that lie in the cache before the step: unlike numbers up to `past`, the last sequence has all of them."""
    return [max(0, c["past"] - (37 * (c["seqs"] - 1 - i)) % (c["past"] // 3 + 1)) for i in range(c["seqs"])]


def _ctxs(c):
    return [max(1, c["ctx"] - (53 * i) % (c["ctx"] // 4 + 1)) for i in range(c["seqs"])]


def _tables(g, ctxs, spare=3):
    """A block table of scattered pages: (number of pages, [seqs, most pages] on the CPU)."""
    need = [-(-x // PAGE) for x in ctxs]
    total = sum(need) + spare
    perm = torch.randperm(total, generator=g, device=DEV).cpu()
    bt = torch.zeros(len(ctxs), max(need), dtype=torch.int32)
    at = 0
    for b, n in enumerate(need):
        bt[b, :n] = perm[at:at + n].int()
        at += n
    return total, bt


def _gather(cache, bt_row, n):
    """The first n rows of a sequence from a paged cache [pages, 64, ...], in 64 bits."""
    return cache[bt_row[:-(-n // PAGE)].long().to(DEV)].flatten(0, 1)[:n].double()


def _attend(q, k, v, first_pos, scale, window=0, keep_first=0, softcap=0.0, sink=None):
    """q [n, H, d] at positions first_pos .., k [m, G, d], v [m, G, e] -> [n, H, e], all in 64 bits."""
    n, H, _ = q.shape
    m, G = k.shape[0], k.shape[1]
    i = (first_pos + torch.arange(n, device=DEV))[:, None]
    j = torch.arange(m, device=DEV)[None, :]
    ok = j <= i
    if window:
        ok &= (i - j < window) | (j < keep_first)
    out = torch.empty(n, H, v.shape[2], dtype=torch.float64, device=DEV)
    for h in range(H):
        s = q[:, h] @ k[:, h * G // H].T * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        s = s.masked_fill(~ok, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].double().expand(n, 1)], 1)
        out[:, h] = torch.softmax(s, 1)[:, :m] @ v[:, h * G // H]
    return out


def _visible(c):
    """Pairs (row, key) that windowed attention sees, and keys that any row of a sequence sees."""
    pairs = keys = 0
    w, kf = c.get("window", 0), c.get("keep_first", 0)
    for n, p in zip(_lens(c), _pasts(c)):
        pos = np.arange(p, p + n)
        pairs += int(np.sum(np.minimum(pos + 1, w + np.minimum(kf, np.maximum(pos + 1 - w, 0))) if w else pos + 1))
        keys += min(p + n, n + w + kf) if w else p + n
    return pairs, keys


# ------------------------------------------------------------------------------------------ quantised checkpoints
_AWQ_ORDER = [0, 2, 4, 6, 1, 3, 5, 7]


def _raw_linear(g, fmt, bits, k, n):
    """Checkpoint tensors (qweight, qzeros, scales) of a random quantised projection."""
    pack = 32 // bits
    word = lambda *s: torch.randint(-2**31, 2**31 - 1, s, generator=g, device=DEV, dtype=torch.int32)   # noqa: E731
    s = ((torch.rand(k // GROUP, n, generator=g, device=DEV) + 0.5) * (2.0 / (2**bits - 1)) / math.sqrt(k)).half()
    if fmt == "awq":
        return word(k, n // 8), word(k // GROUP, n // 8), s
    # symmetric GPTQ: zero point 2^(bits-1), stored minus one
    z = 0x77777777 if bits == 4 else 0x7F7F7F7F
    return word(k // pack, n), torch.full((k // GROUP, n // pack), z, device=DEV, dtype=torch.int32), s


def _packed(raw, fmt, bits, k, n):
    w = ops.awq_prepack(raw[0]) if fmt == "awq" else ops.gptq_prepack(raw[0], bits)
    return QuantLinear(w.reshape(-1), raw[2], raw[1], k, n)


def _nibbles(w, bits):
    pack = 32 // bits
    return torch.stack([(w >> (bits * j)) & (2**bits - 1) for j in range(pack)], -1)


def _weight64(raw, fmt, bits):
    """The [k, n] matrix that the checkpoint tensors stand for, in 64 bits."""
    qw, qz, s = raw
    if fmt == "awq":
        inv = torch.tensor([_AWQ_ORDER.index(i) for i in range(8)], device=DEV)
        q = _nibbles(qw, 4)[..., inv].flatten(1)
        z = _nibbles(qz, 4)[..., inv].flatten(1)
    else:
        q = _nibbles(qw, bits).permute(0, 2, 1).flatten(0, 1)
        z = _nibbles(qz, bits).flatten(1) + 1
    out = torch.empty(q.shape, dtype=torch.float64, device=DEV)
    for a in range(0, q.shape[0], GROUP):
        out[a:a + GROUP] = (q[a:a + GROUP] - z[a // GROUP]).double() * s[a // GROUP].double()
    return out


def _projections(model):
    hidden, _, H, G, D, inter, _, _ = synthetic.SHAPES[model]
    return dict(qkv=(hidden, (H + 2 * G) * D), o=(H * D, hidden), gate_up=(hidden, 2 * inter), down=(inter, hidden))


# ------------------------------------------------------------------------------------------ linears, mlp
def _linears_inputs(c, seed):
    g = _gen(seed)
    p = _projections(c["model"])
    raw = {n: _raw_linear(g, c["fmt"], c["bits"], *kn) for n, kn in p.items()}
    return p, raw, _randn(g, c["rows"], p["qkv"][0], dtype=torch.float16), _randn(g, c["rows"], p["o"][0], dtype=torch.float16)


def _linears_prepare(c, seed):
    p, raw, x, a = _linears_inputs(c, seed)
    lin = {n: _packed(raw[n], c["fmt"], c["bits"], *p[n]) for n in p}
    ws = ops.wna16_workspace(max(c["rows"], 16), max(n for _, n in p.values()))
    return dict(lin=lin, x=x, a=a, ws=ws, bits=c["bits"], fmt=ops.QFMT_AWQ if c["fmt"] == "awq" else ops.QFMT_GPTQ)


def _linears_run(s):
    def lin(x, name, epi=ops.EPI_NONE):
        q = s["lin"][name]
        return ops.wna16_gemm(x, q.w, q.s, q.z, s["ws"], k=q.k, n=q.n, bits=s["bits"], group_size=GROUP, qfmt=s["fmt"],
                              epilogue=epi)
    qkv = lin(s["x"], "qkv")
    o = lin(s["a"], "o")
    act = lin(s["x"], "gate_up", ops.EPI_SILU_MUL)
    return [qkv, o, act, lin(act, "down")]


def _linears_exact(c, seed):
    p, raw, x, a = _linears_inputs(c, seed)
    w = lambda n: _weight64(raw[n], c["fmt"], c["bits"])         # noqa: E731
    qkv, o, gu = x.double() @ w("qkv"), a.double() @ w("o"), x.double() @ w("gate_up")
    gate, up = gu.chunk(2, 1)
    act = torch.nn.functional.silu(gate) * up
    return [qkv, o, act, act @ w("down")]


def _linears_work(c):
    p, m = _projections(c["model"]), c["rows"]
    kn = sum(k * n for k, n in p.values())
    io = m * 2 * (p["qkv"][0] + p["o"][0] + p["qkv"][1] + p["o"][1] + 2 * p["down"][0] + p["down"][1])
    return dict(bytes=kn * c["bits"] / 8 + kn / GROUP * (2 + c["bits"] / 8) + io, flops=2.0 * m * kn)


def _mlp_inputs(c, seed):
    g = _gen(seed)
    hidden, inter = synthetic.SHAPES[c["model"]][0], synthetic.SHAPES[c["model"]][5]
    f16 = torch.float16
    return ((_randn(g, 2 * inter, hidden) / math.sqrt(hidden)).to(f16), (_randn(g, hidden, inter) / math.sqrt(inter)).to(f16),
            _randn(g, c["rows"], hidden, dtype=f16))


def _mlp_prepare(c, seed):
    return _mlp_inputs(c, seed)


def _mlp_run(s):
    act = ops.silu_mul(ops.dense_gemm(s[2], s[0]))
    return [act, ops.dense_gemm(act, s[1])]


def _mlp_exact(c, seed):
    gu, dn, x = _mlp_inputs(c, seed)
    act = torch.empty(c["rows"], gu.shape[0] // 2, dtype=torch.float64, device=DEV)
    for a in range(0, c["rows"], 1024):
        gate, up = (x[a:a + 1024].double() @ gu.double().T).chunk(2, 1)
        act[a:a + 1024] = torch.nn.functional.silu(gate) * up
    return [act, act @ dn.double().T]


def _mlp_work(c):
    hidden, inter = synthetic.SHAPES[c["model"]][0], synthetic.SHAPES[c["model"]][5]
    return dict(bytes=3.0 * hidden * inter * 2 + c["rows"] * 2 * (2 * hidden + inter), flops=6.0 * c["rows"] * hidden * inter)


# ------------------------------------------------------------------------------------------ attention of the dense decoders
_CACHE = {"f16": torch.float16, "bf16": torch.bfloat16}


def _decode_inputs(c, seed):
    g, ctxs = _gen(seed), _ctxs(c)
    pages, bt = _tables(g, ctxs)
    dt = _CACHE.get(c["cache"], torch.float16)
    k, v = (torch.empty(pages, PAGE, c["kv_heads"], c["dim"], dtype=dt, device=DEV).normal_(generator=g) for _ in range(2))
    if c["cache"] == "fp8":
        k, v = (t.to(torch.float8_e4m3fn) for t in (k, v))
    return ctxs, bt, k, v, _randn(g, c["seqs"], c["heads"], c["dim"], dtype=dt)


def _decode_prepare(c, seed):
    ctxs, bt, k, v, q = _decode_inputs(c, seed)
    if c["cache"] == "fp8":
        k, v = k.view(torch.uint8), v.view(torch.uint8)
    ws = ops.paged_attn_workspace(c["seqs"], c["heads"], c["dim"], bt.shape[1])
    return dict(q=q, k=k, v=v, bt=bt.to(DEV), ctx=_i32(ctxs), ws=ws, scale=c["dim"] ** -0.5)


def _decode_run(s):
    return ops.paged_attention_decode(s["q"], s["k"], s["v"], s["bt"], s["ctx"], s["scale"], workspace=s["ws"])


def _decode_exact(c, seed):
    ctxs, bt, k, v, q = _decode_inputs(c, seed)
    return torch.cat([_attend(q[b:b + 1].double(), _gather(k, bt[b], n), _gather(v, bt[b], n), n - 1, c["dim"] ** -0.5)
                      for b, n in enumerate(ctxs)])


def _decode_work(c):
    keys = sum(_ctxs(c))
    e = 1 if c["cache"] == "fp8" else 2
    return dict(bytes=keys * c["kv_heads"] * c["dim"] * 2 * e + c["seqs"] * c["heads"] * c["dim"] * 4,
                flops=4.0 * keys * c["heads"] * c["dim"])


def _prefill_inputs(c, seed):
    g, dt = _gen(seed), _CACHE[c["dtype"]]
    lens, pasts = _lens(c), _pasts(c)
    ctxs = [a + b for a, b in zip(lens, pasts)]
    pages, bt = _tables(g, ctxs)
    k, v = (torch.empty(pages, PAGE, c["kv_heads"], c["dim"], dtype=dt, device=DEV).normal_(generator=g) for _ in range(2))
    return lens, pasts, ctxs, bt, k, v, _randn(g, sum(lens), c["heads"], c["dim"], dtype=dt)


def _prefill_prepare(c, seed):
    lens, pasts, ctxs, bt, k, v, q = _prefill_inputs(c, seed)
    return dict(q=q, k=k, v=v, bt=bt.to(DEV), ctx=_i32(ctxs), cu=_i32(np.cumsum([0] + lens)), longest=max(lens),
                scale=c["dim"] ** -0.5)


def _prefill_run(s):
    return ops.attention_prefill(s["q"], s["k"], s["v"], s["cu"], s["ctx"], s["bt"], s["longest"], s["scale"])


def _prefill_exact(c, seed):
    lens, pasts, ctxs, bt, k, v, q = _prefill_inputs(c, seed)
    at = np.cumsum([0] + lens)
    return torch.cat([_attend(q[at[b]:at[b + 1]].double(), _gather(k, bt[b], ctxs[b]), _gather(v, bt[b], ctxs[b]), pasts[b],
                              c["dim"] ** -0.5) for b in range(c["seqs"])])


def _prefill_work(c):
    pairs, keys = _visible(c)
    return dict(bytes=keys * c["kv_heads"] * c["dim"] * 4 + sum(_lens(c)) * c["heads"] * c["dim"] * 4,
                flops=4.0 * pairs * c["heads"] * c["dim"])


# ------------------------------------------------------------------------------------------ a whole dense decoder
_EPS = 1e-5


def _llama_inputs(c, seed):
    g = _gen(seed)
    hidden, _, H, G, D, inter, vocab, theta = synthetic.SHAPES[c["model"]]
    ctxs = _ctxs(c)
    pages, bt = _tables(g, ctxs)
    norm = lambda: (1 + 0.05 * _randn(g, hidden)).half()          # noqa: E731
    layers = []
    for _ in range(c["layers"]):
        w = {n: _raw_linear(g, "awq", 4, *kn) for n, kn in _projections(c["model"]).items()}
        w.update(n1=norm(), n2=norm(),
                 **{x: torch.empty(pages, PAGE, G, D, dtype=torch.float16, device=DEV).normal_(generator=g) for x in "kv"})
        layers.append(w)
    embed = _randn(g, vocab, hidden, dtype=torch.float16)
    head = (0.02 * _randn(g, vocab, hidden)).half()
    cos, sin = synthetic.rope_tables_device(D, 8192, theta, DEV)
    ids = torch.randint(0, vocab, (c["seqs"],), generator=g, device=DEV, dtype=torch.int32)
    pos = torch.tensor([n - 1 for n in ctxs])
    slots = torch.tensor([int(bt[b, (n - 1) // PAGE]) * PAGE + (n - 1) % PAGE for b, n in enumerate(ctxs)])
    return dict(layers=layers, embed=embed, head=head, fnorm=norm(), cos=cos, sin=sin, ids=ids, ctxs=ctxs, pages=pages, bt=bt,
                pos=pos.to(DEV), slots=slots.to(DEV))


def _llama_prepare(c, seed):
    hidden, _, H, G, D, inter, vocab, _ = synthetic.SHAPES[c["model"]]
    x = _llama_inputs(c, seed)
    r = ModelRunner(hidden=hidden, num_layers=c["layers"], num_heads=H, num_kv_heads=G, head_dim=D, inter=inter, vocab=vocab,
                    num_blocks=x["pages"], max_blocks_per_seq=x["bt"].shape[1], max_batch=c["seqs"], rms_eps=_EPS)
    proj = _projections(c["model"])
    for i, w in enumerate(x["layers"]):
        r.set_layer(i, input_norm=w["n1"], post_norm=w["n2"], **{n: _packed(w[n], "awq", 4, *proj[n]) for n in proj})
        r.k_cache[i].copy_(w["k"])
        r.v_cache[i].copy_(w["v"])
    r.set_globals(x["embed"], x["fnorm"], x["head"], x["cos"], x["sin"])
    return dict(r=r, ids=x["ids"], pos=x["pos"], slots=x["slots"], bt=x["bt"].to(DEV), ctx=_i32(x["ctxs"]))


def _llama_run(s):
    return s["r"].decode_device(s["ids"], s["pos"], s["slots"], s["bt"], s["ctx"])[0]


def _llama_exact(c, seed):
    _, _, H, G, D, _, _, _ = synthetic.SHAPES[c["model"]]
    x = _llama_inputs(c, seed)
    B = c["seqs"]
    unit = lambda t, w: t / torch.sqrt((t * t).mean(-1, keepdim=True) + _EPS) * w.double()      # noqa: E731
    cos, sin = (x[n].double()[x["pos"]][:, None, :] for n in ("cos", "sin"))

    def rope(t):                          # [B, heads, D], halves
        u, v = t.chunk(2, -1)
        return torch.cat([u * cos - v * sin, v * cos + u * sin], -1)

    h = x["embed"][x["ids"].long()].double()
    for w in x["layers"]:
        y = unit(h, w["n1"]) @ _weight64(w["qkv"], "awq", 4)
        q, k, v = y[:, :H * D].reshape(B, H, D), y[:, H * D:(H + G) * D].reshape(B, G, D), y[:, (H + G) * D:].reshape(B, G, D)
        q, k = rope(q), rope(k)
        o = []
        for b, n in enumerate(x["ctxs"]):
            ks, vs = _gather(w["k"], x["bt"][b], n), _gather(w["v"], x["bt"][b], n)
            ks[n - 1], vs[n - 1] = k[b], v[b]
            o.append(_attend(q[b:b + 1], ks, vs, n - 1, D ** -0.5))
        h = h + torch.cat(o).reshape(B, H * D) @ _weight64(w["o"], "awq", 4)
        gate, up = (unit(h, w["n2"]) @ _weight64(w["gate_up"], "awq", 4)).chunk(2, 1)
        h = h + (torch.nn.functional.silu(gate) * up) @ _weight64(w["down"], "awq", 4)
    return unit(h, x["fnorm"]) @ x["head"].double().T


def _llama_work(c):
    hidden, _, H, G, D, inter, vocab, _ = synthetic.SHAPES[c["model"]]
    keys, kn = sum(_ctxs(c)), sum(k * n for k, n in _projections(c["model"]).values())
    return dict(bytes=c["layers"] * (kn / 2 + kn / GROUP * 2.5 + keys * G * D * 4) + vocab * hidden * 2 + c["seqs"] * vocab * 4,
                flops=c["layers"] * (2.0 * c["seqs"] * kn + 4.0 * keys * H * D) + 2.0 * c["seqs"] * vocab * hidden)


# ------------------------------------------------------------------------------------------ attention of the hybrid decoders
def _window_inputs(c, seed):
    g = _gen(seed)
    lens, pasts = _lens(c), _pasts(c)
    ctxs = [a + b for a, b in zip(lens, pasts)]
    pages, bt = _tables(g, ctxs)
    k = _randn(g, pages, PAGE, c["kv_heads"], c["dim"], dtype=torch.bfloat16)
    v = _randn(g, pages, PAGE, c["kv_heads"], c["vdim"], dtype=torch.bfloat16)
    q = _randn(g, sum(lens), c["heads"], c["dim"])
    gate = _randn(g, sum(lens), c["heads"]) if c["gate"] else None
    return lens, pasts, ctxs, bt, k, v, q, gate, 0.5 * _randn(g, c["heads"])


def _window_prepare(c, seed):
    lens, pasts, ctxs, bt, k, v, q, gate, sink = _window_inputs(c, seed)
    return dict(q=q, k=k, v=v, gate=gate, sink=sink, bt=bt.to(DEV), ctx=_i32(ctxs), cu=_i32(np.cumsum([0] + lens)), case=c)


def _window_run(s):
    c = s["case"]
    return ops.window_attn(s["q"], s["k"], s["v"], s["sink"], s["gate"], s["cu"], s["ctx"], s["bt"], window=c["window"],
                           keep_first=c["keep_first"], scale=c["dim"] ** -0.5, softcap=c["softcap"])


def _window_exact(c, seed):
    lens, pasts, ctxs, bt, k, v, q, gate, sink = _window_inputs(c, seed)
    at = np.cumsum([0] + lens)
    out = torch.cat([_attend(q[at[b]:at[b + 1]].double(), _gather(k, bt[b], ctxs[b]), _gather(v, bt[b], ctxs[b]), pasts[b],
                             c["dim"] ** -0.5, c["window"], c["keep_first"], c["softcap"], sink) for b in range(c["seqs"])])
    return out if gate is None else out * torch.sigmoid(gate.double())[:, :, None]


def _window_work(c):
    pairs, keys = _visible(c)
    return dict(bytes=keys * c["kv_heads"] * (c["dim"] + c["vdim"]) * 2 + c["rows"] * c["heads"] * (c["dim"] * 4 + c["vdim"] * 2),
                flops=2.0 * pairs * c["heads"] * (c["dim"] + c["vdim"]))


def _latent_inputs(c, seed):
    g = _gen(seed)
    lens, pasts = _lens(c), _pasts(c)
    ctxs = [a + b for a, b in zip(lens, pasts)]
    pages, bt = _tables(g, ctxs)
    r, dr = c["kv_rank"], c["rot_dim"]
    cache = _randn(g, pages, PAGE, r + dr, dtype=torch.bfloat16)
    q = _randn(g, sum(lens), c["heads"], r + dr)
    q[..., :r] *= (64 / r) ** 0.5             # 64 unit entries through the absorbed key expansion
    gate = _randn(g, sum(lens), c["heads"]) if c["gate"] else None
    return lens, pasts, ctxs, bt, cache, q, gate, 0.5 * _randn(g, c["heads"])


def _latent_scale(c):
    return (64 + c["rot_dim"]) ** -0.5


def _latent_prepare(c, seed):
    lens, pasts, ctxs, bt, cache, q, gate, sink = _latent_inputs(c, seed)
    return dict(q=q, cache=cache, gate=gate, sink=sink, bt=bt.to(DEV), ctx=_i32(ctxs), cu=_i32(np.cumsum([0] + lens)), case=c)


def _latent_run(s):
    c = s["case"]
    return ops.latent_attn(s["q"], s["cache"], s["sink"], s["cu"], s["ctx"], s["bt"], kv_rank=c["kv_rank"],
                           rot_dim=c["rot_dim"], window=c["window"], scale=_latent_scale(c), gate=s["gate"])


def _latent_exact(c, seed):
    lens, pasts, ctxs, bt, cache, q, gate, sink = _latent_inputs(c, seed)
    at, out = np.cumsum([0] + lens), []
    for b in range(c["seqs"]):
        k = _gather(cache, bt[b], ctxs[b])[:, None, :]
        out.append(_attend(q[at[b]:at[b + 1]].double(), k, k[..., :c["kv_rank"]], pasts[b], _latent_scale(c), c["window"],
                           0, 0.0, sink))
    out = torch.cat(out)
    return out if gate is None else out * torch.sigmoid(gate.double())[:, :, None]


def _latent_work(c):
    pairs, keys = _visible(c)
    r, R = c["kv_rank"], c["kv_rank"] + c["rot_dim"]
    return dict(bytes=keys * R * 2 + c["rows"] * c["heads"] * (R * 4 + r * 2), flops=2.0 * pairs * c["heads"] * (R + r))


# ------------------------------------------------------------------------------------------ routed experts
_CLAMPED = dict(limit=7.0, alpha=1.702, up_add=1.0)


def _experts_inputs(c, seed):
    g = _gen(seed)
    D, F, E, T = c["width"], c["ff"], c["experts"], c["rows"]
    bf = torch.bfloat16
    h = _randn(g, T, D, dtype=bf)
    up = (_randn(g, E, F if c["act"] == "relu2" else 2 * F, D) / math.sqrt(D)).to(bf)
    down = (_randn(g, E, D, F) / math.sqrt(F)).to(bf)
    z = _randn(g, T, E) + 0.5 * _randn(g, E)           # some experts are more popular than others
    w, idx = torch.softmax(z, 1).topk(c["top"], 1)
    return h, up, down, idx.int().contiguous(), w.contiguous()


def _experts_prepare(c, seed):
    h, up, down, idx, w = _experts_inputs(c, seed)
    return dict(h=h, up=up, down=down, idx=idx, w=w, out=torch.zeros(c["rows"], c["width"], device=DEV), act=c["act"])


def _experts_run(s):
    kw = _CLAMPED if s["act"] == "clamped" else {}
    return ops.moe_experts_ex(s["out"], s["h"], s["idx"], s["w"], s["up"], s["down"], act=s["act"], accumulate=False, **kw)


def _experts_exact(c, seed):
    h, up, down, idx, w = _experts_inputs(c, seed)
    out = torch.zeros(c["rows"], c["width"], dtype=torch.float64, device=DEV)
    for e in range(c["experts"]):
        t, j = (idx == e).nonzero(as_tuple=True)
        y = h[t].double() @ up[e].double().T
        if c["act"] == "relu2":
            y = torch.relu(y) ** 2
        else:
            gate, u = y.chunk(2, 1)
            if c["act"] == "clamped":
                gate, u = gate.clamp(max=_CLAMPED["limit"]), u.clamp(-_CLAMPED["limit"], _CLAMPED["limit"])
                y = gate * torch.sigmoid(_CLAMPED["alpha"] * gate) * (u + _CLAMPED["up_add"])
            else:
                y = torch.nn.functional.silu(gate) * u
        out.index_add_(0, t, w[t, j].double()[:, None] * (y @ down[e].double().T))
    return out


def _experts_work(c):
    D, F, T, top = c["width"], c["ff"], c["rows"], c["top"]
    mats = 2 if c["act"] == "relu2" else 3
    return dict(bytes=min(c["experts"], T * top) * mats * D * F * 2.0 + T * D * 6, flops=2.0 * T * top * mats * D * F)


# ------------------------------------------------------------------------------------------ recurrences
def _recurrence_inputs(c, seed):
    g, T = _gen(seed), c["rows"]
    H, G, dk, dv = c["heads"], c["kv_heads"], c["dim"], c["vdim"]
    x = dict(q=_randn(g, T, G, dk), k=_randn(g, T, G, dk), v=_randn(g, T, H, dv),
             state=0.3 * _randn(g, c["seqs"], H, dk, dv), slots=torch.randperm(c["seqs"], generator=g, device=DEV).int())
    if c["rule"] == "delta":
        x.update(b=_randn(g, T, H), a=_randn(g, T, H), a_log=-0.5 + 0.5 * _randn(g, H), dtb=-1.0 + 0.5 * _randn(g, H))
    else:
        x["decay"] = 1.0 - torch.exp2(-(5.0 + torch.arange(H, device=DEV) % 4))
    return x


def _recurrence_prepare(c, seed):
    x = _recurrence_inputs(c, seed)
    lens, pasts = _lens(c), _pasts(c)
    return dict(x, cu=_i32(np.cumsum([0] + lens)), ctx=_i32([a + b for a, b in zip(lens, pasts)]), case=c)


def _recurrence_run(s):
    if s["case"]["rule"] == "delta":
        o = ops.delta_rule(s["q"], s["k"], s["v"], s["b"], s["a"], s["a_log"], s["dtb"], s["state"], s["slots"], s["cu"], s["ctx"])
    else:
        o = ops.decay_attn(s["q"], s["k"], s["v"], s["state"], s["slots"], s["cu"], s["ctx"], head_decay=s["decay"],
                           k_scale=s["case"]["dim"] ** -0.5)
    return [o, s["state"]]


def _scan(q, k, v, S, decay, beta=None):
    """One sequence, all heads: S <- decay S;  S <- S + k (beta (v - S^T k))^T or S + k v^T;  o = S^T q.  q, k [T, H, dk],
    v [T, H, dv], decay [T, H, dk or 1], S [H, dk, dv]; 64 bits.  Returns (o [T, H, dv], S)."""
    o = torch.empty_like(v)
    for t in range(v.shape[0]):
        S = S * decay[t][:, :, None]
        u = v[t]
        if beta is not None:
            u = beta[t][:, None] * (u - (k[t][:, None, :] @ S)[:, 0])
        S = torch.baddbmm(S, k[t][:, :, None], u[:, None, :])
        o[t] = (q[t][:, None, :] @ S)[:, 0]
    return o, S


def _recurrence_exact(c, seed):
    x = _recurrence_inputs(c, seed)
    lens, pasts = _lens(c), _pasts(c)
    rep = c["heads"] // c["kv_heads"]
    q, k, v = (x[n].double() for n in "qkv")
    if c["rule"] == "delta":
        q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * c["dim"] ** -0.5
        k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        beta = torch.sigmoid(x["b"].double())
        decay = torch.exp(-torch.exp(x["a_log"].double()) * torch.nn.functional.softplus(x["a"].double() + x["dtb"].double()))
    else:
        k = k * c["dim"] ** -0.5
        beta, decay = None, x["decay"].double().expand(c["rows"], -1)
    q, k = q.repeat_interleave(rep, 1), k.repeat_interleave(rep, 1)
    state, at, out = x["state"].double().clone(), np.cumsum([0] + lens), []
    for b in range(c["seqs"]):
        r, sl = slice(int(at[b]), int(at[b + 1])), int(x["slots"][b])
        S = state[sl] if pasts[b] else torch.zeros_like(state[sl])
        o, state[sl] = _scan(q[r], k[r], v[r], S, decay[r][:, :, None], None if beta is None else beta[r])
        out.append(o)
    return [torch.cat(out), state]


def _recurrence_work(c):
    T, H, G, dk, dv = c["rows"], c["heads"], c["kv_heads"], c["dim"], c["vdim"]
    state = c["seqs"] * H * dk * dv * 4 * (2 if c["past"] else 1)
    return dict(bytes=4.0 * T * (2 * G * dk + 2 * H * dv) + state, flops=(6.0 if c["rule"] == "delta" else 4.0) * T * H * dk * dv)


# ------------------------------------------------------------------------------------------ a whole hybrid decoder
_W, _FF, _VOCAB, _HEPS = 2048, 5632, 32000, 1e-6
_LEFT = dict(heads=16, kv_heads=4, dim=128, vdim=128, scale=128 ** -0.5, softcap=30.0, mask={"size": 1024, "keep_first": 4},
             rot={"base": 10000.0, "dims": 64, "scaling": None})
_RIGHT = dict(heads=8, dim=128, vdim=256, tau=16.0)
_RANK = 16
_LIGHT = dict(heads=16, dim=128, vdim=128, decay=[1.0 - 2.0 ** -(5 + i % 4) for i in range(16)])
_RET = dict(heads=8, dim=128, vdim=256, decay=[1.0 - 2.0 ** -(5 + i % 4) for i in range(8)])


def _hybrid_config():
    par = dict(left=_LEFT, right=_RIGHT, left_scale=1.0, right_scale=1.0)
    kinds = [("parallel", par), ("parallel", par), ("lightning", _LIGHT), ("retention", _RET)]
    return {"architecture": "Zalalix", "width": _W, "vocab": _VOCAB, "embedding": {"scale": _W ** 0.5}, "norm": {"eps": _HEPS},
            "layers": [{"type": t, "mixer": m, "mlp": {"kind": "dense", "ff": _FF}} for t, m in kinds]}


def _hybrid_inputs(c, seed):
    g, bf = _gen(seed), torch.bfloat16
    lin = lambda n, k: (_randn(g, n, k) / math.sqrt(k)).to(bf)                       # noqa: E731
    vec = lambda n, m=0.0, s=0.1: (m + s * _randn(g, n)).to(bf)                      # noqa: E731
    w = {"embed": (_randn(g, _VOCAB, _W) / math.sqrt(_W)).to(bf), "head": lin(_VOCAB, _W), "final.norm": vec(_W, 1.0)}
    lens, pasts = _lens(c), _pasts(c)
    ctxs = [a + b for a, b in zip(lens, pasts)]
    pages, bt = _tables(g, ctxs)
    kv, rec = {}, {}

    def decayed(key, p, m):
        H, dk, dv = m["heads"], m["dim"], m["vdim"]
        w.update({p + "q": lin(H * dk, _W), p + "k": lin(H * dk, _W), p + "v": lin(H * dv, _W), p + "g": lin(H * dv, _W),
                  p + "o": lin(_W, H * dv)})
        rec[key] = _randn(g, c["seqs"], H, dk, dv)

    cfg = _hybrid_config()
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        w.update({p + n: vec(_W, 1.0) for n in ("norm1", "norm1b", "norm2", "norm2b")})
        if layer["type"] == "parallel":
            a, q = m["left"], p + "mix.left."
            for n, rows in (("q", a["heads"] * a["dim"]), ("k", a["kv_heads"] * a["dim"]), ("v", a["kv_heads"] * a["vdim"])):
                w[q + n], w[q + n + ".b"] = lin(rows, _W), vec(rows)
            w.update({q + "q.norm": vec(a["heads"] * a["dim"], 1.0), q + "k.norm": vec(a["kv_heads"] * a["dim"], 1.0),
                      q + "g": lin(a["heads"], _W), q + "o": lin(_W, a["heads"] * a["vdim"]), q + "o.b": vec(_W)})
            kv[i] = [_randn(g, pages, PAGE, a["kv_heads"], n, dtype=bf) for n in (a["dim"], a["vdim"])]
            q, r = p + "mix.right.", m["right"]
            decayed((i, "side"), q, r)
            w.update({q + "a1": lin(_RANK, _W), q + "a2": lin(r["heads"] * r["dim"], _RANK),
                      q + "a2.b": vec(r["heads"] * r["dim"], 3.0, 1.0), q + "norm": vec(r["vdim"], 1.0)})
        else:
            decayed(i, p + "mix.", m)
            if layer["type"] == "lightning":
                w[p + "mix.norm"] = vec(m["heads"] * m["vdim"], 1.0)
        w.update({p + "mlp.gate": lin(_FF, _W), p + "mlp.up": lin(_FF, _W), p + "mlp.down": lin(_W, _FF)})
    ids = torch.randint(0, _VOCAB, (sum(lens),), generator=g, device=DEV).cpu().numpy().astype(np.uint32)
    return cfg, w, lens, pasts, ctxs, pages, bt, kv, rec, ids


def _hybrid_prepare(c, seed):
    cfg, w, lens, pasts, ctxs, pages, bt, kv, rec, ids = _hybrid_inputs(c, seed)
    B, T = c["seqs"], sum(lens)
    r = models.build_runner(cfg, w, dtype=torch.bfloat16, device=DEV, num_blocks=pages, max_blocks_per_seq=bt.shape[1],
                            max_seqs=B, max_tokens=T, num_state_slots=B)
    for i, (k, v) in kv.items():
        r.kv_cache[i].copy_(k)
        r.v_cache[i].copy_(v)
    for key, s in rec.items():
        r.rec_state[key].copy_(s)
    pos = np.concatenate([np.arange(p, p + n) for n, p in zip(lens, pasts)]).astype(np.int64)
    seq = np.repeat(np.arange(B), lens)
    slots = bt.numpy()[seq, pos // PAGE].astype(np.int64) * PAGE + pos % PAGE
    meta = dict(input_ids=ids, positions=pos, slot_mapping=slots, cu_seqlens_q=np.cumsum([0] + lens).astype(np.uint32),
                context_lens=np.array(ctxs, np.uint32), block_tables=np.ascontiguousarray(bt.numpy().astype(np.uint32).reshape(-1)),
                state_slots=np.arange(B, dtype=np.int32), num_seqs=B, num_tokens=T, max_blocks=bt.shape[1])
    torch.cuda.synchronize()
    return dict(r=r, meta=meta, rows=[int(x) - 1 for x in meta["cu_seqlens_q"][1:]])


def _hybrid_run(s):
    return s["r"].step(s["meta"], s["rows"], want_logits=True, want_ids=False)[0]


def _hybrid_exact(c, seed):
    cfg, w, lens, pasts, ctxs, pages, bt, kv, rec, ids = _hybrid_inputs(c, seed)
    W = {n: t.double() for n, t in w.items()}
    silu, sig = torch.nn.functional.silu, torch.sigmoid
    unit = lambda t: t / torch.sqrt((t * t).mean(-1, keepdim=True) + _HEPS)            # noqa: E731
    freq = 10000.0 ** (-2.0 * torch.arange(32, dtype=torch.float64, device=DEV) / 64)
    logits = []
    at = np.cumsum([0] + lens)
    for b in range(c["seqs"]):
        n, past = lens[b], pasts[b]
        ang = (past + torch.arange(n, dtype=torch.float64, device=DEV))[:, None] * freq

        def rotate(t):
            out, cs, sn = t.clone(), torch.cos(ang)[:, None], torch.sin(ang)[:, None]
            u, v = t[..., 0:64:2], t[..., 1:64:2]
            out[..., 0:64:2], out[..., 1:64:2] = u * cs - v * sn, v * cs + u * sn
            return out

        def decayed(key, h, p, m, act, decay, qs, ks):
            H, dk, dv = m["heads"], m["dim"], m["vdim"]
            q, k, v = (act(h @ W[p + x].T).reshape(n, H, -1) for x in "qkv")
            S = rec[key][b].double() if past else torch.zeros(H, dk, dv, dtype=torch.float64, device=DEV)
            return _scan(q * qs, k * ks, v, S, decay)[0]

        x = W["embed"][torch.from_numpy(ids[at[b]:at[b + 1]].astype(np.int64)).to(DEV)] * _W ** 0.5
        for i, layer in enumerate(cfg["layers"]):
            p, m, t = f"l{i}.", layer["mixer"], layer["type"]
            h = unit(x) * W[p + "norm1"]
            if t == "parallel":
                a, e = m["left"], p + "mix.left."
                q = rotate((unit(h @ W[e + "q"].T + W[e + "q.b"]) * W[e + "q.norm"]).reshape(n, a["heads"], a["dim"]))
                k = rotate((unit(h @ W[e + "k"].T + W[e + "k.b"]) * W[e + "k.norm"]).reshape(n, a["kv_heads"], a["dim"]))
                v = (h @ W[e + "v"].T + W[e + "v.b"]).reshape(n, a["kv_heads"], a["vdim"])
                k, v = (torch.cat([_gather(kv[i][z], bt[b], ctxs[b])[:past], new]) for z, new in ((0, k), (1, v)))
                o = _attend(q, k, v, past, a["scale"], a["mask"]["size"], a["mask"]["keep_first"], a["softcap"],
                            torch.zeros(a["heads"], device=DEV))
                y = (o * sig(h @ W[e + "g"].T)[:, :, None]).flatten(1) @ W[e + "o"].T + W[e + "o.b"]
                r, e = m["right"], p + "mix.right."
                z = (h @ W[e + "a1"].T) @ W[e + "a2"].T + W[e + "a2.b"]
                alpha = torch.exp(torch.nn.functional.logsigmoid(z) / r["tau"]).reshape(n, r["heads"], r["dim"])
                o = decayed((i, "side"), h, e, r, lambda q: q, alpha, r["dim"] ** -0.5, 1.0)
                y = y + ((unit(o) * W[e + "norm"]).flatten(1) * silu(h @ W[e + "g"].T)) @ W[e + "o"].T
            else:
                e = p + "mix."
                dec = torch.tensor(m["decay"], dtype=torch.float64, device=DEV)[None, :, None].expand(n, -1, 1)
                if t == "lightning":
                    o = unit(decayed(i, h, e, m, silu, dec, 1.0, 1.0).flatten(1)) * W[e + "norm"] * sig(h @ W[e + "g"].T)
                else:
                    o = unit(decayed(i, h, e, m, lambda q: q, dec, 1.0, m["dim"] ** -0.5)).flatten(1) * silu(h @ W[e + "g"].T)
                y = o @ W[e + "o"].T
            x = x + unit(y) * W[p + "norm1b"]
            h = unit(x) * W[p + "norm2"]
            x = x + unit((silu(h @ W[p + "mlp.gate"].T) * (h @ W[p + "mlp.up"].T)) @ W[p + "mlp.down"].T) * W[p + "norm2b"]
        logits.append((unit(x[-1:]) * W["final.norm"]) @ W["head"].T)
    return torch.cat(logits)


def _hybrid_work(c):
    T, B = sum(_lens(c)), c["seqs"]
    lin = 4 * 3 * _W * _FF + 2 * _W * (24 * 128 + 16 + 2048 + 6144 + _RANK + 2048) + _W * 5 * 2048 + _W * (2048 + 6144)
    pairs, keys = _visible(dict(c, window=1024, keep_first=4))
    att = 2 * 4.0 * pairs * 16 * 128
    scan = 4.0 * T * (3 * 8 * 128 * 256 + 16 * 128 * 128)
    state = B * 4 * (3 * 8 * 128 * 256 + 16 * 128 * 128) * (2 if c["past"] else 1)
    return dict(bytes=2.0 * lin + 2.0 * _W * _VOCAB + T * _W * 2 + 2 * keys * 4 * 256 * 2 + state,
                flops=2.0 * T * lin + att + scan + 2.0 * B * _W * _VOCAB)


# ------------------------------------------------------------------------------------------ the interface
_KINDS = {
    "linears": (_linears_prepare, _linears_run, _linears_exact, _linears_work),
    "mlp": (_mlp_prepare, _mlp_run, _mlp_exact, _mlp_work),
    "decode_attention": (_decode_prepare, _decode_run, _decode_exact, _decode_work),
    "prefill_attention": (_prefill_prepare, _prefill_run, _prefill_exact, _prefill_work),
    "llama_step": (_llama_prepare, _llama_run, _llama_exact, _llama_work),
    "window_attention": (_window_prepare, _window_run, _window_exact, _window_work),
    "latent_attention": (_latent_prepare, _latent_run, _latent_exact, _latent_work),
    "experts": (_experts_prepare, _experts_run, _experts_exact, _experts_work),
    "recurrence": (_recurrence_prepare, _recurrence_run, _recurrence_exact, _recurrence_work),
    "hybrid_step": (_hybrid_prepare, _hybrid_run, _hybrid_exact, _hybrid_work),
}

# Four times the distance from 64 bits that the path shows, which is what rounding operands and results to the case's
# types gives (seen: 5e-4 quantised and fp16 projections, 2.6e-4 fp16 attention, 9e-4 the decode step, 2.7e-3 bf16
# attention, 1.7e-3 experts, 8e-3 the bf16 hybrid step).  Scans are 32-bit sums of up to thousands of terms.
_TOLERANCE = {
    "linears": 2.4e-3, "mlp": 2e-3, "decode_attention": 1.2e-3, "prefill_attention": 1.2e-3, "llama_step": 4e-3,
    "window_attention": 1.1e-2, "latent_attention": 1.1e-2, "experts": 7e-3, "recurrence": 1e-5, "hybrid_step": 3e-2,
}


def prepare(case, seed):
    with torch.no_grad():
        return dict(kind=case["kind"], state=_KINDS[case["kind"]][0](case, seed))


def run(state):
    return _KINDS[state["kind"]][1](state["state"])


def exact(case, seed):
    with torch.no_grad():
        return _KINDS[case["kind"]][2](case, seed)


def work(case):
    return _KINDS[case["kind"]][3](case)


def tolerance(case):
    bf16_llama = "bf16" in (case.get("cache"), case.get("dtype"))
    return dict(rel=1.1e-2 if bf16_llama else _TOLERANCE[case["kind"]])
