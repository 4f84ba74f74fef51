"""GPU parity: every CUDA kernel through the C ABI vs the CPU oracle (oracle/).

Bars: integer/byte outputs bit-exact (prepack, argmax, cache contents); floating point within
the tolerance written in each test (north star: logits within 1e-3 in fp16 terms; single ops
are held to ~1 fp16 ulp of their output scale).
"""
import ctypes
import math

import numpy as np
import pytest
import torch

from oracle import model as om
from oracle import quant as oq

pytestmark = pytest.mark.gpu
F16 = torch.float16


@pytest.fixture(scope="module")
def ops(lib):
    from vllm_rs_b200 import ops as _ops
    return _ops


def _close(a, b, atol, rtol=0.0):
    a, b = a.float().cpu(), b.float().cpu()
    err = (a - b).abs()
    tol = atol + rtol * b.abs()
    assert bool((err <= tol).all()), f"max err {err.max().item():.3e} (tol {atol}, {rtol})"


# ---------------------------------------------------------------- glue
@pytest.mark.parametrize("T,hidden", [(1, 2048), (32, 4096), (7, 8192)])
def test_rmsnorm(ops, T, hidden):
    g = torch.Generator().manual_seed(T)
    x = torch.randn(T, hidden, generator=g).to(F16)
    w = (1 + 0.1 * torch.randn(hidden, generator=g)).to(F16)
    ref = om.rmsnorm(x, w, 1e-5)
    out = ops.rmsnorm(x.cuda(), w.cuda(), 1e-5)
    _close(out, ref, 2e-3, 1e-3)          # 1 fp16 ulp at |x| ~ 4
    # fused residual add: residual rounded to fp16 first (llama.rs:126-130)
    res = torch.randn(T, hidden, generator=g).to(F16)
    res_d = res.cuda().clone()
    out2 = ops.add_rmsnorm(res_d, x.cuda(), w.cuda(), 1e-5)
    new_res = (res.float() + x.float()).to(F16)
    assert torch.equal(res_d.cpu(), new_res)
    _close(out2, om.rmsnorm(new_res, w, 1e-5), 2e-3, 1e-3)


def test_silu_mul_embedding_argmax(ops):
    g = torch.Generator().manual_seed(0)
    gu = torch.randn(5, 2 * 5632, generator=g).to(F16)
    ref = om.silu_mul(gu[:, :5632], gu[:, 5632:])
    _close(ops.silu_mul(gu.cuda()), ref, 1e-3, 2e-3)
    table = torch.randn(1000, 256, generator=g).to(F16)
    ids = torch.randint(0, 1000, (17,), generator=g, dtype=torch.int32)
    assert torch.equal(ops.embedding(table.cuda(), ids.cuda()).cpu(), table[ids.long()])
    logits = torch.randn(9, 128256, generator=g)
    logits[3, 77] = logits[3, 90000] = 50.0     # tie -> first index wins
    assert torch.equal(ops.argmax(logits.cuda()).cpu().long(), logits.argmax(-1))
    assert int(ops.argmax(logits.cuda())[3]) == 77


@pytest.mark.parametrize("H,Hkv,D", [(32, 8, 128), (32, 4, 64)])
def test_rope_kv_write(ops, H, Hkv, D):
    cfg = om.ModelConfig(H * D, 1, H, Hkv, D, 64, 64, rope_theta=500000.0, max_pos=4096)
    cos, sin = om.rope_tables(cfg)
    g = torch.Generator().manual_seed(1)
    T, nb = 19, 8
    q = torch.randn(T, H, D, generator=g).to(F16)
    k = torch.randn(T, Hkv, D, generator=g).to(F16)
    v = torch.randn(T, Hkv, D, generator=g).to(F16)
    pos = torch.randint(0, 4096, (T,), generator=g)
    slots = torch.randperm(nb * 64, generator=g)[:T]
    slots[4] = -1
    kc = torch.zeros(nb, 64, Hkv, D, dtype=F16)
    vc = torch.zeros_like(kc)
    q_ref, k_ref = om.apply_rope(q, k, cos, sin, pos)
    om.kv_write(k_ref, v, kc, vc, slots)
    qd, kd, vd = q.cuda(), k.cuda(), v.cuda()
    kcd, vcd = torch.zeros_like(kc).cuda(), torch.zeros_like(vc).cuda()
    ops.rope_kv_write(qd, kd, vd, cos.cuda(), sin.cuda(), pos.cuda(), slots.cuda(), kcd, vcd)
    _close(qd, q_ref, 2e-3, 1e-3)
    _close(kd, k_ref, 2e-3, 1e-3)
    # cache holds exactly what was written back to k / v, at exactly the mapped slots
    exp_k = torch.zeros_like(kc)
    om.kv_write(kd.cpu(), v, exp_k, torch.zeros_like(vc), slots)
    assert torch.equal(kcd.cpu(), exp_k)
    assert torch.equal(vcd.cpu(), vc)


# ---------------------------------------------------------------- paged attention
def _paged_case(B, H, Hkv, D, ctxs, seed, nb_extra=5):
    g = torch.Generator().manual_seed(seed)
    max_blocks = max(-(-c // 64) for c in ctxs) if max(ctxs) > 0 else 1
    need = sum(-(-c // 64) for c in ctxs)
    nb = need + nb_extra
    perm = torch.randperm(nb, generator=g).tolist()      # non-contiguous pages
    kc = torch.randn(nb, 64, Hkv, D, generator=g).to(F16)
    vc = torch.randn(nb, 64, Hkv, D, generator=g).to(F16)
    bt = torch.zeros(B, max_blocks, dtype=torch.int32)
    off = 0
    for b, c in enumerate(ctxs):
        n = -(-c // 64)
        bt[b, :n] = torch.tensor(perm[off:off + n], dtype=torch.int32)
        off += n
    q = torch.randn(B, H, D, generator=g).to(F16)
    return q, kc, vc, bt, torch.tensor(ctxs, dtype=torch.int32)


@pytest.mark.parametrize("H,Hkv,D,ctxs", [
    (32, 8, 128, [1, 63, 64, 65, 127, 129, 700, 4096]),     # Llama-3-8B shapes, ragged
    (32, 4, 64, [37, 1, 500, 0, 2048]),                     # TinyLlama shapes, a ctx=0 row
    (8, 1, 128, [333, 4097]),                               # TP=8 shard of L70 (G=8)
    (16, 1, 128, [130]),                                    # G=16 (both row halves)
    (4, 4, 128, [200, 77]),                                 # MHA (G=1)
])
def test_paged_attention_decode(ops, H, Hkv, D, ctxs):
    B = len(ctxs)
    q, kc, vc, bt, cl = _paged_case(B, H, Hkv, D, ctxs, seed=H + D)
    scale = 1.0 / math.sqrt(D)
    ref = om.paged_attention_decode(q, kc, vc, bt.tolist(), cl.tolist(), scale)
    out = ops.paged_attention_decode(q.cuda(), kc.cuda(), vc.cuda(), bt.cuda(), cl.cuda(), scale)
    # outputs are convex combinations of N(0,1) values: |o| <~ 1; fp16 P/V rounding ~1e-3
    _close(out, ref, 2e-3, 2e-3)


def test_paged_attention_nan_garbage_and_window(ops):
    """Stale cache rows past context_len may hold NaN; they must not leak (p == 0 * NaN)."""
    q, kc, vc, bt, cl = _paged_case(2, 32, 8, 128, [70, 5], seed=9)
    # poison everything beyond the context inside the last pages
    for b, c in enumerate(cl.tolist()):
        blk = int(bt[b, (c - 1) // 64])
        kc[blk, c % 64 if c % 64 else 64:] = float("nan")
        vc[blk, c % 64 if c % 64 else 64:] = float("nan")
    scale = 1.0 / math.sqrt(128)
    ref = om.paged_attention_decode(q, kc, vc, bt.tolist(), cl.tolist(), scale)
    out = ops.paged_attention_decode(q.cuda(), kc.cuda(), vc.cuda(), bt.cuda(), cl.cuda(), scale)
    assert not torch.isnan(out).any()
    _close(out, ref, 2e-3, 2e-3)
    # sliding window + softcap
    q, kc, vc, bt, cl = _paged_case(3, 32, 8, 128, [700, 100, 64], seed=10)
    ref = om.paged_attention_decode(q, kc, vc, bt.tolist(), cl.tolist(), scale, softcap=30.0,
                                    window=256)
    out = ops.paged_attention_decode(q.cuda(), kc.cuda(), vc.cuda(), bt.cuda(), cl.cuda(), scale,
                                     softcap=30.0, window=256)
    _close(out, ref, 2e-3, 2e-3)


def test_paged_attention_full_size_properties(ops):
    """BASELINE config 2 size (b=32, ctx=4096, L3-8B heads): too big for the torch oracle in
    seconds, so check size-independent properties: (1) V == const => output == const;
    (2) permuting pages + block table together leaves the output bit-identical."""
    B, H, Hkv, D, ctx = 32, 32, 8, 128, 4096
    g = torch.Generator(device="cuda").manual_seed(3)
    nb = B * 64 + 64
    kc = torch.randn(nb, 64, Hkv, D, generator=g, device="cuda", dtype=F16)
    vc = torch.randn(nb, 64, Hkv, D, generator=g, device="cuda", dtype=F16)
    q = torch.randn(B, H, D, generator=g, device="cuda", dtype=F16)
    perm = torch.randperm(nb, device="cuda", generator=g)
    bt = perm[:B * 64].reshape(B, 64).to(torch.int32)
    cl = torch.full((B,), ctx, dtype=torch.int32, device="cuda")
    scale = 1 / math.sqrt(D)
    out1 = ops.paged_attention_decode(q, kc, vc, bt, cl, scale)
    # (2) relocate every page
    perm2 = torch.randperm(nb, device="cuda", generator=g)
    kc2, vc2 = torch.empty_like(kc), torch.empty_like(vc)
    kc2[perm2] = kc
    vc2[perm2] = vc
    bt2 = perm2[bt.long()].to(torch.int32)
    out2 = ops.paged_attention_decode(q, kc2, vc2, bt2, cl, scale)
    assert torch.equal(out1, out2)
    # (1) constant V per (head, d)
    const = torch.randn(Hkv, D, generator=g, device="cuda", dtype=F16)
    vc[:] = const
    out3 = ops.paged_attention_decode(q, kc, vc, bt, cl, scale)
    exp = const.repeat_interleave(H // Hkv, 0).unsqueeze(0).expand(B, H, D)
    _close(out3, exp, 2e-3, 2e-3)
    # spot-check 2 sequences against the oracle
    ref = om.paged_attention_decode(q[:2].cpu(), kc.cpu(), vc.cpu(), bt[:2].cpu().tolist(),
                                    [ctx, ctx], scale)
    _close(out3[:2], ref, 2e-3, 2e-3)


# ---------------------------------------------------------------- W4A16 / W8A16
def _wna_case(K, N, M, fmt, bits, seed, group=128):
    rng = np.random.default_rng(seed)
    if fmt == "awq":
        qw, qz, s = oq.random_awq(rng, K, N, group)
        W = oq.dequant_awq(qw, qz, s, group)
    else:
        qw, qz, s = oq.random_gptq(rng, K, N, group, bits, sym=(fmt == "gptq_sym"))
        if fmt == "gptq_sym":
            qz = None
        W = oq.dequant_gptq(qw, qz, s, group, bits)
    x = torch.from_numpy(rng.standard_normal((M, K)).astype(np.float16))
    return qw, qz, s, torch.from_numpy(W), x


# flat GEMV / unit or tile-split tcgen05 decode kernel (M <= 64) / general tcgen05 / stream-K tcgen05 decode kernel (M <= 32), two
# flavours / unit kernel (8-bit: M <= 32) / tile-split kernel
@pytest.mark.parametrize("variant", [1, 2, 4, 5, 6, 8, 9])
@pytest.mark.parametrize("fmt,bits,K,N,M", [
    ("awq", 4, 4096, 1024, 1), ("awq", 4, 4096, 6144, 32), ("awq", 4, 14336, 4096, 5),
    ("gptq", 4, 2048, 256, 3), ("gptq_sym", 4, 1024, 512, 16), ("gptq", 8, 2048, 512, 7),
    ("awq", 4, 512, 128, 64), ("gptq", 4, 1792, 4096, 33),
])
def test_wna16_gemm(ops, fmt, bits, K, N, M, variant):
    if variant >= 2 and not _tc_available(ops):
        pytest.skip("tcgen05 variant not built yet")
    if variant in (5, 6) and M > 32:
        pytest.skip("the stream-K decode kernel takes M <= 32")
    if variant == 6 and bits != 4:
        pytest.skip("the mma.sync stream-K flavour is 4-bit only")
    qw, qz, s, W, x = _wna_case(K, N, M, fmt, bits, seed=K + N + M)
    qwd = torch.from_numpy(qw).cuda()
    packed = ops.awq_prepack(qwd) if fmt == "awq" else ops.gptq_prepack(qwd, bits)
    ws = ops.wna16_workspace(max(M, 16), N)
    y = ops.wna16_gemm(x.cuda(), packed, torch.from_numpy(s).cuda(),
                       None if qz is None else torch.from_numpy(qz).cuda(), ws, k=K, n=N,
                       bits=bits, group_size=128,
                       qfmt=ops.QFMT_AWQ if fmt == "awq" else ops.QFMT_GPTQ, variant=variant)
    ref = om.linear(x, W)
    # |y| ~ 1; fp32 accumulation both sides, one fp16 rounding on output
    _close(y, ref, 2e-3, 2e-3)
    assert int(ws[:16384].view(torch.int32).abs().sum()) == 0      # arrival counters back at rest
    # second call reuses the workspace and must agree with the first
    y2 = ops.wna16_gemm(x.cuda(), packed, torch.from_numpy(s).cuda(),
                        None if qz is None else torch.from_numpy(qz).cuda(), ws, k=K, n=N,
                        bits=bits, group_size=128,
                        qfmt=ops.QFMT_AWQ if fmt == "awq" else ops.QFMT_GPTQ, variant=variant)
    assert torch.equal(y2, y)                   # split-K partials are reduced in a fixed order


@pytest.mark.parametrize("fmt,bits,K,N,M,group,epi", [
    ("awq", 4, 4096, 28672, 32, 128, "silu"),      # gate|up of Llama-3-8B: 3 tile segments per CTA, gate / up pairs
    ("awq", 4, 14336, 4096, 17, 128, "none"),      # down: every tile cut 4-5 ways
    ("gptq", 4, 4096, 4096, 32, 4096, "none"),     # one group per channel
    ("gptq_sym", 4, 2048, 1536, 8, 256, "bias"),   # groups of two units, bias in the finaliser / direct store
    ("gptq", 8, 4096, 1024, 32, 128, "none"),      # W8A16
    ("awq", 4, 256, 128, 1, 128, "none"),          # one tile, two units, one CTA
    ("awq", 4, 8192, 7168, 32, 128, "silu"),       # Llama-3-70B gate|up shard at TP = 8
])
@pytest.mark.parametrize("variant", [5, 6])
def test_wna16_streamk_decode(ops, fmt, bits, K, N, M, group, epi, variant):
    """wna16_sk.cu (variant 5 = tcgen05 flavour, 6 = mma.sync register flavour): CTA ranges that cut tiles anywhere, per-CTA partial slots, every epilogue the
    public entry exposes; and the post-MMA scale is at least as close to the fp32 truth as the fp16-rounded
    weights the reference multiplies with."""
    if variant == 6 and bits != 4:
        pytest.skip("the mma.sync stream-K flavour is 4-bit only")
    qw, qz, s, W, x = _wna_case(K, N, M, fmt, bits, seed=K + N + M + group, group=group)
    qwd = torch.from_numpy(qw).cuda()
    packed = ops.awq_prepack(qwd) if fmt == "awq" else ops.gptq_prepack(qwd, bits)
    ws = ops.wna16_workspace(max(M, 16), N)
    sd = torch.from_numpy(s).cuda()
    zd = None if qz is None else torch.from_numpy(qz).cuda()
    qf = ops.QFMT_AWQ if fmt == "awq" else ops.QFMT_GPTQ
    bias = torch.randn(N).to(F16) if epi == "bias" else None
    kw = dict(k=K, n=N, bits=bits, group_size=group, qfmt=qf,
              epilogue=ops.EPI_SILU_MUL if epi == "silu" else ops.EPI_NONE,
              bias=None if bias is None else bias.cuda())
    y = ops.wna16_gemm(x.cuda(), packed, sd, zd, ws, variant=variant, **kw)
    full = om.linear(x, W, bias)
    ref = om.silu_mul(full[:, :N // 2], full[:, N // 2:]) if epi == "silu" else full
    _close(y, ref, 2e-3, 4e-3 if epi == "silu" else 2e-3)
    assert int(ws[:16384].view(torch.int32).abs().sum()) == 0      # arrival counters back at rest
    y2 = ops.wna16_gemm(x.cuda(), packed, sd, zd, ws, variant=variant, **kw)
    assert torch.equal(y2, y)                                      # contributor-ordered sums: deterministic
    if epi == "none":
        # the exact product x @ ((q - z) * s), no fp16 rounding of the weights: the post-MMA scale must be at least
        # as close to it as the tile-split kernel, which multiplies with the reference's fp16-rounded weights
        q = oq.unpack_awq(qw) if fmt == "awq" else oq.unpack_gptq(qw, bits)
        if qz is None:
            z = np.full((K // group, N), 1 << (bits - 1), dtype=np.int32)
        else:
            z = oq.unpack_awq(qz).astype(np.int32) if fmt == "awq" else oq.unpack_gptq_zeros(qz, bits)
        gi = np.arange(K) // group
        wexact = (q.astype(np.float64) - z[gi]) * s[gi].astype(np.float64)
        truth = torch.from_numpy(x.numpy().astype(np.float64) @ wexact)
        y_old = ops.wna16_gemm(x.cuda(), packed, sd, zd, ws, variant=9, **kw)
        e_new = (y.cpu().double() - truth).abs().max().item()
        e_old = (y_old.cpu().double() - truth).abs().max().item()
        assert e_new <= e_old + 5e-4, (e_new, e_old)


def _wna_run(ops, fmt, bits, K, N, M, group, epi, seed):
    """(call with a variant, reference, exact product as a function) of one quantised projection."""
    qw, qz, s, W, x = _wna_case(K, N, M, fmt, bits, seed=seed, group=group)
    qwd = torch.from_numpy(qw).cuda()
    packed = ops.awq_prepack(qwd) if fmt == "awq" else ops.gptq_prepack(qwd, bits)
    ws = ops.wna16_workspace(max(M, 16), N)
    sd, zd = torch.from_numpy(s).cuda(), None if qz is None else torch.from_numpy(qz).cuda()
    bias = torch.randn(N).to(F16) if epi == "bias" else None
    kw = dict(k=K, n=N, bits=bits, group_size=group, qfmt=ops.QFMT_AWQ if fmt == "awq" else ops.QFMT_GPTQ,
              epilogue=ops.EPI_SILU_MUL if epi == "silu" else ops.EPI_NONE, bias=None if bias is None else bias.cuda())
    full = om.linear(x, W, bias)
    ref = om.silu_mul(full[:, :N // 2], full[:, N // 2:]) if epi == "silu" else full

    def call(variant):
        y = ops.wna16_gemm(x.cuda(), packed, sd, zd, ws, variant=variant, **kw)
        assert int(ws[:16384].view(torch.int32).abs().sum()) == 0      # arrival counters back at rest
        return y

    def truth():
        q = oq.unpack_awq(qw) if fmt == "awq" else oq.unpack_gptq(qw, bits)
        z = oq.unpack_awq(qz).astype(np.int32) if fmt == "awq" else oq.unpack_gptq_zeros(qz, bits)
        g = np.arange(K) // group
        return torch.from_numpy(x.numpy().astype(np.float64) @ ((q.astype(np.float64) - z[g]) * s[g].astype(np.float64)))

    return call, ref, truth


@pytest.mark.parametrize("fmt,bits,K,N,M,group,epi", [
    ("awq", 4, 128, 128, 1, 128, "none"),          # one unit: the second group of warps has none
    ("awq", 4, 384, 256, 9, 128, "silu"),          # three units per tile, pairs of gate and up
    ("gptq", 4, 640, 384, 8, 640, "bias"),         # one quantisation group; tiles of five units
    ("gptq_sym", 4, 2048, 1536, 16, 256, "none"),  # no zero points, two units per group
    ("awq", 4, 4096, 28672, 3, 128, "silu"),       # ranges cut anywhere: two tiles in a block
    ("awq", 4, 256, 40960, 5, 128, "none"),        # more tiles than blocks, whole tiles and parts in one block
    ("awq", 4, 14336, 4096, 2, 128, "none"),       # eight parts per tile
    ("awq", 4, 2048, 34816, 16, 128, "none"),      # as many units as the sixteen tokens want
])
def test_wna16_decode_of_few_tokens(ops, fmt, bits, K, N, M, group, epi):
    """wna16_mma.cu (variant 7, and what variant 0 takes at up to 8 tokens, and to 16 of wide products of short K)."""
    call, ref, truth = _wna_run(ops, fmt, bits, K, N, M, group, epi, K + N + M)
    y = call(7)
    _close(y, ref, 2e-3, 4e-3 if epi == "silu" else 2e-3)          # the bound of the other variants: fp32 sums, fp16 results
    assert torch.equal(call(7), y)                 # parts are summed in the order of K
    if M <= 8 or K // 128 * (N // 128) >= 4096:
        assert torch.equal(call(0), y)
    if epi == "none" and "sym" not in fmt:
        t = truth()
        e_new, e_old = ((v.cpu().double() - t).norm() for v in (y, call(9)))
        assert e_new <= e_old * 1.05, (e_new, e_old)               # the same weights, sums in another order


@pytest.mark.parametrize("fmt,bits,K,N,M,group,epi", [
    ("awq", 4, 128, 128, 9, 128, "none"),           # one unit: one accumulator, one group of warps
    ("awq", 4, 384, 256, 17, 128, "silu"),          # three blocks of a unit each meet in a cluster
    ("gptq", 4, 640, 384, 33, 640, "bias"),         # five units in five blocks; rows that not every block has as many of
    ("gptq_sym", 4, 2048, 1536, 64, 256, "none"),   # no zero points, two units per group
    ("awq", 4, 4096, 6144, 11, 128, "bias"),        # two blocks per tile
    ("awq", 4, 4096, 28672, 32, 128, "silu"),       # ranges cut anywhere: two or three tiles in a block, meetings in memory
    ("awq", 4, 1280, 40960, 50, 128, "none"),       # whole tiles and parts of an odd number of units in one block
    ("awq", 4, 14336, 4096, 16, 128, "none"),       # rings that go round many times
    ("awq", 4, 8192, 1280, 64, 128, "none"),        # seven blocks would meet, but as many clusters do not fit
    ("awq", 4, 128, 76800, 17, 128, "none"),        # tiles of one unit, four in a block: the issuers take turns
    ("awq", 4, 128, 40960, 12, 128, "silu"),
    ("awq", 4, 256, 29440, 33, 128, "none"),        # first and last parts of one unit beside tiles of two
    ("gptq", 8, 128, 38400, 9, 128, "bias"),
    ("gptq", 8, 384, 256, 1, 128, "silu"),
    ("gptq", 8, 4096, 12288, 32, 128, "none"),
    ("gptq", 8, 14336, 4096, 9, 128, "bias"),
])
def test_wna16_units_cut_evenly(ops, fmt, bits, K, N, M, group, epi):
    """wna16_ts.cu (variant 8, and what variant 0 takes from 9 tokens on)."""
    call, ref, truth = _wna_run(ops, fmt, bits, K, N, M, group, epi, K + N + M)
    y = call(8)
    _close(y, ref, 2e-3, 4e-3 if epi == "silu" else 2e-3)          # the bound of the other variants: fp32 sums, fp16 results
    assert all(torch.equal(call(8), y) for _ in range(20))         # parts are summed in the order of K
    if M > 8 and (K, N) not in ((128, 128), (4096, 12288)):        # (there wna16_tc_dec.cu is the faster: test_wna16_units_or_tiles)
        assert torch.equal(call(0), y)
    if epi == "none" and "sym" not in fmt:
        t = truth()
        e_new, e_old = ((v.cpu().double() - t).norm() for v in (y, call(9)))      # 9: wna16_tc_dec.cu
        assert e_new <= e_old * 1.05, (e_new, e_old)               # the same weights, sums in another order


@pytest.mark.parametrize("M,variants", [(3, (0, 1, 2, 4, 5, 6, 7, 8, 9)), (12, (0, 2, 4, 5, 6, 7, 8, 9)), (40, (0, 2, 4, 8, 9))])
def test_wna16_silu_quotient_is_a_division(ops, M, variants):
    """silu(-88) is -88 / (1 + e^88), whose denominator is above 2^126: small, not zero, so that an infinite up makes it infinite."""
    K, N, g = 512, 256, 128
    q, z, s = np.full((K, N), 7, np.uint8), np.full((K // g, N), 8, np.uint8), np.ones((K // g, N), np.float16)
    q[:, N // 2:], z[:, N // 2:], s[:, N // 2:] = 15, 5, 100                 # gate weights -1, up weights 1000
    packed = ops.awq_prepack(torch.from_numpy(oq.pack_awq(q)).cuda())
    sd, zd, ws = torch.from_numpy(s).cuda(), torch.from_numpy(oq.pack_awq(z)).cuda(), ops.wna16_workspace(64, N)
    x = torch.full((M, K), 88 / K, dtype=F16, device="cuda")                 # exact: the sums are -88 and 88 000, past fp16
    for v in variants:
        y = ops.wna16_gemm(x, packed, sd, zd, ws, k=K, n=N, epilogue=ops.EPI_SILU_MUL, variant=v)
        assert torch.equal(y, torch.full_like(y, -float("inf"))), v


@pytest.mark.parametrize("K,N,M,group", [(512, 19456, 3, 128),          # as many tiles as SMs: no kernel splits them
                                         (8192, 9728, 33, 64)])         # more groups than an unsplit tile of wna16_tc_dec.cu stages
@pytest.mark.parametrize("off_bias,off_y", [(1, 0), (0, 1), (2, 2)])
def test_wna16_bias_and_result_off_eight_bytes(ops, K, N, M, group, off_bias, off_y):
    """Where a kernel writes a tile's results one by one, they and the bias may begin anywhere."""
    qw, qz, s, W, x = _wna_case(K, N, M, "awq", 4, seed=5, group=group)
    bias = torch.randn(N).to(F16)
    at = torch.zeros(N + 4, dtype=F16)
    at[off_bias:off_bias + N] = bias
    y = torch.zeros(M * N + 4, dtype=F16).cuda()
    ops.wna16_gemm(x.cuda(), ops.awq_prepack(torch.from_numpy(qw).cuda()), torch.from_numpy(s).cuda(), torch.from_numpy(qz).cuda(),
                   ops.wna16_workspace(64, N), k=K, n=N, group_size=group, bias=at.cuda()[off_bias:off_bias + N],
                   out=y[off_y:off_y + M * N].view(M, N))
    _close(y[off_y:off_y + M * N].view(M, N), om.linear(x, W, bias), 2e-3, 2e-3)
    rest = torch.ones(M * N + 4, dtype=torch.bool)
    rest[off_y:off_y + M * N] = False
    assert not y.cpu()[rest].any()


@pytest.mark.parametrize("M,off_s,off_z", [(1, 1, 0), (9, 0, 1), (16, 3, 2)])
def test_wna16_scales_and_zeros_off_sixteen_bytes(ops, M, off_s, off_z):
    """Large 4-bit products of few tokens whose scales or zero points begin anywhere (views of fused ones): the stream-K kernel, as
    the others copy them by 16 bytes."""
    K, N = 4096, 28672
    qw, qz, s, W, x = _wna_case(K, N, M, "awq", 4, seed=M)
    at = lambda a, n: torch.cat([torch.zeros(n, dtype=a.dtype), a.flatten()]).cuda()[n:].view(a.shape)      # noqa: E731
    args = (x.cuda(), ops.awq_prepack(torch.from_numpy(qw).cuda()), at(torch.from_numpy(s), off_s), at(torch.from_numpy(qz), off_z),
            ops.wna16_workspace(16, N))
    y = ops.wna16_gemm(*args, k=K, n=N)
    _close(y, om.linear(x, W, None), 2e-3, 2e-3)
    assert torch.equal(y, ops.wna16_gemm(*args, k=K, n=N, variant=5))


@pytest.mark.parametrize("K,N,M,group,off_s,off_z", [(8192, 9728, 33, 64, 1, 0), (4096, 9728, 17, 64, 0, 1), (16384, 1280, 64, 32, 1, 1)])
def test_wna16_many_groups_off_sixteen_bytes(ops, K, N, M, group, off_s, off_z):
    """Scales or zero points that begin anywhere, of more groups than the tile-split kernel stages for one piece of K: the general
    kernel, which reads them one by one."""
    qw, qz, s, W, x = _wna_case(K, N, M, "awq", 4, seed=M, group=group)
    at = lambda a, n: torch.cat([torch.zeros(n, dtype=a.dtype), a.flatten()]).cuda()[n:].view(a.shape)      # noqa: E731
    args = (x.cuda(), ops.awq_prepack(torch.from_numpy(qw).cuda()), at(torch.from_numpy(s), off_s), at(torch.from_numpy(qz), off_z),
            ops.wna16_workspace(64, N))
    y = ops.wna16_gemm(*args, k=K, n=N, group_size=group)
    _close(y, om.linear(x, W, None), 2e-3, 2e-3)
    assert torch.equal(y, ops.wna16_gemm(*args, k=K, n=N, group_size=group, variant=4))


@pytest.mark.parametrize("M", [1, 16])
def test_wna16_decode_of_more_than_65536_units(ops, M):
    """Sizes at which a product by the number of all units does not fit 32 bits (wna16_mma.cu, ranges cut anywhere): every tile is
    written, and the counters are back at rest.  fp32 sums of the weights rounded to fp16, a group of 128 K at a time."""
    K, N = 34944, 30848
    g = torch.Generator(device="cuda").manual_seed(M)
    words = lambda r: torch.randint(-2 ** 31, 2 ** 31, (r, N // 8), generator=g, device="cuda", dtype=torch.int64).int()      # noqa: E731
    qw, qz = words(K), words(K // 128)
    s = (0.005 + 0.01 * torch.rand(K // 128, N, generator=g, device="cuda")).to(F16)
    x = (0.05 * torch.randn(M, K, generator=g, device="cuda")).to(F16)
    at = torch.tensor([4 * j for j in (0, 4, 1, 5, 2, 6, 3, 7)], device="cuda", dtype=torch.int32)      # nibble of output 8 c + i
    nib = lambda w: ((w[..., None] >> at) & 15).reshape(w.shape[0], N)              # noqa: E731
    ref = torch.zeros(M, N, device="cuda", dtype=torch.float64)
    for i in range(K // 128):
        rows = slice(i * 128, i * 128 + 128)
        w = ((nib(qw[rows]) - nib(qz[i:i + 1])).to(F16) * s[i]).float()
        ref += (x[:, rows].float() @ w).double()
    packed, ws = ops.awq_prepack(qw), ops.wna16_workspace(16, N)
    for variant in (7, 0):
        y = ops.wna16_gemm(x, packed, s, qz, ws, k=K, n=N, bits=4, group_size=128, qfmt=ops.QFMT_AWQ, variant=variant)
        _close(y, ref.cpu(), 2e-3, 2e-3)
        assert int(ws[:16384].view(torch.int32).abs().sum()) == 0


@pytest.mark.parametrize("M", [1, 16])
def test_wna16_decode_repeats_itself(ops, M):
    """The same bits from every call: no warp reads a place of the ring that a later unit's copies are on their way to.  Weights that
    have just been written keep the activations out of L2, so that copies take their longest."""
    K, N = 34944, 30848
    g = torch.Generator(device="cuda").manual_seed(M)
    words = lambda r: torch.randint(-2 ** 31, 2 ** 31, (r, N // 8), generator=g, device="cuda", dtype=torch.int64).int()      # noqa: E731
    qw, qz = words(K), words(K // 128)
    s = (0.005 + 0.01 * torch.rand(K // 128, N, generator=g, device="cuda")).to(F16)
    x = (0.05 * torch.randn(M, K, generator=g, device="cuda")).to(F16)
    ws, first, differ = ops.wna16_workspace(16, N), None, 0
    for _ in range(500):
        y = ops.wna16_gemm(x, ops.awq_prepack(qw), s, qz, ws, k=K, n=N, variant=7)
        first = y if first is None else first
        differ += int((y != first).any())
    assert differ == 0


class _FusedEpi(ctypes.Structure):                   # wna16.cuh, FusedEpi
    _fields_ = ([("ssq_in", ctypes.c_void_p), ("ssq_tiles", ctypes.c_int), ("inv_dim", ctypes.c_float), ("eps", ctypes.c_float)] +
                [(n, ctypes.c_void_p) for n in ("resid", "norm_w", "ssq_out", "positions", "slots", "cos", "sin", "k_cache", "v_cache")] +
                [(n, ctypes.c_int) for n in ("H", "Hkv", "D", "kv_fp8")] +
                [("push", ctypes.c_void_p * 8), ("push_cnt", ctypes.c_void_p * 8), ("push_world", ctypes.c_int), ("out_bf16", ctypes.c_int)])


class _WnaParams(ctypes.Structure):                  # wna16.cuh, WnaParams
    _fields_ = ([(n, ctypes.c_void_p) for n in ("a", "bp", "scales", "qzeros", "bias", "c")] +
                [(n, ctypes.c_int) for n in ("M", "K", "N", "bits", "group_size", "qfmt", "epilogue", "no_split")] +
                [("workspace", ctypes.c_void_p), ("fe", ctypes.c_void_p)])


def _same_members(cls, struct):
    """The header's struct has these members in this order (a launch with others would be one with wrong addresses)."""
    import re
    from pathlib import Path
    text = (Path(__file__).resolve().parent.parent / "vllm_rs_b200" / "csrc" / "wna16.cuh").read_text()
    body = re.sub(r"//[^\n]*", "", text[text.index(f"struct {struct} {{"):].split("{", 1)[1].split("};", 1)[0])
    kind = {"int": ctypes.c_int, "float": ctypes.c_float}
    got = []
    for decl in filter(None, (d.strip() for d in body.split(";"))):
        base, names = re.fullmatch(r"(?:const )?(?:struct )?(\w+)(.*)", decl, re.S).groups()
        for n in names.split(","):
            size = re.search(r"\[kMaxTpRanks\]", n)
            got.append((re.search(r"\w+", n).group(), ctypes.c_void_p * 8 if size else ctypes.c_void_p if "*" in n else kind[base]))
    assert "constexpr int kMaxTpRanks = 8;" in text and got == cls._fields_


@pytest.mark.parametrize("kernel,M", [("mma", 1), ("mma", 8), ("mma", 9), ("mma", 16), ("dec", 9), ("dec", 17), ("dec", 33), ("dec", 64)])
def test_wna16_push_to_peers(ops, kernel, M):
    """The epilogue of a tensor-parallel rank's row-parallel products: the fp16 partial in every rank's receive buffer, one count per
    tile and rank.  Nothing waits for the counts here, so the three receive areas lie on this GPU."""
    from vllm_rs_b200 import _lib
    _same_members(_FusedEpi, "FusedEpi")
    _same_members(_WnaParams, "WnaParams")
    K, N, world = 1024, 2048, 3
    qw, qz, s, W, x = _wna_case(K, N, M, "awq", 4, seed=M)
    xd, packed, sd, zd = x.cuda(), ops.awq_prepack(torch.from_numpy(qw).cuda()), torch.from_numpy(s).cuda(), torch.from_numpy(qz).cuda()
    ws = ops.wna16_workspace(64, N)
    recv, cnt = torch.full((world, 64, N), float("nan"), dtype=F16, device="cuda"), torch.zeros(world, 16, dtype=torch.int32, device="cuda")
    fe, p = _FusedEpi(), _WnaParams()
    for r in range(world):
        fe.push[r], fe.push_cnt[r] = recv[r].data_ptr(), cnt[r, 5:].data_ptr()
    fe.push_world = world
    for n, v in dict(a=xd.data_ptr(), bp=packed.data_ptr(), scales=sd.data_ptr(), qzeros=zd.data_ptr(), M=M, K=K, N=N, bits=4,
                     group_size=128, qfmt=ops.QFMT_AWQ, epilogue=4, workspace=ws.data_ptr(), fe=ctypes.addressof(fe)).items():
        setattr(p, n, v)
    name, more = {"mma": ("_ZN4b20016launch_wna16_mmaERKNS_9WnaParamsEP11CUstream_stb", (ctypes.c_bool(True),)),
                  "dec": ("_ZN4b20019launch_wna16_tc_decERKNS_9WnaParamsEP11CUstream_st", ())}[kernel]
    launch = getattr(_lib.lib(), name)
    launch.restype = ctypes.c_bool
    for calls in (1, 2):
        assert launch(ctypes.byref(p), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), *more)
        _lib.check()
        want = torch.zeros(world, 16, dtype=torch.int32)
        want[:, 5] = calls * (N // 128)
        assert torch.equal(cnt.cpu(), want)
        for r in range(world):
            _close(recv[r, :M], om.linear(x, W, None), 2e-3, 2e-3)
            assert recv[r, M:].isnan().all()
        assert int(ws[:16384].view(torch.int32).abs().sum()) == 0


@pytest.mark.parametrize("K,N,M", [(1024, 2048, 9), (1024, 2048, 64), (2048, 20480, 33)])     # parts of a tile; whole tiles as well
def test_wna16_units_push_to_peers(ops, K, N, M):
    """test_wna16_push_to_peers for wna16_ts.cu, whose blocks meet in memory here."""
    from vllm_rs_b200 import _lib
    qw, qz, s, W, x = _wna_case(K, N, M, "awq", 4, seed=M)
    hold = [x.cuda(), ops.awq_prepack(torch.from_numpy(qw).cuda()), torch.from_numpy(s).cuda(), torch.from_numpy(qz).cuda()]
    ws, world = ops.wna16_workspace(64, N), 2
    recv, cnt = torch.full((world, 64, N), float("nan"), dtype=F16, device="cuda"), torch.zeros(world, 16, dtype=torch.int32, device="cuda")
    fe, p = _FusedEpi(push_world=world), _WnaParams(M=M, K=K, N=N, bits=4, group_size=128, qfmt=ops.QFMT_AWQ, epilogue=4)
    for r in range(world):
        fe.push[r], fe.push_cnt[r] = recv[r].data_ptr(), cnt[r, 5:].data_ptr()
    p.a, p.bp, p.scales, p.qzeros = (t.data_ptr() for t in hold)
    p.workspace, p.fe = ws.data_ptr(), ctypes.addressof(fe)
    launch = getattr(_lib.lib(), "_ZN4b20015launch_wna16_tsERKNS_9WnaParamsEP11CUstream_stb")
    launch.restype = ctypes.c_bool
    assert launch(ctypes.byref(p), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), ctypes.c_bool(True))
    _lib.check()
    assert cnt.cpu()[:, 5].tolist() == [N // 128] * world and int(cnt.sum()) == world * (N // 128)
    for r in range(world):
        _close(recv[r, :M], om.linear(x, W, None), 2e-3, 2e-3)
        assert recv[r, M:].isnan().all()
    assert int(ws[:16384].view(torch.int32).abs().sum()) == 0


@pytest.mark.parametrize("variant,bits,K,N,M,epi", [(9, 8, 4096, 28672, 48, "silu"), (9, 8, 14336, 4096, 64, "none"), (9, 4, 4096, 28672, 64, "none"),
                                                    (4, 8, 4096, 8192, 64, "none"), (4, 4, 8192, 4096, 200, "none"),
                                                    (5, 8, 4096, 28672, 16, "silu"), (5, 4, 14336, 4096, 32, "none"), (6, 4, 8192, 8192, 16, "none")])
def test_wna16_rings_repeat_themselves(ops, variant, bits, K, N, M, epi):
    """The same bits from 400 calls of the kernels whose warps read packed weights from a ring of copies, weights cold and not."""
    g = torch.Generator(device="cuda").manual_seed(M)
    words = lambda n: torch.randint(-2 ** 31, 2 ** 31, (n,), generator=g, device="cuda", dtype=torch.int64).int()      # noqa: E731
    packed, qz = words(K * N * bits // 32), words(K // 128 * N * bits // 32).view(K // 128, -1)
    s = (0.005 + 0.01 * torch.rand(K // 128, N, generator=g, device="cuda")).to(F16) / 2 ** (bits - 4)
    x = (0.05 * torch.randn(M, K, generator=g, device="cuda")).to(F16)
    ws, cold = ops.wna16_workspace(M, N), torch.empty(64 << 20, device="cuda")
    kw = dict(k=K, n=N, bits=bits, qfmt=ops.QFMT_AWQ if bits == 4 else ops.QFMT_GPTQ, variant=variant,
              epilogue=ops.EPI_SILU_MUL if epi == "silu" else ops.EPI_NONE)
    first, differ = ops.wna16_gemm(x, packed, s, qz, ws, **kw), torch.zeros((), dtype=torch.int64, device="cuda")
    for i in range(400):
        if i % 8 == 0:
            cold.zero_()
        differ += (ops.wna16_gemm(x, packed, s, qz, ws, **kw).view(torch.int16) != first.view(torch.int16)).any()
    assert int(differ) == 0


def test_wna16_streamk_switch():
    """B200_DEC_SK=1 gives the stream-K kernel every product of up to 32 tokens that it takes, before all others (read once per process)."""
    import os
    import subprocess
    import sys
    program = """
import test_kernels_gpu as t
from vllm_rs_b200 import ops
for fmt, bits, M in (("awq", 4, 3), ("awq", 4, 16), ("awq", 4, 32), ("gptq", 8, 1), ("gptq", 8, 32)):
    call, _, _ = t._wna_run(ops, fmt, bits, 2048, 1536, M, 128, "none", M)
    assert t.torch.equal(call(0), call(5)), (bits, M)
print("equal")
"""
    env = dict(os.environ, B200_DEC_SK="1", PYTHONPATH=os.pathsep.join([os.path.dirname(os.path.abspath(__file__))] + sys.path))
    r = subprocess.run([sys.executable, "-c", program], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "equal" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]


@pytest.mark.parametrize("K,N,M,group", [(4096, 9728, 17, 64), (8192, 9728, 33, 64), (8192, 1280, 64, 128)])
def test_wna16_decode_of_many_groups(ops, K, N, M, group):
    """wna16_tc_dec.cu where one K piece has exactly as many quantisation groups as are staged, and where it takes more pieces."""
    call, ref, _ = _wna_run(ops, "awq", 4, K, N, M, group, "none", K + N + M)
    y = call(9)
    _close(y, ref, 2e-3, 2e-3)
    assert torch.equal(call(9), y)
    if group < 128:                                                # (of 128 and more wna16_ts.cu takes them)
        assert torch.equal(call(0), y)


@pytest.mark.parametrize("K,N,M,epi", [(2048, 512, 33, "bias"), (14336, 4096, 64, "none"), (4096, 28672, 48, "silu"), (128, 256, 40, "silu"),
                                       (1024, 20480, 64, "bias"), (4096, 1280, 57, "none")])
def test_wna16_eight_bits_of_many_tokens(ops, K, N, M, epi):
    """8-bit weights of 33 to 64 tokens, which are wna16_tc_dec.cu's: pieces that meet, tiles that store themselves, pairs of tiles."""
    call, ref, _ = _wna_run(ops, "gptq", 8, K, N, M, 128, epi, K + N + M)
    y = call(9)
    _close(y, ref, 2e-3, 4e-3 if epi == "silu" else 2e-3)          # the bound of the other variants: fp32 sums, fp16 results
    assert torch.equal(call(9), y) and torch.equal(call(0), y)


@pytest.mark.parametrize("fmt,bits,K,N,M,epi,unit", [
    ("awq", 4, 128, 1024, 9, "none", 0), ("awq", 4, 128, 1024, 9, "silu", 1),      # one unit per tile; pairs of tiles meet over there
    ("awq", 4, 384, 4096, 32, "bias", 0), ("awq", 4, 512, 4096, 32, "bias", 1),    # clusters of blocks of one unit, and split tiles there
    ("awq", 4, 1536, 12800, 16, "none", 0), ("awq", 4, 2048, 12800, 16, "none", 1),            # a tile each
    ("awq", 4, 4096, 12800, 32, "none", 0), ("awq", 4, 6144, 12800, 32, "none", 1),            # ranges cut anywhere: few units less, more
    ("awq", 4, 18944, 1024, 33, "none", 0),                                        # sums of many parts
    ("awq", 4, 14336, 5120, 16, "none", 1), ("gptq", 8, 14336, 5120, 16, "none", 0),           # sizes that go on to other kernels, or not
    ("gptq", 8, 1024, 10240, 1, "none", 0), ("gptq", 8, 14336, 4608, 4, "none", 0), ("gptq", 8, 4096, 6144, 4, "silu", 1),
    ("gptq", 8, 2048, 9728, 9, "silu", 0), ("gptq", 8, 2048, 9728, 32, "silu", 1),
])
def test_wna16_units_or_tiles(ops, fmt, bits, K, N, M, epi, unit):
    """On either side of the line between wna16_ts.cu (8) and wna16_tc_dec.cu (9): variants 0 and 2 are that kernel, and both agree."""
    call, ref, _ = _wna_run(ops, fmt, bits, K, N, M, 128, epi, K + N + M)
    ys = [call(9), call(8)]
    for y in ys:
        _close(y, ref, 2e-3, 4e-3 if epi == "silu" else 2e-3)      # the bound of the other variants: fp32 sums, fp16 results
    assert torch.equal(call(0), ys[unit]) and torch.equal(call(2), ys[unit])


def _tc_available(ops):
    from vllm_rs_b200 import _lib
    rng = np.random.default_rng(0)
    qw, qz, s = oq.random_awq(rng, 128, 128, 128)
    x = torch.zeros(16, 128, dtype=F16, device="cuda")
    ws = ops.wna16_workspace(16, 128)
    try:
        ops.wna16_gemm(x, ops.awq_prepack(torch.from_numpy(qw).cuda()),
                       torch.from_numpy(s).cuda(), torch.from_numpy(qz).cuda(), ws, k=128, n=128,
                       variant=2)
        return True
    except _lib.B200Error:
        return False


@pytest.mark.parametrize("bits,K,N,M,group", [(8, 2048, 512, 7, 128), (4, 4096, 1024, 32, 128), (4, 1024, 256, 200, 64)])
def test_gemm_half_q_half_alt_exact_signature(ops, bits, K, N, M, group):
    """The reference's own argument list (gptq.rs:183-195): checkpoint-format qweight, g_idx, no group size, no
    workspace.  Second call hits the cached tile-major copy and must agree bit for bit."""
    from vllm_rs_b200 import _lib
    l = _lib.lib()
    qw, qz, s, W, x = _wna_case(K, N, M, "gptq", bits, seed=K + N + M + bits, group=group)
    qwd, qzd, sd = (torch.from_numpy(t).cuda() for t in (qw, qz, s))
    xd = x.cuda()
    g_idx = (torch.arange(K, dtype=torch.int32) // group + 5).cuda()       # a TP shard's g_idx starts at its first group
    outs = []
    for _ in range(2):
        y = torch.empty(M, N, dtype=F16, device="cuda")
        l.b200_gemm_half_q_half_alt(xd.data_ptr(), qwd.data_ptr(), qzd.data_ptr(), sd.data_ptr(), g_idx.data_ptr(),
                                    y.data_ptr(), M, N, K, bits, torch.cuda.current_stream().cuda_stream)
        _lib.check()
        outs.append(y)
    _close(outs[0], om.linear(x, W), 2e-3, 2e-3)
    assert torch.equal(outs[0], outs[1])
    l.b200_gemm_half_q_half_alt_release()
    _lib.check()


@pytest.mark.parametrize("fmt,K,N,M,group", [("awq", 4096, 6144, 32, 128), ("gptq", 2048, 1024, 5, 128),
                                             ("gptq_sym", 1024, 512, 70, 256), ("awq", 4096, 14336, 1, 128)])
def test_marlin_bf16_entry_points(ops, fmt, K, N, M, group):
    """marlin_awq_4bit_bf16 / marlin_4bit_bf16 (gptq.rs:150-178) with the reference's argument list: bf16 activations,
    bf16 scales, bf16 output.  Checked against the exact product of the bf16 inputs (fp64) within bf16 output
    rounding, and against the reference-style pipeline (weights rounded to bf16 first) within its own error."""
    from vllm_rs_b200 import _lib
    l = _lib.lib()
    BF = torch.bfloat16
    qw, qz, s, W, x = _wna_case(K, N, M, fmt, 4, seed=K + N + M + 1, group=group)
    s_bf = torch.from_numpy(s.astype(np.float32)).to(BF)              # the loader casts the scales to the model dtype
    x_bf = x.to(BF)
    q = oq.unpack_awq(qw) if fmt == "awq" else oq.unpack_gptq(qw, 4)
    if qz is None:
        z = np.full((K // group, N), 8, dtype=np.int32)
    else:
        z = oq.unpack_awq(qz).astype(np.int32) if fmt == "awq" else oq.unpack_gptq_zeros(qz, 4)
    gi = np.arange(K) // group
    d = torch.from_numpy((q.astype(np.int32) - z[gi]).astype(np.float64))
    sg = s_bf.double()[torch.from_numpy(gi)]
    truth = x_bf.double() @ (d * sg)
    w_ref = (d * sg).to(BF)                                           # Marlin bf16: the weight is rounded to bf16
    ref = (x_bf.double() @ w_ref.double()).to(BF)
    qwd = torch.from_numpy(qw).cuda()
    packed = ops.awq_prepack(qwd) if fmt == "awq" else ops.gptq_prepack(qwd, 4)
    ws = ops.wna16_workspace(max(M, 16), N)
    zd = None if qz is None else torch.from_numpy(qz).cuda()
    xd, sd = x_bf.cuda(), s_bf.cuda()
    y = torch.empty(M, N, dtype=BF, device="cuda")
    fn = l.b200_marlin_awq_4bit_bf16 if fmt == "awq" else l.b200_marlin_4bit_bf16
    fn(xd.data_ptr(), packed.data_ptr(), sd.data_ptr(), 0 if zd is None else zd.data_ptr(), 0, y.data_ptr(),
       M, K, N, ws.data_ptr(), group, torch.cuda.current_stream().cuda_stream)
    _lib.check()
    e_new = (y.cpu().double() - truth).abs().max().item()
    e_ref = (ref.double() - truth).abs().max().item()
    scale = truth.abs().max().item()
    assert e_new <= 2.0 ** -8 * scale + 1e-3, (e_new, scale)          # half a bf16 ulp of the largest output, + slack
    assert e_new <= e_ref + 2.0 ** -9 * scale, (e_new, e_ref)         # never worse than the reference-style pipeline
    assert int(ws[:16384].view(torch.int32).abs().sum()) == 0


def test_prepack_bit_exact(ops):
    """Prepacked words decode back to the checkpoint nibbles (layout in include/b200_vllm.h)."""
    rng = np.random.default_rng(5)
    K, N = 256, 256
    q = rng.integers(0, 16, size=(K, N), dtype=np.uint8)
    for fmt in ("awq", "gptq"):
        qw = oq.pack_awq(q) if fmt == "awq" else oq.pack_gptq(q, 4)
        d = torch.from_numpy(qw).cuda()
        p = (ops.awq_prepack(d) if fmt == "awq" else ops.gptq_prepack(d, 4)).cpu().numpy()
        p = p.view(np.uint32).reshape(N // 128, K // 64, 2, 128, 4)
        dec = np.zeros((K, N), dtype=np.uint8)
        for pnib in range(8):
            j = 2 * pnib if pnib < 4 else 2 * (pnib - 4) + 1
            vals = (p >> np.uint32(4 * pnib)) & 0xF            # [nt, kc, h, ch, w]
            nt, kc, h, ch, w = np.meshgrid(*[np.arange(s) for s in p.shape], indexing="ij")
            dec[kc * 64 + h * 32 + w * 8 + j, nt * 128 + ch] = vals
        assert np.array_equal(dec, q), fmt
    q8 = rng.integers(0, 256, size=(K, N), dtype=np.uint8)
    p = ops.gptq_prepack(torch.from_numpy(oq.pack_gptq(q8, 8)).cuda(), 8).cpu().numpy()
    p = p.view(np.uint32).reshape(N // 128, K // 64, 4, 128, 4)
    dec = np.zeros((K, N), dtype=np.uint8)
    for j in range(4):
        vals = (p >> np.uint32(8 * j)) & 0xFF
        nt, kc, h, ch, w = np.meshgrid(*[np.arange(s) for s in p.shape], indexing="ij")
        dec[kc * 64 + h * 16 + w * 4 + j, nt * 128 + ch] = vals
    assert np.array_equal(dec, q8)


def test_wna16_silu_mul_epilogue_and_bias(ops):
    K, inter, M = 1024, 512, 9
    qw, qz, s, W, x = _wna_case(K, 2 * inter, M, "awq", 4, seed=11)
    packed = ops.awq_prepack(torch.from_numpy(qw).cuda())
    ws = ops.wna16_workspace(16, 2 * inter)
    y = ops.wna16_gemm(x.cuda(), packed, torch.from_numpy(s).cuda(), torch.from_numpy(qz).cuda(),
                       ws, k=K, n=2 * inter, epilogue=ops.EPI_SILU_MUL)
    gu = om.linear(x, W)
    _close(y, om.silu_mul(gu[:, :inter], gu[:, inter:]), 2e-3, 4e-3)
    bias = torch.randn(2 * inter).to(F16)
    yb = ops.wna16_gemm(x.cuda(), packed, torch.from_numpy(s).cuda(), torch.from_numpy(qz).cuda(),
                        ws, k=K, n=2 * inter, bias=bias.cuda())
    _close(yb, om.linear(x, W, bias), 3e-3, 2e-3)


def test_dense_gemm(ops):
    g = torch.Generator().manual_seed(2)
    x = torch.randn(32, 1024, generator=g).to(F16)
    w = (torch.randn(4096, 1024, generator=g) * 0.03).to(F16)
    ref = x.float() @ w.float().t()
    _close(ops.dense_gemm(x.cuda(), w.cuda(), out_f32=True), ref, 2e-3, 1e-3)
    _close(ops.dense_gemm(x.cuda(), w.cuda()), ref.to(F16), 2e-3, 2e-3)


def test_errors_are_latched(ops):
    from vllm_rs_b200 import _lib
    x = torch.zeros(2, 100, dtype=F16, device="cuda")
    with pytest.raises(_lib.B200Error):
        ops.rmsnorm(x, torch.zeros(100, dtype=F16, device="cuda"), 1e-5)   # hidden % 8 != 0
    ops.rmsnorm(torch.zeros(2, 128, dtype=F16, device="cuda"),
                torch.ones(128, dtype=F16, device="cuda"), 1e-5)           # state cleared


# ---------------------------------------------------------------- prefill attention
@pytest.mark.parametrize("H,Hkv,D,cases", [
    (32, 8, 128, [(37, 0), (64, 0), (65, 0), (130, 64), (1, 0), (200, 128)]),   # (new tokens, cached)
    (32, 4, 64, [(300, 0), (5, 192)]),                                           # TinyLlama shapes
    (8, 8, 128, [(100, 0), (33, 64)]),                                           # MHA
    (4, 2, 64, [(129, 0)]),
])
def test_attention_prefill_paged(ops, H, Hkv, D, cases):
    """Varlen causal prefill over the paged cache vs the oracle, fresh prompts and chunks that
    attend to cached context (runner.rs:1068-1082).  Stale rows past the context are NaN."""
    g = torch.Generator().manual_seed(H * D + len(cases))
    B = len(cases)
    ctxs = [n + c for n, c in cases]
    nblk = [-(-c // 64) for c in ctxs]
    nb = sum(nblk) + 3
    perm = torch.randperm(nb, generator=g).tolist()
    kc = torch.randn(nb, 64, Hkv, D, generator=g).to(F16)
    vc = torch.randn(nb, 64, Hkv, D, generator=g).to(F16)
    bt = torch.zeros(B, max(nblk), dtype=torch.int32)
    off = 0
    for b, n in enumerate(nblk):
        bt[b, :n] = torch.tensor(perm[off:off + n], dtype=torch.int32)
        off += n
    ref = None
    cu = [0]
    for n, _ in cases:
        cu.append(cu[-1] + n)
    T = cu[-1]
    q = torch.randn(T, H, D, generator=g).to(F16)
    scale = 1.0 / math.sqrt(D)
    dummy = torch.zeros(T, Hkv, D, dtype=F16)           # keys / values come from the paged cache
    ref = om.attention_prefill(q, dummy, dummy, cu, kc, vc, bt.tolist(), ctxs, scale)
    for b, n in enumerate(nblk):                       # poison the tail of every last page
        last = ctxs[b] % 64
        if last:
            kc[bt[b, n - 1], last:] = float("nan")
            vc[bt[b, n - 1], last:] = float("nan")
    out = ops.attention_prefill(q.cuda(), kc.cuda(), vc.cuda(),
                                torch.tensor(cu, dtype=torch.int32).cuda(),
                                torch.tensor(ctxs, dtype=torch.int32).cuda(), bt.cuda(),
                                max(n for n, _ in cases), scale)
    assert not torch.isnan(out).any()
    _close(out, ref, 2e-3, 2e-3)


@pytest.mark.parametrize("M", [100, 256, 300, 700])
def test_wna16_gemm_prefill_sizes(ops, M):
    """tcgen05 variant at prefill token counts (NT = 128 / 256, several token tiles)."""
    K, N = 1024, 512
    qw, qz, s, W, x = _wna_case(K, N, M, "awq", 4, seed=M)
    packed = ops.awq_prepack(torch.from_numpy(qw).cuda())
    ws = ops.wna16_workspace(M, N)
    y = ops.wna16_gemm(x.cuda(), packed, torch.from_numpy(s).cuda(), torch.from_numpy(qz).cuda(), ws,
                       k=K, n=N, variant=2)
    _close(y, om.linear(x, W), 2e-3, 2e-3)


# ---------------------------------------------------------------- cache::swap_blocks (data path)
@pytest.mark.parametrize("dtype", [torch.float16, torch.uint8])
def test_swap_blocks_gpu_cpu_round_trip(ops, dtype):
    """swap_kvcache (runner.rs:1626-1645): GPU -> pinned CPU swap space -> other GPU blocks, whole blocks by
    a {src: dst} mapping in one launch per cache tensor; byte-exact, untouched blocks stay untouched."""
    g = torch.Generator().manual_seed(5)
    nb_gpu, nb_cpu, Hkv, D = 24, 16, 8, 128
    gpu = torch.randint(0, 255, (nb_gpu, 64, Hkv, D), generator=g, dtype=torch.uint8)
    if dtype == torch.float16:
        gpu = torch.randn(nb_gpu, 64, Hkv, D, generator=g).to(dtype)
    ref_gpu = gpu.clone()
    ref_cpu = torch.zeros(nb_cpu, 64, Hkv, D, dtype=dtype)
    cpu = torch.zeros(nb_cpu, 64, Hkv, D, dtype=dtype).pin_memory()
    dgpu = gpu.cuda()
    out_map = {3: 7, 20: 0, 11: 15, 0: 1}                      # swap out: GPU block -> CPU block
    keep = ops.swap_blocks(dgpu, cpu, out_map)
    torch.cuda.synchronize()
    for s, d in out_map.items():
        ref_cpu[d] = ref_gpu[s]
    assert torch.equal(cpu, ref_cpu)
    in_map = {7: 22, 0: 5, 15: 3, 1: 9}                        # swap in: CPU block -> (different) GPU block
    keep = ops.swap_blocks(cpu, dgpu, in_map)
    torch.cuda.synchronize()
    for s, d in in_map.items():
        ref_gpu[d] = ref_cpu[s]
    assert torch.equal(dgpu.cpu(), ref_gpu)
    # device to device (the PD transfer path uses the same call between two GPU caches)
    dst = torch.zeros_like(dgpu)
    keep = ops.swap_blocks(dgpu, dst, [(i, nb_gpu - 1 - i) for i in range(nb_gpu)])
    torch.cuda.synchronize()
    assert torch.equal(dst.cpu(), ref_gpu.flip(0))
    del keep


# ---------------------------------------------------------------- bf16 flavours (the reference's default dtype)
BF16 = torch.bfloat16
# one bf16 ulp is 8 fp16 ulps: the fp16 bars above, times 8


def test_bf16_glue(ops):
    g = torch.Generator().manual_seed(3)
    with om.model_dtype(BF16):
        T, hidden = 9, 4096
        x = torch.randn(T, hidden, generator=g).to(BF16)
        w = (1 + 0.1 * torch.randn(hidden, generator=g)).to(BF16)
        out = ops.rmsnorm(x.cuda(), w.cuda(), 1e-5)
        assert out.dtype == BF16
        _close(out, om.rmsnorm(x, w, 1e-5), 1.6e-2, 8e-3)
        res = torch.randn(T, hidden, generator=g).to(BF16)
        res_d = res.cuda().clone()
        out2 = ops.add_rmsnorm(res_d, x.cuda(), w.cuda(), 1e-5)
        new_res = (res.float() + x.float()).to(BF16)              # the add rounds once, to bf16
        assert torch.equal(res_d.cpu(), new_res)
        _close(out2, om.rmsnorm(new_res, w, 1e-5), 1.6e-2, 8e-3)
        gu = torch.randn(5, 2 * 5632, generator=g).to(BF16)
        _close(ops.silu_mul(gu.cuda()), om.silu_mul(gu[:, :5632], gu[:, 5632:]), 8e-3, 1.6e-2)
        table = torch.randn(1000, 256, generator=g).to(BF16)
        ids = torch.randint(0, 1000, (17,), generator=g, dtype=torch.int32)
        assert torch.equal(ops.embedding(table.cuda(), ids.cuda()).cpu(), table[ids.long()])


@pytest.mark.parametrize("H,Hkv,D,f32_tables", [(32, 8, 128, False), (32, 4, 64, True)])
def test_bf16_rope_kv_write(ops, H, Hkv, D, f32_tables):
    cfg = om.ModelConfig(H * D, 1, H, Hkv, D, 64, 64, rope_theta=500000.0, max_pos=4096)
    cos, sin = om.rope_tables(cfg, dtype=torch.float32 if f32_tables else BF16)
    g = torch.Generator().manual_seed(1)
    T, nb = 19, 8
    q = torch.randn(T, H, D, generator=g).to(BF16)
    k = torch.randn(T, Hkv, D, generator=g).to(BF16)
    v = torch.randn(T, Hkv, D, generator=g).to(BF16)
    pos = torch.randint(0, 4096, (T,), generator=g)
    slots = torch.randperm(nb * 64, generator=g)[:T]
    slots[4] = -1
    kc = torch.zeros(nb, 64, Hkv, D, dtype=BF16)
    vc = torch.zeros_like(kc)
    with om.model_dtype(BF16):
        q_ref, k_ref = om.apply_rope(q, k, cos, sin, pos)
    om.kv_write(k_ref, v, kc, vc, slots)
    qd, kd, vd = q.cuda(), k.cuda(), v.cuda()
    kcd, vcd = torch.zeros_like(kc).cuda(), torch.zeros_like(vc).cuda()
    ops.rope_kv_write(qd, kd, vd, cos.cuda(), sin.cuda(), pos.cuda(), slots.cuda(), kcd, vcd)
    _close(qd, q_ref, 1.6e-2, 8e-3)
    _close(kd, k_ref, 1.6e-2, 8e-3)
    exp_k = torch.zeros_like(kc)
    om.kv_write(kd.cpu(), v, exp_k, torch.zeros_like(vc), slots)
    assert torch.equal(kcd.cpu(), exp_k)
    assert torch.equal(vcd.cpu(), vc)


@pytest.mark.parametrize("H,Hkv,D,ctxs", [
    (32, 8, 128, [1, 63, 64, 65, 127, 129, 700, 4096]),
    (32, 4, 64, [37, 1, 500, 0, 2048]),
    (16, 1, 128, [130]),
])
def test_bf16_paged_attention_decode(ops, H, Hkv, D, ctxs):
    B = len(ctxs)
    q, kc, vc, bt, cl = (t.to(BF16) if t.dtype == F16 else t for t in _paged_case(B, H, Hkv, D, ctxs, seed=H + D))
    scale = 1.0 / math.sqrt(D)
    with om.model_dtype(BF16):
        ref = om.paged_attention_decode(q, kc, vc, bt.tolist(), cl.tolist(), scale)
    out = ops.paged_attention_decode(q.cuda(), kc.cuda(), vc.cuda(), bt.cuda(), cl.cuda(), scale)
    assert out.dtype == BF16
    _close(out, ref, 1.6e-2, 1.6e-2)
    # the fp16 kernel on the same (bf16-representable) values agrees to the bf16 rounding of the output
    out16 = ops.paged_attention_decode(q.to(F16).cuda(), kc.to(F16).cuda(), vc.to(F16).cuda(), bt.cuda(), cl.cuda(),
                                       scale)
    _close(out, out16, 1.6e-2, 1.6e-2)


@pytest.mark.parametrize("H,Hkv,D,cases,mode", [
    (32, 8, 128, [(37, 0), (64, 0), (65, 0), (130, 64), (1, 0), (200, 128)], -1),     # tcgen05 kernel
    (32, 8, 128, [(70, 0), (5, 192)], 0),                                             # mma.sync kernel
    (32, 4, 64, [(300, 0), (5, 192)], -1),
])
def test_bf16_attention_prefill_paged(ops, H, Hkv, D, cases, mode):
    g = torch.Generator().manual_seed(H * D + len(cases))
    B = len(cases)
    ctxs = [n + c for n, c in cases]
    nblk = [-(-c // 64) for c in ctxs]
    nb = sum(nblk) + 3
    perm = torch.randperm(nb, generator=g).tolist()
    kc = torch.randn(nb, 64, Hkv, D, generator=g).to(BF16)
    vc = torch.randn(nb, 64, Hkv, D, generator=g).to(BF16)
    bt = torch.zeros(B, max(nblk), dtype=torch.int32)
    off = 0
    for b, n in enumerate(nblk):
        bt[b, :n] = torch.tensor(perm[off:off + n], dtype=torch.int32)
        off += n
    cu = [0]
    for n, _ in cases:
        cu.append(cu[-1] + n)
    T = cu[-1]
    q = torch.randn(T, H, D, generator=g).to(BF16)
    scale = 1.0 / math.sqrt(D)
    dummy = torch.zeros(T, Hkv, D, dtype=BF16)
    with om.model_dtype(BF16):
        ref = om.attention_prefill(q, dummy, dummy, cu, kc, vc, bt.tolist(), ctxs, scale)
    for b, n in enumerate(nblk):
        last = ctxs[b] % 64
        if last:
            kc[bt[b, n - 1], last:] = float("nan")
            vc[bt[b, n - 1], last:] = float("nan")
    out = ops.attention_prefill(q.cuda(), kc.cuda(), vc.cuda(), torch.tensor(cu, dtype=torch.int32).cuda(),
                                torch.tensor(ctxs, dtype=torch.int32).cuda(), bt.cuda(),
                                max(n for n, _ in cases), scale, mode=mode)
    assert out.dtype == BF16 and not torch.isnan(out).any()
    _close(out, ref, 1.6e-2, 1.6e-2)


# ---------------------------------------------------------------- the reference's default-build cache layout (L1)
# kvcache_allocator.rs:150-173: K [nb, Hkv, D/8, 64, 8], V [nb, Hkv, D, 64].  Same oracle, caches permuted.
@pytest.mark.parametrize("dt", [F16, BF16])
@pytest.mark.parametrize("H,Hkv,D", [(32, 8, 128), (32, 4, 64)])
def test_l1_layout_cache_writes(ops, H, Hkv, D, dt):
    cfg = om.ModelConfig(H * D, 1, H, Hkv, D, 64, 64, rope_theta=500000.0, max_pos=4096)
    cos, sin = om.rope_tables(cfg, dtype=dt)
    g = torch.Generator().manual_seed(5)
    T, nb = 23, 6
    q = torch.randn(T, H, D, generator=g).to(dt)
    k = torch.randn(T, Hkv, D, generator=g).to(dt)
    v = torch.randn(T, Hkv, D, generator=g).to(dt)
    pos = torch.randint(0, 4096, (T,), generator=g)
    slots = torch.randperm(nb * 64, generator=g)[:T]
    slots[7] = -1
    zeros = torch.zeros(nb, 64, Hkv, D, dtype=dt)
    # reshape_and_cache only
    kc1, vc1 = (t.cuda() for t in om.to_l1_layout(zeros, zeros))
    ops.kv_write(k.cuda(), v.cuda(), kc1, vc1, slots.cuda())
    exp_k, exp_v = zeros.clone(), zeros.clone()
    om.kv_write(k, v, exp_k, exp_v, slots)
    got_k, got_v = om.from_l1_layout(kc1.cpu(), vc1.cpu())
    assert torch.equal(got_k, exp_k) and torch.equal(got_v, exp_v)
    # RoPE + cache write in one launch: the same rotated values as the flash-layout call, at the L1 positions
    qd, kd = q.cuda(), k.cuda()
    kc1, vc1 = (t.cuda() for t in om.to_l1_layout(zeros, zeros))
    ops.rope_kv_write(qd, kd, v.cuda(), cos.cuda(), sin.cuda(), pos.cuda(), slots.cuda(), kc1, vc1)
    q2, k2 = q.cuda(), k.cuda()
    kc2, vc2 = zeros.clone().cuda(), zeros.clone().cuda()
    ops.rope_kv_write(q2, k2, v.cuda(), cos.cuda(), sin.cuda(), pos.cuda(), slots.cuda(), kc2, vc2)
    assert torch.equal(qd, q2) and torch.equal(kd, k2)
    got_k, got_v = om.from_l1_layout(kc1.cpu(), vc1.cpu())
    assert torch.equal(got_k, kc2.cpu()) and torch.equal(got_v, vc2.cpu())


@pytest.mark.parametrize("dt", [F16, BF16])
@pytest.mark.parametrize("H,Hkv,D,ctxs", [
    (32, 8, 128, [1, 63, 64, 65, 127, 129, 700, 4096]),
    (32, 4, 64, [37, 1, 500, 0, 2048]),
    (16, 1, 128, [130]),
])
def test_l1_layout_paged_attention_decode(ops, H, Hkv, D, ctxs, dt):
    B = len(ctxs)
    q, kc, vc, bt, cl = (t.to(dt) if t.dtype == F16 else t for t in _paged_case(B, H, Hkv, D, ctxs, seed=H + D + 1))
    scale = 1.0 / math.sqrt(D)
    with om.model_dtype(dt):
        ref = om.paged_attention_decode(q, kc, vc, bt.tolist(), cl.tolist(), scale)
    for b, c in enumerate(ctxs):                       # stale rows past the context must not leak
        if c % 64:
            kc[bt[b, (c - 1) // 64], c % 64:] = float("nan")
            vc[bt[b, (c - 1) // 64], c % 64:] = float("nan")
    k1, v1 = om.to_l1_layout(kc, vc)
    out = ops.paged_attention_decode(q.cuda(), k1.cuda(), v1.cuda(), bt.cuda(), cl.cuda(), scale)
    assert not torch.isnan(out).any()
    tol = 2e-3 if dt == F16 else 1.6e-2
    _close(out, ref, tol, tol)
    # and it is the flash-layout kernel's answer to the last bit of the dtype: same MMAs on the same fragments
    out2 = ops.paged_attention_decode(q.cuda(), kc.cuda(), vc.cuda(), bt.cuda(), cl.cuda(), scale)
    assert torch.equal(out, out2)


@pytest.mark.parametrize("dt,mode", [(F16, -1), (BF16, -1), (F16, 0)])
@pytest.mark.parametrize("H,Hkv,D,cases", [
    (32, 8, 128, [(37, 0), (64, 0), (65, 0), (130, 64), (1, 0), (200, 128)]),
    (32, 4, 64, [(300, 0), (5, 192)]),
])
def test_l1_layout_attention_prefill(ops, H, Hkv, D, cases, dt, mode):
    g = torch.Generator().manual_seed(H * D + len(cases) + 1)
    B = len(cases)
    ctxs = [n + c for n, c in cases]
    nblk = [-(-c // 64) for c in ctxs]
    nb = sum(nblk) + 3
    perm = torch.randperm(nb, generator=g).tolist()
    kc = torch.randn(nb, 64, Hkv, D, generator=g).to(dt)
    vc = torch.randn(nb, 64, Hkv, D, generator=g).to(dt)
    bt = torch.zeros(B, max(nblk), dtype=torch.int32)
    off = 0
    for b, n in enumerate(nblk):
        bt[b, :n] = torch.tensor(perm[off:off + n], dtype=torch.int32)
        off += n
    cu = [0]
    for n, _ in cases:
        cu.append(cu[-1] + n)
    T = cu[-1]
    q = torch.randn(T, H, D, generator=g).to(dt)
    scale = 1.0 / math.sqrt(D)
    dummy = torch.zeros(T, Hkv, D, dtype=dt)
    with om.model_dtype(dt):
        ref = om.attention_prefill(q, dummy, dummy, cu, kc, vc, bt.tolist(), ctxs, scale)
    for b, n in enumerate(nblk):
        last = ctxs[b] % 64
        if last:
            kc[bt[b, n - 1], last:] = float("nan")
            vc[bt[b, n - 1], last:] = float("nan")
    k1, v1 = om.to_l1_layout(kc, vc)
    out = ops.attention_prefill(q.cuda(), k1.cuda(), v1.cuda(), torch.tensor(cu, dtype=torch.int32).cuda(),
                                torch.tensor(ctxs, dtype=torch.int32).cuda(), bt.cuda(),
                                max(n for n, _ in cases), scale, mode=mode)
    assert not torch.isnan(out).any()
    tol = 2e-3 if dt == F16 else 1.6e-2
    _close(out, ref, tol, tol)
