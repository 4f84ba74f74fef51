"""GPU parity of the tcgen05 prefill attention (csrc/attn_prefill_tc.cu, head_dim 128) against the
CPU oracle (oracle/model.py::attention_prefill), with the mma.sync kernel as a third arm.

Floating point: fp32 scores / softmax on both sides, P rounded to fp16 before the PV product on the
GPU (as flash attention does) => tolerance 2e-3 + 2e-3 |x| on outputs of magnitude <= 1 (the same bar
as the mma.sync kernel's test).  Stale cache rows past the context are poisoned with NaN.
"""
import math

import pytest
import torch

from oracle import model as om

pytestmark = pytest.mark.gpu
F16 = torch.float16


@pytest.fixture(scope="module")
def ops(lib):
    from vllm_rs_b200 import ops as _ops
    return _ops


def _case(H, Hkv, cases, seed, big_scores=False):
    D = 128
    g = torch.Generator().manual_seed(seed)
    B = len(cases)
    ctxs = [n + c for n, c in cases]
    nblk = [-(-c // 64) for c in ctxs]
    nb = sum(nblk) + 3
    perm = torch.randperm(nb, generator=g).tolist()
    kc = torch.randn(nb, 64, Hkv, D, generator=g).to(F16)
    vc = torch.randn(nb, 64, Hkv, D, generator=g).to(F16)
    if big_scores:                       # widely varying row maxima: exercises the lazy-rescale branch
        kc = (kc.float() * torch.linspace(0.2, 6.0, nb).view(nb, 1, 1, 1)).to(F16)
    bt = torch.zeros(B, max(nblk), dtype=torch.int32)
    off = 0
    for b, n in enumerate(nblk):
        bt[b, :n] = torch.tensor(perm[off:off + n], dtype=torch.int32)
        off += n
    cu = [0]
    for n, _ in cases:
        cu.append(cu[-1] + n)
    T = cu[-1]
    q = torch.randn(T, H, D, generator=g).to(F16)
    scale = 1.0 / math.sqrt(D)
    dummy = torch.zeros(T, Hkv, D, dtype=F16)
    ref = om.attention_prefill(q, dummy, dummy, cu, kc, vc, bt.tolist(), ctxs, scale)
    for b, n in enumerate(nblk):         # poison the tail of every last page
        last = ctxs[b] % 64
        if last:
            kc[bt[b, n - 1], last:] = float("nan")
            vc[bt[b, n - 1], last:] = float("nan")
    args = (q.cuda(), kc.cuda(), vc.cuda(), torch.tensor(cu, dtype=torch.int32).cuda(),
            torch.tensor(ctxs, dtype=torch.int32).cuda(), bt.cuda(), max(n for n, _ in cases), scale)
    return args, ref


CASES = [
    (32, 8, [(37, 0), (64, 0), (65, 0), (130, 64), (1, 0), (200, 128)]),     # Llama-3-8B heads, ragged + cached
    (8, 8, [(100, 0), (33, 64)]),                                            # MHA (G = 1: 128 tokens per CTA)
    (8, 1, [(129, 0), (17, 300)]),                                           # TP rank shape, G = 8
    (4, 2, [(700, 0)]),                                                      # G = 2, many pages
]


@pytest.mark.parametrize("H,Hkv,cases", CASES)
def test_attn_prefill_tc_matches_oracle(ops, H, Hkv, cases):
    args, ref = _case(H, Hkv, cases, seed=H * 131 + len(cases))
    errs = {}
    for name, mode in (("mma", ops.ATTN_MMA), ("tc", ops.ATTN_TC), ("tc_swapdesc", ops.ATTN_TC_SWAPDESC)):
        out = ops.attention_prefill(*args, mode=mode).float().cpu()
        nan = int(torch.isnan(out).sum())
        err = (out - ref.float()).abs()
        tol = 2e-3 + 2e-3 * ref.float().abs()
        errs[name] = (nan, float(err[~torch.isnan(err)].max()) if nan < out.numel() else float("nan"),
                      int((err > tol).sum()))
    print(f"H={H} Hkv={Hkv} {cases}: (nan, max err, #bad) = {errs}")
    assert errs["mma"][0] == 0 and errs["mma"][2] == 0
    assert errs["tc"][0] == 0 and errs["tc"][2] == 0, errs


def test_attn_prefill_tc_lazy_rescale_and_long_rows(ops):
    """Row maxima that keep growing along the sequence (scaled key pages) force O rescales; 3000-token
    sequences walk 47 pages through both ring stages and both barrier parities."""
    args, ref = _case(32, 8, [(1000, 0), (3000, 64)], seed=7, big_scores=True)
    out = ops.attention_prefill(*args, mode=ops.ATTN_TC).float().cpu()
    assert not torch.isnan(out).any()
    err = (out - ref.float()).abs()
    assert bool((err <= 3e-3 + 3e-3 * ref.float().abs()).all()), float(err.max())
    # the default dispatch is the tcgen05 kernel: identical bits
    assert torch.equal(out, ops.attention_prefill(*args).float().cpu())


@pytest.mark.parametrize("warp", range(4))
@pytest.mark.parametrize("dt,l1", [(F16, False), (F16, True), (torch.bfloat16, False), (torch.bfloat16, True)])
def test_attn_prefill_tc_one_warp_rescales_at_every_page(ops, dt, l1, warp):
    """Every tile's rows of ONE softmax warp (8 of 32 tokens, four heads each) meet keys whose scores grow by some 2^10 a page,
    so that this warp rescales at every page; the other rows' queries are at right angles to what grows, and their warps run ahead.
    fp64 reference from the rounded operands; the bounds of the other tests of this kernel (weights and results of 16 bits)."""
    H, Hkv, D, n, past = 32, 8, 128, 323, 1000
    ctx, scale = n + past, 1.0 / math.sqrt(D)
    pages = -(-ctx // 64)
    g = torch.Generator().manual_seed(warp)
    u = torch.randn(D, generator=g)
    u /= u.norm()
    q, k = torch.randn(n, H, D, generator=g), torch.randn(ctx, Hkv, D, generator=g)
    q -= (q @ u)[..., None] * u
    q[torch.arange(n) % 32 // 8 == warp] += 32 * u
    k += (2.5 * (torch.arange(ctx) // 64))[:, None, None] * u
    q, k, v = q.to(dt), k.to(dt), torch.randn(ctx, Hkv, D, generator=g).to(dt)
    s = torch.einsum("thd,chd->htc", q.double(), k.double().repeat_interleave(H // Hkv, 1)) * scale
    s += torch.full((n, ctx), float("-inf"), dtype=torch.float64).triu(past + 1)
    ref = torch.einsum("htc,chd->thd", torch.softmax(s, -1), v.double().repeat_interleave(H // Hkv, 1))
    order = torch.randperm(pages + 2, generator=g)[:pages]
    kc, vc = (torch.full((pages + 2, 64, Hkv, D), float("nan"), dtype=dt) for _ in range(2))
    for at, t in ((kc, k), (vc, v)):
        for p in range(pages):
            rows = t[p * 64:(p + 1) * 64]
            at[order[p], :len(rows)] = rows
    if l1:
        kc, vc = om.to_l1_layout(kc, vc)
    out = ops.attention_prefill(q.cuda(), kc.cuda(), vc.cuda(), torch.tensor([0, n], dtype=torch.int32).cuda(),
                                torch.tensor([ctx], dtype=torch.int32).cuda(), order.int()[None].contiguous().cuda(), n, scale,
                                mode=ops.ATTN_TC).double().cpu()
    tol = 2e-3 if dt == F16 else 1.6e-2
    assert not torch.isnan(out).any()
    assert bool(((out - ref).abs() <= tol + tol * ref.abs()).all()), float((out - ref).abs().max())
