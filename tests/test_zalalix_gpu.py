"""Zalalix on the GPU against the plain restatement in tests/zalalix_ref.py: each mechanism alone (as a kernel and as a
one-layer model), whole prompts against token-by-token decoding, portions down to two tokens, unequal batches against
each request alone, pages and slots that are used again, window / kept-token / page edges with inputs made so that the
edge key stands out, keys far back, the first tokens of a sequence, long decoding, several sizes, and greedy generation
through LLMEngine.  fp32 runs are held to 2e-4 of the logits' spread, bf16 runs to 6e-2."""
import numpy as np
import pytest
import torch

import zalalix_ref as R
from fidasun_util import Driver, rel_err
from zalalix_util import (full_cfg, gla_cfg, layer, make_cfg, random_layer, random_schedule, random_tensors,
                          window_cfg)

pytestmark = pytest.mark.gpu
F32_TOL, BF16_TOL = 2e-4, 6e-2


def ref_logits(cfg, tensors, tokens):
    return R.forward(cfg, tensors, tokens, torch.float64).numpy()


def toks(n, vocab, seed):
    return np.random.default_rng(seed).integers(0, vocab, size=n).tolist()


def _i32(a):
    return torch.tensor(a, dtype=torch.int32, device="cuda")


# ------------------------------------------------------------------ each mechanism alone (one-layer models)
@pytest.mark.parametrize("kind,kw", [
    ("lightning", {}),
    ("lightning", dict(heads=1, dim=70, vdim=9, decay=[1.0])),
    ("retention", {}),
    ("retention", dict(heads=5, dim=8, vdim=130, decay=[0.5, 0.9, 0.99, 0.999, 1.0])),
    ("parallel", {}),
    ("parallel", dict(left=window_cfg(heads=9, kv_heads=1, dim=8, vdim=40, mask=None, rot=None, softcap=None),
                      right=gla_cfg(heads=1, dim=136, vdim=8, tau=1.0), left_scale=1.0, right_scale=1.0)),
    ("parallel", dict(left=window_cfg(heads=3, kv_heads=3, dim=32, vdim=64, mask={"size": 64, "keep_first": 0},
                                      rot={"base": 500.0, "dims": 32, "scaling": None}),          # tensor-core form
                      right=gla_cfg(), left_scale=0.0, right_scale=1.0)),
    ("parallel", dict(left=window_cfg(heads=16, kv_heads=2, dim=48, vdim=32, mask={"size": 37, "keep_first": 70}),
                      right=gla_cfg(heads=2, dim=64, vdim=64), left_scale=2.0, right_scale=0.0)),
])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_one_mixer_alone(lib, kind, kw, dtype):
    cfg = make_cfg([layer(kind, mlp=False, **kw)])
    w = random_tensors(cfg, seed=3)
    t = toks(90, cfg["vocab"], 1)
    d = Driver(cfg, w, dtype, trace=True)
    d.step([("a", t)])
    tr = []
    want = R.forward(cfg, w, t, torch.float64, tr).numpy()
    resid = d.runner.trace[0, :len(t)].cpu().numpy()
    tol = F32_TOL if dtype == torch.float32 else BF16_TOL
    assert np.abs(resid - tr[0].numpy()).max() <= tol * np.abs(tr[0].numpy()).max()
    assert rel_err(d.result("a"), want) <= tol


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_dense_feed_forward_and_both_norms(lib, dtype):
    cfg = make_cfg([layer("retention", mlp={"kind": "dense", "ff": 56})], embed_scale=0.25)
    w = random_tensors(cfg, seed=5)
    t = toks(40, cfg["vocab"], 2)
    d = Driver(cfg, w, dtype)
    d.step([("a", t)])
    assert rel_err(d.result("a"), ref_logits(cfg, w, t)) <= (F32_TOL if dtype == torch.float32 else BF16_TOL)


def test_norm_ops(lib):
    from vllm_rs_b200 import ops
    g = torch.Generator().manual_seed(1)
    y, gate = torch.randn(9, 48, generator=g), torch.randn(9, 48, generator=g)
    wn = torch.randn(48, generator=g)
    want = R.norm(y.double(), wn.double(), 1e-5) * torch.sigmoid(gate.double())                 # one group, sigmoid gate
    got = ops.gated_group_norm(y.cuda(), gate.cuda(), wn.cuda(), 48, 1e-5, False, torch.float32, gate_act="sigmoid").cpu()
    assert torch.allclose(got, want.float(), atol=2e-5)
    want = R.rms_unit(y.double().reshape(9, 4, 12), 1e-5).reshape(9, 48) * R.silu(gate.double())   # per head, no weight
    got = ops.gated_group_norm(y.cuda(), gate.cuda(), None, 12, 1e-5, False, torch.float32).cpu()
    assert torch.allclose(got, want.float(), atol=2e-5)
    x, w = torch.randn(9, 48, generator=g) * 4, torch.randn(48, generator=g)
    want = x.double() + R.norm(y.double(), w.double(), 1e-3)
    got = ops.resid_add_rmsnorm(x.cuda(), y.cuda(), w.cuda(), 1e-3).cpu()
    assert torch.allclose(got, want.float(), atol=2e-5)
    low, w2, b = torch.randn(7, 5, generator=g), torch.randn(33, 5, generator=g) * 3, torch.randn(33, generator=g) * 4
    for tau in (1.0, 16.0):
        want = torch.sigmoid(low.double() @ w2.double().T + b.double()) ** (1.0 / tau)
        got = ops.lowrank_decay(low.cuda(), w2.cuda(), b.cuda(), tau).cpu()
        assert torch.allclose(got, want.float(), atol=1e-6, rtol=1e-5)


@pytest.mark.parametrize("dk,dv", [(20, 50), (130, 8), (64, 64)])
@pytest.mark.parametrize("chan", [False, True])
def test_decay_attention_op_in_portions(lib, dk, dv, chan):
    """The kernel alone against the token-by-token recurrence: portions of 1, 2 and many tokens on a slot whose old
    contents are stale; a head whose decay is exactly one keeps a far key at full weight."""
    from vllm_rs_b200 import ops
    g = torch.Generator().manual_seed(4)
    T, H = 300, 3
    q, k, v = torch.randn(T, H, dk, generator=g), torch.randn(T, H, dk, generator=g), torch.randn(T, H, dv, generator=g)
    q[-1] = 30.0 * k[0]                                   # the last query asks for the first token
    v[0] = 100.0
    hd = torch.tensor([1.0, 0.9, 0.999])
    cd = torch.rand(T, H, dk, generator=g) * 0.2 + 0.8
    cd[:, 0] = 1.0
    act, qs, ks = (True, 1.0, dk ** -0.5) if chan else (False, 0.7, 1.0)
    f = (lambda z: R.silu(z.double())) if act else (lambda z: z.double())
    decay = cd.double() if chan else hd.double()[None, :, None].expand(T, H, dk)
    want = torch.stack([R.decayed_state_readout(f(q[:, h]) * qs, f(k[:, h]) * ks, f(v[:, h]), decay[:, h]) for h in range(H)], 1)
    state = torch.full((2, H, dk, dv), 3.0, device="cuda")
    got = []
    for lo, hi in ((0, 1), (1, 3), (3, 30), (30, 299), (299, 300)):
        c = lambda z: z[lo:hi].cuda().contiguous()                             # noqa: E731
        got.append(ops.decay_attn(c(q), c(k), c(v), state, _i32([1]), _i32([0, hi - lo]), _i32([hi]),
                                  head_decay=None if chan else hd.cuda(), chan_decay=c(cd) if chan else None,
                                  q_scale=qs, k_scale=ks, act=act).cpu())
    got = torch.cat(got).numpy()
    for h in range(H):
        assert np.abs(got[:, h] - want[:, h].numpy()).max() <= 2e-5 * want[:, h].abs().max().item(), h
    assert np.abs(want[-1, 0].numpy()).max() > 10.0 * np.abs(want[-1, 1].numpy()).max()   # the far key shows in head 0


# ------------------------------------------------------------------ window, kept tokens and page edges, made to show
def _plain_window_attention(q, k, v, gate, rows_pos, window, keep, scale, cap, sink):
    """q [T, H, dk] at positions rows_pos; k [n, G, dk], v [n, G, dv]: the mask rule spelled out per pair."""
    T, H, _ = q.shape
    G = k.shape[1]
    out = torch.zeros(T, H, v.shape[2], dtype=torch.float64)
    for r, i in enumerate(rows_pos):
        seen = [j for j in range(i + 1) if window <= 0 or i - j < window or j < keep]
        for h in range(H):
            s = (k[seen, h // (H // G)] @ q[r, h]) * scale
            if cap > 0:
                s = cap * torch.tanh(s / cap)
            e = torch.exp(s - s.max())
            den = e.sum() + (torch.exp(-s.max()) if sink else 0.0)
            out[r, h] = (e[:, None] * v[seen, h // (H // G)]).sum(0) / den
            if gate is not None:
                out[r, h] *= torch.sigmoid(gate[r, h])
    return out


@pytest.mark.parametrize("window,keep", [(0, 0), (5, 0), (5, 3), (64, 64), (64, 1), (70, 3), (130, 70), (1, 0)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("split", [True, False])
@pytest.mark.parametrize("dk,dv,H,G", [(12, 20, 4, 2), (32, 64, 3, 1), (16, 160, 2, 1)])   # the last two: tensor-core forms
def test_window_attention_sees_exactly_its_window_and_kept_tokens(lib, window, keep, dtype, split, dk, dv, H, G):
    _check_window_attention(window, keep, dtype, split, dk, dv, H, G)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_window_attention_with_a_group_wider_than_a_tile(lib, dtype):
    """17 query heads per key / value head: more than the 16 rows of an MMA tile and than the warps of a block."""
    _check_window_attention(70, 3, dtype, True, 16, 32, 34, 2, row_sets=([199], [64], list(range(100, 200))))


def _check_window_attention(window, keep, dtype, split, dk, dv, H, G, row_sets=None):
    """Keys carry a position tag u and its square, so a query can put a sharp peak on any position.  Four queries per
    row: a ramp that prefers the earliest visible key, a ramp that prefers the latest, a peak on the key JUST OUTSIDE
    the window's far edge, and a peak on the first key that is NOT kept: had the kernel seen a key one place beyond an
    edge, that key would take most of the weight.  Prompt rows and single decoded rows, edges at page borders and far
    back, on a shuffled block table, against the mask rule spelled out; with and without cap, sink and gate."""
    from vllm_rs_b200 import ops
    n = 200
    pages = [5, 2, 7, 0]
    g = torch.Generator().manual_seed(0)
    u = (torch.arange(n) - 128.0) / 256.0
    k = torch.randn(n, G, dk, generator=g) * 0.05
    k[:, :, 0], k[:, :, 1] = u[:, None], (u * u)[:, None]
    v = torch.randn(n, G, dv, generator=g)
    kc = torch.zeros(8, 64, G, dk, dtype=dtype, device="cuda")
    vc = torch.zeros(8, 64, G, dv, dtype=dtype, device="cuda")
    for j in range(n):
        kc[pages[j // 64], j % 64], vc[pages[j // 64], j % 64] = k[j].to(dtype).cuda(), v[j].to(dtype).cuda()
    kr, vr = k.to(dtype).double(), v.to(dtype).double()
    bt = _i32([pages])
    tol = 2e-3 if dtype == torch.float32 else 4e-2
    sharp = 16384.0
    for rows_pos in row_sets or ([199], [64], [63], [0], list(range(100, 200)), list(range(120, 200)), list(range(0, 70)),
                                 list(range(0, 129))):
        T = len(rows_pos)
        pos = torch.tensor(rows_pos, dtype=torch.float32)
        for form, cap, sink in (("early", 0.0, False), ("early", 300.0, True), ("late", 0.0, True), ("window", 0.0, False),
                                ("kept", 0.0, True)):
            q = torch.randn(T, H, dk, generator=g) * 0.1
            if form in ("early", "late"):
                q[:, :, 0], q[:, :, 1] = (-256.0 if form == "early" else 64.0), 0.0
            else:
                target = (pos - window) if form == "window" else torch.full((T,), float(keep))
                ut = (target - 128.0) / 256.0
                q[:, :, 0], q[:, :, 1] = (2.0 * sharp * ut)[:, None], -sharp
            q = q.to(dtype).float()
            gate = torch.randn(T, H, generator=g)
            sk = torch.zeros(H, device="cuda") if sink else None
            out = ops.window_attn(q.cuda().contiguous(), kc, vc, sk, gate.cuda(), _i32([0, T]), _i32([rows_pos[-1] + 1]),
                                  bt, window=window, keep_first=keep, scale=1.0, softcap=cap, split=split).float().cpu()
            want = _plain_window_attention(q.double(), kr, vr, gate.double(), rows_pos, window, keep, 1.0, cap, sink)
            assert (out.double() - want).abs().max() <= tol * max(1.0, want.abs().max().item()), (rows_pos[0], T, form)


def test_window_attention_prep_op(lib):
    """Biases, whole-projection norms, partial rotary and the cache rows, against the plain formulas."""
    from vllm_rs_b200 import ops
    from vllm_rs_b200.rotary import banded_rotary_frequencies
    g = torch.Generator().manual_seed(3)
    T, H, G, dk, dv, rd = 6, 4, 2, 10, 7, 6
    rot = {"base": 100.0, "dims": rd, "scaling": {"factor": 4.0, "low": 1.0, "high": 3.0, "original": 20}}
    n = H * dk + G * (dk + dv)
    proj = torch.randn(T, n + H, generator=g)                         # gate logits ride along, untouched
    bias, qn, kn = torch.randn(n, generator=g), torch.randn(H * dk, generator=g), torch.randn(G * dk, generator=g)
    pos = torch.tensor([0, 1, 5, 63, 64, 1000])
    slots = torch.tensor([3, 64, 2, 0, 130, 191])
    kc, vc = torch.zeros(3, 64, G, dk, device="cuda"), torch.zeros(3, 64, G, dv, device="cuda")
    freq = torch.from_numpy(banded_rotary_frequencies(rd, rot["base"], rot["scaling"])).cuda()
    q = ops.window_attn_prep(proj.cuda(), bias.cuda(), qn.cuda(), kn.cuda(), freq, pos.cuda(), slots.cuda(), kc, vc,
                             heads=H, rot_dims=rd, eps=1e-4).cpu()
    x = proj.double()[:, :n] + bias.double()
    wq = R.norm(x[:, :H * dk], qn.double(), 1e-4).reshape(T, H, dk)
    wk = R.norm(x[:, H * dk:H * dk + G * dk], kn.double(), 1e-4).reshape(T, G, dk)
    wv = x[:, H * dk + G * dk:].reshape(T, G, dv)
    for t in range(T):
        for h in range(H):
            assert torch.allclose(q[t, h].double(), R.rotate(wq[t, h], int(pos[t]), rot), atol=2e-5)
        s = int(slots[t])
        for a in range(G):
            assert torch.allclose(kc.cpu()[s // 64, s % 64, a].double(), R.rotate(wk[t, a], int(pos[t]), rot), atol=2e-5)
        assert torch.allclose(vc.cpu()[s // 64, s % 64].double(), wv[t], atol=2e-5)


@pytest.mark.parametrize("T,H,G,dk,dv,rd,bias,norm,bf16,vk,extra", [
    (37, 16, 4, 128, 128, 64, True, True, True, False, 16),       # the rows a hybrid step has, part of a head rotated
    (5, 32, 8, 128, 128, 128, True, True, True, False, 0),        # four queries of a thread, the largest table of rotations
    (9, 4, 2, 64, 96, 34, False, True, False, False, 4),          # half a group of four rotated
    (3, 8, 8, 32, 32, 30, True, False, True, True, 8),            # values taken from the keys
    (1, 2, 1, 4, 8, 2, False, False, False, False, 0),            # threads without an entry
    (64, 12, 12, 64, 64, 0, True, True, True, False, 0)])         # no rotation
def test_window_attn_prep_aligned_rows_match_unaligned(lib, T, H, G, dk, dv, rd, bias, norm, bf16, vk, extra):
    """Projections that lie on 16 bytes are read four entries at a time; a view that starts one float further on takes the
    general form.  The sums of squares meet in another order, so fp32 may differ by a few roundings of them (2e-6 of an entry of
    up to the largest value) and bf16 by one step of the larger entry (2^-7)."""
    from vllm_rs_b200 import ops
    g = torch.Generator().manual_seed(T)
    nq, nk, nv = H * dk, G * dk, 0 if vk else G * dv
    n, ld, dt = nq + nk + nv, nq + nk + nv + extra, torch.bfloat16 if bf16 else torch.float32
    proj = torch.randn(T, ld, generator=g).cuda()
    b = torch.randn(n, generator=g).cuda() if bias else None
    qn, kn = (torch.randn(nq, generator=g).cuda(), torch.randn(nk, generator=g).cuda()) if norm else (None, None)
    f = 10000.0 ** (-torch.arange(max(1, rd // 2), dtype=torch.float64) / max(1, rd // 2)).cuda()
    pos, slots = torch.randint(0, 5000, (T,), generator=g).cuda(), torch.randperm(128, generator=g)[:T]
    if T > 4:
        slots[3] = -1                                             # a row that is not kept
    got = []
    for off in (0, 1):
        at = torch.empty(T * ld + 1, device="cuda")[off:off + T * ld].view(T, ld)
        at.copy_(proj)
        kc = torch.zeros(2, 64, G, dk, device="cuda", dtype=dt)
        vc = torch.zeros(2, 64, G, dv, device="cuda", dtype=dt)
        q = ops.window_attn_prep(at, b, qn, kn, f, pos, slots.cuda(), kc, vc, heads=H, rot_dims=rd, eps=1e-6,
                                 v_from_k=vk, q_temp=(0.3, 100), rot_mag=1.1)
        got.append((q, kc, vc))
    for x, y in zip(*got):
        top = max(1.0, y.float().abs().max().item())
        assert (x.float() - y.float()).abs().max().item() <= (2.0 ** -7 if x.dtype == torch.bfloat16 else 2e-6) * top


@pytest.mark.parametrize("H", [8, 16, 32])
def test_window_attn_prep_norms_are_as_exact_in_both_forms(lib, H):
    """Normed queries of aligned rows (sums of squares of four entries a thread) against 64 bits, beside the general form's.  The rows'
    common factor is what the sum's order moves: over 8 x 4096 rows its error is known to half a percent."""
    from vllm_rs_b200 import ops
    T, dk, off = 4096, 128, [0.0, 0.0]
    slots, f = torch.full((T,), -1, device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda")
    kc = torch.zeros(1, 64, 1, dk, device="cuda")
    one = torch.ones(H * dk, device="cuda")
    for seed in range(8):
        g = torch.Generator(device="cuda").manual_seed(seed)
        proj = torch.randn(T, (H + 2) * dk, generator=g, device="cuda")
        x = proj[:, :H * dk].double()
        want = x / torch.sqrt((x * x).mean(1, keepdim=True) + 1e-6)
        for i in (0, 1):
            at = torch.empty(proj.numel() + 1, device="cuda")[i:i + proj.numel()].view(proj.shape)
            at.copy_(proj)
            q = ops.window_attn_prep(at, None, one, one[:dk], f, slots, slots, kc, kc.clone(), heads=H, rot_dims=0, eps=1e-6)
            off[i] += float(((q.reshape(T, -1).double() - want) ** 2).sum() / (want ** 2).sum())
    print(H, [(e / 8) ** 0.5 for e in off])
    assert (off[0] / off[1]) ** 0.5 <= 1.01, [(e / 8) ** 0.5 for e in off]


@pytest.mark.parametrize("window,keep", [(3, 2), (64, 5), (65, 64)])
def test_model_edges_show_in_logits(lib, window, keep):
    """A one-layer model whose recurrent side is switched off: replacing the token at one place changes the last row's
    logits exactly while that place is inside the last row's window or among the kept first tokens (the plain model
    gives identical logits otherwise), by far more than the tolerance; the last row is decoded alone."""
    cfg = make_cfg([layer("parallel", mlp=False, left=window_cfg(mask={"size": window, "keep_first": keep}),
                          right=gla_cfg(), left_scale=1.0, right_scale=0.0)])
    w = random_tensors(cfg, seed=11)
    n = window + keep + 70
    base = toks(n, cfg["vocab"] - 1, 5)
    special = cfg["vocab"] - 1
    other = ref_logits(cfg, w, base)
    for pos_x, visible in ((n - 1 - window, False), (n - window, True), (keep - 1, True), (keep, False)):
        t = list(base)
        t[pos_x] = special
        want = ref_logits(cfg, w, t)
        d = Driver(cfg, w, torch.float32)
        d.step([("a", t[:n - 1])])
        d.step([("a", t[n - 1:])])
        assert rel_err(d.result("a"), want) <= F32_TOL
        diff = np.abs(want[-1] - other[-1]).max()
        assert (diff > 5 * F32_TOL * want.std()) if visible else diff == 0.0, (pos_x, visible)


# ------------------------------------------------------------------ schedules
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_whole_decode_and_portions_agree_with_the_plain_model(lib, dtype):
    cfg = full_cfg()
    w = random_tensors(cfg, seed=7)
    t = toks(150, cfg["vocab"], 3)
    want = ref_logits(cfg, w, t)
    tol = F32_TOL if dtype == torch.float32 else BF16_TOL
    d = Driver(cfg, w, dtype)
    d.step([("whole", t)])
    assert rel_err(d.result("whole"), want) <= tol
    d.close("whole")
    d.step([("dec", t[:60])])
    for x in t[60:]:
        d.step([("dec", [x])])
    assert rel_err(d.result("dec"), want) <= tol
    d.close("dec")
    cuts = [2, 1, 2, 61, 2, 3, 64, 2, 13]                            # 150 tokens; cuts inside pages and windows
    at = 0
    for c in cuts:
        d.step([("cut", t[at:at + c])])
        at += c
    assert at == len(t)
    assert rel_err(d.result("cut"), want) <= tol
    if dtype == torch.float32:                                       # the cut must not matter beyond rounding
        assert rel_err(d.result("cut"), d.result("dec")) <= 2e-5


def test_unequal_batches_and_reuse_of_pages_and_slots(lib):
    cfg = full_cfg()
    w = random_tensors(cfg, seed=9)
    V = cfg["vocab"]
    reqs = {"a": toks(130, V, 1), "b": toks(3, V, 2), "c": toks(70, V, 3), "d": toks(65, V, 4), "e": toks(40, V, 5),
            "f": toks(129, V, 6)}
    want = {k: ref_logits(cfg, w, v) for k, v in reqs.items()}
    d = Driver(cfg, w, torch.float32, num_blocks=7, max_seqs=4, slots=4)      # 7 pages: a(3) + c(2) + d(2) fill it
    at = {k: 0 for k in reqs}

    def portion(k, n):
        p = (k, reqs[k][at[k]:at[k] + n])
        at[k] += n
        return p

    d.step([portion("a", 64), portion("b", 2)])
    d.step([portion("a", 1), portion("b", 1), portion("c", 30)])
    d.close("b")                                                      # its page and slot go back
    d.step([portion("c", 40), portion("a", 2), portion("d", 65)])
    d.step([portion("a", 63)])
    d.close("a"), d.close("c")
    assert d.sched.num_free_blocks == 5 and d.sched.num_free_state_slots == 3
    d.step([portion("e", 39), portion("f", 128)])                     # reuses a's and c's pages and slots
    d.step([portion("f", 1), portion("e", 1)])
    for k in "abcdef":
        assert at[k] == len(reqs[k])
        assert rel_err(d.result(k), want[k]) <= F32_TOL, k


def test_first_tokens_and_long_decoding(lib):
    cfg = full_cfg()
    w = random_tensors(cfg, seed=13)
    t = toks(260, cfg["vocab"], 8)
    want = ref_logits(cfg, w, t)
    d = Driver(cfg, w, torch.float32)
    for x in t:                                                       # every token alone, from the very first
        d.step([("a", [x])])
    got = d.result("a")
    assert rel_err(got[:6], want[:6]) <= F32_TOL
    assert rel_err(got, want) <= F32_TOL


def test_other_sizes(lib):
    """Sizes of one, equal scales, a window of one token, more kept tokens than the window, no feed-forward at all."""
    cfg = make_cfg([layer("parallel", mlp={"kind": "dense", "ff": 7},
                          left=window_cfg(heads=1, kv_heads=1, dim=2, vdim=1, scale=1.0, softcap=0.5,
                                          mask={"size": 1, "keep_first": 4},
                                          rot={"base": 77.0, "dims": 2, "scaling": {"factor": 2.0, "low": 1.0, "high": 2.0, "original": 8}}),
                          right=gla_cfg(heads=1, dim=1, vdim=3, tau=1.0), left_scale=1.0, right_scale=1.0),
                    layer("lightning", mlp=False, heads=1, dim=3, vdim=130, decay=[1.0]),
                    layer("retention", mlp=False, heads=7, dim=17, vdim=5, decay=[0.3] * 7)],
                   width=24, vocab=50, eps=1e-3, embed_scale=1.0)
    w = random_tensors(cfg, seed=17, rank=1)
    t = toks(80, cfg["vocab"], 9)
    want = ref_logits(cfg, w, t)
    d = Driver(cfg, w, torch.float32)
    d.step([("a", t[:7])]), d.step([("a", t[7:9])]), d.step([("a", t[9:])])
    assert rel_err(d.result("a"), want) <= F32_TOL


def test_greedy_generation_through_the_engine(lib):
    """LLMEngine (schedule -> chunked prefill -> decode, state slots from the scheduler) against greedy decoding with
    the plain model."""
    from vllm_rs_b200 import engine, models
    cfg = full_cfg()
    w = random_tensors(cfg, seed=21)
    V = cfg["vocab"]
    prompts = [toks(75, V, 1), toks(5, V, 2), toks(40, V, 3)]
    new = 12
    runner = models.build_runner(cfg, w, dtype=torch.float32, device="cuda", num_blocks=12, max_blocks_per_seq=4,
                                 max_seqs=5, max_tokens=64, num_state_slots=5)
    eng = engine.LLMEngine(runner, 12, 3, chunk_size=32)              # prompts longer than a chunk are cut
    sids = [eng.add_request(p, new) for p in prompts]
    out = eng.run_to_completion()
    for sid, p in zip(sids, prompts):
        seq, want = list(p), []
        for _ in range(new):
            lg = ref_logits(cfg, w, seq)[-1]
            top2 = np.sort(lg)[-2:]
            nxt = int(lg.argmax())
            want.append(nxt)
            seq.append(nxt)
            if top2[1] - top2[0] < 1e-3:                              # a near tie may flip in fp32: stop comparing there
                break
        assert out[sid][:len(want)] == want
    assert eng.sched.num_free_state_slots == 5


# ------------------------------------------------------------------ random configurations under random schedules
@pytest.mark.parametrize("seed", [11, 12, 13, 14, 15, 16])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_random_configurations_under_random_schedules(lib, seed, dtype):
    """Sizes, layer orders and constants drawn at random (key sizes above 128 and odd ones, groups wider than a block's
    warps, windows of one token, no window at all); five requests of 5 .. 420 tokens share four state slots and just
    enough pages, so both are used again.  bf16 runs are judged at the 0.9 quantile of the rows: a recurrent layer
    normalises its read-out per head, so where a head's first read-outs q.k are within rounding of zero their sign,
    and with it the whole normalised head, can flip with 16-bit operands."""
    rng = np.random.default_rng(seed)
    pick = lambda *xs: xs[int(rng.integers(len(xs)))]              # noqa: E731
    kinds = [pick("parallel", "parallel", "lightning", "retention") for _ in range(int(rng.integers(2, 5)))]
    cfg = make_cfg([random_layer(rng, k) for k in kinds], width=pick(64, 128, 192), vocab=pick(300, 512),
                   eps=pick(1e-6, 1e-5), embed_scale=pick(1.0, 8.0, 11.3))
    w = random_tensors(cfg, seed=seed, rank=pick(1, 4, 16))
    reqs = {f"r{i}": toks(pick(5, 40, 150, 260, 420), cfg["vocab"], seed + i) for i in range(5)}
    pages = sum(sorted((len(v) + 63) // 64 for v in reqs.values())[-4:])
    d = Driver(cfg, w, dtype, num_blocks=pages, max_seqs=4, slots=4)
    for st, ends in random_schedule(rng, reqs):
        d.step(st)
        for k in ends:
            d.close(k)
    tol, q = (F32_TOL, 1.0) if dtype == torch.float32 else (BF16_TOL, 0.9)
    for k, v in reqs.items():
        assert rel_err(d.result(k), ref_logits(cfg, w, v), q) <= tol, (k, kinds)


@pytest.mark.parametrize("T,width,off", [(3, 4, 0), (2, 1020, 0), (37, 2048, 0), (5, 4096, 0), (3, 4100, 0), (3, 2047, 0), (4, 512, 1)])
@pytest.mark.parametrize("dt", [0, 1])
def test_norm_after_update(T, width, off, dt):
    """The norm made with the update of the stream against the two launches, aligned or not, wider than the registers or not.  The
    stream's bits are the same.  The squares meet in the same tree, of at most 16 terms and 8 levels, but not with the same multiplies
    fused: 24 roundings of 2^-24 on either side, halved by the root, are below 2^-18; bf16 rounds to the neighbour at worst."""
    import ctypes
    from vllm_rs_b200 import _lib
    g = torch.Generator().manual_seed(width)
    row = lambda *n: torch.randn(*n, generator=g).cuda()                       # noqa: E731
    rows = torch.randn(T * width + off, generator=g).cuda()
    x, xs = rows[off:], rows.clone()[off:]                  # both at the same offset: the two sides sum in the same order
    y, w, w2 = row(T, width), row(width), row(width)
    outs = [torch.zeros(T, width, dtype=torch.float32 if dt else torch.bfloat16, device="cuda") for _ in range(2)]
    p = lambda t: None if t is None else ctypes.c_void_p(t.data_ptr())         # noqa: E731
    f, i, L = ctypes.c_float, ctypes.c_int, _lib.lib()
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    add = getattr(L, "_ZN4b20024launch_resid_add_rmsnormEPfPKfS2_iiffPvP11CUstream_stS3_S2_i")
    norm = getattr(L, "_ZN4b20020launch_resid_rmsnormEPvPKfS2_iiffPKjiP11CUstream_sti")
    add(p(x), p(y), p(w), T, width, f(1e-6), f(1.0), None, st, p(outs[0]), p(w2), i(dt))
    add(p(xs), p(y), p(w), T, width, f(1e-6), f(1.0), None, st, None, None, i(0))
    norm(p(outs[1]), p(xs), p(w2), T, width, f(1e-6), f(1.0), None, i(dt), st, i(0))
    torch.cuda.synchronize()
    _lib.check()
    a, b = (o.double() for o in outs)
    assert torch.equal(x, xs) and ((a - b).abs() <= b.abs() * (2.0 ** -18 if dt else 2.0 ** -7)).all() and float(b.abs().sum()) > 0


@pytest.mark.parametrize("T,n,off", [(1, 8, 0), (5, 1032, 0), (300, 2048, 0), (3, 4096, 0), (3, 36, 0), (2, 512, 1)])
def test_row_kernels_wide_and_not(T, n, off):
    """Embedding rows and bias rows by wide accesses and by single entries: exact products and one fused multiply-add, so exact
    against the same in 64 bits rounded once (bias), or in 32 bits (a power of two as scale)."""
    import ctypes
    from vllm_rs_b200 import _lib
    g = torch.Generator().manual_seed(n)
    L, st = _lib.lib(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = lambda t: None if t is None else ctypes.c_void_p(t.data_ptr())         # noqa: E731
    f, i = ctypes.c_float, ctypes.c_int
    embed = getattr(L, "_ZN4b20016launch_embed_f32EPfPKvPKjPKlfiiifiPvP11CUstream_st")
    ids = torch.randint(0, 12, (T,), generator=g)                             # 11 is out of range: row 0
    rows = torch.where(ids < 11, ids, torch.zeros_like(ids))
    for dt, ty in ((0, torch.bfloat16), (1, torch.float32)):
        table = torch.randn(11 * n + off, generator=g).to(ty).cuda()[off:]
        x, cast = torch.zeros(T, n, device="cuda"), torch.zeros(T, n, dtype=ty, device="cuda")
        embed(p(x), p(table), p(_i32(ids.tolist())), None, f(0.0), T, n, 11, f(4.0), i(dt), p(cast), st)
        want = table.view(11, n)[rows.cuda()].float() * 4
        assert torch.equal(x, want) and (dt or torch.equal(cast, want.to(ty)))
    y = torch.randn(T * n + off, generator=g).cuda()[off:]
    b = torch.randn(n, generator=g).cuda()
    want = (y.view(T, n).double() + 0.75 * b.double()).float()
    getattr(L, "_ZN4b20016launch_bias_rowsEPfPKffiiP11CUstream_st")(p(y), p(b), f(0.75), T, n, st)
    torch.cuda.synchronize()
    _lib.check()
    assert torch.equal(y.view(T, n), want)


@pytest.mark.parametrize("T,C,rank", [(1, 1, 4), (17, 300, 16), (16, 256, 6), (40, 33, 12)])
def test_lowrank_decay_tiles(lib, T, C, rank):
    """Tiles of 16 tokens, rows of w2 by four entries where the rank allows it.  exp and log1p are within 2 units, z within rank + 1
    roundings of its terms: the bound of the op's other test holds."""
    from vllm_rs_b200 import ops
    g = torch.Generator().manual_seed(T * C)
    low, w2, b = torch.randn(T, rank, generator=g), torch.randn(C, rank, generator=g), torch.randn(C, generator=g) * 4
    want = torch.sigmoid(low.double() @ w2.double().T + b.double()) ** (1.0 / 16.0)
    got = ops.lowrank_decay(low.cuda(), w2.cuda(), b.cuda(), 16.0).cpu()
    assert torch.allclose(got, want.float(), atol=1e-6, rtol=1e-5)
