"""The recurrent scans (gated delta rule, decayed linear attention, state-space scan) against the recurrence token by token in 64
bits: sequences that end at, just before and just after a block of eight tokens and the sixteen up to which they are walked token
by token, single tokens on a kept state, sizes with padding, unaligned rows, decays near zero and one, several sequences at once."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device="cuda")


def _walk(q, k, v, decay, w, S, corrected):
    """q, k [T, H, d], v [T, H, e], decay [T, H, d or 1], w [T, H] write strengths, S [H, d, e]."""
    out = torch.empty_like(v)
    for t in range(v.shape[0]):
        S = S * decay[t][:, :, None]
        u = v[t] - (torch.einsum("hd,hde->he", k[t], S) if corrected else 0)
        S = S + torch.einsum("hd,he->hde", k[t], w[t][:, None] * u)
        out[t] = torch.einsum("hd,hde->he", q[t], S)
    return out, S


@pytest.mark.parametrize("lens", [[1], [1, 1, 1], [7, 8, 9], [15, 16, 17], [33, 1, 130]])
@pytest.mark.parametrize("H,G,d,e", [(2, 1, 128, 128), (3, 3, 20, 50), (2, 2, 33, 16), (1, 1, 200, 36), (2, 2, 64, 40)])
@pytest.mark.parametrize("kind", ["delta", "delta_chan", "decay", "decay_chan", "ssd"])
def test_scans(lib, kind, H, G, d, e, lens):
    from vllm_rs_b200 import ops
    if kind.startswith("decay"):
        G = H
    g = torch.Generator().manual_seed(d * e + sum(lens))
    T, n, D = sum(lens), len(lens), torch.float64
    r = lambda *s: torch.randn(*s, generator=g)                               # noqa: E731
    q, k, v, state = r(T, G, d), r(T, G, d), r(T, H, e), r(n + 1, H, d, e)
    slots = torch.randperm(n + 1, generator=g)[:n]
    past = [0 if i % 2 else 5 for i in range(n)]                              # every other sequence starts here
    cu, ctx = _i32([0] + [sum(lens[:i + 1]) for i in range(n)]), _i32([a + b for a, b in zip(lens, past)])
    c = lambda t: t.cuda().contiguous()                                       # noqa: E731
    dev_state, rep = c(state), H // G
    wide = lambda t: t.double().repeat_interleave(rep, 1)                     # noqa: E731
    corrected, skip = kind.startswith("delta"), 0.0
    chan = torch.sigmoid(4 * r(T, H, d)) ** 0.5
    chan[::5, :, 0] = 0.0                                                     # a channel that forgets everything
    if corrected:
        braw, araw, alog, dtb = r(T, H), r(T, H), r(H) * 0.5, r(H)
        unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)      # noqa: E731
        Q, K, w = unit(wide(q)) * d ** -0.5, unit(wide(k)), torch.sigmoid(braw.double())
        dec = torch.exp(-torch.exp(alog.double()) * torch.nn.functional.softplus(araw.double() + dtb.double()))[..., None]
        if kind == "delta":
            got = ops.delta_rule(c(q), c(k), c(v), c(braw), c(araw), c(alog), c(dtb), dev_state, c(slots.int()), cu, ctx)
        else:
            dec = chan.double()
            got = ops.delta_rule_chan(c(q), c(k), c(v), c(braw), c(chan), dev_state, c(slots.int()), cu, ctx)
        V = v.double()
    elif kind == "ssd":
        dt, alog, dtb, dsk = r(T, H), r(H) * 0.5, r(H), r(H)
        w = torch.nn.functional.softplus(dt.double() + dtb.double())
        Q, K, V, skip = wide(q), wide(k), v.double(), dsk.double()[:, None] * v.double()
        dec = torch.exp(-torch.exp(alog.double()) * w)[..., None]
        got = ops.ssd_scan(c(v), c(k), c(q), c(dt), c(alog), c(dtb), c(dsk), dev_state, c(slots.int()), cu, ctx)
    else:
        act = kind == "decay_chan"
        f = torch.nn.functional.silu if act else (lambda t: t)
        Q, K, V, w = f(q.double()) * 0.3, f(k.double()), f(v.double()), torch.full((T, H), 0.7, dtype=D)
        hd = torch.linspace(0.3, 1.0, H)
        dec = chan.double() if act else hd.double()[None, :, None].expand(T, H, 1)
        got = ops.decay_attn(c(q), c(k), c(v), dev_state, c(slots.int()), cu, ctx, q_scale=0.3, k_scale=0.7, act=act,
                             **(dict(chan_decay=c(chan)) if act else dict(head_decay=c(hd))))
    want, want_state, at = torch.empty(T, H, e, dtype=D), state.double().clone(), 0
    for i, m in enumerate(lens):
        if m == 0:                                                            # its state stays
            continue
        sl, s = slice(at, at + m), int(slots[i])
        S0 = state[s].double() if past[i] else torch.zeros(H, d, e, dtype=D)
        want[sl], want_state[s] = _walk(Q[sl], K[sl], V[sl], dec[sl], w[sl], S0, corrected)
        at += m
    want = want + skip
    # fp32 sums of up to d terms, thousands of them below 2^-24 of the largest entries each
    assert (got.double().cpu() - want).abs().max() <= 1e-5 * want.abs().max()
    assert (dev_state.double().cpu() - want_state).abs().max() <= 1e-5 * want_state.abs().max()


# More column blocks x heads x sequences than the chip has SMs: 32 columns per block, and blocks that walk several sequences (16
# heads of 128 x 128: 4 x 16 x 9 blocks for 24 sequences), odd and even numbers of blocks of eight tokens one after another.
MANY = [17, 2, 24, 70, 1, 25, 0, 33, 40, 16, 9, 18]


@pytest.mark.parametrize("e", [128, 40])
@pytest.mark.parametrize("kind", ["delta", "delta_chan", "decay", "decay_chan", "ssd"])
def test_many_sequences(lib, kind, e):
    test_scans(lib, kind, 16, 8, 128, e, MANY + [m + 1 if m > 16 else m for m in MANY[::-1]])


@pytest.mark.parametrize("H,G,d,e", [(2, 1, 128, 128), (3, 3, 20, 50), (1, 1, 200, 36)])
@pytest.mark.parametrize("kind", ["delta", "delta_chan", "decay", "decay_chan", "ssd"])
def test_ends_of_blocks(lib, kind, H, G, d, e):
    test_scans(lib, kind, H, G, d, e, [23, 24, 25])
    test_scans(lib, kind, H, G, d, e, [0, 6, 0, 31, 32])


@pytest.mark.parametrize("H,G,d,e,lens", [(2, 1, 128, 128, [300]),            # four blocks of columns share what they prepare
                                          (2, 2, 64, 96, [65, 66]),            # two do
                                          (40, 20, 128, 64, [200, 1, 150]),    # two of 32 columns; a short sequence between
                                          (2, 1, 200, 256, [257]), (3, 1, 128, 40, [130])])      # unaligned rows; alone
@pytest.mark.parametrize("kind", ["delta", "delta_chan", "decay", "decay_chan", "ssd"])
def test_shared_preparation(lib, kind, H, G, d, e, lens):
    test_scans(lib, kind, H, G, d, e, lens)


@pytest.mark.parametrize("d,e", [(128, 128), (256, 64)])
@pytest.mark.parametrize("kind", ["delta", "decay"])
def test_long_portion_beside_decoded_tokens(lib, kind, d, e):
    """Short sequences on average with a long one among them go to two launches by their length, and every one has the bits that it has
    alone (one launch, shared or not)."""
    from vllm_rs_b200 import ops
    lens, H, G = [1, 600, 20, 1, 113, 64, 1, 65, 16, 17, 33, 112, 0, 1] + [1] * 30, 4, 2 if kind == "delta" else 4
    g = torch.Generator().manual_seed(d)
    r = lambda *s: torch.randn(*s, generator=g).cuda()                        # noqa: E731
    T, n = sum(lens), len(lens)
    q, k, v, b, a, alog, dtb, state = r(T, G, d), r(T, G, d), r(T, H, e), r(T, H), r(T, H), r(H) - 1, r(H), r(n, H, d, e)
    dec = torch.linspace(0.9, 1.0, H).cuda()

    def run(i, j, st):
        at, T = sum(lens[:i]), sum(lens[i:j])
        x = [t[at:at + T] for t in (q, k, v, b, a)]
        tail = (st, torch.arange(i, j).int().cuda(), _i32([sum(lens[i:m]) for m in range(i, j + 1)]), _i32([m + 3 for m in lens[i:j]]))
        if kind == "delta":
            return ops.delta_rule(*x, alog, dtb, *tail)
        return ops.decay_attn(*x[:3], *tail, head_decay=dec, k_scale=0.1)
    one, many = state.clone(), state.clone()
    got = run(0, n, many)
    want = torch.cat([run(i, i + 1, one) for i in range(n) if lens[i]])
    assert torch.equal(got, want) and torch.equal(many, one)


def test_operands_as_they_lie(lib):
    """Views with other strides and one row per token (the form that mixed types take) give the same bits as packed operands."""
    from vllm_rs_b200 import _lib, ops
    T, G, H, d, e = 21, 2, 4, 36, 20
    g = torch.Generator().manual_seed(5)
    r = lambda *s: torch.randn(*s, generator=g).cuda()                        # noqa: E731
    q, k, v, b, a, alog, dtb, state = r(T, G, d), r(T, G, d), r(T, H, e), r(T, H), r(T, H), r(H), r(H), r(2, H, d, e)
    tail = (_i32([1]), _i32([0, T]), _i32([T + 3]))
    states = [state.clone() for _ in range(3)]
    want = ops.delta_rule(q, k, v, b, a, alog, dtb, states[0], *tail)
    lie = lambda t: torch.stack([t, t + 1], -1).transpose(0, 1).contiguous().transpose(0, 1)[..., 0]      # noqa: E731
    views = ops.delta_rule(lie(q), lie(k), lie(v), lie(b), lie(a), alog, dtb, states[1], *tail)
    row = torch.cat([t.reshape(T, -1) for t in (q, k, v, b, a)], 1).contiguous()
    out, at, n = torch.empty_like(want), row.data_ptr(), G * d
    _lib.lib().b200_delta_rule(out.data_ptr(), at, at + 4 * n, at + 8 * n, row.shape[1], at + 4 * (2 * n + H * e),
                               at + 4 * (2 * n + H * e + H), row.shape[1], alog.data_ptr(), dtb.data_ptr(), states[2].data_ptr(),
                               *(t.data_ptr() for t in tail), 1, H, G, d, e, torch.cuda.current_stream().cuda_stream)
    _lib.check()
    for o, s in ((views, states[1]), (out, states[2])):
        assert torch.equal(o, want) and torch.equal(s, states[0])


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("kind", ["delta", "delta_chan", "decay", "decay_chan", "ssd"])
def test_non_finite_tokens_stay_behind(lib, kind, bad):
    """An entry that is not finite, in a key, a query, a value, a strength or a decay of one token, leaves the outputs before that
    token as they are, wherever in a block of eight it stands."""
    from vllm_rs_b200 import ops
    T, H, d, e = 40, 2, 64, 32
    g = torch.Generator().manual_seed(11)
    r = lambda *s: torch.randn(*s, generator=g).cuda()                        # noqa: E731
    q, k, v, b, a, dec = r(T, H, d), r(T, H, d), r(T, H, e), r(T, H), r(T, H), torch.sigmoid(r(T, H, d) + 2)
    alog, dtb, state, tail = r(H) * 0.5, r(H), r(1, H, d, e), (_i32([0]), _i32([0, T]), _i32([T + 3]))

    def run(**x):
        o = dict(q=q, k=k, v=v, b=b, a=a, dec=dec)
        o.update(x)
        s = state.clone()
        if kind == "delta":
            return ops.delta_rule(o["q"], o["k"], o["v"], o["b"], o["a"], alog, dtb, s, *tail)
        if kind == "delta_chan":
            return ops.delta_rule_chan(o["q"], o["k"], o["v"], o["b"], o["dec"], s, *tail)
        if kind == "ssd":
            return ops.ssd_scan(o["v"], o["k"], o["q"], o["a"], alog, dtb, r(H), s, *tail)
        kw = dict(chan_decay=o["dec"]) if kind == "decay_chan" else dict(head_decay=torch.full((H,), 0.9, device="cuda"))
        return ops.decay_attn(o["q"], o["k"], o["v"], s, *tail, **kw)

    g.manual_seed(12)
    want = run()
    assert torch.isfinite(want).all()
    names = {"delta": "qkvba", "delta_chan": ["q", "k", "v", "b", "dec"], "ssd": "qkva", "decay": "qkv",
             "decay_chan": ["q", "k", "v", "dec"]}[kind]
    for name in names:
        for t in (1, 7, 11, 12, 38):
            x = dict(q=q, k=k, v=v, b=b, a=a, dec=dec)[name].clone()
            x[t].view(-1)[5 % x[t].numel()] = bad
            g.manual_seed(12)
            got = run(**{name: x})
            assert torch.equal(got[:t], want[:t]), (name, t)
            if name == "v" and bad != bad:
                assert not torch.isfinite(got[t]).all()


def test_operands_the_row_form_judges(lib):
    """More value heads than query heads (the first ones count), and tensors whose sign is pending, take the row form."""
    from vllm_rs_b200 import ops
    T, H, d, e = 13, 2, 16, 8
    g = torch.Generator().manual_seed(6)
    r = lambda *s: torch.randn(*s, generator=g).cuda()                        # noqa: E731
    q, k, v, state, hd = r(T, H, d), r(T, H, d), r(T, H + 2, e), r(1, H, d, e), torch.full((H,), 0.8, device="cuda")
    tail = (_i32([0]), _i32([0, T]), _i32([T + 2]))
    run = lambda q, k, v: ops.decay_attn(q, k, v, state.clone(), *tail, head_decay=hd)      # noqa: E731
    want = run(q, k, v[:, :H])
    assert torch.equal(run(q, k, v), want)
    assert torch.equal(run(q, torch._neg_view(-k), v[:, :H]), want)


@pytest.mark.parametrize("kind", ["delta", "delta_chan", "decay", "ssd"])
def test_bits_do_not_tell_the_company(lib, kind):
    """A sequence alone (16 columns per block, its own launch) and among others (32 columns, blocks that walk several)."""
    from vllm_rs_b200 import ops
    H, d, e = 8, 128, 128
    lens = [40, 5, 1, 17, 70, 16, 33, 2, 24, 90]
    T, n = sum(lens), len(lens)
    g = torch.Generator().manual_seed(4)
    r = lambda *s: torch.randn(*s, generator=g).cuda()                        # noqa: E731
    q, k, v, b, a, dec = r(T, H, d), r(T, H, d), r(T, H, e), r(T, H), r(T, H), torch.sigmoid(r(T, H, d) + 2)
    alog, dtb, dsk, state = r(H) * 0.5, r(H), r(H), r(n, H, d, e)

    def run(rows, slots, ns):
        s, tail = state.clone(), (_i32(slots), _i32([0] + [sum(ns[:i + 1]) for i in range(len(ns))]), _i32([m + 3 for m in ns]))
        x = [t[rows].contiguous() for t in (q, k, v, b, a, dec)]
        if kind == "delta":
            o = ops.delta_rule(x[0], x[1], x[2], x[3], x[4], alog, dtb, s, *tail)
        elif kind == "delta_chan":
            o = ops.delta_rule_chan(x[0], x[1], x[2], x[3], x[5], s, *tail)
        elif kind == "ssd":
            o = ops.ssd_scan(x[2], x[1], x[0], x[4], alog, dtb, dsk, s, *tail)
        else:
            o = ops.decay_attn(x[0], x[1], x[2], s, *tail, head_decay=torch.full((H,), 0.9, device="cuda"), act=True)
        return o, s
    out, after = run(slice(0, T), list(range(n)), lens)
    at = 0
    for i, m in enumerate(lens):
        o, s = run(slice(at, at + m), [i], [m])
        assert torch.equal(o, out[at:at + m]) and torch.equal(s[i], after[i]), (i, m)
        at += m


@pytest.mark.parametrize("n", [2, 63, 64, 65])
@pytest.mark.parametrize("kind", ["delta", "decay"])
def test_bits_do_not_tell_the_order(lib, kind, n):
    """Up to 64 sequences of a step are walked longest first, more as they come: every one has the bits that it has alone, in steps of
    equal lengths, short ones and several per block (at most 18 blocks of 32 columns share a head's sequences here)."""
    from vllm_rs_b200 import ops
    H, d, e = 8, 128, 128
    lens = [[40, 5, 90, 17, 16, 1, 40, 33][i % 8] + (i * 29) % 23 * (i % 3) for i in range(n)]
    assert n < 8 or (len(set(lens)) < n and min(lens) <= 16 < 4 * 148 // 32 < sum(m > 16 for m in lens))
    T, at = sum(lens), [sum(lens[:i]) for i in range(n + 1)]
    g = torch.Generator().manual_seed(n)
    r = lambda *s: torch.randn(*s, generator=g).cuda()                        # noqa: E731
    q, k, v, b, a = r(T, H, d), r(T, H, d), r(T, H, e), r(T, H), r(T, H)
    alog, dtb, state, past = r(H) * 0.5, r(H), r(n, H, d, e), [0 if i % 5 == 2 else 3 for i in range(n)]

    def run(first, last):
        rows, ids = slice(at[first], at[last]), list(range(first, last))
        s, tail = state.clone(), (_i32(ids), _i32([at[i] - at[first] for i in range(first, last + 1)]),
                                  _i32([lens[i] + past[i] for i in ids]))
        x = [t[rows].contiguous() for t in (q, k, v, b, a)]
        if kind == "delta":
            return ops.delta_rule(*x, alog, dtb, s, *tail), s
        return ops.decay_attn(*x[:3], s, *tail, head_decay=torch.full((H,), 0.9, device="cuda"), act=True), s
    out, after = run(0, n)
    for i in range(n):
        o, s = run(i, i + 1)
        assert torch.equal(o, out[at[i]:at[i + 1]]) and torch.equal(s[i], after[i]), (i, lens[i])


def test_one_decay_for_long(lib):
    """Hundreds of tokens of one decay and one sign: what a block's decay is off by may not add up from block to block.  Outputs of
    the walk token by token are 0.7e-7 off in the 2-norm, a block's rounded decay by itself made it 2.6e-7."""
    from vllm_rs_b200 import ops
    T, H, d, e = 700, 4, 64, 64
    g = torch.Generator().manual_seed(9)
    q, k, v = (torch.rand(T, H, n, generator=g) for n in (d, d, e))
    hd = 1 - 2.0 ** -(5 + torch.arange(H).float())
    s = torch.zeros(1, H, d, e, device="cuda")
    got = ops.decay_attn(q.cuda(), k.cuda(), v.cuda(), s, _i32([0]), _i32([0, T]), _i32([T]), head_decay=hd.cuda())
    D = torch.float64
    want, S = _walk(q.double(), k.double(), v.double(), hd.double()[None, :, None].expand(T, H, 1), torch.ones(T, H, dtype=D),
                    torch.zeros(H, d, e, dtype=D), False)
    off = lambda a, b: float((a.double().cpu() - b).norm() / b.norm())        # noqa: E731
    # eight roundings per block and state entry of random sign, and one of each decay and sum per output, 2^-25 on average each
    assert off(got, want) <= 1.5e-7 and off(s[0], S) <= 3e-7, (off(got, want), off(s[0], S))
