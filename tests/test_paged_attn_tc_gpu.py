"""The tcgen05 attention of the hybrid decoders (grouped heads and latent rows) against plain 64-bit attention, at the sizes
where its tiles end: groups that do not divide 128 rows, key rows with a 32-wide tail, several passes over the value columns,
queries kept in tensor memory, split keys, windows and chunks that start inside a page, cache rows that hold NaN."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
D64 = torch.float64


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device="cuda")


def _pages(g, ctxs, shape):
    """A cache of scattered pages filled with NaN, its block table, and a writer of a sequence's rows."""
    need = [-(-c // 64) for c in ctxs]
    perm = torch.randperm(sum(need) + 2, generator=g).tolist()
    cache = torch.full((len(perm), 64, *shape), float("nan"), dtype=torch.bfloat16)
    bt = torch.zeros(len(ctxs), max(need), dtype=torch.int32)
    at = 0
    for b, n in enumerate(need):
        bt[b, :n] = torch.tensor(perm[at:at + n])
        at += n

    def put(c, b, rows):
        for i in range(0, rows.shape[0], 64):
            c[int(bt[b, i // 64]), :min(64, rows.shape[0] - i)] = rows[i:i + 64]
    return cache, bt, put


def _want(q, k, v, pos, scale, window, keep, chunk, cap, sink, gate, slopes, table):
    """(result, sum of weights times |values|): q [n, H, d], k [m, G, d], v [m, Gv, e], pos [n]; 64 bits."""
    n, H, _ = q.shape
    m, G, Gv = k.shape[0], k.shape[1], v.shape[1]
    i, j = pos[:, None], torch.arange(m)[None]
    lo = (i - window + 1 if window else torch.zeros_like(i)).clamp(min=0)
    if chunk:
        lo = torch.maximum(lo, i // chunk * chunk)
    ok = (j <= i) & ((j >= lo) | (j < keep))
    out, mag = torch.zeros(n, H, v.shape[2], dtype=D64), torch.zeros(n, H, v.shape[2], dtype=D64)
    for h in range(H):
        g = h // (H // G)
        s = q[:, h] @ k[:, g].T * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if slopes is not None:
            s = s - slopes[h] * (i - j)
        if table is not None:
            s = s + table[h][(i - j).clamp(0, table.shape[1] - 1)]
        s = s.masked_fill(~ok, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(n, 1)], 1)
        w = torch.softmax(s, 1)[:, :m]
        out[:, h], mag[:, h] = w @ v[:, g % Gv], w @ v[:, g % Gv].abs()
    gt = torch.sigmoid(gate) if gate is not None else torch.ones(n, H, dtype=D64)
    gt = gt.reshape(n, H, -1)
    return out * gt, mag * gt


def _check(out, want, mag):
    # weights are rounded to bf16 once (unit roundoff 2^-8 for its 8 significant bits) and the result once more; the fp32 sums
    # and exponentials of scores up to ~50 add a few 1e-6 of the same sum
    err = (out.double().cpu() - want).abs()
    assert torch.isfinite(out).all()
    assert bool((err <= mag * (2.0 ** -7) * 1.02 + 1e-6).all()), (err / mag.clamp(min=1e-9)).max().item()


def _check32(out, want, mag):
    # everything but the cache rows is fp32: sums of up to 320 products and of some hundred weights, and the rounding of the result
    err = (out.double().cpu() - want).abs()
    assert bool((err <= mag * 2e-5 + want.abs() * (2.0 ** -8 if out.dtype == torch.bfloat16 else 0) + 1e-6).all()), err.max().item()


LENS = [([1], [1]), ([1, 1, 1], [64, 129, 700]), ([5, 1, 70], [5, 65, 333]), ([130, 257], [130, 300])]


@pytest.mark.parametrize("lens,ctxs", LENS)
@pytest.mark.parametrize("H,G,Gv,dk,dv,opt", [
    (16, 4, 4, 128, 128, dict(window=100, keep=3, cap=9.0, sink=True, gate="head")),
    (16, 4, 4, 128, 128, dict()),
    (6, 2, 2, 96, 64, dict(window=64, sink=True, f32=True)),
    (8, 1, 1, 64, 192, dict(window=1, gate="elem")),
    (5, 5, 5, 256, 256, dict(chunk=96, slopes=True)),
    (8, 4, 2, 64, 64, dict(chunk=50, table=40, f32=True)),
    (40, 1, 1, 160, 320, dict(window=333, keep=70, table=90, cap=20.0)),
])
def test_grouped_heads(lib, H, G, Gv, dk, dv, opt, lens, ctxs):
    from vllm_rs_b200 import ops
    g = torch.Generator().manual_seed(H * dk + sum(ctxs))
    kc, bt, put = _pages(g, ctxs, (G, dk))
    vc = torch.full((kc.shape[0], 64, Gv, dv), float("nan"), dtype=torch.bfloat16)
    T = sum(lens)
    q = torch.randn(T, H, dk, generator=g) * 1.5
    q = q if opt.get("q32") else q.bfloat16()
    f = lambda name, *shape: torch.randn(*shape, generator=g) if opt.get(name) else None      # noqa: E731
    sink, slopes = f("sink", H), f("slopes", H)
    slopes = slopes.abs() * 0.02 if slopes is not None else None
    if "low" in opt:
        sink[::2] = opt["low"]
    table = torch.randn(H, opt["table"], generator=g) if opt.get("table") else None
    gate = {"head": torch.randn(T, H, generator=g), "elem": torch.randn(T, H * dv, generator=g)}.get(opt.get("gate"))
    scale, window, keep, chunk, cap = dk ** -0.5, opt.get("window", 0), opt.get("keep", 0), opt.get("chunk", 0), opt.get("cap", 0.0)
    d = lambda t: None if t is None else t.double()                                           # noqa: E731
    want, mag, at = [], [], 0
    for b, (n, c) in enumerate(zip(lens, ctxs)):
        k, v = torch.randn(c, G, dk, generator=g).bfloat16(), torch.randn(c, Gv, dv, generator=g).bfloat16()
        put(kc, b, k)
        put(vc, b, v)
        w, m = _want(q[at:at + n].double(), k.double(), v.double(), torch.arange(c - n, c), scale, window, keep, chunk, cap,
                     d(sink), None if gate is None else gate[at:at + n].double(), d(slopes), d(table))
        want.append(w)
        mag.append(m)
        at += n
    cu = _i32([0] + [sum(lens[:i + 1]) for i in range(len(lens))])
    c_ = lambda t: None if t is None else t.cuda().contiguous()                               # noqa: E731
    for split in (True, False):
        out = ops.window_attn(q.float().cuda(), kc.cuda(), vc.cuda(), c_(sink), c_(gate), cu, _i32(ctxs), bt.cuda(), window=window,
                              keep_first=keep, scale=scale, softcap=cap, split=split, dist_slopes=c_(slopes), chunk=chunk,
                              out_f32=opt.get("f32", False), dist_bias=c_(table))
        (_check32 if opt.get("q32") else _check)(out, torch.cat(want), torch.cat(mag))


@pytest.mark.parametrize("lens,ctxs", LENS + [([420], [420])])
@pytest.mark.parametrize("H,rank,rot,window", [(16, 256, 32, 100), (32, 512, 32, 0), (24, 512, 64, 129), (20, 320, 32, 64),
                                               (3, 64, 0, 1), (128, 128, 32, 77), (9, 448, 32, 0)])
def test_latent_rows(lib, H, rank, rot, window, lens, ctxs, low=None, q32=False):
    from vllm_rs_b200 import ops
    g = torch.Generator().manual_seed(H * rank + sum(ctxs))
    R, T = rank + rot, sum(lens)
    cache, bt, put = _pages(g, ctxs, (R,))
    q = torch.randn(T, H, R, generator=g) * 0.7
    q = q if q32 else q.bfloat16()
    sink, gate = torch.randn(H, generator=g), torch.randn(T, H, generator=g)
    if low is not None:
        sink[::2] = low
    want, mag, at = [], [], 0
    for b, (n, c) in enumerate(zip(lens, ctxs)):
        k = torch.randn(c, R, generator=g).bfloat16()
        put(cache, b, k)
        k = k.double()[:, None]
        w, m = _want(q[at:at + n].double(), k, k[..., :rank], torch.arange(c - n, c), 0.1, window, 0, 0, 0.0, sink.double(),
                     gate[at:at + n].double(), None, None)
        want.append(w)
        mag.append(m)
        at += n
    cu = _i32([0] + [sum(lens[:i + 1]) for i in range(len(lens))])
    for split in (True, False):
        out = ops.latent_attn(q.float().cuda(), cache.cuda(), sink.cuda(), cu, _i32(ctxs), bt.cuda(), kv_rank=rank, rot_dim=rot,
                              window=window, scale=0.1, split=split, gate=gate.cuda())
        (_check32 if q32 else _check)(out, torch.cat(want), torch.cat(mag))


@pytest.mark.parametrize("low", [-math.inf, torch.finfo(torch.float32).min])
@pytest.mark.parametrize("lens,ctxs", [([1, 1], [64, 700]), ([70], [333]), ([130, 257], [130, 300])])
def test_sinks_below_all_scores(lib, low, lens, ctxs):
    """A sink that weighs nothing: heads that have it are heads without one, also where a row's first page holds no key that
    it sees (windows and chunks that start inside a page, for the later tokens of a tile)."""
    for opt in (dict(window=100), dict(window=65, keep=3, cap=9.0, gate="head"), dict(chunk=96, slopes=True)):
        test_grouped_heads(lib, 16, 4, 4, 128, 128, dict(opt, sink=True, low=low), lens, ctxs)
    test_latent_rows(lib, 8, 256, 32, 100, lens, ctxs, low)


@pytest.mark.parametrize("lens,ctxs", [([1, 1], [64, 700]), ([70], [333]), ([130, 257], [130, 300])])
def test_sizes_without_a_tensor_core_form(lib, lens, ctxs):
    """Values wider than 256, ranks past 512 and, at few rows, more score maps over one set of values than fit in shared memory:
    queries and weights stay in fp32."""
    test_grouped_heads(lib, 6, 2, 2, 128, 320, dict(window=100, sink=True, f32=True, q32=True), lens, ctxs)
    test_grouped_heads(lib, 4, 4, 4, 64, 384, dict(cap=9.0, gate="head", f32=True, q32=True), lens, ctxs)
    if sum(lens) <= 74:
        test_grouped_heads(lib, 12, 12, 1, 128, 64, dict(f32=True, q32=True), lens, ctxs)
    test_latent_rows(lib, 5, 576, 32, 100, lens, ctxs, q32=True)


@pytest.mark.parametrize("n", [1, 5])
def test_largest_weight_of_a_page_is_exact(lib, n):
    """Steps of few rows: one key per page counts, and each page's weight lies half way between two bf16 numbers relative to the
    first page's.  Relative to its own page it is one, so that nothing but fp32 sums is left (no split: one reference per row)."""
    from vllm_rs_b200 import ops
    pages, dk, dv = 6, 64, 64
    k = torch.zeros(pages * 64, 1, dk)
    k[:, 0, 0] = -30.0                                                        # weight 2^-43 at most
    step = math.log(2 ** -1 * (1 + 3 * 2.0 ** -9))                            # 3 x 2^-9: bf16 rounds the weight by 2^-9
    q = torch.zeros(n, 1, dk)
    q[:, 0, 0], q[:, 0, 1] = 1.0, step
    for p in range(pages):
        k[p * 64, 0, 0], k[p * 64, 0, 1] = 0.0, 1.0 if p else 0.0
    q = q.bfloat16().float()
    scale = step / q[0, 0, 1].item()                                          # the second entry's product is `step` again
    g = torch.Generator().manual_seed(3)
    v = torch.randn(pages * 64, 1, dv, generator=g).bfloat16()
    want, mag = _want(q.double(), k.double(), v.double(), torch.arange(pages * 64 - n, pages * 64), scale, 0, 0, 0, 0.0, None, None,
                      None, None)
    out = ops.window_attn(q.cuda(), k.bfloat16().cuda().reshape(pages, 64, 1, dk), v.cuda().reshape(pages, 64, 1, dv), None, None,
                          _i32([0, n]), _i32([pages * 64]), _i32([list(range(pages))]), window=0, keep_first=0, scale=scale,
                          split=False, out_f32=True)
    assert bool(((out.double().cpu() - want).abs() <= 2e-5 * mag).all())


@pytest.mark.parametrize("n", [1, 90])
def test_capped_scores_in_other_company(lib, n):
    """A head's bits do not depend on the scores of the heads and tokens beside it (small arguments of tanh take another form)."""
    from vllm_rs_b200 import ops
    ctx, H, G, d = 200, 8, 2, 64
    g = torch.Generator().manual_seed(n)
    k, v = (torch.randn(4, 64, G, d, generator=g).bfloat16().cuda() for _ in range(2))
    q = torch.randn(n, H, d, generator=g).cuda()
    other = q.clone()
    other[:, 1] *= 40.0
    other[1:, 5] *= 40.0
    args = (None, None, _i32([0, n]), _i32([ctx]), _i32([[2, 0, 3, 1]]))
    a, b = (ops.window_attn(x, k, v, *args, window=0, keep_first=0, scale=0.3, softcap=9.0, out_f32=True) for x in (q, other))
    same = torch.ones(n, H, dtype=torch.bool)
    same[:, 1] = same[1:, 5] = False
    assert torch.equal(a[same.cuda()], b[same.cuda()])
    _check(a, *_want(q.bfloat16().double().cpu(), *(t[[2, 0, 3, 1]].reshape(256, G, d)[:ctx].double().cpu() for t in (k, v)),
                     torch.arange(ctx - n, ctx), 0.3, 0, 0, 0, 9.0, None, None, None, None))
    assert not torch.equal(a[:, 1], b[:, 1])


@pytest.mark.parametrize("bad", [math.nan, math.inf])
@pytest.mark.parametrize("H,G,tile", [(16, 4, 32), (8, 8, 128), (32, 1, 4)])
def test_later_tokens_of_a_page_stay_out(lib, H, G, tile, bad):
    """A key and a value that are not finite leave the tiles before their token alone, also where tiles end inside a page."""
    from vllm_rs_b200 import ops
    n, d, past = 300, 64, 20
    g = torch.Generator().manual_seed(tile)
    pages = -(-(n + past) // 64)
    k, v = (torch.randn(pages * 64, G, d, generator=g).bfloat16().cuda() for _ in range(2))
    q = torch.randn(n, H, d, generator=g).cuda()
    args = (None, None, _i32([0, n]), _i32([n + past]), _i32([list(range(pages))]))
    run = lambda: ops.window_attn(q, *(t.reshape(pages, 64, G, d) for t in (k, v)), *args, window=0, keep_first=0, scale=0.2)  # noqa: E731
    want = run()
    for t in (tile, 2 * tile + 1, n - 1):
        kept = k[past + t].clone(), v[past + t].clone()
        k[past + t], v[past + t] = bad, bad
        got = run()
        clean = t // tile * tile
        assert torch.equal(got[:clean], want[:clean]) and not torch.isfinite(got[t]).all()
        k[past + t], v[past + t] = kept


@pytest.mark.parametrize("H,rank,rot,window,lens,ctxs", [
    (128, 320, 32, 0, [170, 130], [170, 199]), (128, 512, 0, 70, [160, 150], [222, 150]), (64, 448, 64, 100, [300, 311], [300, 340])])
def test_passes_of_one_block(lib, H, rank, rot, window, lens, ctxs):
    """Two passes over the value columns in one block, equal and unequal: enough tiles (128 / heads tokens each) for two per SM."""
    assert sum(-(-n // (128 // H)) for n in lens) + 1 > 2 * 148
    test_latent_rows(lib, H, rank, rot, window, lens, ctxs)


def test_several_maps_over_one_set_of_values_at_decode(lib):
    """Key head g reads value head g % v_heads: maps that share the values, in the tensor-core form's sizes."""
    for H, G, Gv in ((8, 4, 2), (12, 6, 1), (16, 8, 4)):
        test_grouped_heads(lib, H, G, Gv, 64, 128, dict(window=90, sink=True), [1, 1, 1], [64, 129, 700])


@pytest.mark.parametrize("lens,ctxs", [([1], [256]), ([1], [257]), ([1] * 20, [300] * 20), ([3, 1], [64, 1100])])
def test_parts_of_a_few_pages(lib, lens, ctxs):
    """Key splits of one and two pages per part, an odd page left over, and contexts shorter than the longest (empty parts)."""
    test_grouped_heads(lib, 16, 4, 4, 64, 64, dict(sink=True, gate="head"), lens, ctxs)
    test_grouped_heads(lib, 6, 2, 2, 96, 64, dict(window=200, keep=70, f32=True), lens, ctxs)
    test_latent_rows(lib, 4, 64, 32, 0, lens, ctxs)
