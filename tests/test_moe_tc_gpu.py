"""The grouped products of routed experts, on tcgen05 and (short rows) on mma.sync, against 64-bit experts: buckets that are empty, hold one row, end inside a tile
or take several; features and inner sizes that end inside a tile; every activation; identity experts; all three tile widths of
both products (on 148 SMs 256 columns where that makes 296 tiles, 128 where it makes 111, else 64)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("act", ["silu_gate", "relu2", "clamped"])
@pytest.mark.parametrize("T,E,top,D,F,skew", [
    (1, 4, 2, 64, 32, 0), (37, 5, 3, 72, 40, 0), (3, 64, 1, 512, 8, 0), (300, 3, 2, 136, 264, 0), (700, 16, 4, 64, 520, 3),
    (513, 2, 1, 264, 1032, 0), (2100, 20, 2, 96, 4100 // 8 * 8, 0), (129, 1, 1, 8, 16, 0),
    (350, 16, 2, 2056, 40, 0),             # second product: 16 row tiles x 17 of 128 columns, the last one 8 wide
    (600, 20, 4, 4104, 72, 0),             # 20 x 17 of 256 columns, the last one 8 wide
    (300, 16, 2, 72, 1032, 0),             # 16 x 9 of 128 columns without a gate
    # rows long enough for tcgen05 in both products, whatever their number
    (1, 4, 2, 776, 264, 0), (37, 5, 3, 776, 264, 0), (3, 64, 1, 1032, 256, 0), (700, 16, 4, 776, 520, 3), (513, 2, 1, 840, 1032, 0),
    (300, 16, 2, 776, 1032, 0), (2100, 20, 2, 776, 296, 0)])
def test_experts(lib, act, T, E, top, D, F, skew):
    from vllm_rs_b200 import ops
    g = torch.Generator().manual_seed(T * E + F)
    bf, dev = torch.bfloat16, "cuda"
    ident = 2 if T == 37 else 0
    h = torch.randn(T, D, generator=g).to(bf)
    wu = (torch.randn(E, F if act == "relu2" else 2 * F, D, generator=g) / D ** 0.5).to(bf)
    wd = (torch.randn(E, D, F, generator=g) / F ** 0.5).to(bf)
    z = torch.randn(T, E + ident, generator=g) - skew * torch.arange(E + ident).float()       # skew leaves buckets empty
    w, idx = torch.softmax(z, 1).topk(top, 1)
    x = torch.randn(T, D, generator=g)
    limit, alpha, add = 1.5, 1.702, 1.0
    want, tol = x.double().to(dev), torch.zeros(T, D, dtype=torch.float64, device=dev)
    H, u24 = h.double().to(dev), 2.0 ** -24
    for e in range(E):
        t, j = (idx == e).nonzero(as_tuple=True)
        if not len(t):
            continue
        t, wt = t.to(dev), w[t, j].double().to(dev)[:, None]
        a, b, m = H[t], wu[e].double().to(dev), wd[e].double().to(dev)
        y, dy = a @ b.T, D * u24 * (a.abs() @ b.abs().T)          # a product and what its fp32 sum may be off by
        if act == "relu2":
            r = torch.relu(y)
            y, dy = r * r, 2 * r * dy + dy * dy
        else:
            gt, up, dg, du = *y.chunk(2, 1), *dy.chunk(2, 1)
            if act == "clamped":
                gt, up = gt.clamp(max=limit), up.clamp(-limit, limit)
                s = gt * torch.sigmoid(alpha * gt)
                y, dy = s * (up + add), 1.2 * (up + add).abs() * dg + s.abs() * du
            else:
                s = torch.nn.functional.silu(gt)
                y, dy = s * up, 1.2 * up.abs() * dg + s.abs() * du          # |d silu| < 1.1
        want.index_add_(0, t, wt * (y @ m.T))
        # the activation is rounded to bf16 (2^-8 of itself), the second product sums F terms in fp32
        tol.index_add_(0, t, wt * (((2.0 ** -8 + F * u24) * y.abs() + dy) @ m.abs().T))
    for e in range(E, E + ident):
        t, j = (idx == e).nonzero(as_tuple=True)
        want.index_add_(0, t.to(dev), w[t, j].double().to(dev)[:, None] * H[t.to(dev)])
    kw = dict(limit=limit, alpha=alpha, up_add=add) if act == "clamped" else {}
    c = lambda v: v.to(dev).contiguous()                                     # noqa: E731
    out = ops.moe_experts_ex(c(x), c(h), c(idx.int()), c(w), c(wu), c(wd), act=act, identity=ident, **kw)
    err = (out.double() - want).abs()
    assert bool((err <= 1.02 * tol + 1e-5 * want.abs().clamp(min=1.0)).all()), (err - tol).max().item()


@pytest.mark.parametrize("act", ["silu_gate", "relu2"])
@pytest.mark.parametrize("E,D,F", [(8, 512, 128), (4, 256, 256), (8, 128, 1024)])
def test_same_bits_in_steps_of_any_size(lib, act, E, D, F):
    """Steps of few rows take mma.sync for these sizes and steps of many tcgen05: a row's result does not tell which."""
    from vllm_rs_b200 import ops
    g = torch.Generator().manual_seed(D)
    c = lambda t: t.cuda().contiguous()                                      # noqa: E731
    wu = c((torch.randn(E, F if act == "relu2" else 2 * F, D, generator=g) / D ** 0.5).bfloat16())
    wd = c((torch.randn(E, D, F, generator=g) / F ** 0.5).bfloat16())
    T = 6000
    h, z, x = c(torch.randn(T, D, generator=g).bfloat16()), torch.randn(T, E, generator=g), torch.zeros(T, D).cuda()
    w, idx = torch.softmax(z, 1).topk(2, 1)
    w, idx = c(w), c(idx.int())
    run = lambda n: ops.moe_experts_ex(x[:n].clone(), h[:n], idx[:n], w[:n], wu, wd, act=act)      # noqa: E731
    few, many = run(70), run(T)
    assert torch.equal(few, many[:70])


@pytest.mark.parametrize("T,E,top", [(4096, 33, 4), (4097, 33, 4), (13000, 70, 3)])
def test_buckets_of_many_pairs(lib, T, E, top):
    """The sort keeps up to 16 384 pairs in registers and walks more of them in several rounds: every row of a large step has the
    bits that it has in a portion of 1000 rows, as sums are taken in the order of a token's choices."""
    from vllm_rs_b200 import ops
    g = torch.Generator().manual_seed(T)
    c = lambda t: t.cuda().contiguous()                                      # noqa: E731
    D, F = 64, 32
    wu, wd = c(torch.randn(E, 2 * F, D, generator=g).bfloat16()), c(torch.randn(E, D, F, generator=g).bfloat16())
    h, z, x = c(torch.randn(T, D, generator=g).bfloat16()), torch.randn(T, E, generator=g), torch.zeros(T, D).cuda()
    w, idx = torch.softmax(z, 1).topk(top, 1)
    w, idx = c(w), c(idx.int())
    run = lambda a, b: ops.moe_experts_ex(x[a:b].clone(), h[a:b], idx[a:b], w[a:b], wu, wd, act="silu_gate")      # noqa: E731
    whole = run(0, T)
    assert torch.equal(whole, torch.cat([run(a, min(a + 1000, T)) for a in range(0, T, 1000)]))
    assert whole.abs().sum() > 0


@pytest.mark.parametrize("act", ["silu_gate", "relu2", "clamped"])
@pytest.mark.parametrize("T,E,skew", [(6000, 3, 0), (5003, 4, 2), (9000, 2, 9)])
def test_pairs_of_blocks(lib, act, T, E, skew):
    """Tiles of 256 slots, which two blocks share: buckets that end in either block's half, hold few rows or none, features that end
    inside a tile.  Every row has the bits that it has in portions of 500 rows, whose tiles are a block's own."""
    from vllm_rs_b200 import ops
    g = torch.Generator().manual_seed(T)
    c = lambda t: t.cuda().contiguous()                                      # noqa: E731
    D, F = 776, 520
    wu = c((torch.randn(E, F if act == "relu2" else 2 * F, D, generator=g) / D ** 0.5).bfloat16())
    wd = c((torch.randn(E, D, F, generator=g) / F ** 0.5).bfloat16())
    h, x = c(torch.randn(T, D, generator=g).bfloat16()), torch.zeros(T, D).cuda()
    z = torch.randn(T, E, generator=g) - skew * torch.arange(E).float()
    w, idx = torch.softmax(z, 1).topk(2 if skew < 9 else 1, 1)
    w, idx = c(w), c(idx.int())
    kw = dict(limit=1.5, alpha=1.702, up_add=1.0) if act == "clamped" else {}
    run = lambda a, b: ops.moe_experts_ex(x[a:b].clone(), h[a:b], idx[a:b], w[a:b], wu, wd, act=act, **kw)      # noqa: E731
    whole = run(0, T)
    assert torch.equal(whole, torch.cat([run(a, min(a + 500, T)) for a in range(0, T, 500)])) and float(whole.abs().sum()) > 0
