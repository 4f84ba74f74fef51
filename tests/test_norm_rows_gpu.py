"""Row norms with 16-byte accesses against 64 bits: widths at the edges of one, two and four vectors per thread and past them
(entry by entry), widths that are no multiple of four, groups a warp and a block wide, gates before and after."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _close(got, want, dtype):
    # the result is rounded once; the sum of squares is an fp32 sum, relative error well below 1e-5 at these widths
    tol = (2.0 ** -8 if dtype == torch.bfloat16 else 1e-5) * want.abs() + 1e-6
    assert bool(((got.double().cpu() - want).abs() <= tol).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n", [1, 4, 6, 1020, 1024, 1028, 2048, 2052, 4096, 4100])
def test_row_norms(lib, n, dtype):
    from vllm_rs_b200 import ops
    g = torch.Generator().manual_seed(n)
    x, y, w = torch.randn(5, n, generator=g) * 3, torch.randn(5, n, generator=g), torch.randn(n, generator=g)
    unit = lambda t: t / torch.sqrt((t * t).mean(-1, keepdim=True) + 1e-6)          # noqa: E731
    c = lambda t: t.cuda().contiguous()                                             # noqa: E731
    _close(ops.resid_rmsnorm(c(x), c(w), 1e-6, 1.0, dtype), unit(x.double()) * (1.0 + w.double()), dtype)
    s = c(x)
    ops.resid_add_rmsnorm(s, c(y), c(w), 1e-6, 0.5)
    want = x.double() + unit(y.double()) * (0.5 + w.double())
    assert (s.double().cpu() - want).abs().max() <= 1e-5 * want.abs().max()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("gate_first,act", [(True, "silu"), (False, "sigmoid")])
@pytest.mark.parametrize("C,group,wn", [(24, 8, 8), (30, 6, 30), (256, 128, 128), (1024, 512, 1024), (2048, 2048, 2048),
                                        (4160, 1040, 0), (8192, 8192, 8192)])
def test_gated_group_norm(lib, C, group, wn, gate_first, act, dtype, T=7):
    from vllm_rs_b200 import ops
    g = torch.Generator().manual_seed(C + group)
    y, gate = torch.randn(T, C, generator=g), torch.randn(T, C, generator=g) * 2
    w = torch.randn(wn, generator=g) if wn else None
    G, Y = gate.double(), y.double()
    s = torch.sigmoid(G) * (G if act == "silu" else 1.0)
    u = (Y * s if gate_first else Y).reshape(T, -1, group)
    want = (u / torch.sqrt((u * u).mean(-1, keepdim=True) + 1e-6)).reshape(T, C)
    if w is not None:
        want = want * w.double().repeat(C // wn)
    want = want if gate_first else want * s
    got = ops.gated_group_norm(y.cuda(), gate.cuda(), None if w is None else w.cuda(), group, 1e-6, gate_first, dtype, act)
    _close(got, want, dtype)


@pytest.mark.parametrize("C,group", [(1024, 256), (2048, 512), (1040, 260), (768, 192), (768, 384)])
def test_gated_group_norm_of_few_and_many_groups(lib, C, group):
    """Rows on both sides of the line between several warps per group and one, a last block that is not full; and the same bits."""
    from vllm_rs_b200 import ops
    many = 3 * torch.cuda.get_device_properties(0).multi_processor_count * group // 128
    for T in (-(-many // (C // group)) - 1, -(-many // (C // group)) + 1):
        test_gated_group_norm(lib, C, group, C, True, "silu", torch.float32, T)
        test_gated_group_norm(lib, C, group, group, False, "sigmoid", torch.bfloat16, T)
    y, gate, w = (torch.randn(n, C, device="cuda") for n in (many, many, 1))
    for first in (True, False):
        run = lambda n: ops.gated_group_norm(y[:n], gate[:n], w[0], group, 1e-6, first, torch.float32, "silu")      # noqa: E731
        assert torch.equal(run(many)[:5], run(5))
