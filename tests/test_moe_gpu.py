"""MoE dispatch / grouped tcgen05 GEMM / combine on the GPU against the CPU reference paths."""
import pytest
import torch

from flex_shard_b200 import ops
from flex_shard_b200.ops import moe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,k,E,D,F", [(300, 2, 4, 256, 384), (2048, 6, 64, 512, 256), (64, 1, 8, 128, 128)])
def test_moe_layer_matches_cpu_reference(T, k, E, D, F):
    torch.manual_seed(0)
    idx = torch.stack([torch.randperm(E)[:k] for _ in range(T)])
    x = torch.randn(T, D).bfloat16()
    w1 = (0.1 * torch.randn(E, F, D)).bfloat16()
    gw = torch.rand(T, k)
    res = {}
    for dev in ("cpu", "cuda"):
        xi = x.clone().to(dev).requires_grad_()
        wi = w1.clone().to(dev).requires_grad_()
        gi = gw.clone().to(dev).requires_grad_()
        plan = moe.plan_routes(idx.to(dev), E)
        y = moe.moe_combine(moe.grouped_linear(moe.moe_dispatch(xi, plan), wi, plan), gi, plan)
        y.float().square().sum().backward()
        res[dev] = [t.detach().float().cpu() for t in (y, xi.grad, wi.grad, gi.grad)]
    ops.check_status()
    names = ["y", "dx", "dw", "dgate"]
    for n, a, b in zip(names, res["cpu"], res["cuda"]):
        scale = max(a.abs().max().item(), 1e-3)
        assert (a - b).abs().max().item() < 4e-2 * scale, (n, (a - b).abs().max().item(), scale)


@pytest.mark.parametrize("mode,normalize,E,k", [("sigmoid", True, 256, 8), ("softmax", True, 8, 2),
                                                ("softmax", False, 64, 6), ("sigmoid", True, 40, 3)])
def test_router_kernel_matches_reference(mode, normalize, E, k):
    torch.manual_seed(3)
    T = 1000
    logits = torch.randn(T, E) * 2
    bias = torch.randn(E) * 0.1 if mode == "sigmoid" else None
    res = {}
    for dev in ("cpu", "cuda"):
        lg = logits.clone().to(dev).requires_grad_()
        counts = torch.zeros(E, device=dev)
        idx, w = moe.route_topk(lg, k, bias=None if bias is None else bias.to(dev), mode=mode, scale=2.5,
                                normalize=normalize, counts=counts)
        (w * torch.arange(1, k + 1, device=dev)).sum().backward()
        res[dev] = (idx.cpu(), w.detach().cpu(), counts.cpu(), lg.grad.cpu())
    assert torch.equal(res["cpu"][0], res["cuda"][0])
    torch.testing.assert_close(res["cpu"][1], res["cuda"][1], rtol=1e-4, atol=1e-6)
    assert torch.equal(res["cpu"][2], res["cuda"][2])
    torch.testing.assert_close(res["cpu"][3], res["cuda"][3], rtol=1e-4, atol=1e-6)


@pytest.mark.parametrize("T,k,E", [(300, 2, 4), (4096, 6, 64), (7, 1, 8), (50000, 1, 16), (1000, 8, 256), (33, 3, 5)])
def test_route_plan_kernel_equals_operator_plan(T, k, E):
    """Histogram, padded offsets, tile table and stable rows from the one-launch kernel equal the plan
    computed with sort / bincount / cumsum operators, exactly; skewed and empty experts included."""
    g = torch.Generator().manual_seed(T + E)
    idx = torch.randint(0, E, (T, k), generator=g)
    idx[idx == E - 1] = 0                      # the last expert stays empty, the first is overloaded
    for dtype in (torch.int64, torch.int32):
        before = ops.launch_count()
        got = moe.plan_routes(idx.to("cuda", dtype), E)
        assert ops.launch_count() - before == 1
        want = moe.plan_routes(idx, E)         # CPU tensors take the operator path
        torch.cuda.synchronize()
        assert torch.equal(got.pos.cpu(), want.pos)
        assert torch.equal(got.src.cpu(), want.src)
        assert torch.equal(got.offs.cpu(), want.offs)
        assert int(got.num_mtiles) == int(want.num_mtiles)
        n_tiles = int(want.num_mtiles)
        assert torch.equal(got.tile_expert.cpu()[:n_tiles], want.tile_expert[:n_tiles])
        assert got.max_rows == want.max_rows
    ops.check_status()


@pytest.mark.parametrize("B,S,H,nope,rope,value", [(1, 1, 1, 8, 8, 8), (2, 37, 3, 64, 32, 64), (1, 200, 16, 128, 64, 128),
                                                   (3, 5, 5, 24, 16, 40)])
def test_latent_attention_operands_match_the_torch_steps(B, S, H, nope, rope, value):
    from flex_shard_b200.ops import elementwise as ew
    from flex_shard_b200.ops import mla

    torch.manual_seed(8)
    dev = torch.device("cuda")
    table = ew.rope_table(S + 3, rope, 10000.0, dev)[:S]
    q = torch.randn(B, S, H, nope + rope, device=dev).bfloat16()
    kvb = torch.randn(B, S, H, nope + value, device=dev).bfloat16()
    kv = torch.randn(B, S, 16 + rope, device=dev).bfloat16()
    grads = [torch.randn(B, S, H, n, device=dev).bfloat16() for n in (nope + rope, nope + rope, value)]
    grads[0] = grads[0].transpose(1, 2).contiguous().transpose(1, 2)     # another memory order than the outputs'
    assert mla._native(q, kvb, kv[..., 16:], table, nope)
    res = []
    for fn, cast in ((mla.mla_operands, lambda t: t), (mla.mla_operands_ref, torch.Tensor.double)):
        leaves = [cast(t).clone().requires_grad_() for t in (q, kvb, kv)]
        outs = fn(leaves[0], leaves[1], leaves[2][..., 16:], table, nope)
        torch.autograd.backward(outs, [cast(g) for g in grads])
        res.append([t.detach().double() for t in (*outs, *(x.grad for x in leaves))])
    for got, ref in zip(*res):
        # the reference rotates in fp32 (2^-22 of |x| + |y| < 2^3 H) on double inputs; one rounding to bf16 on top
        assert ((got - ref).abs() <= ref.abs() * 2.0 ** -8 + H * 2.0 ** -18).all()
    ops.check_status()


def test_latent_attention_operands_under_the_transforms_of_autograd():
    """Batched gradients, second derivatives and forward mode of what is a linear map of its inputs, against the torch
    steps; the kernel's sum over heads is rounded once, theirs between heads."""
    import torch.autograd.forward_ad as fwd

    from flex_shard_b200.ops import elementwise as ew
    from flex_shard_b200.ops import mla

    torch.manual_seed(8)
    dev = torch.device("cuda")
    B, S, H, nope, rope, value = 2, 5, 3, 16, 8, 24
    table = ew.rope_table(S, rope, 10000.0, dev)
    shapes = [(B, S, H, nope + rope), (B, S, H, nope + value), (B, S, rope)]
    rand = lambda *s: torch.randn(*s, device=dev).bfloat16()   # noqa: E731
    xs, vs = [rand(*s).requires_grad_() for s in shapes], [rand(*s) for s in shapes]
    dys = [rand(4, B, S, H, n) for n in (nope + rope, nope + rope, value)]
    assert mla._native(*xs, table, nope)
    close = lambda a, b: torch.testing.assert_close(a.float(), b.float(), rtol=2.0 ** -6, atol=H * 2.0 ** -6)   # noqa: E731
    res = []
    for fn in (mla.mla_operands, mla.mla_operands_ref):
        outs = fn(*xs, table, nope)
        batched = torch.autograd.grad(outs, xs, dys, is_grads_batched=True, retain_graph=True)
        first = [d[0].clone().requires_grad_() for d in dys]
        grads = torch.autograd.grad(outs, xs, first, create_graph=True)
        second = torch.autograd.grad(grads, first, vs)
        with fwd.dual_level():
            ts = [fwd.unpack_dual(o).tangent for o in fn(*(fwd.make_dual(x.detach(), v) for x, v in zip(xs, vs)), table, nope)]
        res.append([*batched, *grads, *second, *ts])
    for a, b in zip(*res):
        close(a, b)
    ops.check_status()


@pytest.mark.parametrize("counts,D,F,dtype", [([0, 700, 1, 0, 513, 256, 1200, 0], 512, 320, torch.bfloat16),
                                              ([385, 130, 900, 0], 264, 640, torch.float32), ([3000], 256, 256, torch.bfloat16)])
def test_grouped_products_on_sm_pairs(counts, D, F, dtype):
    """Groups of an odd number of 128-row tiles, empty groups at both ends, widths that no tile divides; each product
    against fp64 on the same bf16 operands (fp32 sums of at most 1280 terms, one rounding)."""
    torch.manual_seed(4)
    dev = torch.device("cuda")
    E = len(counts)
    idx = torch.cat([torch.full((c,), e) for e, c in enumerate(counts)])[torch.randperm(sum(counts))].view(-1, 1).to(dev)
    plan = moe.plan_routes(idx, E)
    x = moe.moe_dispatch(torch.randn(idx.shape[0], D, device=dev).bfloat16(), plan).requires_grad_()
    w = torch.randn(E, F, D, device=dev).bfloat16().requires_grad_()
    if dtype == torch.float32:
        w.main_grad, w.main_grad_written = torch.zeros(E, F, D, device=dev), False
    y = moe.grouped_linear(x, w, plan)
    offs = plan.offs.tolist()
    dy = torch.zeros_like(y)
    dy[:offs[-1]] = torch.randn(offs[-1], F, device=dev).bfloat16()
    y.backward(dy)
    ops.check_status()
    dw = w.main_grad if dtype == torch.float32 else w.grad
    for e in range(E):
        r = slice(offs[e], offs[e + 1])
        xe, we, de = x.detach()[r].double(), w.detach()[e].double(), dy[r].double()
        pairs = [(dw[e], de.t() @ xe, de.abs().t() @ xe.abs())]
        pairs += [(y[r], xe @ we.t(), xe.abs() @ we.abs().t()), (x.grad[r], de @ we, de.abs() @ we.abs())]
        for got, ref, mag in pairs:
            bound = mag * (1280 * 2.0 ** -24) + ref.abs() * (2.0 ** -8 if got.dtype == torch.bfloat16 else 0)
            assert ((got.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("counts,D,F,dtype", [([1500, 0, 130, 2400, 901], 1032, 1248, torch.bfloat16),
                                              ([640] * 4, 1024, 1024, torch.bfloat16), ([639] * 4, 1024, 1024, torch.bfloat16),
                                              ([3000, 129, 1700], 264, 1248, torch.float32)])
@pytest.mark.parametrize("pairs", [1, 0])
def test_grouped_products_either_way(counts, D, F, dtype, pairs):
    """Sizes at which the rule takes SM pairs (and just does not), on pairs and with pairs switched off: groups that end
    in half a pair tile, an empty one, ragged widths; fp32 destinations written anew. Sums of n products in fp32."""
    from flex_shard_b200.ops import _lib

    torch.manual_seed(4)
    dev = torch.device("cuda")
    E = len(counts)
    idx = torch.cat([torch.full((c,), e) for e, c in enumerate(counts)])[torch.randperm(sum(counts))].view(-1, 1).to(dev)
    plan = moe.plan_routes(idx, E)
    x = moe.moe_dispatch(torch.randn(idx.shape[0], D, device=dev).bfloat16(), plan).requires_grad_()
    w = torch.randn(E, F, D, device=dev).bfloat16().requires_grad_()
    if dtype == torch.float32:
        w.main_grad, w.main_grad_written = torch.full((E, F, D), 7.0, device=dev), False
    offs = plan.offs.tolist()
    dy = torch.zeros(plan.max_rows, F, device=dev, dtype=torch.bfloat16)
    dy[:offs[-1]] = torch.randn(offs[-1], F, device=dev).bfloat16()
    lib = _lib.load()
    lib.fsb_gemm_set_pair_mode(pairs)
    try:
        y = moe.grouped_linear(x, w, plan)
        y.backward(dy)
    finally:
        lib.fsb_gemm_set_pair_mode(1)
    ops.check_status()
    dw = w.main_grad if dtype == torch.float32 else w.grad
    for e in range(E):
        r = slice(offs[e], offs[e + 1])
        xe, we, de = x.detach()[r].double(), w.detach()[e].double(), dy[r].double()
        for got, ref, mag, n in ((dw[e], de.t() @ xe, de.abs().t() @ xe.abs(), max(counts)),
                                 (y[r], xe @ we.t(), xe.abs() @ we.abs().t(), D), (x.grad[r], de @ we, de.abs() @ we.abs(), F)):
            bound = mag * (n * 2.0 ** -24) + ref.abs() * (2.0 ** -8 if got.dtype == torch.bfloat16 else 0)
            assert ((got.double() - ref).abs() <= bound).all()
