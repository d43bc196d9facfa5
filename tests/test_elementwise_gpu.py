"""Bandwidth kernels against fp32 PyTorch references (the CPU path of the same wrappers)."""
import numpy as np
import pytest
import torch

from flex_shard_b200 import ops
from flex_shard_b200.ops import elementwise as ew

pytestmark = pytest.mark.gpu
DEV = "cuda"


def test_rmsnorm_fwd_bwd():
    torch.manual_seed(0)
    x = torch.randn(3, 70, 512, device=DEV).bfloat16().requires_grad_()
    w = (1 + 0.1 * torch.randn(512, device=DEV)).bfloat16().requires_grad_()
    y = ew.rmsnorm(x, w, 1e-5)
    g = torch.randn_like(y)
    y.backward(g)
    xc = x.detach().cpu().requires_grad_()
    wc = w.detach().cpu().requires_grad_()
    yc = ew.rmsnorm(xc, wc, 1e-5)
    yc.backward(g.cpu())
    torch.testing.assert_close(y.cpu().float(), yc.float(), rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(x.grad.cpu().float(), xc.grad.float(), rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(w.grad.cpu().float(), wc.grad.float(), rtol=3e-2, atol=1e-1)


def test_add_rmsnorm():
    torch.manual_seed(1)
    x = torch.randn(130, 256, device=DEV).bfloat16().requires_grad_()
    r = torch.randn(130, 256, device=DEV).bfloat16().requires_grad_()
    w = torch.ones(256, device=DEV).bfloat16().requires_grad_()
    y, s = ew.add_rmsnorm(x, r, w)
    (y.float().sum() + 2 * s.float().sum()).backward()
    xc, rc_, wc = (t.detach().cpu().requires_grad_() for t in (x, r, w))
    yc, sc = ew.add_rmsnorm(xc, rc_, wc)
    (yc.float().sum() + 2 * sc.float().sum()).backward()
    torch.testing.assert_close(y.cpu().float(), yc.float(), rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(s.cpu().float(), sc.float(), rtol=1e-2, atol=1e-2)
    torch.testing.assert_close(x.grad.cpu().float(), xc.grad.float(), rtol=2e-2, atol=3e-2)
    torch.testing.assert_close(r.grad.cpu().float(), rc_.grad.float(), rtol=2e-2, atol=3e-2)


def test_rope_roundtrip_and_reference():
    torch.manual_seed(2)
    B, S, H, hd = 2, 48, 4, 64
    table = ew.rope_table(S, hd, 5e5, DEV)
    x = torch.randn(B, S, H, hd, device=DEV).bfloat16()
    ref = ew._rope_ref(x.cpu(), table.cpu(), False)
    xr = x.clone().requires_grad_()
    y = ew.rope(xr * 1.0, table)
    torch.testing.assert_close(y.cpu().float(), ref.float(), rtol=1e-2, atol=1e-2)
    g = torch.randn_like(y)
    y.backward(g)
    gref = ew._rope_ref(g.cpu(), table.cpu(), True)
    torch.testing.assert_close(xr.grad.cpu().float(), gref.float(), rtol=1e-2, atol=1e-2)


def test_swiglu():
    torch.manual_seed(3)
    gu = torch.randn(100, 2 * 320, device=DEV).bfloat16().requires_grad_()
    h = ew.swiglu(gu)
    g = torch.randn_like(h)
    h.backward(g)
    gc = gu.detach().cpu().requires_grad_()
    hc = ew.swiglu(gc)
    hc.backward(g.cpu())
    torch.testing.assert_close(h.cpu().float(), hc.float(), rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(gu.grad.cpu().float(), gc.grad.float(), rtol=2e-2, atol=2e-2)


def test_cross_entropy_matches_torch():
    torch.manual_seed(4)
    T, V = 64, 1024
    logits = (3 * torch.randn(T, V, device=DEV)).bfloat16()
    tgt = torch.randint(0, V, (T,), device=DEV)
    tgt[5] = -100
    lf = logits.float().requires_grad_()
    ref = torch.nn.functional.cross_entropy(lf, tgt, reduction="sum") / T
    ref.backward()
    lg = logits.clone().requires_grad_()
    loss = ew.cross_entropy(lg * 1.0, tgt)
    loss.backward()
    torch.testing.assert_close(loss, ref.detach(), rtol=1e-3, atol=1e-3)
    torch.testing.assert_close(lg.grad.float(), lf.grad, rtol=2e-2, atol=2e-4)


@pytest.mark.parametrize("pdt,gdt", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32),
                                     (torch.float32, torch.bfloat16)])
def test_adamw_matches_torch(pdt, gdt):
    torch.manual_seed(5)
    n = 10007
    p0 = torch.randn(n, device=DEV)
    p = p0.to(pdt).clone()
    ref = torch.nn.Parameter(p.float().clone())
    opt = torch.optim.AdamW([ref], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    m = torch.zeros(n, device=DEV)
    v = torch.zeros(n, device=DEV)
    for step in range(1, 4):
        g = torch.randn(n, device=DEV).to(gdt)
        ref.grad = g.float()
        opt.step()
        ew.adamw_step_(p, g, m, v, lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=step)
        if pdt == torch.bfloat16:
            ref.data.copy_(ref.data.bfloat16().float())
    tol = 1e-5 if pdt == torch.float32 else 2e-2
    torch.testing.assert_close(p.float(), ref.data, rtol=tol, atol=tol)
    ops.check_status()


def test_cast_scale():
    a = torch.randn(5000, device=DEV)
    b = torch.zeros(5000, device=DEV, dtype=torch.bfloat16)
    ew.cast_scale_(b, a, 0.5)
    torch.testing.assert_close(b.float(), (a * 0.5).bfloat16().float())
    c = torch.ones(5000, device=DEV)
    ew.cast_scale_(c, b, 2.0, accumulate=True)
    torch.testing.assert_close(c, 1 + 2 * b.float())


def test_swiglu_over_the_range_of_the_gate():
    """Gates down to where the exponential nears the largest fp32 value (the quotient is tiny there, and not 0). Bound:
    an argument of up to 88.5 in the fast exponential is good to 88.5 * 2^-23; one rounding to bf16."""
    gate = torch.cat([torch.linspace(-88.5, 88.5, 355), torch.linspace(-2, 2, 45)]).bfloat16()
    x = torch.stack([gate, torch.ones_like(gate)]).to(DEV).view(1, -1).requires_grad_()
    h = ew.swiglu(x)
    h.backward(torch.ones_like(h))
    ops.check_status()
    g = gate.double()
    silu, sg = g * torch.sigmoid(g), torch.sigmoid(g)
    rel = 2.0 ** -8 + 88.5 * 2.0 ** -23
    for got, want in ((h[0], silu), (x.grad[0, 400:], silu)):
        assert ((got.detach().double().cpu() - want).abs() <= want.abs() * rel).all()
    # the gate's gradient is a difference of terms: their size counts
    size = sg + silu.abs() * (1 - sg)
    assert ((x.grad[0, :400].double().cpu() - (sg + silu * (1 - sg))).abs() <= size * rel).all()


@pytest.mark.parametrize("offset", [0, 8, 1])
@pytest.mark.parametrize("gdt", [torch.float32, torch.bfloat16])
def test_adamw_at_every_alignment(offset, gdt):
    """32-byte, 16-byte and element-wise accesses give the same result, and it is that of fp64 arithmetic: moments to a few
    fp32 roundings, a bf16 parameter to its own rounding (and, where that lies close to a tie, one step of it)."""
    torch.manual_seed(12)
    n = 8 * 1000 + 3
    flat = lambda t: torch.cat([t.new_zeros(offset), t])[offset:]   # noqa: E731
    p0 = torch.randn(n, device=DEV).bfloat16()
    g0, m0 = torch.randn(n, device=DEV).to(gdt), torch.randn(n, device=DEV) * 0.1
    v0 = torch.randn(n, device=DEV).square() * 10.0 ** torch.randint(-12, 1, (n,), device=DEV)
    p, g, m, v = flat(p0), flat(g0), flat(m0), flat(v0)
    ew.adamw_step_(p, g, m, v, lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=3)
    gd = g0.double()
    md, vd = m0.double() * 0.9 + gd * 0.1, v0.double() * 0.95 + gd.square() * 0.05
    step = 1e-2 / (1 - 0.9 ** 3) * md / (vd.sqrt() / (1 - 0.95 ** 3) ** 0.5 + 1e-8)
    want = p0.double() * (1 - 1e-3) - step
    mag = m0.abs().double() + gd.abs()
    assert ((m.double() - md).abs() <= mag * 2.0 ** -22).all()
    assert ((v.double() - vd).abs() <= vd * 2.0 ** -21).all()
    assert ((p.double() - want).abs() <= (want.abs() * 2.0 ** -8 + (p0.abs().double() + step.abs()) * 2.0 ** -18)).all()
    ops.check_status()


@pytest.mark.parametrize("pdt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("offset", [0, 8, 1])
def test_adamw_update_is_correctly_rounded(pdt, offset):
    """From a parameter of 0 without decay the stored value is the update itself. At the first step its factors are exact
    in fp32, so from the stored moments it has to be, bit for bit, what IEEE square root, quotients and product give."""
    torch.manual_seed(14)
    n, lr, b1, b2, eps = 8 * 2 ** 16 + 3, 1e-2, 0.9, 0.95, 1e-8
    flat = lambda t: torch.cat([t.new_zeros(offset), t])[offset:]   # noqa: E731
    p, g, m = (flat(t) for t in (torch.zeros(n, device=DEV, dtype=pdt), torch.randn(n, device=DEV),
                                 torch.randn(n, device=DEV) * 0.1))
    v = flat(torch.randn(n, device=DEV).square() * 10.0 ** torch.randint(-12, 1, (n,), device=DEV))
    ew.adamw_step_(p, g, m, v, lr=lr, beta1=b1, beta2=b2, eps=eps, weight_decay=0.0, step=1)
    f = np.float32
    root = np.sqrt(v.cpu().numpy()) / np.sqrt(f(1) - f(b2)) + f(eps)
    want = -(f(lr) / (f(1) - f(b1)) * (m.cpu().numpy() / root))
    assert want.dtype == f and torch.equal(p.cpu(), torch.from_numpy(want).to(pdt))
    ops.check_status()


@pytest.mark.parametrize("sizes", [[1], [7, 32768, 32769, 65543], [3] * 97 + [200001]])
def test_clip_over_many_tensors(sizes):
    """Edges: one element, a chunk and one more, odd remainders, unaligned views, more tensors than a launch takes."""
    from flex_shard_b200.ops import multi_tensor

    torch.manual_seed(11)
    base = [torch.randn(n + 1, device=DEV) for n in sizes]
    grads = [b[i % 2:i % 2 + n] if i % 3 else b[:n].bfloat16() for i, (b, n) in enumerate(zip(base, sizes))]
    want = torch.stack([g.double().square().sum() for g in grads]).sum()
    got = multi_tensor.sum_squares(grads)
    # fp32 partial sums of at most 128 terms a thread and a tree over them: well within 200 roundings of 2^-24
    assert abs(float(got) - float(want)) <= 1.2e-5 * float(want)
    norm = got.sqrt()
    limit = 0.25 * float(norm)
    ref = [g.double() * (limit / (float(norm) + 1e-6)) for g in grads]
    kept = [g.clone() for g in grads]
    multi_tensor.clip_by_norm_(grads, norm, 2 * float(norm))            # below the limit: bit for bit the same
    assert all(torch.equal(a, b) for a, b in zip(grads, kept))
    multi_tensor.clip_by_norm_(grads, norm, limit)
    for g, r in zip(grads, ref):
        # one rounding of the product to the stored type, plus three fp32 roundings in the coefficient
        torch.testing.assert_close(g.double(), r, rtol=2.0 ** -8 if g.dtype == torch.bfloat16 else 2.0 ** -21, atol=0)
    multi_tensor.clip_by_norm_(grads, torch.full((), float("nan"), device=DEV), 1.0)
    assert all(g.isnan().all() for g in grads)
    ops.check_status()


@pytest.mark.parametrize("shape", [(3, 8), (5, 1000), (257, 4096)])
@pytest.mark.parametrize("factor", [1.0, 0.37])
def test_cross_entropy_gradient_of_a_scaled_loss(shape, factor):
    """The saved gradient is scaled in place when the graph ends with this backward and kept when it does not."""
    torch.manual_seed(3)
    x = torch.randn(*shape, device=DEV).bfloat16()
    target = torch.randint(0, shape[1], (shape[0],), device=DEV)
    ref = x.double().requires_grad_()
    (torch.nn.functional.cross_entropy(ref, target) * factor).backward()
    leaf = x.clone().requires_grad_()
    loss = ew.cross_entropy(leaf.clone(), target) * factor
    again = torch.autograd.grad(loss, leaf, retain_graph=True)[0].clone()
    twice = torch.autograd.grad(loss, leaf, retain_graph=True)[0].clone()
    last = torch.autograd.grad(loss, leaf)[0]
    scaled = torch.full((), factor, device=DEV, requires_grad=True)       # a gradient that is differentiated again
    graph = torch.autograd.grad(ew.cross_entropy(leaf.clone(), target) * scaled, leaf, create_graph=True, retain_graph=False)[0]
    assert graph.requires_grad
    for got in (again, twice, last, graph.detach()):
        # two roundings to bf16 (the saved gradient, its scaled copy) of values below 1 / T
        torch.testing.assert_close(got.double(), ref.grad, rtol=2.0 ** -7, atol=2.0 ** -12 / shape[0])
    assert torch.equal(again, twice)
    ops.check_status()


@pytest.mark.parametrize("V", [1000, 56320, 102400, 133120, 145416])
def test_cross_entropy_of_masked_logits(V):
    """Logits of -inf: a whole row but one, either half, the first groups of eight, every other group."""
    torch.manual_seed(16)
    x = torch.randn(6, V, device=DEV).bfloat16()
    tgt = torch.tensor([V // 2, V - 1, 3, V - 2, 8, V - 8], device=DEV)
    x[0, :] = -torch.inf
    x[0, V // 2] = 1.0
    x[1, : V // 2] = -torch.inf
    x[2, V // 2:] = -torch.inf
    x[3, : V - 16] = -torch.inf
    x[4].view(-1, 8)[::2] = -torch.inf
    x[5, : V - 8] = -torch.inf
    ref = x.double().requires_grad_()
    want = torch.nn.functional.cross_entropy(ref, tgt)
    want.backward()
    leaf = x.clone().requires_grad_()
    loss = ew.cross_entropy(leaf * 1.0, tgt)
    loss.backward()
    assert abs(float(loss.detach()) - float(want.detach())) <= 1e-5 * abs(float(want.detach()))
    torch.testing.assert_close(leaf.grad.double(), ref.grad, rtol=2.0 ** -8 + 2e-5, atol=1e-9)
    ops.check_status()


def test_cross_entropy_takes_batched_loss_gradients():
    torch.manual_seed(3)
    x, target = torch.randn(5, 1000, device=DEV).bfloat16(), torch.randint(0, 1000, (5,), device=DEV)
    factors = torch.tensor([1.0, 0.37, -2.0], device=DEV)
    ref = x.double().requires_grad_()
    (want,) = torch.autograd.grad(torch.nn.functional.cross_entropy(ref, target), ref)
    leaf = x.clone().requires_grad_()
    (got,) = torch.autograd.grad(ew.cross_entropy(leaf.clone(), target), leaf, factors, is_grads_batched=True)
    # three roundings to bf16: the saved gradient, the factor, their product
    torch.testing.assert_close(got.double(), factors.double()[:, None, None] * want, rtol=3 * 2.0 ** -8, atol=2.0 ** -12)
    ops.check_status()


@pytest.mark.parametrize("T,V,D,kind", [(1, 3, 8, "any"), (300, 50, 264, "any"), (5000, 7, 2056, "one"), (4097, 4000, 4096, "any"),
                                        (2048, 100, 8192, "one"), (777, 1, 64, "any")])
@pytest.mark.parametrize("main", [None, False, True])
def test_embedding_gradient(T, V, D, kind, main):
    """Values read once, never, and more often than a block orders at a time; a new bf16 gradient, an fp32 destination that
    is overwritten (main False) or added to (main True)."""
    from flex_shard_b200.ops.embedding import embedding

    torch.manual_seed(13)
    w = torch.randn(V, D, device=DEV).bfloat16().requires_grad_()
    tokens = torch.randint(0, V, (T,), device=DEV) if kind == "any" else torch.full((T,), V - 1, device=DEV)
    if T % 2:
        tokens = tokens.int()
    dy = torch.randn(T, D, device=DEV).bfloat16()
    got = []
    for _ in range(2):
        base = torch.randn(V, D, device=DEV, generator=torch.Generator(DEV).manual_seed(1))
        w.grad = None
        if main is not None:
            w.main_grad, w.main_grad_written = base.clone(), main
        y = embedding(tokens.view(1, -1), w)
        assert torch.equal(y[0], w.detach()[tokens])
        y.backward(dy[None])
        got.append(w.grad if main is None else w.main_grad)
    ops.check_status()
    assert torch.equal(*got)                                          # the same bits on every run
    want = torch.zeros(V, D, device=DEV, dtype=torch.float64).index_add_(0, tokens.long(), dy.double())
    mag = torch.zeros_like(want).index_add_(0, tokens.long(), dy.double().abs())
    if main:
        want, mag = want + base.double(), mag + base.double().abs()
    count = torch.bincount(tokens, minlength=V).clamp_min(1)[:, None]
    bound = mag * (count * 2.0 ** -23) + (want.abs() * 2.0 ** -8 if main is None else 0)
    assert ((got[0].double() - want).abs() <= bound).all()


@pytest.mark.parametrize("counts,V", [([64, 65, 63, 1], 9), ([2048, 2049, 128, 3], 5000), ([70000, 100, 65], 300), ([65], 1)])
@pytest.mark.parametrize("main", [None, True])
def test_embedding_gradient_of_frequent_tokens(counts, V, main):
    """Values on either side of what one block adds (64 rows), of what it orders at once (2048 positions) and far above,
    with others never read: the same bits on every run, and as good as a sum in fp32."""
    from flex_shard_b200.ops.embedding import embedding

    torch.manual_seed(15)
    D, T = 40, sum(counts)
    values = torch.linspace(0, V - 1, len(counts)).long()
    tokens = torch.repeat_interleave(values, torch.tensor(counts))[torch.randperm(T)].to(DEV)
    w = torch.randn(V, D, device=DEV).bfloat16().requires_grad_()
    dy, base, got = torch.randn(T, D, device=DEV).bfloat16(), torch.randn(V, D, device=DEV), []
    for _ in range(2):
        w.grad = None
        if main is not None:
            w.main_grad, w.main_grad_written = base.clone(), main
        embedding(tokens, w).backward(dy)
        got.append(w.grad if main is None else w.main_grad)
    assert torch.equal(*got)
    want = torch.zeros(V, D, device=DEV, dtype=torch.float64).index_add_(0, tokens, dy.double())
    mag = torch.zeros_like(want).index_add_(0, tokens, dy.double().abs())
    if main:
        want, mag = want + base, mag + base.abs()
    # at most 64 additions, then one per 64 of them
    n = 64 + max(counts) / 64 + 2
    bound = mag * (n * 2.0 ** -24) + (want.abs() * 2.0 ** -8 if main is None else 0)
    assert ((got[0].double() - want).abs() <= bound).all()
    ops.check_status()


@pytest.mark.parametrize("dtype", [torch.int64, torch.int32])
def test_embedding_under_the_transforms_of_autograd(dtype):
    """What PyTorch's operator can do besides a backward pass: batched gradients, second derivatives, forward mode,
    ``torch.func``, hooks on a weight whose gradient would go elsewhere. All sums here are exact."""
    import torch.autograd.forward_ad as fwd

    from flex_shard_b200.ops.embedding import TokenEmbedding, embedding

    torch.manual_seed(13)
    V, D = 11, 16
    small = lambda *shape: torch.randint(-4, 5, shape, device=DEV).bfloat16()   # noqa: E731
    tokens = torch.randint(0, V, (2, 3), device=DEV, dtype=dtype)
    w = small(V, D).requires_grad_()
    dys = small(4, 2, 3, D)
    want = torch.stack([torch.zeros(V, D, device=DEV).index_add_(0, tokens.long().view(-1), d.float().view(-1, D))
                        for d in dys]).bfloat16()
    (got,) = torch.autograd.grad(embedding(tokens, w), w, dys, is_grads_batched=True)
    assert torch.equal(got, want)
    dy = dys[0].clone().requires_grad_()
    (dw,) = torch.autograd.grad(embedding(tokens, w), w, dy, create_graph=True)
    assert torch.equal(dw, want[0])
    v = small(V, D)
    assert torch.equal(torch.autograd.grad(dw, dy, v)[0], v[tokens.long()])
    with fwd.dual_level():
        y = embedding(tokens, fwd.make_dual(w.detach(), v))
        assert torch.equal(fwd.unpack_dual(y).tangent, v[tokens.long()])
    assert torch.equal(torch.func.grad(lambda t: (embedding(tokens, t) * dys[0]).sum())(w.detach()), want[0])
    stack = torch.stack([w.detach(), v])
    assert torch.equal(torch.vmap(embedding, in_dims=(None, 0))(tokens, stack), stack[:, tokens.long()])
    m = TokenEmbedding(V, D, dtype=torch.bfloat16, device=DEV)
    m.weight.main_grad, m.weight.main_grad_written, seen = torch.zeros(V, D, device=DEV), False, []
    m.weight.register_hook(seen.append)
    m(tokens).backward(dys[0])
    assert torch.equal(seen[0], want[0]) and torch.equal(m.weight.grad, want[0]) and not m.weight.main_grad_written
    ops.check_status()


@pytest.mark.parametrize("V", [56320, 56328, 102400, 145408, 145416])
def test_cross_entropy_of_rows_on_either_side_of_the_splits(V):
    """Rows of one CTA, of a pair of CTAs (odd halves, the largest) and too long to stay on chip; targets in both halves,
    ignored ones, and a maximum far above the rest in either half."""
    torch.manual_seed(6)
    T = 9
    x = torch.randn(T, V, device=DEV).bfloat16()
    x[0, 5], x[1, V - 3] = 60.0, 60.0
    tgt = torch.randint(0, V, (T,), device=DEV)
    tgt[2], tgt[3], tgt[4] = 0, V - 1, -100
    tgt[5], tgt[6] = (V // 8 + 1) // 2 * 8 - 1, (V // 8 + 1) // 2 * 8
    ref = x.double().requires_grad_()
    want = torch.nn.functional.cross_entropy(ref, tgt, reduction="sum") / T
    want.backward()
    got_x = x.clone().requires_grad_()
    loss = ew.cross_entropy(got_x * 1.0, tgt)
    loss.backward()
    # fp32 sums over V terms and the fast exponential (2 ulp of an argument of up to 70): 1e-5; one rounding to bf16
    assert abs(float(loss.detach()) - float(want.detach())) <= 1e-5 * abs(float(want.detach()))
    torch.testing.assert_close(got_x.grad.double(), ref.grad, rtol=2.0 ** -8 + 2e-5, atol=1e-9)
    ops.check_status()
