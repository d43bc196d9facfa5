"""Newton-Schulz on the tcgen05 GEMM and the Muon elementwise kernels against the CPU path."""
import pytest
import torch

from flex_shard_b200 import ops
from flex_shard_b200.ops import newton_schulz as ns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(256, 1024), (1024, 256), (512, 512)])
def test_newton_schulz_matches_cpu_reference(shape):
    torch.manual_seed(0)
    g = torch.randn(*shape)
    ref = ns.newton_schulz_kernel_reference(g).float()
    out = ns.newton_schulz(g.cuda()).float().cpu()
    ops.check_status()
    # bf16 rounding differs between the two GEMM implementations and is amplified along the
    # small singular directions of a square matrix, so compare in a relative Frobenius sense
    assert (out - ref).norm() / ref.norm() < 3e-2
    sv = torch.linalg.svdvals(out)
    assert sv.max() < 1.3
    if shape[0] != shape[1]:
        assert 0.5 < sv.min()


def test_muon_direction_and_apply_match_cpu():
    torch.manual_seed(1)
    g = torch.randn(384, 640)
    m_cpu = 0.1 * torch.randn(384, 640)
    m_gpu = m_cpu.clone().cuda()
    x_cpu = ns.muon_direction_(m_cpu, g, 0.95, True, 5)
    x_gpu = ns.muon_direction_(m_gpu, g.cuda(), 0.95, True, 5)
    torch.testing.assert_close(m_gpu.cpu(), m_cpu, rtol=1e-5, atol=1e-6)
    torch.testing.assert_close(x_gpu.float().cpu(), x_cpu.float(), rtol=0, atol=4e-2)
    for dt in (torch.float32, torch.bfloat16):
        p = torch.randn(384, 640).to(dt)
        pg = p.clone().cuda()
        ns.muon_apply_(p, x_cpu, 0.02, 0.1, 1.5)
        ns.muon_apply_(pg, x_cpu.cuda(), 0.02, 0.1, 1.5)
        torch.testing.assert_close(pg.float().cpu(), p.float(), rtol=1e-2, atol=1e-2)
    ops.check_status()


def test_prepare_sum_is_reproducible_and_vector_paths_match_scalar():
    """The sum of squares is formed from per-block partials in index order: identical bits on every run.
    An odd length and a misaligned view go through the scalar loop and must agree with the vector path."""
    torch.manual_seed(3)
    dev = torch.device("cuda")
    for n, off in ((4096 * 3000, 0), (1234567, 0), (4096 * 64, 1)):
        g = torch.randn(n + off, device=dev)[off:].view(1, -1)
        m0 = 0.1 * torch.randn(n + off, device=dev)[off:].view(1, -1)
        outs = []
        for _ in range(3):
            m = torch.empty(n + off, device=dev)[off:].view(1, -1)
            m.copy_(m0)
            u = ns.muon_momentum_direction_(m, g, 0.95, True)
            outs.append((m.clone(), u.clone()))
        m_ref = torch.lerp(m0, g, 0.05)
        u_ref = torch.lerp(g, m_ref, 0.95).bfloat16()
        for m, u in outs:
            torch.testing.assert_close(m, m_ref, rtol=1e-6, atol=1e-7)
            assert (u.float() - u_ref.float()).abs().max() <= 2 ** -7 * u_ref.float().abs().max()
            assert torch.equal(u, outs[0][1]) and torch.equal(m, outs[0][0])
    g = torch.randn(2048, 3000, device=dev)
    xs = []
    for _ in range(3):
        m = torch.zeros_like(g)
        xs.append(ns.muon_direction_(m, g, 0.95, True, 0))      # zero iterations: the normalised matrix itself
    assert torch.equal(xs[0], xs[1]) and torch.equal(xs[0], xs[2])
    ref = torch.lerp(g, 0.05 * g, 0.95).bfloat16().float()
    torch.testing.assert_close(xs[0].float(), ref / ref.norm(), rtol=2e-2, atol=1e-6)
    ops.check_status()


@pytest.mark.parametrize("shape", [(6, 256, 512), (4, 512, 256), (3, 384, 384)])
def test_batched_newton_schulz_matches_one_matrix_at_a_time(shape):
    """A stack of equal matrices runs each product of an iteration as one grouped launch; every matrix must
    come out as if it had been orthogonalised alone."""
    torch.manual_seed(4)
    g = torch.randn(*shape, device="cuda")
    assert ns.batched_ns_supported(g)
    before = ops.launch_count()
    out = ns.newton_schulz(g)
    assert ops.launch_count() - before == 15                       # 3 launches per iteration for the whole stack
    for i in range(shape[0]):
        one = ns.newton_schulz(g[i])
        assert (out[i].float() - one.float()).norm() / one.float().norm() < 1e-2
        ref = ns.newton_schulz_kernel_reference(g[i]).float()
        assert (out[i].float().cpu() - ref).norm() / ref.norm() < 3e-2
    ops.check_status()


def test_dist_muon_steps_a_stack_of_equal_matrices_in_one_go():
    """A 3-D parameter (experts) takes the batched path: same update, up to the arithmetic of the iteration, as the
    same matrices held as separate 2-D parameters; far fewer launches."""
    import torch.nn as nn

    from flex_shard_b200.dist_muon import DistMuon

    torch.manual_seed(6)
    E, r, c = 6, 256, 384
    w = torch.randn(E, r, c, device="cuda")
    stacked = nn.Parameter(w.clone())
    singles = [nn.Parameter(w[i].clone()) for i in range(E)]
    opt_a = DistMuon([stacked], param_names=["experts"], lr=0.02)
    opt_b = DistMuon(singles, param_names=[f"e{i}" for i in range(E)], lr=0.02)
    launches = []
    for step in range(2):
        g = torch.randn(E, r, c, device="cuda")
        stacked.grad = g.clone()
        for i, p in enumerate(singles):
            p.grad = g[i].clone()
        for opt in (opt_a, opt_b):
            before = ops.launch_count()
            opt.step()
            launches.append(ops.launch_count() - before)
    for i, p in enumerate(singles):
        torch.testing.assert_close(stacked.detach()[i], p.detach(), rtol=0, atol=2e-3)
        # and the steps themselves: two directions, each within 1e-2 of the matrix's own (as above)
        moved, alone = stacked.detach()[i] - w[i], p.detach() - w[i]
        assert (moved - alone).norm() <= 1e-2 * alone.norm()
    assert launches[0] * 3 < launches[1]            # 1 + 15 + 1 launches (plus normalisation) against 6 x 18
    ops.check_status()


@pytest.mark.parametrize("E,rows,cols", [(5, 192, 1536), (3, 40, 72), (4, 520, 264), (2, 1000, 8), (70, 8, 128), (2, 256, 512)])
def test_batched_products_of_any_size_stay_inside_their_matrix(E, rows, cols):
    """Every product form of the iteration on stacks whose matrices end inside a tile. Bound: one bf16 rounding of the
    result (2^-8 of each element) and fp32 sums over at most 1536 terms of unit variance."""
    torch.manual_seed(8)
    x = torch.randn(E, rows, cols, device="cuda").bfloat16()
    xd = x.double()
    s = min(rows, cols)
    gram = xd @ xd.mT if rows <= cols else xd.mT @ xd

    def check(out, ref):
        assert bool(((out.double() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-3).all())

    buf = torch.full((E + 1, s, s), 7.0, device="cuda", dtype=torch.bfloat16)
    A = buf[:E]
    if rows <= cols:
        ns._batched(x, x, A, s, s, cols, symmetric=True)
    else:
        ns._batched(x, x, A, s, s, rows, a_t=True, b_t=True, symmetric=True)
    check(A, gram)
    assert torch.equal(A, A.mT) and bool((buf[E] == 7.0).all())
    A = (A.float() / s).bfloat16()
    B = torch.empty_like(A)
    ns._batched(A, A, B, s, s, s, c=A, alpha=0.5, beta=-1.5, symmetric=True)
    check(B, 0.5 * (A.double() @ A.double()) - 1.5 * A.double())
    assert torch.equal(B, B.mT)
    nxt = torch.empty_like(x)
    if rows <= cols:
        ns._batched(B, x, nxt, s, cols, s, b_t=True, c=x, beta=2.0)
        check(nxt, B.double() @ xd + 2.0 * xd)
    else:
        ns._batched(x, B, nxt, rows, s, s, c=x, beta=2.0)
        check(nxt, xd @ B.double() + 2.0 * xd)
    ops.check_status()


@pytest.mark.parametrize("E,rows,cols", [(3, 40, 72), (2, 5, 9), (1, 300, 700), (5, 1408, 4096)])
def test_prepare_and_scale_of_a_stack_match_the_matrices_alone(E, rows, cols):
    """One launch over a stack gives the bits of one launch per matrix, sums of squares included, whatever else the stack
    holds (here matrices of very different norms); scaling divides every matrix by its own norm, rounded once to bf16."""
    torch.manual_seed(9)
    size = 10.0 ** torch.arange(E, device="cuda").view(E, 1, 1)
    g = torch.randn(E, rows, cols, device="cuda") * size
    m = torch.randn(E, rows, cols, device="cuda") * size
    ms = m.clone()
    u, ws = ns._prepare(m, g, 0.95, True, E)
    for e in range(E):
        u1, ws1 = ns._prepare(ms[e], g[e], 0.95, True, 1)
        assert torch.equal(u[e], u1) and torch.equal(m[e], ms[e])
        if (rows * cols) % 8 == 0:
            assert torch.equal(ws[e, 0], ws1[0, 0])      # (matrices off the 16-byte grid are added in another order)
        torch.testing.assert_close(ws[e, 0].double(), u1.double().square().sum(), rtol=1e-5, atol=0)
    if (rows * cols) % 8 == 0:
        assert torch.equal(ns._sum_squares(u)[:, 0], ws[:, 0])
    norm = ws[:, 0].sqrt().view(E, 1, 1)
    want = (u.float() / norm).bfloat16()
    got = ns._normalise_(u.clone(), ws, 1e-7)
    assert torch.equal(got, want)                        # the quotient in fp32, rounded once
    ns._normalise_(u[0], ws[:1], 1e-7)                    # a matrix alone: times the reciprocal, two fp32 roundings more
    torch.testing.assert_close(u[0].double(), want[0].double(), rtol=2.0 ** -7, atol=0)
    assert (u[0] != want[0]).float().mean() < 0.01
    ops.check_status()


@pytest.mark.parametrize("E,rows,cols", [(4, 192, 1536), (3, 256, 128)])
def test_stacks_have_the_same_direction_wherever_they_are_orthogonalised(E, rows, cols):
    """Momentum, norm and iteration in one go (stacks that stay where they are stored) and in two steps around an
    exchange (any part of a stack, the gradients' rows elsewhere) give the same bits."""
    torch.manual_seed(11)
    g, m = torch.randn(E, rows, cols, device="cuda"), torch.randn(E, rows, cols, device="cuda")
    m2 = m.clone()
    x = ns.muon_direction_(m, g, 0.95, True, 5)
    u = ns.muon_momentum_direction_(m2, g, 0.95, True)
    assert torch.equal(m, m2)
    part = u[1:].clone()
    assert torch.equal(x, ns.orthogonalise_stack_(u, 5, ns.NS_COEFFS, 1e-7))
    assert torch.equal(x[1:], ns.orthogonalise_stack_(part, 5, ns.NS_COEFFS, 1e-7))
    ops.check_status()


def test_redistributed_stacks_take_the_shared_arithmetic():
    """The computing stage of redistributed parameters gives a stack the direction it would have where it is stored."""
    from types import SimpleNamespace

    from flex_shard_b200.dist_muon import DistMuon

    torch.manual_seed(12)
    g = torch.randn(3, 64, 128, device="cuda")
    opt = DistMuon([torch.nn.Parameter(torch.zeros(3, 64, 128, device="cuda"))], param_names=["experts"], lr=0.02)
    group = opt.param_groups[0]
    m = torch.zeros_like(g)
    want = ns.muon_direction_(m.clone(), g, group["momentum"], group["nesterov"], group["ns_steps"],
                              group["ns_coefficients"], group["eps"])
    u = ns.muon_momentum_direction_(m, g, group["momentum"], group["nesterov"])
    plan = SimpleNamespace(matrices=[(i, i + 1, 0) for i in range(3)])
    kept = u.clone()
    got = opt._compute(SimpleNamespace(resolved=SimpleNamespace(batch=True)), plan, u)
    assert torch.equal(got, want) and torch.equal(u, kept)
    ops.check_status()


def test_stacks_without_sm_pairs_take_a_matrix_at_a_time():
    """With the kernels on SM pairs switched off (or where they do not fit), a stack gives what its matrices give alone."""
    from flex_shard_b200.ops import _lib

    torch.manual_seed(10)
    g = torch.randn(3, 128, 256, device="cuda")
    lib = _lib.load()
    assert ns.batched_ns_supported(g)
    lib.fsb_gemm_set_pair_mode(0)
    try:
        assert not ns.batched_ns_supported(g)
        out = ns.newton_schulz(g)
        assert torch.equal(out, torch.stack([ns.newton_schulz(m) for m in g]))
        with pytest.raises(RuntimeError):
            ns._batched(out, out, torch.empty(3, 128, 128, device="cuda", dtype=out.dtype), 128, 128, 256)
    finally:
        lib.fsb_gemm_set_pair_mode(1)
    ops.check_status()
