"""Training kernels at the sizes where their tiles, vector forms and dispatch change."""
import pytest
import torch

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("T,H,E", [(1, 8, 2), (63, 50, 7), (65, 512, 8), (130, 72, 9), (64, 200, 16), (100, 64, 17), (257, 130, 33),
                                   (128, 2048, 64), (70, 96, 65), (33, 128, 256)])
def test_router_logits_against_fp64(T, H, E):
    """fp32 sums in ascending k: H roundings of partial sums, each at most 2^-24 of the terms' sum so far."""
    from summa_b200 import ops
    torch.manual_seed(T + H + E)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    w = torch.randn(H, E, device="cuda")
    ref = x.double() @ w.double()
    tol = H * 2.0 ** -24 * (x.double().abs() @ w.double().abs())
    assert bool(((ops.router_logits(x, w).double() - ref).abs() <= tol).all())
    wide = torch.zeros(T, H + 8, device="cuda", dtype=torch.bfloat16)
    wide[:, :H] = x
    assert torch.equal(ops.router_logits(wide[:, :H], w), ops.router_logits(x, w))


@gpu
@pytest.mark.parametrize("n,off", [(1, 0), (4, 0), (7, 0), (2053, 0), (4096, 0), (1023, 1), (2048, 4)])
@pytest.mark.parametrize("copy", [True, False])
def test_adamw_vector_and_scalar_ranges(n, off, copy):
    """Ranges that are and are not 16-byte aligned, with remainders, against the same update in fp64 (a few fp32 roundings;
    the compute copy is the master rounded)."""
    from summa_b200.ops import native
    torch.manual_seed(n)
    lr, b1, b2, eps, wd, bc1, bc2, gs = 1e-2, 0.9, 0.95, 1e-8, 0.1, 0.19, 0.0975, 0.5
    mk = lambda: torch.randn(n + off, device="cuda")[off:]
    p, m, v, g = mk(), mk(), mk().abs(), mk()
    pb = torch.zeros(n + off, device="cuda", dtype=torch.bfloat16)[off:] if copy else None
    scale = torch.tensor([gs], device="cuda")
    P, M, V, G = p.double(), m.double(), v.double(), g.double() * gs
    M = b1 * M + (1 - b1) * G
    V = b2 * V + (1 - b2) * G * G
    P = P - lr * wd * P - lr * (M / bc1) / ((V / bc2).sqrt() + eps)
    native.call("sb_adamw", p.data_ptr(), m.data_ptr(), v.data_ptr(), g.data_ptr(), native.ptr(pb), n, scale.data_ptr(), lr, b1, b2,
                eps, wd, bc1, bc2, native.stream())
    for a, b in ((p, P), (m, M), (v, V)):
        torch.testing.assert_close(a.double(), b, rtol=2e-5, atol=2e-6)
    if copy:
        assert torch.equal(pb, p.to(torch.bfloat16))


@gpu
@pytest.mark.parametrize("rows,N,ld", [(1, 8, 8), (63, 264, 264), (65, 256, 512), (5000, 1024, 1024), (27648, 40, 48), (7, 2048, 2048)])
def test_column_sum(rows, N, ld):
    """fp32 sums of bf16 values, deterministic: at most `rows` roundings of 2^-24 of the terms' sum."""
    from summa_b200.ops import cuda_ops
    torch.manual_seed(rows)
    x = torch.randn(rows, ld, device="cuda").to(torch.bfloat16)[:, :N]
    got = cuda_ops.column_sum(x)
    tol = rows * 2.0 ** -24 * x.double().abs().sum(0) + 1e-30
    assert bool(((got.double() - x.double().sum(0)).abs() <= tol).all())
    assert torch.equal(got, cuda_ops.column_sum(x))


@gpu
@pytest.mark.parametrize("shape", [(1, 8, 8), (3, 40, 24), (5, 64, 1032)])
def test_newton_schulz_elementwise_steps(shape):
    """One rounding to bf16 of the fp32 result each."""
    from summa_b200.ops import cuda_ops
    torch.manual_seed(shape[2])
    x, y = torch.randn(shape, device="cuda").to(torch.bfloat16), torch.randn(shape, device="cuda").to(torch.bfloat16)
    want = 3.4445 * x.double() - 4.775 * y.double()
    assert bool(((cuda_ops.axpby(3.4445, x, -4.775, y).double() - want).abs()
                 <= 2.0 ** -8 * want.abs() + 2.0 ** -22 * (3.4445 * x.double().abs() + 4.775 * y.double().abs())).all())
    d = torch.rand(shape[0], 1, 1, device="cuda").to(torch.bfloat16) + 0.5
    assert torch.equal(cuda_ops.matrix_div(x, d), x / d)


@gpu
@pytest.mark.parametrize("shape,off", [((2, 24, 40), 1), ((1, 64, 32), 4), ((3, 16, 16), 8)])
def test_newton_schulz_of_a_view_that_starts_anywhere(shape, off):
    """A contiguous bf16 batch whose first element is off a 16-byte boundary gives the same bits as its aligned copy, and the raw
    entry points refuse it on the host."""
    from summa_b200.ops import cuda_ops, native
    from summa_b200.train.muon import newton_schulz
    torch.manual_seed(off)
    n = shape[0] * shape[1] * shape[2]
    g = torch.randn(n + off, device="cuda").to(torch.bfloat16)[off:].view(shape)
    assert g.is_contiguous() and (g.data_ptr() % 16 != 0) == (off % 8 != 0)
    assert torch.equal(newton_schulz(g), newton_schulz(g.clone()))
    if off % 8:
        with pytest.raises(native.NativeError):
            cuda_ops.axpby(1.0, g, 1.0, g)
        with pytest.raises(native.NativeError):
            cuda_ops.matrix_div(g, torch.ones(shape[0], 1, 1, device="cuda", dtype=torch.bfloat16))


@gpu
@pytest.mark.parametrize("T,Hq,Hkv,D", [(1, 1, 1, 64), (9, 3, 1, 128), (12000, 8, 4, 64)])
def test_qk_norm_rope_backward_gains(T, Hq, Hkv, D):
    """Input and gain gradients with fewer and more (token, head) items than one round of the grid, against fp64 autograd
    (bf16 rounding between norm and rotation and of the result: 2^-8 of a term each)."""
    from summa_b200.ops import cuda_ops, reference
    torch.manual_seed(T)
    W = (Hq + 2 * Hkv) * D
    qkv = torch.randn(1, T, W, device="cuda").to(torch.bfloat16).requires_grad_()
    qg, kg = [(1 + 0.1 * torch.randn(D, device="cuda")).requires_grad_() for _ in range(2)]
    cos, sin = reference.rope_table(T, D, 10000.0, None, "cuda")
    dout = torch.randn(1, T, W, device="cuda").to(torch.bfloat16)
    out = cuda_ops.qkv_rope(qkv, qg, kg, 1e-5, cos, sin, Hq, Hkv, D)
    out.backward(dout)
    x = qkv.detach().double().requires_grad_()
    g64 = [g.detach().double().requires_grad_() for g in (qg, kg)]
    v = x.view(T, Hq + 2 * Hkv, D)
    n = v[:, :Hq + Hkv] * torch.rsqrt(v[:, :Hq + Hkv].pow(2).mean(-1, keepdim=True) + 1e-5)
    n = torch.cat([n[:, :Hq] * g64[0], n[:, Hq:] * g64[1]], 1)
    c, s = cos.double().view(T, 1, D // 2), sin.double().view(T, 1, D // 2)
    a, b = n[..., 0::2], n[..., 1::2]
    r = torch.stack([a * c - b * s, a * s + b * c], -1).flatten(-2)
    torch.cat([r, v[:, Hq + Hkv:]], 1).view(1, T, W).backward(dout.double())
    for got, want in ((qkv.grad, x.grad), (qg.grad, g64[0].grad), (kg.grad, g64[1].grad)):
        assert float((got.double() - want).norm() / want.norm()) <= 2.0 ** -7


@gpu
@pytest.mark.parametrize("T,E,k", [(1, 2, 1), (5, 8, 2), (300, 33, 8), (2049, 64, 4), (2100, 256, 3)])
def test_moe_route_gates_and_plan(T, E, k):
    """Indices, gates and their gradient against the torch ops they stand for (fp32 rounding of 64-bit results), the packed
    plan against a stable sort, with fewer and more routes than a round of the packing block; also a second derivative."""
    from summa_b200 import ops
    torch.manual_seed(T + E)
    logits = torch.randn(T, E, device="cuda").requires_grad_()
    idx, gates = ops.moe_route(logits, k)
    val, want = logits.detach().topk(k, dim=-1)
    assert torch.equal(logits.detach().gather(1, idx), val) and idx.dtype == torch.int64
    ref = logits.detach().double().requires_grad_()
    rg = torch.softmax(ref.gather(1, idx), -1)
    torch.testing.assert_close(gates.double(), rg, rtol=2.0 ** -23, atol=1e-30)
    dg = torch.randn_like(gates)
    (d1,) = torch.autograd.grad(gates, logits, dg, retain_graph=True)
    (r1,) = torch.autograd.grad(rg, ref, dg.double(), retain_graph=True)
    torch.testing.assert_close(d1.double(), r1, rtol=1e-5, atol=1e-6)
    (d2,) = torch.autograd.grad((torch.autograd.grad(gates, logits, dg, create_graph=True)[0] ** 2).sum(), logits)
    (r2,) = torch.autograd.grad((torch.autograd.grad(rg, ref, dg.double(), create_graph=True)[0] ** 2).sum(), ref)
    torch.testing.assert_close(d2.double(), r2, rtol=1e-4, atol=1e-5)
    plan = idx._sb_plan
    flat, meta = idx.view(-1).cpu(), plan.meta.cpu()
    counts = torch.bincount(flat, minlength=E)
    assert torch.equal(plan.counts.cpu().long(), counts)
    row_route, dest = plan.row_route.cpu(), plan.dest.cpu()
    for e in range(E):
        lo, hi, n = int(meta[e]), int(meta[e + 1]), int(counts[e])
        routes = (flat == e).nonzero().view(-1)
        assert hi - lo == -(-n // 128) * 128
        assert torch.equal(row_route[lo:lo + n].long(), routes) and bool((row_route[lo + n:hi] == -1).all())
        assert torch.equal(dest[routes].long(), torch.arange(lo, lo + n))


@gpu
def test_scan_and_convolution_inference_forms():
    """a_log and bf16 taps inside the kernels against the same kernels on prepared operands."""
    from summa_b200 import ops
    from summa_b200.ops import cuda_ops
    torch.manual_seed(0)
    for B, T, C, Ns in ((2, 37, 64, 16), (1, 5, 96, 128)):
        u, d, Bm, Cm = [torch.randn(*s, device="cuda").to(torch.bfloat16) for s in ((B, T, C), (B, T, C), (B, T, Ns), (B, T, Ns))]
        a_log, D = torch.rand(C, Ns, device="cuda") * 3 - 1, torch.randn(C, device="cuda")
        h0 = torch.randn(B, C, Ns, device="cuda")
        with torch.no_grad():
            y, h = ops.selective_scan_log(u, d, a_log, Bm, Cm, D, h0, True)
            yr, hr = cuda_ops.selective_scan(u, d, -torch.exp(a_log), Bm, Cm, D, h0, True)
        torch.testing.assert_close(h, hr, rtol=1e-5, atol=1e-5)
        torch.testing.assert_close(y.float(), yr.float(), rtol=2.0 ** -7, atol=2.0 ** -7)
        for K in (2, 3, 4):
            w, b = torch.randn(C, 1, K, device="cuda").to(torch.bfloat16), torch.randn(C, device="cuda")
            assert torch.equal(cuda_ops.conv1d_silu(u, w, b), cuda_ops.conv1d_silu(u, w.float(), b))
            v = torch.empty(C * K + 1, device="cuda")[1:].view(C, 1, K).copy_(w.float())      # taps that are not 16-byte aligned
            assert torch.equal(cuda_ops.conv1d_silu(u, v, b), cuda_ops.conv1d_silu(u, w.float(), b))


@gpu
@pytest.mark.parametrize("B,T,C,Ns", [(1, 17, 40, 16), (2, 33, 34, 16), (75, 5, 128, 16), (2, 19, 72, 32), (1, 18, 64, 64), (1, 21, 36, 128)])
def test_scan_backward_tiles(B, T, C, Ns):
    """Every gradient for ragged channel tiles and segments, on both sides of the channel-tile rule (75 x 128 / 32 blocks are
    more than two per SM), against fp64 autograd of the recurrence. bf16 outputs round to 2^-9 and the inputs of dA and dD
    are sums of B T products in fp32."""
    from summa_b200.ops import cuda_ops
    torch.manual_seed(B + T + C)
    u, d, Bm, Cm = [torch.randn(*s, device="cuda").to(torch.bfloat16) for s in ((B, T, C), (B, T, C), (B, T, Ns), (B, T, Ns))]
    A, D = -torch.rand(C, Ns, device="cuda") - 0.1, torch.randn(C, device="cuda")
    dy = torch.randn(B, T, C, device="cuda").to(torch.bfloat16)
    lo = [t.detach().clone().requires_grad_() for t in (u, d, A, Bm, Cm, D)]
    y, _ = cuda_ops.selective_scan(*lo)
    y.backward(dy)
    hi = [t.detach().double().requires_grad_() for t in (u, d, A, Bm, Cm, D)]
    dt = torch.nn.functional.softplus(hi[1])
    h, ys = torch.zeros(B, C, Ns, device="cuda", dtype=torch.float64), []
    for t in range(T):
        h = torch.exp(dt[:, t, :, None] * hi[2]) * h + (dt[:, t] * hi[0][:, t])[..., None] * hi[3][:, t, None]
        ys.append((h * hi[4][:, t, None]).sum(-1) + hi[5] * hi[0][:, t])
    torch.stack(ys, 1).backward(dy.double())
    for a, b in zip(lo, hi):
        assert float((a.grad.double() - b.grad).norm() / b.grad.norm()) <= 2.0 ** -8


@gpu
def test_scan_without_gradients_does_not_drop_a_forward_mode_tangent():
    from summa_b200 import ops
    import torch.autograd.forward_ad as fwd
    torch.manual_seed(0)
    u, delta, Bm, Cm = [torch.randn(1, 9, n, device="cuda").to(torch.bfloat16) for n in (16, 16, 8, 8)]
    a_log, D = torch.rand(16, 8, device="cuda"), torch.ones(16, device="cuda")
    with torch.no_grad():
        y, _ = ops.selective_scan_log(u, delta, a_log, Bm, Cm, D)
        with fwd.dual_level():
            with pytest.raises((RuntimeError, NotImplementedError)):
                ops.selective_scan_log(u, delta, fwd.make_dual(a_log, torch.ones_like(a_log)), Bm, Cm, D)
            again, _ = ops.selective_scan_log(u, delta, a_log, Bm, Cm, D)
    # without a tangent the autograd function runs: A from the library's exponential, one unit in the last place of fp32 away
    torch.testing.assert_close(again.float(), y.float(), rtol=2 ** -7, atol=2 ** -10)


@gpu
def test_bias_gradient_stays_differentiable():
    """The gradient of a bias under `create_graph`, differentiated once more with respect to what came from above."""
    from summa_b200 import ops
    torch.manual_seed(2)
    x, w = torch.randn(40, 32, device="cuda").to(torch.bfloat16), torch.randn(32, 16, device="cuda").to(torch.bfloat16)
    b = torch.zeros(16, device="cuda", requires_grad=True)
    up = torch.randn(40, 16, device="cuda").to(torch.bfloat16).requires_grad_(True)
    db, = torch.autograd.grad(ops.linear(x, w, b), b, up, create_graph=True)
    again, = torch.autograd.grad(db.pow(2).sum(), up)
    want = (2 * up.detach().double().sum(0)).expand(40, 16)
    torch.testing.assert_close(again.double(), want, rtol=2 ** -8, atol=1e-6)


@gpu
@pytest.mark.parametrize("B,T,C,N", [(1, 19, 40, 8), (2, 33, 72, 16), (3, 17, 40, 32), (2, 16, 24, 64), (2, 17, 2368, 128), (2, 17, 2370, 128),
                                     (11, 9, 1076, 128), (12, 9, 1024, 128), (1, 17, 24, 256)])
def test_scan_forward_tilings_against_fp64(B, T, C, N):
    """Every number of states per thread and channels per block, with N 128 on both sides of its two lines (148 blocks of 32
    channels, 11840 channels in all). The states are fp32 sums with decays of a few 2^-22 each; y is rounded to bf16."""
    from summa_b200.ops import cuda_ops
    torch.manual_seed(B + C + N)
    u, delta, Bm, Cm = [torch.randn(B, T, n, device="cuda").to(torch.bfloat16) for n in (C, C, N, N)]
    a_log, D, h0 = torch.rand(C, N, device="cuda") * 2 - 1, torch.randn(C, device="cuda"), torch.randn(B, C, N, device="cuda")
    with torch.no_grad():
        y, h = cuda_ops.selective_scan_log(u, delta, a_log, Bm, Cm, D, h0, True)
    hs, mag, A = h0.double(), h0.double().abs(), -torch.exp(a_log.double())
    for t in range(T):
        dt, x = torch.nn.functional.softplus(delta[:, t].double()), u[:, t].double()
        decay, inp = torch.exp(dt[..., None] * A), (dt * x)[..., None] * Bm[:, t].double()[:, None]
        hs, mag = decay * hs + inp, decay * mag + inp.abs()
        want = (hs * Cm[:, t].double()[:, None]).sum(-1) + D.double() * x
        tol = 2.0 ** -15 * ((mag * Cm[:, t].double().abs()[:, None]).sum(-1) + (D.double() * x).abs()) + 2.0 ** -8 * want.abs()
        assert bool(((y[:, t].double() - want).abs() <= tol).all())
    assert bool(((h.double() - hs).abs() <= 2.0 ** -15 * mag).all())
