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
