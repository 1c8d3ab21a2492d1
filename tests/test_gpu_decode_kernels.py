"""Kernels of a decode step at the sizes where their dispatch, tiles and remainders change."""
import pytest
import torch

gpu = pytest.mark.gpu


def _w4(K, N, seed):
    from summa_b200.ops import reference
    torch.manual_seed(seed)
    packed, scales = reference.quantize_int4_g128(torch.randn(K, N) * 0.05)
    packed, scales = packed.cuda(), scales.cuda()
    return packed, scales, reference.repack_int4_k8(packed), reference.dequantize_int4_g128(packed.cpu(), scales.cpu()).double().cuda()


@gpu
@pytest.mark.parametrize("M,K,N", [
    (1, 128, 4), (2, 256, 20), (3, 2048, 16), (1, 2176, 132), (8, 1920, 68),        # one group; fewer and more than 16 groups; ragged tiles
    (2, 14464, 36), (1, 20480, 28), (4, 9088, 44), (8, 4352, 2400),                 # K in passes / the last that fits one pass
    (8, 4736, 52), (5, 14336, 40)])                                                 # rows 5..8 beyond one pass: the other kernel
@pytest.mark.parametrize("spread", [0, 24])
def test_w4_projection_against_fp64(M, K, N, spread):
    """x spreads over 2^-spread .. 1: a group's fixed-point step is 2^-21 of its largest magnitude, so a product is off by at
    most 2^-21 max|x| |w| per term, next to fp32 sums (2^-20 of the terms' sum is above both) and one rounding to bf16."""
    from summa_b200 import ops
    packed, scales, k8, wq = _w4(K, N, M + K + N)
    x = (torch.randn(M, K, device="cuda") * torch.exp2(-spread * torch.rand(M, K, device="cuda"))).to(torch.bfloat16)
    res = torch.randn(M, N, device="cuda").to(torch.bfloat16)
    ref = x.double() @ wq
    big = x.double().view(M, K // 128, 128).abs().amax(-1, keepdim=True).expand(M, K // 128, 128).reshape(M, K)
    slack = 2.0 ** -20 * (big @ wq.abs())
    if M > 4 and 3 * M * K > 104 * 1024:                                            # that kernel rounds the weights to bf16
        slack += 2.0 ** -9 * (x.double().abs() @ wq.abs())
    for got, want in ((ops.int4_gemv(x, packed, scales, None, k8), ref), (ops.int4_gemv(x, packed, scales, res, k8), ref + res.double())):
        assert bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + slack + 1e-30).all())


@gpu
def test_w4_projection_keeps_nan_and_inf_in_their_row():
    from summa_b200 import ops
    packed, scales, k8, wq = _w4(512, 40, 3)
    x = torch.randn(4, 512, device="cuda").to(torch.bfloat16)
    clean = ops.int4_gemv(x, packed, scales, None, k8)
    x[1, 7], x[2, 300] = float("inf"), float("nan")
    got = ops.int4_gemv(x, packed, scales, None, k8)
    assert bool(got[1].isnan().all()) and bool(got[2].isnan().all())
    assert torch.equal(got[0], clean[0]) and torch.equal(got[3], clean[3])


@gpu
def test_w4_projection_takes_unaligned_operand_views():
    from summa_b200 import ops
    packed, scales, k8, wq = _w4(256, 24, 5)
    s1 = torch.empty(scales.numel() + 1, device="cuda", dtype=scales.dtype)[1:].view_as(scales).copy_(scales)
    k1 = torch.empty(k8.numel() + 1, device="cuda", dtype=k8.dtype)[1:].view_as(k8).copy_(k8)
    assert s1.data_ptr() % 8 and k1.data_ptr() % 16
    x = torch.randn(2, 256, device="cuda").to(torch.bfloat16)
    assert torch.equal(ops.int4_gemv(x, packed, s1, None, k1), ops.int4_gemv(x, packed, scales, None, k8))


@gpu
@pytest.mark.parametrize("M,K,I", [(1, 128, 4), (3, 9088, 20), (2, 14464, 12)])
def test_w4_gated_projection_edges(M, K, I):
    from summa_b200.ops import cuda_ops
    packed, scales, k8, wq = _w4(K, 2 * I, M + K + I)
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    got = cuda_ops.int4_gemv_swiglu(x, k8, scales).double()
    u = (x.double() @ wq).to(torch.bfloat16).double()
    ref = torch.nn.functional.silu(u[:, :I]) * u[:, I:]
    # gate and value are rounded to bf16 first and may fall to the other side of a rounding boundary (2^-8 each)
    assert bool(((got - ref).abs() <= 2.0 ** -6 * ref.abs() + 2.0 ** -7 * u.abs().amax()).all())


@gpu
@pytest.mark.parametrize("M,K,N", [(9, 512, 132), (33, 4096, 260), (64, 14336, 128), (64, 1024, 2052), (128, 4096, 384), (257, 2048, 516)])
def test_w4a16_split_k_reduction(M, K, N):
    """K split over a cluster with ragged rows and columns; the residual also as a view that is not 8-byte aligned. The kernel
    rounds the weights to bf16 (2^-9 of each term), sums in fp32 and rounds once."""
    from summa_b200.ops import cuda_ops, native
    packed, scales, k8, wq = _w4(K, N, M + K + N)
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    res = torch.randn(M * N + 1, device="cuda").to(torch.bfloat16)
    slack = 2.0 ** -9 * (x.double().abs() @ wq.abs())
    for r in (res[:-1].view(M, N), res[1:].view(M, N)):
        y = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
        native.call("sb_w4a16_gemm", x.data_ptr(), k8.data_ptr(), scales.data_ptr(), None, r.data_ptr(), y.data_ptr(), M, N, K, K,
                    native.stream())
        want = x.double() @ wq + r.double()
        assert bool(((y.double() - want).abs() <= 2.0 ** -7 * (want.abs() + r.double().abs()) + slack).all())
    assert native.read_error_flag() == 0


@gpu
@pytest.mark.parametrize("M,K,N", [
    (1, 8, 2), (2, 96, 3072), (3, 1000, 353), (8, 4104, 2366), (5, 1032, 2369),     # K and N tails; the last N of 16-column tiles
    (8, 14344, 48), (6, 14336, 4100), (1, 40968, 24)])                              # K in passes, both tile widths
def test_bf16_projection_against_fp64(M, K, N):
    """`ops.linear` with up to 8 rows and the decode form (bias, residual, fused norm) on a weight with padded rows. fp32 sums
    (2^-18 of the terms' sum), one rounding to bf16, one more before a residual."""
    from summa_b200 import ops
    from summa_b200.ops import cuda_ops, native
    torch.manual_seed(M + K + N)
    w = (torch.randn(K, (N + 15) // 8 * 8, device="cuda") * 0.05).to(torch.bfloat16)[:, :N]
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    bias, res = torch.randn(N, device="cuda"), torch.randn(M, N, device="cuda").to(torch.bfloat16)
    gamma = 1 + 0.1 * torch.randn(K, device="cuda")
    xn = ops.rmsnorm(x, gamma, 1e-5)

    def check(got, inp, b, r):
        proj = inp.double() @ w.double() + (0 if b is None else b.double())
        want = proj if r is None else proj + r.double()
        tol = 2.0 ** -8 * (want.abs() + (0 if r is None else proj.abs())) + 2.0 ** -18 * (inp.double().abs() @ w.double().abs())
        assert bool(((got.double() - want).abs() <= tol + 1e-30).all())
    if N % 8 == 0:                                        # the general entry's own shape rule
        check(ops.linear(x, w, None), x, None, None)
        check(ops.linear(x, w, bias), x, bias, None)
    check(cuda_ops.decode_linear(x, w, bias.to(torch.bfloat16), res), x, bias.to(torch.bfloat16), res)
    got = cuda_ops.decode_linear(x, w, None, res, norm=(gamma, 1e-5))
    # the fused norm may round single elements of the normed row the other way (2^-8 of one term each)
    proj = xn.double() @ w.double()
    tol = 2.0 ** -7 * (proj.abs() + res.double().abs()) + 2.0 ** -8 * (xn.double().pow(2) @ w.double().pow(2)).sqrt() + 2.0 ** -18 * (xn.double().abs() @ w.double().abs())
    assert bool(((got.double() - proj - res.double()).abs() <= tol + 1e-30).all())
    assert native.read_error_flag() == 0


@gpu
@pytest.mark.parametrize("rows,H", [(1, 2048), (64, 4096), (7, 8192), (3, 2056), (1184, 2048), (1185, 2048), (5, 8200)])
def test_rmsnorm_row_per_cta(rows, H):
    from summa_b200 import ops
    torch.manual_seed(rows + H)
    x, r = torch.randn(rows, H, device="cuda").to(torch.bfloat16), torch.randn(rows, H, device="cuda").to(torch.bfloat16)
    gamma = 1 + 0.1 * torch.randn(H, device="cuda")
    for res in (None, r):
        s = x if res is None else (x.float() + res.float()).to(torch.bfloat16)
        ref = s.double() * torch.rsqrt(s.double().pow(2).mean(-1, keepdim=True) + 1e-5) * gamma.double()
        y = ops.rmsnorm(x, gamma, 1e-5) if res is None else ops.add_rmsnorm(x, res, gamma, 1e-5)
        if res is not None:
            assert torch.equal(y[1], s)
            y = y[0]
        # one rounding to bf16 next to fp32 statistics
        assert bool(((y.double() - ref).abs() <= (2.0 ** -8 + 2.0 ** -18) * ref.abs() + 1e-30).all())
