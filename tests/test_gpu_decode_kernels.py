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


@pytest.mark.parametrize("norm", [0, 1])
@pytest.mark.parametrize("M", range(1, 9))
def test_w4_stream_cuts_every_k_to_fit_shared_memory(M, norm):
    """The host's cut of a call, without a GPU: whatever K, rows, columns and SMs, its launches fit the 220 KB of a CTA."""
    import ctypes
    from summa_b200.ops import native
    passes, seen = ctypes.c_int(0), set()
    for K in list(range(128, 131072, 128)) + [196608, 262144]:
        for N, sms in ((4, 148), (4096, 148), (152064, 148), (28672, 20)):
            got = native.lib().sb_w4_stream_smem(M, N, K, norm, sms, ctypes.byref(passes))
            assert 0 < got <= 220 * 1024 and passes.value >= 1, (K, N, sms)
            seen.add(passes.value)
    assert 1 in seen and 2 in seen


@gpu
@pytest.mark.parametrize("M,K,N", [
    (1, 28032, 20), (1, 28672, 40), (2, 28672, 24), (1, 53376, 12), (1, 86016, 8),  # one row around the last K of one pass
    (1, 128, 4), (2, 256, 20), (3, 2048, 16), (1, 2176, 132), (8, 1920, 68),        # one group; fewer and more than 16 groups; ragged tiles
    (2, 14464, 36), (1, 20480, 28), (4, 9088, 44), (8, 4352, 2400),                 # K in passes / the last that fits one pass
    (8, 4736, 52), (5, 14336, 40)])                                                 # rows 5..8 beyond one pass: the other kernel
@pytest.mark.parametrize("spread", [0, 24])
def test_w4_projection_against_fp64(M, K, N, spread):
    """x spreads over 2^-spread .. 1. Exact products, fp32 sums (2^-18 of the terms' sum) and one rounding to bf16."""
    import ctypes
    from summa_b200 import ops
    from summa_b200.ops import native
    packed, scales, k8, wq = _w4(K, N, M + K + N)
    x = (torch.randn(M, K, device="cuda") * torch.exp2(-spread * torch.rand(M, K, device="cuda"))).to(torch.bfloat16)
    res = torch.randn(M, N, device="cuda").to(torch.bfloat16)
    ref = x.double() @ wq
    passes = ctypes.c_int(0)
    native.lib().sb_w4_stream_smem(M, N, K, 0, 148, ctypes.byref(passes))
    # rows 5..8 beyond one pass: that kernel rounds the weights to bf16
    slack = (2.0 ** -9 if M > 4 and passes.value > 1 else 2.0 ** -18) * (x.double().abs() @ wq.abs())
    for got, want in ((ops.int4_gemv(x, packed, scales, None, k8), ref), (ops.int4_gemv(x, packed, scales, res, k8), ref + res.double())):
        assert bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + slack + 1e-30).all())


@gpu
@pytest.mark.parametrize("M,N", [(1, 36), (2, 16), (4, 52), (8, 20)])
@pytest.mark.parametrize("big", [12, 40])
def test_w4_projection_keeps_small_elements_beside_an_outlier(M, N, big):
    """One element of a scale group is 2^big, its weights are zero: the columns are what the other elements make of them, at
    the same precision (exact products, fp32 sums: 2^-18 of the terms' sum, one rounding to bf16)."""
    from summa_b200 import ops
    from summa_b200.ops import reference
    torch.manual_seed(M + N)
    w = torch.randn(512, N) * 0.05
    w[5::128] = 0
    packed, scales = reference.quantize_int4_g128(w)
    wq = reference.dequantize_int4_g128(packed, scales).double().cuda()
    assert float(wq[5::128].abs().max()) == 0
    packed, scales = packed.cuda(), scales.cuda()
    x = torch.randn(M, 512, device="cuda")
    x[:, 5::128] = 2.0 ** big
    x = x.to(torch.bfloat16)
    ref = x.double() @ wq
    got = ops.int4_gemv(x, packed, scales, None, reference.repack_int4_k8(packed))
    assert bool(((got.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -18 * (x.double().abs() @ wq.abs())).all())


@gpu
@pytest.mark.parametrize("M", [2, 4, 8])
def test_w4_projection_keeps_nan_and_inf_in_their_row(M):
    """An infinite element makes a column infinite, of the sign of its weight, or NaN where that is zero, and a NaN makes the row
    NaN, as IEEE sums do; the other rows do not see either."""
    from summa_b200 import ops
    packed, scales, k8, wq = _w4(512, 40, 3)
    x = torch.randn(M, 512, device="cuda").to(torch.bfloat16)
    clean = ops.int4_gemv(x, packed, scales, None, k8)
    nan = 0 if M == 2 else 2
    x[1, 7], x[nan, 300] = float("inf"), float("nan")
    got = ops.int4_gemv(x, packed, scales, None, k8)
    torch.testing.assert_close(got[1].float(), float("inf") * wq[7].float(), rtol=0, atol=0, equal_nan=True)
    assert bool((wq[7] == 0).any()) and bool(got[nan].isnan().all())
    for m in set(range(M)) - {1, nan}:
        assert torch.equal(got[m], clean[m])


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
@pytest.mark.parametrize("M", [2, 7])
def test_w4_layer_marks_its_weights_settled_only_once_they_are(M, monkeypatch):
    """The first call of a layer repacks (and aligns) right in front of the kernel, which must not read the weights early then;
    later calls may. A raw call never may unless its caller says so, and a copy made for the call never is."""
    from summa_b200 import ops
    from summa_b200.models.quantized import QuantLinear
    from summa_b200.ops import cuda_ops
    packed, scales, k8, wq = _w4(512, 32, 7)
    off = torch.empty(scales.numel() + 1, device="cuda", dtype=scales.dtype)[1:].view_as(scales).copy_(scales)
    x = torch.randn(M, 512, device="cuda").to(torch.bfloat16)
    flags, call = [], cuda_ops.N.call
    monkeypatch.setattr(cuda_ops.N, "call", lambda name, *a: (flags.append(a[-2]) if name == "sb_w4_gemv_cluster" else None, call(name, *a))[1])
    layer, unaligned = QuantLinear(packed, scales), QuantLinear(packed, off)
    assert unaligned.scales.data_ptr() % 8
    want = [ops.int4_gemv(x, packed, scales, None, k8), ops.int4_gemv(x, packed, off, None, k8, static_w=True),
            ops.int4_gemv(x, packed, scales, None, k8, static_w=True)]
    got = [m(x) for m in (layer, layer, unaligned, unaligned)]
    # five to eight rows of unsettled weights go through the entry that has no such flag
    assert flags == ([0, 0, 1, 0, 1, 0, 1] if M <= 4 else [1, 1, 1])
    assert all(torch.equal(t, want[0]) for t in want + got)


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


def _hybrid(state_dim, taps, layers=3, hidden=256):
    from summa_b200 import mal
    src = f"""
attention a {{ num_heads: {hidden // 128}  bias: false }}
ssm s {{ state_dim: {state_dim}  conv_kernel: {taps}  expand: 2 }}
ffn f {{ hidden_dim: 512  activation: swiglu  bias: false }}
block ab {{ attention: a  ffn: f  norm: rmsnorm {{ eps: 1e-5 }}  norm_position: pre  residual: true }}
block mb {{ ssm: s  ffn: f  norm: rmsnorm {{ eps: 1e-5 }}  norm_position: pre  residual: true }}
model t {{ vocab_size: 512  max_seq_len: 64  hidden_size: {hidden}  num_layers: {layers}  block: ab  pattern: [mb, ab, mb] }}
"""
    return mal.parse_mal(src)


@gpu
@pytest.mark.parametrize("B,state_dim,taps", [(1, 8, 2), (3, 16, 4), (2, 32, 3), (8, 64, 4), (9, 128, 4), (1, 256, 4)])
def test_mamba_decode_step_matches_the_general_path(B, state_dim, taps):
    """Output and in-place states of the step against the mixer's own forward over one token (scan kernel). Both round at the
    same places; fp32 sums in another order move single bf16 results by one step (2^-8)."""
    from summa_b200.models import Transformer
    from summa_b200.ops import cuda_ops
    torch.manual_seed(state_dim + taps)
    with torch.device("cuda"):
        model = Transformer(_hybrid(state_dim, taps), init_std=0.1)
    model.prepare_inference(torch.bfloat16)
    mx = model.layers[0].ssm
    with torch.no_grad():
        mx.a_log.copy_(torch.rand_like(mx.a_log) * 3 - 1)
    assert cuda_ops.mamba_decode_usable(mx)
    x = torch.randn(B, 256, device="cuda").to(torch.bfloat16)
    st = mx.make_state(B, "cuda", torch.bfloat16)
    st.conv.normal_()
    st.h.normal_()
    conv, h = st.conv.clone(), st.h.clone()
    with torch.no_grad():
        want = mx(x.view(B, 1, 256), st).view(B, 256)
        got = cuda_ops.decode_linear(cuda_ops.mamba_decode_step(mx, cuda_ops.decode_linear(x, mx.in_proj.weight), conv, h), mx.out_proj.weight)
    assert torch.equal(conv, st.conv.view_as(conv)) or float((conv.float() - st.conv.float()).abs().max()) <= 2.0 ** -7 * float(st.conv.float().abs().max())
    for a, b in ((h, st.h), (got, want)):
        assert float((a.double() - b.double()).norm() / b.double().norm()) <= 2.0 ** -7


@gpu
@pytest.mark.parametrize("B,C,N", [(1, 8, 8), (3, 72, 16), (2, 40, 64), (1, 3072, 128), (2, 24, 256)])
def test_mamba_scan_step_walks_the_prefill_recurrence(B, C, N):
    """One token through the decode step and through the prefill scan from the same state, fast-decaying states included
    (A = -exp(a_log) down to -3000): the new states are the same bits."""
    from summa_b200.ops import cuda_ops, native
    torch.manual_seed(C + N)
    u, delta, z, Bm, Cm = [torch.randn(B, 1, n, device="cuda").to(torch.bfloat16) for n in (C, C, C, N, N)]
    delta = (delta - 4).to(torch.bfloat16)
    a_log, D, h0 = torch.rand(C, N, device="cuda") * 9 - 1, torch.randn(C, device="cuda"), torch.randn(B, C, N, device="cuda")
    with torch.no_grad():
        _, want = cuda_ops.selective_scan_log(u, delta, a_log, Bm, Cm, D, h0, True)
    h, out = h0.clone(), torch.empty(B, C, device="cuda", dtype=torch.bfloat16)
    native.call("sb_mamba_scan_step", u.data_ptr(), delta.data_ptr(), a_log.data_ptr(), Bm.data_ptr(), Cm.data_ptr(), N, D.data_ptr(),
                z.data_ptr(), C, h.data_ptr(), out.data_ptr(), B, C, N, native.stream())
    assert torch.equal(h, want)


@gpu
@pytest.mark.parametrize("B", [1, 5, 9])
def test_hybrid_graph_decode_against_eager(B):
    """The captured step of a model with recurrent blocks: states after one token, repeated and continued requests."""
    from summa_b200.models import Transformer
    from summa_b200.models.engine import InferenceEngine
    from summa_b200.ops import native
    torch.manual_seed(B)
    with torch.device("cuda"):
        model = Transformer(_hybrid(16, 4), init_std=0.1)
    model.prepare_inference(torch.bfloat16)
    prompt = torch.randint(0, 512, (B, 7), device="cuda")

    def after(use_graph, steps):
        eng = InferenceEngine(model)
        eng.use_graph = use_graph
        eng.reset(B, 40)
        first = eng.prefill(prompt)
        eng.decode(first, steps)
        assert (eng._graph is not None) == use_graph
        return eng
    g, e = after(True, 1), after(False, 1)
    for a, b in zip(g.state.layers, e.state.layers):
        for k in vars(b):
            u, v = getattr(a, k), getattr(b, k)
            if not torch.is_tensor(u):
                assert u == v
                continue
            assert u.dtype == v.dtype and float((u.double() - v.double()).norm() / v.double().norm().clamp_min(1e-9)) <= 2e-2
    # the same request again on the kept graph, and in two halves: identical
    eng = after(True, 6)
    assert eng._graph.graph is not None
    runs = []
    for split in ((6,), (6,), (2, 4)):
        eng.reset(B, 40)
        tok, out = eng.prefill(prompt), []
        for n in split:
            out.append(eng.decode(tok, n))
            tok = out[-1][:, -1:]
        runs.append((torch.cat(out, 1), [vars(s).copy() for s in eng.state.layers]))
    for toks, states in runs[1:]:
        assert torch.equal(toks, runs[0][0])
        for a, b in zip(states, runs[0][1]):
            assert "h" not in a or torch.equal(a["h"], b["h"])
    assert native.read_error_flag() == 0


@gpu
@pytest.mark.parametrize("short", [False, True])
def test_decode_capture_empties_the_cache_only_when_memory_is_short(short, monkeypatch):
    """Whole numbers: both ways of capturing give the same tokens as the eager decode."""
    from summa_b200.models import Transformer
    from summa_b200.models.engine import InferenceEngine
    torch.manual_seed(3)
    with torch.device("cuda"):
        model = Transformer(_hybrid(16, 4), init_std=0.1)
    model.prepare_inference(torch.bfloat16)
    eng = InferenceEngine(model)
    eng.reset(2, 24)
    prompt = torch.randint(0, 512, (2, 7), device="cuda")
    first = eng.prefill(prompt)
    free, calls, empty_cache = 0 if short else 1 << 40, [], torch.cuda.empty_cache
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (free, 1 << 40))
    monkeypatch.setattr(torch.cuda, "empty_cache", lambda: (calls.append(1), empty_cache()))
    tokens = eng.decode(first, 6)
    assert eng._graph is not None and eng._graph.graph is not None and len(calls) == int(short)
    plain = InferenceEngine(model)
    plain.use_graph = False
    plain.reset(2, 24)
    again = plain.prefill(prompt)
    assert torch.equal(first, again) and torch.equal(tokens, plain.decode(again, 6))


@gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,vocab,ld,off", [(1, 1, 8, 0), (3, 32000, 32064, 0), (2, 8191, 8192, 0), (2, 1003, 1003, 0), (2, 50, 64, 1)])
def test_argmax_rows_vector_and_scalar(dtype, rows, vocab, ld, off):
    """Aligned and unaligned rows against torch (lowest index among equals: values are drawn from few)."""
    from summa_b200 import ops
    torch.manual_seed(vocab)
    buf = torch.randint(-9, 9, (rows * ld + off,), device="cuda").to(dtype)
    x = buf[off:].view(rows, ld)[:, :vocab]
    want = torch.tensor([int((r == r.max()).nonzero()[0]) for r in x.float().cpu()])
    assert torch.equal(ops.argmax(x).cpu(), want)
    x[0].fill_(float("-inf"))
    assert int(ops.argmax(x)[0]) == 0


@pytest.mark.parametrize("ctas,blocks,one", [
    (148, 1, 0), (149, 1, 1), (512, 2, 1), (512, 6, 1), (512, 7, 0), (512, 33, 0), (296, 9, 0), (296, 6, 1), (304, 4, 1), (320, 33, 1),
    (384, 17, 1), (444, 33, 1), (445, 33, 0), (768, 17, 1), (1024, 17, 0), (1024, 5, 1)])
def test_decode_attention_form(ctas, blocks, one):
    """The rule on a GPU of 148 SMs, at shapes where the two forms were timed against each other."""
    from summa_b200.ops import native
    import ctypes
    f = native.lib().sb_attention_decode_one_stage
    f.argtypes = [ctypes.c_long, ctypes.c_int, ctypes.c_int]
    assert f(ctas, blocks, 148) == one


@gpu
@pytest.mark.parametrize("B,Hq,Hkv,Sk", [(38, 16, 8, 1), (40, 32, 8, 127), (64, 8, 8, 129), (75, 12, 4, 300), (37, 64, 8, 513), (5, 8, 8, 140),
                                         (2, 16, 8, 2100), (16, 16, 8, 2100), (64, 8, 8, 1100), (37, 8, 8, 1100)])
def test_decode_attention_many_sequences(B, Hq, Hkv, Sk):
    """Both forms of the kernel (one stage and three), each with split keys and with whole ones, where it writes the output
    itself; (5, 8, 8, 140) has fewer CTAs than SMs. bf16 probabilities and values: 2^-8 of the weighted sum's terms."""
    from summa_b200.ops import cuda_ops, native
    torch.manual_seed(B + Sk)
    q = torch.randn(B, 1, Hq, 128, device="cuda").to(torch.bfloat16)
    kc, vc = [torch.randn(B, Sk + 9, Hkv, 128, device="cuda").to(torch.bfloat16) for _ in range(2)]
    with torch.no_grad():
        o = cuda_ops.decode_attention(q, kc[:, :Sk], vc[:, :Sk], True, None, Sk - 1)
    k, v = [t[:, :Sk].double().repeat_interleave(Hq // Hkv, 2).transpose(1, 2) for t in (kc, vc)]
    p = torch.softmax(q.double().transpose(1, 2) @ k.transpose(-1, -2) / 128 ** 0.5, -1)
    want = (p @ v).transpose(1, 2)
    assert bool(((o.double() - want).abs() <= 2.0 ** -7 * (p @ v.abs()).transpose(1, 2) + 2.0 ** -8 * want.abs()).all())
    assert native.read_error_flag() == 0


@pytest.mark.parametrize("device", ["cpu", pytest.param("cuda", marks=gpu)])
@pytest.mark.parametrize("before", [0, 1, 3])
def test_decoding_no_tokens_leaves_the_state_alone(device, before):
    """`decode(first, 0)` on a fresh engine, after one step (no graph kept yet) and after several: nothing moves, and what
    follows is what follows without it. A negative count is an error."""
    from summa_b200.models import Transformer
    from summa_b200.models.engine import InferenceEngine
    torch.manual_seed(before)
    cfg = _hybrid(8, 2)
    with torch.device(device):
        model = Transformer(cfg, init_std=0.1)
    if device == "cuda":
        model.prepare_inference(torch.bfloat16)
    eng = InferenceEngine(model)
    eng.reset(2, 24)
    tok = eng.prefill(torch.randint(0, 512, (2, 5), device=device))
    if before:
        tok = eng.decode(tok, before)[:, -1:]
    held = [{k: v.clone() if torch.is_tensor(v) else v for k, v in vars(s).items()} for s in eng.state.layers]
    pos = eng.state.pos
    none = eng.decode(tok, 0)
    assert none.shape == (2, 0) and none.dtype == torch.long and eng.state.pos == pos
    for s, old in zip(eng.state.layers, held):
        for k, v in old.items():
            assert torch.equal(getattr(s, k), v) if torch.is_tensor(v) else getattr(s, k) == v
    with pytest.raises(ValueError):
        eng.decode(tok, -1)
    assert eng.decode(tok, 2).shape == (2, 2)


@gpu
def test_hybrid_decode_runs_hooks_and_subclasses():
    """A forward hook on a mixer or a projection sees every token, before and after a graph was kept, and may change the output; a
    subclass of the mixer or of a projection computes what its own forward says."""
    from summa_b200.models import Transformer
    from summa_b200.models.engine import InferenceEngine
    from summa_b200.models.layers import Linear, MambaMixer
    from summa_b200.ops import cuda_ops
    torch.manual_seed(5)
    with torch.device("cuda"):
        model = Transformer(_hybrid(16, 4), init_std=0.1)
    model.prepare_inference(torch.bfloat16)
    prompt, eng = torch.randint(0, 512, (2, 7), device="cuda"), InferenceEngine(model)

    def tokens(use_graph=True):
        eng.use_graph = use_graph
        eng.reset(2, 24)
        return eng.decode(eng.prefill(prompt), 4)
    plain, seen = tokens(), []
    assert eng._graph is not None
    for mod in (model.layers[0].ssm, model.layers[2].ssm.in_proj, model.final_norm):
        hook, n = mod.register_forward_hook(lambda *a: seen.append(1)), len(seen)
        assert torch.equal(tokens(), tokens(False)) and len(seen) - n == 2 * 5        # the prompt and four tokens, twice
        hook.remove()
    assert torch.equal(tokens(), plain)

    class Off(MambaMixer):
        def forward(self, x, state=None):
            return torch.zeros_like(x)

    class Double(Linear):
        def forward(self, x):
            return 2 * super().forward(x)
    assert cuda_ops.mamba_decode_usable(model.layers[0].ssm)
    model.layers[0].ssm.__class__ = Off
    assert not cuda_ops.mamba_decode_usable(model.layers[0].ssm)
    model.layers[0].ssm.__class__ = MambaMixer
    model.layers[0].ssm.out_proj.__class__ = Double
    assert not cuda_ops.mamba_decode_usable(model.layers[0].ssm)


@pytest.mark.parametrize("device", ["cpu", pytest.param("cuda", marks=gpu)])
def test_w4_layer_follows_its_buffers(device):
    """New codes and scales in a layer's buffers are what it computes with: the repacked codes and the aligned scales are made again
    (in place, so that an address held by a captured step stays good), and the call that does it is not a settled one."""
    from summa_b200.models.quantized import QuantLinear
    from summa_b200.ops import reference
    torch.manual_seed(11)
    a, b = [[t.to(device) for t in reference.quantize_int4_g128(torch.randn(256, 24) * 0.05)] for _ in range(2)]
    off = torch.empty(a[1].numel() + 1, device=device, dtype=a[1].dtype)[1:].view_as(a[1]).copy_(a[1])
    x = torch.randn(2, 256, device=device).to(torch.bfloat16)
    for scales in (a[1], off):
        layer, other = QuantLinear(a[0].clone(), scales), QuantLinear(*b)
        layer(x)
        k8 = layer.decode_operands()[0]
        assert torch.equal(k8, reference.repack_int4_k8(a[0])) and layer.decode_operands()[2]
        layer.load_state_dict(other.state_dict())
        again, s, settled = layer.decode_operands()
        assert not settled and again.data_ptr() == k8.data_ptr()
        assert torch.equal(again, reference.repack_int4_k8(b[0])) and torch.equal(s, b[1])
        assert torch.equal(layer(x), other(x)) and layer.decode_operands()[2]
        layer.scales.mul_(2)
        assert not layer.decode_operands()[2] and torch.equal(layer(x), 2 * other(x))
