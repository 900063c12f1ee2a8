"""tcgen05 GEMM numerics vs fp32 PyTorch for every operand-major combination used by a linear layer."""
import pytest
import torch

from realhf_b200.ops import gemm as G

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _ref(a, b, a_mn, b_mn):
    A = a.float().t() if a_mn else a.float()
    B = b.float() if b_mn else b.float().t()
    return A @ B


@pytest.mark.parametrize("bn", [0, 256, 128, 64, 32])
@pytest.mark.parametrize("shape", [(128, 256, 64), (256, 512, 256), (1000, 1032, 520), (4096, 4096, 4096), (77, 40, 72)])
def test_gemm_kmajor(shape, bn):
    M, N, K = shape
    torch.manual_seed(0)
    a = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    b = torch.randn(N, K, device=DEV, dtype=torch.bfloat16)
    c = G.gemm(a, b, bn=bn)
    ref = _ref(a, b, False, False)
    torch.testing.assert_close(c.float(), ref, atol=K ** 0.5 * 0.05, rtol=2e-2)


@pytest.mark.parametrize("majors", [(False, True), (True, True), (True, False)])
@pytest.mark.parametrize("shape", [(128, 256, 64), (512, 384, 256), (1000, 1032, 520), (4096, 11008, 2048)])
def test_gemm_mn_major(shape, majors):
    M, N, K = shape
    a_mn, b_mn = majors
    torch.manual_seed(1)
    a = torch.randn((K, M) if a_mn else (M, K), device=DEV, dtype=torch.bfloat16)
    b = torch.randn((K, N) if b_mn else (N, K), device=DEV, dtype=torch.bfloat16)
    c = G.gemm(a, b, a_mn=a_mn, b_mn=b_mn)
    ref = _ref(a, b, a_mn, b_mn)
    torch.testing.assert_close(c.float(), ref, atol=K ** 0.5 * 0.05, rtol=2e-2)


def test_gemm_bias_fp32_out_accumulate_fp16():
    torch.manual_seed(2)
    M, N, K = 300, 520, 264
    a = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    b = torch.randn(N, K, device=DEV, dtype=torch.bfloat16)
    bias = torch.randn(N, device=DEV, dtype=torch.bfloat16)
    c = G.gemm(a, b, bias=bias)
    torch.testing.assert_close(c.float(), _ref(a, b, False, False) + bias.float(), atol=1.0, rtol=2e-2)
    acc = torch.randn(M, N, device=DEV, dtype=torch.float32)
    acc0 = acc.clone()
    G.gemm(a, b, out=acc, accumulate=True)
    torch.testing.assert_close(acc, acc0 + _ref(a, b, False, False), atol=1e-2, rtol=1e-3)
    ah, bh = a.half(), b.half()
    ch = G.gemm(ah, bh)
    torch.testing.assert_close(ch.float(), _ref(ah, bh, False, False), atol=0.5, rtol=1e-2)


def test_linear_autograd_matches_torch():
    torch.manual_seed(3)
    T, K, N = 777, 512, 1024
    x = torch.randn(T, K, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    w = (torch.randn(N, K, device=DEV) * 0.05).to(torch.bfloat16).requires_grad_(True)
    bias = torch.randn(N, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    y = G.linear(x, w, bias)
    dy = torch.randn_like(y)
    y.backward(dy)
    xr, wr, br = (t.detach().float().requires_grad_(True) for t in (x, w, bias))
    yr = torch.nn.functional.linear(xr, wr, br)
    yr.backward(dy.float())
    torch.testing.assert_close(y.float(), yr, atol=0.1, rtol=2e-2)
    torch.testing.assert_close(x.grad.float(), xr.grad, atol=0.1, rtol=2e-2)
    torch.testing.assert_close(w.grad.float(), wr.grad, atol=0.5, rtol=2e-2)
    torch.testing.assert_close(bias.grad.float(), br.grad, atol=0.5, rtol=2e-2)


def test_gemm_strided_operand():
    torch.manual_seed(4)
    big = torch.randn(640, 3 * 512, device=DEV, dtype=torch.bfloat16)
    a = big[:, 512:1024]  # row pitch 1536, offset 1024 bytes
    b = torch.randn(256, 512, device=DEV, dtype=torch.bfloat16)
    c = G.gemm(a, b)
    torch.testing.assert_close(c.float(), a.float() @ b.float().t(), atol=1.5, rtol=2e-2)


@pytest.mark.parametrize("shape", [(128, 4096, 4096), (64, 12288, 4096), (128, 22016, 4096), (1, 4096, 512), (100, 11008, 1024),
                                   (128, 32000, 4096), (7, 264, 136)])
def test_gemm_small_m(shape):
    """M <= 128 and K-major operands: the stream-K kernel, and the plain tiles that `mc` other than 2 asks for."""
    M, N, K = shape
    torch.manual_seed(5)
    a = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    b = torch.randn(N, K, device=DEV, dtype=torch.bfloat16)
    for _ in range(3):  # repeated launches exercise barrier phase carry-over
        c = G.gemm(a, b)
    ref = a.float() @ b.float().t()
    torch.testing.assert_close(c.float(), ref, atol=K ** 0.5 * 0.05, rtol=2e-2)
    for mc in (0, 1):
        torch.testing.assert_close(G.gemm(a, b, mc=mc).float(), ref, atol=K ** 0.5 * 0.05, rtol=2e-2)


@pytest.mark.parametrize("shape", [(128, 4096, 4096), (64, 4096, 11008), (17, 12288, 4096), (128, 22016, 4096), (1, 32000, 4096),
                                   (100, 1000, 520), (128, 256, 256), (8, 4104, 264)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_streamk_decode_gemm(shape, dtype):
    """Stream-K small-M GEMM vs fp32 reference; repeated calls check that the flags self-reset."""
    M, N, K = shape
    torch.manual_seed(M + N + K)
    a = (torch.randn(M, K, device=DEV) * 0.5).to(dtype)
    b = (torch.randn(N, K, device=DEV) * 0.05).to(dtype)
    bias = torch.randn(N, device=DEV).to(dtype)
    ref = a.float() @ b.float().t()
    for bn, split in ((0, 0), (128, 0), (48, 0), (96, 1), (256, 3), (32, 2)):
        for it in range(3):
            y = G.gemm_streamk(a, b, bn=bn, split=split)
        torch.testing.assert_close(y.float(), ref, atol=2e-2 * (K / 4096) ** 0.5 + 1e-2, rtol=2e-2)
    yb = G.gemm_streamk(a, b, bias=bias)
    torch.testing.assert_close(yb.float(), ref + bias.float(), atol=2e-2 * (K / 4096) ** 0.5 + 2e-2, rtol=2e-2)
    y32 = G.gemm_streamk(a, b, out_dtype=torch.float32)
    torch.testing.assert_close(y32, ref, atol=5e-3 * (K / 4096) ** 0.5 + 1e-3, rtol=1e-3)
    ws, flags = G.streamk_workspace(a.device)
    assert int(flags.abs().sum()) == 0
    # the default route for small M is the stream-K kernel, also under CUDA graph capture
    g = torch.cuda.CUDAGraph()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        G.gemm(a, b)
        with torch.cuda.graph(g):
            yg = G.gemm(a, b)
    torch.cuda.current_stream().wait_stream(s)
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    torch.testing.assert_close(yg.float(), ref, atol=2e-2 * (K / 4096) ** 0.5 + 1e-2, rtol=2e-2)


@pytest.mark.parametrize("majors", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("shape", [(256, 256, 64), (512, 384, 256), (1000, 1032, 520), (4096, 4096, 1024), (2048, 11008, 512), (304, 128, 136)])
@pytest.mark.parametrize("bn", [0, 128, 256])
def test_gemm_cta_pair(shape, majors, bn):
    """cta_group::2 kernel (256 x BN tiles on SM pairs), every operand-major combination, ragged edges."""
    M, N, K = shape
    a_mn, b_mn = majors
    torch.manual_seed(3)
    a = torch.randn((K, M) if a_mn else (M, K), device=DEV, dtype=torch.bfloat16)
    b = torch.randn((K, N) if b_mn else (N, K), device=DEV, dtype=torch.bfloat16)
    ref = _ref(a, b, a_mn, b_mn)
    for _ in range(2):
        c = G.gemm(a, b, a_mn=a_mn, b_mn=b_mn, bn=bn, mc=2)
    torch.testing.assert_close(c.float(), ref, atol=K ** 0.5 * 0.05, rtol=2e-2)


def test_gemm_cta_pair_epilogues():
    torch.manual_seed(4)
    M, N, K = 600, 520, 264
    a = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    b = torch.randn(N, K, device=DEV, dtype=torch.bfloat16)
    bias = torch.randn(N, device=DEV, dtype=torch.bfloat16)
    c = G.gemm(a, b, bias=bias, mc=2)
    torch.testing.assert_close(c.float(), _ref(a, b, False, False) + bias.float(), atol=1.0, rtol=2e-2)
    acc = torch.randn(M, N, device=DEV, dtype=torch.float32)
    acc0 = acc.clone()
    G.gemm(a, b, out=acc, accumulate=True, mc=2)
    torch.testing.assert_close(acc, acc0 + _ref(a, b, False, False), atol=1e-2, rtol=1e-3)
    ah, bh = a.half(), b.half()
    torch.testing.assert_close(G.gemm(ah, bh, mc=2).float(), _ref(ah, bh, False, False), atol=0.5, rtol=1e-2)


def test_linear_wgrad_accumulates_into_flat_grad_view():
    """With a same-dtype flat gradient buffer the wgrad GEMM adds into the parameter's .grad view (two micro-batches)."""
    torch.manual_seed(5)
    T, K, N = 512, 256, 384
    w = (torch.randn(N, K, device=DEV) * 0.05).to(torch.bfloat16).requires_grad_(True)
    flat = torch.zeros(N * K, device=DEV, dtype=torch.bfloat16)
    w.grad = flat.view(N, K)
    w._grad_in_flat_buffer = True
    ref = torch.zeros(N, K, device=DEV)
    for _ in range(2):
        x = torch.randn(T, K, device=DEV, dtype=torch.bfloat16)
        dy = torch.randn(T, N, device=DEV, dtype=torch.bfloat16) * 0.1
        G.linear(x, w).backward(dy)
        ref += dy.float().t() @ x.float()
    assert w.grad.data_ptr() == flat.data_ptr()
    torch.testing.assert_close(flat.view(N, K).float(), ref, atol=0.2, rtol=3e-2)


@pytest.mark.parametrize("counts", [[130, 0, 257, 64, 5, 1024], [8, 8, 8, 8], [0, 0, 300, 0], [513]])
def test_grouped_gemm_moe(counts):
    """One-launch grouped GEMM over expert row groups (empty and ragged groups) incl. its backward."""
    torch.manual_seed(7)
    E, K, N = len(counts), 256, 384
    M = sum(counts)
    x = (torch.randn(M, K, device=DEV) * 0.5).to(torch.bfloat16).requires_grad_(True)
    w = (torch.randn(E, N, K, device=DEV) * 0.05).to(torch.bfloat16).requires_grad_(True)
    off = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), device=DEV, dtype=torch.int32)
    y = G.grouped_linear(x, w, off)
    dy = (torch.randn(M, N, device=DEV) * 0.1).to(torch.bfloat16)
    y.backward(dy)
    xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    outs, o = [], 0
    for e, n in enumerate(counts):
        outs.append(xr[o:o + n] @ wr[e].t())
        o += n
    yr = torch.cat(outs)
    yr.backward(dy.float())
    torch.testing.assert_close(y.float(), yr, atol=0.1, rtol=2e-2)
    torch.testing.assert_close(x.grad.float(), xr.grad, atol=0.05, rtol=3e-2)
    torch.testing.assert_close(w.grad.float(), wr.grad, atol=0.3, rtol=3e-2)


@pytest.mark.parametrize("counts,M,N", [([300, 0, 64, 1000, 5, 77], 256, 512), ([4096, 4096], 1024, 384), ([0, 0, 9], 128, 128)])
def test_grouped_wgrad_single_launch(counts, M, N):
    from realhf_b200.ops import gemm as G
    torch.manual_seed(0)
    T, ng = sum(counts), len(counts)
    offsets = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32, device="cuda")
    dy = torch.randn(T, M, device="cuda", dtype=torch.bfloat16)
    x = torch.randn(T, N, device="cuda", dtype=torch.bfloat16)
    ref = G.grouped_wgrad_ref(dy, x, offsets, ng)
    out = G.grouped_wgrad(dy, x, offsets, ng)
    torch.testing.assert_close(out.float(), ref, atol=2e-2 * max(counts) ** 0.5, rtol=2e-2)
    acc = torch.ones(ng, M, N, device="cuda", dtype=torch.float32)
    G.grouped_wgrad(dy, x, offsets, ng, out=acc, accumulate=True)
    torch.testing.assert_close(acc, ref + 1.0, atol=2e-2 * max(counts) ** 0.5, rtol=2e-2)


@pytest.mark.parametrize("shape", [(300, 1024, 512), (4096, 4096, 11008), (129, 512, 136)])
@pytest.mark.parametrize("kind", ["silu", "gelu_pytorch_tanh"])
def test_gated_linear_fused_epilogue_matches_reference(shape, kind):
    """SwiGLU / GeGLU in the epilogue of the CTA-pair GEMM (gate rows from CTA 0, up rows from CTA 1 of the fused weight):
    forward equals gated_act(x @ W^T), backward (through the saved raw projections) equals autograd of the fp32 reference."""
    from realhf_b200.ops import functional as OF
    from realhf_b200.ops import gemm as G
    OF.set_gemm_impl(G.linear)
    M, K, F_ = shape
    torch.manual_seed(0)
    x = (torch.randn(M, K, device="cuda") * 0.5).to(torch.bfloat16).requires_grad_(True)
    w = (torch.randn(2 * F_, K, device="cuda") * (1.0 / K ** 0.5)).to(torch.bfloat16).requires_grad_(True)
    assert G.gated_linear_supported(x, w)
    a = OF.gated_linear(x, w, kind)
    da = torch.randn_like(a)
    a.backward(da)
    xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    gu = (xr @ wr.t()).to(torch.bfloat16).float() + 0 * (xr @ wr.t())  # the projection is rounded to bf16 before the activation
    gur = xr @ wr.t()
    ar = OF.gated_act_ref(gur, kind)
    ar.backward(da.float())
    torch.testing.assert_close(a.float(), ar, atol=3e-2, rtol=3e-2)
    torch.testing.assert_close(x.grad.float(), xr.grad, atol=6e-2, rtol=6e-2)
    torch.testing.assert_close(w.grad.float(), wr.grad, atol=0.25 if M > 1000 else 8e-2, rtol=6e-2)
    # inference: no raw projection is written
    with torch.no_grad():
        a2 = OF.gated_linear(x.detach(), w.detach(), kind)
    torch.testing.assert_close(a2, a.detach())


def test_grouped_wgrad_tail_rows_of_other_groups():
    """K blocks that reach into the next group's rows, past the last group and past the tensor, with NaN in one group and in the rows of no group: a
    group's gradient is that of its own rows.  Products of 16-bit numbers are exact in fp32; 2^-8 for the rounded result, 2^-20 of the summed magnitudes."""
    from realhf_b200.ops import gemm as G
    torch.manual_seed(1)
    counts, lead, M, N = [1, 63, 64, 65, 127, 0, 5, 130, 64], 7, 264, 136
    off = torch.tensor([lead] + [lead + int(c) for c in torch.tensor(counts).cumsum(0)], dtype=torch.int32, device="cuda")
    T = int(off[-1]) + 3
    dy, x = torch.randn(T, M, device="cuda").to(torch.bfloat16), torch.randn(T, N, device="cuda").to(torch.bfloat16)
    dy[:lead], x[int(off[-1]):] = float("nan"), float("nan")
    dy[int(off[3]): int(off[4])] = float("nan")
    for acc in (False, True):
        out = torch.ones(len(counts), M, N, device="cuda", dtype=torch.bfloat16 if acc else torch.float32)
        G.grouped_wgrad(dy, x, off, len(counts), out=out, accumulate=acc)
        for g in range(len(counts)):
            if g == 3:
                assert out[g].isnan().all()
                continue
            a, b = dy[int(off[g]): int(off[g + 1])].double(), x[int(off[g]): int(off[g + 1])].double()
            ref, mag = a.T @ b + float(acc), a.abs().T @ b.abs() + float(acc)
            assert ((out[g].double() - ref).abs() <= (2.0 ** -8 if acc else 0.0) * ref.abs() + 2.0 ** -20 * mag + 1e-6).all(), g
    assert torch.equal(G.grouped_wgrad(dy[:0], x[:0], torch.zeros(3, dtype=torch.int32, device="cuda"), 2), torch.zeros(2, M, N, device="cuda", dtype=torch.bfloat16))


@pytest.mark.parametrize("M,N,K", [(1, 4096, 4096), (7, 2040, 2048), (16, 6144, 4096), (33, 4104, 4168), (64, 8184, 2048), (128, 4096, 11008), (128, 2040, 136)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_small_products_with_parts_of_k(M, N, K, dtype):
    """Few rows, narrow outputs: K cut into parts that are merged in a cluster or through the workspace; ragged rows, columns and parts.  Products of 16-bit numbers are
    exact in fp32: 2^-20 of the summed magnitudes for the sums, 2^-8 (bf16; fp16 2^-11) of the value for a rounded result; the same every time."""
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a, b = (torch.randn(n, K, device="cuda", generator=g).to(dtype) for n in (M, N))
    bias = torch.randn(N, device="cuda", generator=g).to(dtype)
    ref, mag = a.double() @ b.double().T, a.double().abs() @ b.double().abs().T
    y = G.gemm_streamk(a, b, out_dtype=torch.float32)
    assert ((y.double() - ref).abs() <= 2.0 ** -20 * mag).all()
    assert all(torch.equal(G.gemm_streamk(a, b, out_dtype=torch.float32), y) for _ in range(3))
    z = G.gemm_streamk(a, b, bias=bias)
    want = ref + bias.double()
    assert ((z.double() - want).abs() <= 2.0 ** -20 * mag + want.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11)).all()


@pytest.mark.parametrize("out_dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N,K,shift", [(129, 136, 64, 0), (300, 520, 192, 0), (257, 264, 128, 1), (8, 72, 200, 0), (640, 40, 72, 3)])
def test_gemm_accumulates_into_ragged_outputs(out_dt, M, N, K, shift):
    """C += A B through the staged epilogue: ragged rows and columns, an output that starts off every vector boundary, untouched surroundings.  Bound: one
    rounding of the result and 2^-20 of the summed magnitudes."""
    from realhf_b200.ops import gemm as G
    torch.manual_seed(M + N)
    a, b = torch.randn(K, M, device="cuda").to(torch.bfloat16), torch.randn(K, N, device="cuda").to(torch.bfloat16)
    if M % 8 or N % 8:
        a = torch.randn(K, (M + 7) // 8 * 8, device="cuda").to(torch.bfloat16)[:, :M]
    buf = torch.randn(M + 2, N + 8, device="cuda").to(out_dt)
    before = buf.clone()
    out = buf[1:M + 1, shift:shift + N]
    G.gemm(a, b, out=out, a_mn=True, b_mn=True, accumulate=True)
    ref = before[1:M + 1, shift:shift + N].double() + a.double().T @ b.double()
    mag = before[1:M + 1, shift:shift + N].double().abs() + a.double().abs().T @ b.double().abs()
    assert ((out.double() - ref).abs() <= (2.0 ** -8 if out_dt == torch.bfloat16 else 0.0) * ref.abs() + 2.0 ** -20 * mag).all()
    buf[1:M + 1, shift:shift + N] = before[1:M + 1, shift:shift + N]
    assert torch.equal(buf, before)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K,shift", [(288, 256, 64, 0), (300, 512, 128, 8), (1000, 776, 72, 0), (257, 264, 512, 0), (512, 256, 64, 4)])
def test_gemm_cta_pair_output_edges(M, N, K, shift, dtype):
    """16-bit outputs of the CTA-pair kernel: whole 32 x 64 pieces leave in their own type, the rest through fp32 staging (last rows and columns, rows off a
    16-byte boundary); what surrounds the output stays as it is.  Bound: fp32 sums of K products (2^-22 of their magnitudes) and one rounding."""
    torch.manual_seed(M + N)
    a, b = torch.randn(M, K, device=DEV).to(dtype), torch.randn(N, K, device=DEV).to(dtype)
    wide = torch.full((M + 2, N + 24), 7.0, device=DEV, dtype=dtype)
    out = wide[1:M + 1, 8 + shift:8 + shift + N]
    G.gemm(a, b, out=out, mc=2)
    ref, mag = a.double() @ b.double().t(), a.double().abs() @ b.double().abs().t()
    eps = 2.0 ** (-9 if dtype == torch.bfloat16 else -12)
    assert ((out.double() - ref).abs() <= 2 * eps * ref.abs() + 2.0 ** -22 * mag + 2.0 ** -24).all()
    out.fill_(7.0)
    assert (wide == 7.0).all()


@pytest.mark.parametrize("M,N,K,bn,split", [(80, 512, 8192, 64, 16), (128, 384, 8192, 48, 16), (112, 512, 8192, 64, 16)])
def test_few_row_layout_fills_its_round_trips(M, N, K, bn, split):
    """The reduction of a tile's parts takes eight of them at a time: the layout that is chosen must not be behind one whose parts fill those eights (cold weights, captured loops
    in turn, the best of each; it was 5 .. 6 % behind while every part had a cost of its own)."""
    x = torch.randn(M, K, device="cuda").bfloat16()
    ws = [torch.randn(N, K, device="cuda").bfloat16() * 0.02 for _ in range(30)]

    def loop(**layout):
        graph = torch.cuda.CUDAGraph()
        G.gemm_streamk(x, ws[0], **layout)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):
            for w in ws:
                G.gemm_streamk(x, w, **layout)
        return graph

    def time(graph):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        graph.replay()
        b.record()
        b.synchronize()
        return a.elapsed_time(b)
    chosen, full = loop(), loop(bn=bn, split=split)
    pairs = [(time(chosen), time(full)) for _ in range(25)]
    assert min(t for t, _ in pairs) <= 1.03 * min(t for _, t in pairs)
