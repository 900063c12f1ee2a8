"""Decode attention kernel (fused RoPE + KV append + split-KV softmax) vs the PyTorch reference."""
import pytest
import torch

from realhf_b200.ops import attention as A
from realhf_b200.ops import functional as OF
from realhf_b200.ops import lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("cfg", [(128, 32, 32, 128, 640), (3, 32, 8, 128, 2048), (5, 8, 1, 64, 700), (16, 16, 16, 64, 300),
                                 (2, 32, 4, 128, 4096)])
@pytest.mark.parametrize("rope", [None, "half", "interleaved"])
@pytest.mark.parametrize("layout", ["bshd", "bhsd"])
def test_decode_attention(cfg, rope, layout):
    B, nq, nkv, hd, S = cfg
    torch.manual_seed(0)
    if layout == "bshd":
        kc = torch.randn(B, S, nkv, hd, device=DEV, dtype=torch.bfloat16)
        vc = torch.randn(B, S, nkv, hd, device=DEV, dtype=torch.bfloat16)
    else:
        kc = torch.randn(B, nkv, S, hd, device=DEV, dtype=torch.bfloat16).permute(0, 2, 1, 3)
        vc = torch.randn(B, nkv, S, hd, device=DEV, dtype=torch.bfloat16).permute(0, 2, 1, 3)
    lens = torch.randint(0, S - 1, (B,), device=DEV, dtype=torch.int32)
    lens[0] = 0
    lens[-1] = S - 1
    qkv = torch.randn(B, (nq + 2 * nkv) * hd, device=DEV, dtype=torch.bfloat16)
    cos = sin = None
    if rope:
        cos, sin = OF.rope_tables(S, hd, 10000.0, DEV)
    kc_ref, vc_ref = kc.clone(), vc.clone()
    out = A.decode_attention(qkv, kc, vc, lens, nq, nkv, hd, None, cos, sin, hd, rope == "interleaved")
    # reference: same op through the CPU/PyTorch path
    x = qkv
    if rope:
        x = OF.rope_ref(qkv, cos, sin, lens, nq + nkv, hd, hd, rope == "interleaved")
    q = x[:, : nq * hd].reshape(B, nq, hd)
    k = x[:, nq * hd:(nq + nkv) * hd].reshape(B, nkv, hd)
    v = x[:, (nq + nkv) * hd:].reshape(B, nkv, hd)
    idx = torch.arange(B, device=DEV)
    kc_ref[idx, lens.long()] = k
    vc_ref[idx, lens.long()] = v
    ref = A.decode_attention_ref(q, kc_ref, vc_ref, lens + 1, hd ** -0.5).reshape(B, nq * hd)
    torch.testing.assert_close(out.float(), ref.float(), atol=2e-2, rtol=2e-2)
    torch.testing.assert_close(kc.float(), kc_ref.float(), atol=1e-2, rtol=1e-2)
    assert torch.equal(vc, vc_ref)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("nq,nkv,S", [(5, 5, 200), (6, 3, 131), (16, 4, 700), (8, 1, 4096), (256, 256, 70), (4, 2, 9)])
def test_decode_attention_step_edges(nq, nkv, S, hd, dtype):
    """Lengths around the 16-row steps of a warp and the 64-row steps of a CTA, few pairs (split over a cluster) and many, and cache rows that
    nobody has written yet (NaN), against float64.  Bound: the result's rounding (a relative 2^-8 for bf16's 8 significant bits, 2^-11 for fp16's 11), plus what fp32 scores and sums
    leave: scores of |s| < 64 carry 128 products of relative error 2^-24 each, so weights differ by less than 64 * 128 * 2^-24 / 16 = 3e-5."""
    edges = [0, 1, 15, 16, 17, 63, 64, 65, 127, 129, 255, 1000, 4095]
    lens = [n for n in edges if n < S]
    B = len(lens)
    g = torch.Generator(device=DEV).manual_seed(nq * 1000 + hd)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).to(dtype)  # noqa: E731
    kc, vc = rnd(B, nkv, S, hd).permute(0, 2, 1, 3), rnd(B, S, nkv, hd)
    for b, n in enumerate(lens):
        kc[b, n:] = float("nan")
        vc[b, n:] = float("nan")
    qkv = rnd(B, (nq + 2 * nkv) * hd)
    qkv[:, : nq * hd] *= 3
    q, k, v = (t.reshape(B, -1, hd).double() for t in qkv.split([nq * hd, nkv * hd, nkv * hd], 1))
    out = A.decode_attention(qkv, kc, vc, torch.tensor(lens, dtype=torch.int32, device=DEV), nq, nkv, hd).view(B, nq, hd)
    for b, n in enumerate(lens):
        assert torch.equal(kc[b, n].double(), k[b]) and torch.equal(vc[b, n].double(), v[b])
        kk, vv = (torch.repeat_interleave(t[b, : n + 1].double(), nq // nkv, 1) for t in (kc, vc))
        ref = torch.einsum("hn,nhd->hd", torch.softmax(torch.einsum("hd,nhd->hn", q[b], kk) * hd ** -0.5, -1), vv)
        rounding = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
        bound = rounding * ref.abs() + 3e-5 * vv.abs().amax(0).amax(-1).unsqueeze(-1)
        assert bool(((out[b].double() - ref).abs() <= bound).all()), (n, float((out[b].double() - ref).abs().max()))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("nq,nkv,S", [(3, 3, 200), (4, 2, 1400), (8, 2, 150), (8, 1, 300)])
def test_decode_attention_with_infinities_in_the_cache(nq, nkv, S, hd, dtype):
    """A cached key that scores minus infinity has a weight of 0, an infinite value an infinite output in its column, a NaN a
    NaN there: as float64 has it, and nothing else is touched.  Bound of the finite outputs: as in the test above."""
    inf, n, B = float("inf"), S - 1, 5
    g = torch.Generator(device=DEV).manual_seed(nq * 1000 + hd)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).to(dtype)  # noqa: E731
    kc, vc = rnd(B, S, nkv, hd), rnd(B, S, nkv, hd)
    qkv = rnd(B, (nq + 2 * nkv) * hd)
    qkv[:, : nq * hd] = qkv[:, : nq * hd].abs() + 0.5          # an element of a key has its sign in every score
    rows = torch.arange(0, n, 37, device=DEV)
    kc[0, rows, :, 5] = -inf                                   # sequence 0: weights of 0
    kc[0, 3, 0, 7], vc[1, 11, 0, 9], vc[1, 60, 0, 10] = -inf, inf, -inf
    kc[2, n - 1, 0, 0] = -inf
    vc[3, 0, 0, 3] = float("nan")
    q, k, v = (t.reshape(B, -1, hd).double() for t in qkv.split([nq * hd, nkv * hd, nkv * hd], 1))
    out = A.decode_attention(qkv, kc, vc, torch.full((B,), n, dtype=torch.int32, device=DEV), nq, nkv, hd).view(B, nq, hd).double()
    kk, vv = (torch.repeat_interleave(torch.cat([t[:, :n].double(), x.unsqueeze(1)], 1), nq // nkv, 2) for t, x in ((kc, k), (vc, v)))
    w = torch.softmax(torch.einsum("bhd,bnhd->bhn", q, kk) * hd ** -0.5, -1)
    ref = torch.einsum("bhn,bnhd->bhd", w, vv)
    assert bool(torch.isfinite(ref[0]).all()) and bool(torch.isfinite(ref[4]).all())
    assert torch.equal(torch.isnan(out), torch.isnan(ref)) and torch.equal(out[torch.isinf(ref)], ref[torch.isinf(ref)])
    ok = torch.isfinite(ref)
    most = vv.nan_to_num(0, 0, 0).abs().amax(1).amax(-1, keepdim=True).expand_as(ref)
    rounding = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert bool(((out - ref).abs()[ok] <= (rounding * ref.abs() + 3e-5 * most)[ok]).all())


@pytest.mark.parametrize("heads", [(8, 8), (8, 2)])
def test_packed_qkv_attention_forward_backward(heads):
    """Fused-QKV varlen attention (one d(qkv) buffer written by the backward kernel) vs the fp32 reference on sliced q/k/v."""
    nq, nkv = heads
    hd = 64
    torch.manual_seed(1)
    lens = [37, 128, 5, 200]
    T = sum(lens)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), device=DEV, dtype=torch.int32)
    qkv = (torch.randn(T, (nq + 2 * nkv) * hd, device=DEV) * 0.5).to(torch.bfloat16).requires_grad_(True)
    out = A.varlen_attention_qkv(qkv, cu, max(lens), nq, nkv, hd)
    dout = torch.randn_like(out)
    out.backward(dout)
    g = qkv.grad.clone()
    x = qkv.detach().float().requires_grad_(True)
    q = x[:, : nq * hd].view(T, nq, hd)
    k = x[:, nq * hd:(nq + nkv) * hd].view(T, nkv, hd)
    v = x[:, (nq + nkv) * hd:].view(T, nkv, hd)
    ref = A.varlen_attention_ref(q, k, v, cu, hd ** -0.5, True)
    ref.backward(dout.float())
    torch.testing.assert_close(out.float(), ref, atol=2e-2, rtol=2e-2)
    torch.testing.assert_close(g.float(), x.grad, atol=3e-2, rtol=3e-2)


@pytest.mark.parametrize("hd,nq,nkv,causal", [(128, 8, 8, True), (128, 8, 2, True), (64, 4, 4, True), (128, 4, 4, False)])
def test_attn_fwd_tcgen05_matches_reference(hd, nq, nkv, causal):
    import math

    import numpy as np

    from realhf_b200.ops import lib
    torch.manual_seed(0)
    lens = [1, 37, 128, 129, 300, 640, 5]
    T = sum(lens)
    cu = torch.tensor([0] + list(np.cumsum(lens)), dtype=torch.int32, device=DEV)
    qkv = torch.randn(T, (nq + 2 * nkv) * hd, device=DEV, dtype=torch.bfloat16)
    q = qkv[:, : nq * hd].view(T, nq, hd)
    k = qkv[:, nq * hd:(nq + nkv) * hd].view(T, nkv, hd)
    v = qkv[:, (nq + nkv) * hd:].view(T, nkv, hd)
    scale = 1.0 / math.sqrt(hd)
    out, lse = lib().attn_fwd(q, k, v, cu, max(lens), scale, causal)
    ref = A.varlen_attention_ref(q.float(), k.float(), v.float(), cu, scale, causal)
    torch.testing.assert_close(out.float(), ref, atol=2e-2, rtol=2e-2)
    # LSE [nq, T]: natural log of the softmax denominator with the scale applied
    rep = nq // nkv
    for s, e in zip(cu[:-1].tolist(), cu[1:].tolist()):
        att = torch.einsum("qhd,khd->hqk", q[s:e].float(), k[s:e].float().repeat_interleave(rep, 1)) * scale
        if causal:
            att = att.masked_fill(torch.ones(e - s, e - s, device=DEV, dtype=torch.bool).triu(1), float("-inf"))
        torch.testing.assert_close(lse[:, s:e], torch.logsumexp(att, -1), atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("hd,nq,nkv,causal", [(128, 8, 8, True), (128, 8, 2, True), (64, 4, 4, True), (128, 4, 4, False)])
def test_attn_bwd_tcgen05_matches_autograd_of_the_reference(hd, nq, nkv, causal):
    """dq / dk / dv written into the three column ranges of one d(qkv) buffer vs autograd through the fp32 reference."""
    import math

    import numpy as np

    from realhf_b200.ops import lib
    torch.manual_seed(0)
    lens = [1, 37, 128, 129, 300, 640, 5]
    T = sum(lens)
    cu = torch.tensor([0] + list(np.cumsum(lens)), dtype=torch.int32, device=DEV)
    W = (nq + 2 * nkv) * hd
    qkv = torch.randn(T, W, device=DEV, dtype=torch.bfloat16)
    dout = torch.randn(T, nq, hd, device=DEV, dtype=torch.bfloat16)
    scale = 1.0 / math.sqrt(hd)

    def views(t):
        return (t[:, : nq * hd].view(T, nq, hd), t[:, nq * hd:(nq + nkv) * hd].view(T, nkv, hd), t[:, (nq + nkv) * hd:].view(T, nkv, hd))
    # reference: fp32 autograd, forward statistics from the same math
    x = qkv.float().requires_grad_(True)
    qf, kf, vf = views(x)
    ref = A.varlen_attention_ref(qf, kf, vf, cu, scale, causal)
    ref.backward(dout.float())
    q, k, v = views(qkv)
    rep = nq // nkv
    lse = torch.empty(nq, T, device=DEV, dtype=torch.float32)
    for s, e in zip(cu[:-1].tolist(), cu[1:].tolist()):
        att = torch.einsum("qhd,khd->hqk", q[s:e].float(), k[s:e].float().repeat_interleave(rep, 1)) * scale
        if causal:
            att = att.masked_fill(torch.ones(e - s, e - s, device=DEV, dtype=torch.bool).triu(1), float("-inf"))
        lse[:, s:e] = torch.logsumexp(att, -1)
    dqkv = torch.full_like(qkv, float("nan"))   # every element must be written
    dq, dk, dv = views(dqkv)
    lib().attn_bwd(dout, q, k, v, ref.detach().to(torch.bfloat16), lse, dq, dk, dv, cu, max(lens), scale, causal)
    assert torch.isfinite(dqkv.float()).all()
    torch.testing.assert_close(dqkv.float(), x.grad, atol=6e-2, rtol=6e-2)


def _attention_f64(q, k, v, lens, scale, causal, window):
    """(out, sum of weights * |v|, lse) in float64."""
    out, mag, lse = torch.zeros(q.shape, dtype=torch.float64, device=DEV), torch.zeros(q.shape, dtype=torch.float64, device=DEV), []
    a = 0
    for n in lens:
        qq, kk, vv = (t[a:a + n].double().transpose(0, 1) for t in (q, k, v))
        kk, vv = (t.repeat_interleave(q.shape[1] // k.shape[1], 0) for t in (kk, vv))
        i = torch.arange(n, device=DEV)
        ok = torch.ones(n, n, dtype=torch.bool, device=DEV)
        if causal:
            ok = i[None] <= i[:, None]
            if window:
                ok = ok & (i[None] > i[:, None] - window)
        s = (qq @ kk.transpose(1, 2) * scale).masked_fill(~ok, float("-inf"))
        p = torch.softmax(s, -1)
        out[a:a + n], mag[a:a + n] = (p @ vv).transpose(0, 1), (p @ vv.abs()).transpose(0, 1)
        lse.append(torch.logsumexp(s, -1))
        a += n
    return out, mag, torch.cat(lse, 1)


@pytest.mark.parametrize("heads", [(1, 1, 128), (4, 2, 64), (3, 1, 128), (6, 3, 128), (2, 2, 64), (8, 1, 128)])
@pytest.mark.parametrize("lens", [[1], [127, 128, 129, 255, 256, 257], [0, 5, 0, 640, 1], [33] * 70 + [1100], [1536, 385]])
@pytest.mark.parametrize("form", ["causal", "full", "window", "growing"])
def test_attn_fwd_tile_pairs(heads, lens, form):
    """Tile pairs over heads (even groups) and over rows (odd groups), left-over tiles, empty sequences, more than 32 sequences, windows, and scores
    whose maximum grows by orders of magnitude from tile to tile.  Bound: the weights and the result are rounded to 16 bits once each,
    2^-9 of the weighted sum of |v| and 2^-9 of the result, doubled for the exponentials and the scaling of earlier tiles."""
    nq, nkv, hd = heads
    dt = torch.float16 if form == "window" else torch.bfloat16
    torch.manual_seed(len(lens) + nq)
    T = sum(lens)
    qkv = torch.randn(T, (nq + 2 * nkv) * hd, device=DEV)
    if form == "growing":                    # queries and keys share a direction that grows with the position: row maxima climb by hundreds
        pos = torch.cat([torch.arange(n, device=DEV) for n in lens]).float()
        qkv[:, 0:nq * hd:hd] = 8.0
        qkv[:, nq * hd:(nq + nkv) * hd:hd] = pos[:, None] / 8
    qkv = qkv.to(dt)
    q, k, v = (t.view(T, -1, hd) for t in qkv.split([nq * hd, nkv * hd, nkv * hd], 1))
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    window = 150 if form == "window" else 0
    out, lse = lib().attn_fwd_window(q, k, v, cu, max(lens), hd ** -0.5, form != "full", window)
    assert lib().attn_wait_error() == 0
    ref, mag, rlse = _attention_f64(q, k, v, lens, hd ** -0.5, form != "full", window)
    eps = 2.0 ** (-8 if dt == torch.bfloat16 else -11)
    assert ((out.double() - ref).abs() <= eps * ref.abs() + eps * mag + 1e-6).all()
    torch.testing.assert_close(lse.double(), rlse, atol=2e-5, rtol=2e-6)


@pytest.mark.parametrize("cap,sink,hd", [(20.0, False, 64), (20.0, True, 64), (3.0, False, 128), (50.0, True, 128)])
@pytest.mark.parametrize("form", ["ordinary", "overflowing"])
def test_capped_scores(cap, sink, hd, form):
    """Capped scores against float64, also where the products overflow fp32: an infinite product is a score of +-cap like any other, hidden keys alone are
    left out.  Bound as in test_attn_fwd_tile_pairs, and the capped score's own rounding, a few ulps of cap log2 e in the exponent."""
    H, G, lens = 4, 2, [1, 130, 300]
    T, dt = sum(lens), torch.bfloat16
    torch.manual_seed(hd)
    qkv = torch.randn(T, H * hd + 2 * G * hd, device=DEV)
    if form == "overflowing":               # one sign a key, so that no sum holds both infinities; the first sequences' keys are all negative
        sign = torch.where(torch.rand(T, 1, device=DEV) < 0.7, -1.0, 1.0)
        sign[:131] = -1.0
        qkv[:, :H * hd] = 1e25
        qkv[:, H * hd:(H + G) * hd] = sign * 1e25
    qkv = qkv.to(dt)
    vn = qkv[:, (H + G) * hd:].contiguous()
    logit = torch.randn(H, device=DEV).to(dt) if sink else None
    out = torch.full((T, H * hd), float("nan"), device=DEV, dtype=dt)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    scale = hd ** -0.5
    lib().sink_window_attention_tc(qkv, vn, out, None, logit, cu, max(lens), H, G, hd, scale, 0, 0, -1.0, None, False, 0, cap)
    eps, a = 2.0 ** -8 + 16 * 2.0 ** -23 * cap * 1.45, 0
    for n in lens:
        q, k, v = (t[a:a + n].double().view(n, -1, hd).transpose(0, 1) for t in (qkv[:, :H * hd], qkv[:, H * hd:(H + G) * hd], vn))
        k, v = k.repeat_interleave(H // G, 0), v.repeat_interleave(H // G, 0)
        s = cap * torch.tanh(q @ k.transpose(1, 2) * scale / cap)
        s = s.masked_fill(torch.ones(n, n, dtype=torch.bool, device=DEV).triu(1), float("-inf"))
        if sink:
            s = torch.cat([s, logit.double().view(H, 1, 1).expand(H, n, 1)], 2)
        p = torch.softmax(s, -1)[..., :n]
        ref, mag = (p @ v).transpose(0, 1), (p @ v.abs()).transpose(0, 1)
        assert ((out[a:a + n].double().view(n, H, hd) - ref).abs() <= eps * (ref.abs() + mag) + 1e-6).all()
        a += n


@pytest.mark.parametrize("heads", [(1, 1, 128), (4, 2, 64), (3, 1, 128), (8, 1, 128), (8, 8, 64), (16, 4, 128)])
@pytest.mark.parametrize("lens", [[1], [127, 128, 129, 255, 256, 257], [0, 5, 0, 640, 1], [33] * 70 + [1100], [1536, 385], [640] * 12],
                         ids=lambda x: f"{len(x)}x{x[0]}")
@pytest.mark.parametrize("causal", [True, False])
def test_attn_bwd_items(heads, lens, causal):
    """The backward where CTAs take several items (up to 960 of them), one to three query heads and whole groups a key head, left-over rows and blocks,
    empty sequences and more than 32 of them, in both types; `out` starts off a 16-byte boundary for an odd number of sequences.  Against float64
    gradients from the same 16-bit inputs.  Bound: P and dS are rounded to 16 bits once (half an ulp, doubled for exp2 and its argument; values under
    fp16's normal range lose half of its smallest step), dP and delta are fp32 sums whose difference cancels (2^-16 of the sum of magnitudes), and the
    result is rounded once."""
    nq, nkv, hd = heads
    dt = torch.float16 if nq % 4 else torch.bfloat16
    eps, tiny = (2.0 ** -8, 0.0) if dt == torch.bfloat16 else (2.0 ** -11, 2.0 ** -24)
    torch.manual_seed(len(lens) + nq)
    T, scale, rep = sum(lens), hd ** -0.5, nq // nkv
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    qkv = torch.randn(T, (nq + 2 * nkv) * hd, device=DEV).to(dt)
    dout = torch.randn(T, nq, hd, device=DEV).to(dt)
    split = lambda t: [x.view(T, -1, hd) for x in t.split([nq * hd, nkv * hd, nkv * hd], 1)]
    q, k, v = split(qkv)
    out = torch.empty(T * nq * hd + 1, device=DEV, dtype=dt)[len(lens) % 2:][:T * nq * hd].view(T, nq, hd)
    lse = torch.empty(nq, T, device=DEV)
    want, bound = [torch.zeros(T, n, hd, dtype=torch.float64, device=DEV) for n in (nq, nkv, nkv)], []
    bound = [torch.zeros_like(t) for t in want]
    a = 0
    for n in lens:
        r = slice(a, a + n)
        a += n
        qq, dd = (t[r].double().transpose(0, 1) for t in (q, dout))
        kk, vv = (t[r].double().transpose(0, 1).repeat_interleave(rep, 0) for t in (k, v))
        s = qq @ kk.transpose(1, 2) * scale
        if causal:
            s = s.masked_fill(torch.ones(n, n, dtype=torch.bool, device=DEV).triu(1), float("-inf"))
        P = torch.softmax(s, -1)
        lse[:, r] = torch.logsumexp(s, -1).float()
        out[r] = (P @ vv).transpose(0, 1).to(dt)
        oo = out[r].double().transpose(0, 1)                 # delta is defined by the rounded output
        dP, mag = dd @ vv.transpose(1, 2), dd.abs() @ vv.abs().transpose(1, 2) + (dd * oo).abs().sum(-1, keepdim=True)
        dS = P * (dP - (dd * oo).sum(-1, keepdim=True)) * scale
        e_s, e_p = eps * dS.abs() + 2.0 ** -16 * P * mag * scale + tiny * (P > 0), eps * P + tiny * (P > 0)
        group = lambda t: t.view(nkv, rep, n, hd).sum(1).transpose(0, 1)
        want[0][r], bound[0][r] = (dS @ kk).transpose(0, 1), (e_s @ kk.abs()).transpose(0, 1)
        want[1][r], bound[1][r] = group(dS.transpose(1, 2) @ qq), group(e_s.transpose(1, 2) @ qq.abs())
        want[2][r], bound[2][r] = group(P.transpose(1, 2) @ dd), group(e_p.transpose(1, 2) @ dd.abs())
    dqkv = torch.full_like(qkv, float("nan"))                # every element must be written
    lib().attn_bwd(dout, q, k, v, out, lse, *split(dqkv), cu, max(lens), scale, causal)
    assert lib().attn_wait_error() == 0
    for got, w, b in zip(split(dqkv), want, bound):
        assert ((got.double() - w).abs() <= b + eps * w.abs() + 1e-6).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("nq,nkv,hd", [(4, 4, 64), (8, 2, 128)])
def test_packed_qkv_attention_on_columns_of_a_wider_buffer(nq, nkv, hd, dtype):
    """The fused projection as a range of columns of wider rows: outputs and gradients bit for bit those of a copy, with and without a gradient asked for."""
    lens = [1, 130, 77, 300]
    T, W = sum(lens), (nq + 2 * nkv) * hd
    cu = torch.tensor([0] + lens, device=DEV).cumsum(0).int()
    g = torch.Generator(device=DEV).manual_seed(hd)
    wide = torch.randn(T, W + 64, device=DEV, generator=g).to(dtype)
    dout = torch.randn(T, nq, hd, device=DEV, generator=g).to(dtype)
    a, b = wide[:, 32:32 + W], wide[:, 32:32 + W].contiguous()
    call = lambda x: A.varlen_attention_qkv(x, cu, max(lens), nq, nkv, hd)
    want = call(b)
    assert torch.equal(call(a), want)
    wide.requires_grad_(True)
    leaf = b.requires_grad_(True)
    got, out = call(wide[:, 32:32 + W]), call(leaf)
    assert torch.equal(got, want) and torch.equal(out, want)
    got.backward(dout)
    out.backward(dout)
    assert torch.equal(wide.grad[:, 32:32 + W], leaf.grad) and not wide.grad[:, :32].any() and not wide.grad[:, 32 + W:].any()


def test_packed_qkv_attention_inside_function_transforms():
    """Without a gradient asked for the kernel is called without its autograd function, which is what refuses forward-mode differentiation and function
    transforms: they are refused all the same, and a plain tensor inside a forward-mode level is not."""
    from torch.autograd import forward_ad as fw
    T, n, hd = 40, 2, 64
    cu = torch.tensor([0, T], dtype=torch.int32, device=DEV)
    qkv = torch.randn(T, 3 * n * hd, device=DEV).to(torch.bfloat16)
    call = lambda x: A.varlen_attention_qkv(x, cu, T, n, n, hd)
    want = call(qkv)
    with fw.dual_level():
        assert torch.equal(call(qkv), want)
        with pytest.raises((RuntimeError, NotImplementedError)):
            call(fw.make_dual(qkv, torch.ones_like(qkv)))
    with pytest.raises((RuntimeError, NotImplementedError)):
        torch.func.vmap(call)(qkv.unsqueeze(0).expand(2, -1, -1))
    with pytest.raises((RuntimeError, NotImplementedError)):
        torch.func.grad(lambda x: call(x).float().sum())(qkv)
    assert torch.equal(call(qkv), want)


def test_a_wait_that_ran_out_is_raised_and_the_update_skipped():
    """The status word as a kernel leaves it whose bounded wait ran out (set here by a copy): the next attention call of either direction and the
    engine raise, the optimizer leaves the parameters alone, and clearing the word makes everything run again."""
    from realhf_b200.api.config import ModelName
    from realhf_b200.api.model import FinetuneSpec, Model, ReaLModelConfig
    from realhf_b200.engine.engine import TrainBackend
    from realhf_b200.models.real_model import ReaLModel
    dev = torch.device("cuda", 0)
    cfg = ReaLModelConfig(n_layers=1, n_kv_heads=2, n_q_heads=2, hidden_dim=128, intermediate_dim=256, vocab_size=512, n_positions=64, embd_pdrop=0.0,
                          resid_pdrop=0.0, attn_pdrop=0.0, activation_function="silu", layer_norm_type="rms", mlp_type="llama", apply_rotary=True)
    m = ReaLModel(cfg, dtype=torch.bfloat16, device=dev).init_random_fast()
    engine = TrainBackend(optimizer=dict(lr=1e-2, warmup_steps_proportion=0.0)).initialize(Model(ModelName("actor", 0), m, None, dev),
                                                                                          FinetuneSpec(1, 10, 10)).module
    opt = engine.optim
    q, k, v = (torch.randn(40, 2, 64, device=DEV, dtype=torch.bfloat16) for _ in range(3))
    cu = torch.tensor([0, 40], dtype=torch.int32, device=DEV)
    fwd = lambda: lib().attn_fwd(q, k, v, cu, 40, 0.125, True)
    out, lse = fwd()
    bwd = lambda: lib().attn_bwd(out, q, k, v, out, lse, torch.empty_like(q), torch.empty_like(k), torch.empty_like(v), cu, 40, 0.125, True)

    def step():
        opt.zero_grad()
        opt.flat_grad.fill_(1e-2)
        return float(opt.step()["skipped"])
    assert lib().attn_wait_error() == 0
    word = lib().attn_status(dev)
    word.fill_(1)
    before = m.flat_param.detach().clone()
    assert step() == 1.0 and torch.equal(m.flat_param, before)
    for call in (fwd, bwd, engine._check_device_flags):
        with pytest.raises(RuntimeError, match="gave up"):
            call()
    assert lib().attn_wait_error() == 1 and lib().attn_wait_error() == 0 and int(word) == 0
    assert step() == 0.0 and not torch.equal(m.flat_param, before)
    fwd(), bwd(), engine._check_device_flags()
    torch.cuda.synchronize()


@pytest.mark.parametrize("use_graph", [True, False])
def test_a_wait_that_ran_out_in_a_generation_step_is_raised(use_graph, monkeypatch):
    """A replayed step does not look at the status word (set here behind the last step by a copy): generate() does before it hands the tokens out."""
    from realhf_b200.api.model import GenerationHyperparameters, ReaLModelConfig
    from realhf_b200.models import generation as gen
    from realhf_b200.models.real_model import ReaLModel
    dev = torch.device("cuda", 0)
    cfg = ReaLModelConfig(n_layers=1, n_kv_heads=2, n_q_heads=2, hidden_dim=128, intermediate_dim=256, vocab_size=512, n_positions=64, embd_pdrop=0.0,
                          resid_pdrop=0.0, attn_pdrop=0.0, activation_function="silu", layer_norm_type="rms", mlp_type="llama", apply_rotary=True)
    m = ReaLModel(cfg, dtype=torch.bfloat16, device=dev).init_random_fast()
    ids, cu = torch.arange(3, 23, device=dev), torch.tensor([0, 8, 20], dtype=torch.int32, device=dev)
    g = GenerationHyperparameters(max_new_tokens=4, min_new_tokens=4, greedy=True, use_cuda_graph=use_graph)
    word, steps, final = lib().attn_status(dev), [], gen._final_logits

    def run():
        with torch.no_grad():
            return gen.generate(m, ids, cu, g, eos_id=None, pad_id=0)[0].tokens

    want, m.training = run(), True
    if use_graph:
        count = gen.launches.count_replay
        monkeypatch.setattr(gen.launches, "count_replay", lambda n: (count(n), steps.append(1), word.fill_(int(len(steps) == 3))))
    else:
        monkeypatch.setattr(gen, "_final_logits", lambda *a: (final(*a), steps.append(1), word.fill_(int(len(steps) == 4)))[0])
    with pytest.raises(RuntimeError, match="gave up"):
        run()
    assert m.training and lib().attn_wait_error() == 1
    monkeypatch.undo()
    assert torch.equal(run(), want)


def test_attention_status_says_what_went_wrong():
    """Shared memory that a kernel cannot work in is not reported as a wait that ran out."""
    q = torch.randn(40, 2, 64, device=DEV, dtype=torch.bfloat16)
    cu = torch.tensor([0, 40], dtype=torch.int32, device=DEV)
    word = lib().attn_status(torch.device("cuda", 0))
    assert lib().attn_wait_error() == 0
    for code, text in ((2, "1024 bytes"), (1, "gave up waiting")):
        word.fill_(code)
        torch.cuda.synchronize()
        with pytest.raises(RuntimeError, match=text):
            lib().attn_fwd(q, q, q, cu, 40, 0.125, True)
        assert lib().attn_wait_error() == code and lib().attn_wait_error() == 0


def _scores(cols):
    """Sequences [S, n keys, 128] of scores -> q, k, v of one head whose query r has the scores of column r % 128, one sequence after the other."""
    S, n, _ = cols.shape
    q = torch.eye(128, device=DEV, dtype=torch.bfloat16)[torch.arange(n, device=DEV) % 128].repeat(S, 1).view(S * n, 1, 128)
    k = cols.reshape(S * n, 1, 128).bfloat16()
    assert torch.equal(k.float(), cols.reshape(S * n, 1, 128))
    return q, k, torch.zeros_like(k), torch.arange(S + 1, device=DEV, dtype=torch.int32) * n


def _bits(x, ones, n=128):
    """Scores [..., n]: weights 2^score whose sum is x (< 4, 24 bits): `ones` keys of weight one first."""
    i = torch.arange(n, device=DEV)
    frac = (x - x.floor()).double().unsqueeze(-1)
    bit = (frac * 2.0 ** i.clamp(max=24)).floor() % 2
    s = torch.where((i >= 1) & (i <= 23) & (bit == 1), -i.double(), -256.0)
    return torch.where((i == 0) | ((i > 23) & (i < 23 + ones.unsqueeze(-1))), 0.0, s).float()


LN2 = 0.6931471805599453            # as the scale: a weight is 2^score exactly


def test_attention_statistics_are_rounded_tile_by_tile():
    """The denominator of two key tiles is round(round(l * factor) + sum of the second tile): scores chosen so that the weights are powers of two and their sums exact leave these two
    roundings alone, and a sequence of one tile with that very denominator gives the same statistics bit for bit."""
    g = torch.Generator(device=DEV).manual_seed(3)
    draw = lambda: 1 + torch.randint(0, 2 ** 23, (16, 128), device=DEV, generator=g).float() * 2.0 ** -23  # noqa: E731
    l1, s2 = draw(), draw()
    one = torch.ones_like(l1)
    first = _bits(l1, one)
    cols = torch.cat([torch.where(first > -100, first - 0.5, first), _bits(s2, one)], -1).transpose(1, 2).contiguous()
    factor = torch.exp2(torch.tensor(-0.5, device=DEV))
    total = l1 * factor + s2
    assert (total.double() != (l1.double() * factor.double() + s2.double()).float().double()).sum() > 100       # a contracted sum would show
    q, k, v, cu = _scores(cols)
    lse = lib().attn_fwd(q, k, v, cu, 256, LN2, False)[1].view(16, 2, 128)
    q, k, v, cu = _scores(_bits(total, total.floor()).transpose(1, 2).contiguous())
    want = lib().attn_fwd(q, k, v, cu, 128, LN2, False)[1].view(16, 1, 128)
    assert torch.equal(lse, want.expand_as(lse))


def test_attention_statistics_end_in_one_rounding():
    """log2 of a power of two is exact: the statistics are the maximum's product rounded once, the logarithm's added with one rounding."""
    j = torch.arange(8, device=DEV).repeat(16)
    m = (torch.arange(128, device=DEV) - 64) * 0.5 - 3.5
    i = torch.arange(128, device=DEV)[:, None]
    q, k, v, cu = _scores(torch.where(i < 2 ** j, m, -256.0)[None].float())
    lse = lib().attn_fwd(q, k, v, cu, 128, LN2, False)[1][0]
    ln2 = torch.tensor(LN2, dtype=torch.float32, device=DEV)
    assert torch.equal(lse, (j.double() * ln2.double() + (m.float() * ln2).double()).float())
