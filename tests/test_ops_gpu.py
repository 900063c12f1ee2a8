"""Numerics of every sm_100a kernel against a plain PyTorch fp32 reference of the same op."""
import pytest
import torch

from realhf_b200.ops import functional as OF
from realhf_b200.ops import lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _packed_case(bs=37, max_len=700, seed=0):
    g = torch.Generator().manual_seed(seed)
    lens = torch.randint(1, max_len, (bs,), generator=g)
    cu = torch.zeros(bs + 1, dtype=torch.int32)
    cu[1:] = lens.cumsum(0)
    total = int(cu[-1])
    return lens, cu, total, g


def test_gae_1d_matches_reference():
    lens, cu, total, g = _packed_case()
    bs = lens.numel()
    rewards = torch.randn(total, generator=g)
    values = torch.randn(total + bs, generator=g)
    boot = torch.rand(bs, generator=g) > 0.5
    a_ref, r_ref = OF.gae_1d_misalign_ref(rewards, values, cu, boot, 0.99, 0.95)
    a, r = OF.gae_1d_misalign(rewards.to(DEV), values.to(DEV), cu.to(DEV), boot.to(DEV), 0.99, 0.95)
    torch.testing.assert_close(a.cpu(), a_ref, atol=1e-4, rtol=1e-4)
    torch.testing.assert_close(r.cpu(), r_ref, atol=1e-4, rtol=1e-4)


def test_ppo_rewards_gae_fused():
    lens, cu, total, g = _packed_case(bs=64, max_len=600, seed=1)
    bs = lens.numel()
    logp, ref = torch.randn(total, generator=g), torch.randn(total, generator=g)
    scores = torch.randn(bs, generator=g) * 10
    values = torch.randn(total + bs, generator=g)
    no_eos = torch.rand(bs, generator=g) > 0.7
    ref_out = OF.ppo_rewards_gae_ref(logp, ref, scores, values, cu, no_eos, 1.0, 0.95, 0.1, 5.0)
    out = OF.ppo_rewards_gae(logp.to(DEV), ref.to(DEV), scores.to(DEV), values.to(DEV), cu.to(DEV), no_eos.to(DEV),
                             1.0, 0.95, 0.1, 5.0)
    for o, r in zip(out, ref_out):
        torch.testing.assert_close(o.cpu(), r, atol=2e-4, rtol=1e-4)


@pytest.mark.parametrize("mode", ["olp", "nolp"])
def test_gae_2d(mode):
    g = torch.Generator().manual_seed(2)
    bs, T = 33, 257
    rewards, values = torch.randn(bs, T, generator=g), torch.randn(bs, T + 1, generator=g)
    dones = torch.rand(bs, T + 1, generator=g) > 0.95
    truncs = (torch.rand(bs, T + 1, generator=g) > 0.5) & dones
    a_ref, r_ref = OF.gae_2d_ref(rewards, values, dones, truncs, 0.98, 0.9, mode)
    a, r = OF.gae_2d(rewards.to(DEV), values.to(DEV), dones.to(DEV), truncs.to(DEV), 0.98, 0.9, mode)
    torch.testing.assert_close(a.cpu(), a_ref, atol=1e-4, rtol=1e-4)
    torch.testing.assert_close(r.cpu(), r_ref, atol=1e-4, rtol=1e-4)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("H", [256, 4096, 5120, 8192])
def test_rmsnorm_fwd_bwd(dtype, H):
    torch.manual_seed(0)
    x = torch.randn(300, H, device=DEV, dtype=dtype, requires_grad=True)
    w = (torch.randn(H, device=DEV) * 0.1 + 1).to(dtype).requires_grad_(True)
    y = OF.rmsnorm(x, w, 1e-5, 0.0)
    dy = torch.randn_like(y)
    y.backward(dy)
    xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    yr = OF.rmsnorm_ref(xr, wr, 1e-5, 0.0)
    yr.backward(dy.float())
    tol = dict(atol=2e-2, rtol=2e-2) if dtype != torch.float32 else dict(atol=1e-4, rtol=1e-4)
    torch.testing.assert_close(y.float(), yr, **tol)
    torch.testing.assert_close(x.grad.float(), xr.grad, **tol)
    torch.testing.assert_close(w.grad.float(), wr.grad, atol=0.3 if dtype != torch.float32 else 1e-3, rtol=3e-2)


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs a second GPU")
@pytest.mark.parametrize("dtype,H", [(torch.bfloat16, 1024), (torch.bfloat16, 4096), (torch.float32, 2048)])
def test_rmsnorm_bwd_on_every_device_of_a_process(dtype, H):
    """The kernel's shared-memory opt-in belongs to one device: every further GPU of the process needs its own."""
    torch.manual_seed(H)
    x, w, dy = (torch.randn(*s).to(dtype) for s in ((300, H), (H,), (300, H)))
    rstd = torch.rand(300)
    got = [[t.cpu() for t in lib().rmsnorm_bwd(x.to(d), w.to(d), dy.to(d), rstd.to(d), 0.0, None)] for d in range(torch.cuda.device_count())]
    for other in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], other))


def test_add_rmsnorm_gemma_offset():
    torch.manual_seed(0)
    x = torch.randn(128, 2048, device=DEV, dtype=torch.bfloat16)
    res = torch.randn_like(x)
    w = torch.randn(2048, device=DEV, dtype=torch.bfloat16) * 0.1
    with torch.no_grad():
        y, r = OF.add_rmsnorm(x, res, w, 1e-6, 1.0)
    yr, rr = OF.rmsnorm_ref(x, w, 1e-6, 1.0, residual=res)
    torch.testing.assert_close(r, rr)
    torch.testing.assert_close(y.float(), yr.float(), atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("w_off", [0.0, 1.0])
def test_add_rmsnorm_training_forward_and_fused_backward(dtype, w_off):
    """(h, x_new) = (rmsnorm(x + d), x + d) with autograd: both outputs are used downstream (the norm feeds the block, the sum
    continues as the residual stream), so the backward kernel must add the residual-stream gradient to the norm gradient."""
    torch.manual_seed(0)
    H = 4096
    d = torch.randn(257, H, device=DEV, dtype=dtype, requires_grad=True)
    x = torch.randn(257, H, device=DEV, dtype=dtype, requires_grad=True)
    w = (torch.randn(H, device=DEV) * 0.1 + (0.0 if w_off else 1.0)).to(dtype).requires_grad_(True)
    h, xn = OF.add_rmsnorm(d, x, w, 1e-5, w_off)
    gh, gx = torch.randn_like(h), torch.randn_like(xn)
    torch.autograd.backward([h, xn], [gh, gx])
    dr, xr, wr = (t.detach().float().requires_grad_(True) for t in (d, x, w))
    s = (dr + xr) if dtype == torch.float32 else (dr + xr).to(dtype).float() + 0 * (dr + xr)  # the stream is stored in `dtype`
    sr = dr + xr
    hr = sr * torch.rsqrt(sr.pow(2).mean(-1, keepdim=True) + 1e-5) * (wr + w_off)
    torch.autograd.backward([hr, sr], [gh.float(), gx.float()])
    tol = dict(atol=3e-2, rtol=3e-2) if dtype != torch.float32 else dict(atol=1e-4, rtol=1e-4)
    torch.testing.assert_close(h.float(), hr, **tol)
    torch.testing.assert_close(xn.float(), sr, **tol)
    torch.testing.assert_close(d.grad.float(), dr.grad, **tol)
    torch.testing.assert_close(x.grad.float(), xr.grad, **tol)
    torch.testing.assert_close(w.grad.float(), wr.grad, atol=0.4 if dtype != torch.float32 else 2e-3, rtol=3e-2)
    # only the residual output used (e.g. a stage boundary): gradient passes straight through
    d2, x2 = d.detach().clone().requires_grad_(True), x.detach().clone().requires_grad_(True)
    _, xn2 = OF.add_rmsnorm(d2, x2, w.detach().requires_grad_(True), 1e-5, w_off)
    xn2.backward(gx)
    torch.testing.assert_close(d2.grad, gx)
    torch.testing.assert_close(x2.grad, gx)


@pytest.mark.parametrize("interleaved", [False, True])
def test_rope_inplace_and_grad(interleaved):
    torch.manual_seed(0)
    T, nq, nkv, hd = 513, 8, 2, 128
    row = (nq + 2 * nkv) * hd
    qkv = torch.randn(T, row, device=DEV, dtype=torch.bfloat16)
    pos = torch.randint(0, 2048, (T,), device=DEV, dtype=torch.int32)
    cos, sin = OF.rope_tables(2048, hd, 10000.0, DEV)
    ref = OF.rope_ref(qkv, cos, sin, pos, nq + nkv, hd, hd, interleaved)
    out = OF.apply_rope(qkv.clone(), cos, sin, pos, nq + nkv, hd, hd, interleaved)
    torch.testing.assert_close(out.float(), ref.float(), atol=2e-2, rtol=2e-2)
    assert torch.equal(out[:, (nq + nkv) * hd:], qkv[:, (nq + nkv) * hd:])
    # gradient = inverse rotation
    x = qkv.clone().requires_grad_(True)
    y = OF.apply_rope(x * 1.0, cos, sin, pos, nq + nkv, hd, hd, interleaved)
    dy = torch.randn_like(y)
    y.backward(dy)
    gref = OF.rope_ref(dy, cos, sin, pos, nq + nkv, hd, hd, interleaved, inverse=True)
    torch.testing.assert_close(x.grad.float(), gref.float(), atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("kind", ["silu", "gelu_pytorch_tanh"])
def test_gated_act(kind):
    torch.manual_seed(0)
    gu = torch.randn(777, 2 * 1408, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    out = OF.gated_act(gu, kind)
    d = torch.randn_like(out)
    out.backward(d)
    gr = gu.detach().float().requires_grad_(True)
    outr = OF.gated_act_ref(gr, kind)
    outr.backward(d.float())
    torch.testing.assert_close(out.float(), outr, atol=3e-2, rtol=3e-2)
    torch.testing.assert_close(gu.grad.float(), gr.grad, atol=3e-2, rtol=3e-2)


@pytest.mark.parametrize("V", [32000, 50257])
@pytest.mark.parametrize("masked", [False, True])
def test_logprob_from_logits(V, masked):
    torch.manual_seed(0)
    T = 257
    logits = (torch.randn(T, V, device=DEV) * 3).to(torch.bfloat16)
    labels = torch.randint(0, V, (T,), device=DEV)
    bits = None
    if masked:
        m = torch.rand(T, V, device=DEV) > 0.3
        m[torch.arange(T), labels] = False
        bits = OF.pack_mask_bits(m)
        assert torch.equal(OF.unpack_mask_bits(bits, V), m)
    lp, lse = OF.logprob_from_logits(logits, labels, bits, 1 / 0.7)
    lpr, lser = OF.logprob_from_logits_ref(logits, labels, bits, 1 / 0.7)
    torch.testing.assert_close(lp, lpr, atol=2e-3, rtol=1e-3)
    torch.testing.assert_close(lse, lser, atol=2e-3, rtol=1e-3)


def test_lm_head_logprobs_fwd_bwd():
    torch.manual_seed(0)
    T, H, V = 1000, 512, 32000
    h = (torch.randn(T, H, device=DEV) * 0.5).to(torch.bfloat16).requires_grad_(True)
    w = (torch.randn(V, H, device=DEV) * 0.05).to(torch.bfloat16).requires_grad_(True)
    labels = torch.randint(0, V, (T,), device=DEV)
    lp = OF.lm_head_logprobs(h, w, labels, chunk=384)
    d = torch.randn(T, device=DEV)
    lp.backward(d)
    hr, wr = h.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    lpr = OF.lm_head_logprobs_ref(hr, wr, labels)
    lpr.backward(d)
    torch.testing.assert_close(lp, lpr, atol=5e-2, rtol=2e-2)
    torch.testing.assert_close(h.grad.float(), hr.grad, atol=5e-2, rtol=5e-2)
    torch.testing.assert_close(w.grad.float(), wr.grad, atol=5e-2, rtol=5e-2)


@pytest.mark.parametrize("T,chunk", [(384, 384), (392, 384), (380, 384), (8, 8192)])
@pytest.mark.parametrize("buffer", ["weight_type", "fp32", None])
def test_head_gradient_is_added_to_what_the_buffer_holds(T, chunk, buffer):
    """One chunk, more than one, a token count that is no multiple of 8; a gradient buffer of the weight's type, an fp32 one, none; twice in a row, the weight
    also an embedding, against float64.  Bound: logits and their gradients in 16 bits (2^-9 of values up to 4) move the product by less than 2 %, each of at most
    five sums is rounded to 16 bits; a sum left out or added twice is off by the product itself."""
    from realhf_b200.ops import gemm as G
    impl = OF.gemm_impl()
    OF.set_gemm_impl(G.linear)
    try:
        torch.manual_seed(T)
        H, V = 256, 1000
        h = (torch.randn(T, H, device=DEV) * 0.5).to(torch.bfloat16)
        w = torch.nn.Parameter((torch.randn(V, H, device=DEV) * 0.05).to(torch.bfloat16))
        labels, ids = torch.randint(0, V, (T,), device=DEV), torch.randint(0, V, (T,), device=DEV)
        d, e = torch.randn(T, device=DEV), torch.randn(T, H, device=DEV).to(torch.bfloat16) * 0.3
        wr = w.detach().double().requires_grad_(True)
        lp = torch.log_softmax(h.double() @ wr.t(), -1).gather(1, labels.unsqueeze(1)).squeeze(1)
        (product,) = torch.autograd.grad((lp * d.double()).sum(), wr)
        looked_up = torch.zeros_like(product).index_add_(0, ids, e.double())
        old = torch.randn(V, H, device=DEV) * float(product.std())
        if buffer == "weight_type":
            old = old.to(torch.bfloat16)
            w.grad, w._grad_in_flat_buffer = old.clone(), True
        elif buffer == "fp32":
            w.main_grad = old.clone()
        for _ in range(2):
            ((OF.lm_head_logprobs(h, w, labels, chunk=chunk) * d).sum() + (torch.nn.functional.embedding(ids, w) * e).sum()).backward()
        got = sum(t.double() for t in (w.grad, getattr(w, "main_grad", None)) if t is not None)
        want = 2 * (product + looked_up) + (old.double() if buffer else 0)
        assert float((got - want).norm()) <= 0.02 * 2 * float(product.norm()) + 5 * 2.0 ** -9 * float(want.norm())
    finally:
        OF.set_gemm_impl(impl)


@pytest.mark.parametrize("cfg", [("bf16", "bf16", "fp32", True), ("bf16", "bf16", "bf16", False), ("fp32", "fp32", "fp32", False),
                                 ("bf16", "fp32", "fp32", True)])
def test_adamw_matches_reference(cfg):
    dt = {"bf16": torch.bfloat16, "fp32": torch.float32}
    pd, gd, sd, use_master = dt[cfg[0]], dt[cfg[1]], dt[cfg[2]], cfg[3]
    torch.manual_seed(0)
    n = 1_000_003
    p = torch.randn(n, device=DEV).to(pd)
    g = (torch.randn(n, device=DEV) * 1e-2).to(gd)
    m, v = torch.zeros(n, device=DEV, dtype=sd), torch.zeros(n, device=DEV, dtype=sd)
    master = p.float().clone() if use_master else None
    pr, mr, vr = p.clone(), m.clone(), v.clone()
    masterr = master.clone() if use_master else None
    scale = torch.tensor(0.5, device=DEV)
    skip = torch.zeros(1, dtype=torch.int32, device=DEV)
    for step in (1, 2, 3):
        OF.adamw_step(p, g, m, v, master, 1e-3, 0.9, 0.95, 1e-5, 0.05, step, scale, skip)
        OF.adamw_ref(pr, g, mr, vr, masterr, 1e-3, 0.9, 0.95, 1e-5, 0.05, step, 0.5)
    tol = dict(atol=1e-5, rtol=1e-4) if pd == torch.float32 else dict(atol=1e-2, rtol=1e-2)
    torch.testing.assert_close(p.float(), pr.float(), **tol)
    if use_master:
        torch.testing.assert_close(master, masterr, atol=1e-5, rtol=1e-4)
    # skip flag suppresses the update
    skip.fill_(1)
    before = p.clone()
    OF.adamw_step(p, g, m, v, master, 1e-3, 0.9, 0.95, 1e-5, 0.05, 4, scale, skip)
    assert torch.equal(before, p)


def test_sumsq_and_nonfinite():
    g = torch.randn(3_000_001, device=DEV).to(torch.bfloat16)
    out = torch.zeros(2, device=DEV)
    OF.sumsq_accum(g, out)
    torch.testing.assert_close(out[0], g.float().pow(2).sum(), rtol=1e-3, atol=1)
    assert out[1].item() == 0
    g[12345] = float("inf")
    out.zero_()
    OF.sumsq_accum(g, out)
    assert out[1].item() == 1


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_interval_ops_match_python(dtype):
    torch.manual_seed(0)
    n = 20_000_000
    src = torch.randn(n, device=DEV).to(dtype)
    starts = torch.randperm(n // 1000)[:5000].sort().values * 1000
    lens = torch.randint(1, 999, (5000,))
    iv = [(int(s), int(s + l)) for s, l in zip(starts, lens)]
    perm = torch.randperm(len(iv)).tolist()
    iv = [iv[i] for i in perm]
    packed = OF.slice_intervals(src, iv)
    ref = torch.cat([src[a:b] for a, b in iv])
    assert torch.equal(packed, ref)
    dst = torch.zeros_like(src)
    OF.set_intervals(packed, dst, iv)
    dref = torch.zeros_like(src)
    for a, b in iv:
        dref[a:b] = src[a:b]
    assert torch.equal(dst, dref)


def test_segment_copy_ema():
    src = torch.randn(1 << 20, device=DEV).to(torch.bfloat16)
    dst = torch.randn(1 << 20, device=DEV).to(torch.bfloat16)
    ref = (0.3 * src.float() + 0.7 * dst.float()).to(torch.bfloat16)
    plan = OF.SegmentPlan([0], [0], [src.numel() * 2], DEV)
    plan.run(src, dst, eta=0.3)
    torch.testing.assert_close(dst.float(), ref.float(), atol=1e-2, rtol=1e-2)


@pytest.mark.parametrize("H,dtype", [(768, torch.bfloat16), (1024, torch.float16), (4096, torch.bfloat16), (1600, torch.float32)])
def test_layernorm_native_matches_reference(H, dtype, monkeypatch):
    from realhf_b200.ops import functional as OF
    monkeypatch.setenv("REAL_LAYERNORM", "native")
    torch.manual_seed(0)
    x = (torch.randn(517, H, device="cuda") * 2 + 0.5).to(dtype).requires_grad_(True)
    w = (1 + 0.1 * torch.randn(H, device="cuda")).to(dtype).requires_grad_(True)
    b = (0.1 * torch.randn(H, device="cuda")).to(dtype).requires_grad_(True)
    dy = torch.randn(517, H, device="cuda").to(dtype)
    y = OF.layer_norm(x, w, b, 1e-5)
    y.backward(dy)
    xr, wr, br = (t.detach().float().requires_grad_(True) for t in (x, w, b))
    yr = torch.nn.functional.layer_norm(xr, (H,), wr, br, 1e-5)
    yr.backward(dy.float())
    tol = dict(atol=2e-2, rtol=2e-2) if dtype != torch.float32 else dict(atol=1e-4, rtol=1e-4)
    torch.testing.assert_close(y.float(), yr, **tol)
    torch.testing.assert_close(x.grad.float(), xr.grad, **tol)
    torch.testing.assert_close(w.grad.float(), wr.grad, atol=tol["atol"] * 20, rtol=tol["rtol"])
    torch.testing.assert_close(b.grad.float(), br.grad, atol=tol["atol"] * 20, rtol=tol["rtol"])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,H", [(1, 8), (3, 1024), (593, 1032), (1500, 2048), (149, 2056), (2400, 4096), (37, 4104), (700, 8192)])
@pytest.mark.parametrize("with_dres", [False, True])
def test_rmsnorm_bwd_row_rings(dtype, rows, H, with_dres):
    """The backward kernel against float64 where its rings of rows wrap, end early or stay empty, at the edges of its widths.  dx is one rounding of a
    sum of three terms (each rounded in fp32), dw an fp32 sum over the rows rounded once."""
    torch.manual_seed(rows + H)
    x, dy, dres = (torch.randn(rows, H, device=DEV).to(dtype) for _ in range(3))
    w = (1 + 0.1 * torch.randn(H, device=DEV)).to(dtype)
    y, rstd = lib().rmsnorm_fwd(x, None, w, 1e-5, 0.5)[:2]
    dx, dw = lib().rmsnorm_bwd(x, w, dy, rstd, 0.5, dres if with_dres else None)
    xd, wd = x.double(), w.double() + 0.5
    r = torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-5)
    xh, g = xd * r, dy.double() * wd
    rdx = r * (g - xh * (g * xh).mean(-1, keepdim=True)) + (dres.double() if with_dres else 0.0)
    rdw = (dy.double() * xh).sum(0)
    eps = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -20}[dtype]
    mag = r * (g.abs() + xh.abs() * (g * xh).abs().mean(-1, keepdim=True)) + (dres.double().abs() if with_dres else 0.0)
    assert ((dx.double() - rdx).abs() <= eps * rdx.abs() + 2.0 ** -20 * mag + 1e-7).all()
    assert ((dw.double() - rdw).abs() <= eps * rdw.abs() + 2.0 ** -20 * (dy.double() * xh).abs().sum(0) + 1e-7).all()


@pytest.mark.parametrize("dtype,buffer", [(torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32), (torch.float16, torch.float16), (torch.float32, torch.float32)])
@pytest.mark.parametrize("T,V,H", [(1, 3, 8), (33, 1, 64), (300, 7, 72), (1000, 50, 264), (5000, 4000, 2048), (2000, 2, 1032)])
def test_embedding_gradient_goes_into_the_buffer(T, V, H, dtype, buffer):
    """Against the sums in float64: an fp32 sum of c rows errs by at most c ulps of the sum of their magnitudes, and the result is rounded once to the buffer's type.
    Chains of one token, of up to 32, and longer ones; ids that do not occur; the same every time."""
    from realhf_b200.ops import functional as OF
    g = torch.Generator(device="cuda").manual_seed(T + H)
    ids = torch.randint(0, V, (T,), device="cuda", generator=g)
    ids[: T // 3] = V // 2
    if V > 4:
        ids[ids == V - 1] = 0
    w = torch.nn.Parameter(torch.randn(V, H, device="cuda", generator=g).to(dtype))
    dy = torch.randn(T, H, device="cuda", generator=g).to(dtype)
    start = torch.randn(V, H, device="cuda", generator=g).to(buffer)
    got = []
    for _ in range(2):
        buf = start.clone()
        if buffer == dtype:
            w.grad, w._grad_in_flat_buffer = buf, True
        else:
            w.main_grad = buf
        y = OF.embedding(ids.view(1, -1), w)
        assert torch.equal(y[0], w.detach()[ids])
        y.backward(dy.view(1, T, H))
        got.append(buf)
    assert torch.equal(got[0], got[1])
    want = start.double().index_add(0, ids, dy.double())
    size = start.double().abs().index_add(0, ids, dy.double().abs())
    n = torch.bincount(ids, minlength=V).max().item() + 1
    bound = size * n * 2.0 ** -24 + want.abs() * torch.finfo(buffer).eps / 2 * 1.01 + 1e-12
    if buffer == torch.float16:
        bound = bound + 2.0 ** -25
    assert ((got[0].double() - want).abs() <= bound).all()
    if V > 4:
        assert torch.equal(got[0][V - 1], start[V - 1])


def _positions(B, n):
    return torch.arange(n, device="cuda").repeat(B)


@pytest.mark.parametrize("B,n,H,ids_dtype", [(33, 50, 264, torch.int64), (40, 700, 1032, torch.int32), (512, 30, 72, torch.int64), (513, 30, 72, torch.int32),
                                             (1030, 68, 136, torch.int64), (33, 1, 8, torch.int64)])
def test_embedding_gradient_of_many_long_chains(B, n, H, ids_dtype):
    """Positions of B sequences: every id has B tokens, ranked up to 512 and through a bitmap beyond, over more than one window of 65536 tokens too; some ids outside the
    table, which are passed over.  Small whole numbers, so that the sums are exact; the tokens in any order, and the same for fp32 rows."""
    from realhf_b200.ops import lib
    g = torch.Generator(device="cuda").manual_seed(B + n)
    ids = _positions(B, n)[torch.randperm(B * n, device="cuda", generator=g)]
    ids[ids == n // 2] = torch.where(torch.rand(B, device="cuda", generator=g) < 0.5, -1, n + 3) if n > 1 else 0
    keep = (ids >= 0) & (ids < n)
    dy = torch.randint(-3, 4, (B * n, H), device="cuda", generator=g).float()
    want = torch.ones(n, H, device="cuda").index_add_(0, ids[keep], dy[keep])
    for dtype, buffer in ((torch.float32, torch.float32), (torch.bfloat16, torch.float32), (torch.float16, torch.float16)):
        buf = torch.ones(n, H, device="cuda", dtype=buffer)
        lib().embedding_grad_(dy.to(dtype), ids.to(ids_dtype), buf)
        assert torch.equal(buf, want.to(buffer))


def _best(f):
    times = []
    for _ in range(6):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(5):
            f()
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b))
    return min(times)


@pytest.mark.parametrize("ids,V,H", [(lambda: _positions(64, 1024), 1024, 1024), (lambda: _positions(128, 512), 1024, 768),
                                     (lambda: torch.arange(32768, device="cuda") * 7919 % 256, 256, 1024), (lambda: torch.zeros(100000, device="cuda", dtype=torch.long), 8, 256)],
                         ids=["64x1024 positions", "128x512 positions", "256 ids", "one id"])
def test_embedding_gradient_is_no_slower_than_the_library(ids, V, H):
    """Where every id is frequent: against the library's dense gradient and its sum into the buffer, best of a few (2 .. 8 times as fast when written)."""
    from realhf_b200.ops import lib
    ids, L = ids(), lib()
    dy, buf = torch.randn(ids.numel(), H, device="cuda").bfloat16(), torch.zeros(V, H, device="cuda", dtype=torch.bfloat16)
    ours = _best(lambda: L.embedding_grad_(dy, ids, buf))
    assert ours <= _best(lambda: buf.add_(torch.ops.aten.embedding_dense_backward(dy, ids, V, -1, False)))


@pytest.mark.parametrize("dtype,ids_dtype", [(torch.bfloat16, torch.int64), (torch.float16, torch.int32), (torch.float32, torch.int64)])
@pytest.mark.parametrize("shape,V,H", [((1,), 1, 8), ((16,), 50, 4096), ((3, 5), 7, 1032), ((0,), 3, 64), ((700,), 300, 72), ((300,), 64, 4104), ((9,), 5, 12), ((1535,), 30, 264),
                                       ((1537,), 30, 264), ((3, 1000), 9, 8), ((2500,), 40, 2048), ((2100,), 20, 2056), ((1001,), 16, 8200)])
def test_embedding_rows_are_copied(shape, V, H, dtype, ids_dtype):
    """A lookup without a gradient: few and many rows, rows that end within a block's share of pieces and that are no whole 16-byte pieces, ids in any shape and stride."""
    from realhf_b200.ops import functional as OF
    g = torch.Generator(device="cuda").manual_seed(V + H)
    w = torch.randn(V, H, device="cuda", generator=g).to(dtype)
    ids = torch.randint(0, V, shape, device="cuda", generator=g).to(ids_dtype)
    for i in (ids, ids.flip(0).transpose(0, -1), ids[..., ::2]):
        got = OF.embedding(i, w)
        assert got.dtype == dtype and torch.equal(got, w[i.long()])
    with torch.no_grad():
        assert torch.equal(OF.embedding(ids, torch.nn.Parameter(w)), w[ids.long()])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,H", [(1, 8), (1, 4096), (3, 264), (16, 8192), (148, 4104), (296, 1000), (297, 1000)])
def test_rms_norm_of_few_rows(rows, H, dtype):
    """A piece a thread up to two rows an SM, several beyond.  The sum of squares takes at most 8 + 5 + 5 roundings on a path, the square root and the products a few:
    2^-19 of the value, and half an ulp of the type for the result; the residual sum is rounded once."""
    from realhf_b200.ops import lib
    g = torch.Generator(device="cuda").manual_seed(rows + H)
    x, r, w = (torch.randn(n, device="cuda", generator=g).to(dtype) for n in ((rows, H), (rows, H), (H,)))
    for res, off in ((None, 0.0), (r, 1.0)):
        out = lib().rmsnorm_fwd(x, res, w, 1e-5, off)
        h = x if res is None else (x.float() + res.float()).to(dtype)
        if res is not None:
            assert torch.equal(out[2], h)
        rstd = (h.double().square().mean(-1) + 1e-5).rsqrt()
        want = h.double() * rstd[:, None] * (w.double() + off)
        bound = want.abs() * (2.0 ** -19 + torch.finfo(dtype).eps / 2) + (2.0 ** -24 if dtype == torch.float16 else 0)
        assert ((out[0].double() - want).abs() <= bound).all()
        assert ((out[1].double().flatten() - rstd).abs() <= rstd * 2.0 ** -19).all()


@pytest.mark.parametrize("T,V,H,dtype", [(20480, 50257, 768, torch.bfloat16), (20480, 1024, 1600, torch.float32), (65536, 100, 64, torch.bfloat16), (20480, 32000, 4096, torch.bfloat16)])
def test_embedding_rows_are_no_slower_than_the_library(T, V, H, dtype):
    """Many rows, narrow ones and such that do not fill their blocks among them (1.2 .. 9 times as fast when written), captured: 20 lookups in a row."""
    from realhf_b200.ops import lib
    w, ids = torch.randn(V, H, device="cuda").to(dtype), torch.randint(0, V, (T,), device="cuda")
    L, graphs = lib(), []
    for f in (lambda: L.embedding_rows(w, ids), lambda: torch.nn.functional.embedding(ids, w)):
        f()
        torch.cuda.synchronize()
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1]):
            for _ in range(20):
                f()
    assert _best(graphs[0].replay) <= _best(graphs[1].replay)


def test_embedding_gradient_finds_the_buffer_when_it_comes():
    """The buffer of the backward pass counts, not that of the forward pass; without one the gradient is the library's; ids of two forms; twice through one table."""
    from realhf_b200.ops import functional as OF
    g = torch.Generator(device="cuda").manual_seed(2)
    w = torch.nn.Parameter(torch.randn(40, 64, device="cuda", generator=g).bfloat16())
    ids = torch.randint(0, 40, (2, 30), device="cuda", generator=g)
    dy = torch.randint(-4, 5, (2, 30, 64), device="cuda", generator=g).bfloat16()      # sums are exact
    want = torch.zeros(40, 64, device="cuda").index_add_(0, ids.view(-1), dy.view(-1, 64).float()).bfloat16()
    first, second = torch.zeros_like(w), torch.ones_like(w)
    w.grad, w._grad_in_flat_buffer = first, True
    y = OF.embedding(ids, w)
    w.grad = second
    y.backward(dy)
    assert not first.any() and w.grad is second and torch.equal(second, want + 1)
    w.grad = first
    y = OF.embedding(ids, w)
    w.grad = None
    y.backward(dy)
    assert torch.equal(w.grad, want)
    w.grad = first
    (OF.embedding(ids, w) + OF.embedding(ids.t().int(), w).transpose(0, 1)).backward(dy)
    assert w.grad is first and torch.equal(first, 2 * want)
    with torch.no_grad():
        assert torch.equal(OF.embedding(ids, w), w[ids])


def _table(form):
    """A table with its gradient buffer as `ReaLModel.attach_grad_buffer` leaves it: in .grad, or in fp32 beside it with the hook that folds .grad into it."""
    g = torch.Generator(device="cuda").manual_seed(5)
    w = torch.nn.Parameter(torch.randn(40, 64, device="cuda", generator=g).bfloat16())
    ids = torch.randint(0, 40, (2, 30), device="cuda", generator=g)
    dy = torch.randint(-4, 5, (2, 30, 64), device="cuda", generator=g).bfloat16()
    want = torch.zeros(40, 64, device="cuda").index_add_(0, ids.view(-1), dy.view(-1, 64).float())
    if form == "grad":
        w.grad, w._grad_in_flat_buffer = torch.ones_like(w), True
        return w, ids, dy, want, w.grad
    w.main_grad = torch.ones(40, 64, device="cuda")

    def fold(p):
        if p.grad is not None:
            p.main_grad.add_(p.grad)
            p.grad = None
    w.register_post_accumulate_grad_hook(fold)
    w._main_grad_hooked = True
    return w, ids, dy, want, w.main_grad


@pytest.mark.parametrize("form", ["grad", "main_grad"])
def test_embedding_gradient_is_given_to_who_asks_for_it(form):
    """With a buffer attached: `torch.autograd.grad` returns the table's gradient and leaves the buffer alone, also twice differentiated and over a batch of gradients; hooks get
    it; a plain backward pass and one restricted to the table go into the buffer without a dense gradient."""
    from realhf_b200.ops import functional as OF
    w, ids, dy, want, buf = _table(form)
    one = buf.clone()
    got, = torch.autograd.grad(OF.embedding(ids, w), w, dy)
    assert torch.equal(got.float(), want) and torch.equal(buf, one)
    got, = torch.autograd.grad(OF.embedding(ids, w), w, torch.stack([dy, 2 * dy]), is_grads_batched=True)
    assert torch.equal(got.float(), torch.stack([want, 2 * want])) and torch.equal(buf, one)
    c = torch.ones((), device="cuda", requires_grad=True)
    first, = torch.autograd.grad(OF.embedding(ids, w), w, dy * c.bfloat16(), create_graph=True)
    second, = torch.autograd.grad(first.float().sum(), c)
    assert torch.equal(first.float(), want) and second.item() == dy.float().sum().item() and torch.equal(buf, one)

    OF.embedding(ids, w).backward(dy)
    assert torch.equal(buf.float(), want + 1)
    OF.embedding(ids, w).backward(dy, inputs=[w])
    assert torch.equal(buf.float(), 2 * want + 1)

    seen = []
    handle = w.register_hook(lambda g: seen.append(g.clone()))
    OF.embedding(ids, w).backward(dy)
    handle.remove()
    assert len(seen) == 1 and torch.equal(seen[0].float(), want) and torch.equal(buf.float(), 3 * want + 1)
    after = []
    handle = w.register_post_accumulate_grad_hook(lambda p: after.append(1))
    OF.embedding(ids, w).backward(dy)
    handle.remove()
    assert after == [1] and torch.equal(buf.float(), 4 * want + 1)
    node = w.view_as(w).grad_fn.next_functions[0][0]
    calls = []
    handle = node.register_hook(lambda *a: calls.append(a[1][0].clone()))
    OF.embedding(ids, w).backward(dy)
    handle.remove()
    assert len(calls) == 1 and torch.equal(calls[0].float(), want) and torch.equal(buf.float(), 5 * want + 1)


@pytest.mark.parametrize("form", ["grad", "main_grad"])
def test_embedding_gradient_of_a_plain_pass_is_not_dense(form):
    """A plain backward pass adds to the buffer by the kernels: nothing of the table's size is allocated."""
    from realhf_b200.ops import functional as OF
    w, ids, dy, want, buf = _table(form)
    big = torch.nn.Parameter(torch.zeros(200000, 64, device="cuda", dtype=torch.bfloat16))
    if form == "grad":
        big.grad, big._grad_in_flat_buffer = torch.zeros_like(big), True
    else:
        big.main_grad, big._main_grad_hooked = torch.zeros(200000, 64, device="cuda"), True
        big.register_post_accumulate_grad_hook(lambda p: None)
    y = OF.embedding(ids, big)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    y.backward(dy)
    assert torch.cuda.max_memory_allocated() - before < big.numel()
    assert torch.equal((big.grad if form == "grad" else big.main_grad)[:40].float(), want)


@pytest.mark.parametrize("form", ["grad", "main_grad"])
def test_embedding_gradient_of_two_streams(form):
    """Two lookups of one table on two streams: their gradients are added one after the other, as autograd orders its accumulation.  The second stream is kept behind the first by
    long work of its own on some passes and ahead of it on others; ids and gradients are such that both change the same rows."""
    from realhf_b200.ops import functional as OF
    g = torch.Generator(device="cuda").manual_seed(6)
    w = torch.nn.Parameter(torch.zeros(500, 512, device="cuda", dtype=torch.bfloat16))
    buf = torch.zeros(500, 512, device="cuda", dtype=torch.bfloat16 if form == "grad" else torch.float32)
    if form == "grad":
        w.grad, w._grad_in_flat_buffer = buf, True
    else:
        w.main_grad = buf
    ids = torch.randint(0, 500, (4000,), device="cuda", generator=g)
    dy = torch.randint(-1, 2, (4000, 512), device="cuda", generator=g).bfloat16()
    want = torch.zeros(500, 512, device="cuda").index_add_(0, ids, dy.float())
    side, load = torch.cuda.Stream(), torch.randn(2048, 2048, device="cuda")
    for k in range(6):
        buf.zero_()
        w.grad = buf if form == "grad" else None
        side.wait_stream(torch.cuda.current_stream())
        a = OF.embedding(ids, w)
        with torch.cuda.stream(side):
            b = OF.embedding(ids, w)
            for _ in range(k % 3):
                load = load @ load * 1e-3
        torch.autograd.backward([a, b], [dy, dy])
        torch.cuda.current_stream().wait_stream(side)
        total = buf.float() + (w.grad.float() if form == "main_grad" and w.grad is not None else 0)
        assert torch.equal(total, 2 * want)


def test_gradients_go_past_autograd_on_the_accumulating_stream_only():
    """Asked from backward passes on the stream that the leaf's accumulation belongs to (that of its first use) and on another one."""
    from realhf_b200.ops import lib
    w, said = torch.nn.Parameter(torch.zeros(4, 8, device="cuda")), []

    class Ask(torch.autograd.Function):
        @staticmethod
        def forward(ctx, w):
            ctx.w = w
            return w * 1

        @staticmethod
        def backward(ctx, dy):
            said.append(lib().gradient_goes_past(ctx.w, False))
            return dy

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    a = Ask.apply(w)
    with torch.cuda.stream(side):
        b = Ask.apply(w)
        b.sum().backward()
    torch.cuda.current_stream().wait_stream(side)
    a.sum().backward()
    assert said == [False, True] and torch.equal(w.grad, torch.full_like(w, 2.0))


@pytest.mark.parametrize("ids_dtype", [torch.int64, torch.int32])
@pytest.mark.parametrize("form", ["grad", "main_grad", "none"])
@pytest.mark.parametrize("rank", [0, 1])
def test_embedding_shard_leaves_rows_alone_that_no_token_reads(rank, form, ids_dtype, monkeypatch):
    """A shard of a table: tokens of the other shard are looked up as row 0 and blanked; they add nothing to row 0's gradient, not even zeros (a row of -0.0 stays)."""
    import types

    from realhf_b200.parallel import tp as TP
    monkeypatch.setattr(TP, "reduce_from_tp", lambda x, ctx: x)
    g = torch.Generator(device="cuda").manual_seed(rank)
    V, H, lo = 50, 72, 50 * rank
    ids = torch.randint(1, 100, (3, 400), device="cuda", generator=g)
    ids[ids == 50] = 51
    ids = ids.to(ids_dtype)
    here = (ids >= lo) & (ids < lo + V)
    w = torch.nn.Parameter(torch.randn(V, H, device="cuda", generator=g).bfloat16())
    buf = torch.full((V, H), -0.0, device="cuda", dtype=torch.float32 if form == "main_grad" else torch.bfloat16)
    if form == "grad":
        w.grad, w._grad_in_flat_buffer = buf, True
    elif form == "main_grad":
        w.main_grad = buf
    dy = torch.randint(-2, 3, (3, 400, H), device="cuda", generator=g).bfloat16()
    out = TP.vocab_parallel_embedding(ids, w, types.SimpleNamespace(tp_size=2, tp_rank=rank))
    assert torch.equal(out, torch.where(here.unsqueeze(-1), w[(ids - lo).clamp(0, V - 1).long()], torch.zeros((), device="cuda", dtype=torch.bfloat16)))
    out.backward(dy)
    got = w.grad if form == "none" else buf
    want = torch.zeros(V, H, device="cuda").index_add_(0, (ids - lo)[here].long(), dy[here].float())
    assert torch.equal(got.float(), want)
    assert form == "none" or bool(torch.signbit(buf[0]).all())


@pytest.mark.parametrize("form", ["grad", "main_grad"])
def test_launches_of_the_embedding_gradient_are_counted_when_they_come(form):
    """The lookup counts as one kernel, its gradient as those that the backward pass launched: none without one, none of ours when the library forms the gradient."""
    from realhf_b200.ops import functional as OF, launches
    w, ids, dy, _, _ = _table(form)
    launches.reset()
    y = OF.embedding(ids, w)
    assert launches.total == 1
    y.backward(dy)
    assert launches.total == 1 + 4 and launches.by_op["embedding_grad_"] == 4
    OF.embedding(ids[:, :5], w).backward(dy[:, :5])
    assert launches.total == 5 + 1 + 2                      # (up to 32 tokens: no long chains)
    torch.autograd.grad(OF.embedding(ids, w), w, dy)
    assert launches.total == 8 + 1
    launches.reset()
    launches.begin_capture()
    OF.embedding(ids, w).backward(dy)
    assert launches.end_capture() == 5 and launches.total == 0
    launches.reset()


@pytest.mark.parametrize("dtype,buffer", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16)])
def test_embedding_gradient_keeps_numbers_below_the_normal_ones(dtype, buffer):
    """Sums of subnormal numbers are exact, in short chains and in long ones, as in the sums of a plain lookup's gradient."""
    from realhf_b200.ops import lib
    tiny = 2.0 ** -130                                       # a multiple of bf16's smallest number too
    ids = torch.tensor([0] + [1] * 3 + [2] * 40 + [3] * 600, device="cuda")
    dy = torch.full((ids.numel(), 16), tiny, device="cuda").to(dtype)
    buf = torch.full((5, 16), tiny, device="cuda").to(buffer)
    lib().embedding_grad_(dy, ids, buf)
    want = torch.tensor([2.0, 4.0, 41.0, 601.0, 1.0], dtype=torch.float64, device="cuda") * tiny
    assert torch.equal(buf, want.to(buffer)[:, None].expand(5, 16))
