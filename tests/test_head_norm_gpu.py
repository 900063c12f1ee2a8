"""The per-head norms' kernels at the edges of their access widths: head sizes of one, two and four pieces of 128, sizes and row strides that no
four-element access fits, few rows (a row a warp) and many (several a warp) with a remainder."""
import pytest
import torch

from realhf_b200.api.model import WindowAttentionConfig
from realhf_b200.ops import attention as A
from realhf_b200.ops import recurrent as R

pytestmark = pytest.mark.gpu


def close(got, want, dtype):
    # both round the same fp32 value once; a sum of squares in another order moves it by a few fp32 ulps, at most one step of the storage type
    ulp = {torch.float32: 2.0 ** -20, torch.bfloat16: 2.0 ** -7, torch.float16: 2.0 ** -10}[dtype]
    assert float(((got.double().cpu() - want.double()).abs() / want.double().abs().clamp(min=1e-3)).max()) <= ulp


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("T,G,d,dv,pad", [(37, 3, 128, 128, 0), (4739, 2, 128, 128, 0), (4737, 3, 64, 100, 4), (3200, 3, 256, 132, 0), (9, 2, 128, 512, 0),
                                          (33, 2, 6, 10, 0), (33, 2, 128, 128, 1), (20, 2, 516, 64, 0)])
def test_value_norm_store_widths(T, G, d, dv, pad, dtype):
    a = WindowAttentionConfig(n_heads=2 * G, n_kv_heads=G, qk_dim=d, v_dim=dv, scale=0.1, window=16, keep_first=4)
    g = torch.Generator().manual_seed(T + dv)
    rows = torch.randn(T, 2 * G * d + G * (d + dv) + pad, generator=g).to(dtype)
    n = T // 2                                   # two sequences; the first in slot 1, the second not kept
    pos = torch.cat([torch.arange(n), torch.arange(T - n)]).int()
    slot = torch.cat([torch.ones(n), -torch.ones(T - n)]).int()
    remain = torch.cat([torch.arange(n - 1, -1, -1), torch.arange(T - n - 1, -1, -1)]).int()
    kc, vc = torch.zeros(3, G, 20, d, dtype=dtype), torch.zeros(3, G, 20, dv, dtype=dtype)
    want = A.value_norm_store_ref(rows, a, 1e-5, kc, vc, slot, pos, remain)
    dk, dvc = torch.zeros_like(kc, device="cuda"), torch.zeros_like(vc, device="cuda")
    got = A.value_norm_store(rows.cuda(), a, 1e-5, dk, dvc, slot.cuda(), pos.cuda(), remain.cuda())
    close(got, want, dtype)
    close(dvc, vc, dtype)
    assert torch.equal(dk.cpu(), kc)
    close(A.value_norm_store(rows.cuda(), a, 1e-5, None, None, None, pos.cuda(), None), want, dtype)


@pytest.mark.parametrize("act", ["silu", "sigmoid"])
@pytest.mark.parametrize("T,H,dv,off", [(3, 4, 128, 0), (2369, 4, 128, 8), (601, 16, 96, 0), (3159, 3, 200, 0), (5, 2, 512, 0), (7, 3, 516, 0), (9, 3, 10, 0),
                                        (50, 4, 64, 1)])
def test_gated_head_norm_widths(T, H, dv, off, act):
    g = torch.Generator().manual_seed(T + dv)
    o, w, wide = torch.randn(T, H, dv, generator=g), torch.randn(dv, generator=g).bfloat16(), torch.randn(T, H * dv + 16, generator=g).bfloat16()
    gate = lambda x: x[:, off:off + H * dv]
    want = R.gated_head_norm_ref(o, w, gate(wide), 1e-5, torch.bfloat16, act)
    close(R.gated_head_norm(o.cuda(), w.cuda(), gate(wide.cuda()), 1e-5, torch.bfloat16, act), want, torch.bfloat16)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("taps", [1, 3, 4, 5, 8])
@pytest.mark.parametrize("d,dv", [(64, 96), (200, 40)])
def test_delta_prepare_taps(d, dv, taps, dtype):
    from realhf_b200.api.model import DeltaRuleConfig
    from realhf_b200.models.sharding import delta_sections
    cfg = DeltaRuleConfig(n_heads=4, n_kv_heads=2, qk_dim=d, v_dim=dv, conv_taps=taps)
    g = torch.Generator().manual_seed(taps + d)
    lens = [5, 1, 77, 30]
    T, C = sum(lens), 4 * d + 4 * dv
    rn = lambda *s: torch.randn(*s, generator=g).to(dtype)
    proj, conv, A_log, bias = rn(T, sum(delta_sections(cfg))), rn(C, taps), rn(4), rn(4)
    pos = torch.cat([torch.arange(n) for n in lens]).int()
    remain = torch.cat([torch.arange(n - 1, -1, -1) for n in lens]).int()
    slot = torch.cat([torch.full((n,), s) for n, s in zip(lens, [2, -1, 0, 3])]).int()
    st = torch.zeros(4, max(taps - 1, 1), C)
    c_st = st.clone().cuda()
    args = (st if taps > 1 else None, slot, remain) if taps > 1 else (None, None, None)
    want = R.delta_prepare_ref(proj, conv, A_log, bias, cfg, pos, *args)
    got = R.delta_prepare(proj.cuda(), conv.cuda(), A_log.cuda(), bias.cuda(), cfg, pos.cuda(), c_st if taps > 1 else None,
                          slot.cuda() if taps > 1 else None, remain.cuda() if taps > 1 else None)
    # fp32 on both sides, up to eight products of unit size and their sum's cancellation before a unit-length division
    assert float((got.cpu() - want).abs().max()) <= 2.0 ** -17 * float(want.abs().max())
    if taps > 1:
        assert torch.equal(c_st.cpu(), st)


@pytest.mark.parametrize("T", [100, 9000])
@pytest.mark.parametrize("taps", [3, 8])
def test_delta_prepare_is_the_same_for_every_type(taps, T):
    """Inputs that all three types hold exactly: everything behind the loads is fp32, so the results are the same bits."""
    from realhf_b200.api.model import DeltaRuleConfig
    from realhf_b200.models.sharding import delta_sections
    cfg = DeltaRuleConfig(n_heads=4, n_kv_heads=2, qk_dim=16, v_dim=24, conv_taps=taps)
    g = torch.Generator().manual_seed(taps)
    rn = lambda *s: (torch.randint(-63, 64, s, generator=g) / 32).cuda()
    args = [rn(T, sum(delta_sections(cfg))), rn(4 * 16 + 4 * 24, taps), rn(4), rn(4)]
    pos = torch.cat([torch.arange(41), torch.arange(T - 41)]).int().cuda()
    got = [R.delta_prepare(*(a.to(dt) for a in args), cfg, pos, None, None, None) for dt in (torch.float32, torch.bfloat16, torch.float16)]
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])


@pytest.mark.parametrize("taps", [2, 4, 7])
def test_delta_prepare_many_tokens(taps):
    """Enough tokens that a warp walks 32 of them: sequences that begin and end inside its tiles of 8, a remainder of tokens, the final inputs kept."""
    from realhf_b200.api.model import DeltaRuleConfig
    from realhf_b200.models.sharding import delta_sections
    cfg = DeltaRuleConfig(n_heads=4, n_kv_heads=2, qk_dim=16, v_dim=24, conv_taps=taps)
    g = torch.Generator().manual_seed(taps)
    lens = [3000, 1, 2, 33, 31, 7, 5900]
    T, C = sum(lens), 4 * 16 + 4 * 24
    rn = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16)
    proj, conv, A_log, bias = rn(T, sum(delta_sections(cfg))), rn(C, taps), rn(4), rn(4)
    pos = torch.cat([torch.arange(n) for n in lens]).int()
    remain = torch.cat([torch.arange(n - 1, -1, -1) for n in lens]).int()
    slot = torch.cat([torch.full((n,), s) for n, s in zip(lens, [2, -1, 0, 3, 1, 5, 4])]).int()
    st = torch.zeros(6, taps - 1, C)
    c_st = st.clone().cuda()
    want = R.delta_prepare_ref(proj, conv, A_log, bias, cfg, pos, st, slot, remain)
    got = R.delta_prepare(proj.cuda(), conv.cuda(), A_log.cuda(), bias.cuda(), cfg, pos.cuda(), c_st, slot.cuda(), remain.cuda())
    assert float((got.cpu() - want).abs().max()) <= 2.0 ** -17 * float(want.abs().max())      # the bound of the test above
    assert torch.equal(c_st.cpu(), st)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("G,d,dv,norm", [(3, 128, 128, True), (4, 64, 72, True), (5, 40, 8, False)])
def test_value_norm_of_many_tokens(G, d, dv, norm, dtype):
    """Half a warp a (token, head) unit: unit counts that leave the last block partly empty, values narrower and wider than keys, rows of the cache that later
    tokens overwrite.  Bound: one rounding to the type on each side of the same fp32 value, whose sums differ by a few 2^-24: one unit in the last place."""
    from realhf_b200.api.model import WindowAttentionConfig
    from realhf_b200.ops import attention as A
    a = WindowAttentionConfig(n_heads=G, n_kv_heads=G, qk_dim=d, v_dim=dv, scale=1.0, window=30, keep_first=4, value_norm=norm, out_gate=False)
    g = torch.Generator().manual_seed(G)
    lens = [9000 // G, 1000, 1, 77, 1500]
    T = sum(lens)
    x = torch.randn(T, G * (2 * d + dv), generator=g).to(dtype)
    pos = torch.cat([torch.arange(n) for n in lens]).int()
    remain = torch.cat([torch.arange(n - 1, -1, -1) for n in lens]).int()
    slot = torch.cat([torch.full((n,), s) for n, s in zip(lens, [2, -1, 0, 3, 1])]).int()
    kc, vc = torch.zeros(4, G, 40, d, dtype=dtype), torch.zeros(4, G, 40, dv, dtype=dtype)
    k2, v2 = kc.clone().cuda(), vc.clone().cuda()
    want = A.value_norm_store(x, a, 1e-5, kc, vc, slot, pos, remain)
    got = A.value_norm_store(x.cuda(), a, 1e-5, k2, v2, slot.cuda(), pos.cuda(), remain.cuda())
    rel = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -10
    for w, f in ((want, got), (vc, v2)):
        assert bool(((f.cpu().double() - w.double()).abs() <= rel * w.double().abs()).all())
    assert torch.equal(k2.cpu(), kc)
