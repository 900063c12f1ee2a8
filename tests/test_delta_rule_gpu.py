"""The delta rule's kernel where its bookkeeping can go wrong: decays whose product leaves the range it is carried in (0, tiny, 1, above 1),
head sizes at and between the kernel's lane groups, columns that do not fill a group, empty and one-token sequences, both kinds of decay, and
decode steps that go on from a prompt's state."""
import pytest
import torch

from realhf_b200.api.model import DeltaRuleConfig
from realhf_b200.ops import recurrent as R

pytestmark = pytest.mark.gpu
LENS = [1, 9, 0, 70, 33]


def inputs(d, dv, decays, channel, n, seed):
    g = torch.Generator().manual_seed(seed)
    H, G = 4, 2
    unit = lambda x: torch.nn.functional.normalize(x, dim=-1)
    q, k, v = unit(torch.randn(n, G, d, generator=g)), unit(torch.randn(n, G, d, generator=g)), torch.randn(n, H, dv, generator=g)
    r = torch.rand(n, H * d if channel else H, generator=g)
    decay = {"one": torch.ones_like(r), "mixed": 0.1 + 0.9 * r, "zeros": torch.where(r < 0.2, 0.0, r), "tiny": torch.where(r < 0.3, 1e-30 * r, r),
             "growing": 0.9 + 0.4 * r}[decays]
    cfg = DeltaRuleConfig(n_heads=H, n_kv_heads=G, qk_dim=d, v_dim=dv, conv_taps=1, **(dict(decay_rank=8) if channel else {}))
    return cfg, torch.cat([q.reshape(n, -1), k.reshape(n, -1), v.reshape(n, -1), torch.rand(n, H, generator=g), decay], -1)


@pytest.mark.parametrize("d,dv", [(16, 8), (32, 40), (48, 20), (64, 130), (128, 128), (200, 70), (256, 17), (512, 24)])
@pytest.mark.parametrize("decays,channel", [("one", False), ("mixed", False), ("zeros", False), ("tiny", False), ("growing", False), ("mixed", True),
                                            ("zeros", True)])
def test_delta_rule_decays_and_shapes(d, dv, decays, channel):
    cfg, u = inputs(d, dv, decays, channel, sum(LENS) + 3, d + dv)
    cu = torch.tensor([0] + LENS).cumsum(0).int()
    slots = torch.tensor([4, 0, 2, -1, 3], dtype=torch.int32)
    pick = torch.tensor([0, 4, 3], dtype=torch.int32)            # three decode steps, one on an untouched slot
    n = sum(LENS)

    def run(u, native):
        dev = u.device
        S = torch.full((6, 4, d, dv), 0.25, dtype=u.dtype, device=dev)
        scan, step = (R.delta_rule_scan, R.delta_rule_step) if native else (R.delta_rule_scan_ref, R.delta_rule_step_ref)
        args = cu.to(dev), S, slots.to(dev)
        o = scan(u[:n], cfg, *args)
        o2 = step(u[n:], cfg, S, pick.to(dev))
        return torch.cat([o, o2]).double().cpu(), S.double().cpu()

    want = run(u.double(), False)
    plain, got = run(u, False), run(u.cuda(), True)
    for w, f, x in zip(want, plain, got):
        # The yardstick is fp32's own rounding: the plain fp32 recurrence's largest error, four times it for another order of sums and the
        # decays' product, plus a few ulps of the largest value.
        assert float((x - w).abs().max()) <= 4 * float((f - w).abs().max()) + 8 * 2.0 ** -23 * float(w.abs().max())


@pytest.mark.parametrize("d,dv,n_seqs", [(32, 64, 36), (32, 64, 37), (24, 130, 13), (64, 64, 40), (128, 128, 3), (128, 130, 3)])
def test_delta_rule_on_both_sides_of_the_sequence_count(d, dv, n_seqs):
    """Head sizes up to 32 change kernels with the number of CTAs (36 and 37 sequences x 4 heads lie on either side), and the final state is written four columns
    at a time or one by one."""
    lens = [3 + i % 7 for i in range(n_seqs)]
    cfg, u = inputs(d, dv, "mixed", False, sum(lens), n_seqs)
    cu, slots = torch.tensor([0] + lens).cumsum(0).int(), torch.arange(n_seqs, dtype=torch.int32).flip(0)

    def run(u, scan):
        S = torch.zeros(n_seqs, 4, d, dv, dtype=u.dtype, device=u.device)
        return scan(u, cfg, cu.to(u.device), S, slots.to(u.device)).double().cpu(), S.double().cpu()
    want, plain, got = run(u.double(), R.delta_rule_scan_ref), run(u, R.delta_rule_scan_ref), run(u.cuda(), R.delta_rule_scan)
    for w, f, x in zip(want, plain, got):      # the bound of the test above
        assert float((x - w).abs().max()) <= 4 * float((f - w).abs().max()) + 8 * 2.0 ** -23 * float(w.abs().max())


@pytest.mark.parametrize("keys", ["shifted", "nearly_constant"])
@pytest.mark.parametrize("d,dv", [(128, 128), (64, 64)])
def test_delta_rule_of_keys_that_point_the_same_way(keys, d, dv):
    """Unit keys far from orthogonal, write strengths near 1, no decay: a token takes back most of what the one before wrote, so errors of earlier tokens only
    stay small where each token works from the state as it was rounded.  Yardstick: the plain fp32 recurrence, token by token; sums in another order and a
    k . q shared by the columns leave the same number of roundings of the same sizes, so the 2-norm of the error at most doubles."""
    n, H, G = 512, 4, 2
    g = torch.Generator().manual_seed(d)
    rn = lambda *s: torch.randn(*s, generator=g)
    if keys == "shifted":
        qk = torch.nn.functional.silu(rn(2, n, G, d) + 2)
    else:
        qk = rn(1, 1, G, d) + 0.1 * rn(2, n, G, d)
    q, k = torch.nn.functional.normalize(qk, dim=-1)
    cfg = DeltaRuleConfig(n_heads=H, n_kv_heads=G, qk_dim=d, v_dim=dv, conv_taps=1)
    u = torch.cat([q.reshape(n, -1), k.reshape(n, -1), rn(n, H * dv), 0.98 + 0.02 * torch.rand(n, H, generator=g), torch.ones(n, H)], -1)
    cu, slots = torch.tensor([0, n], dtype=torch.int32), torch.zeros(1, dtype=torch.int32)

    def run(u, scan):
        S = torch.zeros(1, H, d, dv, dtype=u.dtype, device=u.device)
        return scan(u, cfg, cu.to(u.device), S, slots.to(u.device)).double().cpu(), S.double().cpu()
    want, plain, got = run(u.double(), R.delta_rule_scan_ref), run(u, R.delta_rule_scan_ref), run(u.cuda(), R.delta_rule_scan)
    for w, f, x in zip(want, plain, got):
        assert float((x - w).norm()) <= 2 * float((f - w).norm()), (float((x - w).norm() / w.norm()), float((f - w).norm() / w.norm()))


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("column", ["k", "v", "beta", "g"])
@pytest.mark.parametrize("d,dv", [(128, 128), (128, 124), (64, 64)])
def test_delta_rule_tokens_before_a_non_finite_one(d, dv, column, bad):
    """A value that is not finite reaches its own and later tokens of its sequence and heads, nothing else: the rest is bit for bit what it is without it."""
    lens, at = [100, 90], 70
    cfg, u = inputs(d, dv, "mixed", False, sum(lens), d + dv)
    H, nqk = 4, 2 * d
    first = {"k": nqk, "v": 2 * nqk, "beta": 2 * nqk + H * dv, "g": 2 * nqk + H * dv + H}[column]      # key of head group 0, value / gates of head 0
    dirty = u.clone()
    dirty[at, first] = bad
    cu = torch.tensor([0] + lens).cumsum(0).int().cuda()
    a, b = (R.delta_rule_scan(x.cuda(), cfg, cu) for x in (u, dirty))
    heads = 2 if column == "k" else 1
    assert torch.equal(a[:at], b[:at]) and torch.equal(a[lens[0]:], b[lens[0]:]) and torch.equal(a[:, heads:], b[:, heads:])
    assert not bool(torch.isfinite(b[at:lens[0], :heads]).all())
