"""Fused sampling kernel vs the PyTorch reference filter: same kept set (mask), consistent log-probs, valid samples."""
import math

import pytest
import torch

from realhf_b200.api.model import GenerationHyperparameters
from realhf_b200.models import generation as gen
from realhf_b200.ops import functional as OF
from realhf_b200.ops import lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("cfg", [(1000, 0.9, 1.0), (50, 1.0, 0.7), (32000, 0.5, 1.3), (200, 0.95, 1.0)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_sample_matches_reference_filter(cfg, dtype):
    top_k, top_p, temp = cfg
    torch.manual_seed(0)
    B, V = 64, 32000
    logits = (torch.randn(B, V, device=DEV) * 2.5).to(dtype)
    g = GenerationHyperparameters(max_new_tokens=8, min_new_tokens=4, top_k=top_k, top_p=top_p, temperature=temp)
    unfinished = torch.ones(B, dtype=torch.bool, device=DEV)
    unfinished[3] = False
    tok, lp, mb = lib().sample(logits, unfinished, top_k, top_p, 1.0 / temp, 2, True, False, 0, 1234, 1, True)
    # reference keep-set
    x = logits.float() / temp
    x[:, 2] = torch.finfo(torch.float32).min
    xf = gen._filter_logits(x.clone(), g)
    ref_removed = xf == torch.finfo(torch.float32).min
    removed = OF.unpack_mask_bits(mb, V)
    # ties / fp rounding at the top-p boundary may move a handful of tokens
    # (bf16 logits have large tie groups; which members of the boundary group survive is sort-order dependent,
    # so mismatches must be confined to at most two tied values per row: the top-k and the top-p boundary)
    mism = removed != ref_removed
    for r in torch.nonzero(mism.sum(1) > 2).flatten().tolist():
        assert x[r][mism[r]].unique().numel() <= 2, (r, x[r][mism[r]])
    lp_ref = torch.log_softmax(x.masked_fill(removed, float("-inf")), -1)  # log-probs under the kernel's own keep-set
    rows = torch.arange(B, device=DEV)
    live = unfinished
    assert (~removed[rows, tok])[live].all(), "sampled a filtered token"
    torch.testing.assert_close(lp[live], lp_ref[rows, tok][live], atol=2e-3, rtol=1e-3)
    assert tok[3].item() == 0 and lp[3].item() == 0.0


def test_sample_distribution_and_greedy():
    torch.manual_seed(0)
    V = 4096
    base = torch.randn(1, V, device=DEV)
    logits = base.repeat(4096, 1)
    tok, lp, _ = lib().sample(logits, None, 8, 1.0, 1.0, -1, False, False, 0, 99, 0, False)
    top = torch.topk(base[0], 8)
    p_ref = torch.softmax(top.values, 0)
    counts = torch.stack([(tok == i).sum() for i in top.indices]).float()
    assert counts.sum().item() == 4096
    torch.testing.assert_close(counts / 4096, p_ref, atol=0.03, rtol=0.2)
    tok, lp, _ = lib().sample(logits[:8], None, 8, 1.0, 1.0, -1, False, True, 0, 99, 0, False)
    assert (tok == base[0].argmax()).all()
    torch.testing.assert_close(lp, torch.log_softmax(base[0], 0)[tok], atol=1e-3, rtol=1e-3)


def _tiny_llama():
    from realhf_b200.api.model import ReaLModelConfig
    from realhf_b200.models.real_model import ReaLModel
    from realhf_b200.ops import gemm as G
    OF.set_gemm_impl(G.linear)
    cfg = ReaLModelConfig(n_layers=2, n_kv_heads=4, n_q_heads=8, hidden_dim=1024, intermediate_dim=2816, vocab_size=32000, n_positions=2048,
                          embd_pdrop=0.0, resid_pdrop=0.0, attn_pdrop=0.0, activation_function="silu", scale_attn_by_inverse_layer_idx=False,
                          use_attention_bias=False, use_attn_proj_bias=False, use_mlp_bias=False, layer_norm_type="rms", mlp_type="llama",
                          apply_rotary=True)
    m = ReaLModel(cfg, dtype=torch.bfloat16, device=torch.device(DEV)).init_random_fast(std=0.05)
    for p in m.parameters():
        p.requires_grad_(False)
    return m.eval()


@pytest.mark.parametrize("greedy", [True, False])
def test_in_graph_sampling_matches_eager_decode_loop(greedy, monkeypatch):
    """The sampling kernel as the tail of the captured decode step (device-side step counters, history buffers, next-token
    feed, EOS bookkeeping) must reproduce the eager loop: exactly for greedy decoding; for sampling the log-probs must be those
    of the sampled tokens under the model (teacher-forced forward) and EOS / padding semantics must hold."""
    m = _tiny_llama()
    lens = [5, 17, 9, 30]
    ids = torch.randint(3, 32000, (sum(lens),), device=DEV)
    cu = torch.tensor([0, 5, 22, 31, 61], dtype=torch.int32, device=DEV)
    g = GenerationHyperparameters(max_new_tokens=24, min_new_tokens=6, greedy=greedy, top_k=50, top_p=0.9, temperature=0.8,
                                  use_cuda_graph=True, force_cudagraph_recapture=True)
    outs = {}
    for mode in ("1", "0"):
        monkeypatch.setenv("REAL_GEN_SAMPLE_IN_GRAPH", mode)
        gen.seed_sampling(7)
        outs[mode], _ = gen.generate(m, ids, cu, g, eos_id=2, pad_id=0)
    a, b = outs["1"], outs["0"]
    assert a.tokens.shape == b.tokens.shape == (4, 24)
    if greedy:
        assert torch.equal(a.tokens, b.tokens)
        torch.testing.assert_close(a.logprobs, b.logprobs, atol=1e-3, rtol=1e-3)
        assert torch.equal(a.gen_lens, b.gen_lens)
        return
    # sampling: teacher-forced check of the in-graph path
    assert a.mask_bits is not None and a.mask_bits.shape == (4, 24, 4000)
    for i, L in enumerate(lens):
        n = int(a.gen_lens[i])
        seq = torch.cat([ids[int(cu[i]): int(cu[i + 1])], a.tokens[i, :n]])
        out = m(input_ids=seq, cu_seqlens=torch.tensor([0, seq.numel()], dtype=torch.int32, device=DEV), max_seqlen=int(seq.numel()))
        lg = out.logits.float()[L - 1: L - 1 + n] / 0.8
        removed = OF.unpack_mask_bits(a.mask_bits[i, :n], 32000)
        assert not removed[torch.arange(n), a.tokens[i, :n]].any(), "sampled a filtered token"
        lp_ref = torch.log_softmax(lg.masked_fill(removed, float("-inf")), -1)[torch.arange(n), a.tokens[i, :n]]
        torch.testing.assert_close(a.logprobs[i, :n], lp_ref, atol=0.08, rtol=0.05)  # bf16 decode vs packed forward
        assert (a.tokens[i, :min(n, 6) - 1] != 2).all()          # EOS suppressed before min_new_tokens
        assert (a.tokens[i, n:] == 0).all() and (a.logprobs[i, n:] == 0).all()  # padding after EOS


@pytest.mark.parametrize("V,top_k,top_p", [(97, 96, 0.5), (2048, 256, 0.9), (4099, 1, 1.0), (32000, 512, 0.95), (32003, 513, 0.8), (50257, 50, 0.9),
                                           (51200, 200, 1.0), (8192, 8192, 0.7)])
@pytest.mark.parametrize("ties", [False, True])
def test_sample_thresholds_at_the_edges_of_the_candidate_path(V, top_k, top_p, ties):
    """Kept set, draw and log-prob against float64 at both sides of the top_k limit, with unaligned rows and with tie groups that overflow
    the candidate list.  The mask may differ only where the mass above an element is within fp32 rounding of top_p (1e-5 of the total)."""
    torch.manual_seed(V + top_k)
    B = 6
    x = torch.randn(B, V, device=DEV) * 2.0
    if ties:
        x = (x * 2).round() / 2                      # a few dozen values: tie groups of hundreds to thousands of elements
    tok, lp, mb = lib().sample(x, None, top_k, top_p, 1.0, -1, False, False, 0, 77, 3, True)
    xd = x.double()
    kth = torch.topk(xd, min(top_k, V), -1).values[:, -1:]
    p = torch.softmax(xd.masked_fill(xd < kth, float("-inf")), -1)
    srt, idx = torch.sort(xd, -1, descending=True)
    before = p.gather(1, idx).cumsum(-1) - p.gather(1, idx)
    first = torch.searchsorted(-srt, -srt)           # equal logits share the mass above the first of them
    above = torch.zeros_like(p).scatter_(1, idx, before.gather(1, first))
    keep = (p > 0) & ((above < top_p) if top_p < 1 else torch.ones_like(above, dtype=torch.bool))
    removed = OF.unpack_mask_bits(mb, V)
    sure = (above - top_p).abs() > 1e-5
    assert torch.equal(removed[sure | (p == 0)], ~keep[sure | (p == 0)])
    rows = torch.arange(B, device=DEV)
    assert not removed[rows, tok].any()
    ref = torch.log_softmax(xd.masked_fill(removed, float("-inf")), -1)[rows, tok]
    torch.testing.assert_close(lp.double(), ref, atol=2e-5, rtol=1e-5)


@pytest.mark.parametrize("V", [500, 2048, 32003])
@pytest.mark.parametrize("top_k,top_p", [(50, 0.9), (600, 1.0), (None, 1.0), (None, 0.9)])
def test_sample_without_a_finite_mass_takes_the_last_kept_element(V, top_k, top_p):
    """Rows whose kept elements have no probability to draw from (all -infinity, all NaN, a +infinity among finite ones): the last element that the mask
    keeps, as an index inside the row.  Beside them ordinary rows with -infinity in them, which must never draw one."""
    top_k = min(top_k or V, V)
    torch.manual_seed(V)
    x = torch.randn(6, V, device=DEV) * 2
    x[0] = float("-inf")
    x[1] = float("nan")
    x[2, 7] = float("inf")
    x[3, ::2] = float("-inf")
    x[4, 3:] = float("-inf")
    tok, lp, mb = lib().sample(x, None, top_k, top_p, 1.0, -1, False, False, 0, 5, 3, True)
    kept = ~OF.unpack_mask_bits(mb, V)
    last = (V - 1 - kept.flip(1).int().argmax(1)).tolist()
    assert kept.any(1).all() and tok[:3].tolist() == last[:3]
    rows = torch.arange(3, 6, device=DEV)
    assert torch.isfinite(x[rows, tok[3:]]).all() and torch.isfinite(lp[3:]).all() and kept[rows, tok[3:]].all()


@pytest.mark.parametrize("V", [31, 1000, 2048, 4099, 32003, 51200])
def test_sample_unfiltered_draws_by_inverse_cdf(V):
    """No filter: the draw over the whole row.  Logits of one element far above the rest, in every group of a row in turn, and a flat row, whose draws
    over many seeds cover it evenly; the mask removes nothing and ends at the last byte."""
    at = torch.arange(0, V, max(1, V // 97), device=DEV)
    x = torch.randn(at.numel(), V, device=DEV)
    x[torch.arange(at.numel(), device=DEV), at] = 60.0
    tok, lp, mb = lib().sample(x, None, V, 1.0, 1.0, -1, False, False, 0, 9, 1, True)
    assert torch.equal(tok, at) and float(lp.abs().max()) < 1e-6 and int(mb.sum()) == 0
    flat = torch.zeros(4096, V, device=DEV, dtype=torch.bfloat16)
    tok, lp, _ = lib().sample(flat, None, V, 1.0, 1.0, -1, False, False, 0, 9, 1, False)
    torch.testing.assert_close(lp, torch.full_like(lp, -math.log(V)), atol=2e-5, rtol=1e-5)
    # 4096 draws in 16 equal parts of the row (V 31: each part is two elements or one): a part's count is binomial, five standard deviations
    part = tok * 16 // V
    share = torch.bincount(torch.arange(V, device=DEV) * 16 // V, minlength=16).double() / V
    count = torch.bincount(part, minlength=16).double()
    assert ((count - 4096 * share).abs() <= 5 * (4096 * share * (1 - share)).sqrt()).all()


@pytest.mark.parametrize("V,top_k", [(1000, 200), (1003, 126), (264, 60)])
def test_sample_with_fewer_thread_maxima_than_top_k(V, top_k):
    """16-byte loads of 16-bit logits leave V / 8 thread maxima: with fewer than top_k of them nothing bounds the candidates."""
    torch.manual_seed(V)
    x = (torch.randn(5, V, device=DEV) * 2).to(torch.bfloat16)
    _, _, mb = lib().sample(x, None, top_k, 1.0, 1.0, -1, False, False, 0, 5, 3, True)
    kth = torch.topk(x.float(), top_k, -1).values[:, -1:]
    assert torch.equal(OF.unpack_mask_bits(mb, V), x.float() < kth)


@pytest.mark.parametrize("top_k", [63, 64, 65, 127, 128, 129, 512])
@pytest.mark.parametrize("V,dtype", [(32000, torch.bfloat16), (2051, torch.float32), (8192, torch.float16)])
def test_sample_at_the_group_sizes_of_the_bound(V, dtype, top_k):
    """The bound of the candidates comes from 256, 512 or 1024 maxima, by top_k: the kept set on both sides of each change, with ties at the threshold."""
    torch.manual_seed(V + top_k)
    x = (torch.randn(7, V, device=DEV) * 2).to(dtype)
    tok, _, mb = lib().sample(x, None, top_k, 1.0, 1.0, -1, False, False, 0, 5, 3, True)
    kth = torch.topk(x.float(), top_k, -1).values[:, -1:]
    removed = OF.unpack_mask_bits(mb, V)
    assert torch.equal(removed, x.float() < kth) and not removed[torch.arange(7, device=DEV), tok].any()


@pytest.mark.parametrize("greedy", [True, False])
@pytest.mark.parametrize("eos,pad", [(5, 0), (5, 5), (-1, 0)])
def test_sample_next_says_which_rows_go_on(eos, pad, greedy):
    """The last output against the expression it stands for: rows that draw eos, rows that draw another token, finished rows, padding that is eos itself, no eos."""
    B, V = 64, 1000
    x = torch.zeros(B, V, device=DEV)
    x[torch.arange(B, device=DEV), torch.tensor([5, 6, 7, 0], device=DEV).repeat(B // 4)] = 60.0
    live = torch.arange(B, device=DEV) % 3 != 0
    tok, _, _, goes_on = lib().sample_next(x, live, V if greedy else 50, 1.0, 1.0, eos, False, greedy, pad, 3, 1, False)
    assert torch.equal(tok, torch.where(live, x.argmax(-1), pad)) and goes_on.dtype == torch.bool
    assert torch.equal(goes_on, live & (tok != eos))
    assert torch.equal(lib().sample_next(x, None, 50, 1.0, 1.0, eos, False, greedy, pad, 3, 1, False)[3], x.argmax(-1) != eos)
