"""Tile-level emulation of the tcgen05 attention kernels (csrc/attn_fwd_tcgen05.cu, attn_bwd_tcgen05.cu) in PyTorch.

The kernels' ALGORITHM -- which key tiles an item of two query tiles walks and which of the two takes part in each, mask predicates, the output that
accumulates over the stream and is scaled when a row's maximum grows, the LSE convention, the transposed dKV pass with per-column
statistics, the 64-row streamed blocks, the GQA head loop -- is mirrored here (same names, same predicates, bf16 rounding of P / dS where the
kernels round) and checked against the plain fp32 reference and its autograd, or for the walk against the visible keys themselves.  A mistake in
any of those shows up here; what this cannot check is the hardware protocol (barriers, descriptors, swizzles)."""
import math

import pytest
import torch

from realhf_b200.ops.attention import varlen_attention_ref

LOG2E = 1.4426950408889634
kBQ = kBKV = 128   # forward tiles
kR, kX = 128, 64   # backward: resident rows, streamed rows


def _bf16(x):
    return x.to(torch.bfloat16).float()


def emulate_fwd(q, k, v, cu, scale, causal):
    """Per (sequence, head, 128-row q tile); scores in the log2 domain; returns out [T,nq,D] and lse [nq,T]."""
    T, nq, D = q.shape
    nkv = k.shape[1]
    out = torch.zeros(T, nq, D)
    lse = torch.zeros(nq, T)
    sl2 = scale * LOG2E
    for seq in range(len(cu) - 1):
        tok0, L = cu[seq], cu[seq + 1] - cu[seq]
        for head in range(nq):
            hk = head // (nq // nkv)
            for qt in range((L + kBQ - 1) // kBQ):
                q0 = qt * kBQ
                kv_len = min(L, q0 + kBQ) if causal else L
                n_kv = (kv_len + kBKV - 1) // kBKV
                rows = torch.arange(kBQ)
                q_pos = q0 + rows
                # TMA box: rows past the end of the packed tensor are zero-filled, rows of the next sequence are real data
                Q = torch.zeros(kBQ, D)
                n_in = min(kBQ, T - (tok0 + q0))
                Q[:n_in] = q[tok0 + q0: tok0 + q0 + n_in, head]
                m_run = torch.full((kBQ,), -math.inf)
                l_run = torch.zeros(kBQ)
                O = torch.zeros(kBQ, D)
                for j in range(n_kv):
                    kv0 = j * kBKV
                    K = torch.zeros(kBKV, D)
                    V = torch.zeros(kBKV, D)
                    n_in = min(kBKV, T - (tok0 + kv0))
                    K[:n_in] = k[tok0 + kv0: tok0 + kv0 + n_in, hk]
                    V[:n_in] = v[tok0 + kv0: tok0 + kv0 + n_in, hk]
                    S = Q @ K.t()
                    need_mask = (kv0 + kBKV > L) or (causal and kv0 + kBKV - 1 > q0)
                    lim = (torch.minimum(torch.tensor(L), q_pos + 1) if causal else torch.full((kBQ,), L)) - kv0
                    cols = torch.arange(kBKV)
                    masked = need_mask & (cols[None, :] >= lim[:, None])
                    S = S.masked_fill(masked, -math.inf)
                    mx = S.max(dim=1).values * sl2                     # the scale is positive: the maximum is taken over the raw products
                    m_new = torch.maximum(m_run, mx)
                    alpha = torch.where(m_new == m_run, torch.ones_like(m_new), torch.exp2(m_run - m_new))
                    l_run = l_run * alpha
                    O = O * alpha[:, None]                             # (the kernel skips this while no row of a warp has grown)
                    m_run = m_new
                    neg_m = torch.where(torch.isinf(m_run), torch.zeros_like(m_run), -m_run)
                    P = torch.exp2(S * sl2 + neg_m[:, None])
                    l_run = l_run + P.sum(1)
                    O = O + _bf16(P) @ V                               # P is rounded to bf16 before the second product
                ok = q_pos < L
                out[tok0 + q_pos[ok], head] = (O / l_run[:, None])[ok]
                lse[head, tok0 + q_pos[ok]] = (m_run * math.log(2) + torch.log(l_run))[ok]
    return out, lse


def _delta(out, dout):
    return (out * dout).sum(-1).t().contiguous()  # [nq, T]


def _load_rows(x, row0, n, head, T):
    """TMA box of n rows starting at row0 of x[:, head]: zero fill past the end of the packed tensor."""
    D = x.shape[-1]
    tile = torch.zeros(n, D)
    n_in = max(0, min(n, T - row0))
    tile[:n_in] = x[row0: row0 + n_in, head]
    return tile


def emulate_bwd(q, k, v, out, dout, lse, cu, scale, causal):
    T, nq, D = q.shape
    nkv = k.shape[1]
    G = nq // nkv
    delta = _delta(out, dout)
    sl2 = scale * LOG2E
    dq, dk, dv = torch.zeros_like(q), torch.zeros_like(k), torch.zeros_like(v)
    for seq in range(len(cu) - 1):
        tok0, L = cu[seq], cu[seq + 1] - cu[seq]
        nblk_all = (L + kX - 1) // kX
        for tile in range((L + kR - 1) // kR):
            r0 = tile * kR
            r_pos = r0 + torch.arange(kR)
            # ---------------- dKV pass: lanes are keys
            for head in range(nkv):
                Kt, Vt = _load_rows(k, tok0 + r0, kR, head, T), _load_rows(v, tok0 + r0, kR, head, T)
                blk0 = r0 // kX if causal else 0
                nblk = nblk_all - blk0
                accV, accK = torch.zeros(kR, D), torch.zeros(kR, D)
                for t in range(nblk * G):
                    h, blk = head * G + t // nblk, blk0 + t % nblk
                    x0 = blk * kX
                    Qx, dOx = _load_rows(q, tok0 + x0, kX, h, T), _load_rows(dout, tok0 + x0, kX, h, T)
                    qpos = x0 + torch.arange(kX)
                    inb = qpos < L
                    lse_c = torch.full((kX,), math.inf)
                    del_c = torch.zeros(kX)
                    lse_c[inb] = lse[h, tok0 + qpos[inb]] * LOG2E
                    del_c[inb] = delta[h, tok0 + qpos[inb]]
                    St, dPt = Kt @ Qx.t(), Vt @ dOx.t()
                    Pt = torch.exp2(St * sl2 - lse_c[None, :])
                    need_mask = causal and (r0 + kR - 1 > x0)
                    if need_mask:
                        Pt = Pt.masked_fill(~(r_pos[:, None] <= qpos[None, :]), 0.0)
                    dSt = Pt * (dPt - del_c[None, :]) * scale
                    accV += _bf16(Pt) @ dOx
                    accK += _bf16(dSt) @ Qx
                ok = r_pos < L
                dv[tok0 + r_pos[ok], head] = accV[ok]
                dk[tok0 + r_pos[ok], head] = accK[ok]
            # ---------------- dQ pass: lanes are queries
            for head in range(nq):
                hk = head // G
                Qt, dOt = _load_rows(q, tok0 + r0, kR, head, T), _load_rows(dout, tok0 + r0, kR, head, T)
                ok = r_pos < L
                lse_r = torch.full((kR,), math.inf)
                del_r = torch.zeros(kR)
                lse_r[ok] = lse[head, tok0 + r_pos[ok]] * LOG2E
                del_r[ok] = delta[head, tok0 + r_pos[ok]]
                blk1 = (min(L, r0 + kR) + kX - 1) // kX if causal else nblk_all
                acc = torch.zeros(kR, D)
                for t in range(blk1):
                    x0 = t * kX
                    Kx, Vx = _load_rows(k, tok0 + x0, kX, hk, T), _load_rows(v, tok0 + x0, kX, hk, T)
                    xpos = x0 + torch.arange(kX)
                    S, dP = Qt @ Kx.t(), dOt @ Vx.t()
                    P = torch.exp2(S * sl2 - lse_r[:, None])
                    need_mask = (x0 + kX > L) or (causal and x0 + kX - 1 > r0)
                    if need_mask:
                        vis = (xpos[None, :] < L) & ((xpos[None, :] <= r_pos[:, None]) if causal else torch.ones(kR, kX, dtype=torch.bool))
                        P = P.masked_fill(~vis, 0.0)
                    dS = P * (dP - del_r[:, None]) * scale
                    acc += _bf16(dS) @ Kx
                dq[tok0 + r_pos[ok], head] = acc[ok]
    return dq, dk, dv


CASES = [((1, 37, 128, 129, 300, 5), 4, 4, 64, True), ((200, 64, 257), 4, 2, 64, True), ((130, 70), 2, 2, 128, False),
         ((1, 2, 3), 2, 1, 64, True)]


@pytest.mark.parametrize("lens,nq,nkv,hd,causal", CASES)
def test_forward_tile_algorithm_matches_reference(lens, nq, nkv, hd, causal):
    torch.manual_seed(0)
    T = sum(lens)
    cu = [0]
    for l in lens:
        cu.append(cu[-1] + l)
    q, k, v = _bf16(torch.randn(T, nq, hd)), _bf16(torch.randn(T, nkv, hd)), _bf16(torch.randn(T, nkv, hd))
    scale = 1.0 / math.sqrt(hd)
    out, lse = emulate_fwd(q, k, v, cu, scale, causal)
    ref = varlen_attention_ref(q, k, v, torch.tensor(cu), scale, causal)
    torch.testing.assert_close(out, ref, atol=2e-2, rtol=2e-2)
    rep = nq // nkv
    for s, e in zip(cu[:-1], cu[1:]):
        att = torch.einsum("qhd,khd->hqk", q[s:e], k[s:e].repeat_interleave(rep, 1)) * scale
        if causal:
            att = att.masked_fill(torch.ones(e - s, e - s, dtype=torch.bool).triu(1), -math.inf)
        torch.testing.assert_close(lse[:, s:e], torch.logsumexp(att, -1), atol=1e-4, rtol=1e-4)


@pytest.mark.parametrize("lens,nq,nkv,hd,causal", CASES)
def test_backward_tile_algorithm_matches_autograd(lens, nq, nkv, hd, causal):
    torch.manual_seed(1)
    T = sum(lens)
    cu = [0]
    for l in lens:
        cu.append(cu[-1] + l)
    q, k, v = (_bf16(torch.randn(T, h, hd)).requires_grad_(True) for h in (nq, nkv, nkv))
    dout = _bf16(torch.randn(T, nq, hd))
    scale = 1.0 / math.sqrt(hd)
    ref = varlen_attention_ref(q, k, v, torch.tensor(cu), scale, causal)
    ref.backward(dout)
    with torch.no_grad():
        out, lse = emulate_fwd(q, k, v, cu, scale, causal)
        dq, dk, dv = emulate_bwd(q.detach(), k.detach(), v.detach(), out, dout, lse, cu, scale, causal)
    for name, got, want in (("dq", dq, q.grad), ("dk", dk, k.grad), ("dv", dv, v.grad)):
        torch.testing.assert_close(got, want, atol=3e-2, rtol=3e-2, msg=lambda m, n=name: f"{n}: {m}")


def _walk(L, qt0, qt1, causal, window, keep, chunk):
    """The key tiles of an item in order, each with (tile 0 takes part, tile 1 takes part)."""
    win = window if causal and window > 0 else 0
    keep_tiles = -(-keep // kBKV) if win > 0 else 0

    def first(qt):
        q0 = qt * kBQ
        return q0 // chunk * chunk // kBKV if chunk > 0 else max(0, q0 - win + 1) // kBKV if win > 0 else 0

    def end(qt):
        return 0 if qt < 0 else -(-(min(L, qt * kBQ + kBQ) if causal else L) // kBKV)
    firsts, ends = (first(qt0), first(qt0) if qt1 < 0 else first(qt1)), (end(qt0), end(qt1))
    lo = min(firsts)
    nk = min(keep_tiles, lo)
    for k in range(nk + max(ends) - lo):
        j = k if k < nk else lo + k - nk
        yield j, tuple(j < ends[t] and (j >= firsts[t] or j < keep_tiles) for t in range(2))


def _softmax_tiles(L, qt, causal, window, keep, chunk):
    """The key tiles that the softmax warps of a query tile go through."""
    win, q0 = (window if causal and window > 0 else 0), qt * kBQ
    first_tile = q0 // chunk * chunk // kBKV if chunk > 0 else max(0, q0 - win + 1) // kBKV if win > 0 else 0
    n_keep = min(-(-keep // kBKV), first_tile) if win > 0 else 0
    n = n_keep + -(-(min(L, q0 + kBQ) if causal else L) // kBKV) - first_tile
    return [k if k < n_keep else first_tile + k - n_keep for k in range(n)]


@pytest.mark.parametrize("pair_heads", [True, False])
@pytest.mark.parametrize("causal,window,keep,chunk", [(True, 0, 0, 0), (False, 0, 0, 0), (True, 1, 0, 0), (True, 100, 0, 0), (True, 128, 1, 0), (True, 200, 130, 0),
                                                      (True, 300, 600, 0), (True, 5000, 64, 0), (True, 0, 0, 1), (True, 0, 0, 90), (True, 0, 0, 256), (True, 0, 0, 300)])
def test_forward_item_walk_covers_exactly_the_visible_tiles(pair_heads, causal, window, keep, chunk):
    """Both roles of the kernel agree on the tiles of each query tile and their order; every visible key lies in one of them; every tile walked is taken by
    somebody; the items of a sequence cover its query tiles once."""
    for L in (1, 127, 128, 129, 256, 300, 513, 1100):
        tiles = -(-L // kBQ)
        last, units = tiles - 1, tiles if pair_heads else -(-tiles // 2)
        items = [(last - r, last - r) if pair_heads else (last - 2 * r, last - 2 * r - 1) for r in range(units)]
        covered = sorted(q for it in items for q in (it[:1] if pair_heads else it) if q >= 0)
        assert covered == list(range(tiles))
        for qt0, qt1 in items:
            walk = list(_walk(L, qt0, qt1, causal, window, keep, chunk))
            assert all(any(t) for _, t in walk)
            for t, qt in enumerate((qt0, qt1)):
                taken = [j for j, takes in walk if takes[t]]
                assert taken == ([] if qt < 0 else _softmax_tiles(L, qt, causal, window, keep, chunk))
                if qt < 0:
                    continue
                i, j = torch.arange(qt * kBQ, min(L, qt * kBQ + kBQ))[:, None], torch.arange(L)[None]
                ok = (j <= i) if causal else torch.ones(i.numel(), L, dtype=torch.bool)
                if chunk:
                    ok = ok & (j // chunk == i // chunk)
                elif window:
                    ok = ok & ((j > i - window) | (j < keep))
                assert set((ok.any(0).nonzero().flatten() // kBKV).tolist()) <= set(taken)
