"""Performance cases: what a program that uses this framework runs on the GPU, each through a public entry point.

A case is a dict of plain values.  `listed()` holds the standing cases, `draw(rng)` one more of the same ranges, `prepare` makes what
the program has in hand before the call, `run` is one pass, `work` the bytes and operations a pass cannot do without, `tolerance` what
another correct implementation of the same precision may differ by, `exact` the same outputs from plain torch in 64 bits.

Kinds:
  attention   packed causal attention on the fused projection output: "train" forward + backward, "infer" forward alone (prefill,
              reference / reward inference).
  decode_attn one generation step's attention: rotation, append to the key / value cache, attention over the cache.
  norm        residual add + RMSNorm at a layer boundary: "train" forward + backward, "infer" forward alone.
  sample      one sampling step of generation: temperature, top-k, top-p, draw, log-probability, packed mask.
  moe         a mixture-of-experts feed-forward, forward + backward.
  window_attn packed prefill attention of the heterogeneous stacks: window with kept first tokens, distance penalty, temperature,
              sink and output gate ("sink"), or soft-capped chunks with a sink ("chunk").
  delta       packed prefill of a gated delta-rule mixer: convolution and gates, recurrence, gated head norm.
  train_step  a whole model's training pass: log-probabilities of the labels and the gradients of every weight.
  decode      a whole model's generation step (a captured CUDA graph, as `generate` keeps one): logits and the updated cache.
"""

from __future__ import annotations

import math
import random
from typing import Dict, List

import torch

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


# ------------------------------------------------------------------------------------------------ the cases


def listed() -> List[dict]:
    return [
        # a handful of short prompts through a GPT-2 sized attention: latency and launches count
        dict(name="attention_small_prefill", kind="attention", mode="infer", seqs=4, lo=29, hi=64, lens_seed=1, nq=12, nkv=12, hd=64, dtype="bf16"),
        # one layer of the PPO benchmark's training step: 32 sequences of 128 + 512 tokens (a minibatch), LLaMA-7B heads
        dict(name="attention_train_ppo", kind="attention", mode="train", seqs=32, lo=640, hi=640, lens_seed=2, nq=32, nkv=32, hd=128, dtype="bf16"),
        # long ragged sequences with grouped key / value heads: SFT of a mistral / mixtral shaped model
        dict(name="attention_train_long_gqa", kind="attention", mode="train", seqs=8, lo=1500, hi=4096, lens_seed=3, nq=32, nkv=8, hd=128, dtype="bf16"),
        # generation with 16 sequences per GPU (the benchmark's share on 8 GPUs)
        dict(name="decode_attention_b16", kind="decode_attn", batch=16, lo=128, hi=639, lens_seed=4, room=640, nq=32, nkv=32, hd=128, dtype="bf16"),
        # generation with the benchmark's whole batch on one GPU
        dict(name="decode_attention_b128", kind="decode_attn", batch=128, lo=128, hi=639, lens_seed=5, room=640, nq=32, nkv=32, hd=128, dtype="bf16"),
        # a layer boundary of the PPO benchmark's training step
        dict(name="norm_train_20480x4096", kind="norm", mode="train", rows=20480, width=4096, dtype="bf16"),
        # the sampling step of the PPO benchmark with both filters on
        dict(name="sample_b128_topk_topp", kind="sample", rows=128, vocab=32000, top_k=50, top_p=0.9, greedy=False, dtype="bf16"),
        # one Mixtral-8x7B feed-forward on a small training batch
        dict(name="moe_train_mixtral", kind="moe", tokens=2048, width=4096, ff=14336, experts=8, top=2, dtype="bf16"),
        # prefill of the serving benchmark's heterogeneous stacks: attention and delta-rule mixers
        dict(name="window_attention_prefill", kind="window_attn", form="sink", seqs=32, lo=1024, hi=1024, lens_seed=6, nq=16, nkv=4, hd=128,
             window=512, keep=64, dtype="bf16"),
        dict(name="delta_rule_prefill", kind="delta", seqs=8, lo=700, hi=1024, lens_seed=7, nq=16, nkv=4, hd=128, taps=4, dtype="bf16"),
        # two LLaMA blocks with embedding and head: every kernel of a training step in its place
        dict(name="train_step_2layers", kind="train_step", layers=2, width=2048, heads=16, kv=16, ff=5632, vocab=32000, seqs=8, lo=300, hi=640, lens_seed=8,
             dtype="bf16"),
        # a generation step of four LLaMA-7B blocks and the head at 16 sequences
        dict(name="decode_step_4layers_b16", kind="decode", layers=4, width=4096, heads=32, kv=32, ff=11008, vocab=32000, batch=16, lo=128, hi=639, room=640,
             lens_seed=9, dtype="bf16"),
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


HEADS = [(12, 12, 64), (16, 4, 128), (32, 32, 128), (32, 8, 128), (16, 16, 64), (14, 2, 64)]


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["attention", "attention", "attention", "decode_attn", "decode_attn", "norm", "norm", "sample", "moe", "window_attn", "delta",
                       "train_step", "decode"])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    seed = rng.randrange(1 << 20)
    if kind == "attention":
        nq, nkv, hd = rng.choice(HEADS)
        hi = _log(rng, 17, 4096)
        lo = rng.choice([hi, max(1, hi // 3), max(1, hi // 2)])
        seqs = _log(rng, 1, max(1, min(64, 20480 // hi)))
        return dict(kind=kind, mode=rng.choice(["train", "infer"]), seqs=seqs, lo=lo, hi=hi, lens_seed=seed, nq=nq, nkv=nkv, hd=hd, dtype=dtype)
    if kind == "decode_attn":
        nq, nkv, hd = rng.choice([(32, 32, 128), (32, 8, 128), (12, 12, 64), (16, 4, 128), (8, 1, 128)])
        room = _log(rng, 96, 4096)
        hi = rng.randint(room // 2, room - 1)
        return dict(kind=kind, batch=_log(rng, 1, max(1, min(128, 128 * 640 // room))), lo=max(1, hi // rng.choice([1, 3])), hi=hi, lens_seed=seed, room=room,
                    nq=nq, nkv=nkv, hd=hd, dtype=dtype)
    if kind == "norm":
        return dict(kind=kind, mode=rng.choice(["train", "train", "infer"]), rows=_log(rng, 16, 20480), width=8 * rng.choice([96, 128, 256, 320, 512, 640]),
                    dtype=rng.choice(["bf16", "bf16", "fp16", "fp32"]))
    if kind == "sample":
        return dict(kind=kind, rows=_log(rng, 1, 128), vocab=rng.choice([2048, 32000, 32003, 50257]), top_k=rng.choice([20, 50, 200, 256]),
                    top_p=rng.choice([0.8, 0.9, 0.95, 1.0]), greedy=rng.random() < 0.15, dtype=rng.choice(["bf16", "fp32"]))
    if kind == "moe":
        w = rng.choice([1024, 2048, 4096])
        return dict(kind=kind, tokens=8 * _log(rng, 16, 256), width=w, ff=w // 8 * rng.choice([14, 28, 16]), experts=8, top=2, dtype="bf16")
    if kind == "window_attn":
        nq, nkv, hd = rng.choice([(16, 4, 128), (32, 8, 128), (12, 12, 64)])
        hi = _log(rng, 33, 2048)
        return dict(kind=kind, form=rng.choice(["sink", "chunk"]), seqs=_log(rng, 1, max(1, min(32, 16384 // hi))), lo=max(1, hi // rng.choice([1, 2])), hi=hi,
                    lens_seed=seed, nq=nq, nkv=nkv, hd=hd, window=rng.choice([128, 500, 512, 1024]), keep=rng.choice([0, 16, 64]), dtype=dtype)
    if kind == "delta":
        nq, nkv, hd = rng.choice([(16, 4, 128), (32, 8, 128), (8, 8, 64)])
        hi = _log(rng, 20, 1024)
        return dict(kind=kind, seqs=_log(rng, 1, 8), lo=max(1, hi // rng.choice([1, 2])), hi=hi, lens_seed=seed, nq=nq, nkv=nkv, hd=hd,
                    taps=rng.choice([2, 4]), dtype=dtype)
    if kind == "train_step":
        w = rng.choice([1024, 2048])
        return dict(kind=kind, layers=rng.choice([1, 2]), width=w, heads=w // 128, kv=rng.choice([w // 128, w // 512]), ff=w // 128 * rng.choice([344, 352]) // 8 * 8,
                    vocab=32000, seqs=_log(rng, 2, 8), lo=100, hi=rng.randint(200, 640), lens_seed=seed, dtype="bf16")
    return dict(kind="decode", layers=rng.choice([2, 4]), width=4096, heads=32, kv=rng.choice([8, 32]), ff=11008, vocab=32000, batch=_log(rng, 1, 128), lo=64,
                hi=rng.randint(128, 639), room=640, lens_seed=seed, dtype="bf16")


# ------------------------------------------------------------------------------------------------ helpers


def _lens(case) -> List[int]:
    r = random.Random(case["lens_seed"])
    n = case["seqs"] if "seqs" in case else case["batch"]
    return [r.randint(case["lo"], case["hi"]) for _ in range(n)]


def _rand(g, shape, dtype, std=1.0):
    return torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, std, generator=g)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _cu(lens):
    out = [0]
    for n in lens:
        out.append(out[-1] + n)
    return torch.tensor(out, dtype=torch.int32, device="cuda")


def _pos(lens):
    return torch.cat([torch.arange(n, dtype=torch.int32, device="cuda") for n in lens])


def _llama(case):
    from realhf_b200.api.model import ReaLModelConfig
    return ReaLModelConfig(n_layers=case["layers"], n_kv_heads=case["kv"], n_q_heads=case["heads"], hidden_dim=case["width"], intermediate_dim=case["ff"],
                           vocab_size=case["vocab"], n_positions=4096, embd_pdrop=0.0, resid_pdrop=0.0, attn_pdrop=0.0, activation_function="silu",
                           scale_attn_by_inverse_layer_idx=False, use_attention_bias=False, use_attn_proj_bias=False, use_mlp_bias=False,
                           layer_norm_type="rms", mlp_type="llama", apply_rotary=True)


def _llama_weights(case, g, dtype) -> Dict[str, torch.Tensor]:
    H, F, V, hd = case["width"], case["ff"], case["vocab"], case["width"] // case["heads"]
    w = {"0.wte.weight": _rand(g, (V, H), dtype, 0.02)}
    for i in range(1, case["layers"] + 1):
        w[f"{i}.attn.ln.weight"] = 1 + _rand(g, (H,), dtype, 0.05)
        w[f"{i}.attn.qkv.weight"] = _rand(g, ((case["heads"] + 2 * case["kv"]) * hd, H), dtype, 0.02)
        w[f"{i}.attn.o.weight"] = _rand(g, (H, H), dtype, 0.02)
        w[f"{i}.mlp.ln.weight"] = 1 + _rand(g, (H,), dtype, 0.05)
        w[f"{i}.mlp.gate_up.weight"] = _rand(g, (2 * F, H), dtype, 0.02)
        w[f"{i}.mlp.down.weight"] = _rand(g, (H, F), dtype, 0.02)
    w[f"{case['layers']}.ln_f.weight"] = 1 + _rand(g, (H,), dtype, 0.05)
    w[f"{case['layers'] + 1}.head.weight"] = _rand(g, (V, H), dtype, 0.02)
    return w


def _model(case, weights, dtype):
    from realhf_b200.models.real_model import ReaLModel
    m = ReaLModel(_llama(case), dtype=dtype, device="cuda").instantiate("empty")
    with torch.no_grad():
        m.flat_param.data.zero_()
    m.load_state_dict(weights)
    return m


def _wattn_config(case):
    from realhf_b200.api.model import WindowAttentionConfig
    base = dict(n_heads=case["nq"], n_kv_heads=case["nkv"], qk_dim=case["hd"], v_dim=case["hd"], scale=case["hd"] ** -0.5)
    if case["form"] == "sink":
        return WindowAttentionConfig(window=case["window"], keep_first=case["keep"], **base)
    return WindowAttentionConfig(chunk=case["window"], softcap=30.0, slope_base=None, head_temp=False, sink=False, sink_const=0.0, value_norm=False,
                                 out_gate=False, **base)


def _delta_config(case):
    from realhf_b200.api.model import DeltaRuleConfig
    return DeltaRuleConfig(n_heads=case["nq"], n_kv_heads=case["nkv"], qk_dim=case["hd"], v_dim=case["hd"], conv_taps=case["taps"])


# ------------------------------------------------------------------------------------------------ inputs (plain torch, from the seed alone)


def _inputs(case, seed) -> dict:
    k, dt, g = case["kind"], DTYPES[case["dtype"]], _gen(seed)
    s: dict = dict(case=case)
    if k == "attention":
        lens = _lens(case)
        T, nq, nkv, hd = sum(lens), case["nq"], case["nkv"], case["hd"]
        s.update(lens=lens, cu=_cu(lens), qkv=_rand(g, (T, (nq + 2 * nkv) * hd), dt))
        if case["mode"] == "train":
            s["dout"] = _rand(g, (T, nq, hd), dt)
    elif k == "decode_attn":
        lens, B, S = _lens(case), case["batch"], case["room"]
        nq, nkv, hd = case["nq"], case["nkv"], case["hd"]
        cache = lambda: _rand(g, (B, nkv, S, hd), dt).permute(0, 2, 1, 3)  # noqa: E731
        s.update(lens=torch.tensor(lens, dtype=torch.int32, device="cuda"), qkv=_rand(g, (B, (nq + 2 * nkv) * hd), dt), k=cache(), v=cache())
    elif k == "norm":
        shape = (case["rows"], case["width"])
        s.update(d=_rand(g, shape, dt), x=_rand(g, shape, dt), w=(1 + _rand(g, (case["width"],), torch.float32, 0.1)).to(dt))
        if case["mode"] == "train":
            s.update(dy=_rand(g, shape, dt), dres=_rand(g, shape, dt))
    elif k == "sample":
        # a language model's logits: a few tokens stand out
        lg = _rand(g, (case["rows"], case["vocab"]), torch.float32, 2.0)
        hot = torch.randint(0, case["vocab"], (case["rows"], 12), device="cuda", generator=g)
        lg.scatter_add_(1, hot, _rand(g, (case["rows"], 12), torch.float32, 1.5) + 6.0)
        s.update(logits=lg.to(dt), unfinished=torch.ones(case["rows"], dtype=torch.bool, device="cuda"), draw_seed=int(seed) * 7919 + 12345)
    elif k == "moe":
        T, H, F, E = case["tokens"], case["width"], case["ff"], case["experts"]
        s.update(h=_rand(g, (T, H), dt), dout=_rand(g, (T, H), dt), router=_rand(g, (E, H), dt, 0.02), gate_up=_rand(g, (E, 2 * F, H), dt, 0.02),
                 down=_rand(g, (E, H, F), dt, 0.02))
    elif k == "window_attn":
        lens = _lens(case)
        H, G, hd = case["nq"], case["nkv"], case["hd"]
        gate = (H + 7) // 8 * 8 if case["form"] == "sink" else 0
        s.update(lens=lens, cu=_cu(lens), pos=_pos(lens), rows=_rand(g, (sum(lens), (H + 2 * G) * hd + gate), dt))
        if case["form"] == "sink":
            s.update(temp=1 + _rand(g, (H,), dt, 0.1), sink=_rand(g, (H,), dt))
    elif k == "delta":
        lens = _lens(case)
        H, G, hd = case["nq"], case["nkv"], case["hd"]
        C = 2 * G * hd + H * hd
        s.update(lens=lens, cu=_cu(lens), pos=_pos(lens), proj=_rand(g, (sum(lens), C + H * hd + 2 * H), dt), conv=_rand(g, (C, case["taps"]), dt, 0.4),
                 A_log=_rand(g, (H,), torch.float32, 0.5).to(dt), dt_bias=_rand(g, (H,), torch.float32, 0.5).to(dt), w=(1 + _rand(g, (hd,), torch.float32, 0.1)).to(dt))
    elif k == "train_step":
        lens = _lens(case)
        T = sum(lens) // 8 * 8
        lens[-1] -= sum(lens) - T
        s.update(lens=lens, cu=_cu(lens), weights=_llama_weights(case, g, dt), ids=torch.randint(3, case["vocab"], (T,), device="cuda", generator=g),
                 labels=torch.randint(3, case["vocab"], (T,), device="cuda", generator=g), dlogp=_rand(g, (T,), torch.float32, 1.0 / T))
    else:
        lens, hd = _lens(case), case["width"] // case["heads"]
        cache = lambda: _rand(g, (case["batch"], case["kv"], case["room"], hd), dt)  # noqa: E731
        s.update(lens=torch.tensor(lens, dtype=torch.int32, device="cuda"), weights=_llama_weights(case, g, dt),
                 ids=torch.randint(3, case["vocab"], (case["batch"],), device="cuda", generator=g), k=[cache() for _ in range(case["layers"])],
                 v=[cache() for _ in range(case["layers"])])
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    k, dt = case["kind"], DTYPES[case["dtype"]]
    if k == "attention":
        s["qkv"].requires_grad_(case["mode"] == "train")
    elif k == "decode_attn":
        from realhf_b200.ops import functional as OF
        s["cos"], s["sin"] = OF.rope_tables(case["room"], case["hd"], 10000.0, "cuda")
    elif k == "norm" and case["mode"] == "train":
        for n in ("d", "x", "w"):
            s[n].requires_grad_(True)
    elif k == "sample":
        from realhf_b200.api.model import GenerationHyperparameters
        s["g"] = GenerationHyperparameters(max_new_tokens=512, min_new_tokens=0, greedy=case["greedy"], top_p=case["top_p"],
                                           top_k=min(case["top_k"], case["vocab"]))
    elif k == "moe":
        from realhf_b200.api.model import ReaLModelConfig, ReaLMoEConfig
        from realhf_b200.models.real_model import ReaLModel
        cfg = ReaLModelConfig(n_layers=1, n_kv_heads=case["width"] // 128, n_q_heads=case["width"] // 128, hidden_dim=case["width"],
                              intermediate_dim=case["ff"], vocab_size=64, n_positions=2048, embd_pdrop=0.0, resid_pdrop=0.0, attn_pdrop=0.0,
                              activation_function="silu", scale_attn_by_inverse_layer_idx=False, use_attention_bias=False, use_attn_proj_bias=False,
                              use_mlp_bias=False, layer_norm_type="rms", mlp_type="moe", apply_rotary=True,
                              moe=ReaLMoEConfig(num_experts=case["experts"], top_k=case["top"], aux_loss_coeff=0.0))
        m = ReaLModel(cfg, dtype=dt, device="cuda").instantiate("empty")
        names = {"router": "1.mlp.router.weight", "gate_up": "1.mlp.experts.gate_up.weight", "down": "1.mlp.experts.down.weight"}
        with torch.no_grad():
            m.flat_param.data.zero_()
            for a, b in names.items():
                m.p[b].copy_(s.pop(a))
        m.train()
        s.update(model=m, params=[m.p[b] for b in names.values()])
        s["h"].requires_grad_(True)
    elif k == "window_attn":
        s["a"] = _wattn_config(case)
    elif k == "delta":
        s["dl"] = _delta_config(case)
    elif k == "train_step":
        m = _model(case, s.pop("weights"), dt)
        m.train()
        m.attach_grad_buffer(torch.zeros_like(m.flat_param.data))
        s["model"] = m
    elif k == "decode":
        m = _model(case, s.pop("weights"), dt)
        m.eval()
        m.flat_param.requires_grad_(False)
        s["model"] = m
        s["k"], s["v"] = [t.permute(0, 2, 1, 3) for t in s["k"]], [t.permute(0, 2, 1, 3) for t in s["v"]]
        from realhf_b200.ops import functional as OF

        def step():
            return OF.linear(m.decode_step(s["ids"], s["k"], s["v"], s["lens"]), m.head_weight())

        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.no_grad():
            with torch.cuda.stream(side):
                step()
            torch.cuda.current_stream().wait_stream(side)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                s["logits"] = step()
        s["graph"] = graph
    return s


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "attention":
        from realhf_b200.ops import attention as A
        nq, nkv, hd = case["nq"], case["nkv"], case["hd"]
        if case["mode"] == "infer":
            with torch.no_grad():
                return A.varlen_attention_qkv(s["qkv"], s["cu"], case["hi"], nq, nkv, hd)
        out = A.varlen_attention_qkv(s["qkv"], s["cu"], case["hi"], nq, nkv, hd)
        return out, torch.autograd.grad(out, s["qkv"], s["dout"])[0]
    if k == "decode_attn":
        from realhf_b200.ops import attention as A
        out = A.decode_attention(s["qkv"], s["k"], s["v"], s["lens"], case["nq"], case["nkv"], case["hd"], cos=s["cos"], sin=s["sin"])
        return out, s["k"], s["v"]
    if k == "norm":
        from realhf_b200.ops import functional as OF
        if case["mode"] == "infer":
            with torch.no_grad():
                return OF.add_rmsnorm(s["d"], s["x"], s["w"], 1e-5)
        y, res = OF.add_rmsnorm(s["d"], s["x"], s["w"], 1e-5)
        _, dx, dw = torch.autograd.grad((y, res), (s["d"], s["x"], s["w"]), (s["dy"], s["dres"]))
        return y, res, dx, dw
    if k == "sample":
        from realhf_b200.models import generation as GEN
        GEN.seed_sampling(s["draw_seed"])
        tok, lp, mask, _ = GEN.genstep(s["logits"], s["g"], 5, 2, 0, s["unfinished"])
        return dict(tokens=tok, logprobs=lp, mask=mask) if mask is not None else dict(tokens=tok, logprobs=lp)
    if k == "moe":
        from realhf_b200.models.moe import moe_forward
        out = moe_forward(s["model"], 1, s["h"])
        return (out,) + torch.autograd.grad(out, [s["h"]] + s["params"], s["dout"])
    if k == "window_attn":
        from realhf_b200.ops import attention as A
        a = s["a"]
        with torch.no_grad():
            v = A.value_norm_store(s["rows"], a, 1e-5, None, None, None, s["pos"], None) if a.value_norm else A.window_values(s["rows"], a)
            return A.sink_window_attention(s["rows"], v, a, s.get("temp"), s.get("sink"), s["pos"], s["cu"], case["hi"])
    if k == "delta":
        from realhf_b200.ops import recurrent as R
        d = s["dl"]
        with torch.no_grad():
            u = R.delta_prepare(s["proj"], s["conv"], s["A_log"], s["dt_bias"], d, s["pos"])
            o = R.delta_rule_scan(u, d, s["cu"])
            return R.gated_head_norm(o, s["w"], R.delta_gate(s["proj"], None, d), 1e-5, s["proj"].dtype)
    if k == "train_step":
        m = s["model"]
        m.flat_grad.zero_()
        out = m(input_ids=s["ids"], cu_seqlens=s["cu"], max_seqlen=max(s["lens"]))
        lp = out.logprobs(s["labels"])
        (lp * s["dlogp"]).sum().backward()
        return lp.detach(), {n: p.grad for n, p in m.named_parameters()}
    s["graph"].replay()
    return s["logits"], s["k"], s["v"]


# ------------------------------------------------------------------------------------------------ work, tolerance


def work(case) -> dict:
    k, es = case["kind"], torch.empty(0, dtype=DTYPES[case["dtype"]]).element_size()
    if k == "attention":
        lens = _lens(case)
        T, pairs = sum(lens), sum(n * (n + 1) // 2 for n in lens)
        nq, nkv, hd = case["nq"], case["nkv"], case["hd"]
        f, qkv, out = 4 * hd * nq * pairs, T * (nq + 2 * nkv) * hd * es, T * nq * hd * es
        return dict(bytes=qkv + out, flops=f) if case["mode"] == "infer" else dict(bytes=2 * qkv + 2 * out, flops=3.5 * f)
    if k == "decode_attn":
        n, B = sum(_lens(case)), case["batch"]
        return dict(bytes=2 * n * case["nkv"] * case["hd"] * es + B * (2 * case["nq"] + 4 * case["nkv"]) * case["hd"] * es,
                    flops=4 * (n + B) * case["nq"] * case["hd"])
    if k == "norm":
        n = case["rows"] * case["width"] * es
        return dict(bytes=(7 if case["mode"] == "train" else 4) * n, flops=0)
    if k == "sample":
        return dict(bytes=case["rows"] * (case["vocab"] * es + (0 if case["greedy"] else case["vocab"] / 8) + 12), flops=0)
    if k == "moe":
        w, T = 3 * case["experts"] * case["width"] * case["ff"], case["tokens"]
        return dict(bytes=2 * w * es + 4 * T * case["width"] * es, flops=18.0 * T * case["top"] * case["width"] * case["ff"])
    if k == "window_attn":
        w, keep, pairs = case["window"], case["keep"] if case["form"] == "sink" else 0, 0
        for n in _lens(case):
            for i in range(n):
                pairs += i % w + 1 if case["form"] == "chunk" else min(i + 1, w) + min(max(i + 1 - w, 0), keep)
        T, nq, nkv, hd = sum(_lens(case)), case["nq"], case["nkv"], case["hd"]
        return dict(bytes=T * (2 * nq + 2 * nkv) * hd * es, flops=4.0 * hd * nq * pairs)
    if k == "delta":
        T, H, G, hd = sum(_lens(case)), case["nq"], case["nkv"], case["hd"]
        return dict(bytes=T * (2 * G * hd + 3 * H * hd + 2 * H) * es, flops=7.0 * T * H * hd * hd)
    H, F, L, V = case["width"], case["ff"], case["layers"], case["vocab"]
    hd = H // case["heads"]
    per = (case["heads"] + 2 * case["kv"]) * hd * H + H * H + 3 * H * F
    if k == "train_step":
        lens = _lens(case)
        T, pairs = sum(lens), sum(n * (n + 1) // 2 for n in lens)
        return dict(bytes=2 * (L * per + 2 * V * H) * es, flops=6.0 * T * (L * per + V * H) + 14.0 * H * pairs * L)
    n, B = sum(_lens(case)), case["batch"]
    return dict(bytes=(L * per + V * H + 2 * L * n * case["kv"] * hd + B * V) * es, flops=2.0 * B * (L * per + V * H) + 4.0 * L * n * H)


# kind -> (largest relative error, largest single difference) of bf16 results: about four times what the present kernels differ by from
# `exact` (bf16's rounding of a result alone is 1.7e-3, of gradients through two roundings 2.4e-3; whole models carry it through every
# layer).  fp16 rounds eight times finer; fp32 results are bound by sums over a row or a column.
_TOL = dict(attention=(1e-2, 0.5), decode_attn=(7e-3, 2e-2), norm=(7e-3, 2e-2), moe=(2e-2, 0.25), window_attn=(1e-2, 0.16), delta=(7e-3, 2e-2),
            train_step=(3e-2, 0.99), decode=(3e-2, 0.3))


def tolerance(case):
    if case["kind"] == "sample":     # probabilities and sums are fp32 whatever the logits are; a draw may fall on a rounded boundary
        return dict(rel=1e-5, max=1e-4, differ=0.01)
    rel, most = _TOL[case["kind"]]
    if case["dtype"] == "fp32":
        return dict(rel=2e-6, max=1e-5)
    return dict(rel=rel, max=most) if case["dtype"] == "bf16" else dict(rel=rel / 7, max=most / 7)


# ------------------------------------------------------------------------------------------------ the same outputs in 64 bits


def _attend(q, k, v, scale, ok, sink=None, bias=None, cap=None, temp=None):
    """q [h, n, d], k / v [h, m, d] float64; visibility ok [n, m] -> [h, n, d]."""
    s = q @ k.transpose(1, 2) * scale
    if temp is not None:
        s = s * temp.view(-1, 1, 1)
    if cap is not None:
        s = cap * torch.tanh(s / cap)
    if bias is not None:
        s = s + bias
    s = s.masked_fill(~ok, float("-inf"))
    if sink is not None:
        s = torch.cat([s, sink.view(-1, 1, 1).expand(-1, s.shape[1], 1)], -1)
    p = torch.softmax(s, -1)
    return (p[..., :-1] if sink is not None else p) @ v


def _causal(n):
    i = torch.arange(n, device="cuda")
    return i[None, :] <= i[:, None]


def _packed_attention(qkv, lens, nq, nkv, hd):
    """Causal attention on float64 [T, (nq + 2 nkv) hd] -> [T, nq, hd]."""
    T = qkv.shape[0]
    q, k, v = (t.view(T, -1, hd) for t in qkv.split([nq * hd, nkv * hd, nkv * hd], 1))
    k, v = (t.repeat_interleave(nq // nkv, 1) for t in (k, v))
    parts, a = [], 0
    for n in lens:
        sl = [t[a:a + n].transpose(0, 1) for t in (q, k, v)]
        step = max(1, int(2e8) // (n * n))
        o = [_attend(*(t[h:h + step] for t in sl), hd ** -0.5, _causal(n)) for h in range(0, nq, step)]
        parts.append(torch.cat(o, 0).transpose(0, 1))
        a += n
    return torch.cat(parts, 0)


def _rotate(x, pos, hd):
    """x [T, heads, hd] float64, halves rotated by position (base 10000, the tables rounded to fp32 angles as the model has them)."""
    inv = 1.0 / (10000.0 ** (torch.arange(0, hd, 2, dtype=torch.float32, device="cuda") / hd))
    ang = torch.outer(pos.float(), inv)
    c, s = ang.cos().double().unsqueeze(1), ang.sin().double().unsqueeze(1)
    a, b = x[..., :hd // 2], x[..., hd // 2:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _rms(x, w, eps=1e-5):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _decode_attention(qkv, kc, vc, lens, nq, nkv, hd, pos):
    """qkv [B, ..] float64, kc / vc [B, S, nkv, hd] float64 updated in place -> [B, nq * hd]."""
    B = qkv.shape[0]
    q, k, v = (t.reshape(B, -1, hd) for t in qkv.split([nq * hd, nkv * hd, nkv * hd], 1))
    q, k = _rotate(q, pos, hd), _rotate(k, pos, hd)
    out = torch.empty(B, nq * hd, dtype=torch.float64, device="cuda")
    for b, n in enumerate(lens):
        kc[b, n], vc[b, n] = k[b], v[b]
        kk, vv = (t[b, :n + 1].transpose(0, 1).repeat_interleave(nq // nkv, 0) for t in (kc, vc))
        out[b] = _attend(q[b].unsqueeze(1), kk, vv, hd ** -0.5, torch.ones(1, n + 1, dtype=torch.bool, device="cuda")).reshape(-1)
    return out


def _mix32(x: int) -> int:
    x ^= x >> 16
    x = x * 0x7FEB352D & 0xFFFFFFFF
    x ^= x >> 15
    x = x * 0x846CA68B & 0xFFFFFFFF
    return x ^ (x >> 16)


def _exact_sample(s, case):
    x = s["logits"].double()
    B, V = x.shape
    if case["greedy"]:
        tok = s["logits"].float().argmax(-1)
        return dict(tokens=None, logprobs=(torch.log_softmax(x, -1).gather(1, tok.unsqueeze(1)).squeeze(1)))
    kth = torch.topk(x, min(case["top_k"], V), -1).values[:, -1:]
    p = torch.softmax(x.masked_fill(x < kth, float("-inf")), -1)
    keep = p > 0
    if case["top_p"] < 1.0:          # kept while the mass of strictly larger logits is below top_p
        srt, idx = torch.sort(x.masked_fill(~keep, float("-inf")), -1, descending=True)
        ps = p.gather(1, idx)
        before = ps.cumsum(-1) - ps
        first = torch.searchsorted(-srt.contiguous(), -srt.contiguous())      # equal logits share the mass above the first of them
        keep = torch.zeros_like(keep).scatter_(1, idx, before.gather(1, first.clamp(max=V - 1)) < case["top_p"]) & keep
    p = torch.where(keep, p, torch.zeros_like(p))
    cdf = p.cumsum(-1)
    seed = s["draw_seed"] % (1 << 62)
    lo, hi = seed & 0xFFFFFFFF, seed >> 32
    out = torch.empty(B, dtype=torch.float64, device="cuda")
    for row in range(B):
        r = _mix32(lo ^ _mix32((hi + 0x9E3779B9 * row) & 0xFFFFFFFF) ^ _mix32((5 * 0x85EBCA6B + 1) & 0xFFFFFFFF))
        u = ((r >> 8) + 0.5) / 16777216.0
        t = int((cdf[row] <= u * cdf[row, -1]).sum())
        out[row] = torch.log(p[row, min(t, V - 1)] / cdf[row, -1])
    return dict(tokens=None, logprobs=out, mask=None)


def _exact_llama(case, w, ids, lens, pos):
    """(final hidden states, head weight) of the packed batch from float64 weights."""
    hd = case["width"] // case["heads"]
    nq, nkv = case["heads"], case["kv"]
    x = w["0.wte.weight"][ids]
    for i in range(1, case["layers"] + 1):
        qkv = _rms(x, w[f"{i}.attn.ln.weight"]) @ w[f"{i}.attn.qkv.weight"].T
        T = qkv.shape[0]
        qk = _rotate(qkv[:, :(nq + nkv) * hd].reshape(T, nq + nkv, hd), pos, hd).reshape(T, -1)
        o = _packed_attention(torch.cat([qk, qkv[:, (nq + nkv) * hd:]], 1), lens, nq, nkv, hd)
        x = x + o.reshape(T, -1) @ w[f"{i}.attn.o.weight"].T
        gu = _rms(x, w[f"{i}.mlp.ln.weight"]) @ w[f"{i}.mlp.gate_up.weight"].T
        x = x + (torch.nn.functional.silu(gu[:, :case["ff"]]) * gu[:, case["ff"]:]) @ w[f"{i}.mlp.down.weight"].T
    return _rms(x, w[f"{case['layers']}.ln_f.weight"])


def _exact_window(s, case):
    H, G, hd = case["nq"], case["nkv"], case["hd"]
    rows = s["rows"].double()
    T = rows.shape[0]
    q, k, v = (t.reshape(T, -1, hd) for t in rows[:, :(H + 2 * G) * hd].split([H * hd, G * hd, G * hd], 1))
    sink_form = case["form"] == "sink"
    if sink_form:
        v = v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + 1e-5)
    k, v = (t.repeat_interleave(H // G, 1) for t in (k, v))
    slopes = torch.exp2(-8.0 * torch.arange(1, H + 1, dtype=torch.float64, device="cuda") / H)
    parts, a = [], 0
    for n in s["lens"]:
        i = torch.arange(n, device="cuda")
        dist = i[:, None] - i[None, :]
        if sink_form:
            ok = (dist >= 0) & ((dist < case["window"]) | (i[None, :] < case["keep"]))
        else:
            ok = (dist >= 0) & (i[:, None] // case["window"] == i[None, :] // case["window"])
        sl = [t[a:a + n].transpose(0, 1) for t in (q, k, v)]
        kw = dict(sink=s["sink"].double(), temp=s["temp"].double(), bias=-slopes.view(-1, 1, 1) * dist.double()) if sink_form else \
            dict(sink=torch.zeros(H, dtype=torch.float64, device="cuda"), cap=30.0)
        parts.append(_attend(*sl, hd ** -0.5, ok, **kw).transpose(0, 1))
        a += n
    o = torch.cat(parts, 0)
    if sink_form:
        o = o * torch.sigmoid(rows[:, (H + 2 * G) * hd:(H + 2 * G) * hd + H]).unsqueeze(-1)
    return o.reshape(T, H * hd)


def _exact_delta(s, case):
    H, G, hd, taps = case["nq"], case["nkv"], case["hd"], case["taps"]
    proj, cw = s["proj"].double(), s["conv"].double()
    T, nqk, nv = proj.shape[0], G * hd, H * hd
    C = 2 * nqk + nv
    x = proj[:, :C]
    y = x * cw[:, taps - 1]
    for back in range(1, taps):
        prev = torch.zeros_like(x)
        prev[back:] = x[:-back]
        y = y + prev * (s["pos"] >= back).unsqueeze(-1) * cw[:, taps - 1 - back]
    y = torch.nn.functional.silu(y)
    unit = lambda t: t * torch.rsqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    q = unit(y[:, :nqk].reshape(T, G, hd)).repeat_interleave(H // G, 1) * hd ** -0.5
    k = unit(y[:, nqk:2 * nqk].reshape(T, G, hd)).repeat_interleave(H // G, 1)
    v = y[:, 2 * nqk:].reshape(T, H, hd)
    beta = torch.sigmoid(proj[:, C + nv:C + nv + H])
    g = torch.exp(-torch.exp(s["A_log"].double()) * torch.nn.functional.softplus(proj[:, C + nv + H:C + nv + 2 * H] + s["dt_bias"].double()))
    n_seq, n_max = len(s["lens"]), max(s["lens"])
    start = s["cu"][:-1].long()
    S = torch.zeros(n_seq, H, hd, hd, dtype=torch.float64, device="cuda")
    o = torch.zeros(T, H, hd, dtype=torch.float64, device="cuda")
    lens = torch.tensor(s["lens"], device="cuda")
    for t in range(n_max):
        live = torch.nonzero(lens > t).flatten() if t >= min(s["lens"]) else torch.arange(n_seq, device="cuda")
        r = start[live] + t
        St = S[live] * g[r].view(-1, H, 1, 1)
        u = beta[r].unsqueeze(-1) * (v[r] - (k[r].unsqueeze(-2) @ St).squeeze(-2))
        St = St + k[r].unsqueeze(-1) * u.unsqueeze(-2)
        S[live] = St
        o[r] = (q[r].unsqueeze(-2) @ St).squeeze(-2)
    gate = proj[:, C:C + nv].reshape(T, H, hd)
    return (_rms(o, s["w"].double()) * torch.nn.functional.silu(gate)).reshape(T, H * hd)


def _exact_moe(s, case):
    leaf = {n: s[n].double().requires_grad_(True) for n in ("h", "router", "gate_up", "down")}
    h = leaf["h"]
    probs, idx = torch.topk(torch.softmax(h @ leaf["router"].T, -1), case["top"], -1)
    probs = probs / probs.sum(-1, keepdim=True)
    out = torch.zeros_like(h)
    for e in range(case["experts"]):
        t, c = torch.nonzero(idx == e, as_tuple=True)
        gu = h[t] @ leaf["gate_up"][e].T
        y = (torch.nn.functional.silu(gu[:, :case["ff"]]) * gu[:, case["ff"]:]) @ leaf["down"][e].T
        out = out.index_add(0, t, y * probs[t, c].unsqueeze(-1))
    return (out.detach(),) + torch.autograd.grad(out, list(leaf.values()), s["dout"].double())


def exact(case, seed):
    s = _inputs(case, seed)
    k = case["kind"]
    if k == "attention":
        nq, nkv, hd = case["nq"], case["nkv"], case["hd"]
        qkv = s["qkv"].double().requires_grad_(case["mode"] == "train")
        if case["mode"] == "infer":
            return _packed_attention(qkv, s["lens"], nq, nkv, hd)
        outs, grads, a = [], [], 0
        for n in s["lens"]:                       # sequence by sequence: the scores of one are all the memory it takes
            x = qkv.detach()[a:a + n].requires_grad_(True)
            o = _packed_attention(x, [n], nq, nkv, hd)
            grads.append(torch.autograd.grad(o, x, s["dout"][a:a + n].double())[0])
            outs.append(o.detach())
            a += n
        return torch.cat(outs, 0), torch.cat(grads, 0)
    if k == "decode_attn":
        kc, vc = s["k"].double(), s["v"].double()
        out = _decode_attention(s["qkv"].double(), kc, vc, s["lens"].tolist(), case["nq"], case["nkv"], case["hd"], s["lens"])
        return out, kc, vc
    if k == "norm":
        d, x, w = (s[n].double() for n in ("d", "x", "w"))
        res = d + x
        if case["mode"] == "infer":
            return _rms(res, w), res
        # the residual stream is stored in its own type and normalised as stored
        stored = (s["d"].float() + s["x"].float()).to(s["x"].dtype).double().requires_grad_(True)
        w.requires_grad_(True)
        y = _rms(stored, w)
        dx, dw = torch.autograd.grad(y, (stored, w), s["dy"].double())
        return y.detach(), res, dx + s["dres"].double(), dw
    if k == "sample":
        return _exact_sample(s, case)
    if k == "moe":
        return _exact_moe(s, case)
    if k == "window_attn":
        return _exact_window(s, case)
    if k == "delta":
        return _exact_delta(s, case)
    if k == "train_step":
        w = {n: t.double().requires_grad_(True) for n, t in s["weights"].items()}
        h = _exact_llama(case, w, s["ids"], s["lens"], _pos(s["lens"]))
        lp = torch.log_softmax(h @ w[f"{case['layers'] + 1}.head.weight"].T, -1).gather(1, s["labels"].unsqueeze(1)).squeeze(1)
        grads = torch.autograd.grad((lp * s["dlogp"].double()).sum(), list(w.values()))
        return lp.detach(), dict(zip(w, grads))
    hd, lens = case["width"] // case["heads"], s["lens"].tolist()
    w = {n: t.double() for n, t in s["weights"].items()}
    kc, vc = ([t.permute(0, 2, 1, 3).double() for t in s[n]] for n in ("k", "v"))
    x = w["0.wte.weight"][s["ids"]]
    for i in range(1, case["layers"] + 1):
        qkv = _rms(x, w[f"{i}.attn.ln.weight"]) @ w[f"{i}.attn.qkv.weight"].T
        x = x + _decode_attention(qkv, kc[i - 1], vc[i - 1], lens, case["heads"], case["kv"], hd, s["lens"]) @ w[f"{i}.attn.o.weight"].T
        gu = _rms(x, w[f"{i}.mlp.ln.weight"]) @ w[f"{i}.mlp.gate_up.weight"].T
        x = x + (torch.nn.functional.silu(gu[:, :case["ff"]]) * gu[:, case["ff"]:]) @ w[f"{i}.mlp.down.weight"].T
    return _rms(x, w[f"{case['layers']}.ln_f.weight"]) @ w[f"{case['layers'] + 1}.head.weight"].T, kc, vc
