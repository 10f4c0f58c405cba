"""The work a user of this framework has it do, as measurable cases.

Reinforcement learning of a language model spends its time in two places: the training step (packed sequences through
attention, projections, norms, MLP or experts, the fused output head, forward and backward) and the rollout (prefill, then
decode steps over a paged cache). Every case is one layer, block or whole call of those, through the entry point that the
trainer, the rollout engine or a model file uses, on the shapes of the architectures this repository names.

``listed()`` has the cases, ``draw()`` more of the same ranges, ``prepare()`` makes what a program holds before the call,
``run()`` is one pass, ``exact()`` the same result in 64-bit torch without this repository's code.
"""
import math
import random

import torch

# The architectures of this repository: hidden size, query heads, kv heads, MLP size, vocabulary, qkv bias, per-head q/k norm, rope base
ARCHS = {
    "qwen2.5-7b": dict(dim=3584, hq=28, hkv=4, ffn=18944, vocab=152064, bias=True, qk_norm=False, theta=1e6),
    "llama3-8b": dict(dim=4096, hq=32, hkv=8, ffn=14336, vocab=128256, bias=False, qk_norm=False, theta=5e5),
    "qwen3-32b": dict(dim=5120, hq=64, hkv=8, ffn=25600, vocab=151936, bias=False, qk_norm=True, theta=1e6),
    "tiny-qwen2-d128": dict(dim=512, hq=4, hkv=2, ffn=1024, vocab=32000, bias=True, qk_norm=False, theta=1e6),
}
HEAD_DIM = 128
EPS = 1e-6
PAGE = 128


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one micro-batch of rollouts in training: seven sequences of uneven length packed to 8192 tokens (the packing
        # size of the GRPO benchmark), attention alone, forward and backward
        {"name": "attn_packed_8k", "kind": "attention", "hq": 28, "hkv": 4, "causal": True,
         "lens": "1536,1200,977,1536,640,1311,992"},
        # long-context training: one sequence that fills a micro-batch of 16384 tokens
        {"name": "attn_long_16k", "kind": "attention", "hq": 32, "hkv": 8, "causal": True, "lens": "16384"},
        # bidirectional attention of the diffusion transformer (dit-2b: 16 heads), two videos of uneven token count
        {"name": "attn_full_dit", "kind": "attention", "hq": 16, "hkv": 16, "causal": False, "lens": "3600,2340"},
        # a whole transformer block in training, the 7B benchmark model at its 8192-token micro-batch
        {"name": "block_7b_8k", "kind": "block", "arch": "qwen2.5-7b", "lens": "1536,1536,1536,1536,1536,512"},
        # the same on a short, ragged micro-batch: fine-tuning on short samples
        {"name": "block_8b_ragged", "kind": "block", "arch": "llama3-8b", "lens": "301,77,150,475"},
        # smallest call: prompt through a small model to logits, no gradients; launches and host work count
        {"name": "tiny_prefill", "kind": "model", "arch": "tiny-qwen2-d128", "layers": 2, "lens": "57"},
        # residual add + RMSNorm of the 7B model, forward and backward; twice per block
        {"name": "norm_8k", "kind": "norm", "tokens": 8192, "dim": 3584},
        # output head in training: log-probability and entropy of 2048 response tokens over the full vocabulary,
        # forward and the gradients of hidden states and head weight
        {"name": "head_2k", "kind": "head", "tokens": 2048, "dim": 3584, "vocab": 152064},
        # one block of a decode step at the rollout benchmark's 128 sequences, replayed from a CUDA graph as the engine does
        {"name": "decode_b128", "kind": "decode", "arch": "qwen2.5-7b", "batch": 128, "max_len": 1536},
        # the tail of a rollout: five sequences left
        {"name": "decode_b5", "kind": "decode", "arch": "llama3-8b", "batch": 5, "max_len": 700},
        # mixture-of-experts layer of the Qwen3-30B-A3B shape in training: routing, experts, gradients
        {"name": "moe_4k", "kind": "moe", "tokens": 4096, "dim": 2048, "ffn": 768, "experts": 128, "top_k": 8},
        # rollout on block-scaled fp8 weights: prefill of 4096 tokens through the gate/up projection
        {"name": "fp8_linear_4k", "kind": "fp8", "tokens": 4096, "n": 37888, "k": 3584},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_lens(rng, total):
    """`total` tokens cut into one to eight sequences of uneven length."""
    n = min(rng.choice([1, 2, 3, 5, 8]), total)
    cuts = sorted(rng.sample(range(1, total), n - 1)) if n > 1 else []
    return ",".join(str(b - a) for a, b in zip([0] + cuts, cuts + [total]))


def draw(rng):
    kind = rng.choice(["attention", "attention", "attention", "block", "block", "model", "norm", "head", "decode", "decode",
                       "decode", "moe", "fp8"])
    if kind == "attention":
        causal = rng.random() < 0.7
        hq, hkv = rng.choice([(28, 4), (32, 8), (16, 16), (4, 2)])
        return {"kind": kind, "hq": hq, "hkv": hkv, "causal": causal,
                "lens": _draw_lens(rng, _log_int(rng, 40, 16384 if causal else 8192))}
    if kind == "block":
        arch = rng.choice(["qwen2.5-7b", "llama3-8b", "qwen3-32b", "tiny-qwen2-d128"])
        return {"kind": kind, "arch": arch, "lens": _draw_lens(rng, _log_int(rng, 64, 3500 if arch == "qwen3-32b" else 8192))}
    if kind == "model":
        return {"kind": kind, "arch": "tiny-qwen2-d128", "layers": 2, "lens": _draw_lens(rng, _log_int(rng, 8, 2048))}
    if kind == "norm":
        return {"kind": kind, "tokens": _log_int(rng, 16, 16384), "dim": rng.choice([512, 2048, 3584, 4096, 5120, 7168])}
    if kind == "head":
        arch = rng.choice(["qwen2.5-7b", "llama3-8b", "tiny-qwen2-d128"])
        return {"kind": kind, "tokens": _log_int(rng, 64, 2048), "dim": ARCHS[arch]["dim"], "vocab": ARCHS[arch]["vocab"]}
    if kind == "decode":
        arch = rng.choice(["qwen2.5-7b", "llama3-8b", "tiny-qwen2-d128"])
        batch = _log_int(rng, 1, 256)
        return {"kind": kind, "arch": arch, "batch": batch, "max_len": _log_int(rng, 32, min(16384, 262144 // batch))}
    if kind == "moe":
        experts, top_k, dim, ffn = rng.choice([(128, 8, 2048, 768), (16, 8, 2048, 768), (8, 2, 256, 128)])
        return {"kind": kind, "tokens": _log_int(rng, 64, 8192), "dim": dim, "ffn": ffn, "experts": experts, "top_k": top_k}
    arch = ARCHS[rng.choice(["qwen2.5-7b", "llama3-8b"])]
    n, k = rng.choice([(2 * arch["ffn"], arch["dim"]), (arch["dim"], arch["ffn"]),
                       ((arch["hq"] + 2 * arch["hkv"]) * HEAD_DIM, arch["dim"])])
    return {"kind": "fp8", "tokens": _log_int(rng, 1, 8192), "n": n, "k": k}


def _lens(case):
    return [int(x) for x in case["lens"].split(",")]


def _context_lens(case):
    """Cached tokens per sequence of a decode step: spread between a quarter of the longest and the longest."""
    rng = random.Random(case["batch"] * 100003 + case["max_len"])
    lo = max(1, case["max_len"] // 4)
    return [case["max_len"]] + [rng.randint(lo, case["max_len"]) for _ in range(case["batch"] - 1)]


# ------------------------------------------------------------------------------------------------ inputs
def _inputs(case, seed):
    """Plain tensors, made from the seed alone. Weights have the initialisation's spread (0.02), activations that of
    normalised hidden states (1), gradients that of a mean over the micro-batch."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))

    def bf(*shape, std=1.0):
        return torch.empty(*shape, dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=g)

    def gain(n):
        return torch.empty(n, dtype=torch.bfloat16, device="cuda").uniform_(0.5, 1.5, generator=g)

    kind = case["kind"]
    d = HEAD_DIM

    def packed(lens):
        cu = torch.tensor([0] + lens, device="cuda").cumsum(0).to(torch.int32)
        pos = torch.cat([torch.arange(n, device="cuda") for n in lens])
        return cu, pos

    def block_weights(a):
        w = {"input_layernorm": gain(a["dim"]),
             "self_attn.qkv_proj.weight": bf((a["hq"] + 2 * a["hkv"]) * d, a["dim"], std=0.02),
             "self_attn.o_proj.weight": bf(a["dim"], a["hq"] * d, std=0.02),
             "post_attention_layernorm": gain(a["dim"]),
             "mlp.gate_up_proj.weight": bf(2 * a["ffn"], a["dim"], std=0.02),
             "mlp.down_proj.weight": bf(a["dim"], a["ffn"], std=0.02)}
        if a["bias"]:
            w["self_attn.qkv_proj.bias"] = bf((a["hq"] + 2 * a["hkv"]) * d, std=0.5)
        if a["qk_norm"]:
            w["self_attn.q_norm"], w["self_attn.k_norm"] = gain(d), gain(d)
        return w

    if kind == "attention":
        lens, hq, hkv = _lens(case), case["hq"], case["hkv"]
        T = sum(lens)
        cu, _ = packed(lens)
        return {"qkv": bf(T, (hq + 2 * hkv) * d), "dout": bf(T, hq, d), "cu": cu, "lens": lens}
    if kind == "block":
        a, lens = ARCHS[case["arch"]], _lens(case)
        T = sum(lens)
        cu, pos = packed(lens)
        return {"w": block_weights(a), "h": bf(T, a["dim"]), "res": bf(T, a["dim"]), "dh": bf(T, a["dim"]),
                "dres": bf(T, a["dim"]), "cu": cu, "pos": pos, "lens": lens}
    if kind == "model":
        a, lens = ARCHS[case["arch"]], _lens(case)
        cu, pos = packed(lens)
        w = {"embed_tokens.weight": bf(a["vocab"], a["dim"]), "norm": gain(a["dim"]),
             "lm_head.weight": bf(a["vocab"], a["dim"], std=0.02)}
        for i in range(case["layers"]):
            w.update({"layers.%d.%s" % (i, k): v for k, v in block_weights(a).items()})
        ids = torch.randint(0, a["vocab"], (sum(lens),), device="cuda", generator=g)
        return {"w": w, "ids": ids, "cu": cu, "pos": pos, "lens": lens}
    if kind == "norm":
        T, H = case["tokens"], case["dim"]
        return {"x": bf(T, H), "res": bf(T, H, std=3.0), "w": gain(H), "dy": bf(T, H), "dres": bf(T, H)}
    if kind == "head":
        T, H, V = case["tokens"], case["dim"], case["vocab"]
        return {"hidden": bf(T, H), "w": bf(V, H, std=0.02),
                "labels": torch.randint(0, V, (T,), device="cuda", generator=g),
                "dlp": torch.empty(T, device="cuda").normal_(0.0, 1.0 / T, generator=g)}
    if kind == "decode":
        a, B = ARCHS[case["arch"]], case["batch"]
        lens = _context_lens(case)
        per = [(n + PAGE - 1) // PAGE for n in lens]
        total = sum(per)
        order = (torch.randperm(total, generator=torch.Generator().manual_seed(int(seed))) + 1).tolist()  # page 0 is scratch
        table = torch.zeros(B, max(per) + 1, dtype=torch.int32)
        at = 0
        for b, n in enumerate(per):
            table[b, :n] = torch.tensor(order[at:at + n], dtype=torch.int32)
            at += n
        last = torch.tensor([n - 1 for n in lens])
        slots = table[torch.arange(B), last // PAGE].long() * PAGE + last % PAGE
        return {"w": block_weights(a), "next_norm": gain(a["dim"]), "x": bf(B, a["dim"]), "res": bf(B, a["dim"], std=3.0),
                "cache": bf(total + 1, 2, a["hkv"], PAGE, d), "table": table.cuda(), "lens": lens,
                "seq_lens": torch.tensor(lens, dtype=torch.int32, device="cuda"), "pos": last.cuda(),
                "slots": slots.to(torch.int32).cuda()}
    if kind == "moe":
        T, H, I, E = case["tokens"], case["dim"], case["ffn"], case["experts"]
        logits = torch.empty(T, E, device="cuda").normal_(generator=g)
        logits += 0.5 * torch.empty(E, device="cuda").normal_(generator=g)    # some experts are more popular than others
        return {"x": bf(T, H), "logits": logits, "w_gate_up": bf(E, 2 * I, H, std=0.02), "w_down": bf(E, H, I, std=0.02),
                "dout": bf(T, H)}
    if kind == "fp8":
        return {"x": bf(case["tokens"], case["k"]), "w": bf(case["n"], case["k"], std=0.02)}
    raise ValueError(kind)


def prepare(case, seed):
    from cosmos_rl_b200.models.gpt import GPT, GPTArgs, GPTBlock
    from cosmos_rl_b200.ops import functional as F

    s = _inputs(case, seed)
    kind = s["kind"] = case["kind"]

    def args(a, layers):
        return GPTArgs(vocab_size=a["vocab"], dim=a["dim"], n_layers=layers, n_heads=a["hq"], n_kv_heads=a["hkv"],
                       head_dim=HEAD_DIM, ffn_dim=a["ffn"], norm_eps=EPS, rope_theta=a["theta"], qkv_bias=a["bias"],
                       qk_norm=a["qk_norm"])

    def load(module, weights):
        module = module.to_empty(device="cuda").to(torch.bfloat16)
        with torch.no_grad():
            for name, p in module.named_parameters():
                p.copy_(weights[name])
        return module

    if kind == "attention":
        s["qkv"].requires_grad_(True)
        s["heads"], s["causal"], s["max_len"] = (case["hq"], case["hkv"]), case["causal"], max(s["lens"])
    elif kind == "block":
        with torch.device("meta"):
            block = GPTBlock(args(ARCHS[case["arch"]], 1))
        s["block"] = load(block, s.pop("w"))
        for p in s["block"].parameters():
            p.grad = torch.zeros_like(p)        # the trainer keeps its gradients in one buffer for the whole run
        s["grads"] = [p.grad for p in s["block"].parameters()]
        s["h"].requires_grad_(True)
        s["res"].requires_grad_(True)
        s["max_len"] = max(s["lens"])
    elif kind == "model":
        with torch.device("meta"):
            model = GPT(args(ARCHS[case["arch"]], case["layers"]))
        s["model"] = load(model, s.pop("w"))
        s["max_len"] = max(s["lens"])
    elif kind == "norm":
        for k in ("x", "res", "w"):
            s[k].requires_grad_(True)
    elif kind == "head":
        s["hidden"].requires_grad_(True)
        s["w"].requires_grad_(True)
    elif kind == "decode":
        a = ARCHS[case["arch"]]
        s["arch"] = a
        # the layout that this head size and page size are served in: V slabs [d, page]; the engine keeps its cache so
        assert F.tc_decode_supported(HEAD_DIM, PAGE, a["hq"], a["hkv"])
        s["out"] = None

        def step():
            w, d = s["w"], HEAD_DIM
            q = F.skinny_qkv_rope_append(s["x"], w["self_attn.qkv_proj.weight"], w.get("self_attn.qkv_proj.bias"), s["pos"],
                                         s["slots"], a["theta"], a["hq"], a["hkv"], d, s["cache"], True)
            o = F.paged_decode(q, s["cache"], s["table"], s["seq_lens"], v_transposed=True)
            x, res = F.skinny_linear_residual_rmsnorm(o.reshape(o.shape[0], -1), w["self_attn.o_proj.weight"], s["res"],
                                                      w["post_attention_layernorm"], EPS)
            act = F.skinny_gate_up_swiglu(x, w["mlp.gate_up_proj.weight"])
            y, res = F.skinny_linear_residual_rmsnorm(act, w["mlp.down_proj.weight"], res, s["next_norm"], EPS)
            return {"q": q, "y": y, "res": res, "cache": s["cache"]}

        # as the rollout engine does: warm up on a side stream, then capture the step once and replay it
        with torch.no_grad():
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                step()
            torch.cuda.current_stream().wait_stream(side)
            s["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s["graph"]):
                s["out"] = step()
    elif kind == "moe":
        s["top_k"], s["experts"] = case["top_k"], case["experts"]
        for k in ("x", "w_gate_up", "w_down"):
            s[k].requires_grad_(True)
    elif kind == "fp8":
        s["w"]._fp8 = F.quant_fp8_block(s["w"], 128)     # what the rollout's fp8 weight store attaches
    return s


# ------------------------------------------------------------------------------------------------ one pass
def run(s):
    from cosmos_rl_b200.ops import functional as F
    kind = s["kind"]
    if kind == "attention":
        hq, hkv = s["heads"]
        d = HEAD_DIM
        q, k, v = s["qkv"].split([hq * d, hkv * d, hkv * d], dim=-1)
        q, k, v = q.unflatten(-1, (hq, d)), k.unflatten(-1, (hkv, d)), v.unflatten(-1, (hkv, d))
        if s["causal"]:
            o = F.varlen_attention(q, k, v, s["cu"], s["max_len"])
        else:
            o = F.full_attention(q, k, v, s["cu"], s["cu"], s["max_len"], s["max_len"])
        dqkv, = torch.autograd.grad(o, s["qkv"], s["dout"])
        return {"o": o, "dqkv": dqkv}
    if kind == "block":
        torch._foreach_zero_(s["grads"])
        s["h"].grad = s["res"].grad = None
        h, res = s["block"](s["h"], s["res"], s["pos"], s["cu"], s["max_len"])
        torch.autograd.backward([h, res], [s["dh"], s["dres"]])
        out = {"h": h, "res": res, "dh": s["h"].grad, "dres": s["res"].grad}
        out.update({n: p.grad for n, p in s["block"].named_parameters()})
        return out
    if kind == "model":
        with torch.no_grad():
            hidden = s["model"](s["ids"], s["pos"], s["cu"], s["max_len"])
            return {"hidden": hidden, "logits": s["model"].logits(hidden)}
    if kind == "norm":
        y, res = F.rms_norm(s["x"], s["w"], EPS, residual=s["res"])
        dx, dw = torch.autograd.grad([y, res], [s["x"], s["w"]], [s["dy"], s["dres"]])
        return {"y": y, "res": res, "dx": dx, "dw": dw}
    if kind == "head":
        lp, ent = F.fused_logprob(s["hidden"], s["w"], s["labels"])
        dh, dw = torch.autograd.grad(lp, [s["hidden"], s["w"]], s["dlp"])
        return {"logprob": lp, "entropy": ent, "dh": dh, "dw": dw}
    if kind == "decode":
        s["graph"].replay()
        return s["out"]
    if kind == "moe":
        from cosmos_rl_b200.ops import moe
        counts = torch.zeros(s["experts"], dtype=torch.int32, device="cuda")
        probs, idx = moe.route_topk(s["logits"], s["top_k"], True, counts)
        probs.requires_grad_(True)
        o = moe.moe_experts(s["x"], probs, idx, s["w_gate_up"], s["w_down"], counts)
        dx, dp, dgu, dd = torch.autograd.grad(o, [s["x"], probs, s["w_gate_up"], s["w_down"]], s["dout"])
        return {"o": o, "idx": idx, "probs": probs, "dx": dx, "dprobs": dp, "dw_gate_up": dgu, "dw_down": dd}
    with torch.no_grad():
        return {"y": F.linear_maybe_fp8(s["x"], s["w"])}


# ------------------------------------------------------------------------------------------------ floors, tolerances
def _pairs(lens, causal):
    """(query, key) pairs that attention has to score."""
    return sum(n * (n + 1) // 2 if causal else n * n for n in lens)


def work(case):
    kind, d = case["kind"], HEAD_DIM
    if kind == "attention":
        lens, hq, hkv = _lens(case), case["hq"], case["hkv"]
        T = sum(lens)
        # read qkv, dout; write o, dqkv. Two products forward, five backward.
        return {"bytes": 2 * T * d * (2 * (hq + 2 * hkv) + 2 * hq), "flops": 14 * d * hq * _pairs(lens, case["causal"])}
    if kind in ("block", "model"):
        a, lens = ARCHS[case["arch"]], _lens(case)
        T = sum(lens)
        weights = a["dim"] * (2 * a["hq"] + 2 * a["hkv"]) * d + 3 * a["dim"] * a["ffn"]
        if kind == "block":
            return {"bytes": 2 * (2 * weights + 8 * T * a["dim"]), "flops": 6 * T * weights + 14 * d * a["hq"] * _pairs(lens, True)}
        head = a["vocab"] * a["dim"]
        return {"bytes": 2 * (case["layers"] * weights + head + T * (2 * a["dim"] + a["vocab"])),
                "flops": 2 * T * (case["layers"] * weights + head) + case["layers"] * 4 * d * a["hq"] * _pairs(lens, True)}
    if kind == "norm":
        # read x, res, dy, dres; write y, res', dx
        return {"bytes": 2 * (7 * case["tokens"] * case["dim"] + 2 * case["dim"]), "flops": 20 * case["tokens"] * case["dim"]}
    if kind == "head":
        T, H, V = case["tokens"], case["dim"], case["vocab"]
        # logits, and once their gradient is known two more products; the logits are formed again in backward, since they are not kept
        return {"bytes": 2 * (2 * V * H + 2 * T * H) + 16 * T, "flops": 6 * T * H * V}
    if kind == "decode":
        a, lens = ARCHS[case["arch"]], _context_lens(case)
        weights = a["dim"] * (2 * a["hq"] + 2 * a["hkv"]) * d + 3 * a["dim"] * a["ffn"]
        B = case["batch"]
        return {"bytes": 2 * (weights + 2 * a["hkv"] * d * sum(lens) + B * (4 * a["dim"] + a["hq"] * d)),
                "flops": 2 * B * weights + 4 * a["hq"] * d * sum(lens)}
    if kind == "moe":
        T, H, I, E, k = case["tokens"], case["dim"], case["ffn"], case["experts"], case["top_k"]
        return {"bytes": 2 * (2 * 3 * E * H * I + 4 * T * H) + 4 * T * E, "flops": 18 * T * k * H * I}
    T, N, K = case["tokens"], case["n"], case["k"]
    return {"bytes": 2 * T * K + N * K + 2 * T * N, "flops": 2 * T * N * K}


def tolerance(case):
    """About four times the measured distance between the path and 64-bit torch on the same inputs (2-norm, worst output):
    attention 2.5e-3, block 1.1e-2 (the weight gradient of its first norm, at the end of the chain), model 4.2e-3, norm
    2.4e-3, head 2.4e-3, decode 3.6e-3, experts 4.2e-3, fp8 5.5e-3. One rounding to bf16 alone gives 1.7e-3."""
    return {"rel": {"attention": 1e-2, "block": 4e-2, "model": 1.7e-2, "norm": 1e-2, "head": 1e-2, "decode": 1.5e-2,
                    "moe": 1.7e-2, "fp8": 2.2e-2}[case["kind"]], "differ": 0.0}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms64(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w


def _rope64(x, pos, theta):
    """Rotate-half rotary embedding of [T, heads, d]."""
    d = x.shape[-1]
    inv = theta ** (-torch.arange(0, d, 2, device=x.device, dtype=torch.float64) / d)
    ang = pos.double()[:, None] * inv
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b = x[..., :d // 2], x[..., d // 2:]
    return torch.cat([a * c - b * s, b * c + a * s], dim=-1)


def _attention64(q, k, v, lens, causal, dout=None):
    """o [T, hq, d]; with `dout` also dq, dk, dv. One head of one sequence at a time."""
    hq, hkv, d = q.shape[1], k.shape[1], q.shape[2]
    scale, o = 1.0 / math.sqrt(d), torch.zeros_like(q)
    grads = [torch.zeros_like(t) for t in (q, k, v)] if dout is not None else None
    at = 0
    for n in lens:
        rows = slice(at, at + n)
        at += n
        for h in range(hq):
            kv = h // (hq // hkv)
            p = (q[rows, h] @ k[rows, kv].T).mul_(scale)
            if causal:
                p.masked_fill_(torch.ones(n, n, dtype=torch.bool, device=q.device).triu_(1), float("-inf"))
            p = torch.softmax(p, dim=-1)
            o[rows, h] = p @ v[rows, kv]
            if dout is not None:
                grads[2][rows, kv] += p.T @ dout[rows, h]
                dp = dout[rows, h] @ v[rows, kv].T
                dp.sub_((o[rows, h] * dout[rows, h]).sum(-1, keepdim=True)).mul_(p).mul_(scale)
                grads[0][rows, h] = dp @ k[rows, kv]
                grads[1][rows, kv] += dp.T @ q[rows, h]
    return o if dout is None else (o, *grads)


class _Attention64(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, lens):
        ctx.save_for_backward(q, k, v)
        ctx.lens = lens
        return _attention64(q, k, v, lens, True)

    @staticmethod
    def backward(ctx, dout):
        return (*_attention64(*ctx.saved_tensors, ctx.lens, True, dout)[1:], None)


def _block64(a, w, h, res, pos, lens):
    """(h, res) -> (mlp output, residual stream); h + res is the stream, res is None for the first block."""
    d, hq, hkv = HEAD_DIM, a["hq"], a["hkv"]
    res = h if res is None else h + res
    x = _rms64(res, w["input_layernorm"])
    qkv = x @ w["self_attn.qkv_proj.weight"].T
    if a["bias"]:
        qkv = qkv + w["self_attn.qkv_proj.bias"]
    q, k, v = (t.unflatten(-1, (-1, d)) for t in qkv.split([hq * d, hkv * d, hkv * d], dim=-1))
    if a["qk_norm"]:
        q, k = _rms64(q, w["self_attn.q_norm"]), _rms64(k, w["self_attn.k_norm"])
    o = _Attention64.apply(_rope64(q, pos, a["theta"]), _rope64(k, pos, a["theta"]), v, lens)
    res = res + o.flatten(1) @ w["self_attn.o_proj.weight"].T
    gate, up = (_rms64(res, w["post_attention_layernorm"]) @ w["mlp.gate_up_proj.weight"].T).chunk(2, dim=-1)
    return (torch.nn.functional.silu(gate) * up) @ w["mlp.down_proj.weight"].T, res


def _quant64(x, rows):
    """x rounded to e4m3 with one scale per `rows` x 128 values, and scaled back; scales are held in 32 bits."""
    R, C = x.shape
    nr, nc = -(-R // rows), -(-C // 128)
    pad = x.new_zeros(nr * rows, nc * 128, dtype=torch.float32)
    pad[:R, :C] = x
    blocks = pad.view(nr, rows, nc, 128)
    scale = (blocks.abs().amax(dim=(1, 3)).clamp_min(1e-12) / 448.0)[:, None, :, None]
    q = (blocks / scale).clamp(-448.0, 448.0).to(torch.float8_e4m3fn)
    return (q.double() * scale.double()).view(nr * rows, nc * 128)[:R, :C]


def exact(case, seed):
    kind, d = case["kind"], HEAD_DIM
    s = _inputs(case, seed)
    with torch.no_grad():
        if kind == "attention":
            hq, hkv = case["hq"], case["hkv"]
            q, k, v = (t.unflatten(-1, (-1, d)) for t in s["qkv"].double().split([hq * d, hkv * d, hkv * d], dim=-1))
            o, dq, dk, dv = _attention64(q, k, v, s["lens"], case["causal"], s["dout"].double())
            return {"o": o, "dqkv": torch.cat([dq.flatten(1), dk.flatten(1), dv.flatten(1)], dim=-1)}
        if kind == "model":
            w = {k: v.double() for k, v in s["w"].items()}
            h, res = w["embed_tokens.weight"][s["ids"]], None
            for i in range(case["layers"]):
                pre = "layers.%d." % i
                h, res = _block64(ARCHS[case["arch"]], {k[len(pre):]: v for k, v in w.items() if k.startswith(pre)}, h, res,
                                  s["pos"], s["lens"])
            hidden = _rms64(h + res, w["norm"])
            return {"hidden": hidden, "logits": hidden @ w["lm_head.weight"].T}
        if kind == "head":
            x, w, T = s["hidden"].double(), s["w"].double(), case["tokens"]
            logits = x @ w.T
            lse = torch.logsumexp(logits, dim=-1)
            lp = logits.gather(-1, s["labels"][:, None]).squeeze(-1) - lse
            p = (logits - lse[:, None]).exp_()
            ent = lse - p.mul(logits).sum(-1)
            del logits
            g = s["dlp"].double()
            p.mul_(-g[:, None])
            p[torch.arange(T, device="cuda"), s["labels"]] += g
            return {"logprob": lp, "entropy": ent, "dh": p @ w, "dw": p.T @ x}
        if kind == "decode":
            a, B, lens = ARCHS[case["arch"]], case["batch"], s["lens"]
            hq, hkv = a["hq"], a["hkv"]
            w = {k: v.double() for k, v in s["w"].items()}
            qkv = s["x"].double() @ w["self_attn.qkv_proj.weight"].T
            if a["bias"]:
                qkv = qkv + w["self_attn.qkv_proj.bias"]
            q, k, v = (t.unflatten(-1, (-1, d)) for t in qkv.split([hq * d, hkv * d, hkv * d], dim=-1))
            q, k = _rope64(q, s["pos"], a["theta"]), _rope64(k, s["pos"], a["theta"])
            cache = s["cache"].double()
            o = torch.empty(B, hq, d, dtype=torch.float64, device="cuda")
            for b, n in enumerate(lens):
                page, off = divmod(int(s["slots"][b]), PAGE)
                cache[page, 0, :, off] = k[b]
                cache[page, 1].view(hkv, d, PAGE)[:, :, off] = v[b]           # V slabs are stored [d, page]
                pages = s["table"][b, :(n + PAGE - 1) // PAGE].long()
                kk = cache[pages, 0].transpose(0, 1).reshape(hkv, -1, d)[:, :n]
                vv = cache[pages, 1].view(-1, hkv, d, PAGE).permute(1, 0, 3, 2).reshape(hkv, -1, d)[:, :n]
                p = torch.softmax(q[b].view(hkv, hq // hkv, d) @ kk.transpose(1, 2) / math.sqrt(d), dim=-1)
                o[b] = (p @ vv).reshape(hq, d)
            res = s["res"].double() + o.flatten(1) @ w["self_attn.o_proj.weight"].T
            gate, up = (_rms64(res, w["post_attention_layernorm"]) @ w["mlp.gate_up_proj.weight"].T).chunk(2, dim=-1)
            res = res + (torch.nn.functional.silu(gate) * up) @ w["mlp.down_proj.weight"].T
            return {"q": q, "y": _rms64(res, s["next_norm"].double()), "res": res, "cache": cache}
        if kind == "moe":
            x, dout = s["x"].double(), s["dout"].double()
            p = torch.softmax(s["logits"].double(), dim=-1)
            probs, idx = torch.topk(p, case["top_k"], dim=-1)
            probs = probs / probs.sum(-1, keepdim=True)
            o, dx, dp = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(probs)
            dgu, dd = (torch.zeros_like(s[k], dtype=torch.float64) for k in ("w_gate_up", "w_down"))
            for e in range(case["experts"]):
                tok, slot = (idx == e).nonzero(as_tuple=True)
                wg, wd = s["w_gate_up"][e].double(), s["w_down"][e].double()
                gate, up = (x[tok] @ wg.T).chunk(2, dim=-1)
                sg = torch.sigmoid(gate)
                act = gate * sg * up
                y, pr = act @ wd.T, probs[tok, slot][:, None]
                o.index_add_(0, tok, y * pr)
                dp[tok, slot] = (y * dout[tok]).sum(-1)
                dy = dout[tok] * pr
                dd[e] = dy.T @ act
                dact = dy @ wd
                dgate_up = torch.cat([dact * up * (sg + gate * sg * (1 - sg)), dact * gate * sg], dim=-1)
                dgu[e] = dgate_up.T @ x[tok]
                dx.index_add_(0, tok, dgate_up @ wg)
            return {"o": o, "idx": idx.to(torch.int32), "probs": probs, "dx": dx, "dprobs": dp, "dw_gate_up": dgu,
                    "dw_down": dd}
        if kind == "fp8":
            return {"y": _quant64(s["x"], 1) @ _quant64(s["w"], 128).T}
    if kind == "norm":
        x, res, w = (s[k].double().requires_grad_(True) for k in ("x", "res", "w"))
        total = x + res
        y = _rms64(total, w)
        dx, dw = torch.autograd.grad([y, total], [x, w], [s["dy"].double(), s["dres"].double()])
        return {"y": y, "res": total, "dx": dx, "dw": dw}
    a = ARCHS[case["arch"]]
    w = {k: v.double().requires_grad_(True) for k, v in s["w"].items()}
    h, res = s["h"].double().requires_grad_(True), s["res"].double().requires_grad_(True)
    out = _block64(a, w, h, res, s["pos"], s["lens"])
    names = sorted(w)
    grads = torch.autograd.grad(out, [h, res] + [w[n] for n in names], [s["dh"].double(), s["dres"].double()])
    return {"h": out[0], "res": out[1], "dh": grads[0], "dres": grads[1], **dict(zip(names, grads[2:]))}
