"""The workloads of the FP8 linear path as its users run them, for timing and for comparison.

Two kinds of program call this package.  Engines (``kernels.*``, ``stack.LinearStack``) own their
buffers, enqueue a layer stack once and replay it as a CUDA graph for every inference.  Models
whose ``nn.Linear`` modules were replaced by ``runtime.SM100FP8Linear`` call one projection after
the other from Python.  The families below are those calls, over the sizes of the configurations in
``stack.SPECS``, the tests and the benchmark:

``module``    one replaced projection on bf16 activations (dynamic per-tensor pack + GEMM + bias)
``linear``    one engine linear: per-token quantiser, GEMM with row / column scales and bias
``gemma``     decoder layers with gated feed-forward: vision-language prefix and action expert
``wan``       diffusion-transformer blocks (self / cross attention projections, GELU feed-forward)
``qkv``       the consumer of a fused QKV accumulator of a decoder layer (rotary, cache rows)
``wan_qkv``   the same for a diffusion block (full-width norm, three-axis rotary, pooled K / V)
``combine``   merge of split-KV attention partials, quantised for the output projection

All random data is drawn on the GPU from the seed: activations N(0, 1) with a few large channels
(what the per-token scales are for), weights N(0, 0.02).
"""
import torch

from instinctflash_b200 import stack as _stack
from instinctflash_b200.kernels import attention as _attention
from instinctflash_b200.kernels import fp8 as _fp8
from instinctflash_b200.kernels import norm as _norm
from instinctflash_b200.kernels import rope as _rope
from instinctflash_b200.kernels import wan as _wan
from instinctflash_b200.runtime.torch_fp8_linear import SM100FP8Linear

DEV = "cuda"
E4M3 = torch.float8_e4m3fn
BF16 = torch.bfloat16
F16 = torch.float16


def listed():
    return [
        # one attention projection of an action-expert layer, called from Python for one episode's
        # 50 tokens: the smallest call there is, all latency
        dict(name="module_small", family="module", M=50, N=1024, K=1024, bias=False),
        # an odd number of vision-language tokens through a biased projection
        dict(name="module_ragged", family="module", M=333, N=2560, K=2048, bias=True),
        # first feed-forward projection of a video diffusion block, all tokens of a request
        dict(name="module_large", family="module", M=4680, N=14336, K=3072, bias=True),
        # the single linear of the benchmark's first configuration, called operator by operator
        dict(name="linear_single", family="linear", M=64, N=4096, K=1024, bias=True),
        # one pass of the action expert at the engine's own shapes (QKV of 10 heads of 256, output projection)
        dict(name="expert_pass", family="gemma", M=50, layers=18, hidden=1024, ffn=4096, qkv=2560, o_in=2048, episodes=1),
        # eight episodes' expert passes served together, as parallel branches of one graph
        dict(name="expert_episodes", family="gemma", M=50, layers=18, hidden=1024, ffn=4096, qkv=1536, o_in=0, episodes=8),
        # the vision-language prefix: three 256-token images and 48 text tokens
        dict(name="prefix", family="gemma", M=816, layers=4, hidden=2048, ffn=16384, qkv=2560, o_in=2048, episodes=1),
        # one image and a short, odd prompt
        dict(name="prefix_one_image", family="gemma", M=301, layers=4, hidden=2048, ffn=16384, qkv=2560, o_in=2048, episodes=1),
        # video diffusion blocks at the 5B shape, all video and action tokens
        dict(name="video_5b", family="wan", M=4680, layers=2, hidden=3072, ffn=14336, qkv=9216),
        # a block at the 14B shape with classifier-free guidance (2 x 8192 tokens): the largest
        dict(name="video_14b", family="wan", M=16384, layers=1, hidden=5120, ffn=13824, qkv=15360),
        # QKV consumer of the 5B-shape block
        dict(name="video_qkv", family="wan_qkv", batch=1, tokens=4680, heads=24, head_dim=128),
        # attention output of the expert's tokens merged over eight key ranges
        dict(name="expert_combine", family="combine", tokens=50, heads_q=8, heads_kv=1, head_dim=256, splits=8),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    family = rng.choice(("module", "module", "linear", "gemma", "gemma", "wan", "wan", "qkv", "wan_qkv", "combine"))
    if family in ("module", "linear"):
        while True:
            c = dict(family=family, M=_log_int(rng, 1, 8192), N=16 * _log_int(rng, 16, 960), K=16 * _log_int(rng, 32, 896),
                     bias=rng.random() < 0.5)
            if c["M"] * c["N"] * c["K"] < 4680 * 14336 * 3072:
                return c
    if family == "gemma":
        if rng.random() < 0.5:   # expert widths, few tokens
            return dict(family=family, M=_log_int(rng, 8, 400), layers=rng.choice((6, 12, 18)), hidden=rng.choice((768, 1024, 1280)),
                        ffn=128 * rng.randint(20, 40), qkv=rng.choice((1536, 2560)), o_in=rng.choice((0, 2048)),
                        episodes=rng.choice((1, 1, 1, 4)))
        return dict(family=family, M=_log_int(rng, 64, 1100), layers=rng.choice((1, 2, 4)), hidden=2048,
                    ffn=rng.choice((8192, 11008, 16384)), qkv=rng.choice((2560, 3072)), o_in=2048, episodes=1)
    if family == "wan":
        hidden = rng.choice((1536, 2048, 3072, 4096, 5120))
        return dict(family=family, M=_log_int(rng, 256, 16384), layers=1, hidden=hidden, ffn=256 * rng.randint(hidden // 102, 54),
                    qkv=3 * hidden)
    if family == "qkv":
        return dict(family=family, tokens=_log_int(rng, 16, 4096), heads_q=rng.choice((8, 12, 16)), heads_kv=rng.choice((1, 2, 4)),
                    head_dim=rng.choice((64, 128, 256)))
    if family == "wan_qkv":
        return dict(family=family, batch=rng.choice((1, 2)), tokens=_log_int(rng, 64, 8192), heads=rng.choice((12, 24, 40)), head_dim=128)
    return dict(family=family, tokens=_log_int(rng, 8, 1024), heads_q=rng.choice((8, 16)), heads_kv=rng.choice((1, 2, 8)),
                head_dim=rng.choice((64, 128, 256)), splits=rng.randint(2, 16))


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _activations(gen, rows, width):
    x = torch.randn(rows, width, device=DEV, generator=gen)
    x[:, torch.randperm(width, device=DEV, generator=gen)[: max(1, width // 100)]] *= 20.0
    return x.to(BF16)


def _spec(case, seed):
    return _stack.StackSpec("case", case["family"], case["layers"], case["M"], case["hidden"], case["ffn"], case["qkv"],
                            o_in=case["hidden"] if case["family"] == "wan" else case["o_in"], cross=case["family"] == "wan",
                            seed=seed % (1 << 30))


def prepare(case, seed):
    gen = _generator(seed)
    kind = case["family"]
    if kind == "module":
        lin = torch.nn.Linear(case["K"], case["N"], bias=case["bias"], device=DEV, dtype=BF16)
        with torch.no_grad():
            lin.weight.normal_(0.0, 0.02, generator=gen)
            if case["bias"]:
                lin.bias.normal_(0.0, 0.01, generator=gen)
        return dict(kind=kind, module=SM100FP8Linear(lin), x=_activations(gen, case["M"], case["K"]))
    if kind == "linear":
        M, N, K = case["M"], case["N"], case["K"]
        bias = torch.randn(N, device=DEV, generator=gen) * 0.01 if case["bias"] else None
        w = _fp8.quantize_weight(torch.randn(N, K, device=DEV, generator=gen) * 0.02, bias)
        return dict(kind=kind, x=_activations(gen, M, K), w=w, q=torch.empty(M, K, device=DEV, dtype=E4M3),
                    s=torch.empty(M, device=DEV), y=torch.empty(M, N, device=DEV, dtype=BF16))
    if kind in ("gemma", "wan"):
        spec = _spec(case, seed)
        weights = _stack.make_weights(spec, DEV)
        attn = torch.randn(spec.M, max(spec.o_in, 16), device=DEV, generator=gen).to(F16 if kind == "wan" else BF16)
        episodes = case.get("episodes", 1)
        x = [_activations(gen, spec.M, spec.hidden) for _ in range(episodes)]
        st = _stack.LinearStack(spec, weights, DEV) if episodes == 1 else _stack.EpisodeBatch(spec, weights, DEV, episodes)
        x = x[0] if episodes == 1 else x
        st.load(x, attn)
        graph = st.capture()
        res = st.res if episodes == 1 else [s.res for s in st.stacks]
        return dict(kind="stack", stack=st, graph=graph, x=x, attn=attn, res=res)
    if kind == "qkv":
        T, HQ, HKV, HD = case["tokens"], case["heads_q"], case["heads_kv"], case["head_dim"]
        width = (HQ + 2 * HKV) * HD
        k = torch.empty(T + 16, HKV, HD, device=DEV, dtype=F16)
        k.zero_()
        kw = dict(heads_q=HQ, heads_kv=HKV, head_dim=HD, row=torch.rand(T, device=DEV, generator=gen) * 0.02,
                  col=torch.rand(width, device=DEV, generator=gen), inv_freq=_rope.rope_inv_freq(HD, 10000.0, DEV),
                  pos=torch.arange(T, device=DEV).float()[:, None].contiguous(), kv_base=7)
        return dict(kind=kind, raw=torch.randn(T, width, device=DEV, generator=gen).to(BF16),
                    q=torch.empty(T, HQ, HD, device=DEV, dtype=F16), k=k, v=k.clone(), kw=kw)
    if kind == "wan_qkv":
        B, T, H, HD = case["batch"], case["tokens"], case["heads"], case["head_dim"]
        D, R = H * HD, B * T
        k = torch.empty(B, T, D, device=DEV, dtype=F16)
        kw = dict(heads=H, head_dim=HD, tokens=T, row=torch.rand(R, device=DEV, generator=gen) * 0.02,
                  col=torch.rand(3 * D, device=DEV, generator=gen), bias=torch.randn(3 * D, device=DEV, generator=gen),
                  q_norm=torch.rand(D, device=DEV, generator=gen) + 0.5, k_norm=torch.rand(D, device=DEV, generator=gen) + 0.5,
                  pos=(torch.rand(T, 3, device=DEV, generator=gen) * 60).floor(),
                  sections=(torch.arange(HD // 2, device=DEV) % 3).int(), inv_freq=_rope.rope_inv_freq(HD, 10000.0, DEV))
        return dict(kind=kind, raw=torch.randn(R, 3 * D, device=DEV, generator=gen).to(BF16),
                    q=torch.empty(R, D, device=DEV, dtype=F16), k=k, v=torch.empty_like(k), kw=kw)
    T, HQ, HD = case["tokens"], case["heads_q"], case["head_dim"]
    ws = _attention.SplitWorkspace(1, T, HQ, case["heads_kv"], HD, case["splits"], DEV)
    ws.po.normal_(generator=gen)
    ws.pm.normal_(generator=gen)
    ws.pl.uniform_(1.0, 50.0, generator=gen)
    return dict(kind="combine", ws=ws, q8=torch.empty(T, HQ * HD, device=DEV, dtype=E4M3), s=torch.empty(T, device=DEV),
                kw=dict(heads_q=HQ, heads_kv=case["heads_kv"], head_dim=HD, tokens=T))


def run(state):
    kind = state["kind"]
    if kind == "module":
        return state["module"](state["x"])
    if kind == "linear":
        _norm.row_quant(state["x"], state["q"], state["s"])
        _fp8.fp8_linear(state["q"], state["s"], state["w"], state["y"])
        return state["q"], state["s"], state["y"]
    if kind == "stack":
        state["stack"].load(state["x"], state["attn"])
        state["graph"].replay()
        return state["res"]
    if kind == "qkv":
        _rope.qkv_split(state["raw"], state["q"], state["k"], state["v"], **state["kw"])
        return state["q"], state["k"], state["v"]
    if kind == "wan_qkv":
        _wan.wan_qkv(state["raw"], state["q"], k_pool=state["k"], v_pool=state["v"], **state["kw"])
        return state["q"], state["k"], state["v"]
    _attention.attn_combine(state["ws"], q8=state["q8"], q8_scale=state["s"], **state["kw"])
    return state["q8"], state["s"]


def work(case):
    kind = case["family"]
    if kind in ("module", "linear"):
        M, N, K = case["M"], case["N"], case["K"]
        out = 2 * M * N + (M * K + 4 * M if kind == "linear" else 0)   # the engine linear hands its codes and scales on too
        return {"bytes": N * K + 2 * M * K + out + (4 * N if case["bias"] else 0), "flops": 2 * M * N * K}
    if kind in ("gemma", "wan"):
        spec, n = _spec(case, 0), case.get("episodes", 1)
        res = 2 if kind == "wan" else 4
        io = n * spec.M * spec.hidden * (2 + res) + spec.M * spec.o_in * 2
        return {"bytes": int(spec.weight_bytes()) + io, "flops": int(n * spec.flops())}
    if kind == "qkv":
        n = case["tokens"] * (case["heads_q"] + 2 * case["heads_kv"]) * case["head_dim"]
        return {"bytes": 4 * n, "flops": 8 * n}
    if kind == "wan_qkv":
        n = 3 * case["batch"] * case["tokens"] * case["heads"] * case["head_dim"]
        return {"bytes": 4 * n, "flops": 8 * n}
    n = case["tokens"] * case["heads_q"] * case["head_dim"]
    return {"bytes": case["splits"] * (4 * n + 8 * case["tokens"] * case["heads_q"]) + n + 4 * case["tokens"],
            "flops": n * (2 * case["splits"] + 3)}


def tolerance(case):
    kind = case["family"]
    if kind == "module":        # bf16 results of fp32 sums: half an ulp is 2^-9, rarely one ulp apart
        return {"rel": 4e-3, "max": 1.6e-2}
    if kind in ("linear", "combine"):   # codes too: a value at a rounding boundary may take the neighbouring e4m3 code (1/8)
        return {"rel": 4e-3, "max": 0.13}
    if kind in ("qkv", "wan_qkv"):      # f16 results; the order of the sum of squares is free
        return {"rel": 1e-3, "max": 4e-3}
    # a stack of layers: every layer quantises its input again, so that one e4m3 code on the other side
    # of a rounding boundary (the order of a 32-bit sum) is carried on and multiplied by the layers behind it;
    # adding the same K ranges in one order or another puts four prefix layers 0.9e-2 apart
    return {"rel": 2e-2, "max": 0.3}
