"""The work whose speed counts for this framework, as cases that can be timed and whose outputs can be compared.

Five kinds of work, each through the public entry points (`nanoserve_b200.ops.Kernels`, `nanoserve_b200.qwen.Qwen2Runner`):
  linear    one eager `w4_linear`: a drop-in call from a user's own model, decode to prefill
  layers    the four linears (q|k|v, o, gate|up, down) of several decoder layers, captured once in a CUDA graph and
            replayed for every step, as a batched decode loop runs them
  quantize  one `w4_quantize` of a bf16 weight matrix, as a checkpoint is loaded
  prefill   `Qwen2Runner.prefill`: a prompt through the whole model, KV cache filled, first token picked
  generate  `Qwen2Runner.generate`: prompt and greedy decoding, batch 1
Sizes are those of the benchmark configurations (7B-shaped and 70B-class layers), of the tests, or generic.  Weights
are uniform random nibbles with scales 0.005 + |N(0, 0.01)|, activations N(0, 1), as in the benchmark.
"""
import math

import torch

from nanoserve_b200.ops import Kernels
from nanoserve_b200.qwen import Qwen2Config, Qwen2Runner

# (hidden, query width, key/value width, intermediate) of one decoder layer
SHAPE_7B = dict(hidden=3584, q=3584, kv=512, inter=18944)
SHAPE_70B = dict(hidden=8192, q=8192, kv=1024, inter=28672)

# the largest listed work, which no drawn case exceeds: bytes of weights or flops of one pass
MOST_LAYER_BYTES = 1.0e9
MOST_LINEAR_FLOPS = 2.0 * 4096 * 28672 * 8192
MOST_LINEAR_WEIGHTS = 28672 * 8192

_kernels = None


def kernels():
    global _kernels
    if _kernels is None:
        _kernels = Kernels()
        _kernels.init()
    return _kernels


def listed():
    return [
        # the key or value projection of one token, called eagerly: the smallest call of the path
        dict(name="linear_m1_kv", kind="linear", M=1, N=512, K=3584, G=128),
        # single-stream decode: the linears of a 7B-shaped model's layers, one token (weights exceed the L2)
        dict(name="layers_m1", kind="layers", M=1, n_layers=4, G=128, **SHAPE_7B),
        # a few concurrent requests, or a few speculated tokens
        dict(name="layers_m4", kind="layers", M=4, n_layers=4, G=128, **SHAPE_7B),
        # a batch of requests at the odd count a server happens to have
        dict(name="layers_m13", kind="layers", M=13, n_layers=4, G=128, **SHAPE_7B),
        # the same on 70B-class layers
        dict(name="layers_70b_m8", kind="layers", M=8, n_layers=2, G=128, **SHAPE_70B),
        # a busy server: decode batch above the GEMV's sixteen tokens
        dict(name="layers_m48", kind="layers", M=48, n_layers=4, G=128, **SHAPE_7B),
        # a ragged chunk of a prompt through a generic layer with finer groups
        dict(name="linear_m777_g64", kind="linear", M=777, N=5000, K=4096, G=64),
        # prefill of a short prompt, the projection with the long contraction
        dict(name="linear_m512_down", kind="linear", M=512, N=3584, K=18944, G=128),
        # prefill of a long prompt, 70B-class: the largest matrix product
        dict(name="linear_m4096_70b", kind="linear", M=4096, N=28672, K=8192, G=128),
        # loading a checkpoint: one gate or up projection
        dict(name="quantize_7b_gate", kind="quantize", N=18944, K=3584, G=128),
        # time to first token of a 7B-shaped model
        dict(name="prefill_7b_t512", kind="prefill", T=512, n_layers=28),
        # a whole request: prompt and greedy decoding
        dict(name="generate_7b", kind="generate", T=512, n_new=64, n_layers=28),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "layers", "layers", "layers", "quantize", "prefill", "generate"])
    G = rng.choice([128, 128, 128, 128, 64, 32])
    if kind == "linear":
        while True:
            M, N = _log_int(rng, 1, 8192), _log_int(rng, 256, 28672)
            K = 128 * _log_int(rng, 4, 224)
            if M * N * K * 2.0 <= MOST_LINEAR_FLOPS and N * K <= MOST_LINEAR_WEIGHTS:
                return dict(kind=kind, M=M, N=N, K=K, G=G)
    if kind == "layers":
        shape = rng.choice([SHAPE_7B, SHAPE_7B, SHAPE_70B, None])
        if shape is None:  # a generic decoder: grouped-query attention, intermediate two to five times the hidden size
            hidden = 256 * _log_int(rng, 8, 32)
            shape = dict(hidden=hidden, q=hidden, kv=hidden // rng.choice([4, 8]), inter=256 * int(hidden * rng.uniform(2, 5) / 256))
        per_layer = shape["hidden"] * (2 * shape["q"] + 2 * shape["kv"] + 3 * shape["inter"]) * 0.52
        most = max(1, int(MOST_LAYER_BYTES / per_layer))
        least = min(most, int(math.ceil(2.5e8 / per_layer)))  # the weights of a pass exceed the L2
        return dict(kind=kind, M=_log_int(rng, 1, 200), n_layers=rng.randint(least, min(most, least + 4)), G=G, **shape)
    if kind == "quantize":
        return dict(kind=kind, N=_log_int(rng, 512, 28672), K=128 * _log_int(rng, 4, 148), G=G)
    if kind == "prefill":
        return dict(kind=kind, T=_log_int(rng, 17, 2048), n_layers=rng.randint(4, 14))
    return dict(kind=kind, T=_log_int(rng, 17, 1024), n_new=rng.randint(8, 64), n_layers=rng.randint(4, 28))


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _weights(N, K, G, gen):
    Wq = torch.randint(-2**31, 2**31 - 1, (N, K // 8), dtype=torch.int32, device="cuda", generator=gen)
    S = (0.005 + (torch.randn(N, K // G, device="cuda", generator=gen) * 0.01).abs()).to(torch.bfloat16)
    return Wq, S


def _activations(M, K, gen):
    return torch.randn(M, K, device="cuda", generator=gen).to(torch.bfloat16)


def _layer_linears(c):
    """(rows, columns) of the four matrices of one layer: q|k|v, o, gate|up, down."""
    return [(c["q"] + 2 * c["kv"], c["hidden"]), (c["hidden"], c["q"]), (2 * c["inter"], c["hidden"]), (c["hidden"], c["inter"])]


def _runner(c, seed, k):
    cfg = Qwen2Config.qwen25_7b()
    cfg.n_layers = c["n_layers"]
    r = Qwen2Runner(cfg, k, torch.device("cuda"), seed=seed, max_len=c["T"] + c.get("n_new", 0) + 8)
    prompt = torch.randint(0, cfg.vocab, (c["T"],), device="cuda", generator=_gen(seed + 1000003))
    return r, prompt


def prepare(case, seed):
    k, kind, gen = kernels(), case["kind"], _gen(seed)
    if kind == "linear":
        Wq, S = _weights(case["N"], case["K"], case["G"], gen)
        return dict(kind=kind, k=k, Wq=Wq, S=S, G=case["G"], x=_activations(case["M"], case["K"], gen))
    if kind == "layers":
        # one input per kind of matrix, shared by the layers: what a step holds at each layer boundary
        shapes = _layer_linears(case)
        xs = [_activations(case["M"], K, gen) for _, K in shapes]
        weights = [[_weights(N, K, case["G"], gen) for N, K in shapes] for _ in range(case["n_layers"])]
        outs = [[torch.empty(case["M"], N, dtype=torch.bfloat16, device="cuda") for N, _ in shapes]
                for _ in range(case["n_layers"])]
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())

        def step():
            for ws, ys in zip(weights, outs):
                for x, (Wq, S), y in zip(xs, ws, ys):
                    k.w4_linear(x, Wq, S, case["G"], out=y)

        with torch.cuda.stream(stream):
            step()
            stream.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                step()
        return dict(kind=kind, k=k, xs=xs, weights=weights, outs=outs, graph=graph)
    if kind == "quantize":
        # weights as a checkpoint holds them: small, with a spread of its own in every row
        W = torch.randn(case["N"], case["K"], device="cuda", generator=gen)
        W *= 0.02 * (0.5 + torch.rand(case["N"], 1, device="cuda", generator=gen))
        return dict(kind=kind, k=k, W=W.to(torch.bfloat16), G=case["G"])
    r, prompt = _runner(case, seed, k)
    torch.cuda.synchronize()  # the runner works on a stream of its own: weights and prompt are there before it starts
    if kind == "prefill":
        r.prefill(prompt)  # the kernels of the model are loaded
    else:
        r.generate(prompt, 4)  # captures the decode graph, which a server keeps
    return dict(kind=kind, r=r, prompt=prompt, n_new=case.get("n_new", 0))


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["k"].w4_linear(state["x"], state["Wq"], state["S"], state["G"])
    if kind == "layers":
        state["graph"].replay()
        return state["outs"]
    if kind == "quantize":
        return state["k"].w4_quantize(state["W"], state["G"])
    r, prompt = state["r"], state["prompt"]
    if kind == "prefill":
        token = r.prefill(prompt)
        T = prompt.shape[0]
    else:
        token = torch.tensor(r.generate(prompt, state["n_new"]))
        T = prompt.shape[0] + state["n_new"] - 1
    return dict(tokens=token, logits=r.logits, cache_k=r.cache_k[:, :, :T], cache_v=r.cache_v[:, :, :T])


def work(case):
    kind = case["kind"]
    if kind in ("linear", "layers"):
        shapes = [(case["N"], case["K"])] if kind == "linear" else _layer_linears(case)
        M, G, n = case["M"], case["G"], case.get("n_layers", 1)
        return {"bytes": n * sum(N * K // 2 + N * (K // G) * 2 + 2 * M * (N + K) for N, K in shapes),
                "flops": n * sum(2.0 * M * N * K for N, K in shapes)}
    if kind == "quantize":
        N, K, G = case["N"], case["K"], case["G"]
        return {"bytes": 2 * N * K + N * K // 2 + 2 * N * (K // G), "flops": 0}
    cfg, T, L = Qwen2Config.qwen25_7b(), case["T"], case["n_layers"]
    c = dict(hidden=cfg.hidden, q=cfg.n_heads * cfg.head_dim, kv=cfg.n_kv_heads * cfg.head_dim, inter=cfg.intermediate)
    per_layer = sum(N * K for N, K in _layer_linears(c))
    weights = L * per_layer * (0.5 + 2 / cfg.group)
    head, kv_row, qd = cfg.vocab * cfg.hidden, L * 2 * c["kv"] * 2, c["q"]
    # prompt: every weight and the vocabulary projection once, the embeddings read, the KV cache written; causal attention
    bytes_ = weights + 2 * head + T * (2 * cfg.hidden + kv_row)
    flops = 2.0 * T * L * per_layer + L * 2.0 * T * T * qd + 2.0 * head
    for i in range(case.get("n_new", 1) - 1):  # each further token: every weight, and the KV cache so far
        bytes_ += weights + 2 * head + (T + i + 1) * kv_row
        flops += 2.0 * L * per_layer + L * 4.0 * (T + i) * qd + 2.0 * head
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """About four times what was measured: a decode linear of group 128 (exact integer weights) against the product in 64
    bits rounded once, 1e-4; weights rounded to bf16 (prefill, finer groups) against exact ones, 2.4e-3; a whole model
    with such linears in 32 bits, logits 3.9e-3 and cache 1.4e-3.  The largest differences were one bf16 step."""
    kind = case["kind"]
    if kind == "quantize":
        return "exact"
    if kind in ("linear", "layers"):
        exact_weights = case["M"] <= 16 and case["G"] == 128
        return {"rel": 1e-3 if exact_weights else 8e-3, "max": 3e-2}
    return {"rel": 1.5e-2, "max": 8e-2, "differ": 0.0}


def _exact_linear(x, Wq, S, G):
    """x . ((q - 8) * s)^T in 64 bits, a block of rows at a time."""
    shifts = torch.arange(0, 32, 4, device="cuda", dtype=torch.int32)
    x = x.double()
    rows = []
    for lo in range(0, Wq.shape[0], 4096):
        q = ((Wq[lo:lo + 4096, :, None] >> shifts) & 15).flatten(1).double() - 8
        rows.append(x @ (q * S[lo:lo + 4096].double().repeat_interleave(G, dim=1)).T)
    return torch.cat(rows, dim=1)


def exact(case, seed):
    """What `run` returns, in 64 bits and without this package's code.  A quantized matrix is whole numbers; a model's
    logits and cache depend on every intermediate's rounding to bf16, so no 64-bit value is theirs."""
    kind, gen = case["kind"], _gen(seed)
    if kind == "linear":
        Wq, S = _weights(case["N"], case["K"], case["G"], gen)
        return _exact_linear(_activations(case["M"], case["K"], gen), Wq, S, case["G"])
    if kind == "layers":
        shapes = _layer_linears(case)
        xs = [_activations(case["M"], K, gen) for _, K in shapes]
        return [[_exact_linear(x, *_weights(N, K, case["G"], gen), case["G"]) for x, (N, K) in zip(xs, shapes)]
                for _ in range(case["n_layers"])]
    return None
