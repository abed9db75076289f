"""The work a host program has this library do, as cases that can be timed: single decode tokens, small
batches of sequences, prompt chunks, the decode loop over a model's layers, the model's other INT4
matrices (LM head, projections), the host-buffer entry, and the quantizer that makes the weights.

Sizes are the repository's own: the 1024 x 3072 layer of its first configuration, the Qwen3-4B layer
(2560 x 9728), the 27B layer (5120 x 17408), that layer's tensor-parallel slices (an intermediate size of
8704, 4352 or 2176 is what one of 2, 4 or 8 ranks runs), the 27B LM head (248320 x 5120) and its
projections; `draw` adds ragged token counts and any other whole number of 128-wide groups.
"""
import math

import torch

from haskell_infer_demo_b200 import ops

GROUP = 128
SMALL, QWEN3_4B, DENSE_27B = (1024, 3072), (2560, 9728), (5120, 17408)
LAYERS = (SMALL, QWEN3_4B, DENSE_27B, (5120, 8704), (5120, 4352), (5120, 2176), (2560, 4864), (4096, 14336))
MATRICES = ((248320, 5120), (34816, 5120), (12288, 5120), (5120, 17408), (4096, 5120), (19456, 2560), (151936, 2560))
LARGEST = 1.45e9      # bytes, or floating-point operations / 50: no drawn case costs more


def _ffn(name, tokens, shape, norm):
    return {"name": name, "kind": "ffn", "tokens": tokens, "hidden": shape[0], "inter": shape[1], "norm": norm}


def listed():
    return [
        # the smallest call: one token through a small layer; launch and start-up are most of it
        _ffn("decode_small", 1, SMALL, False),
        # two sequences of a 4B model, norm included: the layer as an engine calls it
        _ffn("decode_4b_pair", 2, QWEN3_4B, True),
        # single-stream decode of the 27B layer: the call the library exists for
        _ffn("decode_27b", 1, DENSE_27B, False),
        # the same for a caller whose activations live in pinned host memory, synchronous
        {"name": "decode_27b_host", "kind": "host", "tokens": 1, "hidden": 5120, "inter": 17408},
        # batched decode: eight sequences, and a ragged number of them
        _ffn("batch_8_27b", 8, DENSE_27B, False),
        _ffn("batch_27_27b", 27, DENSE_27B, False),
        # a prompt chunk of the default maximum, with the norm
        _ffn("chunk_128_27b", 128, DENSE_27B, True),
        # a longer, ragged prompt on the 4B layer
        _ffn("chunk_500_4b", 500, QWEN3_4B, True),
        # one decode step over the FFN sublayers of a 36-layer 4B model
        {"name": "stack_4b", "kind": "stack", "tokens": 1, "hidden": 2560, "inter": 9728, "layers": 36},
        # the LM head for five sequences
        {"name": "lm_head_5", "kind": "gemm", "rows": 5, "n": 248320, "k": 5120},
        # an attention projection over a ragged prompt chunk
        {"name": "proj_100", "kind": "gemm", "rows": 100, "n": 12288, "k": 5120},
        # weights to INT4: one gate (or up) matrix of the 27B layer
        {"name": "quantize_27b", "kind": "quantize", "n": 17408, "k": 5120},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def _draw(rng):
    kind = rng.choice(("ffn", "ffn", "ffn", "ffn", "gemm", "gemm", "stack", "host", "quantize"))
    if kind == "gemm":
        n, k = rng.choice(MATRICES) if rng.random() < 0.6 else (8 * _log_int(rng, 32, 8192), GROUP * _log_int(rng, 4, 136))
        return {"kind": kind, "rows": _log_int(rng, 1, 512), "n": n, "k": k}
    if kind == "quantize":
        return {"kind": kind, "n": 8 * _log_int(rng, 16, 4352), "k": GROUP * _log_int(rng, 4, 136)}
    hidden, inter = rng.choice(LAYERS) if rng.random() < 0.6 else (GROUP * _log_int(rng, 4, 64), GROUP * _log_int(rng, 8, 192))
    case = {"kind": kind, "tokens": 0, "hidden": hidden, "inter": inter}
    if kind == "ffn":
        case.update(tokens=_log_int(rng, 1, 512), norm=rng.random() < 0.5)
    elif kind == "host":
        case.update(tokens=_log_int(rng, 1, 8))
    else:
        case.update(tokens=_log_int(rng, 1, 64), layers=_log_int(rng, 2, 36))
    return case


def draw(rng):
    while True:
        case = _draw(rng)
        if _cost(case) <= LARGEST:
            return case


def _weights(gen, n, k):
    """A trained-looking matrix, N(0, 0.02), in the library's format (made a slab of rows at a time)."""
    slab = max(8, (1 << 28) // k // 8 * 8)
    parts = []
    for r in range(0, n, slab):
        w = torch.empty((min(slab, n - r), k), dtype=torch.float32, device="cuda").normal_(0.0, 0.02, generator=gen)
        parts.append(ops.quantize_int4(w))
    if len(parts) == 1:
        return parts[0]
    return torch.cat([p for p, _ in parts]), torch.cat([s for _, s in parts])


def _layer(gen, hidden, inter, norm, tokens):
    gate_up, gate_up_scales = _weights(gen, 2 * inter, hidden)
    down, down_scales = _weights(gen, hidden, inter)
    w_norm = torch.randn(hidden, generator=gen, device="cuda").mul_(0.1).to(torch.bfloat16) if norm else None
    return ops.DenseMlp(gate_up, gate_up_scales, down, down_scales, post_norm_w=w_norm, max_chunk=max(128, tokens))


def _activations(gen, rows, cols):
    return torch.randn((rows, cols), generator=gen, device="cuda").to(torch.bfloat16)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "quantize":
        w = torch.empty((case["n"], case["k"]), dtype=torch.float32, device="cuda").normal_(0.0, 0.02, generator=gen)
        return {"kind": kind, "w": w}
    if kind == "gemm":
        packed, scales = _weights(gen, case["n"], case["k"])
        return {"kind": kind, "a": _activations(gen, case["rows"], case["k"]), "packed": packed, "scales": scales}
    hidden, inter, tokens = case["hidden"], case["inter"], case["tokens"]
    if kind == "stack":
        mlps = [_layer(gen, hidden, inter, True, tokens) for _ in range(case["layers"])]
        embedded = _activations(gen, tokens, hidden)
        return {"kind": kind, "mlps": mlps, "embedded": embedded, "h": torch.empty_like(embedded),
                "ws": mlps[0].workspace(tokens), "out": torch.empty_like(embedded)}
    norm = bool(case.get("norm"))
    mlp = _layer(gen, hidden, inter, norm, tokens)
    x = _activations(gen, tokens, hidden)
    state = {"kind": kind, "mlp": mlp, "norm": norm, "ws": mlp.workspace(tokens)}
    if kind == "host":
        x_host, y_host = x.cpu().pin_memory(), torch.empty((tokens, hidden), dtype=torch.bfloat16).pin_memory()
        staging = torch.empty(2 * tokens * hidden, dtype=torch.bfloat16, device="cuda")
        state["call"] = ops.bind_forward_mlp_host(mlp, x_host, y_host, staging, state["ws"])
    else:
        state.update(x=x, out=torch.empty_like(x))
    return state


def run(state):
    kind = state["kind"]
    if kind == "ffn":
        forward = state["mlp"].forward_mlp if state["norm"] else state["mlp"].forward_mlp_prepared
        return forward(state["x"], state["ws"], state["out"])
    if kind == "host":
        return state["call"]()
    if kind == "stack":     # the step's embedded tokens become the residual stream, which the layers update in place
        state["h"].copy_(state["embedded"])
        return ops.decode_stack(state["mlps"], state["h"], ws=state["ws"], layer_out=state["out"]), state["out"]
    if kind == "gemm":
        return ops.gemm_int4_bf16(state["a"], state["packed"], state["scales"])
    return ops.quantize_int4(state["w"])


def _matrix_bytes(n, k):
    return n * k // 2 + n * (k // GROUP) * 2


def work(case):
    kind = case["kind"]
    if kind == "quantize":      # every weight read once, its code and its group's scale written once
        n, k = case["n"], case["k"]
        return {"bytes": 4 * n * k + _matrix_bytes(n, k), "flops": 3 * n * k}
    if kind == "gemm":
        m, n, k = case["rows"], case["n"], case["k"]
        return {"bytes": _matrix_bytes(n, k) + 2 * m * (n + k), "flops": 2 * m * n * k}
    m, h, i = case["tokens"], case["hidden"], case["inter"]
    layers = case.get("layers", 1)
    weights = _matrix_bytes(2 * i, h) + _matrix_bytes(h, i)
    normed = kind == "stack" or case.get("norm")
    return {"bytes": layers * (weights + (2 * h if normed else 0)) + 2 * 2 * m * h, "flops": layers * 6 * m * h * i}


def tolerance(case):
    kind = case["kind"]
    if kind == "quantize":
        return "exact"
    if kind == "gemm":
        return {"rel": 4e-3}
    if kind == "stack":
        return {"rel": 8e-2}
    return {"rel": 1e-2}


def _plain_quantize(w):
    """The format in plain torch: a 128-group's scale is its largest magnitude over 7 in BF16, codes -7..7."""
    groups = w.view(w.shape[0], -1, GROUP)
    top = groups.abs().amax(dim=2)
    scales = torch.where(top == 0, torch.ones_like(top), top / torch.full_like(top, 7)).to(torch.bfloat16)
    codes = (groups / scales.float()[:, :, None]).round_().clamp_(-7, 7).to(torch.int8)
    return codes, scales


def _plain_matrix(gen, n, k):
    """The matrix that `_weights` draws, slab by slab, as FP64 (rows, k) blocks of code * scale."""
    slab = max(8, (1 << 28) // k // 8 * 8)
    for r in range(0, n, slab):
        w = torch.empty((min(slab, n - r), k), dtype=torch.float32, device="cuda").normal_(0.0, 0.02, generator=gen)
        codes, scales = _plain_quantize(w)
        yield (codes.double() * scales.double()[:, :, None]).view(w.shape)


def _plain_ffn(x, gate_up, down, w_norm):
    if w_norm is not None:
        x = x * torch.rsqrt(x.square().mean(dim=1, keepdim=True) + 1e-6) * (1 + w_norm)
    g, u = (x @ gate_up.T).chunk(2, dim=1)
    return (torch.nn.functional.silu(g) * u) @ down.T


def exact(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "quantize":
        w = torch.empty((case["n"], case["k"]), dtype=torch.float32, device="cuda").normal_(0.0, 0.02, generator=gen)
        codes, scales = _plain_quantize(w)
        pairs = codes.view(case["n"], -1, 2).to(torch.uint8) & 15
        return pairs[:, :, 0] | pairs[:, :, 1] << 4, scales
    if kind == "gemm":      # the weights are drawn before the activations
        state = torch.Generator(device="cuda").manual_seed(seed)
        for _ in _plain_matrix(gen, case["n"], case["k"]):
            pass
        a = _activations(gen, case["rows"], case["k"]).double()
        return torch.cat([a @ w.T for w in _plain_matrix(state, case["n"], case["k"])], dim=1)
    hidden, inter, tokens = case["hidden"], case["inter"], case["tokens"]
    normed = kind == "stack" or bool(case.get("norm"))
    again = torch.Generator(device="cuda").manual_seed(seed)

    def layer(g):
        gate_up = torch.cat(list(_plain_matrix(g, 2 * inter, hidden)))
        down = torch.cat(list(_plain_matrix(g, hidden, inter)))
        w_norm = torch.randn(hidden, generator=g, device="cuda").mul_(0.1).to(torch.bfloat16).double() if normed else None
        return gate_up, down, w_norm

    for _ in range(case.get("layers", 1)):
        layer(gen)
    x = _activations(gen, tokens, hidden).double()
    if kind != "stack":
        y = _plain_ffn(x, *layer(again))
        return y.cpu() if kind == "host" else y
    for _ in range(case["layers"]):
        y = _plain_ffn(x, *layer(again))
        x = x + y
    return x, y
