"""The framework's work at the sizes it is used at: single layers and blocks of the speculative
decoding step through the C ABI, and whole runner calls (one verify step, prompt prefill).

Widths are Gemma-4-31B's (hidden 5376, FFN 21504, vocabulary 262144, sliding layers 32 query / 16 KV
heads of 256, global layers 32 / 4 of 512) and its drafter's (hidden 1024, FFN 8192). Rows follow the
serving configurations: up to 24 request slots times a verify depth of 1 to 9 tokens for decoding,
up to 256 rows a linear call for BF16 prefill. Weights are N(0, 0.02) as in a fresh initialisation,
activations N(0, 1) as they leave a norm.
"""
import ctypes
import math
import random

import torch

import carat_b200
from carat_b200 import capi
from carat_b200.capi import check
from carat_b200.runner import Int4Bf16Linear, quantize_tensor_to_fp8

HIDDEN, FFN, VOCABULARY, WINDOW, EPSILON = 5376, 21504, 262144, 1024, 1e-6
DRAFT_HIDDEN, DRAFT_FFN = 1024, 8192
HEADS = 32
SLIDING, GLOBAL = (16, 256), (4, 512)          # KV heads, head dimension
LAYERS = ("sliding",) * 5 + ("global",)        # one period of the 31B layer pattern

# (input width, output width) of the linears a step runs.
TARGET_LINEARS = ((5376, 16384), (5376, 18432), (8192, 5376), (16384, 5376), (5376, 43008),
                  (21504, 5376))
DRAFT_LINEARS = ((10752, 1024), (1024, 8192), (1024, 16384), (8192, 1024), (16384, 1024),
                 (1024, 5376))


def listed():
    return [
        # One request alone verifies five rows: the output projection of a sliding layer. The
        # smallest call of the path; latency is what counts.
        {"name": "o_proj_one_request", "kind": "fp8_linear", "rows": 5, "k": 8192, "n": 5376},
        # 24 slots at nine proposal rows (k = 8): the largest row count one linear call takes.
        {"name": "down_proj_k8", "kind": "fp8_linear", "rows": 216, "k": 21504, "n": 5376},
        # The MLP of a verify step, 24 slots x 5 rows: pre-MLP norm + quantise, gate_up, GeGLU +
        # quantise, down. Three quarters of a layer's weights.
        {"name": "mlp_verify", "kind": "mlp", "rows": 120},
        # The weight-only INT4 form of the same gate_up projection.
        {"name": "int4_gate_up", "kind": "int4_linear", "rows": 120, "k": 5376, "n": 43008,
         "group": 128},
        # The target's LM head with the fused argmax, once a verify step.
        {"name": "lm_head_verify", "kind": "fp8_head", "rows": 120, "k": 5376, "n": VOCABULARY},
        # The drafter's BF16 LM head, four times a step.
        {"name": "draft_head", "kind": "bf16_head", "rows": 24, "k": 1024, "n": VOCABULARY},
        # A full 256-row BF16 linear call, the unit of prompt prefill.
        {"name": "prefill_gate_up", "kind": "bf16_linear", "rows": 256, "k": 5376, "n": 43008},
        # Verify attention of a sliding layer over mostly wrapped rings, ragged contexts.
        {"name": "sliding_attention", "kind": "sliding", "requests": 24, "depth": 5,
         "shortest": 128, "longest": 6144, "mix": 3},
        # Verify attention of a global layer at the same contexts.
        {"name": "global_attention", "kind": "global", "requests": 24, "depth": 5,
         "shortest": 128, "longest": 6144, "mix": 3},
        # A whole verify step of 24 requests through the runner.
        {"name": "verify_step", "kind": "verify", "requests": 24, "depth": 5, "shortest": 128,
         "longest": 6144, "mix": 3},
        # A lone prompt of ordinary, odd length becomes resident: time to first token.
        {"name": "prefill_prompt", "kind": "prefill", "requests": 1, "shortest": 777,
         "longest": 777, "chunk": 1024, "mix": 1},
        # Several ragged prompts together, some of them past the sliding window, in the
        # scheduler's quanta.
        {"name": "prefill_batch", "kind": "prefill", "requests": 6, "shortest": 200,
         "longest": 2600, "chunk": 512, "mix": 5},
    ]


def _log(rng, low, high):
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    kind = rng.choice(("fp8_linear", "fp8_linear", "mlp", "int4_linear", "fp8_head", "bf16_head",
                       "bf16_linear", "bf16_linear", "sliding", "sliding", "global", "global",
                       "verify", "prefill", "prefill"))
    if kind in ("fp8_linear", "bf16_linear", "int4_linear"):
        k, n = rng.choice(TARGET_LINEARS + (DRAFT_LINEARS if kind != "int4_linear" else ()))
        if rng.random() < 0.3:         # other models' widths, odd ones among them
            k, n = 128 * _log(rng, 4, 160), 8 * _log(rng, 32, 5000)
        case = {"kind": kind, "rows": _log(rng, 1, 128 if kind == "int4_linear" else 256),
                "k": k, "n": n}
        if kind == "int4_linear":
            case["group"] = 256 if k % 256 == 0 and rng.random() < 0.5 else 128
        return case
    if kind == "mlp":
        return {"kind": kind, "rows": _log(rng, 1, 128)}
    if kind == "fp8_head":
        return {"kind": kind, "rows": _log(rng, 1, 128), "k": 5376, "n": VOCABULARY}
    if kind == "bf16_head":
        return {"kind": kind, "rows": _log(rng, 1, 64), "k": 1024, "n": VOCABULARY}
    if kind == "prefill":
        longest = _log(rng, 16, 2600)
        return {"kind": kind, "requests": rng.randint(1, 6),
                "shortest": max(1, int(longest * rng.random())), "longest": longest,
                "chunk": rng.choice((256, 512, 1024, 4096)), "mix": rng.randrange(1 << 16)}
    longest = _log(rng, 16, 6144)
    return {"kind": kind, "requests": rng.randint(1, 24), "depth": rng.randint(1, 5),
            "shortest": max(1, int(longest * rng.random())), "longest": longest,
            "mix": rng.randrange(1 << 16)}


def _lengths(case):
    """The context or prompt length of every request, from the case's own numbers."""
    rng = random.Random(case["mix"])
    return [rng.randint(case["shortest"], case["longest"]) for _ in range(case["requests"])]


# ------------------------------------------------------------------------------ inputs
def _normal(generator, *shape, std=1.0):
    return torch.randn(*shape, device="cuda", dtype=torch.bfloat16, generator=generator).mul_(std)


def _stream():
    return torch.cuda.current_stream().cuda_stream


class _View:
    """Device memory of the runner as a tensor, without a copy; the tensor keeps the runner alive."""

    def __init__(self, runner, which, layer, shape):
        self.runner = runner
        address = runner.device_pointer(which, layer)[0]
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<i2",
                                         "data": (address, False), "version": 2}

    def tensor(self):
        return torch.as_tensor(self, device="cuda").view(torch.bfloat16)


def _buffer(runner, which, layer, shape):
    return _View(runner, which, layer, shape).tensor()


def _model(generator, slots, context):
    """One period of the 31B layer pattern with its tied LM head, and a runner over it."""
    layers = [carat_b200.Gemma4LayerConfig("sliding", HEADS, *SLIDING, 1e4, False)
              if kind == "sliding" else
              carat_b200.Gemma4LayerConfig("global", HEADS, *GLOBAL, 1e6, True)
              for kind in LAYERS]
    config = carat_b200.Gemma4Config(HIDDEN, FFN, VOCABULARY, WINDOW, EPSILON, layers)
    tensors = {"token_embedding": _normal(generator, VOCABULARY, HIDDEN, std=0.02)}

    def norm(width, mean=1.0):
        return (mean * (1 + 0.1 * torch.randn(width, device="cuda", generator=generator))).bfloat16()

    for index, layer in enumerate(layers):
        prefix = f"layer.{index}."
        for name in ("input_norm", "pre_mlp_norm"):
            tensors[prefix + name] = norm(HIDDEN)
        # As in a trained checkpoint, a block adds a fraction of the stream's size to it (unit
        # weights would make a last-bit flip in one layer grow in every layer that follows), and
        # the attention scores have a spread of a few units.
        for name in ("post_attention_norm", "post_mlp_norm"):
            tensors[prefix + name] = norm(HIDDEN, 0.25)
        tensors[prefix + "q_norm"] = norm(layer.head_dimension, 0.35)
        tensors[prefix + "k_norm"] = norm(layer.head_dimension, 0.35)
        tensors[prefix + "scalar"] = torch.ones(1, device="cuda", dtype=torch.bfloat16)
        for name, rows, columns in (("qkv", layer.packed_width(), HIDDEN),
                                    ("o", HIDDEN, layer.query_width()),
                                    ("gate_up", 2 * FFN, HIDDEN), ("down", HIDDEN, FFN)):
            tensors[prefix + name] = _normal(generator, rows, columns, std=0.02)
    tensors["final_norm"] = norm(HIDDEN)
    weights = carat_b200.DeviceWeightArena(tensors)
    fp8 = carat_b200.Fp8WeightArena.quantize(weights)
    runner = carat_b200.Gemma4BatchModelRunner(config, weights, slots, context, fp8)
    return {"config": config, "weights": weights, "fp8": fp8, "runner": runner}


def _caches(runner, slots, context):
    """[(K, V)] of every layer as views of the runner's arenas."""
    found = []
    for index, kind in enumerate(LAYERS):
        kv_heads, dim = SLIDING if kind == "sliding" else GLOBAL
        shape = (slots, kv_heads, min(context, WINDOW) if kind == "sliding" else context, dim)
        found.append((_buffer(runner, 0, index, shape), _buffer(runner, 1, index, shape)))
    return found


def _context_capacity(case):
    return (case["longest"] + case.get("depth", 0) + 128) // 128 * 128


def prepare(case, seed):
    library = capi.library()
    generator = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    state = {"case": case, "library": library}
    if kind in ("fp8_linear", "fp8_head"):
        rows, k, n = case["rows"], case["k"], case["n"]
        state["x"], state["x_scale"] = quantize_tensor_to_fp8(_normal(generator, rows, k))
        state["w"], state["w_scale"] = quantize_tensor_to_fp8(_normal(generator, n, k, std=0.02))
    elif kind in ("bf16_linear", "bf16_head"):
        rows, k, n = case["rows"], case["k"], case["n"]
        state["x"] = _normal(generator, rows, k)
        state["w"] = _normal(generator, n, k, std=0.02)
    if kind in ("fp8_linear", "bf16_linear"):
        state["out"] = torch.empty(rows, n, dtype=torch.bfloat16, device="cuda")
        needed = (library.carat_b200_fp8_linear_workspace_bytes if kind == "fp8_linear"
                  else library.carat_b200_bf16_linear_workspace_bytes)(rows, k, n)
        state["needed"] = needed
        state["workspace"] = torch.empty(max(needed, 16), dtype=torch.uint8, device="cuda")
    elif kind in ("fp8_head", "bf16_head"):
        state["out"] = torch.empty(rows, dtype=torch.int32, device="cuda")
        state["keys"] = torch.empty(rows, dtype=torch.int64, device="cuda")
    elif kind == "int4_linear":
        state["linear"] = Int4Bf16Linear(_normal(generator, case["n"], case["k"], std=0.02),
                                         case["k"], case["n"], case["group"])
        state["x"] = _normal(generator, case["rows"], case["k"])
        state["out"] = torch.empty(case["rows"], case["n"], dtype=torch.bfloat16, device="cuda")
    elif kind == "mlp":
        rows = case["rows"]
        state["hidden"] = _normal(generator, rows, HIDDEN, std=3.0)
        state["norm"] = _normal(generator, HIDDEN, std=0.1).add_(1.0)
        state["gate_up"], state["gate_up_scale"] = quantize_tensor_to_fp8(
            _normal(generator, 2 * FFN, HIDDEN, std=0.02))
        state["down"], state["down_scale"] = quantize_tensor_to_fp8(
            _normal(generator, HIDDEN, FFN, std=0.02))
        for name, width in (("normed", HIDDEN), ("activated", FFN)):
            state[name] = torch.empty(rows, width, dtype=torch.uint8, device="cuda")
            state[name + "_scale"] = torch.zeros(1, dtype=torch.float32, device="cuda")
            state[name + "_scratch"] = torch.zeros(1, dtype=torch.int32, device="cuda")
        state["packed"] = torch.empty(rows, 2 * FFN, dtype=torch.bfloat16, device="cuda")
        state["out"] = torch.empty(rows, HIDDEN, dtype=torch.bfloat16, device="cuda")
        needed = max(library.carat_b200_fp8_linear_workspace_bytes(rows, HIDDEN, 2 * FFN),
                     library.carat_b200_fp8_linear_workspace_bytes(rows, FFN, HIDDEN))
        state["needed"] = needed
        state["workspace"] = torch.empty(max(needed, 16), dtype=torch.uint8, device="cuda")
    elif kind in ("sliding", "global"):
        kv_heads, dim = SLIDING if kind == "sliding" else GLOBAL
        requests, depth = case["requests"], case["depth"]
        lengths = _lengths(case)
        longest = max(lengths)
        capacity = WINDOW if kind == "sliding" else _context_capacity(case)
        # Norm weights that give the scores of a trained layer a spread near one.
        state["queries"] = _normal(generator, requests, HEADS, depth, dim, std=0.3)
        for name in ("keys", "values"):
            state[name] = _normal(generator, requests, kv_heads, capacity, dim, std=0.3)
            state["new_" + name] = (_normal(generator, requests, kv_heads, depth, dim, std=0.3)
                                    if kind == "sliding" else None)
        participating = min(longest, capacity) if kind == "sliding" else longest + depth
        state["stride"] = 16 + (participating + 127) // 128 * 128
        state["positions"] = torch.tensor(lengths, dtype=torch.int32, device="cuda")
        state["out"] = torch.empty(requests * depth, HEADS * dim, dtype=torch.bfloat16,
                                   device="cuda")
        state["scores"] = torch.empty(requests * HEADS * depth * state["stride"],
                                      dtype=torch.bfloat16, device="cuda")
        state["capacity"], state["longest"], state["lengths"] = capacity, longest, lengths
    elif kind == "verify":
        requests, depth = case["requests"], case["depth"]
        lengths, context = _lengths(case), _context_capacity(case)
        state.update(_model(generator, requests, context))
        state["runner"].seed_slot_positions(lengths)
        state["caches"] = _caches(state["runner"], requests, context)
        for keys, values in state["caches"]:
            keys.copy_(_normal(generator, *keys.shape, std=0.35))
            values.copy_(_normal(generator, *values.shape))
        rng = random.Random(seed)
        # The drafts are random, and so is the token that the slot's last step predicted: every
        # request is rejected at its first row and the step leaves its slot as it found it.
        state["proposals"] = [[rng.randrange(3, VOCABULARY) for _ in range(depth)]
                              for _ in range(requests)]
        state["first"] = [row[0] - 1 for row in state["proposals"]]
        state["final_hidden"] = _buffer(state["runner"], 3, 0, (requests * depth, HIDDEN))
        state["lengths"] = lengths
    else:
        lengths, context = _lengths(case), _context_capacity(case)
        state.update(_model(generator, case["requests"], context))
        state["runner"].set_bf16_weights()
        state["caches"] = _caches(state["runner"], case["requests"], context)
        state["hand_off"] = _buffer(state["runner"], 2, 0, (case["requests"], HIDDEN))
        rng = random.Random(seed)
        state["prompts"] = [capi.int_array([rng.randrange(3, VOCABULARY) for _ in range(length)])
                            for length in lengths]
        state["lengths"] = lengths
    return state


# ------------------------------------------------------------------------------ one pass
def run(state):
    library, case = state["library"], state["case"]
    kind = case["kind"]
    if kind == "fp8_linear":
        check(library.carat_b200_fp8_linear(
            state["x"].data_ptr(), state["x_scale"].data_ptr(), state["w"].data_ptr(),
            state["w_scale"].data_ptr(), state["out"].data_ptr(), case["rows"], case["k"],
            case["n"], state["workspace"].data_ptr(), state["needed"], _stream()))
        return state["out"]
    if kind == "bf16_linear":
        check(library.carat_b200_bf16_linear(
            state["x"].data_ptr(), state["w"].data_ptr(), state["out"].data_ptr(), case["rows"],
            case["k"], case["n"], state["workspace"].data_ptr(), state["needed"], _stream()))
        return state["out"]
    if kind == "fp8_head":
        check(library.carat_b200_fp8_linear_argmax(
            state["x"].data_ptr(), state["x_scale"].data_ptr(), state["w"].data_ptr(),
            state["w_scale"].data_ptr(), state["out"].data_ptr(), state["keys"].data_ptr(),
            case["rows"], case["k"], case["n"], _stream()))
        return state["out"]
    if kind == "bf16_head":
        check(library.carat_b200_bf16_linear_argmax(
            state["x"].data_ptr(), state["w"].data_ptr(), state["out"].data_ptr(),
            state["keys"].data_ptr(), case["rows"], case["k"], case["n"], _stream()))
        return state["out"]
    if kind == "int4_linear":
        return state["linear"].run(state["x"], state["out"])
    if kind == "mlp":
        rows, stream = case["rows"], _stream()
        check(library.carat_b200_rms_norm_quantize(
            state["hidden"].data_ptr(), state["norm"].data_ptr(), None, state["normed"].data_ptr(),
            state["normed_scale"].data_ptr(), state["normed_scratch"].data_ptr(), rows, HIDDEN,
            EPSILON, stream))
        check(library.carat_b200_fp8_linear(
            state["normed"].data_ptr(), state["normed_scale"].data_ptr(),
            state["gate_up"].data_ptr(), state["gate_up_scale"].data_ptr(),
            state["packed"].data_ptr(), rows, HIDDEN, 2 * FFN, state["workspace"].data_ptr(),
            state["needed"], stream))
        check(library.carat_b200_gelu_gate_quantize(
            state["packed"].data_ptr(), state["activated"].data_ptr(),
            state["activated_scale"].data_ptr(), state["activated_scratch"].data_ptr(), rows, FFN,
            stream))
        check(library.carat_b200_fp8_linear(
            state["activated"].data_ptr(), state["activated_scale"].data_ptr(),
            state["down"].data_ptr(), state["down_scale"].data_ptr(), state["out"].data_ptr(),
            rows, FFN, HIDDEN, state["workspace"].data_ptr(), state["needed"], stream))
        return state["out"]
    if kind in ("sliding", "global"):
        kv_heads, dim = SLIDING if kind == "sliding" else GLOBAL
        new_keys, new_values = state["new_keys"], state["new_values"]
        check(library.carat_b200_verify_attention(
            state["queries"].data_ptr(), state["keys"].data_ptr(), state["values"].data_ptr(),
            None if new_keys is None else new_keys.data_ptr(),
            None if new_values is None else new_values.data_ptr(),
            state["positions"].data_ptr(), state["out"].data_ptr(), state["scores"].data_ptr(),
            state["stride"], case["requests"], case["depth"], HEADS, kv_heads, dim,
            state["capacity"], WINDOW if kind == "sliding" else 0, state["longest"], _stream()))
        return state["out"]
    runner = state["runner"]
    slots = list(range(case["requests"]))
    if kind == "verify":
        result = runner.verify_greedy_proposals(state["proposals"], state["first"], slots)
        return {"accepted": torch.tensor(result.accepted_tokens),
                "predictions": torch.tensor(
                    runner.last_predictions(case["requests"] * case["depth"])),
                "hidden": state["final_hidden"]}
    for slot in slots:
        runner.reset_slot(slot)
    tokens = [None] * len(slots)
    pending = slots
    while pending:
        first = runner.prefill_slots_chunks(pending, [state["prompts"][slot] for slot in pending],
                                            case["chunk"])
        for slot, token in zip(pending, first):
            tokens[slot] = token
        pending = [slot for slot, token in zip(pending, first) if token is None]
    return {"tokens": torch.tensor(tokens), "hidden": state["hand_off"],
            "caches": state["caches"]}


# ------------------------------------------------------------------------------ what it takes
def _layer_parameters(kind):
    kv_heads, dim = SLIDING if kind == "sliding" else GLOBAL
    packed = (HEADS + kv_heads * (2 if kind == "sliding" else 1)) * dim
    return packed * HIDDEN + HEADS * dim * HIDDEN + 3 * FFN * HIDDEN


def _attention_work(kind, lengths, depth):
    """(bytes of K and V, flops) of `depth` new rows of each request over its context."""
    kv_heads, dim = SLIDING if kind == "sliding" else GLOBAL
    rows = pairs = 0
    for length in lengths:
        seen = min(length, WINDOW - 1) if kind == "sliding" else length
        rows += seen + depth
        for t in range(depth):
            pairs += min(length + t + 1, WINDOW) if kind == "sliding" else length + t + 1
    return rows * kv_heads * dim * 4, pairs * HEADS * dim * 4


def work(case):
    kind = case["kind"]
    if kind in ("fp8_linear", "fp8_head", "bf16_linear", "bf16_head", "int4_linear"):
        rows, k, n = case["rows"], case["k"], case["n"]
        each = 1 if kind.startswith("fp8") else 2
        weight = k * n * each if kind != "int4_linear" else k * n // 2 + k // case["group"] * n * 2
        out = rows * 4 if kind.endswith("head") else rows * n * 2
        return {"bytes": weight + rows * k * each + out, "flops": 2 * rows * k * n}
    if kind == "mlp":
        rows = case["rows"]
        return {"bytes": 3 * HIDDEN * FFN + 4 * rows * HIDDEN, "flops": 6 * rows * HIDDEN * FFN}
    if kind in ("sliding", "global"):
        dim = (SLIDING if kind == "sliding" else GLOBAL)[1]
        moved, flops = _attention_work(kind, _lengths(case), case["depth"])
        return {"bytes": moved + 4 * case["requests"] * case["depth"] * HEADS * dim,
                "flops": flops}
    parameters = sum(_layer_parameters(kind_) for kind_ in LAYERS)
    lengths = _lengths(case)
    if kind == "verify":
        rows = case["requests"] * case["depth"]
        moved = flops = 0
        for layer in LAYERS:
            of = _attention_work(layer, lengths, case["depth"])
            moved, flops = moved + of[0], flops + of[1]
        head = HIDDEN * VOCABULARY
        return {"bytes": parameters + head + moved + 4 * rows * HIDDEN,
                "flops": flops + 2 * rows * (parameters + head)}
    rows = sum(lengths)
    moved = flops = 0
    for layer in LAYERS:
        kv_heads, dim = SLIDING if layer == "sliding" else GLOBAL
        moved += rows * kv_heads * dim * 4
        for length in lengths:
            seen = min(length, WINDOW) if layer == "sliding" else length
            flops += (seen * (seen + 1) // 2 + (length - seen) * seen) * HEADS * dim * 4
    head = HIDDEN * VOCABULARY
    return {"bytes": 2 * (parameters + head) + moved + 2 * rows * HIDDEN,
            "flops": flops + 2 * rows * parameters + 2 * len(lengths) * head}


def tolerance(case):
    kind = case["kind"]
    if kind in ("fp8_linear", "bf16_linear", "int4_linear"):
        # fp32 sums in another order, rounded once to bf16 (which alone is 1.7e-3 off 64 bits).
        return {"rel": 4e-3, "max": 2e-2}
    if kind in ("fp8_head", "bf16_head"):
        return {"rel": 0.0, "differ": 1e-2}
    if kind == "mlp":
        # Last-bit flips of bf16 values across e4m3 boundaries: 3.7e-2 off 64 bits.
        return {"rel": 3e-2, "max": 0.5}
    if kind in ("sliding", "global"):
        # Scores rounded to bf16 or not: 0.7e-2 to 1.1e-2 off 64 bits.
        return {"rel": 2.5e-2, "max": 0.3}
    # Six layers carry every flip on: up to 1e-2 off 64 bits in bf16 (prefill), 3.6e-2 with e4m3
    # activations (verify).
    return {"rel": 3e-2, "max": 0.9, "differ": 1e-2}


# ------------------------------------------------------------------------------ 64 bits
def _fp8(tensor):
    return tensor.view(torch.float8_e4m3fn).double()


def _product(x, weight, as_double=lambda part: part.double()):
    """x . weight^T in 64 bits, the weight widened a part at a time."""
    step = max(1, (1 << 27) // weight.shape[1])
    return torch.cat([x @ as_double(weight[at:at + step]).t()
                      for at in range(0, weight.shape[0], step)], 1)


def _best(logits):
    """argmax of the bf16 logits, ties to the lowest index."""
    logits = logits.bfloat16()
    index = torch.arange(logits.shape[1], device=logits.device)
    top = logits.max(1, keepdim=True).values
    return torch.where(logits == top, index, logits.shape[1]).min(1).values.int()


def _norm(x, weight=None):
    y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPSILON)
    return y if weight is None else y * weight.double()


def _quantised(x):
    """x as the tensor-wide e4m3 quantiser leaves it."""
    scale = x.abs().max() / 448
    return (x / scale).clamp(-448, 448).float().to(torch.float8_e4m3fn).double() * scale


def _geglu(packed):
    gate, up = packed.chunk(2, 1)
    return torch.nn.functional.gelu(gate, approximate="tanh") * up


def _attend(queries, keys, values, visible):
    """queries [heads, q, D] over keys and values [kv heads, k, D]; visible [q, k]."""
    heads, rows, dim = queries.shape
    grouped = queries.reshape(keys.shape[0], -1, dim)
    scores = (grouped @ keys.transpose(1, 2)).reshape(heads, rows, -1)
    scores = scores.masked_fill(~visible, -math.inf).softmax(-1)
    return (scores.reshape(keys.shape[0], -1, keys.shape[1]) @ values).reshape(heads, rows, dim)


def _visible(first, rows, count, window, offset=0):
    """Which of the positions offset .. offset + count - 1 the queries first .. see."""
    query = torch.arange(first, first + rows, device="cuda")[:, None]
    key = torch.arange(offset, offset + count, device="cuda")[None, :]
    seen = key <= query
    return seen & (key > query - window) if window else seen


def _rope(x, first, kind):
    """Rotate-half RoPE of [heads, rows, D]; the tables are bf16 by the model's definition."""
    dim = x.shape[-1]
    index = torch.arange(dim // 2, dtype=torch.float32, device="cuda")
    theta = 1e4 if kind == "sliding" else 1e6
    frequency = torch.pow(torch.tensor(theta, device="cuda"), -2.0 * index / dim)
    if kind == "global":
        frequency = torch.where(index < dim // 8, frequency, 0.0)
    angle = torch.arange(first, first + x.shape[1], dtype=torch.float32,
                         device="cuda")[:, None] * frequency
    cosine, sine = angle.cos().bfloat16().double(), angle.sin().bfloat16().double()
    low, high = x.chunk(2, -1)
    return torch.cat([low * cosine - high * sine, high * cosine + low * sine], -1)


def _forward(state, tokens, firsts, counts, quantised):
    """Final-normed hidden rows of `counts[r]` tokens of each request r from position firsts[r] on,
    and their K and V rows: [(layer, request)] of [kv heads, rows, D]. Earlier rows are read from
    state["caches"] as they stand."""
    weights, fp8 = state["weights"], state["fp8"]

    def linear(x, name):
        if not quantised:
            return _product(x, weights.at(name))
        return _product(_quantised(x), fp8.at(name), _fp8) * fp8.scale(name).double()

    embedding = weights.at("token_embedding")
    hidden = embedding[tokens].double() * float(torch.tensor(math.sqrt(HIDDEN)).bfloat16())
    rows = {}
    for index, kind in enumerate(LAYERS):
        prefix = f"layer.{index}."
        kv_heads, dim = SLIDING if kind == "sliding" else GLOBAL
        window = WINDOW if kind == "sliding" else 0
        packed = linear(_norm(hidden, weights.at(prefix + "input_norm")), prefix + "qkv")
        packed = packed.reshape(len(tokens), -1, dim).transpose(0, 1)
        attended, at = [], 0
        for request, (first, count) in enumerate(zip(firsts, counts)):
            part = packed[:, at:at + count]
            at += count
            query = _rope(_norm(part[:HEADS], weights.at(prefix + "q_norm")), first, kind)
            raw = part[HEADS:HEADS + kv_heads]
            key = _rope(_norm(raw, weights.at(prefix + "k_norm")), first, kind)
            value = _norm(part[HEADS + kv_heads:] if kind == "sliding" else raw)
            rows[index, request] = key, value
            start = max(0, first - WINDOW + 1) if window else 0
            place = torch.arange(start, first, device="cuda")
            keys, values = state["caches"][index]
            if window:
                place = place % keys.shape[2]
            key = torch.cat([keys[request][:, place].double(), key], 1)
            value = torch.cat([values[request][:, place].double(), value], 1)
            out = _attend(query, key, value, _visible(first, count, key.shape[1], window, start))
            attended.append(out.transpose(0, 1).reshape(count, -1))
        residual = hidden
        projected = linear(torch.cat(attended), prefix + "o")
        residual = _norm(projected, weights.at(prefix + "post_attention_norm")) + residual
        packed = linear(_norm(residual, weights.at(prefix + "pre_mlp_norm")), prefix + "gate_up")
        down = linear(_geglu(packed), prefix + "down")
        hidden = ((_norm(down, weights.at(prefix + "post_mlp_norm")) + residual)
                  * weights.at(prefix + "scalar").double())
    return _norm(hidden, weights.at("final_norm")), rows


def exact(case, seed):
    state = prepare(case, seed)
    kind = case["kind"]
    if kind in ("fp8_linear", "fp8_head"):
        out = (_product(_fp8(state["x"]), state["w"], _fp8)
               * (state["x_scale"].double() * state["w_scale"].double()))
        return out if kind == "fp8_linear" else _best(out)
    if kind in ("bf16_linear", "bf16_head"):
        out = _product(state["x"].double(), state["w"])
        return out if kind == "bf16_linear" else _best(out)
    if kind == "int4_linear":
        linear, group = state["linear"], case["group"]
        packed = linear.packed
        codes = torch.stack([packed & 15, packed >> 4], 2).reshape(case["n"], case["k"]).int()
        codes = torch.where(codes > 7, codes - 16, codes).float()
        scales = linear.scales.t().float().repeat_interleave(group, 1)
        return _product(state["x"].double(), (codes * scales).bfloat16())
    if kind == "mlp":
        x = _quantised(_norm(state["hidden"].double(), state["norm"]))
        packed = _product(x, state["gate_up"], _fp8) * state["gate_up_scale"].double()
        return (_product(_quantised(_geglu(packed)), state["down"], _fp8)
                * state["down_scale"].double())
    if kind in ("sliding", "global"):
        depth, out = case["depth"], []
        window = WINDOW if kind == "sliding" else 0
        for request, length in enumerate(state["lengths"]):
            start = max(0, length - WINDOW + 1) if window else 0
            rows = torch.arange(start, length + (0 if window else depth),
                                device="cuda") % state["capacity"]
            both = []
            for name in ("keys", "values"):
                part = state[name][request][:, rows].double()
                if window:
                    part = torch.cat([part, state["new_" + name][request].double()], 1)
                both.append(part)
            seen = _visible(length, depth, both[0].shape[1], window, start)
            out.append(_attend(state["queries"][request].double(), *both, seen)
                       .transpose(0, 1).reshape(depth, -1))
        return torch.cat(out)
    lengths = state["lengths"]
    if kind == "verify":
        depth = case["depth"]
        tokens = torch.tensor([t for row in state["proposals"] for t in row], device="cuda")
        hidden, _ = _forward(state, tokens, lengths, [depth] * len(lengths), True)
        head = state["fp8"]
        logits = (_product(_quantised(hidden), head.at("token_embedding"), _fp8)
                  * head.scale("token_embedding").double())
        return {"accepted": torch.zeros(len(lengths), dtype=torch.int64),
                "predictions": _best(logits), "hidden": hidden}
    tokens = torch.tensor([t for prompt in state["prompts"] for t in prompt], device="cuda")
    hidden, rows = _forward(state, tokens, [0] * len(lengths), lengths, False)
    ends = [sum(lengths[:r + 1]) - 1 for r in range(len(lengths))]
    caches = []
    for index, (keys, values) in enumerate(state["caches"]):
        pair = []
        for which, cache in ((0, keys), (1, values)):
            filled = torch.zeros(cache.shape, dtype=torch.float64, device="cuda")
            for request, length in enumerate(lengths):
                place = torch.arange(max(0, length - cache.shape[2]), length, device="cuda")
                filled[request][:, place % cache.shape[2]] = rows[index, request][which][:, place]
            pair.append(filled)
        caches.append(tuple(pair))
    last = hidden[ends]
    tokens = _best(_product(last, state["weights"].at("token_embedding")))
    return {"tokens": tokens, "hidden": last, "caches": caches}
