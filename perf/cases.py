"""What the framework is timed on: the calls that a program built on it makes, over the sizes it makes them at.

Kinds of work and the entry points they go through:
  linear   `QuantLinear.forward`: a packed CherryQ layer applied to m activation rows (decode, small serving batches,
           prefill), weights packed beforehand
  decode   `CherryDecoder.generate(1)`: one token for every sequence of a LLaMA-architecture model over a filled KV cache
           (the captured step), logits read back by the sampler; the fed token is given, as in a perplexity evaluation
  prefill  `CherryDecoder.prefill`: prompts through the same model into its KV cache
  pack     `QuantLinear.pack`: fp16 weights to codes, scales and cherry columns (converting a trained model)
  unpack   `QuantLinear.unpack`: back to the dense fp16 matrix
  speed    `quant_cuda.vecquant3matmul_cherryq(fp16=False)`: the operator's 32-bit form
  train    `CherryLinear` forward and backward (quantisation-aware training, straight-through gradient)

Layer and model sizes are those of LLaMA-2 7B / 13B / 70B (the configurations of `decoder.py`), with fewer decoder layers
where a whole model would only repeat the same layer.  Weights are N(0, 0.02) with cherry columns N(0, 0.2), activations
N(0, 1).
"""
import math
from types import SimpleNamespace

import torch

import cherryq_b200
from cherryq_b200 import CherryLinear, QuantLinear
from cherryq_b200 import decoder as D

ARCH = {
    "7b": dict(hidden=4096, n_heads=32, n_kv_heads=32, ffn=11008),
    "13b": dict(hidden=5120, n_heads=40, n_kv_heads=40, ffn=13824),
    "70b": dict(hidden=8192, n_heads=64, n_kv_heads=8, ffn=28672),
}
FRACTION = 1 / 256          # share of cherry columns
VOCAB = 32000
# no drawn case costs more than the largest listed ones
MAX_FLOPS = 1.0e13
MAX_BYTES = 6.0e9


def listed():
    return [
        # one token through one attention projection of a 7B layer, called from Python: launch latency and host work
        {"name": "linear_4096x4096_m1", "kind": "linear", "k": 4096, "n": 4096, "m": 1, "bits": 4, "group": 128, "bias": False},
        # sixteen sequences decoded together, the 7B gate projection
        {"name": "linear_4096x11008_m16", "kind": "linear", "k": 4096, "n": 11008, "m": 16, "bits": 4, "group": 128, "bias": False},
        # a serving step of mixed requests: an odd number of rows, the narrow group size, a layer with a bias
        {"name": "linear_5120x13824_m45", "kind": "linear", "k": 5120, "n": 13824, "m": 45, "bits": 3, "group": 64, "bias": True},
        # a 2048-token prompt through the 7B gate projection
        {"name": "linear_4096x11008_m2048", "kind": "linear", "k": 4096, "n": 11008, "m": 2048, "bits": 4, "group": 128, "bias": False},
        # the widest layer at a long prompt: 70B gate projection, 3-bit
        {"name": "linear_8192x28672_m4096", "kind": "linear", "k": 8192, "n": 28672, "m": 4096, "bits": 3, "group": 128, "bias": False},
        # interactive decoding: the whole 7B model, 4-bit, one sequence, short context
        {"name": "decode_7b_b1", "kind": "decode", "arch": "7b", "layers": 32, "bits": 4, "group": 128, "batch": 1, "context": 256, "max_seq": 512},
        # throughput decoding: 70B layers (grouped-query attention), 3-bit, sixteen sequences at a long context
        {"name": "decode_70b_b16", "kind": "decode", "arch": "70b", "layers": 8, "bits": 3, "group": 128, "batch": 16, "context": 4000, "max_seq": 4096},
        # a 2048-token prompt through 13B layers, 3-bit
        {"name": "prefill_13b_2048", "kind": "prefill", "arch": "13b", "layers": 8, "bits": 3, "group": 128, "batch": 1, "tokens": 2048, "max_seq": 2304},
        # converting a trained model: one 7B gate projection
        {"name": "pack_4096x11008", "kind": "pack", "k": 4096, "n": 11008, "bits": 4, "group": 128},
        # back to a dense matrix: one 7B down projection, 3-bit
        {"name": "unpack_11008x4096", "kind": "unpack", "k": 11008, "n": 4096, "bits": 3, "group": 128},
        # the operator's own speed check: 32-bit activations, sixteen rows
        {"name": "speed_4096x13824_m16", "kind": "speed", "k": 4096, "n": 13824, "m": 16, "group": 128},
        # a training step of one 7B gate projection on 2048 tokens
        {"name": "train_4096x11008_m2048", "kind": "train", "k": 4096, "n": 11008, "m": 2048, "bits": 4, "group": 128},
    ]


# ---------------------------------------------------------------------------------- drawn cases
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo, hi):
    """A layer width: usually a multiple of 128 as in the configurations, sometimes only of 8."""
    w = _log_int(rng, lo, hi)
    step = 128 if rng.random() < 0.6 else 8
    return max(lo, w // step * step)


def draw(rng):
    while True:
        case = _draw(rng)
        w = work(case)
        if w["flops"] <= MAX_FLOPS and w["bytes"] <= MAX_BYTES:
            return case


def _draw(rng):
    kind = rng.choices(["linear", "decode", "prefill", "pack", "unpack", "speed", "train"], [9, 3, 2, 2, 2, 1, 2])[0]
    bits = rng.choice([3, 4])
    group = rng.choice([128, 128, 128, 256, -1] + ([64] if bits == 3 else []))
    if kind in ("decode", "prefill"):
        arch = rng.choice(sorted(ARCH))
        bits = bits if arch == "7b" else 3                # as configured
        case = {"kind": kind, "arch": arch, "layers": rng.randint(3, 8), "bits": bits, "group": 128}
        if kind == "decode":
            context = _log_int(rng, 64, 4000)
            case.update(batch=_log_int(rng, 1, 32), context=context, max_seq=context + _log_int(rng, 64, 512))
        else:
            batch, tokens = rng.choice([1, 1, 1, 2, 4]), _log_int(rng, 32, 2048)
            case.update(batch=batch, tokens=tokens, max_seq=tokens + _log_int(rng, 64, 512))
        return case
    k, n = _width(rng, 1024, 16384), _width(rng, 1024, 28672)
    if group == -1 and k % 128:          # one group per row: the kernels want whole blocks of 128 columns
        group = 128
    case = {"kind": kind, "k": k, "n": n, "group": group}
    if kind == "linear":
        case.update(m=_log_int(rng, 1, 4096), bits=bits, bias=rng.random() < 0.25)
    elif kind == "speed":
        case.update(m=_log_int(rng, 1, 64), group=rng.choice([64, 128]))
    elif kind == "train":
        case.update(m=_log_int(rng, 128, 4096), bits=bits, group=128)
    else:
        case.update(bits=bits)
    return case


# ---------------------------------------------------------------------------------- preparation
def _cherries(k):
    return math.ceil(k * FRACTION) // 8 * 8


def _weights(k, n, g, dtype=torch.float16):
    """(n, k) weights with their cherry columns, and the columns' indices in no particular order."""
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.02).to(dtype)
    idx = torch.randperm(k, device="cuda", generator=g)[:_cherries(k)].to(torch.int32)
    w[:, idx.long()] = (torch.randn(n, idx.numel(), device="cuda", generator=g) * 0.2).to(dtype)
    return w, idx


def _layer(case, g):
    """A packed layer, and the weights it was packed from."""
    k, n = case["k"], case["n"]
    w, idx = _weights(k, n, g)
    bias = (torch.randn(n, device="cuda", generator=g) * 0.1).half() if case.get("bias") else None
    src = SimpleNamespace(weight=w, bias=bias, cherry_indices=idx, group_size=case["group"])
    layer = QuantLinear(case.get("bits", 3), case["group"], None, FRACTION, k, n, bias=bias is not None).to("cuda")
    layer.pack(src)
    return layer, src


def _config(case):
    return D.DecoderConfig(n_layers=case["layers"], vocab=VOCAB, bits=case["bits"], group=case["group"], cherry_fraction=FRACTION,
                           max_seq=case["max_seq"], **ARCH[case["arch"]])


def prepare(case, seed):
    kind = case["kind"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    if kind in ("decode", "prefill"):
        dec = D.CherryDecoder(_config(case), device="cuda", seed=seed, release_reference_buffers=True, batch=case["batch"])
        if kind == "prefill":
            return {"kind": kind, "dec": dec, "tokens": torch.randint(0, VOCAB, (case["batch"], case["tokens"]), device="cuda", generator=g)}
        # a filled cache: keys and values of this architecture with weights as above have a deviation of about 1.5
        for cache in (dec.k_cache, dec.v_cache):
            for layer in cache[:, :, :case["context"]]:
                layer.copy_(torch.randn(layer.shape, device="cuda", generator=g, dtype=torch.float16) * 1.5)
        dec.capture()
        return {"kind": kind, "dec": dec, "context": case["context"], "tokens": torch.randint(0, VOCAB, (case["batch"],), device="cuda", generator=g)}
    if kind == "train":
        k, n, m = case["k"], case["n"], case["m"]
        with torch.device("cuda"):
            layer = CherryLinear(k, n, w_bits=case["bits"], group_size=case["group"], cherryq=True, cherry_fraction=FRACTION)
        layer = layer.to(torch.bfloat16).train()
        w, idx = _weights(k, n, g, torch.bfloat16)
        layer.weight.data.copy_(w)
        layer.register_cherry_indices(idx)
        x = torch.randn(m, k, device="cuda", generator=g, dtype=torch.bfloat16).requires_grad_()
        gy = torch.randn(m, n, device="cuda", generator=g, dtype=torch.bfloat16)
        return {"kind": kind, "layer": layer, "x": x, "gy": gy}
    layer, src = _layer(case, g)
    state = {"kind": kind, "layer": layer}
    if kind == "linear":
        state["x"] = torch.randn(case["m"], case["k"], device="cuda", generator=g).half()
    elif kind == "pack":
        state["src"] = src
    elif kind == "speed":
        state.update(x=torch.randn(case["m"], case["k"], device="cuda", generator=g), qweight=layer.qweight, cherry=layer.cherry_weight.float(),
                     indices=layer.cherry_indices.int(), scales=layer.scales.float(), group=case["group"], op=cherryq_b200.load_quant_cuda())
    return state


# ---------------------------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["layer"](state["x"])
    if kind == "decode":
        dec, p = state["dec"], state["context"]
        dec.tok.copy_(state["tokens"])
        dec.pos.fill_(p)
        dec.pos_host = p
        dec.generate(1)
        return {"logits": dec.graph_logits, "k_cache": dec.k_cache, "v_cache": dec.v_cache}
    if kind == "prefill":
        dec = state["dec"]
        return {"logits": dec.prefill(state["tokens"]), "k_cache": dec.k_cache, "v_cache": dec.v_cache}
    if kind == "pack":
        layer = state["layer"]
        layer.pack(state["src"])
        return [layer.qweight, layer.scales, layer.cherry_weight, layer.cherry_indices]
    if kind == "unpack":
        return state["layer"].unpack()
    if kind == "speed":
        x, q = state["x"], state["qweight"]
        y = torch.zeros(x.shape[0], q.shape[1], device=x.device)
        state["op"].vecquant3matmul_cherryq(x, q, state["cherry"], state["indices"], state["scales"], y, state["group"], False)
        return y
    layer, x = state["layer"], state["x"]
    x.grad = layer.weight.grad = None
    y = layer(x)
    y.backward(state["gy"])
    return {"y": y, "x_grad": x.grad, "weight_grad": layer.weight.grad}


# ---------------------------------------------------------------------------------- what a pass cannot do without
def _packed_bytes(k, n, bits, group, scale_bytes=2):
    c = _cherries(k)
    group = k if group == -1 else group
    return (k - c) // 8 * bits * n + math.ceil((k - c) / group) * n * scale_bytes + c * n * scale_bytes + 2 * c


def work(case):
    kind = case["kind"]
    if kind in ("decode", "prefill"):
        cfg = _config(case)
        shapes = [(cfg.hidden, cfg.hidden)] * 2 + [(cfg.hidden, cfg.n_kv_heads * cfg.head_dim)] * 2 + [(cfg.hidden, cfg.ffn)] * 2 + [(cfg.ffn, cfg.hidden)]
        weights = case["layers"] * sum(_packed_bytes(k, n, cfg.bits, cfg.group) for k, n in shapes)
        params = case["layers"] * sum(k * n for k, n in shapes)
        row = 2 * cfg.n_kv_heads * cfg.head_dim * 2 * case["layers"]               # K and V of one position, all layers
        head = VOCAB * cfg.hidden
        b = case["batch"]
        if kind == "decode":
            pos = case["context"] + 1
            return {"bytes": weights + 2 * head + b * pos * row + b * VOCAB * 2,
                    "flops": 2 * b * (params + head) + 4 * b * pos * cfg.hidden * case["layers"]}
        t = case["tokens"]
        return {"bytes": weights + 2 * head + b * t * (row + 2 * cfg.hidden) + b * VOCAB * 2,
                "flops": 2 * b * t * params + 2 * b * head + 2 * b * t * (t + 1) * cfg.hidden * case["layers"]}
    k, n = case["k"], case["n"]
    if kind == "linear":
        m = case["m"]
        return {"bytes": _packed_bytes(k, n, case["bits"], case["group"]) + 2 * m * (k + n), "flops": 2 * m * k * n}
    if kind in ("pack", "unpack"):
        return {"bytes": 2 * n * k + _packed_bytes(k, n, case["bits"], case["group"]), "flops": 0}
    if kind == "speed":
        m = case["m"]
        return {"bytes": _packed_bytes(k, n, 3, case["group"], 4) + 4 * m * (k + n), "flops": 2 * m * k * n}
    m = case["m"]
    return {"bytes": 2 * (2 * n * k + 2 * m * k + 2 * m * n), "flops": 6 * m * k * n}


def tolerance(case):
    """About four times the error seen of each path: against the same product in 64 bits, for whole models against the same
    model with every projection as a dense fp16 product (`dense=True`)."""
    kind = case["kind"]
    if kind in ("pack", "unpack"):
        return "exact"
    if kind == "linear":                                   # seen: 2.1e-4 .. 2.9e-4, largest 9.8e-4 (fp16 outputs)
        return {"rel": 1.2e-3, "max": 4e-3}
    if kind in ("decode", "prefill"):                      # seen: 2.6e-3 at 3 layers, 3.2e-3 at 8, 5.9e-3 at 32; largest 2.6e-2
        return {"rel": max(1.1e-2, 4.2e-3 * math.sqrt(case["layers"])), "max": 0.1}
    if kind == "speed":                                    # seen: 1.5e-7 .. 1.9e-7, largest 8.7e-7 (fp32 sums)
        return {"rel": 1e-6, "max": 5e-6}
    return {"rel": 7e-3, "max": 1.6e-2}                    # train, seen: 1.7e-3, largest 3.9e-3 (bf16 outputs)
