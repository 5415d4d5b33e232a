"""The calls a user of this framework makes, as cases that can be prepared, run, counted and checked.

Kinds of case
  block      the seven packed linears of decoder blocks (q, k, v, o, gate, up, down; siblings grouped as
             ``mk.optimize`` groups them) called as modules inside one ``mk.capture``: decode and batched decode
  prefill    the same modules called eagerly on a prompt of more than 128 rows
  head       a tied output head: token embeddings decoded from its packed rows, then its logits
  transform  the randomised Hadamard transform of a batch of activations
  encode     rounding a weight matrix to a packed format, as ``mk.quantize`` does for every linear
  step       one captured decode step of the tensor-parallel decoder (on one GPU): logits and caches
"""

import math

import torch
from torch import nn

import mlkit_b200 as mk
from mlkit_b200 import tp

DEVICE = "cuda"
DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
CODEBOOK3 = [-1.0, -0.5, -0.25, 0.0, 0.25, 0.5, 1.0]
NF4 = [-1.0, -0.6961928, -0.52507305, -0.39491749, -0.28444138, -0.18477343, -0.09105004, 0.0,
       0.07958030, 0.16093020, 0.24611230, 0.33791524, 0.44070983, 0.56261700, 0.72295684, 1.0]
# codec -> (bits, group, asymmetric); the first is what most checkpoints use
CODECS = {"int4_g128": (4, 128, False), "int4_g64": (4, 64, False), "int4_g32": (4, 32, False),
          "int4_g128_asym": (4, 128, True), "int4_g64_asym": (4, 64, True), "int2_g128": (2, 128, False),
          "int3_g128": (3, 128, False), "int5_g128": (5, 128, False), "int6_g128": (6, 128, False),
          "int8_g128": (8, 128, False), "nf4_g64": (4, 64, False), "codebook3_g64": (3, 64, False)}
ROTATED = ("o_proj", "down_proj")


def listed():
    return [
        # a small model (hidden 896, MLP 4864, biases on q, k, v) decoding one token: launches and latency
        dict(name="decode_small_m1", kind="block", hidden=896, kv=128, mlp=4864, blocks=4, rows=1, codec="int4_g128",
             dtype="fp16", bias=True, rotated=False),
        # the common case: an 8B-shaped model decoding one sequence
        dict(name="decode_int4_m1", kind="block", hidden=4096, kv=1024, mlp=14336, blocks=2, rows=1, codec="int4_g128",
             dtype="fp16", bias=False, rotated=False),
        # most checkpoints are bf16: the same model with its own activations type, four sequences
        dict(name="decode_int4_bf16_m4", kind="block", hidden=4096, kv=1024, mlp=14336, blocks=2, rows=4,
             codec="int4_g128", dtype="bf16", bias=False, rotated=False),
        # a table codec with the largest batch the matvec takes at once
        dict(name="decode_nf4_m8", kind="block", hidden=4096, kv=1024, mlp=14336, blocks=2, rows=8, codec="nf4_g64",
             dtype="fp16", bias=False, rotated=False),
        # scales with offsets, the layout asymmetric post-training methods write
        dict(name="decode_asym_m2", kind="block", hidden=4096, kv=1024, mlp=14336, blocks=2, rows=2,
             codec="int4_g128_asym", dtype="fp16", bias=False, rotated=False),
        # online rotation ahead of o and down (4096 and 14336 = 28 x 512 wide), outliers in the activations
        dict(name="decode_rotated_m1", kind="block", hidden=4096, kv=1024, mlp=14336, blocks=2, rows=1,
             codec="int4_g128", dtype="fp16", bias=False, rotated=True),
        # batched decode: more rows than the matvec takes
        dict(name="batch_int4_m64", kind="block", hidden=4096, kv=1024, mlp=14336, blocks=2, rows=64, codec="int4_g128",
             dtype="fp16", bias=False, rotated=False),
        # a prompt of odd length in bf16
        dict(name="prefill_bf16_1537", kind="prefill", hidden=4096, kv=1024, mlp=14336, blocks=1, rows=1537,
             codec="int4_g128", dtype="bf16", bias=False, rotated=False),
        # a tied eight-bit head of a 128k vocabulary: embeddings of the tokens, then logits
        dict(name="head_int8_bf16_m3", kind="head", vocab=128256, hidden=4096, rows=3, codec="int8_g128", dtype="bf16"),
        # the rotation of a prompt's activations in front of the down projection
        dict(name="rht_4099x14336", kind="transform", rows=4099, width=14336, dtype="fp16", inverse=False),
        # converting one bf16 gate projection
        dict(name="encode_int4", kind="encode", outputs=14336, width=4096, codec="int4_g128", scale="absmax",
             dtype="bf16"),
        # a whole decode step, eight sequences at a context of about 500
        dict(name="decode_step_b8", kind="step", hidden=4096, kv_heads=8, mlp=14336, layers=4, vocab=32000, rows=8,
             context=500, codec="int4_g128"),
    ]


def _log_between(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _log_multiple(rng, low, high, unit):
    return unit * _log_between(rng, low // unit, high // unit)


def draw(rng):
    kind = rng.choice(["block", "block", "block", "block", "prefill", "head", "transform", "encode", "step"])
    dtype = rng.choice(["fp16", "bf16"])
    if kind in ("block", "prefill"):
        codec = rng.choice(sorted(CODECS))
        if rng.random() < 0.4:
            codec = "int4_g128"
        hidden = _log_multiple(rng, 640, 5120, 128)
        case = dict(kind=kind, hidden=hidden, kv=max(64, hidden // rng.choice([1, 2, 4, 8]) // 64 * 64),
                    mlp=128 * _log_between(rng, 2 * hidden // 128, min(4 * hidden, 14336) // 128),
                    blocks=rng.choice([1, 2]) if kind == "block" else 1, codec=codec, dtype=dtype,
                    bias=rng.random() < 0.25, rotated=rng.random() < 0.15)
        if kind == "prefill":
            case["rows"] = _log_between(rng, 129, 1400)
        else:
            case["rows"] = rng.randint(1, 8) if rng.random() < 0.75 else _log_between(rng, 9, 128)
        return case
    if kind == "head":
        return dict(kind=kind, vocab=_log_between(rng, 16000, 120000), hidden=_log_multiple(rng, 640, 4096, 128),
                    rows=rng.randint(1, 8), codec=rng.choice(["int8_g128", "int6_g128", "int4_g128", "nf4_g64"]), dtype=dtype)
    if kind == "transform":
        width = rng.choice([1024, 2048, 4096, 8192, 16384]) if rng.random() < 0.5 else 512 * rng.choice([12, 20, 24, 28, 36])
        return dict(kind=kind, rows=min(_log_between(rng, 64, 16384), 60_000_000 // width), width=width, dtype=dtype,
                    inverse=rng.random() < 0.25)
    if kind == "encode":
        return dict(kind=kind, outputs=_log_between(rng, 500, 12000), width=_log_multiple(rng, 640, 5120, 128),
                    codec=rng.choice(sorted(CODECS)), scale="mse" if rng.random() < 0.2 else "absmax", dtype=dtype)
    heads = rng.choice([8, 16, 24, 32])
    return dict(kind=kind, hidden=128 * heads, kv_heads=heads // rng.choice([1, 2, 4, 8]),
                mlp=_log_multiple(rng, 2048, 14336, 128), layers=rng.randint(1, 4), vocab=_log_between(rng, 8000, 32000),
                rows=rng.randint(1, 8), context=_log_between(rng, 30, 900), codec="int4_g128")


# ------------------------------------------------------------------------------------------- inputs


def _generator(seed, stream=0):
    return torch.Generator(device=DEVICE).manual_seed((seed * 1000003 + stream) % (1 << 62))


def _format(codec, scale="absmax"):
    bits, group, asym = CODECS[codec]
    if codec.startswith("nf4"):
        return mk.nf4(group=group, scale=scale)
    if codec.startswith("codebook3"):
        return mk.scaled(mk.grid.values(CODEBOOK3, bits=3), group=group, scale=scale)
    return mk.int(bits, group=group, asym=asym, scale=scale)


def _shapes(case):
    hidden, kv, mlp = case["hidden"], case["kv"], case["mlp"]
    return {"q_proj": (hidden, hidden), "k_proj": (kv, hidden), "v_proj": (kv, hidden), "o_proj": (hidden, hidden),
            "gate_proj": (mlp, hidden), "up_proj": (mlp, hidden), "down_proj": (hidden, mlp)}


def _weight(outputs, width, dtype, generator):
    return (torch.randn(outputs, width, generator=generator, device=DEVICE) * 0.02).to(dtype)


def _biased(case, name):
    return case["bias"] and name in ("q_proj", "k_proj", "v_proj")


def _block_parts(case, seed):
    """(block, name, weight, bias or None) of every linear, in the order they are made."""
    generator = _generator(seed)
    dtype = DTYPES[case["dtype"]]
    for block in range(case["blocks"]):
        for name, (outputs, width) in _shapes(case).items():
            weight = _weight(outputs, width, dtype, generator)
            bias = (torch.randn(outputs, generator=generator, device=DEVICE) * 0.1).to(dtype) if _biased(case, name) else None
            yield block, name, weight, bias


def _block_inputs(case, seed):
    """Activations [blocks, rows, width] into q/k/v/gate/up, o, and down; with outlier channels where a rotation follows."""
    generator = _generator(seed, 1)
    inputs = []
    for width, outliers in ((case["hidden"], False), (case["hidden"], case["rotated"]), (case["mlp"], case["rotated"])):
        x = torch.randn(case["blocks"], case["rows"], width, generator=generator, device=DEVICE)
        if outliers:
            x[..., torch.randperm(width, generator=generator, device=DEVICE)[: max(1, width // 100)]] *= 50
        inputs.append(x.to(DTYPES[case["dtype"]]))
    return tuple(inputs)


def _rotation_seed(block, name):
    return 1000 + 10 * block + ROTATED.index(name)


class Blocks(nn.Module):
    """Decoder blocks' linears, each on the input it reads in a model."""

    def __init__(self, blocks):
        super().__init__()
        self.blocks = nn.ModuleList(blocks)

    def forward(self, hidden, attention, mlp):
        outputs = []
        for block, h, a, m in zip(self.blocks, hidden.unbind(0), attention.unbind(0), mlp.unbind(0)):
            outputs += [block.q_proj(h), block.k_proj(h), block.v_proj(h), block.o_proj(a), block.gate_proj(h),
                        block.up_proj(h), block.down_proj(m)]
        return tuple(outputs)


def _packed_linear(weight, bias, codec, parent=None, name=None, rotation=None):
    linear = nn.Linear(weight.shape[1], weight.shape[0], bias=bias is not None, device=DEVICE, dtype=weight.dtype)
    with torch.no_grad():
        linear.weight.copy_(weight)
        if bias is not None:
            linear.bias.copy_(bias)
    if rotation is not None:
        setattr(parent, name, linear)
        mk.install_transform(parent, {"kind": "rotation", "name": name, "seed": rotation})
    return mk.PackedLinear(linear, _format(codec)(weight.float(), mk.Ctx(device=DEVICE)))


def _prepare_block(case, seed):
    blocks = [nn.Module() for _ in range(case["blocks"])]
    for block, name, weight, bias in _block_parts(case, seed):
        rotation = _rotation_seed(block, name) if case["rotated"] and name in ROTATED else None
        setattr(blocks[block], name, _packed_linear(weight, bias, case["codec"], blocks[block], name, rotation))
    for block in blocks:
        mk.fuse_siblings(block)
    module, inputs = Blocks(blocks).eval(), _block_inputs(case, seed)
    if case["kind"] == "prefill":
        return {"call": module, "inputs": inputs}
    call = mk.capture(module)
    call(*inputs)      # a serving program captures its step before it serves
    return {"call": call, "inputs": inputs}


def _prepare_head(case, seed):
    dtype, generator = DTYPES[case["dtype"]], _generator(seed)
    weight = _weight(case["vocab"], case["hidden"], dtype, generator)
    head = _packed_linear(weight, None, case["codec"])
    embedding = mk.PackedEmbedding(head, nn.Embedding(1, case["hidden"], device="meta"))
    tokens = torch.randint(0, case["vocab"], (case["rows"],), generator=generator, device=DEVICE)
    x = torch.randn(case["rows"], case["hidden"], generator=generator, device=DEVICE).to(dtype)
    call = mk.capture(_TiedHead(head, embedding))
    call(tokens, x)
    return {"call": call, "inputs": (tokens, x)}


class _TiedHead(nn.Module):
    def __init__(self, head, embedding):
        super().__init__()
        self.head, self.embedding = head, embedding

    def forward(self, tokens, hidden):
        return self.embedding(tokens), self.head(hidden)


def _transform_inputs(case, seed):
    generator = _generator(seed)
    x = torch.randn(case["rows"], case["width"], generator=generator, device=DEVICE)
    x[:, torch.randperm(case["width"], generator=generator, device=DEVICE)[: case["width"] // 100]] *= 50
    signs = (torch.randint(0, 2, (case["width"],), generator=generator, device=DEVICE) * 2 - 1).to(torch.int8)
    return x.to(DTYPES[case["dtype"]]), signs


def _step_config(case):
    heads = case["hidden"] // 128
    return tp.DecoderConfig(layers=case["layers"], hidden=case["hidden"], q_heads=heads, kv_heads=case["kv_heads"],
                            head_dim=128, intermediate=case["mlp"], vocab=case["vocab"])


def _step_parts(case, seed):
    """The tensors of a step in a fixed order: per layer its seven weights, norms and caches, then the rest."""
    generator = _generator(seed)
    heads, kv = case["hidden"] // 128, case["kv_heads"] * 128
    half = lambda *shape, scale=1.0: (torch.randn(*shape, generator=generator, device=DEVICE) * scale).half()
    shapes = {"q": (heads * 128, case["hidden"]), "k": (kv, case["hidden"]), "v": (kv, case["hidden"]),
              "o": (case["hidden"], heads * 128), "gate": (case["mlp"], case["hidden"]),
              "up": (case["mlp"], case["hidden"]), "down": (case["hidden"], case["mlp"])}
    for _ in range(case["layers"]):
        weights = {name: half(*shape, scale=0.02) for name, shape in shapes.items()}
        norms = tuple((1 + 0.1 * half(case["hidden"]).float()).half() for _ in range(2))
        caches = tuple(half(case["rows"], case["kv_heads"], case["context"], 128) for _ in range(2))
        yield weights, norms, caches
    embedding = half(case["vocab"], case["hidden"])
    final_norm = (1 + 0.1 * half(case["hidden"]).float()).half()
    head = half(case["vocab"], case["hidden"], scale=0.02)
    tokens = torch.randint(0, case["vocab"], (case["rows"],), generator=generator, device=DEVICE)
    positions = case["context"] - torch.randint(0, max(1, case["context"] // 8), (case["rows"],), generator=generator, device=DEVICE)
    yield embedding, final_norm, head, tokens, positions.to(torch.int32)


def _prepare_step(case, seed):
    config, device = _step_config(case), torch.device(DEVICE, torch.cuda.current_device())
    model = tp.TensorParallelDecoder(config, device=device, max_batch=case["rows"], capacity=case["context"] + 1)
    contexts, fmt = [], _format(case["codec"])
    for part in _step_parts(case, seed):
        if len(part) == 3:
            weights, norms, caches = part
            block = {name: fmt(weight.float(), mk.Ctx(name, device=DEVICE)) for name, weight in weights.items()}
            model.add_block(tp.shard_block(block, config, 0, 1, device), *norms)
            contexts.append(caches)
        else:
            embedding, final_norm, head, tokens, positions = part
            model.set_head(embedding, final_norm, _format("int8_g128")(head.float(), mk.Ctx("head", device=DEVICE)))
    step = model.capture(case["rows"])
    for (keys, values), k_cache, v_cache in zip(contexts, model.k_cache, model.v_cache):
        k_cache[:, :, :case["context"]].copy_(keys)
        v_cache[:, :, :case["context"]].copy_(values)
        k_cache[:, :, case["context"]:].zero_()
        v_cache[:, :, case["context"]:].zero_()
    return {"step": step, "model": model, "tokens": tokens, "positions": positions}


def prepare(case, seed):
    kind = case["kind"]
    with torch.inference_mode():
        if kind in ("block", "prefill"):
            state = _prepare_block(case, seed)
        elif kind == "head":
            state = _prepare_head(case, seed)
        elif kind == "transform":
            x, signs = _transform_inputs(case, seed)
            state = {"x": x, "signs": signs, "inverse": case["inverse"]}
        elif kind == "encode":
            weight = _weight(case["outputs"], case["width"], DTYPES[case["dtype"]], _generator(seed))
            state = {"weight": weight, "format": _format(case["codec"], case["scale"])}
        else:
            state = _prepare_step(case, seed)
    return {"kind": kind, **state}


def run(state):
    kind = state["kind"]
    with torch.inference_mode():
        if kind in ("block", "prefill", "head"):
            return state["call"](*state["inputs"])
        if kind == "transform":
            return mk.rht(state["x"], signs=state["signs"], inverse=state["inverse"])
        if kind == "encode":
            quantized = state["format"](state["weight"], mk.Ctx(device=DEVICE))
            packed = quantized.packed_stream(quantized.metadata["code_bits"])
            return [quantized.codes, packed, quantized.params["scales"], quantized.params["zero"]]
        state["step"].tokens.copy_(state["tokens"])
        state["step"].positions.copy_(state["positions"])
        logits = state["step"].replay()
        return [logits, state["model"].k_cache, state["model"].v_cache]


# ------------------------------------------------------------------------------------------- counting


def _weight_bytes(outputs, width, codec):
    bits, group, asym = CODECS[codec]
    return outputs * width * bits / 8 + outputs * math.ceil(width / group) * 2 * (2 if asym else 1)


def work(case):
    kind = case["kind"]
    moved = flops = 0.0
    if kind in ("block", "prefill"):
        for name, (outputs, width) in _shapes(case).items():
            moved += _weight_bytes(outputs, width, case["codec"]) + case["rows"] * outputs * 2
            moved += outputs * 2 if _biased(case, name) else 0
            flops += 2.0 * case["rows"] * outputs * width
        moved += case["rows"] * (2 * case["hidden"] + case["mlp"]) * 2
        return {"bytes": moved * case["blocks"], "flops": flops * case["blocks"]}
    if kind == "head":
        moved = _weight_bytes(case["vocab"], case["hidden"], case["codec"]) + case["rows"] * case["vocab"] * 2
        moved += case["rows"] * (_weight_bytes(1, case["hidden"], case["codec"]) + 4 * case["hidden"] + 8)
        return {"bytes": moved, "flops": 2.0 * case["rows"] * case["vocab"] * case["hidden"]}
    if kind == "transform":
        factor, power, _ = _factor(case["width"])
        size = case["rows"] * case["width"]
        return {"bytes": 4.0 * size + case["width"], "flops": size * (math.log2(power) + (2 * factor if factor > 1 else 0))}
    if kind == "encode":
        size = case["outputs"] * case["width"]   # scales come back as fp32, codes as bytes beside the packed stream
        bits, group, asym = CODECS[case["codec"]]
        groups = case["outputs"] * math.ceil(case["width"] / group)
        return {"bytes": 2.0 * size + size + size * bits / 8 + groups * 4 * (2 if asym else 1), "flops": 4.0 * size}
    hidden, kv, rows = case["hidden"], case["kv_heads"] * 128, case["rows"]
    shapes = ((hidden + 2 * kv, hidden), (hidden, hidden), (2 * case["mlp"], hidden), (hidden, case["mlp"]))
    per_layer = sum(_weight_bytes(n, k, case["codec"]) for n, k in shapes) + rows * (case["context"] + 1) * kv * 2 * 2 + 4 * hidden
    moved = case["layers"] * per_layer + _weight_bytes(case["vocab"], hidden, "int8_g128") + rows * (case["vocab"] * 2 + hidden * 2 + 12)
    flops = case["layers"] * sum(2.0 * rows * n * k for n, k in shapes) + 2.0 * rows * case["vocab"] * hidden
    return {"bytes": moved, "flops": flops + case["layers"] * rows * 4.0 * (case["context"] + 1) * hidden}


def tolerance(case):
    kind = case["kind"]
    if kind == "encode":
        return "exact"      # codes, packed bytes and the stored scales follow one arithmetic, operation for operation
    if kind == "step":
        return {"rel": 4e-3}    # fp16 rounding between operators, through up to four layers
    if kind == "transform":
        return {"rel": 8e-4, "max": 8e-3} if case["dtype"] == "fp16" else {"rel": 6e-3, "max": 4e-2}
    # one rounding of the output; weights of the dense and table routes are rounded to 16 bits too
    return {"rel": 1.5e-3, "max": 1.5e-2} if case["dtype"] == "fp16" else {"rel": 8e-3, "max": 6e-2}


# ------------------------------------------------------------------------------------------- 64 bits


def _plain_quantized(weight, codec):
    """The reconstruction a format stores for ``weight``: round to nearest in fp32, values times scales in 64 bits."""
    bits, group, asym = CODECS[codec]
    w = weight.float()
    rows, width = w.shape
    blocks = w.reshape(rows, width // group, group)
    if codec.startswith("nf4") or codec.startswith("codebook3"):
        levels = torch.tensor(NF4 if codec.startswith("nf4") else CODEBOOK3, device=w.device)
    else:
        levels = torch.arange(-(2 ** (bits - 1)), 2 ** (bits - 1), device=w.device).float()
    low, high = float(levels[0]), float(levels[-1])
    span = high - low if asym else float(levels.abs().max())
    reciprocal = float(torch.tensor(1.0) / torch.tensor(span))
    zero = None
    if asym:
        scale = (blocks.amax(-1) - blocks.amin(-1)).clamp_min(1e-12) * reciprocal
        zero = blocks.amin(-1) - low * scale
    else:
        scale = torch.maximum(blocks.amax(-1), -blocks.amin(-1)).clamp_min(1e-12) * reciprocal
    scale = scale.clamp(2**-24, 65504).half().float()
    if zero is not None:
        zero = zero.abs().clamp_min(1e-12).clamp(2**-24, 65504).half().float() * zero.sign()
        blocks = blocks - zero[..., None]
    normalized = blocks / scale[..., None]
    if codec.startswith("int"):
        chosen = normalized.round().clamp(low, high)
    else:
        above = torch.searchsorted(levels, normalized.contiguous()).clamp_max(levels.numel() - 1)
        below = (above - 1).clamp_min(0)
        nearer = (normalized - levels[below]).abs() <= (normalized - levels[above]).abs()
        chosen = levels[torch.where(nearer, below, above)]
    dense = chosen.double() * scale[..., None].double()
    if zero is not None:
        dense = dense + zero[..., None].double()
    return dense.reshape(rows, width)


def _is_prime(value):
    return value >= 2 and all(value % d for d in range(2, math.isqrt(value) + 1))


def _paley(order):
    """Orthonormal Hadamard matrix of the first or second Paley construction over a prime field, else None."""
    def character(q):
        squares = {(i * i) % q for i in range(1, q)}
        return torch.tensor([[0.0 if i == j else 1.0 if (i - j) % q in squares else -1.0 for j in range(q)] for i in range(q)],
                            dtype=torch.float64)
    q = order - 1
    if _is_prime(q) and q % 4 == 3:
        matrix = torch.ones(order, order, dtype=torch.float64)
        matrix[1:, 0] = -1
        matrix[1:, 1:] = character(q) + torch.eye(q, dtype=torch.float64)
        return matrix / math.sqrt(order)
    q = order // 2 - 1
    if order % 2 == 0 and _is_prime(q) and q % 4 == 1:
        core = torch.ones(q + 1, q + 1, dtype=torch.float64)
        core[0, 0] = 0
        core[1:, 1:] = character(q)
        eye = torch.eye(q + 1, dtype=torch.float64)
        return torch.cat((torch.cat((core + eye, core - eye), 1), torch.cat((core - eye, -core - eye), 1)), 0) / math.sqrt(order)
    return None


def _factor(width):
    odd = width
    while odd % 2 == 0:
        odd //= 2
    power = width // odd
    if odd == 1:
        return 1, width, None
    for multiple in (1, 2, 4, 8, 16):
        if power % multiple == 0 and _paley(odd * multiple) is not None:
            return odd * multiple, power // multiple, _paley(odd * multiple)
    index = torch.arange(odd, dtype=torch.float64)
    basis = torch.cos(math.pi / odd * (index[None, :] + 0.5) * index[:, None])
    basis[0] *= 1 / math.sqrt(odd)
    basis[1:] *= math.sqrt(2 / odd)
    return odd, power, basis


def _plain_transform(x, signs, inverse=False):
    factor, power, basis = _factor(x.shape[-1])
    y = x.double() if inverse else x.double() * signs
    shape, span = y.shape, 1
    while span < power:
        pairs = y.reshape(-1, 2, span)
        y = torch.stack((pairs[:, 0] + pairs[:, 1], pairs[:, 0] - pairs[:, 1]), 1)
        span *= 2
    y = (y / math.sqrt(power)).reshape(-1, factor, power)
    if basis is not None:
        basis = basis.to(y.device)
        y = torch.matmul(basis.t() if inverse else basis, y)
    y = y.reshape(shape)
    return y * signs if inverse else y


def _exact_block(case, seed):
    hidden, attention, mlp = _block_inputs(case, seed)
    outputs = []
    for block, name, weight, bias in _block_parts(case, seed):
        x = (attention if name == "o_proj" else mlp if name == "down_proj" else hidden)[block]
        if case["rotated"] and name in ROTATED:
            generator = torch.Generator(device=DEVICE).manual_seed(_rotation_seed(block, name))
            signs = torch.randint(2, (x.shape[-1],), generator=generator, device=DEVICE) * 2 - 1
            x = _plain_transform(x, signs)
        y = x.double() @ _plain_quantized(weight, case["codec"]).t()
        outputs.append(y if bias is None else y + bias.double())
    return tuple(outputs)


def _exact_head(case, seed):
    generator = _generator(seed)
    dtype = DTYPES[case["dtype"]]
    weight = _plain_quantized(_weight(case["vocab"], case["hidden"], dtype, generator), case["codec"])
    tokens = torch.randint(0, case["vocab"], (case["rows"],), generator=generator, device=DEVICE)
    x = torch.randn(case["rows"], case["hidden"], generator=generator, device=DEVICE).to(dtype)
    return weight[tokens], x.double() @ weight.t()


def _exact_step(case, seed):
    parts = list(_step_parts(case, seed))
    embedding, final_norm, head, tokens, positions = parts.pop()
    rows, dim, kv_heads = case["rows"], 128, case["kv_heads"]
    config = _step_config(case)

    def norm(x, weight):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + config.eps) * weight.double()

    def rope(x):
        frequency = config.rope_theta ** (-torch.arange(0, dim, 2, device=DEVICE).double() / dim)
        angle = (positions.double()[:, None] * frequency)[:, None, :]
        a, b = x[..., : dim // 2], x[..., dim // 2:]
        return torch.cat((a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()), -1)

    x = embedding.double()[tokens]
    k_caches, v_caches = [], []
    for weights, (attention_norm, mlp_norm), (keys, values) in parts:
        dense = lambda name: _plain_quantized(weights[name], case["codec"]).t()
        h = norm(x, attention_norm)
        q, k = rope((h @ dense("q")).view(rows, -1, dim)), rope((h @ dense("k")).view(rows, kv_heads, dim))
        v = (h @ dense("v")).view(rows, kv_heads, dim)
        pad = torch.zeros(rows, kv_heads, 1, dim, dtype=torch.float64, device=DEVICE)
        keys, values = torch.cat((keys.double(), pad), 2), torch.cat((values.double(), pad), 2)
        index = torch.arange(rows, device=DEVICE)
        keys[index, :, positions.long()], values[index, :, positions.long()] = k, v
        k_caches.append(keys)
        v_caches.append(values)
        repeat = q.shape[1] // kv_heads
        scores = torch.einsum("mhd,mhpd->mhp", q, keys.repeat_interleave(repeat, 1)) / math.sqrt(dim)
        later = torch.arange(keys.shape[2], device=DEVICE)[None, None, :] > positions[:, None, None]
        mixed = torch.einsum("mhp,mhpd->mhd", torch.softmax(scores.masked_fill(later, -math.inf), -1),
                             values.repeat_interleave(repeat, 1))
        x = x + mixed.reshape(rows, -1) @ dense("o")
        h = norm(x, mlp_norm)
        x = x + (nn.functional.silu(h @ dense("gate")) * (h @ dense("up"))) @ dense("down")
    return [norm(x, final_norm) @ _plain_quantized(head, "int8_g128").t(), k_caches, v_caches]


def exact(case, seed):
    """What ``run`` returns for these inputs, from plain torch in 64 bits."""
    kind = case["kind"]
    with torch.inference_mode():
        if kind in ("block", "prefill"):
            return _exact_block(case, seed)
        if kind == "head":
            return _exact_head(case, seed)
        if kind == "transform":
            x, signs = _transform_inputs(case, seed)
            return _plain_transform(x, signs, case["inverse"])
        if kind == "encode":
            return None     # whole numbers, and scales that are roundings of a maximum
        return _exact_step(case, seed)
