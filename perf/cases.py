"""Performance cases of the library: the calls that programs built on it make, over the sizes they make them at.

Every case goes through the public entry points.  Dense and packed triangle attention carry most of the weight because
they carry most of the time of a pair block; layer norm, the gated form, the triangle multiplicative update and token
attention with a pair bias are the operators around it.  Values follow the distributions of the benchmark
configurations: query, key and value N(0, 1) / 2, bias and upstream gradient N(0, 1).
"""

from __future__ import annotations

import math

import torch

import oops_b200 as oops

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


def _triangle(name, dtype, n, *, batch=1, heads=4, dim=32, train=True, valid=0, mask="none", node="starting", projected=False):
    """`valid` tokens of `n` are real when mask is "tokens"; `projected`: the bias is the permuted view a linear map gives."""
    return {"name": name, "op": "triangle", "dtype": dtype, "n": n, "batch": batch, "heads": heads, "dim": dim, "train": train,
            "valid": valid or n, "mask": mask, "node": node, "projected": projected}


def listed():
    return [
        # f32 training step of a small complex: the precision used to validate a model, launches and latency count
        _triangle("f32 n64 train", "f32", 64, mask="ones"),
        # the smallest 16-bit calls: short chains at inference
        _triangle("bf16 n100 infer", "bf16", 100, train=False),
        # the usual training crop, two samples per GPU, some of the tokens padding
        _triangle("bf16 n256 b2 train", "bf16", 256, batch=2, valid=241, mask="tokens"),
        # padded inference
        _triangle("bf16 n384 infer padded", "bf16", 384, train=False, valid=350, mask="tokens"),
        # odd length, ending node (views with the pair axes exchanged), the bias as its projection leaves it
        _triangle("f16 n499 infer ending", "f16", 499, train=False, node="ending", projected=True),
        # the training shape of the benchmark
        _triangle("bf16 n768 train", "bf16", 768, mask="ones"),
        # the large training shape of the benchmark
        _triangle("bf16 n2048 train", "bf16", 2048, mask="ones"),
        # ending node on a packed ragged batch, the pair mask built from the token masks of the batch
        {"name": "bf16 ragged train", "op": "ragged", "dtype": "bf16", "n0": 1024, "n1": 700, "valid0": 1000, "valid1": 700,
         "heads": 4, "dim": 32, "train": True},
        # attention with the gate of the output projection, at inference
        {"name": "bf16 n512 gated infer", "op": "gated", "dtype": "bf16", "n": 512, "batch": 1, "heads": 4, "dim": 32, "train": False},
        # layer norm of the pair representation in front of the projections, f32 parameters
        {"name": "bf16 n768 layer norm", "op": "layer_norm", "dtype": "bf16", "rows": 768 * 768, "width": 128, "train": True},
        # triangle multiplicative update of a training crop, f32 parameters with 16-bit activations
        {"name": "bf16 n384 multiplication", "op": "multiplication", "dtype": "bf16", "n": 384, "channels": 128,
         "direction": "outgoing", "train": True},
        # token attention of several samples that share the pair bias, then its gated output projection
        {"name": "bf16 n512 token attention", "op": "tokens", "dtype": "bf16", "n": 512, "samples": 4, "heads": 16, "dim": 64,
         "train": True},
    ]


def _between(rng, low, high):
    """An integer spread over the logarithm of the range, odd ones as likely as even ones."""
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    op = rng.choice(["triangle"] * 6 + ["ragged", "gated", "layer_norm", "multiplication", "tokens"])
    half = rng.choice(["bf16", "bf16", "f16"])
    if op == "triangle":
        dtype = rng.choice(["f32", half, half, half, half])
        n = _between(rng, 48, 256 if dtype == "f32" else 1600)
        batch = rng.choice([1, 2]) if n <= 384 else 1
        mask = rng.choice(["none", "ones", "tokens"])
        case = _triangle("", dtype, n, batch=batch, train=rng.random() < 0.6, mask=mask,
                         valid=max(1, int(n * rng.uniform(0.7, 1.0))) if mask == "tokens" else n,
                         node=rng.choice(["starting", "ending"]), projected=rng.random() < 0.5)
    elif op == "ragged":
        n0, n1 = _between(rng, 64, 1024), _between(rng, 64, 1024)
        case = {"op": op, "dtype": half, "n0": n0, "n1": n1, "valid0": max(1, int(n0 * rng.uniform(0.8, 1.0))), "valid1": n1,
                "heads": 4, "dim": 32, "train": rng.random() < 0.6}
    elif op == "gated":
        case = {"op": op, "dtype": half, "n": _between(rng, 64, 1024), "batch": 1, "heads": 4, "dim": 32, "train": rng.random() < 0.4}
    elif op == "layer_norm":
        case = {"op": op, "dtype": rng.choice(["f32", half, half]), "rows": _between(rng, 64 * 64, 1024 * 1024),
                "width": rng.choice([64, 128, 256, 384]), "train": rng.random() < 0.6}
    elif op == "multiplication":
        case = {"op": op, "dtype": rng.choice(["f32", half, half, half]), "n": _between(rng, 48, 512),
                "channels": rng.choice([64, 128]), "direction": rng.choice(["outgoing", "incoming"]), "train": rng.random() < 0.6}
    else:
        case = {"op": op, "dtype": half, "n": _between(rng, 64, 768), "samples": rng.choice([1, 2, 4]), "heads": rng.choice([8, 16]),
                "dim": rng.choice([16, 24, 32, 48, 64]), "train": rng.random() < 0.6}
    case.pop("name", None)
    return case


def _token_pairs(valid, n):
    tokens = torch.arange(n, device="cuda") < valid
    return tokens[:, None] & tokens[None, :]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    dtype, train, op = DTYPES[case["dtype"]], case["train"], case["op"]

    def normal(*shape, scale=1.0, of=dtype, leaf=True):
        t = torch.randn(*shape, device="cuda", dtype=of, generator=gen)
        if scale != 1.0:
            t.mul_(scale)
        return t.requires_grad_(True) if leaf and train else t

    if op in ("triangle", "gated"):
        b, n, h, d = case["batch"], case["n"], case["heads"], case["dim"]
        shape = (b, n, n, h, d)
        leaves = [normal(*shape, scale=0.5) for _ in range(3)]
        if case.get("projected"):
            leaves.append(normal(b, n, n, h))
            bias = leaves[3].permute(0, 3, 1, 2).unsqueeze(1)
        else:
            leaves.append(normal(b, 1, h, n, n))
            bias = leaves[3]
        mask = None
        if case.get("mask") == "ones":
            mask = torch.ones(b, n, n, dtype=torch.bool, device="cuda")
        elif case.get("mask") == "tokens":
            mask = _token_pairs(case["valid"], n).expand(b, n, n).contiguous()
        state = {"leaves": leaves, "bias": bias, "mask": mask}
        if op == "gated":
            leaves.append(normal(*shape))
        if train:
            state["upstream"] = normal(*shape, leaf=False)
    elif op == "ragged":
        h, d, sizes = case["heads"], case["dim"], (case["n0"], case["n1"])
        state = {"leaves": [], "nested": []}
        for _ in range(3):
            packed = oops.NestedTensor([normal(n, n, h, d, scale=0.5, leaf=False) for n in sizes], ragged_dims=(0, 1))
            values = packed.concat.requires_grad_(train)
            state["leaves"].append(values)
            state["nested"].append(packed.packed_like(values).transpose(-4, -3))
        packed = oops.NestedTensor([normal(1, h, n, n, leaf=False) for n in sizes], ragged_dims=(2, 3))
        values = packed.concat.requires_grad_(train)
        state["leaves"].append(values)
        state["bias"] = packed.packed_like(values).transpose(-2, -1)
        state["tokens"] = oops.NestedTensor(
            [torch.arange(n, device="cuda") < valid for n, valid in zip(sizes, (case["valid0"], case["valid1"]))], ragged_dims=(0,))
        if train:
            state["upstream"] = normal(*state["leaves"][0].shape, leaf=False)
    elif op == "layer_norm":
        rows, width = case["rows"], case["width"]
        state = {"leaves": [normal(rows, width), normal(width, of=torch.float32), normal(width, of=torch.float32)]}
        if train:
            state["upstream"] = normal(rows, width, leaf=False)
    elif op == "multiplication":
        n, c = case["n"], case["channels"]
        master = {"of": torch.float32}
        weights = {f"{which}_norm_{what}": normal(c, **master) for which in ("input", "output") for what in ("weight", "bias")}
        for which in ("left_value", "left_gate", "right_value", "right_gate", "output", "output_gate"):
            weights[f"{which}_weight"] = normal(c, c, scale=c**-0.5, **master)
        pair = normal(1, n, n, c)
        mask = torch.ones(1, n, n, device="cuda")
        mask[:, n - n // 8:] = 0
        state = {"leaves": [pair, *weights.values()], "pair": pair, "weights": weights, "mask": mask, "direction": case["direction"]}
        if train:
            state["upstream"] = normal(1, n, n, c, leaf=False)
    else:
        s, h, n, d = case["samples"], case["heads"], case["n"], case["dim"]
        channels = 384
        leaves = [normal(s, h, n, d, scale=0.5) for _ in range(3)] + [normal(1, h, n, n)]
        leaves += [normal(s, n, channels), normal(h * d, channels, scale=channels**-0.5), normal(channels, h * d, scale=(h * d)**-0.5)]
        state = {"leaves": leaves}
        if train:
            state["upstream"] = normal(s, n, channels, leaf=False)
    state.update(op=op, train=train, node=case.get("node", "starting"))
    return state


def _forward(state):
    op = state["op"]
    if op == "triangle":
        q, k, v = state["leaves"][:3]
        mask = state["mask"]
        if state["node"] == "ending":
            q, k, v = (t.transpose(1, 2) for t in (q, k, v))
            mask = None if mask is None else mask.transpose(1, 2)
        return oops.triangle_attention(q, k, v, mask, state["bias"])
    if op == "gated":
        q, k, v, bias, gate = state["leaves"]
        return oops.triangle_attention_gated(q, k, v, gate, state["mask"], bias)
    if op == "ragged":
        mask = oops.pair_mask_from_token_mask(state["tokens"]).transpose(-2, -1)
        return oops.triangle_attention(*state["nested"], mask, state["bias"]).concat
    if op == "layer_norm":
        x, weight, bias = state["leaves"]
        return oops.layer_norm(x, x.shape[-1], weight, bias)
    if op == "multiplication":
        return oops.triangle_multiplication(state["pair"], state["mask"], direction=state["direction"], **state["weights"])
    q, k, v, bias, single, gate_weight, output_weight = state["leaves"]
    return oops.gate_attention_output(oops.pair_bias_attention(q, k, v, pair_bias=bias), single, gate_weight, output_weight)


def run(state):
    if not state["train"]:
        with torch.no_grad():
            return _forward(state)
    out = _forward(state)
    upstream = state["upstream"]
    if state["node"] == "ending":
        upstream = upstream.transpose(1, 2)
    return [out, *torch.autograd.grad(out, state["leaves"], upstream)]


def _attention_work(cells, logits, heads, dim, size, bias, mask, train, extra=0):
    """`cells` pair positions, `logits` kept (row, query, key) triples per head, `extra` further tensors of a call."""
    tensor = cells * heads * dim * size
    return {"bytes": tensor * ((8 if train else 4) + extra) + bias * size * (2 if train else 1) + mask,
            "flops": (14.0 if train else 4.0) * logits * heads * dim}


def work(case):
    size, train, op = 4 if case["dtype"] == "f32" else 2, case["train"], case["op"]
    if op in ("triangle", "gated"):
        b, n, h, d = case["batch"], case["n"], case["heads"], case["dim"]
        valid = case.get("valid", n)  # rows without a kept key give zeros and dropped keys give nothing
        return _attention_work(b * n * n, b * valid * n * valid, h, d, size, b * h * n * n,
                               b * n * n if case.get("mask", "none") != "none" else 0, train,
                               extra=0 if op == "triangle" else 2 if train else 1)
    if op == "ragged":
        h, d, pairs = case["heads"], case["dim"], ((case["n0"], case["valid0"]), (case["n1"], case["valid1"]))
        cells = sum(n * n for n, _ in pairs)
        return _attention_work(cells, sum(v * n * v for n, v in pairs), h, d, size, h * cells, cells, train)
    if op == "layer_norm":
        tensor = case["rows"] * case["width"] * size
        return {"bytes": tensor * (4 if train else 2) + case["width"] * (16 if train else 8), "flops": 0}
    if op == "multiplication":
        n, c = case["n"], case["channels"]
        forward = 2.0 * n * n * c * c * 6 + 2.0 * n * n * n * c
        return {"bytes": n * n * c * size * (4 if train else 2) + n * n * 4 + c * (6 * c + 4) * (8 if train else 4),
                "flops": forward * (3 if train else 1)}
    s, h, n, d, channels = case["samples"], case["heads"], case["n"], case["dim"], 384
    tensor, rest = s * h * n * d * size, 2 * s * n * channels * size + 2 * channels * h * d * size
    linear = 2.0 * s * n * channels * h * d * 2
    return {"bytes": tensor * (6 if train else 3) + (rest + h * n * n * size) * (2 if train else 1),
            "flops": (14.0 if train else 4.0) * s * n * n * h * d + linear * (3 if train else 1)}


def tolerance(case):
    """What rounding to the data type leaves open: operands of 16-bit products and results are rounded, f32 sums reordered."""
    if case["op"] == "multiplication":  # a chain of six projections, a contraction, two normalisations and three gates
        return {"rel": {"f32": 1e-4, "f16": 4e-3, "bf16": 2e-2}[case["dtype"]]}
    return {"rel": {"f32": 1e-5, "f16": 2e-3, "bf16": 1e-2}[case["dtype"]]}
