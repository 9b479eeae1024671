"""The calls a user of this library makes, at the sizes they make them: the cases its speed is measured on.

Six kinds of call, all through the public Python entry points:

layer        one fully connected ``LUTLayer``: forward, or forward + backward under one of the three gradient policies
projection   one ``ProjectionLUTLayer`` (sparse lookup -> output connectivity), forward + backward
convnet      the sparse conv-net for 28 x 28 images (three projection layers and a readout), forward or training pass
transformer  the character ``LUTTransformer``, logits or training pass
attention    one sequence layer, product or concatenation mode, forward + backward
inference    ``LUTInference``: the large forward-only layer with fp32 or int8 tables

Table indices are discontinuous in a layer's input, so in a stack of layers the rounding of one layer's sums would pick
other rows in the next.  The stacked kinds (convnet, transformer) therefore hold tables and embeddings on a grid of
2^-16: a sum of such entries is exact in fp32 in every order, the indices of all layers are reproducible, and only the
gradients round.  The single layers use tables that are not on any grid.
"""
import math

import torch
import torch.nn.functional as F

from spiky_b200.inference import LUTInference
from spiky_b200.lut_layer import (GradientPolicy, GradientType, LUTLayer, PointSamplingPolicy, PointSamplingType,
                                  ProjectionLUTLayer, SynapseMeta)
from spiky_b200.lut_transformer import LUTTransformer

DEVICE = "cuda:0"
GRID = 2.0 ** 16
TABLE_STD = 0.02
META = dict(min_weight=-1.0, max_weight=1.0)
POLICY = {"dense": GradientType.Dense, "sparse": GradientType.Sparse, "internal": GradientType.Internal}
LEARNING_RATE = 0.01
# (input side, output side, positions per side, tables per position) of the conv-net's projection layers, and its
# readout (inputs, outputs, tables, anchor pairs); 5 x 5 receptive fields, stride 2, 4 x 4 projections, 256-row tables
PROJECTIONS = [(28, 24, 12, 32), (24, 20, 10, 64), (20, 16, 8, 128)]
READOUT = (256, 10, 64, 8)


def _layer(name, batch, inputs, detectors, anchors, outputs, policy="dense", train=True):
    return dict(name=name, kind="layer", batch=batch, inputs=inputs, detectors=detectors, anchors=anchors,
                outputs=outputs, policy=policy, train=train)


def _attention(name, mode, batch, context, width, detectors, anchors, positional, policy="dense"):
    return dict(name=name, kind="attention", mode=mode, batch=batch, context=context, width=width,
                detectors=detectors, anchors=anchors, positional=positional, policy=policy)


def _transformer(name, batch, context, width, layers, heads, vocab, anchors, train):
    return dict(name=name, kind="transformer", batch=batch, context=context, width=width, layers=layers, heads=heads,
                vocab=vocab, anchors=anchors, train=train)


def _inference(name, tables, batch, inputs, detectors, anchors, outputs):
    return dict(name=name, kind="inference", tables=tables, batch=batch, inputs=inputs, detectors=detectors,
                anchors=anchors, outputs=outputs)


def listed():
    return [
        # the single-layer configuration at its own batch: a training step of a small model, where launches count
        _layer("layer, batch 256", 256, 784, 64, 6, 32),
        # the same layer fed with a large batch
        _layer("layer, batch 65536", 65536, 784, 64, 6, 32),
        # the feed-forward block of the character transformer over 64 sequences of 128 tokens
        _layer("feed-forward, 8192 tokens", 8192, 256, 16, 8, 256),
        # sizes nobody tuned for, table gradients as (cell, value) lists and an SGD step with them
        _layer("ragged layer, sparse SGD", 1111, 300, 50, 7, 33, policy="sparse"),
        # training pass of the conv-net, dense table gradients for the optimiser of the user's choice
        dict(name="conv-net step, batch 512", kind="convnet", batch=512, train=True),
        # its widest layer with the SGD update inside the backward pass, at a batch that fills no tile
        dict(name="projection, in-place SGD", kind="projection", which=2, batch=100, policy="internal"),
        # training pass of the character transformer at its own configuration
        _transformer("transformer step, batch 64", 64, 128, 256, 4, 4, 65, 8, True),
        # the same model asked for the logits of one sequence
        _transformer("transformer logits, batch 1", 1, 128, 256, 4, 4, 65, 8, False),
        # long context, 1024-row tables: four of the sixteen heads of the large transformer's attention layer
        _attention("long attention, 1024 tokens", "product", 1, 1024, 1024, 64, 10, 4),
        # concatenation mode, 65536-row tables updated in place: the attention layer of the byte-level language model
        _attention("concat attention, batch 32", "concat", 32, 32, 32, 64, 6, 4, policy="internal"),
        # the large inference layer: throughput with fp32 tables, and the small end of the batch sweep with int8 tables
        _inference("inference fp32, batch 16384", "fp32", 16384, 4096, 4096, 8, 64),
        _inference("inference int8, batch 4096", "int8", 4096, 4096, 4096, 8, 64),
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["layer", "layer", "projection", "convnet", "transformer", "attention", "attention", "inference"])
    if kind == "layer":
        detectors, outputs = _log(rng, 8, 256), _log(rng, 4, 256)
        batch = _log(rng, 1, max(1, min(65536, 65536 * 64 * 32 // (detectors * outputs))))
        c = _layer("", batch, rng.randint(16, 1024), detectors, rng.randint(4, 8), outputs,
                   policy=rng.choice(["dense", "dense", "sparse", "internal"]), train=rng.random() < 0.75)
    elif kind == "projection":
        c = dict(kind=kind, which=rng.randrange(3), batch=_log(rng, 16, 512), policy=rng.choice(["dense", "internal"]))
    elif kind == "convnet":
        c = dict(kind=kind, batch=_log(rng, 16, 512), train=rng.random() < 0.7)
    elif kind == "transformer":
        c = _transformer("", _log(rng, 1, 64), _log(rng, 16, 128), 32 * rng.randint(2, 8), rng.randint(1, 4),
                         rng.randint(1, 4), rng.randint(33, 256), rng.randint(6, 8), rng.random() < 0.6)
    elif kind == "attention" and rng.random() < 0.6:
        context = _log(rng, 64, 1024)
        c = _attention("", "product", _log(rng, 1, max(1, min(8, 1024 // context))), context, 32 * rng.randint(4, 32),
                       rng.randint(8, 64), rng.randint(7, 10), rng.choice([0, 4]),
                       policy=rng.choice(["dense", "internal"]))
    elif kind == "attention":
        c = _attention("", "concat", _log(rng, 1, 64), _log(rng, 8, 32), 32, rng.randint(16, 64), rng.randint(4, 6), 4,
                       policy=rng.choice(["dense", "internal"]))
    else:
        c = _inference("", rng.choice(["fp32", "int8"]), _log(rng, 1, 16384), rng.randint(512, 4096),
                       32 * rng.randint(16, 128), rng.randint(6, 8), 4 * rng.randint(4, 16))
    c.pop("name", None)
    return c


# ------------------------------------------------------------------------------------------------ preparation
def _policy(case):
    return GradientPolicy(POLICY[case.get("policy", "dense")])


def _fill_tables(layer, gen, on_grid=False):
    with torch.no_grad():
        layer._weights.normal_(0.0, TABLE_STD, generator=gen)
        if on_grid:
            layer._weights.mul_(GRID).round_().div_(GRID)


def _finish_layer(layer, gen, case, on_grid=False):
    layer.to(device=DEVICE)
    _fill_tables(layer, gen, on_grid)
    if case.get("policy") == "internal":
        layer.set_external_learning_rate_hook(lambda weights: LEARNING_RATE)
    return layer.train(case.get("train", True))


def _projection(which, seed, policy=None):
    side, out, grid, per = PROJECTIONS[which]
    return ProjectionLUTLayer(
        (side, side), (out, out), 8, grid * grid, per, (5, 5), (4, 4), synapse_meta=SynapseMeta(**META),
        detectors_sampling_policy=PointSamplingPolicy(PointSamplingType.Grid, grid_h=grid, grid_w=grid, stride_h=2,
                                                      stride_w=2, pad_h=2, pad_w=2),
        weights_gradient_policy=policy, random_seed=seed)


def _images(gen, batch, side):
    """About 19 % of the pixels lit, their values uniform in [0.5, 1)."""
    lit = torch.rand(batch, 1, side, side, device=DEVICE, generator=gen) < 0.19
    return torch.where(lit, 0.5 + 0.5 * torch.rand(lit.shape, device=DEVICE, generator=gen), 0.0)


def _zipf_tokens(gen, shape, vocab, s):
    p = torch.arange(1, vocab + 1, dtype=torch.float64, device=DEVICE) ** -s
    n = math.prod(shape)
    return torch.multinomial(p / p.sum(), n, replacement=True, generator=gen).view(shape)


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    kind = case["kind"]
    if kind == "layer":
        layer = LUTLayer(case["inputs"], case["anchors"], case["detectors"], case["outputs"],
                         synapse_meta=SynapseMeta(**META), weights_gradient_policy=_policy(case), random_seed=seed)
        _finish_layer(layer, gen, case)
        return dict(run=_run_layer if case["train"] else _run_forward, layer=layer,
                    x=torch.rand(case["batch"], 1, case["inputs"], device=DEVICE, generator=gen),
                    dy=torch.randn(case["batch"], 1, case["outputs"], device=DEVICE, generator=gen))
    if kind == "projection":
        layer = _finish_layer(_projection(case["which"], seed, _policy(case)), gen, case)
        side, out = PROJECTIONS[case["which"]][:2]
        x = _images(gen, case["batch"], side) if case["which"] == 0 else torch.randn(
            case["batch"], 1, side, side, device=DEVICE, generator=gen)
        return dict(run=_run_layer, layer=layer, x=x,
                    dy=torch.randn(case["batch"], 1, out, out, device=DEVICE, generator=gen))
    if kind == "convnet":
        layers = [_projection(i, seed + i) for i in range(3)]
        inputs, outputs, tables, anchors = READOUT
        layers.append(LUTLayer(inputs, anchors, tables, outputs, synapse_meta=SynapseMeta(**META), random_seed=seed + 3))
        for layer in layers:
            _finish_layer(layer, gen, case, on_grid=True)
        return dict(run=_run_convnet, layers=layers, train=case["train"], x=_images(gen, case["batch"], 28),
                    labels=torch.randint(0, 10, (case["batch"],), device=DEVICE, generator=gen))
    if kind == "transformer":
        model = LUTTransformer(case["vocab"], case["width"], case["context"], 4, case["layers"], case["heads"], 16,
                               case["anchors"], concatenation_product=False, seed=seed, device=DEVICE,
                               synapse_meta=SynapseMeta(**META))
        for layer in model._lut_layers():
            _fill_tables(layer, gen, on_grid=True)
        with torch.no_grad():
            model.token_embedder.weight.mul_(GRID).round_().div_(GRID)
        model.train(case["train"])
        return dict(run=_run_transformer, model=model, train=case["train"],
                    params=[p for p in model.parameters() if p.requires_grad],
                    tokens=_zipf_tokens(gen, (case["batch"], case["context"] + 1), case["vocab"], 1.1))
    if kind == "attention":
        product = case["mode"] == "product"
        layer = LUTLayer(case["width"], case["anchors"], case["detectors"], case["width"],
                         sequence_length=case["context"], concatenation_product=not product,
                         positional_dim=case["positional"], synapse_meta=SynapseMeta(**META),
                         weights_gradient_policy=_policy(case), random_seed=seed)
        _finish_layer(layer, gen, case)
        shape = (case["batch"], case["context"], case["width"])
        return dict(run=_run_layer, layer=layer, x=2 * torch.rand(shape, device=DEVICE, generator=gen) - 1,
                    dy=torch.randn(shape, device=DEVICE, generator=gen))
    detectors, inputs = case["detectors"], case["inputs"]
    first = torch.randint(0, inputs, (detectors, case["anchors"]), device=DEVICE, generator=gen)
    step = torch.randint(1, inputs, (detectors, case["anchors"]), device=DEVICE, generator=gen)
    anchors = torch.stack([first, (first + step) % inputs], dim=-1)
    n = detectors * (1 << case["anchors"]) * case["outputs"]
    if case["tables"] == "int8":
        tables = torch.randint(-127, 128, (n,), device=DEVICE, generator=gen, dtype=torch.int8)
        scales = (TABLE_STD / 127) * (0.5 + torch.rand(detectors, device=DEVICE, generator=gen))
    else:
        tables, scales = TABLE_STD * torch.randn(n, device=DEVICE, generator=gen), None
    layer = LUTInference(inputs, case["outputs"], detectors, case["anchors"], anchors, tables, scales,
                         int_rescaler=0.05, device=DEVICE)
    return dict(run=_run_forward, layer=layer, x=torch.randn(case["batch"], inputs, device=DEVICE, generator=gen))


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    return state["run"](state)


def _run_forward(state):
    with torch.no_grad():
        return state["layer"](state["x"])


def _run_layer(state):
    layer = state["layer"]
    for p in layer.parameters():
        p.grad = None
    x = state["x"].detach().requires_grad_(True)
    y = layer(x)
    y.backward(state["dy"])
    out = [y.detach(), x.grad]
    for p in layer.parameters():
        if p.grad is not None and p.grad.is_sparse:
            # how many cells the list holds differs from batch to batch: one SGD step takes it up
            p.data.add_(p.grad, alpha=-LEARNING_RATE)
        # where the update is in place (this list, or the policy without gradients) the new tables are the result
        out.append(p.detach() if p.grad is None or p.grad.is_sparse else p.grad)
    return out


def _run_convnet(state):
    layers, x = state["layers"], state["x"]
    with torch.set_grad_enabled(state["train"]):
        for layer in layers:
            layer._weights.grad = None
        z = x
        for layer in layers[:-1]:
            z = layer(z)
        logits = layers[-1](z.reshape(z.shape[0], 1, -1)).reshape(z.shape[0], -1)
        if not state["train"]:
            return logits
        loss = F.cross_entropy(logits, state["labels"])
        loss.backward()
    return [loss.detach(), logits.detach()] + [layer._weights.grad for layer in layers]


def _run_transformer(state):
    model, tokens = state["model"], state["tokens"]
    with torch.set_grad_enabled(state["train"]):
        logits = model(tokens[:, :-1])
        if not state["train"]:
            return logits
        for p in state["params"]:
            p.grad = None
        loss = F.cross_entropy(logits.reshape(-1, logits.shape[-1]), tokens[:, 1:].reshape(-1))
        loss.backward()
    return [loss.detach(), logits.detach()] + [p.grad for p in state["params"]]


# ------------------------------------------------------------------------------------------------ work and tolerance
def _fc_work(rows, inputs, detectors, table_rows, outputs, train, policy="dense"):
    """(bytes, adds and multiplies) of a fully connected layer on `rows` inputs: inputs, outputs, the tables (or the rows
    the batch can touch) once; backward: both gradients, and the tables' gradient or update."""
    tables = detectors * min(table_rows, rows) * outputs
    size, ops = rows * (inputs + outputs) + tables, rows * detectors * outputs
    if train:
        written = detectors * table_rows * outputs if policy == "dense" else tables
        size, ops = size + rows * (inputs + outputs) + written, 5 * ops
    return 4 * size, ops


def _projection_work(which, batch, train):
    side, out, grid, per = PROJECTIONS[which]
    # 4 x 4 projections cover 16 to 25 outputs of a position: 16 is the number that every position has
    tables, row = grid * grid * per, 16
    entries = tables * min(256, batch) * row
    size, ops = batch * (side * side + out * out) + entries, batch * tables * row
    if train:
        size, ops = 2 * size, 5 * ops
    return 4 * size, ops


def work(case):
    kind = case["kind"]
    if kind == "layer":
        b, f = _fc_work(case["batch"], case["inputs"], case["detectors"], 1 << case["anchors"], case["outputs"],
                        case["train"], case["policy"])
    elif kind == "projection":
        b, f = _projection_work(case["which"], case["batch"], True)
    elif kind == "convnet":
        parts = [_projection_work(i, case["batch"], case["train"]) for i in range(3)]
        inputs, outputs, tables, anchors = READOUT
        parts.append(_fc_work(case["batch"], inputs, tables, 1 << anchors, outputs, case["train"]))
        b, f = (sum(v) for v in zip(*parts))
    elif kind == "transformer":
        tokens, T, E = case["batch"] * case["context"], 1 << case["anchors"], case["width"]
        heads = 16 * case["heads"]
        ffn = _fc_work(tokens, E, 16, T, E, case["train"])
        out = _fc_work(tokens, E, 16, T, case["vocab"], case["train"])
        att = _fc_work(tokens, E, heads, T, E, case["train"])
        keys = (case["context"] - 1) / 2   # every query adds one row per key and detector
        b = case["layers"] * (ffn[0] + att[0]) + out[0]
        f = case["layers"] * (ffn[1] + keys * att[1]) + out[1]
    elif kind == "attention":
        bits = case["anchors"] if case["mode"] == "product" else 2 * case["anchors"] + case["positional"]
        pairs = case["batch"] * case["context"] * (case["context"] - 1) // 2
        rows = min(1 << bits, pairs)
        tokens = case["batch"] * case["context"]
        touched = case["detectors"] * rows * case["width"]
        written = case["detectors"] * (1 << bits) * case["width"] if case["policy"] == "dense" else touched
        b = 4 * (4 * tokens * case["width"] + touched + written)
        f = 5 * pairs * case["detectors"] * case["width"]
    else:
        entry = 1 if case["tables"] == "int8" else 4
        rows = min(1 << case["anchors"], case["batch"])
        b = (4 * case["batch"] * (case["inputs"] + case["outputs"])
             + entry * case["detectors"] * rows * case["outputs"])
        f = case["batch"] * case["detectors"] * case["outputs"]
    return {"bytes": b, "flops": f}


def tolerance(case):
    """Largest differences between correct fp32 evaluations: about four times what the same sums in 64 bits, another
    summation order and another kernel of the library show (largest seen: layers 5.7e-7, conv-net 3.4e-7, inference
    1e-7, product attention 2.9e-6 between row by row sums and histogram contractions, transformer 3.2e-6)."""
    kind = case["kind"]
    if kind == "inference":
        # int8 tables: fixed-point sums, the same bits in any order
        return "exact" if case["tables"] == "int8" else {"rel": 5e-7, "max": 5e-6}
    if kind == "attention" and case["mode"] == "product" or kind == "transformer":
        return {"rel": 1.2e-5, "max": 7e-4}
    return {"rel": 2.4e-6, "max": 6e-5}
