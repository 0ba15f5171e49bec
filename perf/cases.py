"""The workloads this framework's speed is measured on, and how their results are compared.

Every case is one call a user makes on a compiled model: ``CompiledModel.train_step(inputs, labels)`` (forward, loss,
backward, optimizer, and the loss read back) or ``CompiledModel.forward(inputs)`` on a model compiled for inference.
The models are the zoo's (``flexflow_train_b200.api.compile`` by name), at the sizes of the benchmark, the zoo's
defaults and the tests, with fewer layers or smaller tables where the deep model only repeats the same layer.
"""
import math

import torch

from flexflow_train_b200 import _ffcore as core
from flexflow_train_b200 import api
from flexflow_train_b200.runtime.executor import OptimizerConfig

CLASSIFY, REGRESS = "sparse_categorical_crossentropy", "mean_squared_error_avg_reduce"


def listed():
    return [
        # A small classifier on flattened images at the batch most people start with: launches and host time only.
        {"name": "mlp_train", "family": "mlp", "train": True, "dtype": "bf16", "batch": 64, "features": 784, "width": 512, "layers": 2,
         "classes": 10},
        # The recommendation benchmark: 8 tables, dot interaction, batch 4096, plain SGD with row-wise table updates.
        {"name": "dlrm_train", "family": "dlrm", "train": True, "dtype": "bf16", "batch": 4096, "tables": 8, "rows": 250000, "dim": 64,
         "dense": 13, "interaction": "DOT"},
        # Drug-response regression: seven feature inputs of odd widths (1, 942, 5270, 2048), wide layers, a small batch.
        {"name": "candle_uno_train", "family": "candle", "train": True, "dtype": "bf16", "batch": 64, "width": 1024, "feature_layers": 4,
         "layers": 3},
        # The benchmark's small language model: a training step short enough for launches to show.
        {"name": "lm_small_train", "family": "lm", "train": True, "dtype": "bf16", "batch": 8, "seq": 256, "heads": 8, "head_dim": 64,
         "layers": 2, "vocab": 4096},
        # One short prompt through a language model of that width: the latency of a single answer.
        {"name": "lm_forward_one", "family": "lm", "train": False, "dtype": "bf16", "batch": 1, "seq": 128, "heads": 8, "head_dim": 64,
         "layers": 6, "vocab": 4096},
        # The encoder-decoder Transformer in fp32 (tf32 products): 16 heads of 128, the precision the reference trains in.
        {"name": "transformer_fp32_train", "family": "transformer", "train": True, "dtype": "fp32", "batch": 8, "seq": 512, "heads": 16,
         "ffn": 2048, "layers": 3, "vocab": 64},
        # The same model as the zoo builds it by default (8 heads, so 256 wide ones), bf16, at a sequence that fills no tile.
        {"name": "transformer_default_train", "family": "transformer", "train": True, "dtype": "bf16", "batch": 16, "seq": 500, "heads": 8,
         "ffn": 2048, "layers": 3, "vocab": 64},
        # BERT-base layers on token ids at sequence 512 with the full vocabulary on the head.
        {"name": "bert_train", "family": "bert", "train": True, "dtype": "bf16", "batch": 16, "seq": 512, "hidden": 768, "heads": 12,
         "layers": 3, "vocab": 30528},
        # The headline model's layers and batch (2048 wide, 16 heads, FFN 8192, 32 x 1024 tokens, vocabulary 32000), Adam.
        {"name": "lm_large_train", "family": "lm", "train": True, "dtype": "bf16", "batch": 32, "seq": 1024, "heads": 16, "head_dim": 128,
         "layers": 4, "vocab": 32000},
        # The same model scoring a batch of documents whose length is no multiple of anything.
        {"name": "lm_large_forward", "family": "lm", "train": False, "dtype": "bf16", "batch": 4, "seq": 1001, "heads": 16, "head_dim": 128,
         "layers": 4, "vocab": 32000},
        # Inception-v3 with the auxiliary head, SGD with momentum: convolutions, batch norm and pooling, both directions.
        {"name": "inception_train", "family": "inception", "train": True, "dtype": "bf16", "batch": 64, "classes": 1000},
        # A handful of images through the same network: many small layers.
        {"name": "inception_forward", "family": "inception", "train": False, "dtype": "bf16", "batch": 5, "classes": 1000},
    ]


def _spread(rng, lo, hi, step=1):
    """A whole number of [lo, hi], spread over its logarithm, on the grid of `step`."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    family = rng.choice(("mlp", "dlrm", "candle", "lm", "lm", "transformer", "bert", "inception"))
    train = rng.random() < 0.7
    c = {"family": family, "train": train, "dtype": "bf16"}
    if family == "mlp":
        c.update(batch=_spread(rng, 16, 4096), features=_spread(rng, 64, 2048), width=_spread(rng, 64, 2048, 8), layers=rng.randint(1, 4),
                 classes=_spread(rng, 8, 1000))
    elif family == "dlrm":
        c.update(train=True, batch=_spread(rng, 64, 4096), tables=rng.randint(2, 8), rows=_spread(rng, 1000, 250000), dim=rng.choice((16, 32, 64)),
                 dense=rng.randint(4, 16), interaction=rng.choice(("DOT", "DOT", "CAT")))
    elif family == "candle":
        c.update(train=True, batch=_spread(rng, 16, 512), width=_spread(rng, 128, 1024, 8), feature_layers=rng.randint(2, 4), layers=rng.randint(2, 4))
    elif family == "lm":
        c.update(batch=_spread(rng, 1, 32), seq=_spread(rng, 32, 1024), heads=rng.choice((4, 8, 12, 16)), head_dim=rng.choice((64, 128)),
                 layers=rng.randint(1, 4), vocab=_spread(rng, 1000, 32000, 8))
    elif family == "transformer":
        heads = rng.choice((8, 16, 32))
        c.update(train=True, dtype=rng.choice(("bf16", "fp32")), batch=_spread(rng, 2, 16), seq=_spread(rng, 64, 512), heads=heads, ffn=2048,
                 layers=rng.randint(1, 3), vocab=64)
    elif family == "bert":
        heads = rng.choice((4, 8, 12))
        c.update(batch=_spread(rng, 1, 16), seq=_spread(rng, 32, 512), hidden=64 * heads, heads=heads, layers=rng.randint(1, 3),
                 vocab=_spread(rng, 1000, 30528, 8))
    else:
        c.update(batch=_spread(rng, 1, 64), classes=_spread(rng, 10, 1000))
    return c


def _model(case):
    """(zoo name, model configuration) of a case."""
    f = case["family"]
    if f == "mlp":
        return "mlp", {"batch_size": case["batch"], "input_dim": case["features"], "hidden": [case["width"]] * case["layers"],
                       "num_classes": case["classes"]}
    if f == "dlrm":
        return "dlrm", {"batch_size": case["batch"], "embedding_dim": case["dim"], "embedding_bag_size": 1,
                        "embedding_size": [case["rows"]] * case["tables"], "dense_arch_layer_sizes": [case["dense"], 512, 256, case["dim"]],
                        "over_arch_layer_sizes": [512, 512, 256, 1], "arch_interaction_op": case["interaction"], "final_activation": "SIGMOID",
                        "embedding_data_type": "FLOAT", "embedding_init_range": 0.01}
    if f == "candle":
        return "candle_uno", {"batch_size": case["batch"], "dense_layers": [case["width"]] * case["layers"],
                              "dense_feature_layers": [case["width"]] * case["feature_layers"]}
    if f == "lm":
        d = case["heads"] * case["head_dim"]
        return "transformer_lm", {"batch_size": case["batch"], "sequence_length": case["seq"], "num_features": d, "dim_feedforward": 4 * d,
                                  "num_heads": case["heads"], "num_decoder_layers": case["layers"], "vocab_size": case["vocab"], "dropout": 0.1}
    if f == "transformer":
        return "transformer", {"batch_size": case["batch"], "sequence_length": case["seq"], "num_heads": case["heads"],
                               "dim_feedforward": case["ffn"], "num_encoder_layers": case["layers"], "num_decoder_layers": case["layers"],
                               "vocab_size": case["vocab"]}
    if f == "bert":
        return "bert", {"batch_size": case["batch"], "sequence_length": case["seq"], "hidden_size": case["hidden"], "num_heads": case["heads"],
                        "dim_feedforward": 4 * case["hidden"], "num_encoder_layers": case["layers"], "vocab_size": case["vocab"],
                        "token_ids": True}
    return "inception_v3", {"batch_size": case["batch"], "num_classes": case["classes"]}


def _training(case):
    """(optimizer, loss) as the benchmark and the tests train the family.  Inception-v3 starts at the rate of a warm-up's
    first steps: from random weights the full rate moves it so far in one step that rounding decides where it lands."""
    f = case["family"]
    if f == "dlrm":
        return OptimizerConfig(kind="sgd", lr=0.01), REGRESS
    if f == "inception":
        return OptimizerConfig(kind="sgd", lr=1e-4, momentum=0.9), CLASSIFY
    if f == "mlp":
        return OptimizerConfig(kind="sgd", lr=0.05, momentum=0.9), CLASSIFY
    return OptimizerConfig(kind="adam", lr=1e-4), (REGRESS if f == "candle" else CLASSIFY)


def prepare(case, seed):
    """The compiled model (weights of the seed, as a program keeps them) and one batch on the device."""
    name, cfg = _model(case)
    graph = core.build_model(name, cfg)
    optimizer, loss = _training(case)
    model = api.compile(graph, config=api.FFConfig(compute_dtype=case["dtype"], seed=seed % 1000003), optimizer=optimizer, loss=loss,
                        training=case["train"])
    gen = torch.Generator(device="cuda").manual_seed(seed)
    inputs, rows, cols = {}, 1, 1
    nodes = {n["id"]: n for n in graph.nodes()}
    for n in nodes.values():
        if n["type"] != "INPUT":
            continue
        shape = n["outputs"][0][1]
        if shape.dtype in ("INT32", "INT64"):
            dt = torch.int32 if shape.dtype == "INT32" else torch.int64
            table = next(c for c in nodes.values() if c["type"] == "EMBEDDING" and (n["id"], "OUTPUT") in [tuple(v) for _, v in c["inputs"]])
            if n["name"] == "position_ids":
                t = torch.arange(shape.sizes[1], device="cuda", dtype=dt).view(1, -1, 1).repeat(shape.sizes[0], 1, 1)
            else:
                t = torch.randint(0, int(table["attrs"]["num_entries"]), list(shape.sizes), generator=gen, device="cuda", dtype=dt)
        else:
            t = torch.randn(list(shape.sizes), generator=gen, device="cuda")
        inputs[n["name"]] = t
    labels = None
    if case["train"]:
        *lead, cols = graph.shape(model.executable.loss_value).sizes
        rows = math.prod(lead)
        if loss == CLASSIFY:
            labels = torch.randint(0, cols, (rows,), generator=gen, device="cuda", dtype=torch.int32)
        else:
            labels = torch.randint(0, 2, (rows, cols), generator=gen, device="cuda").float()
    return {"model": model, "inputs": inputs, "labels": labels}


def run(state):
    """One training step (the loss and every updated weight come back) or one forward pass (the class probabilities come
    back)."""
    model = state["model"]
    if state["labels"] is None:
        return model.forward(state["inputs"])
    loss = model.train_step(state["inputs"], state["labels"])
    return {"loss": loss, "weights": [t for k, t in model.state_dict().items() if k == "master" or k.startswith("table.")]}


def work(case):
    """Products of the linear, attention, batched-matmul and convolution operators (three passes in training, two for an
    operator whose input needs no gradient); inputs and weights read once, results and updated state written once."""
    name, cfg = _model(case)
    graph = core.build_model(name, cfg)
    train = case["train"]
    act = 2 if case["dtype"] == "bf16" else 4
    fed, flops, nbytes, params, table_bytes, out_bytes = {}, 0.0, 0.0, 0, 0, 0

    def size(v):
        return math.prod(graph.shape(v).sizes)

    sparse = set()
    for n in graph.nodes():
        ins = {s: tuple(v) for s, v in n["inputs"]}
        a = n["attrs"]
        if n["type"] == "EMBEDDING" and _training(case)[0].kind == "sgd":
            sparse.add(ins["WEIGHT"])
        fed[n["id"]] = n["type"] == "WEIGHT" or any(fed[v[0]] for v in ins.values())
        if n["type"] == "INPUT":
            nbytes += size((n["id"], "OUTPUT")) * (8 if n["outputs"][0][1].dtype == "INT64" else 4)
            continue
        if n["type"] == "LINEAR":
            one = 2.0 * size((n["id"], "OUTPUT")) * graph.shape(ins["INPUT"]).sizes[-1]
            data = fed[ins["INPUT"][0]]
        elif n["type"] == "CONV2D":
            _, ch, kh, kw = graph.shape(ins["FILTER"]).sizes
            one = 2.0 * size((n["id"], "OUTPUT")) * ch * kh * kw
            data = fed[ins["INPUT"][0]]
        elif n["type"] == "BATCHMATMUL":
            one = 2.0 * size((n["id"], "OUTPUT")) * graph.shape(ins["LHS_INPUT"]).sizes[-1]
            data = True
        elif n["type"] == "MULTIHEAD_ATTENTION":
            (b, sq, dq), (_, sk, dk) = graph.shape(ins["QUERY"]).sizes, graph.shape(ins["KEY"]).sizes
            wide = a["num_heads"] * a["kdim"]
            one = 2.0 * b * wide * (sq * dq + 2 * sk * dk + sq * a["embed_dim"] + 2 * sq * sk)
            data = True
        else:
            one, data = 0.0, True
        flops += one * ((3 if data else 2) if train else 1)
        if n["type"] == "EMBEDDING":
            rows = size(ins["INPUT"]) * graph.shape(ins["WEIGHT"]).sizes[1] * 4
            table_bytes += rows * (2 if train and ins["WEIGHT"] in sparse else 1)
        if n["type"] == "SOFTMAX":
            out_bytes = size((n["id"], "OUTPUT")) * act
    for n in graph.nodes():
        v = (n["id"], "OUTPUT")
        if n["type"] == "WEIGHT" and not (train and v in sparse):
            params += size(v)
    if train:
        # weights and optimizer state are read and written in fp32
        kind = _training(case)[0]
        nbytes += params * 8 * (3 if kind.kind == "adam" else 2 if kind.momentum else 1) + table_bytes
    else:
        nbytes += params * act + out_bytes
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times what two correct ways of computing the case differ by after two steps, measured over the listed
    and 30 drawn cases: fused against unfused attention, implicit against im2col convolution, bf16 against fp32
    activations (Adam turns the sign of a gradient near zero into a whole step, hence the largest differences)."""
    f = case["family"]
    if not case["train"]:
        return {"rel": 2.5e-2, "max": 0.2}  # probabilities in bf16: 8e-3, 0.044
    if f == "mlp":
        return {"rel": 1.5e-3, "max": 0.06}  # weights 4e-4, 0.014
    if f == "dlrm":
        return {"rel": 2.5e-3, "max": 2.5e-3}  # loss 7e-4; weights and tables 2e-6, 1e-4
    if f == "candle":
        return {"rel": 1e-2, "max": 0.06}  # weights 1.8e-3, 0.016; loss up to 1e-2
    if f == "inception":
        return {"rel": 2.5e-2, "max": 0.4}  # weights 6e-4, 0.08; loss up to 1.3e-2
    if case["dtype"] == "fp32":
        return {"rel": 4e-4, "max": 0.1}  # tf32 products: 8e-5, 0.024
    return {"rel": 4.5e-3, "max": 0.1}  # 1.2e-3, 0.024
