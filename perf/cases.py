r"""The work that the speed of this package is judged by: its operators as a user's program calls them.

``listed()`` holds twelve cases, from a query of a few hundred points, where the launch and the Python around
it count, to the largest benchmark configuration.  ``draw(rng)`` gives further cases of the same ranges: point
and row counts over their logarithm (odd ones among them), the layer widths, depths, activations, biases and
data types the layers take.  ``prepare`` makes inputs and parameters from a seed, ``run`` is one call of the
public entry points: module or functional forward, or forward and the gradients of everything trainable, or
one optimisation step.

Operators (``case["op"]``):

``encode`` / ``encode_grad``   ``hash_encoding`` forward; forward and the table's gradient
``mlp`` / ``mlp_grad``         ``FullyFusedMLP`` forward; forward and the gradients of input and parameters
``rev`` / ``rev_grad``         ``ReversibleMLP``, the same two
``field`` / ``field_grad``     ``hash_encoded_mlp``, the same two
``train``                      ``NeuralFieldTrainer.step``: forward, loss, backward, Adam
"""
import math

import torch

from triton_helpers_b200.layers.fully_fused_mlp import FullyFusedMLP
from triton_helpers_b200.layers.hash_encoding import HashEncoding, hash_encoding
from triton_helpers_b200.layers.hash_encoding.helpers import level_geometry
from triton_helpers_b200.layers.neural_field import hash_encoded_mlp
from triton_helpers_b200.layers.reversible_mlp import ReversibleMLP
from triton_helpers_b200.training import NeuralFieldTrainer

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
BYTES = {"f32": 4, "f16": 2, "bf16": 2}


def _encode(op, n, dtype, d=3, feats=2, cap=2**19, max_res=2048, levels=16, clustered=False):
    return dict(op=op, n=n, dtype=dtype, d=d, feats=feats, cap=cap, max_res=max_res, levels=levels, clustered=clustered)


def _mlp(op, n, dtype, d_in=32, hidden=64, d_out=16, depth=2, activation="relu", bias=False):
    return dict(op=op, n=n, dtype=dtype, d_in=d_in, hidden=hidden, d_out=d_out, depth=depth, activation=activation, bias=bias)


def _rev(op, n, dtype, d_model=128, hidden=64, blocks=8, activation="relu", bias=False):
    return dict(op=op, n=n, dtype=dtype, d_model=d_model, hidden=hidden, blocks=blocks, activation=activation, bias=bias)


def _field(op, n, dtype, d=3, feats=2, cap=2**19, max_res=2048, levels=16, hidden=64, d_out=16, depth=2):
    return dict(op=op, n=n, dtype=dtype, d=d, feats=feats, cap=cap, max_res=max_res, levels=levels, clustered=False,
                hidden=hidden, d_out=d_out, depth=depth)  # fmt: skip


def listed():
    named = lambda name, case: dict(case, name=name)  # noqa: E731
    return [
        # a few rays' samples looked up in the default layer (2^14 rows per level, finest grid 512): latency
        named("encode_query", _encode("encode", 777, "f32", cap=2**14, max_res=512)),
        # benchmark configuration 0: a training batch of the float32 encoding by itself
        named("encode_grad", _encode("encode_grad", 65536, "f32")),
        # benchmark configuration 4: clustered points on a table far larger than L2; the largest case
        named("encode_grad_clustered", _encode("encode_grad", 2**22, "f32", feats=4, cap=2**22, max_res=4096, clustered=True)),
        # a decoder asked for one small batch: latency
        named("mlp_query", _mlp("mlp", 1000, "f16")),
        # the operator benchmark's network (64 wide, eight hidden layers after the first, biases): deep inference
        named("mlp_deep", _mlp("mlp", 32 * 8192, "f16", d_in=64, d_out=64, depth=9, bias=True)),
        # benchmark configuration 1: training step of the network by itself
        named("mlp_grad", _mlp("mlp_grad", 2**20, "f16", depth=4)),
        # a colour head as the module builds it: biases, smooth activation, three outputs, a ragged batch
        named("mlp_grad_rgb", _mlp("mlp_grad", 300_007, "bf16", d_out=3, depth=3, activation="silu", bias=True)),
        # a small ragged batch through the reversible stack
        named("rev_grad_small", _rev("rev_grad", 5003, "f16")),
        # benchmark configuration 2: the reversible stack
        named("rev_grad", _rev("rev_grad", 2**20, "bf16")),
        # an image (two coordinates) fitted with the fused operator, an odd number of pixels
        named("field_grad_image", _field("field_grad", 200_003, "f16", d=2, cap=2**17, max_res=4096)),
        # benchmark configuration 3: the training step
        named("train_step", _field("train", 2**21, "f16")),
        # float32 parameters throughout (the modules as constructed), a small batch: the autograd training step
        named("train_step_f32", _field("train", 2**14, "f32", cap=2**17, max_res=1024)),
    ]


def _count(rng, low, high):
    r"""A count between ``low`` and ``high``, even over its logarithm; half of them a multiple of 128."""
    n = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    return max(128, n // 128 * 128) if rng.random() < 0.5 else n


def draw(rng):
    op = rng.choice(("encode", "encode_grad", "mlp", "mlp_grad", "rev", "rev_grad", "field", "field_grad", "train"))
    if op in ("encode", "encode_grad"):
        # bfloat16 tables are looked up, not trained: eight bits are too few for sums over a batch
        dtype = rng.choice(("f32", "f16", "bf16") if op == "encode" else ("f32", "f16"))
        return _encode(op, _count(rng, 500, 2**21), dtype, rng.choice((2, 3, 3)), rng.choice((2, 2, 4)), 2 ** rng.randint(14, 21),
                       rng.choice((512, 1024, 2048, 4096)), rng.choice((8, 16, 16)), rng.random() < 0.3)  # fmt: skip
    if op in ("mlp", "mlp_grad"):
        dtype = rng.choice(("f16", "bf16", "f32"))
        depth = rng.randint(1, 9) if op == "mlp" else rng.randint(1, 3 if dtype == "f32" else 4)
        return _mlp(op, _count(rng, 500, 2**20), dtype, rng.choice((16, 27, 32, 32, 64)), rng.choice((32, 64, 64)),
                    rng.choice((1, 3, 16, 16, 64)), depth, rng.choice(("relu", "relu", "silu")), rng.random() < 0.5)  # fmt: skip
    if op in ("rev", "rev_grad"):
        plain = rng.random() < 0.7
        return _rev(op, _count(rng, 500, 2**19), rng.choice(("f16", "bf16")), rng.choice((64, 128, 128)), rng.choice((32, 64, 64)),
                    rng.randint(2, 10), "relu" if plain else "silu", not plain)  # fmt: skip
    dtype = rng.choice(("f16", "f16", "f32")) if op == "train" else "f16"
    return _field(op, _count(rng, 4000, 2**21 if dtype == "f16" else 2**18), dtype, rng.choice((2, 3, 3)), 2, 2 ** rng.randint(14, 20),
                  rng.choice((512, 1024, 2048)), rng.choice((8, 16, 16)), 64, rng.choice((8, 16)), rng.randint(1, 3))  # fmt: skip


# ---- inputs and parameters ---------------------------------------------------------------------------------


def _points(case, gen):
    n, d = case["n"], case["d"]
    if not case["clustered"]:
        return torch.rand(n, d, device="cuda", generator=gen)
    # samples near a few surfaces: a mixture of eight narrow Gaussians
    centres = torch.rand(8, d, device="cuda", generator=gen) * 0.6 + 0.2
    which = torch.randint(0, 8, (n,), device="cuda", generator=gen)
    return (centres[which] + 0.02 * torch.randn(n, d, device="cuda", generator=gen)).clamp_(0, 1 - 2**-24)


def _table(case, gen, dtype):
    rows = level_geometry(case["levels"], case["cap"], case["d"], 16, case["max_res"]).total_rows
    # entries of a table in training are of the order of 0.1
    return torch.randn(rows, case["feats"], device="cuda", generator=gen).mul_(0.1).to(dtype)


def prepare(case, seed):
    op, dtype = case["op"], DTYPES[case["dtype"]]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    torch.manual_seed(seed)  # the modules' own initialisation
    grad = op.endswith("_grad")
    normal = lambda *shape, scale=1.0: (torch.randn(*shape, device="cuda", generator=gen) * scale).to(dtype)  # noqa: E731
    state = {"op": op, "case": case}
    if op in ("encode", "encode_grad"):
        state["coords"] = _points(case, gen)
        state["table"] = _table(case, gen, dtype).requires_grad_(grad)
        if grad:
            state["grad_out"] = normal(case["n"], case["levels"] * case["feats"])
    elif op in ("mlp", "mlp_grad"):
        module = FullyFusedMLP(case["d_in"], case["hidden"], case["d_out"], case["depth"], case["activation"], bias=case["bias"])
        state["module"] = module.to("cuda", dtype)
        state["x"] = normal(1, case["n"], case["d_in"]).requires_grad_(grad)
        if grad:
            state["grad_out"] = normal(1, case["n"], case["d_out"], scale=1e-2)
    elif op in ("rev", "rev_grad"):
        module = ReversibleMLP(case["d_model"], case["blocks"], case["hidden"], case["activation"], bias=case["bias"])
        state["module"] = module.to("cuda", dtype)
        state["x"] = normal(case["n"], case["d_model"]).requires_grad_(grad)
        if grad:
            state["grad_out"] = normal(case["n"], case["d_model"])
    elif op in ("field", "field_grad"):
        state["coords"] = _points(case, gen)
        state["table"] = _table(case, gen, dtype).requires_grad_(grad)
        mlp = FullyFusedMLP(case["levels"] * case["feats"], case["hidden"], case["d_out"], case["depth"], bias=False).to("cuda", dtype)
        state["weights"] = [None if w is None else w.detach().requires_grad_(grad) for w in (mlp.w_in, mlp.w_out, mlp.w_hid)]
        if grad:
            state["grad_out"] = normal(case["n"], case["d_out"], scale=1e-2)
    else:
        encoding = HashEncoding(case["cap"], case["levels"], case["d"], case["feats"], 16, case["max_res"])
        with torch.no_grad():
            encoding.embeddings.mul_(0.1)
        mlp = FullyFusedMLP(case["levels"] * case["feats"], case["hidden"], case["d_out"], case["depth"], bias=case["dtype"] == "f32")
        state["trainer"] = NeuralFieldTrainer(encoding.to("cuda", dtype), mlp.to("cuda", dtype), lr=1e-2, betas=(0.9, 0.99), eps=1e-15)
        state["coords"] = _points(case, gen)
        state["targets"] = torch.rand(case["n"], case["d_out"], device="cuda", generator=gen).to(dtype)
    return state


# ---- one pass ----------------------------------------------------------------------------------------------


def _encode_call(state):
    c = state["case"]
    return hash_encoding(state["coords"], state["table"], None, None, c["cap"], 16, c["max_res"], c["levels"])


def _field_call(state):
    c = state["case"]
    w_in, w_out, w_hid = state["weights"]
    return hash_encoded_mlp(state["coords"], state["table"], w_in, w_out, w_hid, None, c["cap"], 16, c["max_res"], c["levels"])


def run(state):
    op = state["op"]
    if op == "train":
        loss = state["trainer"].step(state["coords"], state["targets"])
        return [loss] + [p.data for p in state["trainer"].parameters()]
    if not op.endswith("_grad"):
        with torch.no_grad():
            return _encode_call(state) if op == "encode" else _field_call(state) if op == "field" else state["module"](state["x"])
    if op == "encode_grad":
        y, wanted = _encode_call(state), [state["table"]]
    elif op == "field_grad":
        y, wanted = _field_call(state), [state["table"]] + [w for w in state["weights"] if w is not None]
    else:
        y, wanted = state["module"](state["x"]), [state["x"], *state["module"].parameters()]
    return [y.detach(), *torch.autograd.grad(y, wanted, state["grad_out"])]


# ---- what a pass cannot do without ---------------------------------------------------------------------------


def _table_rows(case):
    return level_geometry(case["levels"], case["cap"], case["d"], 16, case["max_res"]).total_rows


def _mlp_weights(case, d_in):
    return d_in * case["hidden"] + (case["depth"] - 1) * case["hidden"] ** 2 + case["hidden"] * case["d_out"]


def work(case):
    op, n, size = case["op"], case["n"], BYTES[case["dtype"]]
    grad = op.endswith("_grad")
    total = flops = 0
    if "cap" in case:
        corners, feats = n * case["levels"] * 2 ** case["d"], case["feats"]
        table = _table_rows(case) * feats * size
        # coordinates and the rows that are looked up, each once; a gradient fills the table's whole shape
        total += n * case["d"] * 4 + min(table, corners * feats * size) + (table if grad else 0)
        flops += (2 if grad or op == "train" else 1) * 2 * corners * feats
    if op in ("encode", "encode_grad"):
        total += (2 if grad else 1) * n * case["levels"] * case["feats"] * size
    elif op in ("mlp", "mlp_grad"):
        weights = _mlp_weights(case, case["d_in"])
        total += (2 if grad else 1) * (n * (case["d_in"] + case["d_out"]) + weights) * size
        flops += (3 if grad else 1) * 2 * weights * n
    elif op in ("rev", "rev_grad"):
        weights = case["blocks"] * 4 * (case["d_model"] // 2) * case["hidden"]
        total += (2 if grad else 1) * (2 * n * case["d_model"] + weights) * size
        flops += (3 if grad else 1) * 2 * weights * n
    else:
        weights = _mlp_weights(case, case["levels"] * case["feats"])
        total += (2 if grad else 1) * (n * case["d_out"] + weights) * size  # outputs and their gradient, or the targets
        flops += (3 if grad or op == "train" else 1) * 2 * weights * n
        if op == "train":
            # every parameter is written once more than it is read; two float32 moments are read and written
            total += table + (table + weights * size) // size * 16
    return {"bytes": total, "flops": flops}


def tolerance(case):
    op, dtype = case["op"], case["dtype"]
    if op == "encode":
        return {"rel": {"f32": 1e-6, "f16": 1e-3, "bf16": 8e-3}[dtype]}
    if op == "encode_grad":
        # float16 gradients of a row are sums of float16 contributions, in no fixed order
        return {"rel": 1e-5, "max": 1e-3} if dtype == "f32" else {"rel": 1e-2}
    if op == "train":
        # Adam's first steps move a parameter by lr times its gradient's sign: entries whose gradient is a sum that
        # nearly cancels may move the other way
        return {"rel": 1e-2, "max": 0.9}
    if op in ("mlp", "rev", "field"):
        return {"rel": 1e-2, "max": 0.1}
    # 16-bit activations within a rounding of zero switch their ReLU: single rows of the input's gradient differ
    return {"rel": 2e-2 if op == "rev_grad" else 1e-2, "max": 0.9}
