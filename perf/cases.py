"""The forward passes a user of this backend has it do, as cases for timing and comparison.

One case is one call of Handle.forward, the call NeuralNet::getOutput makes for a batch of positions: page-locked host
buffers in, host buffers out.  `listed` names the ordinary ones, `draw` gives others of the same ranges, `prepare` makes
what a program holds before the call (the handle of a loaded net, the positions of a batch, the result buffers), `run`
is the call.

Nets are the architectures of katago_b200.modelfile.  Their generators draw weights at N(0, 1/fan_in), which in a deep
residual net lets every block add as much as the stream already holds; a trained net's blocks add little each (they
start from scaled-down residual branches).  `_net` scales the last layer of every residual branch accordingly, so that
a rounding of the storage type is not blown up from block to block.
"""
import functools

import numpy as np

import katago_b200 as kb
from katago_b200 import capi
from katago_b200 import modelfile as mf

_PRECISION = {"fp32": kb.PRECISION_FP32, "fp16": kb.PRECISION_FP16, "bf16": kb.PRECISION_BF16}
_BYTES = {"fp32": 4, "fp16": 2, "bf16": 2}

# The batches of each net and type that are drawn, smallest and largest: fp16 is what an interactive search runs, from
# single positions up; bf16 the type of self-play servers' batches; fp32 that of accuracy checks and of small nets.
_BATCHES = {
    ("b6c96", "fp32"): (1, 64), ("b6c96", "fp16"): (1, 512),
    ("b18", "fp32"): (1, 8), ("b18", "fp16"): (1, 512), ("b18", "bf16"): (8, 256),
    ("b18human", "fp16"): (1, 128),
    ("b28", "fp16"): (1, 256), ("b28", "bf16"): (8, 512),
    ("transformer", "fp16"): (1, 256), ("transformer", "bf16"): (8, 128),
    ("transformer_relbias", "fp16"): (1, 192),
}


def listed():
    def case(name, net, dtype, n, edge=19, boards="full", symmetry=True):
        return dict(name=name, net=net, dtype=dtype, n=n, edge=edge, boards=boards, symmetry=symmetry)

    return [
        # one position at a time: a single-threaded search, or the raw net queried from a GUI
        case("b18_one_position", "b18", "fp16", 1),
        # a human-imitation net queried for the few candidate moves of one turn; metadata rows, no random symmetry
        case("b18human_few", "b18human", "fp16", 5, symmetry=False),
        # what a search with some dozen threads gathers in one batch
        case("b18_search_batch", "b18", "fp16", 37),
        # the headline: a full batch of a server thread
        case("b18_full_batch", "b18", "fp16", 256),
        # self-play on mixed board sizes, padded to 19x19 with the on-board mask
        case("b18_mixed_boards", "b18", "fp16", 128, boards="mixed"),
        # a server for 9x9 games only
        case("b18_9x9", "b18", "bf16", 193, edge=9),
        # the largest convolutional net under a small search, and under a full self-play batch
        case("b28_small_batch", "b28", "fp16", 12),
        case("b28_full_batch", "b28", "bf16", 512),
        # the transformer trunk in a full batch, and its relative-position variant in a small odd one
        case("transformer_full_batch", "transformer", "fp16", 128),
        case("relbias_small_batch", "transformer_relbias", "fp16", 11),
        # a small net in the exact type, and in the fast type as a policy prior for many positions
        case("b6_fp32", "b6c96", "fp32", 8),
        case("b6_fp16", "b6c96", "fp16", 100, boards="mixed"),
    ]


def draw(rng):
    net, dtype = rng.choice(sorted(_BATCHES))
    edge = rng.choice((19, 19, 19, 13, 9))
    least, most = _BATCHES[net, dtype]
    most *= 1 if edge == 19 else 2  # smaller boards, larger batches
    n = min(most, round(least * (most / least) ** rng.random()))
    boards = rng.choice(("full", "full", "mixed")) if edge == 19 else "full"
    return dict(net=net, dtype=dtype, n=n, edge=edge, boards=boards, symmetry=rng.random() < 0.75)


# ---- nets ----

def _branch_ends(blocks):
    """The layers whose output is added to a residual stream."""
    for b in blocks:
        kind = b["kind"]
        if kind == "ordinary_block":
            yield b["conv2"]
        elif kind == "gpool_block":
            yield b["finalConv"]
        elif kind == "nested_bottleneck_block":
            yield b["postConv"]
            yield from _branch_ends(b["blocks"])
        elif kind == "transformer_attention_block":
            yield b["out"]
        elif kind == "transformer_ffn_block":
            yield b["linear2"]


@functools.lru_cache(maxsize=2)
def _net(net):
    """(tree, Model) of a net; its weights are the same for every seed, as a program's are for every batch."""
    tree = {
        "b6c96": mf.make_b6c96,
        "b18": mf.make_b18c384nbt,
        "b18human": lambda: mf.add_meta_encoder(mf.make_b18c384nbt()),
        "b28": mf.make_b28c512nbt,
        "transformer": mf.make_transformer,
        "transformer_relbias": mf.make_transformer_relbias,
    }[net]()
    blocks = tree["trunk"]["blocks"]
    if not net.startswith("transformer"):  # those are drawn small already
        for layer in _branch_ends(blocks):
            layer["w"] = layer["w"] * np.float32(len(blocks) ** -0.5)
    return tree, kb.Model(mf.to_blob(tree))


@functools.lru_cache(maxsize=1)
def _handle(net, dtype, edge, max_batch):
    return kb.Handle(_net(net)[1], max_batch, nn_x=edge, nn_y=edge, precision=_PRECISION[dtype])


def _sizes(case):
    """Board edges of the batch: all full, or 9, 13 and 19 as 1:1:2."""
    if case["boards"] == "full":
        return [case["edge"]] * case["n"]
    return ([9, 13, 19, 19] * (case["n"] // 4 + 1))[:case["n"]]


# ---- the state before a call, and the call ----

class _Owner:
    """Array interface of page-locked memory that keeps the memory alive: arrays made from it outlive the state."""

    def __init__(self, shape, dtype):
        self.memory = capi.PinnedArray(shape, dtype)
        self.__array_interface__ = self.memory.array.__array_interface__


def _pinned(shape, dtype=np.float32, values=None):
    a = np.asarray(_Owner(shape, dtype))
    a[...] = 0 if values is None else values
    return a


def prepare(case, seed):
    n, edge = case["n"], case["edge"]
    model = _net(case["net"])[1]
    # a server's batch limit is a power of two; the batches it gets are not
    handle = _handle(case["net"], case["dtype"], edge, 1 << (n - 1).bit_length())
    spatial, glob = mf.random_positions(n, seed=seed, nn_len=edge, board_sizes=_sizes(case), num_spatial=model.in_c,
                                        num_global=model.in_global_c)
    state = {"handle": handle, "spatial": _pinned(spatial.shape, values=spatial), "glob": _pinned(glob.shape, values=glob),
             "symmetry": None, "meta": None}
    if case["symmetry"]:
        state["symmetry"] = _pinned((n,), np.int32, np.random.default_rng(seed + 1).integers(0, 8, n))
    if model.meta_c:
        meta = mf.random_meta_rows(n, seed=seed + 2, channels=model.meta_c)
        state["meta"] = _pinned(meta.shape, values=meta)
    shapes = {"policy": (n, edge * edge, model.policy_c), "policyPass": (n, model.policy_c), "value": (n, model.value_c),
              "scoreValue": (n, model.score_c), "ownership": (n, edge * edge)}
    state["out"] = {k: _pinned(shape) for k, shape in shapes.items()}
    return state


def run(state):
    return state["handle"].forward(state["spatial"], state["glob"], state["symmetry"], out=state["out"], meta=state["meta"])


# ---- what a pass cannot do without ----

def _layers(tree):
    """(multiply-adds per board point, multiply-adds per board, multiply-adds per pair of points, parameters) of a net."""
    point = board = pair = params = 0

    def walk(x):
        nonlocal point, board, pair, params
        if isinstance(x, list):
            for v in x:
                walk(v)
        if not isinstance(x, dict):
            return
        for v in x.values():
            if isinstance(v, np.ndarray):
                params += v.size
            else:
                walk(v)
        if x.get("kind") == "conv":
            point += x["kY"] * x["kX"] * x["inC"] * x["outC"]
        elif x.get("kind") == "transformer_attention_block":
            for key in ("q", "k", "v", "out"):
                point += x[key]["inC"] * x[key]["outC"]
                board -= x[key]["inC"] * x[key]["outC"]
            pair += x["heads"] * (x["qDim"] + x["vDim"])
        elif x.get("kind") == "transformer_ffn_block":
            for key in ("linear1", "gate", "linear2"):
                point += x[key]["inC"] * x[key]["outC"]
                board -= x[key]["inC"] * x[key]["outC"]
        elif x.get("kind") == "matmul":
            board += x["inC"] * x["outC"]

    walk(tree)
    return point, board, pair, params


def work(case):
    tree, model = _net(case["net"])
    point, board, pair, params = _layers(tree)
    area = [s * s for s in _sizes(case)]
    n, grid = case["n"], case["edge"] ** 2
    flops = 2 * (point * sum(area) + board * n + pair * sum(a * a for a in area))
    inputs = n * (grid * model.in_c + model.in_global_c + model.meta_c + (1 if case["symmetry"] else 0))
    outputs = n * (grid * (model.policy_c + 1) + model.policy_c + model.value_c + model.score_c)
    return {"bytes": 4 * (inputs + outputs) + params * _BYTES[case["dtype"]], "flops": flops}


# Relative 2-norm error and largest error of an output over its root mean square.  Measured for every net at one and at
# eight positions, reduced types against fp32 on the same net: fp16 0.0001 to 0.0027 and at most 0.01, bf16 (eight
# positions) 0.0002 to 0.012 and at most 0.05; fp32 against the same sums in another order on a CPU 7e-8 to 1e-6 and at most 3e-6.
_TOLERANCE = {"fp32": {"rel": 5e-6, "max": 2e-5}, "fp16": {"rel": 0.01, "max": 0.05}, "bf16": {"rel": 0.03, "max": 0.2}}


def tolerance(case):
    return _TOLERANCE[case["dtype"]]
