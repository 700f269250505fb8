"""The workloads whose speed matters to a user of this library, as measurable cases.

A case is one call (or one short job) through the public entry points: `forward` of one sample, `forward_batch` on device
or host buffers, `train`, and `save` + `load`.  `listed()` names the ones to watch; `draw(rng)` gives others of the same
ranges: 1 to 65536 rows, the three configured nets and nets of ragged widths, the six stored precisions, the three math
modes, the five optimisers.

A served model stays loaded while inputs come and go, so nets of the inference cases are made once per process (fixed
seed) and shared by every prepared input; training and file jobs get a net of their own.
"""
import functools
import os
import tempfile

import numpy as np
import torch

import spingalett_b200 as spg
from spingalett_b200 import abi, configs

ACTS = {"sigmoid": abi.ACT_SIGMOID, "relu": abi.ACT_RELU, "tanh": abi.ACT_TANH, "leaky": abi.ACT_LEAKY_RELU,
        "foo52": abi.ACT_FOO52, "softmax": abi.ACT_SOFTMAX}
ACT_NAMES = {v: k for k, v in ACTS.items()}
BITS = {"fp32": 32, "fp16": 16, "bf16": 16, "int8": 8, "int4": 4, "int2": 2}
MODES = {"fast": abi.MATH_FAST, "exact": abi.MATH_EXACT, "auto": abi.MATH_AUTO}
OPTIMIZERS = {"sgd": abi.OPTIMIZER_SGD, "momentum": abi.OPTIMIZER_MOMENTUM, "rmsprop": abi.OPTIMIZER_RMSPROP,
              "adam": abi.OPTIMIZER_ADAM, "adamw": abi.OPTIMIZER_ADAMW}


def _net(topology, acts):
    """The two fields of a case that describe a net."""
    return {"net": "-".join(map(str, topology)), "acts": ",".join(ACT_NAMES.get(a, a) for a in acts)}


MLP = _net(configs.A_TOPO, configs.A_ACTS)
WIDE = _net(configs.W_TOPO, configs.W_ACTS)
LARGE = _net(configs.L_TOPO, configs.L_ACTS)


def _topology(case):
    return [int(v) for v in case["net"].split("-")]


def _weights(case):
    t = _topology(case)
    return sum(a * b for a, b in zip(t, t[1:]))


def listed():
    return [
        # one sample through the C API's forward() from host memory, on a net built with layer() (fp32): an interactive caller
        {"name": "sample_mlp_fp32", "kind": "sample", **MLP, "precision": "fp32", "rows": 1, "mode": "auto"},
        # a small served batch of the benchmark MLP, device buffers: launches and latency
        {"name": "mlp_int4_b256", "kind": "device", **MLP, "precision": "int4", "rows": 256, "mode": "auto"},
        # the headline configuration: bulk scoring with the benchmark MLP
        {"name": "mlp_int8_b65536", "kind": "device", **MLP, "precision": "int8", "rows": 65536, "mode": "auto"},
        # a data set of 60000 rows scored from ordinary (pageable) host arrays into host arrays
        {"name": "host_mlp_fp32_b60000", "kind": "host", **MLP, "precision": "fp32", "rows": 60000, "mode": "auto"},
        # a regression net of widths that are no multiple of anything, full-quality products, a batch that ends in a ragged tile
        {"name": "ragged_fp16_b3001_exact", "kind": "device", **_net([301, 777, 333, 129, 37], ["tanh", "leaky", "relu", "sigmoid"]),
         "precision": "fp16", "rows": 3001, "mode": "exact"},
        # the wide configuration: bulk scoring, bound by the tensor cores
        {"name": "wide_bf16_b16384", "kind": "device", **WIDE, "precision": "bf16", "rows": 16384, "mode": "auto"},
        # the large INT4 configuration's batch sweep: one request, a handful, a served batch, a large one
        {"name": "large_int4_b1", "kind": "device", **LARGE, "precision": "int4", "rows": 1, "mode": "auto"},
        {"name": "large_int4_b8", "kind": "device", **LARGE, "precision": "int4", "rows": 8, "mode": "auto"},
        {"name": "large_int4_b64", "kind": "device", **LARGE, "precision": "int4", "rows": 64, "mode": "auto"},
        {"name": "large_int4_b256", "kind": "device", **LARGE, "precision": "int4", "rows": 256, "mode": "auto"},
        # the training configuration: mini-batches of 256 with Adam over a few epochs, host arrays in, trained host arrays out
        {"name": "train_mlp_adam_b256", "kind": "train", **MLP, "samples": 4096, "epochs": 4, "batch": 256, "optimizer": "adam"},
        # a trained net of 25 million weights written as an INT8 file and read back
        {"name": "file_int8", "kind": "file", **_net([1024, 4096, 4096, 1000], ["relu", "relu", "softmax"]), "precision": "int8"},
    ]


class _View(np.ndarray):
    """Parameters of a net, in the net's own memory: holds on to the net."""
    net = None


def _parameters(net):
    views = {"weights": net.weights.view(_View), "biases": net.biases.view(_View)}
    for v in views.values():
        v.net = net
    return views


def _log(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, round(lo * (hi / lo) ** rng.random())))


def _ragged(rng, lo, hi, most_hidden):
    hidden = rng.randint(1, most_hidden)
    topology = [_log(rng, lo, hi) for _ in range(hidden + 1)] + [_log(rng, 2, 128)]
    acts = [rng.choice(["relu", "leaky", "tanh", "sigmoid", "foo52"]) for _ in range(hidden)] + [rng.choice(["softmax", "softmax", "sigmoid"])]
    return _net(topology, acts)


def draw(rng):
    kind = rng.choice(["mlp", "mlp", "large", "large", "wide", "ragged", "ragged", "host", "sample", "train", "file"])
    if kind == "mlp":
        return {"kind": "device", **MLP, "precision": rng.choice(list(BITS)), "rows": _log(rng, 1, 65536), "mode": rng.choice(["auto", "auto", "exact", "fast"])}
    if kind == "large":
        return {"kind": "device", **LARGE, "precision": rng.choice(["int4", "int4", "int8", "int2"]), "rows": _log(rng, 1, 512), "mode": "auto"}
    if kind == "wide":
        return {"kind": "device", **WIDE, "precision": rng.choice(["bf16", "fp16"]), "rows": _log(rng, 16, 16384), "mode": rng.choice(["auto", "fast"])}
    if kind == "ragged":
        return {"kind": "device", **_ragged(rng, 24, 2048, 4), "precision": rng.choice(list(BITS)), "rows": _log(rng, 1, 32768), "mode": rng.choice(["auto", "exact"])}
    if kind == "host":
        return {"kind": "host", **MLP, "precision": rng.choice(list(BITS)), "rows": _log(rng, 64, 65536), "mode": "auto"}
    if kind == "sample":
        return {"kind": "sample", **_ragged(rng, 24, 2048, 3), "precision": rng.choice(list(BITS)), "rows": 1, "mode": "auto"}
    if kind == "train":
        batch = _log(rng, 24, 512)
        return {"kind": "train", **(MLP if rng.random() < 0.5 else _ragged(rng, 24, 1024, 3)), "samples": batch * rng.randint(4, 16) + rng.choice([0, 0, batch // 3]),
                "epochs": rng.randint(1, 4), "batch": batch, "optimizer": rng.choice(list(OPTIMIZERS))}
    return {"kind": "file", **_net([_log(rng, 256, 4096), _log(rng, 512, 4096), _log(rng, 10, 1000)], ["relu", "softmax"]), "precision": rng.choice(list(BITS))}


def _built(net_text, acts_text, seed, loss=abi.LOSS_CROSS_ENTROPY):
    """A net built with layer() whose weights are N(0, gain/fan_in) (He for rectifiers, "Xavier" otherwise), biases small."""
    case = {"net": net_text}
    topology, acts = _topology(case), [ACTS[a] for a in acts_text.split(",")]
    net = spg.Network.build(topology, acts, abi.WEIGHT_INITIALIZATION_NONE, loss)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    w, b, pos = torch.from_numpy(net.weights), torch.from_numpy(net.biases), 0
    for fan_in, fan_out, act in zip(topology, topology[1:], acts_text.split(",")):
        gain = 2.0 if act in ("relu", "leaky", "foo52", "softmax") else 1.0
        count = fan_in * fan_out
        w[pos:pos + count] = (torch.randn(count, generator=gen, device="cuda") * (gain / fan_in) ** 0.5).cpu()
        pos += count
    b.copy_(torch.randn(b.numel(), generator=gen, device="cuda") * 0.01)
    return net


@functools.lru_cache(maxsize=2)
def _served(net_text, acts_text, precision):
    """The model a serving program has loaded: read from a .nn file of the wanted precision; fp32 ones stay as built."""
    net = _built(net_text, acts_text, seed=1234)
    if precision != "fp32":
        with tempfile.TemporaryDirectory() as folder:
            path = os.path.join(folder, "model.nn")
            net.save(path, abi.PRECISION_NAMES[precision])
            net.free()
            net = spg.Network.load(path)
    net.set_stream(torch.cuda.current_stream().cuda_stream)
    return net


def _inputs(rows, width, seed, uniform):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    make = torch.rand if uniform else torch.randn
    return make(rows, width, generator=gen, device="cuda")


def prepare(case, seed):
    spg.lib().spingalett_set_log_level(abi.LOG_WARNING)
    topology = _topology(case)
    kind = case["kind"]
    if kind in ("device", "host", "sample"):
        spg.set_math_mode(MODES[case["mode"]])
        net = _served(case["net"], case["acts"], case["precision"])
        # pixels for the benchmark MLP, standardised features otherwise, as configured
        x = _inputs(case["rows"], topology[0], seed, uniform=case["net"] == MLP["net"])
        if kind == "device":
            return {"kind": kind, "net": net, "rows": case["rows"], "x": x, "y": torch.empty(case["rows"], topology[-1], device="cuda")}
        if kind == "host":
            return {"kind": kind, "net": net, "x": x.cpu().numpy(), "y": np.zeros((case["rows"], topology[-1]), np.float32)}
        return {"kind": kind, "net": net, "x": x[0].cpu().numpy()}
    if kind == "train":
        softmax = case["acts"].endswith("softmax")
        net = _built(case["net"], case["acts"], seed, abi.LOSS_CROSS_ENTROPY if softmax else abi.LOSS_MSE)
        x = _inputs(case["samples"], topology[0], seed, uniform=True)
        gen = torch.Generator(device="cuda").manual_seed(seed + 1)
        classes = torch.randint(topology[-1], (case["samples"],), generator=gen, device="cuda")
        t = torch.nn.functional.one_hot(classes, topology[-1]).float()
        return {"kind": kind, "net": net, "x": x.cpu().numpy(), "t": t.cpu().numpy(), "w0": net.weights.copy(), "b0": net.biases.copy(),
                "epochs": case["epochs"], "batch": case["batch"], "optimizer": OPTIMIZERS[case["optimizer"]]}
    folder = tempfile.TemporaryDirectory()
    return {"kind": kind, "net": _built(case["net"], case["acts"], seed), "precision": abi.PRECISION_NAMES[case["precision"]], "folder": folder,
            "path": os.path.join(folder.name, "model.nn")}


def run(state):
    kind, net = state["kind"], state["net"]
    if kind == "device":
        net.forward_batch_ptr(state["x"].data_ptr(), state["rows"], state["y"].data_ptr())
        return state["y"]
    if kind == "host":
        return net.forward_batch(state["x"], state["y"])
    if kind == "sample":
        return net.forward(state["x"])
    if kind == "train":
        # a job that trains from the same checkpoint with the same shuffles, as one of a sweep does
        net.weights[:] = state["w0"]
        net.biases[:] = state["b0"]
        spg.lib().spingalett_seed(7)
        net.train(state["x"], state["t"], epochs=state["epochs"], batch_size=state["batch"], optimizer=state["optimizer"],
                  learning_rate=1e-3, reset_optimizer=True)
        return _parameters(net)
    net.save(state["path"], state["precision"])
    state["loaded"] = spg.Network.load(state["path"])
    return _parameters(state["loaded"])


def work(case):
    t, count = _topology(case), _weights(case)
    biases = sum(t[1:])
    if case["kind"] == "train":
        # samples and one-hot targets in, parameters in and out; three products per weight and row, but for the input's delta
        steps_rows = case["samples"] * case["epochs"]
        return {"bytes": 4 * case["samples"] * (t[0] + t[-1]) + 8 * (count + biases), "flops": 2 * steps_rows * (3 * count - t[0] * t[1])}
    stored = (count + biases) * BITS[case["precision"]] / 8
    if case["kind"] == "file":
        return {"bytes": 8 * (count + biases) + 2 * stored, "flops": 0}
    return {"bytes": stored + 4 * case["rows"] * (t[0] + t[-1]), "flops": 2 * case["rows"] * count}


def tolerance(case):
    if case["kind"] == "file":
        return "exact"
    if case["kind"] == "train":
        # fp32 sums in another order; Adam and RMSProp turn a gradient that is nearly zero into a full step of either sign
        return {"rel": 1e-4, "max": 0.1}
    if case["rows"] > 512 and case["mode"] != "exact" or case["mode"] == "fast":
        return {"rel": 5e-3}    # one 16-bit term per operand
    return {"rel": 1e-4}        # two 16-bit terms per activation, logits of some ten units in a softmax


def _activation(name, z):
    if name == "relu":
        return z.clamp(min=0)
    if name == "leaky":
        return torch.where(z > 0, z, 0.01 * z)
    if name == "foo52":
        return torch.where(z > 1, 1 + 0.01 * (z - 1), torch.where(z < 0, 0.01 * z, z))
    return {"sigmoid": torch.sigmoid, "tanh": torch.tanh, "softmax": lambda v: torch.softmax(v, 1)}[name](z)


def exact(case, seed):
    """The forward pass in 64 bits, on the weights that the loaded file stands for.  Files are compared byte for byte; a
    training job's result hangs on the order of the library's own shuffles and has no such value."""
    if case["kind"] not in ("device", "host", "sample"):
        return None
    topology = _topology(case)
    net = _served(case["net"], case["acts"], case["precision"])
    weights, biases = torch.from_numpy(np.array(net.weights)), torch.from_numpy(np.array(net.biases))
    a = _inputs(case["rows"], topology[0], seed, uniform=case["net"] == MLP["net"]).double()
    w_pos = b_pos = 0
    for fan_in, fan_out, act in zip(topology, topology[1:], case["acts"].split(",")):
        w = weights[w_pos:w_pos + fan_in * fan_out].cuda().double().view(fan_out, fan_in)
        a = _activation(act, a @ w.T + biases[b_pos:b_pos + fan_out].cuda().double())
        w_pos += fan_in * fan_out
        b_pos += fan_out
    return a[0].cpu().numpy() if case["kind"] == "sample" else a if case["kind"] == "device" else a.cpu().numpy()
