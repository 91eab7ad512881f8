"""Performance cases of the training step, through the public entry points.

The five PDE losses of `quabla_b200.workloads`, over the sizes, dtypes and options a training program meets, in the
three ways such a program calls the backend:

  train   `optim.Trainer`: `steps` optimizer steps, then what is written at a logging or checkpoint interval: the
          last loss, the parameters and the optimizer state.  The collocation points are resident on the device,
          or a new batch comes from host arrays every step, or a new batch is drawn on the device every step.
  grad    `jit(value_and_grad(loss))`: one call, for code that drives its own optimizer (L-BFGS, a line search):
          parameters and points in, value and gradients out, as host arrays.
  loss    `Trainer.loss()`: the forward pass alone, as for a validation loss.

Arrays are NumPy arrays because the surface is one of host arrays (the device holds the plan's own copies).
"""

import math

import numpy as np

import quabla_b200 as qb
from quabla_b200 import workloads

# Interior streams (value and derivatives along every direction the residual needs) and network inputs.
STREAMS = {"poisson1d": 3, "poisson2d": 4, "burgers": 4, "heat3d": 6, "beam": 5}
INPUTS = {"poisson1d": 1, "poisson2d": 2, "burgers": 2, "heat3d": 4, "beam": 1}
# Interior box, one (low, high) per input.
BOX = {"poisson1d": [(-1.0, 1.0)], "poisson2d": [(0.0, 1.0)] * 2, "burgers": [(-1.0, 1.0), (0.0, 1.0)],
       "heat3d": [(0.0, 1.0)] * 4, "beam": [(0.0, 1.0)]}


def _case(name, problem, mode, points, width, depth, dtype, activation="tanh", data="resident", optimizer="adam",
          steps=1):
    return {"name": name, "problem": problem, "mode": mode, "points": points, "width": width, "depth": depth,
            "dtype": dtype, "activation": activation, "data": data, "optimizer": optimizer, "steps": steps}


def listed():
    return [
        # The tutorial-sized problem: a step is a handful of short launches.
        _case("poisson1d train", "poisson1d", "train", 128, 16, 2, "float64", steps=50),
        # The same, one call at a time from a host optimizer: argument binding and read-back count.
        _case("poisson1d grad", "poisson1d", "grad", 128, 16, 2, "float64"),
        # 2-D Poisson at the configured size, a freshly sampled batch from the host every step.
        _case("poisson2d train, host batches", "poisson2d", "train", 65536, 64, 4, "float32", data="host", steps=8),
        # The same network at a small, ragged batch, gradients for a host optimizer.
        _case("poisson2d grad, 10007 points", "poisson2d", "grad", 10007, 64, 4, "float32"),
        # A hidden width that is no power of two, as hand-picked networks have.
        _case("poisson2d train, width 50", "poisson2d", "train", 20000, 50, 4, "float32", steps=10),
        # float64 is the default dtype of the surface's arrays; few points.
        _case("poisson2d train, float64", "poisson2d", "train", 8192, 64, 4, "float64", steps=10),
        # Viscous Burgers at the configured size.
        _case("burgers train", "burgers", "train", 262144, 128, 8, "float64"),
        # The usual ten thousand collocation points, ragged, gradients for L-BFGS.
        _case("burgers grad, 10007 points", "burgers", "grad", 10007, 128, 8, "float64"),
        # 3-D heat equation at the configured size: the largest case.
        _case("heat3d train", "heat3d", "train", 1048576, 256, 6, "float32"),
        # A minibatch of it redrawn on the device every step, decoupled decay and gradient clipping.
        _case("heat3d train, drawn batches", "heat3d", "train", 16411, 256, 6, "float32", data="device",
              optimizer="adamw clip", steps=5),
        # Validation loss of it: the forward direction alone.
        _case("heat3d loss", "heat3d", "loss", 131072, 256, 6, "float32"),
        # Fourth-order beam at the configured size.
        _case("beam train", "beam", "train", 1048576, 64, 4, "float32"),
    ]


def _sizes(case):
    return [INPUTS[case["problem"]]] + [case["width"]] * case["depth"] + [1]


def _parameter_count(case):
    sizes = _sizes(case)
    return sum(m * n + n for m, n in zip(sizes[:-1], sizes[1:]))


def _sets(case):
    """(points, streams) of every point set: the interior, then boundary and initial points."""
    n = case["points"]
    extra = {"poisson1d": [(2, 1)], "poisson2d": [(_edge_points(n, 16, 4), 1)],
             "burgers": [(_edge_points(n, 32, 2), 1)] * 2, "heat3d": [], "beam": [(2, 2)]}
    return [(n, STREAMS[case["problem"]])] + extra[case["problem"]]


def _edge_points(n, share, multiple):
    return max(multiple, n // share // multiple * multiple)


def _step_flops(case):
    """Matmul FLOPs of one step: forward 2 S Q, data and weight gradient twice that, the first layer without a data
    gradient."""
    sizes = _sizes(case)
    inner = sum(m * n for m, n in zip(sizes[1:-1], sizes[2:]))
    first = sizes[0] * sizes[1]
    forward_only = case["mode"] == "loss"
    total = 0.0
    for points, streams in _sets(case):
        forward = 2.0 * streams * inner + 2.0 * first
        total += points * (forward if forward_only else 3.0 * 2.0 * streams * inner + 2.0 * first * (2 + streams))
    return total


def work(case):
    item = 4 if case["dtype"] == "float32" else 8
    point_bytes = sum(points for points, _ in _sets(case)) * INPUTS[case["problem"]] * item
    parameter_bytes = _parameter_count(case) * item
    steps = case["steps"]
    if case["mode"] == "train":
        # Parameters and, for Adam, two moments, in and out; the points once, or once per batch.
        state = 6 if case["optimizer"].startswith("adam") else 2
        moved = state * parameter_bytes + point_bytes * (steps if case["data"] != "resident" else 1)
    elif case["mode"] == "grad":
        moved = 2 * parameter_bytes + point_bytes
    else:
        moved = parameter_bytes + point_bytes
    return {"bytes": float(moved), "flops": steps * _step_flops(case)}


def tolerance(case):
    # Value and gradients: sums over points of products carried in the dtype.  Optimizer state: Adam divides a
    # gradient by its own size, so an entry f times the leaf's largest carries the leaf's error times 1/f; "max"
    # admits single entries whose gradient is next to nothing.
    if case["dtype"] == "float32":
        return {"rel": 1e-4, "max": 0.05} if case["mode"] == "train" else {"rel": 1e-5}
    return {"rel": 1e-9, "max": 1e-6} if case["mode"] == "train" else {"rel": 1e-11}


def draw(rng):
    largest = _cost(next(c for c in listed() if c["name"] == "heat3d train"))
    while True:
        problem = rng.choice(sorted(STREAMS))
        mode = rng.choice(["train", "train", "grad", "loss"])
        dtype = rng.choice(["float64" if problem in ("poisson1d", "burgers") else "float32"] * 3 + ["float32", "float64"])
        width = rng.choice([16, 32, 50, 64, 64, 100, 128, 256])
        depth = rng.randint(2, 4 if problem == "beam" else 8)
        points = int(round(math.exp(rng.uniform(math.log(100), math.log(1048576)))))
        if rng.random() < 0.4:  # a third to a half of real batches are round numbers
            points = max(128, points // 128 * 128)
        activation = rng.choice(["tanh"] * 5 + ["sin", "sin", "gelu"])
        optimizer = rng.choice(["adam", "adam", "adamw clip", "sgd"]) if mode == "train" else "adam"
        data = rng.choice(["resident", "resident", "host", "device"]) if mode == "train" else "resident"
        if data == "device" and problem in ("poisson1d", "beam"):
            data = "host"  # one-column points: not what Trainer.resample draws
        case = _case("", problem, mode, points, width, depth, dtype, activation, data, optimizer, 1)
        del case["name"]
        if mode == "train":  # short steps are logged less often
            case["steps"] = max(1, min(20, int(2e11 / _cost(case))))
        if _cost(case) * case["steps"] <= largest:
            return case


def _cost(case):
    """FLOPs of a step, weighted by how much slower float64 and widths off the tensor cores' tiles run."""
    return _step_flops(case) * (8 if case["dtype"] == "float64" or case["width"] % 64 else 1)


def _points(case, rng):
    """The data arguments of the loss: points of every set, uniform in their domain."""
    problem, dtype = case["problem"], np.dtype(case["dtype"])
    sets = [points for points, _ in _sets(case)]

    def box(n):
        return np.stack([rng.uniform(low, high, n).astype(dtype) for low, high in BOX[problem]], axis=1)

    interior = box(sets[0])
    if problem == "heat3d":
        return (interior,)
    if problem in ("poisson1d", "beam"):
        return interior[:, 0].copy(), np.array(BOX[problem][0], dtype=dtype)
    edge = box(sets[1])
    if problem == "poisson2d":  # the four sides in turn
        side = np.arange(sets[1]) % 4
        edge[side < 2, 0] = side[side < 2]
        edge[side >= 2, 1] = side[side >= 2] - 2
        return interior, edge
    edge[:, 1] = 0.0
    target = (-np.sin(math.pi * edge[:, 0])).astype(dtype)
    wall = box(sets[2])
    wall[:, 0] = np.where(np.arange(sets[2]) % 2 == 0, -1.0, 1.0)
    return interior, edge, target, wall


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    loss = workloads.make(case["problem"], 128, activation=case["activation"]).loss
    params = workloads.init_mlp(qb.random.key(seed), _sizes(case), np.dtype(case["dtype"]))
    data = _points(case, rng)
    state = {"case": case, "params": params, "data": data, "key": qb.random.key(seed), "draws": 0}
    if case["mode"] == "grad":
        state["step"] = qb.jit(qb.value_and_grad(loss), device="cuda:0")
        state["step"](params, *data)  # traced and compiled, as after a program's first iteration
        return state
    optimizer = {"adam": qb.optim.Adam(1e-3), "adamw clip": qb.optim.AdamW(1e-3, clip_norm=1.0),
                 "sgd": qb.optim.SGD(1e-6)}[case["optimizer"]]  # a small rate: the losses are not normalised
    batch = () if case["data"] == "resident" else (0,) if case["data"] == "device" else tuple(range(len(data)))
    state["trainer"] = qb.optim.Trainer(loss, params, optimizer, *data, device="cuda:0", batch_argnums=batch)
    if case["data"] == "host":
        state["batches"] = [_points(case, rng) for _ in range(case["steps"])]
    return state


def run(state):
    case = state["case"]
    if case["mode"] == "grad":
        return state["step"](state["params"], *state["data"])
    trainer = state["trainer"]
    if case["mode"] == "loss":
        return trainer.loss()
    for i in range(case["steps"]):
        if case["data"] == "host":
            trainer.step(*state["batches"][i])
        else:
            if case["data"] == "device":
                state["draws"] += 1
                trainer.resample(0, qb.random.fold_in(state["key"], state["draws"]), BOX[case["problem"]])
            trainer.step()
    return {"loss": trainer.value, "state": trainer.export_state()}
