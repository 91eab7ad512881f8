"""The tensor-core fused kernels (split float32, FP64 MMA) against the CPU oracle at the edges of what they take: every padded width, unequal
widths, one to many hidden layers (running weight-gradient sums in shared and in global memory), ragged point counts,
every derivative signature, and operands that differ by many orders of magnitude, between streams and inside one block."""

import math

import numpy as np
import pytest

import quabla_b200 as qb
from oracle import contracted
from quabla_b200 import _lib, workloads
from quabla_b200._plan import Plan
from quabla_b200._transforms import CompiledLoss

from _util import TOLERANCE, relative_error

pytestmark = pytest.mark.gpu


def _residual(kind):
    def residual(f, q):
        if kind == "value":
            return f(q) - qb.sin(q[0])
        g = qb.grad(f)
        if kind == "first":
            return g(q)[0] + f(q)
        if kind == "second":
            return qb.hessian(f)(q)[0, 0] - f(q)
        if kind == "laplacian":
            h = qb.hessian(f)(q)
            total = h[0, 0]
            for i in range(1, q.shape[0]):
                total = total + (i + 1.0) * h[i, i]
            return total + f(q) * g(q)[0]
        if kind == "burgers":
            return g(q)[1] + f(q) * g(q)[0] - 0.1 * qb.hessian(f)(q)[0, 0]
        raise ValueError(kind)

    return residual


def _check(sizes, points, kind, activation="tanh", scale=1.0, dtype=np.float32):
    u = workloads.make_u(qb, activation)
    params = workloads.init_mlp(qb.random.key(11), sizes, dtype)
    for i, layer in enumerate(params):
        layer["b"] = qb.random.uniform(qb.random.key(50 + i), layer["b"].shape, dtype, -0.5, 0.5)
    if scale != 1.0:  # input directions on very different scales: streams of very different size
        params[0]["w"] = params[0]["w"] * dtype(scale)
    p = np.stack([qb.random.uniform(qb.random.fold_in(qb.random.key(5), j), (points,), dtype, -1.0, 1.0)
                  for j in range(sizes[0])], axis=1)

    def loss(params, p):
        return qb.mean(qb.vmap(lambda q: _residual(kind)(lambda s: u(params, s), q))(p) ** 2)

    args = (params, p)
    compiled = CompiledLoss(loss, args, (0,), 0)
    assert compiled.plan.query(_lib.Q_ENGINE) in (1, 2)
    assert compiled.plan.query(_lib.Q_FUSED_KERNEL) == (2 if np.dtype(dtype) == np.float32 else 3)
    spec = compiled.spec.unmerged or compiled.spec
    value, grads = contracted.value_and_grad(spec, compiled.named_inputs(args), threads=contracted.max_threads())
    compiled.bind(args)
    compiled.plan.execute()
    got = compiled.plan.outputs()
    tol = TOLERANCE[np.dtype(dtype)]
    assert relative_error(got[0], value) <= tol
    for (name, _, _), g, expected in zip(compiled.spec.parameters, got[1:], grads):
        assert relative_error(g.reshape(expected.shape), expected) <= tol, name


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("sizes,points", [
    ([1, 16, 1], 1), ([2, 16, 16, 1], 17), ([2, 32, 32, 32, 1], 255), ([2, 64, 64, 64, 64, 1], 15),
    ([2, 3, 5, 1], 1024), ([3, 17, 17, 17, 1], 1025), ([4, 48, 48, 48, 1], 1031), ([2, 33, 64, 20, 1], 1100),
    ([2, 63, 50, 1], 1999), ([1] + [64] * 12 + [1], 1050), ([2] + [16] * 12 + [1], 5000), ([2, 64, 64, 64, 64, 1], 9001),
], ids=lambda v: "-".join(map(str, v)) if isinstance(v, list) else str(v))
def test_widths_depths_and_point_counts(cuda_device, sizes, points, dtype):
    _check(sizes, points, "second", dtype=dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("activation", ["tanh", "sin"])
@pytest.mark.parametrize("width,kind,inputs", [
    (64, "value", 2), (64, "first", 2), (64, "burgers", 2), (64, "laplacian", 2), (64, "laplacian", 3), (64, "laplacian", 4),
    (50, "laplacian", 4), (48, "burgers", 2), (32, "laplacian", 3), (16, "laplacian", 4)])
def test_signatures(cuda_device, activation, width, kind, inputs, dtype):
    _check([inputs, width, width, width, 1], 1037, kind, activation, dtype=dtype)


@pytest.mark.parametrize("scale", [2.0 ** -40, 2.0 ** -12, 16.0])
def test_streams_of_very_different_size(cuda_device, scale):
    # Derivative streams grow with the scale of the first weights, to the first and second power: the parts have
    # float32's range (a float16 operand would be subnormal or infinite here).
    _check([2, 64, 64, 1], 1040, "burgers", "sin", scale=scale)


@pytest.mark.parametrize("width", [16, 32, 50, 64])
def test_truncation_leaves_no_common_factor(cuda_device, width):
    # The tensor core's truncation would lower every contraction by up to 4e-8 of itself, which no sum over points
    # averages out and which the residual of the heat equation amplifies (2e-6 on these gradients).  What is left is
    # random: float32's rounding (2^-24) in every factor, averaged over 10,007 points; 5e-7 allows for the residual.
    loss = workloads.make("heat3d", 128).loss
    params = workloads.init_mlp(qb.random.key(10007 + width), [4] + [width] * 4 + [1], np.float32)
    points = np.random.default_rng(10007 + width).uniform(0.0, 1.0, (10007, 4)).astype(np.float32)

    def flat(tree):
        return np.concatenate([np.asarray(layer[k], np.float64).ravel() for layer in tree for k in ("w", "b")])

    wide = [{k: v.astype(np.float64) for k, v in layer.items()} for layer in params]
    step = qb.jit(qb.value_and_grad(loss), device="cuda:0")
    value, grads = step(params, points)
    exact_value, exact = step(wide, points.astype(np.float64))
    assert np.linalg.norm(flat(grads) - flat(exact)) <= 5e-7 * np.linalg.norm(flat(exact))
    assert abs(float(value) - float(exact_value)) <= 5e-7 * abs(float(exact_value))


@pytest.mark.parametrize("width", [16, 50, 64])
@pytest.mark.parametrize("place", ["columns", "rows", "output"])
@pytest.mark.parametrize("power", [12, 30])
def test_every_entry_keeps_its_own_size(cuda_device, width, place, power):
    # Every third column or row of a hidden weight, or every third output weight, is 2^-power of its neighbours in the same
    # 16 x 16 block.  Columns and rows of all weight gradients are right relative to themselves, not to the largest
    # (with an exponent shared by a block they were off by up to 5e-2 at 2^-30): 2^-24 for each of some hundred factors
    # and sums per entry and an amplification of a few by the second derivative.
    loss = workloads.make("poisson2d", 128).loss
    params = workloads.init_mlp(qb.random.key(3), [2] + [width] * 3 + [1], np.float32)
    f = np.where(np.arange(width) % 3 == 1, 2.0 ** -power, 1.0).astype(np.float32)
    if place == "columns":
        params[1]["w"] = params[1]["w"] * f[None, :]
    elif place == "rows":
        params[1]["w"] = params[1]["w"] * f[:, None]
    else:
        params[-1]["w"] = params[-1]["w"] * f[:, None]
    rng = np.random.default_rng(width)
    interior = rng.uniform(0.0, 1.0, (2003, 2)).astype(np.float32)
    edge = rng.uniform(0.0, 1.0, (124, 2)).astype(np.float32)
    step = qb.jit(qb.value_and_grad(loss), device="cuda:0")
    _, grads = step(params, interior, edge)
    _, exact = step([{k: v.astype(np.float64) for k, v in layer.items()} for layer in params],
                    interior.astype(np.float64), edge.astype(np.float64))
    for i in range(3):
        g, e = grads[i]["w"].astype(np.float64), exact[i]["w"]
        for axis in (0, 1):
            error = np.linalg.norm(g - e, axis=axis) / np.linalg.norm(e, axis=axis)
            assert error.max() <= 2e-5, (i, axis, error.max())
