"""Arguments of the transforms as trees of any container type: what is bound and how the gradients come back, on a plan
that only records (no device)."""

from collections import OrderedDict, defaultdict

import numpy as np
import pytest

import quabla_b200 as qb
from quabla_b200 import _transforms


class RecordingPlan:
    """Keeps what was bound; the gradient of a parameter is twice its bound value."""

    def __init__(self, spec, ordinal=0):
        self.names = [n for n, _, _ in spec.parameters] + [n for n, _, _, _ in spec.inputs]
        self.parameters = len(spec.parameters)
        self.bound = {}

    def slot(self, name):
        return self.names.index(name)

    def bind_many(self, slots, values):
        self.bound.update((slot, np.array(value)) for slot, value in zip(slots, values))

    def execute(self):
        pass

    def outputs(self):
        return [np.float64(0.0)] + [2.0 * self.bound[i] for i in range(self.parameters)]

    def close(self):
        pass


class Layers(list):
    pass


def _leaf(shape, seed):
    return np.random.default_rng(seed).normal(size=shape)


def _layer(kind, seed, n_in=2, n_out=3):
    layer = {"w": _leaf((n_in, n_out), seed), "b": _leaf((n_out,), seed + 1)}
    return defaultdict(None, layer) if kind is defaultdict else kind(layer)


def _loss(params, p):
    u = lambda x: (qb.tanh(x.reshape(1, -1) @ params[0]["w"] + params[0]["b"]) @ params[1]["w"] + params[1]["b"]).reshape(())
    return qb.mean(qb.vmap(u)(p) ** 2)


def _params(outer, inner, seed=0):
    return outer([_layer(inner, seed), _layer(inner, seed + 10, 3, 1)])


def _check(step, params, points):
    value, grads = step(params, points)
    assert type(grads) is type(params)
    for layer, given in zip(grads, params):
        assert type(layer) is dict and list(layer) == sorted(given)
        for key in given:
            if given[key] is None:
                assert layer[key] is None
            else:
                np.testing.assert_array_equal(layer[key], 2.0 * given[key])


@pytest.mark.parametrize("outer", [list, tuple, Layers])
@pytest.mark.parametrize("inner", [dict, OrderedDict, defaultdict])
def test_nested_containers(monkeypatch, outer, inner):
    monkeypatch.setattr(_transforms, "Plan", RecordingPlan)
    step = qb.value_and_grad(_loss)
    for seed in (0, 100, 200):  # traced, then repeated
        _check(step, _params(outer, inner, seed), _leaf((5, 2), seed))


def test_other_containers_around_the_same_leaves(monkeypatch):
    # One compiled loss serves them all; the gradients come in the containers of the call at hand.
    monkeypatch.setattr(_transforms, "Plan", RecordingPlan)
    step = qb.value_and_grad(_loss)
    points = _leaf((5, 2), 7)
    for outer, inner in [(list, dict), (tuple, dict), (list, OrderedDict), (Layers, dict), (tuple, dict), (list, dict)]:
        _check(step, _params(outer, inner), points)
    without = _params(list, dict)
    with_none = [dict(layer, extra=None) for layer in without]
    for params in (without, with_none, with_none, without):
        _check(step, params, points)
    assert len(step._cache) == 1
