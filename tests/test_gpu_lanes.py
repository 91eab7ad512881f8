"""Point sets of one plan on two streams: the largest down the first lane, the others down the second."""

import numpy as np
import pytest

import quabla_b200 as qb
from quabla_b200 import _lib
from quabla_b200._plan import Plan
from quabla_b200._transforms import CompiledLoss

from _util import relative_error, traced

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points,scratch", [(64, None), (130, None), (3001, None), (16383, None), (3001, str(64 << 20))])
def test_sets_on_two_lanes_are_repeatable_and_agree_with_one(cuda_device, monkeypatch, points, scratch):
    _, compiled, inputs = traced("burgers", points)
    if scratch is not None:
        monkeypatch.setenv("QB200_SCRATCH_BYTES", scratch)  # the interior is cut into chunks: one lane

    def run(lanes, single=False):
        if lanes is None:
            monkeypatch.delenv("QB200_LANES", raising=False)
        else:
            monkeypatch.setenv("QB200_LANES", lanes)
        plan = Plan(compiled.spec, 0)
        for key, value in inputs.items():
            plan.bind(key, value)
        assert plan.query(_lib.Q_LANES) == (2 if lanes is None and scratch is None else 1)
        if single:
            plan.set_option(_lib.OPT_SINGLE_LANE, 1)
        results, losses = [], []
        for _ in range(4):  # launched one by one, then as a captured sequence
            plan.execute()
            results.append([o.copy() for o in plan.outputs()])
            losses.append(float(plan.loss()))
        plan.close()
        assert len(set(losses)) == 1
        for later in results[1:]:
            for a, b in zip(results[0], later):
                assert a.tobytes() == b.tobytes()
        return results[0]

    one = run("1")
    for other in (run(None), run(None, single=True) if scratch is None else one):
        for a, b in zip(other, one):
            assert relative_error(a, b) <= 1e-12  # two double accumulators added instead of one


def _two_sets(first, second, dtype=np.float64, width=128):
    """A residual of second order on `first` points, values on `second`, one hidden-to-hidden layer."""
    def loss(params, p, q):
        u = lambda x: (qb.tanh(qb.tanh(x.reshape(1, -1) @ params["w"] + params["b"]) @ params["m"]) @ params["v"]).reshape(())
        laplacian = lambda x: (lambda h: h[0, 0] + h[1, 1])(qb.hessian(u)(x))
        return qb.mean(qb.vmap(laplacian)(p) ** 2) + qb.mean(qb.vmap(u)(q) ** 2)

    rng = np.random.default_rng(2)
    params = {"w": rng.normal(size=(2, width)), "b": rng.normal(size=width), "m": rng.normal(size=(width, width)) / 12,
              "v": rng.normal(size=(width, 1)) / 12}
    params = {k: v.astype(dtype) for k, v in params.items()}
    return loss, (params, rng.uniform(size=(first, 2)).astype(dtype), rng.uniform(size=(second, 2)).astype(dtype))


@pytest.mark.parametrize("first,second", [(7000, 9000), (9000, 700), (20480, 700)])
def test_time_of_the_first_set_on_either_lane(cuda_device, first, second):
    # The set goes down the second lane, the first one, or (cut into chunks) both; beside other work it takes as long
    # as alone or longer.
    loss, args = _two_sets(first, second)
    compiled = CompiledLoss(loss, args, (0,), 0)
    plan = compiled.plan
    assert [s.n_points for s in compiled.spec.sets] == [first, second] and plan.query(_lib.Q_LANES) == 2
    compiled.bind(args)

    def times():
        out = []
        for _ in range(6):  # captured from the second on
            plan.execute()
            plan.synchronize()
            out.append(plan.query(_lib.Q_SET0_NANOSECONDS))
        return out[1:]

    both = times()
    plan.set_option(_lib.OPT_SINGLE_LANE, 1)
    alone = sorted(times())[2]
    # Two lanes halve the time of a set cut into chunks at best.
    assert min(both) >= 0.4 * alone, (both, alone)


@pytest.mark.parametrize("first,second,width", [(3001, 312, 128), (130, 3001, 256), (16500, 16500, 64 * 3)])
def test_float32_sets_on_two_lanes(cuda_device, monkeypatch, first, second, width):
    # tcgen05 GEMMs of two lanes at once, launched one by one and captured: repeatable, equal to one lane to the rounding
    # of a float32 result (the lanes' sums are double), and as near to float64 as the parity gate asks.
    loss, args = _two_sets(first, second, np.float32, width)
    results = {}
    for lanes in ("1", None):
        if lanes is None:
            monkeypatch.delenv("QB200_LANES")
        else:
            monkeypatch.setenv("QB200_LANES", lanes)
        compiled = CompiledLoss(loss, args, (0,), 0)
        assert compiled.plan.query(_lib.Q_LANES) == (1 if lanes else 2) and compiled.plan.query(_lib.Q_ENGINE) == 3
        compiled.bind(args)
        runs = []
        for _ in range(4):
            compiled.plan.execute()
            runs.append([o.copy() for o in compiled.plan.outputs()])
        assert all(a.tobytes() == b.tobytes() for later in runs[1:] for a, b in zip(runs[0], later))
        results[lanes] = runs[0]
    wide = ({k: v.astype(np.float64) for k, v in args[0].items()}, *(a.astype(np.float64) for a in args[1:]))
    exact = CompiledLoss(loss, wide, (0,), 0)
    exact.bind(wide)
    exact.plan.execute()
    for two, one, e in zip(results[None], results["1"], exact.plan.outputs()):
        assert relative_error(two, one) <= 2.0 ** -23
        assert relative_error(two, e) <= 1e-5
