"""Point sets of one plan on two streams: the largest down the first lane, the others down the second."""

import pytest

from quabla_b200 import _lib
from quabla_b200._plan import Plan

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
