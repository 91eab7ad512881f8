"""Uploads through the pinned staging blocks, captured step sequences and flat read-backs against the per-name calls
and single launches they stand for: the same bits."""

import ctypes as C
import os
import signal
import threading

import numpy as np
import pytest

import quabla_b200 as qb
from quabla_b200 import _host, _lib, workloads
from quabla_b200._plan import Plan, opt_config
from quabla_b200._transforms import CompiledLoss

from _util import traced

pytestmark = pytest.mark.gpu


# Point sets below and above the size that goes on the copy stream, and ragged around one staging block (1 MiB:
# 131,072 points of two float32 columns, 65,536 of heat's four).
@pytest.mark.parametrize("name,points", [("poisson1d", 64), ("poisson2d", 131072), ("poisson2d", 131075), ("heat3d", 65537)])
def test_staged_uploads_and_captured_steps_equal_single_calls(cuda_device, name, points):
    w, compiled, inputs = traced(name, points)
    plan, single = Plan(compiled.spec, 0), Plan(compiled.spec, 0)
    names = [n for n, _, _ in compiled.spec.parameters] + [n for n, _, _, _ in compiled.spec.inputs]
    plan.bind_many([plan.slot(n) for n in names], [inputs[n] for n in names])
    for n in names:
        np.testing.assert_array_equal(plan.read_input(n, np.shape(inputs[n])), inputs[n])
        single.bind(n, inputs[n])
    single.set_option(_lib.OPT_KERNEL_TIMERS, 1)  # never captured
    config = opt_config("adam", 1e-3)
    data = [n for n, _, _, _ in compiled.spec.inputs]
    for step in range(4):  # the second step captures the sequence, the later ones replay it on new batches
        batch = [np.roll(inputs[n], step, axis=0) for n in data]
        plan.bind_many([plan.slot(n) for n in data], batch)
        for n, value in zip(data, batch):
            single.bind(n, value)
        plan.train_step(config)
        single.execute()
        single.optimizer_step(config)
    for got, expected in zip(plan.outputs(), [single.read_output(i) for i in range(1 + len(compiled.spec.parameters))]):
        assert got.tobytes() == expected.tobytes()
    params, m, v = plan.read_state(moments=True)
    for i in range(len(compiled.spec.parameters)):
        assert params[i].tobytes() == single.read_parameter(i).tobytes()
    flat = np.concatenate([np.pad(a.reshape(-1), (0, -a.size % 4)) for a in v])
    assert flat.tobytes() == single.read_moments(1).tobytes()
    assert plan.loss() == single.loss()


def test_wrong_slots_and_sizes_upload_nothing(cuda_device):
    w, compiled, inputs = traced("poisson1d", 64)
    plan = Plan(compiled.spec, 0)
    names = [n for n, _, _ in compiled.spec.parameters]
    for slots, values in [([0, 99], [inputs[names[0]], inputs[names[1]]]), ([0, 1], [inputs[names[0]], np.zeros(999)])]:
        with pytest.raises(_lib.BackendError):
            plan.bind_many(slots, values)
    with pytest.raises(_lib.BackendError) as caught:
        plan.read_input(names[0], np.shape(inputs[names[0]]))
    assert caught.value.status == _lib.NOT_BOUND


@pytest.mark.parametrize("name", ["poisson1d", "poisson2d"])
@pytest.mark.parametrize("choose", [lambda n: range(0, n, 2), lambda n: range(1, n, 2), lambda n: reversed(range(n)),
                                    lambda n: [2, 1, 3], lambda n: [1, 0, n - 1], lambda n: [0, 0, 1]],
                         ids=["even", "odd", "reversed", "one before its predecessor", "last input", "twice"])
def test_any_choice_and_order_of_slots_leaves_the_others_alone(cuda_device, name, choose):
    # A bias is shorter than the padding a run of slots may contain: it must not be taken for padding.
    w, compiled, inputs = traced(name, 64)
    plan = Plan(compiled.spec, 0)
    names = [n for n, _, _ in compiled.spec.parameters] + [n for n, _, _, _ in compiled.spec.inputs]
    expected = {n: np.asarray(inputs[n]) + 1 for n in names}  # no zeros, biases included
    plan.bind_many([plan.slot(n) for n in names], [expected[n] for n in names])
    chosen = list(choose(len(names)))
    for slot in chosen:
        expected[names[slot]] = expected[names[slot]] * 2
    plan.bind_many(chosen, [expected[names[slot]] for slot in chosen])
    for n in names:
        np.testing.assert_array_equal(plan.read_input(n, expected[n].shape), expected[n], err_msg=n)


def test_a_captured_plan_follows_the_correction_scheme(cuda_device, monkeypatch):
    # QB200_TC_COR is read at every call, by a replayed sequence as by single launches.
    w, compiled, inputs = traced("heat3d", 640)
    plan, fresh = Plan(compiled.spec, 0), {}
    for n, value in inputs.items():
        plan.bind(n, value)

    def outputs(p):
        p.execute()
        return [o.tobytes() for o in p.outputs()] + [p.loss().tobytes()]

    for scheme in ("tf32", "bf16"):
        monkeypatch.setenv("QB200_TC_COR", scheme)
        single = Plan(compiled.spec, 0)
        for n, value in inputs.items():
            single.bind(n, value)
        fresh[scheme] = outputs(single)
        single.close()
    assert fresh["tf32"] != fresh["bf16"]
    for scheme in ("tf32", "tf32", "tf32", "bf16", "bf16", "bf16", "tf32", "bf16"):
        monkeypatch.setenv("QB200_TC_COR", scheme)
        assert outputs(plan) == fresh[scheme]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_plans_of_different_depth_on_two_threads(cuda_device, dtype):
    # They share a kernel and need different amounts of shared memory; single launches, so that every one sets it.
    def plan_of(depth):
        loss = workloads.make("poisson2d", 64).loss
        params = workloads.init_mlp(qb.random.key(depth), [2] + [64] * depth + [1], dtype)
        points = np.random.default_rng(depth).uniform(size=(64, 2)).astype(dtype)
        compiled = CompiledLoss(loss, (params, points, points), (0,), 0)
        compiled.bind((params, points, points))
        compiled.plan.set_option(_lib.OPT_KERNEL_TIMERS, 1)
        compiled.plan.execute()
        return compiled.plan, [o.tobytes() for o in compiled.plan.outputs()]

    failures = []

    def run(plan, expected):
        try:
            for _ in range(400):
                plan.execute()
            assert [o.tobytes() for o in plan.outputs()] == expected
        except Exception as e:  # reported below, on the test's thread
            failures.append(e)

    threads = [threading.Thread(target=run, args=plan_of(depth)) for depth in (1, 8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures


def test_a_refused_page_lock_leaves_the_next_step_alone(cuda_device):
    # More host memory than any machine has: refused on the host, and not the next launch's error.
    w, compiled, inputs = traced("poisson1d", 64)
    plan = Plan(compiled.spec, 0)
    for n, value in inputs.items():
        plan.bind(n, value)
    out = C.c_void_p()
    assert _lib.load().qb200_host_alloc(1 << 60, C.byref(out)) == _lib.CUDA_ERROR and out.value is None
    plan.execute()
    assert np.isfinite(plan.loss())


def test_read_back_buffers_are_recycled_and_bounded(cuda_device):
    first = _host.empty(1000, np.dtype(np.float32))
    address = first.__array_interface__["data"][0]
    view = first[10:20]
    del first
    second = _host.empty(1000, np.dtype(np.float32))  # the view keeps the first block out of the pool
    assert second.__array_interface__["data"][0] != address
    del view
    assert _host.empty(1000, np.dtype(np.float32)).__array_interface__["data"][0] == address
    held = [_host.empty(_host.LIMIT // 16, np.dtype(np.float64)) for _ in range(4)]  # more than the limit in all
    assert all(a.flags.writeable for a in held)
    assert _host._total <= _host.LIMIT
    del held
    assert _host._idle_bytes <= _host.IDLE_LIMIT


@pytest.mark.filterwarnings("ignore::DeprecationWarning")  # fork beside threads: the child only compares and exits
def test_a_forked_child_has_arrays_of_its_own(cuda_device):
    # As when a child writes a checkpoint while its parent trains on; the child makes no CUDA call.
    w, compiled, inputs = traced("heat3d", 64)
    plan = Plan(compiled.spec, 0)
    for n, value in inputs.items():
        plan.bind(n, value)
    plan.execute()
    grads = plan.outputs()[1:]
    kept = [g.copy() for g in grads]
    large = max(range(len(grads)), key=lambda i: grads[i].nbytes)
    (go, went), (answer, told) = os.pipe(), os.pipe()
    child = os.fork()
    if child == 0:
        try:
            signal.alarm(60)
            os.read(go, 1)  # the parent has read the next gradients by now
            same = all(g.tobytes() == k.tobytes() for g, k in zip(grads, kept))
            for g in grads:
                g.fill(7.0)
            del g, grads
            fresh = _host.empty(1000, np.dtype(np.float32))
            os.write(told, b"y" if same and fresh.flags.owndata else b"n")
        finally:
            os._exit(0)
    del grads
    plan.bind(compiled.spec.parameters[1][0], 2.0 * np.asarray(inputs[compiled.spec.parameters[1][0]]))
    plan.execute()
    later = plan.outputs()[1:]
    os.write(went, b"g")
    said = os.read(answer, 1)
    os.waitpid(child, 0)
    for end in (go, went, answer, told):
        os.close(end)
    assert said == b"y"
    assert later[large].tobytes() != kept[large].tobytes()
    for i, g in enumerate(later):
        assert g.tobytes() == plan.read_output(1 + i).tobytes()


def test_repeated_calls_follow_changed_arguments(cuda_device):
    # Same structure: bound without a new signature; another shape, another static value: traced anew.
    def loss(params, p, scale):
        u = qb.vmap(lambda x: (qb.tanh(x.reshape(1, -1) @ params["w"] + params["b"]) @ params["v"]).reshape(()))(p)
        return qb.mean((scale * u - 1.0) ** 2)

    rng = np.random.default_rng(3)
    params = {"w": rng.normal(size=(2, 16)), "b": np.zeros(16), "v": rng.normal(size=(16, 1))}
    step = qb.jit(qb.value_and_grad(loss), device="cuda:0")
    points = rng.normal(size=(40, 2))

    def value_of(p, scale):
        u = np.tanh(p @ params["w"] + params["b"]) @ params["v"]
        return np.mean((scale * u[:, 0] - 1.0) ** 2)

    for p, scale in [(points, 1.0), (points[::-1], 1.0), (points[:7], 1.0), (points, 2.0), (points, 1.0)]:
        value, grads = step(params, p, scale)
        assert abs(value - value_of(p, scale)) <= 1e-12
        assert sorted(grads) == ["b", "v", "w"] and grads["v"].shape == (16, 1)
