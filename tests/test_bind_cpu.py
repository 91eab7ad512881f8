"""What a trainer's executor binds by name, on a library that only records (no device)."""

import ctypes as C

import numpy as np
import pytest

from quabla_b200 import _lib
from quabla_b200._plan import COTANGENT_NAME, Plan
from quabla_b200.optim import CudaTrainerExecutor

from _util import traced


class RecordingLibrary:
    def __init__(self, dtype, names):
        self.dtype, self.names, self.seen = np.dtype(dtype), names, {}

    def _take(self, name, address, nbytes):
        self.seen[name] = np.frombuffer(C.string_at(address, nbytes), self.dtype)

    def qb200_plan_bind(self, handle, name, address, nbytes):
        if name.decode() not in self.names and name.decode() != COTANGENT_NAME:
            return _lib.INVALID
        self._take(name.decode(), address, nbytes)
        return _lib.OK

    def qb200_plan_bind_many(self, handle, slots, hosts, sizes, n):
        for i in range(n):
            self._take(self.names[slots[i]], hosts[i], sizes[i])
        return _lib.OK


def _executor():
    _, compiled, inputs = traced("poisson1d", 8)
    plan = Plan(compiled.spec, 0, _handle=1)
    names = [n for n, _, _ in compiled.spec.parameters] + [n for n, _, _, _ in compiled.spec.inputs]
    plan._lib = RecordingLibrary(plan.dtype, names)
    executor = CudaTrainerExecutor.__new__(CudaTrainerExecutor)
    executor._plan = plan
    return executor, plan._lib, inputs


def test_lists_scalars_other_dtypes_and_the_cotangent():
    executor, library, inputs = _executor()
    x = np.linspace(-1.0, 1.0, 8)
    executor._bind({COTANGENT_NAME: 2.0, "x": x.tolist(), "xb": np.float32([[-1.0], [1.0]])[:, ::1],
                    "params/2/b": np.float64(0.25), "params/0/b": np.arange(32.0)[::2]})
    np.testing.assert_array_equal(library.seen["x"], x)
    np.testing.assert_array_equal(library.seen["xb"], [-1.0, 1.0])
    np.testing.assert_array_equal(library.seen["params/2/b"], [0.25])
    np.testing.assert_array_equal(library.seen["params/0/b"], np.arange(32.0)[::2])
    np.testing.assert_array_equal(library.seen[COTANGENT_NAME], [2.0])


def test_unknown_names_are_the_librarys_to_refuse():
    executor, library, inputs = _executor()
    with pytest.raises(_lib.BackendError):
        executor._bind({"nothing": np.zeros(3)})


@pytest.mark.parametrize("name", ["poisson1d", "heat3d"])
def test_leaves_do_not_keep_the_read_back_buffer(name):
    _, compiled, _ = traced(name, 8)
    plan = Plan(compiled.spec, 0, _handle=1)
    plan._layout()
    flat = np.arange(1 + plan._flat_size, dtype=plan.dtype)
    leaves = plan._leaves(flat, 1)
    for i, (leaf, (_, first)) in enumerate(zip(leaves, plan._layout())):
        assert leaf.flags.writeable and not np.shares_memory(leaf, flat)
        assert not any(np.shares_memory(leaf, other) for other in leaves[:i])
        np.testing.assert_array_equal(leaf.reshape(-1), np.arange(1 + first, 1 + first + leaf.size, dtype=plan.dtype))
