"""The library's host code against runtime calls that fail, on a stand-in for the CUDA runtime (compiled here, no device)."""

import os
import subprocess
import sys

import numpy as np
import pytest

from quabla_b200 import _build, _host, _lib

CUDA_INCLUDE = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_build._nvcc()))), "include")

# Every call can be made to fail; a failure stays the last error until it is read, as in the real runtime.
RUNTIME = r"""
#include <cuda_runtime.h>
#include <cstdio>
#include <cstdlib>
static cudaError_t last = cudaSuccess;
static bool fail_alloc, fail_event, fail_begin, fail_end, fail_instantiate;
static int allocated, capturing, graphs, queries_done;
static cudaError_t result(bool failed, cudaError_t e) { if (failed) last = e; return failed ? e : cudaSuccess; }
extern "C" {
cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    if (!fail_alloc) { *p = malloc(n); ++allocated; }
    return result(fail_alloc, cudaErrorMemoryAllocation);
}
cudaError_t cudaFreeHost(void* p) { free(p); --allocated; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)1; return result(fail_event, cudaErrorMemoryAllocation); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return queries_done ? cudaSuccess : cudaErrorNotReady; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    if (!fail_begin) ++capturing;
    return result(fail_begin, cudaErrorUnknown);
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    --capturing;
    if (!fail_end) { *g = (cudaGraph_t)1; ++graphs; }
    return result(fail_end, cudaErrorStreamCaptureInvalidated);
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    *e = (cudaGraphExec_t)1;
    return result(fail_instantiate, cudaErrorMemoryAllocation);
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { --graphs; return cudaSuccess; }
}
#define CHECK(c) do { if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
"""

STAGING = r"""
#include "host_staging.cu"
using namespace qb;
int main() {
    staging_attach(0);
    StagingBlock *a, *b;
    for (int event = 0; event < 2; ++event) {  // nothing to be had: the caller copies without staging
        fail_alloc = !event;
        fail_event = event;
        CHECK(staging_acquire(0, STAGING_BLOCKS, &a) == cudaSuccess && a == nullptr);
        CHECK(cudaGetLastError() == cudaSuccess && allocated == 0);
    }
    fail_alloc = fail_event = false;
    CHECK(staging_acquire(0, STAGING_BLOCKS, &a) == cudaSuccess && a != nullptr && allocated == 1);
    CHECK(staging_release(0, a, 0) == cudaSuccess);
    fail_alloc = true;  // no second block while the first is in transfer: wait for that one
    CHECK(staging_acquire(0, STAGING_BLOCKS, &b) == cudaSuccess && b == a);
    CHECK(cudaGetLastError() == cudaSuccess);
    CHECK(staging_acquire(0, STAGING_BLOCKS, &a) == cudaSuccess && a == nullptr);
    CHECK(staging_release(0, b, 0) == cudaSuccess);
    staging_detach(0);
    CHECK(allocated == 0);
    return 0;
}
"""

GRAPHS = r"""
#include "step_graph.h"
using namespace qb;
int main() {
    for (int failing = 0; failing < 5; ++failing) {
        fail_begin = failing == 1;
        fail_end = failing == 2;
        fail_instantiate = failing == 3;
        StepGraph g;
        int queued = 0;
        const bool made = capture_sequence((cudaStream_t)1, g, [&] { ++queued; return failing != 4; });
        CHECK(made == (failing == 0) && g.single == (failing != 0) && (g.exec != nullptr) == (failing == 0));
        CHECK(queued == (failing != 1) && capturing == 0 && graphs == 0);
        CHECK(cudaGetLastError() == cudaSuccess);
    }
    return 0;
}
"""


@pytest.mark.parametrize("program", [STAGING, GRAPHS], ids=["staging blocks", "captured sequences"])
def test_failing_runtime_calls_leave_the_plain_path(tmp_path, program):
    source = tmp_path / "program.cpp"
    source.write_text(RUNTIME + program)
    subprocess.run(["g++", "-std=c++17", "-I", _build.CSRC, "-I", CUDA_INCLUDE, str(source), "-o", str(tmp_path / "program")],
                   check=True)
    done = subprocess.run([str(tmp_path / "program")], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0, done.stdout


def test_read_back_falls_back_to_ordinary_memory(monkeypatch):
    class Refusing:
        def qb200_host_alloc(self, nbytes, out):
            return _lib.CUDA_ERROR

    monkeypatch.setattr(_lib, "load", Refusing)
    total = _host._total
    for _ in range(3):
        a = _host.empty(1000, np.dtype(np.float64))
        assert a.flags.owndata and a.shape == (1000,)
    assert _host._total == total


def test_blocks_that_outlive_the_modules_end_quietly():
    # On a stand-in for the library's two calls; builtins and os are cleared after the package.
    program = """
import builtins, ctypes, os
import numpy as np
from quabla_b200 import _host, _lib

class Memory:
    held = {}
    def qb200_host_alloc(self, nbytes, out):
        block = ctypes.create_string_buffer(nbytes)
        out._obj.value = ctypes.addressof(block)
        self.held[out._obj.value] = block
        return _lib.OK

memory = Memory()
_lib.load = lambda: memory
builtins.keep = os.keep = [_host.empty(n, np.dtype(np.float64)) for n in (100, 100, 300000)]
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    done = subprocess.run([sys.executable, "-c", program], cwd=root, capture_output=True, text=True, timeout=120)
    assert done.returncode == 0 and done.stderr == "", done.stderr
