"""A count of arrivals left behind in a context's ordering launch (by replays of captured decodes that ran at the
same time, say) does not outlive the next batch: the batch after it is ordered and decoded as if nothing had
happened. The count is planted in the context's counters between two calls. The batch that meets it is the one
decoded before, so its keys and order are those already in place, whenever they are read."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from pusch_b200 import _native, sim
from pusch_b200.ldpc import LdpcBatchDecoder

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(__file__), "..", "ocudu-dapp-platform_b200", "csrc")
SHIM = """
#include "pg_internal.h"
extern "C" void* counters(void* ctx) { return static_cast<pg_context*>(ctx)->dev.ldpc_counter; }
"""


def counters_of(tmp_path, ctx):
    src, so = tmp_path / "shim.cpp", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", "-I/usr/local/cuda/include", str(src), "-o",
                    str(so)], check=True)
    f = ctypes.CDLL(str(so)).counters
    f.restype, f.argtypes = ctypes.c_void_p, [ctypes.c_void_p]
    return f(ctx.handle)


@pytest.mark.parametrize("kernel", [_native.PG_LDPC_KERNEL_Z384, _native.PG_LDPC_KERNEL_ONE_LANE])
@pytest.mark.parametrize("stale", [1, 3, 399])
def test_stale_arrivals_do_not_survive(tmp_path, kernel, stale):
    import torch
    from cuda.bindings import runtime
    ctx = _native.Context(max_codeblocks=1024)
    dec = LdpcBatchDecoder(context=ctx)
    dec.set_kernel(kernel)
    n = 400  # more than the CTAs of a launch: ordered
    jobs = [sim.ldpc_batch(seed=s, n=n, z=16, ebn0_range=(1.0, 5.0), max_iterations=5).jobs for s in (51, 52)]
    h2d, d2h = runtime.cudaMemcpyKind.cudaMemcpyHostToDevice, runtime.cudaMemcpyKind.cudaMemcpyDeviceToHost
    where = counters_of(tmp_path, ctx)
    first, second = dec.decode_batch(jobs[0]), dec.decode_batch(jobs[1])
    dec.decode_batch(jobs[0])
    torch.cuda.synchronize()
    planted = np.array([0, stale], np.int32)
    assert runtime.cudaMemcpy(where, planted.ctypes.data, 8, h2d)[0] == runtime.cudaError_t.cudaSuccess
    dec.decode_batch(jobs[0])
    left = np.full(2, -1, np.int32)
    assert runtime.cudaMemcpy(left.ctypes.data, where, 8, d2h)[0] == runtime.cudaError_t.cudaSuccess
    assert left[1] == 0
    for j, want in ((jobs[1], second), (jobs[0], first)):
        bits, it = dec.decode_batch(j)
        assert np.array_equal(it, want[1])
        assert all(np.array_equal(a, b) for a, b in zip(bits, want[0]))
    ctx.close()
