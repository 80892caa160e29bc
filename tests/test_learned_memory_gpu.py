"""A net that only infers holds no gradient buffers: they come with the first backward pass, also where that pass is
captured into a graph."""
import numpy as np
import pytest

from pusch_b200 import learned
from pusch_b200 import tclayout as tl

pytestmark = pytest.mark.gpu

ROWS = 100_000


def inputs(rows):
    import torch
    rng = np.random.default_rng(7)
    bf = lambda: torch.from_numpy(tl.to_chunked(tl.bf16_round(rng.standard_normal((rows, 16)).astype(np.float32)))
                                  .view(np.int16)).cuda()
    return bf(), bf(), torch.ones(rows, dtype=torch.uint8, device="cuda")


def test_gradient_buffers_come_with_training(ctx):
    import torch
    rows = 300
    x, dy, valid = inputs(rows)
    y = torch.zeros((2, rows, 8), dtype=torch.int16, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    torch.cuda.synchronize()
    free = lambda: torch.cuda.mem_get_info()[0]
    f0 = free()
    net = learned.LearnedEstimator(ctx, ROWS, params=learned.init_params(3))
    f1 = free()
    net.forward(x.data_ptr(), valid.data_ptr(), rows, y.data_ptr(), st)
    net.status()
    f2 = free()
    net.backward(dy.data_ptr(), rows, st)
    net.status()
    f3 = free()
    net.backward(dy.data_ptr(), rows, st)
    net.status()
    slack = 8 << 20  # granularity of the allocations
    assert f0 - f1 < 1900 * ROWS + slack
    assert f2 > f1 - slack
    assert 13 * 128 * ROWS <= f2 - f3 + slack and f2 - f3 < 13 * 128 * ROWS + slack
    assert free() > f3 - slack
    net.close()
    torch.cuda.synchronize()
    assert free() > f0 - slack


def test_first_backward_captured(ctx):
    import torch
    rows = 1025
    x, dy, valid = inputs(rows)
    y = torch.zeros((2, rows, 8), dtype=torch.int16, device="cuda")
    grads = []
    for captured in (False, True):
        net = learned.LearnedEstimator(ctx, rows, params=learned.init_params(3))
        s = torch.cuda.Stream()
        torch.cuda.synchronize()
        net.forward(x.data_ptr(), valid.data_ptr(), rows, y.data_ptr(), s.cuda_stream)
        s.synchronize()
        if captured:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                net.backward(dy.data_ptr(), rows, s.cuda_stream)
            g.replay()
        else:
            net.backward(dy.data_ptr(), rows, s.cuda_stream)
        torch.cuda.synchronize()
        grads.append(net.grads())
        net.status()
        if captured:
            del g
        net.close()
    # The same kernels on the same inputs; the order of the FP32 atomics differs.
    assert np.linalg.norm(grads[1] - grads[0]) <= 2e-6 * np.linalg.norm(grads[0])
