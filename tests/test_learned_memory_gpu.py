"""A net that a plan uses and that has not trained holds no gradient buffers; a training call allocates them again,
also where it is captured into a graph, and a net that has trained keeps them."""
import numpy as np
import pytest

from pusch_b200 import learned, sim
from pusch_b200 import tclayout as tl
from pusch_b200.pusch import PuschSlotPlan

pytestmark = pytest.mark.gpu

ROWS = 100_000
GRADIENTS = 13 * 128 * ROWS
SLACK = 8 << 20  # granularity of the allocations


def inputs(rows):
    import torch
    rng = np.random.default_rng(7)
    bf = lambda: torch.from_numpy(tl.to_chunked(tl.bf16_round(rng.standard_normal((rows, 16)).astype(np.float32)))
                                  .view(np.int16)).cuda()
    return bf(), bf(), torch.ones(rows, dtype=torch.uint8, device="cuda")


def free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.fixture(scope="module")
def plan(ctx):
    p = PuschSlotPlan(ctx, sim.uneven_cells(seed=3, nof_cells=1, max_ues=4))
    yield p
    p.close()


def train(net, rows, x, dy, valid, y, stream, graph):
    """Gradients of one forward and backward pass; the backward pass captured and replayed when graph is set."""
    import torch
    net.forward(x.data_ptr(), valid.data_ptr(), rows, y.data_ptr(), stream.cuda_stream)
    stream.synchronize()
    if graph:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            net.backward(dy.data_ptr(), rows, stream.cuda_stream)
        g.replay()
        torch.cuda.synchronize()
        del g
    else:
        net.backward(dy.data_ptr(), rows, stream.cuda_stream)
    grads = net.grads()
    net.status()
    return grads


@pytest.mark.parametrize("graph", [False, True])
def test_gradient_buffers_of_a_plan_s_net(ctx, plan, graph):
    import torch
    rows = 1025
    x, dy, valid = inputs(rows)
    y = torch.zeros((2, rows, 8), dtype=torch.int16, device="cuda")
    s = torch.cuda.Stream()
    fresh = learned.LearnedEstimator(ctx, rows, params=learned.init_params(3))
    want = train(fresh, rows, x, dy, valid, y, s, False)
    fresh.close()
    f0 = free()
    net = learned.LearnedEstimator(ctx, ROWS, params=learned.init_params(3))
    f1 = free()
    assert f0 - f1 < 1900 * ROWS + GRADIENTS + SLACK
    plan.set_learned(net)
    f2 = free()
    assert f2 - f1 > GRADIENTS - SLACK
    a = [r.tb_crc_ok for r in plan.execute_host()]
    got = train(net, rows, x, dy, valid, y, s, graph)
    f3 = free()
    assert abs(f2 - f3 - GRADIENTS) < SLACK + (64 << 20 if graph else 0)  # a capture may hold memory of its own
    plan.set_learned(None)
    plan.set_learned(net)  # trained: kept
    assert free() < f3 + GRADIENTS // 2
    assert [r.tb_crc_ok for r in plan.execute_host()] == a
    again = train(net, rows, x, dy, valid, y, s, False)
    plan.set_learned(None)
    net.close()
    # The same kernels on the same inputs; the order of the FP32 atomics differs.
    for g in (got, again):
        assert np.linalg.norm(g - want) <= 2e-6 * np.linalg.norm(want)
