"""The autotuner searches the decoding kernels too: a plan set to the one-lane kernel, about half as fast, leaves it."""
import numpy as np
import pytest

from pusch_b200 import _native, sim
from pusch_b200.pusch import PuschSlotPlan

pytestmark = pytest.mark.gpu


def test_autotune_leaves_the_one_lane_kernel(ctx):
    import torch
    plan = PuschSlotPlan(ctx, sim.uneven_cells(seed=21, nof_cells=2), max_iterations=6)
    t = plan.tuning()
    t.ldpc_kernel = _native.PG_LDPC_KERNEL_ONE_LANE
    plan.set_tuning(t)
    best, _ = plan.autotune(torch.from_numpy(plan.grid.view(np.int32)).cuda().data_ptr(), reps=5)
    assert best.ldpc_kernel != _native.PG_LDPC_KERNEL_ONE_LANE
    assert plan.tuning().ldpc_kernel == best.ldpc_kernel
    plan.close()
