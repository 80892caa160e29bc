"""UCI results can be read with another device current than the plan's, and the current device stays as it was."""
import numpy as np
import pytest

from pusch_b200 import sim
from pusch_b200.pusch import PuschSlotPlan, batch_descriptors
from test_uci_plan_gpu import random_uci

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("current", [0, 1])
def test_read_with_another_device_current(ctx, current):
    import torch
    if torch.cuda.device_count() <= current:
        pytest.skip("one device")
    slots = sim.uneven_cells(seed=11, nof_cells=3)
    descs, _, _, ues = batch_descriptors(slots)
    ucis = random_uci(ctx, np.random.default_rng(21), ues, descs)
    plan = PuschSlotPlan(ctx, slots, uci=ucis)
    plan.execute_host()
    want = bytes(plan.uci_results())
    u = next(i for i, q in enumerate(ucis) if q.nof_harq_ack_bits)
    message = plan.uci_message(u, 0, ucis[u].nof_harq_ack_bits)
    with torch.cuda.device(current):
        assert bytes(plan.uci_results()) == want
        bits, valid = plan.uci_message(u, 0, ucis[u].nof_harq_ack_bits)
        assert np.array_equal(bits, message[0]) and valid == message[1]
        assert torch.cuda.current_device() == current
    plan.close()
