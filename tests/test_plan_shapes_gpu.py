"""Launch shapes that a plan takes from its number of codeblocks until a tuning is set: below one codeblock per
SM and on both sides of 1.75, results and TB bytes equal those of every explicit shape."""
import numpy as np
import pytest

from pusch_b200 import mcs, sim
from pusch_b200.pusch import PuschSlotPlan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [1, 4, 6])  # 51, 204 and 306 codeblocks
def test_plan_shapes_until_tuned(ctx, cells):
    ues, rb = [], 0
    for u, (n, layers, index) in enumerate([(6, 1, 3), (40, 1, 12), (220, 2, 26)]):
        qm, r = mcs.MCS_TABLE_2[index]
        snr = sim.required_snr_db(qm, r, layers, 4) + 3.0
        ues.append(sim.ue_from_mcs(rb, n, layers, 2, index, (2, 11), snr_db=snr, channel="pdp", rnti=0x4100 + u))
        rb += n
    plan = PuschSlotPlan(ctx, [sim.make_pusch_slot(ues, 4, seed=9)] * cells, graph=True)
    want = plan.execute_host()
    assert any(w.tb_crc_ok for w in want)
    for ctas, order in ((1, 0), (1, 1), (2, 0), (2, 1)):
        t = plan.tuning()
        t.ldpc_ctas_per_sm, t.ldpc_order = ctas, order
        plan.set_tuning(t)
        for g, w in zip(plan.execute_host(), want):
            assert (g.tb_crc_ok, g.nof_codeblocks, g.nof_codeblocks_crc_ok, g.mean_iterations) == (
                w.tb_crc_ok, w.nof_codeblocks, w.nof_codeblocks_crc_ok, w.mean_iterations)
            assert np.array_equal(g.transport_block, w.transport_block)
    plan.close()
