"""Slot plans join their transport blocks inside the decoder: results and TB bytes equal those of the
stage-by-stage entry (separate TB assembly and CRC) for TBs of one codeblock with odd and even lifting
sizes, of many codeblocks, decoded and failing, on repeated executions of one plan and with the
one-lane decoder, whose plans keep the separate join."""
import numpy as np
import pytest

from pusch_b200 import _native, sim
from pusch_b200.pusch import PuschProcessor, PuschSlotPlan

pytestmark = pytest.mark.gpu

# (PRBs, layers, MCS index of table 2): lifting sizes from 3 up, 1 to 50 codeblocks.
GRANTS = [(1, 1, 0), (1, 1, 1), (1, 1, 4), (2, 1, 0), (2, 1, 6), (3, 2, 11), (9, 1, 3), (20, 2, 8), (30, 1, 26), (60, 2, 20),
          (100, 2, 27)]


@pytest.mark.parametrize("offset_db", [4.0, -1.5])
def test_join_equals_separate_stages(ctx, offset_db):
    from pusch_b200 import mcs
    ues, rb = [], 0
    for u, (n, layers, index) in enumerate(GRANTS):
        qm, r = mcs.MCS_TABLE_2[index]
        snr = sim.required_snr_db(qm, r, layers, 4) + offset_db - 8.0 * (u % 3 == 2) * (offset_db < 0)
        ues.append(sim.ue_from_mcs(rb, n, layers, 2, index, (2, 11), snr_db=snr, channel="pdp", rnti=0x4000 + u))
        rb += n
    slots = [sim.make_pusch_slot(ues, 4, seed=int(40 + offset_db))]
    want = PuschProcessor(ctx).process_slots(slots)
    assert sorted({w.nof_codeblocks for w in want})[-1] > 8
    plan = PuschSlotPlan(ctx, slots, graph=True)
    for kernel in (_native.PG_LDPC_KERNEL_Z384, _native.PG_LDPC_KERNEL_Z384, _native.PG_LDPC_KERNEL_ONE_LANE,
                   _native.PG_LDPC_KERNEL_Z384):
        t = plan.tuning()
        t.ldpc_kernel = kernel
        plan.set_tuning(t)
        for g, w in zip(plan.execute_host(), want):
            assert (g.tb_crc_ok, g.nof_codeblocks, g.nof_codeblocks_crc_ok, g.mean_iterations) == (
                w.tb_crc_ok, w.nof_codeblocks, w.nof_codeblocks_crc_ok, w.mean_iterations)
            assert not g.tb_crc_ok or np.array_equal(g.transport_block, w.transport_block)
    plan.close()
    ok = [w.tb_crc_ok for w in want]
    assert all(ok) if offset_db > 0 else not all(ok)
