"""A plan's tuning is what the plan runs: read and set again it changes nothing, for plans on both sides of 1.75
codeblocks per SM."""
import pytest

from pusch_b200 import _native, mcs, sim
from pusch_b200.pusch import PgPuschPlanInfo, PuschSlotPlan

pytestmark = pytest.mark.gpu


def nof_kernels(plan):
    info = PgPuschPlanInfo()
    plan.ctx.check(plan.lib.pg_pusch_plan_info(plan.handle, _native.ctypes.byref(info)))
    return info.nof_kernels


@pytest.mark.parametrize("cells,ctas", [(1, 1), (4, 1), (6, 2)])  # 51, 204 and 306 codeblocks
def test_read_and_set_again(ctx, cells, ctas):
    ues, rb = [], 0
    for u, (n, layers, index) in enumerate([(6, 1, 3), (40, 1, 12), (220, 2, 26)]):
        qm, r = mcs.MCS_TABLE_2[index]
        snr = sim.required_snr_db(qm, r, layers, 4) + 3.0
        ues.append(sim.ue_from_mcs(rb, n, layers, 2, index, (2, 11), snr_db=snr, channel="pdp", rnti=0x4100 + u))
        rb += n
    plan = PuschSlotPlan(ctx, [sim.make_pusch_slot(ues, 4, seed=9)] * cells)
    t, kernels = plan.tuning(), nof_kernels(plan)
    assert (t.ldpc_ctas_per_sm, t.ldpc_order) == (ctas, 0)
    plan.set_tuning(t)
    assert plan.tuning().as_dict() == t.as_dict() and nof_kernels(plan) == kernels
    plan.close()
