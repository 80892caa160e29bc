"""Kernels of a slot plan that start before the kernel ahead of them ends read that kernel's output coherently: a
plan whose UEs partly combine (rate dematching reads and writes the soft buffers that the decoder reads next) runs
transmission after transmission with no host wait in between, and every execution's results and TB bytes equal the
CPU chain's over the same LLRs. Small plans take one decoder CTA per SM, which is the shape that starts early."""
import ctypes

import numpy as np
import pytest

from pusch_b200 import _native, sim
from pusch_b200.pusch import PuschSlotPlan, results_from
from test_harq_gpu import device_llrs, oracle_receive, retransmission

pytestmark = pytest.mark.gpu

TRANSMISSIONS = 8  # combined ones, after the first


@pytest.mark.parametrize("seed", [31, 32])
def test_combining_executions_back_to_back(ctx, port, seed):
    import torch
    first = sim.uneven_cells(seed=seed, nof_cells=2, max_ues=6)
    ues = [ue for sl in first for ue in sl.ues]
    n = len(ues)
    combine = [u % 3 != 2 for u in range(n)]

    def again(k):
        out, u0 = [], 0
        for c, sl in enumerate(first):
            out.append(retransmission(sl, combine[u0:u0 + len(sl.ues)], 1000 * seed + 10 * k + c))
            u0 += len(sl.ues)
        return out

    sent = [first] + [again(k) for k in range(TRANSMISSIONS)]
    plan = PuschSlotPlan(ctx, first, max_iterations=6)
    words = [np.concatenate([np.ascontiguousarray(sl.grid, np.uint32).ravel() for sl in s]) for s in sent]
    grids = [torch.from_numpy(w.view(np.int32)).cuda() for w in words]
    size = ctypes.sizeof(_native.PgSchResult)
    tbs = [torch.zeros(max(plan.tb_bytes, 1), dtype=torch.uint8, device="cuda") for _ in sent]
    res = [torch.zeros(n * size, dtype=torch.uint8, device="cuda") for _ in sent]
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    plan.execute_device(grids[0].data_ptr(), tbs[0].data_ptr(), res[0].data_ptr(), stream_ptr=s.cuda_stream)
    s.synchronize()
    plan.set_harq(new_data=[not c for c in combine], rv=[2 if c else 0 for c in combine])
    for k in range(1, len(sent)):
        plan.execute_device(grids[k].data_ptr(), tbs[k].data_ptr(), res[k].data_ptr(), stream_ptr=s.cuda_stream)
    torch.cuda.synchronize()
    got = [results_from(plan.descs, (_native.PgSchResult * n).from_buffer_copy(r.cpu().numpy().tobytes()), None,
                        t.cpu().numpy()) for r, t in zip(res, tbs)]
    soft = [None] * n
    for k, slots in enumerate(sent):
        llrs = [x for sl in slots for x in device_llrs(ctx, sl)]
        for u in range(n):
            comb = k > 0 and combine[u]
            buf, ok, nok, bits = oracle_receive(port, ues[u], llrs[u], 2 if comb else 0, soft[u] if comb else None, 6)
            soft[u] = buf
            assert (got[k][u].tb_crc_ok, got[k][u].nof_codeblocks_crc_ok) == (ok, nok), (k, u)
            if ok:
                assert np.array_equal(np.unpackbits(got[k][u].transport_block), bits), (k, u)
    assert any(g.tb_crc_ok for g in got[-1])
    plan.close()
