"""Calls that share a context's decoder scratch follow one another on the device, whichever entry and stream they
come through: an asynchronous batch decode, a decode of resident descriptors on another stream and a
transport-block decode (the context's own stream) issued one after the other without a host wait give what each of
them gives alone."""
import numpy as np
import pytest

from pusch_b200 import _native, sim
from pusch_b200.ldpc import LdpcBatchDecoder, make_descriptors
from pusch_b200.sch import PuschDecoder, SchTransportBlock
from test_sch_gpu import make_tb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [_native.PG_LDPC_ORDER_LONGEST_FIRST, _native.PG_LDPC_ORDER_GIVEN])
def test_calls_on_several_streams(order):
    import torch
    ctx = _native.Context(max_codeblocks=1024)
    dec = LdpcBatchDecoder(context=ctx)
    dec.set_order(order)
    big = sim.ldpc_batch(seed=41, n=600, z=384, ebn0_range=(1.0, 3.0)).jobs      # ordered, two CTAs per SM
    small = sim.ldpc_batch(seed=42, n=330, z=64, ebn0_range=(1.0, 4.0)).jobs
    rng = np.random.default_rng(43)
    tbs = [SchTransportBlock(make_tb(rng, 12040, 1, 4, 1, 5000, snr_db=6.0)[1], 12040, 1, 4, 1) for _ in range(12)]
    tbs = 15 * tbs  # two codeblocks each: ordered
    streams = [torch.cuda.Stream() for _ in range(3)]
    buf = []
    for jobs in (big, small):
        descs, llrs, nbytes = make_descriptors(jobs)
        buf.append((descs, torch.from_numpy(np.frombuffer(bytes(descs), np.uint8).copy()).cuda(),
                    torch.from_numpy(llrs).cuda(), len(jobs), nbytes))

    def outputs(b):
        return (torch.zeros(b[4], dtype=torch.uint8, device="cuda"), torch.full((b[3],), -7, dtype=torch.int32, device="cuda"))

    def device(b, out, s):
        dec.decode_device(b[0], b[3], b[2].data_ptr(), out[0].data_ptr(), out[1].data_ptr(), s.cuda_stream)

    def resident(b, out, s):
        dec.decode_resident(b[1].data_ptr(), b[3], b[2].data_ptr(), out[0].data_ptr(), out[1].data_ptr(), s.cuda_stream)

    want = []
    for b in buf:
        o = outputs(b)
        torch.cuda.synchronize()
        device(b, o, streams[0])
        torch.cuda.synchronize()
        want.append([t.cpu() for t in o])
    sch = PuschDecoder(ctx)
    want_tb = sch.decode_batch(tbs)
    assert any(t.tb_crc_ok for t in want_tb)
    for _ in range(5):
        outs = [outputs(buf[i]) for i in (0, 1, 0, 1)]
        torch.cuda.synchronize()
        device(buf[0], outs[0], streams[0])
        resident(buf[1], outs[1], streams[1])
        resident(buf[0], outs[2], streams[2])
        got_tb = sch.decode_batch(tbs)
        device(buf[1], outs[3], streams[0])
        torch.cuda.synchronize()
        for o, i in zip(outs, (0, 1, 0, 1)):
            assert torch.equal(o[1].cpu(), want[i][1]) and torch.equal(o[0].cpu(), want[i][0])
        for g, w in zip(got_tb, want_tb):
            assert (g.tb_crc_ok, g.nof_codeblocks_crc_ok, g.mean_iterations) == (
                w.tb_crc_ok, w.nof_codeblocks_crc_ok, w.mean_iterations)
    ctx.close()
