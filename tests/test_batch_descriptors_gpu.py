"""Descriptors of batched calls that travel with the launches (pg_rate_dematch_batch_device,
pg_ldpc_decode_batch_device): batches at and beyond each size that a launch takes, so that the staged path runs
too, give each codeblock what a batch of its own gives it, and calls on two streams of one context follow one
another."""
import ctypes

import numpy as np
import pytest

from pusch_b200 import _native, sim
from pusch_b200.ldpc import LdpcBatchDecoder, make_descriptors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 335, 336, 670, 671, 1340, 1341])
def test_rate_dematch_batches(n):
    import torch
    ctx = _native.Context(max_codeblocks=2048)
    rng = np.random.default_rng(n)
    z, e = 2, 96
    descs = (_native.PgRmCb * n)()
    for i, d in enumerate(descs):
        d.in_offset, d.rm_length, d.out_offset, d.nref = e * i, e, 132 * i, 0
        d.lifting_size, d.nof_filler_bits, d.base_graph = z, i % 7, 1
        d.rv, d.modulation_order, d.new_data = i % 4, (2, 4, 6, 8)[i % 4], i % 2
    llr = torch.from_numpy(rng.integers(-120, 121, n * e).astype(np.int8)).cuda()
    prev = torch.from_numpy(rng.integers(-120, 121, n * 132).astype(np.int8)).cuda()
    whole, single = prev.clone(), prev.clone()
    s = torch.cuda.current_stream().cuda_stream
    lib = ctx.lib
    ctx.check(lib.pg_rate_dematch_batch_device(ctx.handle, ctypes.addressof(descs), n, llr.data_ptr(), whole.data_ptr(), s))
    size = ctypes.sizeof(_native.PgRmCb)
    for i in sorted({0, n // 2, n - 1} | set(range(0, n, 97))):
        ctx.check(lib.pg_rate_dematch_batch_device(ctx.handle, ctypes.addressof(descs) + size * i, 1, llr.data_ptr(),
                                                   single.data_ptr(), s))
        torch.cuda.synchronize()
        assert torch.equal(whole[132 * i:132 * i + 132], single[132 * i:132 * i + 132]), i


@pytest.mark.parametrize("n", [260, 261, 400, 401, 800, 801, 1600, 1601])
def test_ldpc_batches(n):
    import torch
    ctx = _native.Context(max_codeblocks=2048)
    base = sim.ldpc_batch(seed=n, n=24, z=16, ebn0_range=(1.0, 4.0), bgs=np.array([1, 2] * 12, np.int32), max_iterations=4)
    jobs = [base.jobs[i % 24] for i in range(n)]
    dec = LdpcBatchDecoder(context=ctx)

    def run(js, stream):
        descs, llrs, nbits = make_descriptors(js)
        d_llr = torch.from_numpy(llrs).cuda()
        bits = torch.zeros(nbits, dtype=torch.uint8, device="cuda")
        it = torch.full((len(js),), -7, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        dec.decode_device(descs, len(js), d_llr.data_ptr(), bits.data_ptr(), it.data_ptr(), stream.cuda_stream)
        return d_llr, bits, it

    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    a, b, c = run(jobs, s1), run(base.jobs, s2), run(jobs, s2)
    torch.cuda.synchronize()
    reps = -(-n // 24)
    want = b[2].repeat(reps)[:n]
    assert (b[2] >= 0).all()
    assert torch.equal(a[2], want) and torch.equal(c[2], want)
    assert torch.equal(a[1], c[1])
    bits24 = b[1]
    m = min(bits24.numel(), a[1].numel())
    assert torch.equal(a[1][:m], bits24[:m])
