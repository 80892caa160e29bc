"""One context per thread: contexts created by several threads at the same time decode as one created alone."""
import threading

import numpy as np
import pytest

from pusch_b200 import _native, sim
from pusch_b200.ldpc import LdpcBatchDecoder

pytestmark = pytest.mark.gpu


def test_contexts_created_at_the_same_time():
    jobs = [j for z in (6, 64, 384) for j in sim.ldpc_batch(seed=z, n=8, z=z, ebn0_range=(1.0, 4.0)).jobs]
    n = 6
    gate, got, errors = threading.Barrier(n), [None] * n, []

    def work(t):
        try:
            gate.wait()
            ctx = _native.Context(max_codeblocks=64)
            got[t] = LdpcBatchDecoder(context=ctx).decode_batch(jobs)
            ctx.close()
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(n)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    ctx = _native.Context(max_codeblocks=64)
    want = LdpcBatchDecoder(context=ctx).decode_batch(jobs)
    ctx.close()
    assert (want[1] > 0).any()
    for bits, it in got:
        assert np.array_equal(it, want[1])
        assert all(np.array_equal(a, b) for a, b in zip(bits, want[0]))
