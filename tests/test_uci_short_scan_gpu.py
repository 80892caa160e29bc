"""The short-block detector scans a message's soft bits in batches of a size that depends on their number: on both
sides of that line and around the batches' ends, the decision on a stream equals that on the stream folded
beforehand (3 to 11 bits), and one or two bits decode alike with zeros in every other place."""
import numpy as np
import pytest

from test_uci_decoders_gpu import fold32
from test_uci_gpu import detect_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E", [33, 64, 96, 97, 127, 128, 129, 160, 1025])
def test_both_scans(ctx, E):
    rng = np.random.default_rng(E)
    cases, want = [], []
    for K in range(3, 12):
        for lim in (1, 20, 127):
            llr = rng.choice([-lim, -1, 1, lim], E).astype(np.int8)
            if np.count_nonzero(fold32(llr)) >= 17:
                cases.append((K, 2, llr))
                want.append((K, 2, fold32(llr)))
    got, ref = detect_gpu(ctx, cases), detect_gpu(ctx, want)
    assert len(cases) >= 9
    for (gb, gok), (rb, rok), c in zip(got, ref, cases):
        assert gok == rok and np.array_equal(gb, rb), (c[0], E)
    # The span check counts non-zero soft bits: one below its threshold is refused, at it accepted.
    for K, need in ((1, 2), (2, 3), (3, 9), (11, 17)):
        for n in (need - 1, need):
            llr = np.zeros(E, np.int8)
            llr[np.linspace(0, E - 1, n).astype(int)] = 50
            (_, ok), = detect_gpu(ctx, [(K, 2, llr)])
            if n < need:
                assert not ok, (K, E)
