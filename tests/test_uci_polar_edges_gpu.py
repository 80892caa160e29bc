"""The polar decoder's copy of a message's soft bits, taken by aligned words with the first and last ones by bytes:
every alignment of the stream's start and end, the stream ending where the buffer ends, against the CPU restatement
of the decoding (integers: equal)."""
import numpy as np
import pytest

import polar_oracle
from pusch_b200 import uci

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("start", range(4))
def test_first_and_last_soft_bits(ctx, start):
    rng = np.random.default_rng(start)
    dec, nvalid = uci.PolarUciDecoder(ctx), 0
    for A, E in [(12, e) for e in range(24, 32)] + [(40, 511), (40, 512), (40, 513), (40, 514), (361, 2001)]:
        lead = rng.integers(-20, 21, 24 + start).astype(np.int8)
        llr = rng.integers(-20, 21, E).astype(np.int8)
        for x in (llr, np.abs(llr)):
            bits, ok = dec.decode([(12, lead), (A, x)])[1]
            want, want_ok = polar_oracle.uci_polar_decode(A, x, uci.polar_code)
            assert ok == want_ok and np.array_equal(bits, want), (A, E)
            nvalid += ok
    assert nvalid >= 8
