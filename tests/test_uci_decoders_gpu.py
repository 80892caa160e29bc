"""The UCI decoders' paths that depend on where and how long a message's soft bits are: the polar decoder
over every N it reaches (32 to 1024), one and two codeblocks, streams at every byte alignment and soft bits
of every int8 value from -127 to 127, against the CPU restatement of the decoding (polar_oracle); and
the short-block detector's folding of a long stream against its decision on the stream folded beforehand.
Both are integer computations: bits and validity are equal."""
import numpy as np
import pytest

import polar_oracle
from pusch_b200 import uci
from test_uci_gpu import detect_gpu

pytestmark = pytest.mark.gpu

# (A, E): N = 32 to 1024, shortening, puncturing, repetition to eight times and more, E at both sides of a
# triangle number (entries missing from the channel interleaver's last columns), two codeblocks.
POLAR = [(12, 24), (12, 31), (12, 36), (12, 37), (12, 55), (13, 56), (19, 300), (20, 64), (24, 8191), (40, 170),
         (64, 150), (100, 400), (200, 1024), (60, 8192), (359, 1500), (361, 2001), (1013, 1600), (1706, 8000)]


def test_polar_decoder_over_lengths_and_alignments(ctx):
    rng = np.random.default_rng(5)
    msgs = []
    for t, (A, E) in enumerate(POLAR):
        lim = (127, 20, 3)[t % 3]
        llr = rng.integers(-lim, lim + 1, E).astype(np.int8)
        llr[rng.random(E) < 0.1] = 0
        msgs.append((A, llr))
        msgs.append((A, np.abs(llr)))  # the all-zero codeword: a valid CRC
    got = uci.PolarUciDecoder(ctx).decode(msgs)
    nvalid = 0
    for (A, llr), (bits, ok) in zip(msgs, got):
        want, want_ok = polar_oracle.uci_polar_decode(A, llr, uci.polar_code)
        assert ok == want_ok, (A, llr.size)
        assert np.array_equal(bits, want), (A, llr.size)
        nvalid += ok
    assert nvalid >= len(POLAR) // 2


def fold32(llr):
    out = llr[:32].astype(int)
    for i in range(32, llr.size):
        out[i % 32] = max(-120, min(120, out[i % 32] + int(llr[i])))
    return out.astype(np.int8)


@pytest.mark.parametrize("E", [32, 33, 63, 1023, 1024, 1025, 2100])
def test_short_block_folds_long_streams(ctx, E):
    rng = np.random.default_rng(E)
    cases, want = [], []
    for K in range(3, 12):
        for lim in (1, 127):
            llr = rng.choice([-lim, -1, 1, lim], E).astype(np.int8)
            cases.append((K, 2, llr))
            want.append((K, 2, fold32(llr)))
    # The folded stream keeps enough nonzero soft bits for the detector's span check, or is left out.
    keep = [i for i, (K, _, f) in enumerate(want) if np.count_nonzero(f) >= 17]
    got, ref = detect_gpu(ctx, [cases[i] for i in keep]), detect_gpu(ctx, [want[i] for i in keep])
    assert len(keep) >= 9
    for i, (gb, gok), (rb, rok) in zip(keep, got, ref):
        assert gok == rok and np.array_equal(gb, rb), (cases[i][0], E)
