"""Lane-pair LDPC decoder (csrc/ldpc_decoder.cu): every lifting size of both base graphs against the CPU
restatement, with whole and ragged inputs. A ragged tail keeps LLRs that whole nodes clamp: values of
121 to 126 are finite in the first iteration, +-127 infinite. Few codeblocks keep their messages in
shared memory, many in the global slabs: both are taken."""
import numpy as np
import pytest

import golden_io
from pusch_b200 import codec
from pusch_b200.ldpc import CodeblockJob, LdpcDecoderConfiguration

pytestmark = pytest.mark.gpu


def make_job(rng, bg, z, ragged):
    k = golden_io.kbits(bg, z)
    nn = (66 if bg == 1 else 50) * z
    poly = int(rng.choice([1, 2, 255])) if k > 40 else 255
    cw = codec.ldpc_encode(bg, z, codec.attach_crc(1, rng.integers(0, 2, k - 24, dtype=np.uint8)) if k > 40
                           else rng.integers(0, 2, k, dtype=np.uint8))
    sigma = 10 ** (-rng.uniform(0.0, 6.0) / 20)
    llr = np.clip(np.rint((1 - 2.0 * cw + sigma * rng.standard_normal(nn)) * 8 / sigma ** 2), -127, 127).astype(np.int8)
    n = nn
    if ragged and z > 1:
        n = k + 2 * z + int(rng.integers(1, nn - k - 2 * z))
        n += n % z == 0
        n = min(n, nn - 1)
        tail = np.arange(n // z * z, n)
        llr[tail] = rng.choice([121, 122, 125, 126, 127, -121, -124, -126, -127, 3, -7, 0, 120], tail.size)
        llr[n - 1] = 126
    return CodeblockJob(llr[:n].copy(), LdpcDecoderConfiguration(bg, z, 0, 24, int(rng.integers(1, 6))), poly)


@pytest.mark.parametrize("copies", [1, 4])
def test_every_lifting_size_bit_exact(batch_decoder, port, copies):
    rng = np.random.default_rng(2024 + copies)
    jobs = [make_job(rng, bg, z, ragged) for z in codec.LIFTING_SIZES for bg in (1, 2) for ragged in (False, True)]
    outs, iters = batch_decoder.decode_batch(jobs * copies)
    for i, j in enumerate(jobs):
        c = j.cfg
        want_it, want = port.ldpc_decode(c.base_graph, c.lifting_size, j.llrs, filler=0,
                                         crc_poly=-1 if j.crc_poly == 255 else j.crc_poly, max_iter=c.max_iterations)
        k = golden_io.kbits(c.base_graph, c.lifting_size)
        for q in range(copies):
            o, it = outs[i + q * len(jobs)], iters[i + q * len(jobs)]
            assert it == want_it, (c, j.llrs.size, j.crc_poly)
            assert (np.unpackbits(o)[:k] == np.unpackbits(np.asarray(want, np.uint8))[:k]).all(), (c, j.llrs.size)
