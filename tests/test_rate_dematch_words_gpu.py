"""Rate dematching by aligned words of four positions: every byte alignment of the buffer, E at the edges of
the valid positions (none left over, one short, one column more), repetition of several rounds, tiles of the
de-interleaver with a remainder, N_ref, fillers, and soft combining, against the rule restated position by
position: LLR t of the de-interleaved order is summed onto the t-th valid position of the circular buffer from
k0, onto 0 or the previous content, whatever its int8 value (equal bytes, and nothing written outside the
buffer)."""
import ctypes

import numpy as np
import pytest

from pusch_b200 import _native

pytestmark = pytest.mark.gpu


def llr_sum(a, b):
    s = np.clip(a + b, -120, 120)
    s = np.where(np.abs(b) == 127, b, s)
    s = np.where(np.abs(a) == 127, a, s)
    return np.where(a == -b, 0, s)


def dematch(bg, z, llr, rv, qm, nref, f, nd, prev):
    n, sys_ = (66 if bg == 1 else 50) * z, (20 if bg == 1 else 8) * z
    ncb = nref if 0 < nref < n else n
    k0 = ([0, 17, 33, 56] if bg == 1 else [0, 13, 25, 43])[rv] * ncb // n * z
    valid = np.concatenate([np.arange(sys_ - f), np.arange(sys_, ncb)])
    order = np.roll(valid, -int(np.searchsorted(valid, k0)))
    x = llr.astype(int).reshape(-1, qm).T.ravel()  # out[K j + i] = in[i Qm + j]
    out = np.zeros(n, int) if nd else prev.astype(int)
    for t in range(0, x.size, order.size):
        p = order[:x.size - t]
        out[p] = llr_sum(out[p], x[t:t + p.size])
    out[sys_ - f:sys_] = 127
    return out.astype(np.int8)


@pytest.mark.parametrize("bg,z", [(1, 2), (2, 7), (1, 15), (2, 104), (1, 384)])
def test_rate_dematch_every_alignment(ctx, bg, z):
    import torch
    rng = np.random.default_rng(z)
    n, k = (66 if bg == 1 else 50) * z, (22 if bg == 1 else 10) * z
    cases = []
    for t in range(40):
        qm = [1, 2, 4, 6, 8][t % 5]
        f = [0, (k - 2 * z) // 3, k - 2 * z - 1][t % 3]
        nref = [0, int(rng.integers(k - 2 * z + 1, n + 1))][t % 2]
        v = (nref if 0 < nref < n else n) - f
        e = [qm, v // qm * qm, max(qm, v // qm * qm - qm), v // qm * qm + qm, 5 * v // qm * qm,
             qm * int(rng.integers(1, max(2, v // qm)))][t % 6]
        cases.append((qm, f, nref, e, int(rng.integers(0, 4)), bool(rng.integers(0, 2)), t % 4))
    descs = (_native.PgRmCb * len(cases))()
    llrs, out, want, off_in, off_out = [], [], [], 0, 0
    for d, (qm, f, nref, e, rv, nd, mis) in zip(descs, cases):
        llr = rng.integers(-127, 128, e).astype(np.int8)
        prev = rng.integers(-127, 128, n).astype(np.int8)
        pad = 4 + (mis - off_out) % 4
        off_out += pad
        d.in_offset, d.out_offset, d.rm_length, d.nref = off_in, off_out, e, nref
        d.nof_filler_bits, d.lifting_size, d.base_graph, d.rv = f, z, bg, rv
        d.modulation_order, d.new_data = qm, int(nd)
        off_in += e
        off_out += n
        llrs.append(llr)
        out += [np.full(pad, 99, np.int8), prev]
        want += [np.full(pad, 99, np.int8),
                 dematch(bg, z, llr, rv, qm, nref, f, nd, prev)]
    d_in = torch.from_numpy(np.concatenate(llrs)).cuda()
    d_out = torch.from_numpy(np.concatenate(out + [np.full(8, 99, np.int8)])).cuda()
    st = torch.cuda.current_stream()
    ctx.check(ctx.lib.pg_rate_dematch_batch_device(ctx.handle, ctypes.addressof(descs), len(cases), d_in.data_ptr(),
                                                   d_out.data_ptr(), st.cuda_stream))
    st.synchronize()
    assert np.array_equal(d_out.cpu().numpy(), np.concatenate(want + [np.full(8, 99, np.int8)]))
