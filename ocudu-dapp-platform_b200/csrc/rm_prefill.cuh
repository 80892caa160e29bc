// Device code that a slot plan's estimation launch runs for the rate dematcher.
#pragma once

#include "pg_internal.h"

namespace pg {

// The circular buffers of the codeblocks whose LLRs the demodulator stores in place (placed[c]
// = 1: new data, E <= V), before it does: +127 at the filler positions [inf, (Kb - 2) Z) and 0
// everywhere else, which is what rate dematching leaves at every position that no LLR reaches.
// 16-byte stores; the first and last bytes of a buffer that does not start or end on a 16-byte
// boundary are stored one by one. Also zeroes the TB buffer (bytes between the TBs stay zero), the decoders'
// work counter, the arrivals of their ordering launch, and the CRC and arrival words of the TB join. CTA `cta` of kRmFillCtas * n, NT threads each.
template <int NT>
__device__ __forceinline__ void rm_prefill(const rm_fill& f, const int cta)
{
  {
    const size_t nthr = (size_t)kRmFillCtas * f.n * NT;
    const size_t t0   = (size_t)cta * NT + threadIdx.x;
    const size_t head = min(f.tb_bytes, (size_t)((16u - (unsigned)(reinterpret_cast<uintptr_t>(f.tb_out) & 15u)) & 15u));
    const size_t nvec = (f.tb_bytes - head) / 16;
    uint4*       v    = reinterpret_cast<uint4*>(f.tb_out + head);
    for (size_t q = t0; q < nvec; q += nthr) {
      v[q] = make_uint4(0u, 0u, 0u, 0u);
    }
    if (t0 < head) {
      f.tb_out[t0] = 0;
    }
    if (head + 16 * nvec + t0 < f.tb_bytes) {
      f.tb_out[head + 16 * nvec + t0] = 0;
    }
    if (t0 < 2) {
      f.counters[t0] = 0;
    }
    for (size_t q = t0; q < (size_t)f.njoin; q += nthr) {
      f.join[q] = 0u;
    }
  }
  const int c = cta / kRmFillCtas;
  if (f.placed[c] == 0) {
    return;
  }
  const pg_rm_cb d    = f.cbs[c];
  const int      Z    = d.lifting_size;
  const int      N    = (d.base_graph == 1 ? 66 : 50) * Z;
  const int      sys  = ((d.base_graph == 1 ? 22 : 10) - 2) * Z;
  const int      inf  = sys - (int)d.nof_filler_bits;
  int8_t*        out  = f.out + d.out_offset;
  const int      head = min(N, (int)((16u - (unsigned)(reinterpret_cast<uintptr_t>(out) & 15u)) & 15u));
  const int      nch  = (N - head) / 16;
  const int      tail = head + 16 * nch;
  const int      tid  = cta % kRmFillCtas * NT + threadIdx.x;
  const int      nthr = kRmFillCtas * NT;
  auto value = [&](int p) { return (int8_t)((p >= inf && p < sys) ? 127 : 0); };
  if (tid < head) {
    out[tid] = value(tid);
  }
  if (tail + tid < N) {
    out[tail + tid] = value(tail + tid);
  }
  for (int q = tid; q < nch; q += nthr) {
    const int p0  = head + 16 * q;
    const int fil = max(0, min(p0 + 16, sys) - max(p0, inf));
    uint4     w   = make_uint4(0u, 0u, 0u, 0u);
    if (fil == 16) {
      w = make_uint4(0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu);
    } else if (fil > 0) {
      int8_t* b = reinterpret_cast<int8_t*>(&w);
      for (int i = 0; i < 16; ++i) {
        b[i] = value(p0 + i);
      }
    }
    *reinterpret_cast<uint4*>(out + p0) = w;
  }
}

} // namespace pg
