// Batched LDPC rate dematching (TS 38.212 Section 5.4.2), bit-exact with the reference's
// ldpc_rate_dematcher (lib/phy/upper/channel_coding/ldpc/ldpc_rate_dematcher_impl.cpp:29-250) on
// finite LLRs.
//
// The reference walks the E received LLRs sequentially through the circular buffer: bit
// de-interleaving (out[K*j + i] = in[i*Qm + j]), then placement from k0 onward, skipping the
// filler positions, wrapping at N_cb and combining wrapped values with the saturating LLR sum.
// Here every output position is computed independently: the valid (non-filler) positions form a
// cycle of length V = N_cb - F; position p with valid index v receives the de-interleaved inputs
// t = (v - v0) mod V, t + V, t + 2V, ... < E, summed in that order onto 0 (new data) or onto the
// previous buffer content (soft combining). Filler positions hold +127; positions at or beyond N_cb
// are zeroed on new data and untouched otherwise.
#include "pg_internal.h"
#include "pg_device.cuh"

#include <algorithm>
#include <cstring>

namespace {

constexpr int kRmThreads = 256;

__device__ __forceinline__ int llr_sum(int a, int b)
{
  // log_likelihood_ratio::operator+ (lib/phy/upper/log_likelihood_ratio.cpp:21-53).
  if (a == -b) {
    return 0;
  }
  if (a == 127 || a == -127) {
    return a;
  }
  if (b == 127 || b == -127) {
    return b;
  }
  return max(-120, min(120, a + b));
}

constexpr int kRmRepBatch = 4;   // repetitions whose loads a thread issues together

// One codeblock's buffer, and the store of one aligned word of it (positions 4 g - mis ..). EARLY: the kernel
// may have started before the one that writes the LLRs ended.
template <bool EARLY>
struct rm_buffer {
  int8_t*       out;
  const int8_t* in;
  int           mis, N, Ncb, inf, sys, F, V, v0, E, Qm, Kq;
  float         inv_kq;
  bool          nd;

  __device__ __forceinline__ static int llr(const int8_t* p)
  {
    return EARLY ? pg::load_written(p) : (int)__ldg(p);
  }

  // LLR t of the de-interleaved order is at row t mod Kq, column t div Kq; the quotient comes from a float
  // reciprocal, corrected to the exact value (t < 2^24).
  __device__ __forceinline__ void split(int t, int& r, int& q) const
  {
    q = __float2int_rz((float)t * inv_kq);
    r = t - q * Kq;
    if (r < 0) {
      --q;
      r += Kq;
    } else if (r >= Kq) {
      ++q;
      r -= Kq;
    }
  }
  __device__ __forceinline__ int load(int t) const
  {
    int r, q;
    split(t, r, q);
    return llr(in + (r * Qm + q));
  }
  __device__ __forceinline__ static uint32_t pack(const int* x)
  {
    return __byte_perm(__byte_perm((uint32_t)x[0], (uint32_t)x[1], 0x0040),
                       __byte_perm((uint32_t)x[2], (uint32_t)x[3], 0x0040), 0x5410);
  }

  // Without repetition most words hold four LLRs of one column, or none: these take a quarter of the
  // instructions. Returns false for any other word.
  __device__ __forceinline__ bool plain_word(int g) const
  {
    const int p0 = 4 * g - mis;
    if (p0 < 0 || p0 + 4 > Ncb || (p0 + 3 >= inf && p0 < sys)) {
      return false;
    }
    int t = (p0 < inf ? p0 : p0 - F) - v0;
    t += t < 0 ? V : 0;
    uint32_t* const o = reinterpret_cast<uint32_t*>(out + p0);
    if (t >= E && t + 3 < V) {
      if (nd) {
        *o = 0u;
      }
      return true;
    }
    int r, q;
    split(t, r, q);
    if (t + 3 >= E || r + 3 >= Kq) {
      return false;
    }
    const int8_t* const f = in + (r * Qm + q);
    int                 x[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      x[j] = llr(f + j * Qm);
    }
    if (nd) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        x[j] = llr_sum(0, x[j]);
      }
    } else {
      const uint32_t old = *o;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        x[j] = llr_sum((int)(int8_t)(old >> (8 * j)), x[j]);
      }
    }
    *o = pack(x);
    return true;
  }

  // Any word: its LLRs are loaded together and summed in order onto 0 or the previous content.
  template <bool REP>
  __device__ __forceinline__ void word(int g) const
  {
    const int  p0    = 4 * g - mis;
    const bool whole = p0 >= 0 && p0 + 4 <= N;
    uint32_t   old   = 0;
    if (!nd) {
      if (whole) {
        old = *reinterpret_cast<const uint32_t*>(out + p0);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (p0 + j >= 0 && p0 + j < N) {
            old |= (uint32_t)(uint8_t)out[p0 + j] << (8 * j);
          }
        }
      }
    }
    int acc[4], t[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int p = p0 + j;
      acc[j]      = (int)(int8_t)(old >> (8 * j));
      t[j]        = E; // no LLR reaches the position
      if (p >= inf && p < sys) {
        acc[j] = 127;
      } else if (p >= 0 && p < Ncb) {
        const int x = (p < inf ? p : p - F) - v0;
        t[j]        = x < 0 ? x + V : x;
      }
    }
    if (!REP) {
      int x[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        x[j] = t[j] < E ? load(t[j]) : 0;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (t[j] < E) {
          acc[j] = llr_sum(acc[j], x[j]);
        }
      }
    } else {
      // Position p receives t, t + V, ... in that order; four repetitions' loads are issued together.
      for (int r = 0; r < E; r += kRmRepBatch * V) {
        int x[4][kRmRepBatch];
#pragma unroll
        for (int u = 0; u < kRmRepBatch; ++u) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int tu = t[j] + r + u * V;
            x[j][u]      = t[j] < E && tu < E ? load(tu) : 0;
          }
        }
#pragma unroll
        for (int u = 0; u < kRmRepBatch; ++u) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (t[j] < E && t[j] + r + u * V < E) {
              acc[j] = llr_sum(acc[j], x[j][u]);
            }
          }
        }
      }
    }
    if (whole) {
      *reinterpret_cast<uint32_t*>(out + p0) = pack(acc);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (p0 + j >= 0 && p0 + j < N) {
          out[p0 + j] = (int8_t)acc[j];
        }
      }
    }
  }
};

// Each aligned word of four positions is written once, by the thread that loads its LLRs; nothing waits on a
// barrier. Bound: instructions, and the latency of descriptor, LLRs and store. 200 codeblocks of up to 25,344
// positions: 7.0 us on new data, 8.7 us combining (12 us each as tiles of the input transposed through shared
// memory with a second pass over the positions no LLR reaches; 10 us with every word taken the general way;
// 12 us with the words ordered so that one CTA reads each input sector).
template <bool EARLY>
__device__ __forceinline__ void rate_dematch(const pg_rm_cb& d, const int8_t* __restrict__ in_all, int8_t* __restrict__ out_all)
{
  const int      bg = d.base_graph;
  const int      Z  = d.lifting_size;
  const int      Kb = bg == 1 ? 22 : 10;
  const int      sh = bg == 1 ? (d.rv == 0 ? 0 : d.rv == 1 ? 17 : d.rv == 2 ? 33 : 56)
                              : (d.rv == 0 ? 0 : d.rv == 1 ? 13 : d.rv == 2 ? 25 : 43);
  rm_buffer<EARLY> c;
  c.N            = (bg == 1 ? 66 : 50) * Z;
  c.Ncb          = (d.nref > 0 && d.nref < (uint32_t)c.N) ? (int)d.nref : c.N;
  c.F            = d.nof_filler_bits;
  c.sys          = (Kb - 2) * Z;
  c.inf          = c.sys - c.F;
  c.E            = (int)d.rm_length;
  c.Qm           = d.modulation_order;
  c.Kq           = c.E / c.Qm;
  c.inv_kq       = 1.0f / (float)max(1, c.Kq);
  c.V            = c.Ncb - c.F;
  c.in           = in_all + d.in_offset;
  c.out          = out_all + d.out_offset;
  c.nd           = d.new_data != 0;
  c.mis          = (int)(reinterpret_cast<uintptr_t>(c.out) & 3u);
  const int k0   = (sh * c.Ncb) / c.N * Z; // sh * Ncb < 2^21
  c.v0           = k0 < c.inf ? k0 : (k0 < c.sys ? c.inf : k0 - c.F);
  const int nw   = (c.N + c.mis + 3) >> 2;
  const int tid  = threadIdx.x;
  for (int g = blockIdx.y * kRmThreads + tid; g < nw; g += gridDim.y * kRmThreads) {
    if (c.E > c.V) {
      c.template word<true>(g);
    } else if (!c.plain_word(g)) {
      c.template word<false>(g);
    }
  }
}

__global__ void __launch_bounds__(kRmThreads) rate_dematch_kernel(const pg_rm_cb* __restrict__ cbs,
                                                                  const int8_t* __restrict__ in_all,
                                                                  int8_t* __restrict__ out_all,
                                                                  const uint32_t* __restrict__ list)
{
  pg::launch_dependents();
  const pg_rm_cb d = cbs[list != nullptr ? list[blockIdx.x] : blockIdx.x];
  pg::wait_prerequisites();
  rate_dematch<true>(d, in_all, out_all);
}

// The descriptors in the launch's arguments: a copy staged in pinned memory started the kernel 6 us later, and
// a second call waited on the host for the first one's kernel.
template <int N>
struct rm_args {
  pg_rm_cb cb[N];
};
static_assert(sizeof(rm_args<pg::kRmArgs>) <= 32700, "arguments of a launch");

template <int N>
__global__ void __launch_bounds__(kRmThreads) rate_dematch_args_kernel(const __grid_constant__ rm_args<N> args,
                                                                       const int8_t* __restrict__ in_all,
                                                                       int8_t* __restrict__ out_all)
{
  const pg_rm_cb d = args.cb[blockIdx.x];
  rate_dematch<false>(d, in_all, out_all);
}

} // namespace

namespace pg {

int validate_rm_descs(pg_context* ctx, const pg_rm_cb* cbs, int n, size_t in_total, size_t out_total)
{
  if (n < 0 || (n > 0 && cbs == nullptr)) {
    return set_error(ctx, PG_ERR_INVALID, "invalid codeblock list");
  }
  if (n > ctx->max_codeblocks) {
    return set_error(ctx, PG_ERR_CAPACITY, "rate-dematch batch exceeds max_codeblocks");
  }
  for (int i = 0; i < n; ++i) {
    const pg_rm_cb& d = cbs[i];
    char            buf[160];
    const int       qm = d.modulation_order;
    if ((d.base_graph != 1 && d.base_graph != 2) || lifting_set_index(d.lifting_size) < 0 || d.rv > 3 ||
        !(qm == 1 || qm == 2 || qm == 4 || qm == 6 || qm == 8)) {
      snprintf(buf, sizeof(buf), "codeblock %d: invalid base graph, lifting size, rv or modulation", i);
      return set_error(ctx, PG_ERR_INVALID, buf);
    }
    const int Z   = d.lifting_size;
    const int N   = nshort_of(d.base_graph) * Z;
    const int sys = (kb_of(d.base_graph) - 2) * Z;
    const int Ncb = (d.nref > 0 && (int)d.nref < N) ? (int)d.nref : N;
    if ((int)d.nof_filler_bits >= sys || Ncb <= sys) {
      snprintf(buf, sizeof(buf), "codeblock %d: filler bits or N_ref out of range", i);
      return set_error(ctx, PG_ERR_INVALID, buf);
    }
    if (d.rm_length % qm != 0) {
      snprintf(buf, sizeof(buf), "codeblock %d: E=%u not a multiple of Qm=%d", i, d.rm_length, qm);
      return set_error(ctx, PG_ERR_INVALID, buf);
    }
    if (in_total != 0 && (size_t)d.in_offset + d.rm_length > in_total) {
      snprintf(buf, sizeof(buf), "codeblock %d: input beyond the buffer", i);
      return set_error(ctx, PG_ERR_INVALID, buf);
    }
    if (out_total != 0 && (size_t)d.out_offset + (size_t)N > out_total) {
      snprintf(buf, sizeof(buf), "codeblock %d: output beyond the buffer", i);
      return set_error(ctx, PG_ERR_INVALID, buf);
    }
  }
  return PG_OK;
}

// CTAs per codeblock of a batch. A CTA's set-up is worth several words of its threads: five CTAs per SM shared
// among the codeblocks, at least four each. 200 codeblocks: 7.0 us at 4 CTAs each, 7.5 at 8, 8.3 at 13, 10.9 at
// 25 (one word a thread).
static int batch_ctas_per_cb(const pg_context* ctx, int n)
{
  return std::max(4, std::min(16, 5 * ctx->sm_count / std::max(1, n)));
}

int rate_dematch_launch(pg_context* ctx, const pg_rm_cb* descs_dev, int n, const int8_t* in, int8_t* out,
                        cudaStream_t stream)
{
  return rate_dematch_launch(ctx, descs_dev, n, in, out, stream, batch_ctas_per_cb(ctx, n));
}

template <int N>
static void launch_args(pg_context* ctx, const pg_rm_cb* descs, int n, const int8_t* in, int8_t* out, cudaStream_t stream)
{
  rm_args<N> args;
  std::memcpy(args.cb, descs, (size_t)n * sizeof(pg_rm_cb));
  rate_dematch_args_kernel<N><<<dim3(n, batch_ctas_per_cb(ctx, n)), kRmThreads, 0, stream>>>(args, in, out);
}

int rate_dematch_launch_args(pg_context* ctx, const pg_rm_cb* descs, int n, const int8_t* in, int8_t* out,
                             cudaStream_t stream)
{
  // A launch copies its arguments whole: four sizes. The smallest, 20 codeblocks, is for the usual small call: one
  // codeblock of 132 positions takes 9.5 us with it, 10.7 with the next (10.3 by a staged copy).
  if (n <= kRmArgs / 64) {
    launch_args<kRmArgs / 64>(ctx, descs, n, in, out, stream);
  } else if (n <= kRmArgs / 4) {
    launch_args<kRmArgs / 4>(ctx, descs, n, in, out, stream);
  } else if (n <= kRmArgs / 2) {
    launch_args<kRmArgs / 2>(ctx, descs, n, in, out, stream);
  } else {
    launch_args<kRmArgs>(ctx, descs, n, in, out, stream);
  }
  return check_cuda(ctx, cudaGetLastError(), "rate_dematch_args_kernel launch");
}

int rate_dematch_launch(pg_context* ctx, const pg_rm_cb* descs_dev, int n, const int8_t* in, int8_t* out,
                        cudaStream_t stream, int ctas_per_cb, const uint32_t* list, bool overlap)
{
  if (n == 0) {
    return PG_OK;
  }
  // Each codeblock's N <= 25,344 output positions spread over ctas_per_cb CTAs.
  ctas_per_cb = std::max(1, std::min(32, ctas_per_cb));
  if (overlap) {
    return check_cuda(ctx,
                      launch_overlapped(rate_dematch_kernel, dim3(n, ctas_per_cb), kRmThreads, 0, stream, descs_dev, in, out,
                                        list),
                      "rate_dematch_kernel launch");
  }
  rate_dematch_kernel<<<dim3(n, ctas_per_cb), kRmThreads, 0, stream>>>(descs_dev, in, out, list);
  return check_cuda(ctx, cudaGetLastError(), "rate_dematch_kernel launch");
}

} // namespace pg
