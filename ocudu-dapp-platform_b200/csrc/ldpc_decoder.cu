// Batched LDPC decoder for sm_100a: layered normalised min-sum on int8 messages, bit-exact with
// the reference's ldpc_decoder_avx512 / ldpc_decoder_avx2
// (lib/phy/upper/channel_coding/ldpc/ldpc_decoder_impl.cpp:41-306,
//  lib/phy/upper/channel_coding/ldpc/ldpc_decoder_avx512.cpp:69-253).
//
// Mapping: one CTA per codeblock at a time. For base-graph row r, edge e (variable node v_e, lifted shift
// s_e), check lane j (0 <= j < Z) reads soft bit (v_e, (j+s_e) mod Z): the rows of a layer touch every
// lifted variable lane exactly once, so the Z lanes of a row are independent and a barrier separates rows
// that share columns (the layer schedule). Soft bits live in shared memory; check-to-variable messages are
// indexed by (edge, check lane) rather than the reference's rotated-back (variable slot, variable lane):
// the stored values are identical. Two kernels:
// - ldpc_decode_pair_kernel ("Lane-pair decoder" below) runs the batch decodes and the slot plans: even
//   lifting sizes as pairs of lanes in f16x2, messages in shared memory or a global slab per CTA; the
//   odd ones (Z <= 15) with the one-lane code.
// - ldpc_decode_kernel, one thread per lane, messages in global memory (one byte per edge and lane, L2
//   resident): PG_LDPC_KERNEL_ONE_LANE and the static-scratch entry, whose fixed array has room for this
//   layout and not for the padded rows of the other.
//
// Arithmetic, per lane and edge (all exactly as the reference's AVX-512 kernels):
//   v2c = soft == +-127 ? soft : clamp(soft - c2v, -120, 120)
//   min1/min2 over |v2c| starting at 120 (first minimum wins), sign = xor of v2c signs
//   scale: m -> (m * 52428) >> 16     (floor(0.8 * 2^16) = 52428; m <= 120 always)
//   c2v  = (sign xor sign(v2c)) ? -mag : mag,  mag = |v2c| == min1 ? scale(min2) : scale(min1)
//          (equivalent to the reference's index test: a tie at min1 implies min1 == min2)
//   soft = |v2c| == 127 ? v2c : promote(c2v + v2c) with |sum| > 120 -> +-127
// After each iteration: hard bits (soft <= 0), fail if any soft bit is 0, else CRC over the
// K*Z - F significant bits; CRC == 0 stops with iterations = it + 1.
#include "pg_internal.h"
#include "pg_device.cuh"

#include <cuda_fp16.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <mutex>

namespace pg {
#include "ldpc_base_graphs.inc"
} // namespace pg

namespace {

constexpr int kThreads = 384;

__constant__ uint8_t  c_edge_col[2][pg::kBg1Edges];
__constant__ uint16_t c_edge_v[2][pg::kBg1Edges][8];
__constant__ uint8_t  c_row_deg[2][pg::kBg1Rows];
// Layer steps: runs of consecutive base-graph rows whose columns are pairwise disjoint. The rows of
// a step touch disjoint soft bits, so running them between the same two barriers gives exactly
// the results of the reference's one-row-at-a-time order (BG1: 46 rows in 32 steps, BG2: 42 in 28).
__constant__ uint8_t  c_step_row0[2][pg::kBg1Rows]; // first row of each step
__constant__ uint8_t  c_step_nrows[2][pg::kBg1Rows];
__constant__ uint8_t  c_nsteps[2];
__constant__ uint16_t c_row_e0[2][pg::kBg1Rows + 1]; // first edge of each row (prefix sums of the degrees)

__device__ __forceinline__ int dev_set_index(int Z)
{
  const int a_tab[8] = {2, 3, 5, 7, 9, 11, 13, 15};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    int t = Z;
    while ((t & 1) == 0 && t > a_tab[i]) {
      t >>= 1;
    }
    if (t == a_tab[i]) {
      return i;
    }
  }
  return -1;
}

// Steps of a codeblock that processes nof_layers rows: those whose first row is below nof_layers.
__device__ __forceinline__ int steps_for_layers(int g, int nof_layers)
{
  int n = 0;
  while (n < c_nsteps[g] && c_step_row0[g][n] < nof_layers) {
    ++n;
  }
  return n;
}

// Pulls the check-to-variable messages of step st (rows up to nof_layers) into L1 ahead of their
// use: one prefetch per 128-byte line, thread `tid` taking line tid. Message rows are
// row_bytes apart (one per edge) starting at base.
__device__ __forceinline__ void prefetch_step(const int g, const int st, const int nof_layers, const int tid,
                                              const char* base, const int row_bytes)
{
  const int r0    = c_step_row0[g][st];
  const int r1    = min(r0 + (int)c_step_nrows[g][st], nof_layers);
  const int ea    = c_row_e0[g][r0];
  const int lpe   = (row_bytes + 127) >> 7;
  const int lines = (c_row_e0[g][r1] - ea) * lpe;
  if (tid < lines) {
    const int e = tid / lpe;
    const char* p = base + (size_t)(ea + e) * row_bytes + ((tid - e * lpe) << 7);
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
  }
}

__device__ __forceinline__ int scale_mag(int m)
{
  return (m * 52428) >> 16;
}

__device__ __forceinline__ int warp_max(int v)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  }
  return v;
}

__device__ __forceinline__ uint32_t warp_xor(uint32_t v)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v ^= __shfl_xor_sync(0xffffffffu, v, o);
  }
  return v;
}

// One layer (base-graph row) for check lane tid, specialised on the row degree so that the edge
// loops unroll without predication. FIRST selects the first iteration, where every row's
// check-to-variable messages are still zero (the reference copies the soft bits into the v2c
// messages then: ldpc_decoder_impl.cpp:208-212).
template <int DEG, bool FIRST, int ZT>
__device__ __forceinline__ void row_update(const int tid, const int Zr, int8_t* __restrict__ soft,
                                           const uint32_t* __restrict__ edge, int8_t* __restrict__ c2v_row)
{
  const int Z = ZT > 0 ? ZT : Zr;
  int       m[DEG];
  unsigned  pos[DEG];
  int       min1 = 120, min2 = 120, sgn = 0;
#pragma unroll
  for (int e = 0; e < DEG; ++e) {
    const uint32_t ed = edge[e];
    const unsigned p0 = (unsigned)tid + (ed & 0xffffu);
    const unsigned p  = min(p0, p0 - (unsigned)Z) + (ed >> 16);
    pos[e]            = p;
    const int x       = soft[p];
    int       v       = x;
    if (!FIRST) {
      const int c = c2v_row[e * Z];
      v           = max(-120, min(120, x - c));
      v           = (x == 127 || x == -127) ? x : v;
    }
    m[e]        = v;
    const int a = abs(v);
    min2        = min(min2, max(min1, a));
    min1        = min(min1, a);
    sgn ^= v;
  }
  const int s1 = scale_mag(min1);
  const int s2 = scale_mag(min2);
#pragma unroll
  for (int e = 0; e < DEG; ++e) {
    const int v    = m[e];
    const int a    = abs(v);
    const int mag  = (a == min1) ? s2 : s1;
    const int c    = ((v ^ sgn) < 0) ? -mag : mag;
    c2v_row[e * Z] = (int8_t)c;
    int t          = c + v;
    t              = (t > 120) ? 127 : ((t < -120) ? -127 : t);
    t              = (a == 127) ? v : t;
    soft[pos[e]]   = (int8_t)t;
  }
}

// Degree-19 rows (BG1 rows 0-3): the same update as a rolled loop with the v2c messages staged in
// shared memory (one byte per edge and lane), so the wide rows do not raise the register budget
// of the whole kernel; the soft-bit addresses are recomputed in the second pass.
template <bool FIRST, int ZT, int NT>
__device__ __forceinline__ void row_update_wide(const int deg, const int tid, const int Zr, int8_t* __restrict__ soft,
                                                const uint32_t* __restrict__ edge, int8_t* __restrict__ c2v_row,
                                                int8_t* __restrict__ mbuf)
{
  const int Z    = ZT > 0 ? ZT : Zr;
  int       min1 = 120, min2 = 120, sgn = 0;
#pragma unroll 2
  for (int e = 0; e < deg; ++e) {
    const uint32_t ed = edge[e];
    const unsigned p0 = (unsigned)tid + (ed & 0xffffu);
    const unsigned p  = min(p0, p0 - (unsigned)Z) + (ed >> 16);
    const int      x  = soft[p];
    int            v  = x;
    if (!FIRST) {
      const int c = c2v_row[e * Z];
      v           = max(-120, min(120, x - c));
      v           = (x == 127 || x == -127) ? x : v;
    }
    mbuf[e * NT + tid] = (int8_t)v;
    const int a              = abs(v);
    min2                     = min(min2, max(min1, a));
    min1                     = min(min1, a);
    sgn ^= v;
  }
  const int s1 = scale_mag(min1);
  const int s2 = scale_mag(min2);
#pragma unroll 2
  for (int e = 0; e < deg; ++e) {
    const uint32_t ed  = edge[e];
    const unsigned p0  = (unsigned)tid + (ed & 0xffffu);
    const unsigned p   = min(p0, p0 - (unsigned)Z) + (ed >> 16);
    const int      v   = mbuf[e * NT + tid];
    const int      a   = abs(v);
    const int      mag = (a == min1) ? s2 : s1;
    const int      c   = ((v ^ sgn) < 0) ? -mag : mag;
    c2v_row[e * Z]     = (int8_t)c;
    int t              = c + v;
    t                  = (t > 120) ? 127 : ((t < -120) ? -127 : t);
    t                  = (a == 127) ? v : t;
    soft[p]            = (int8_t)t;
  }
}

// Base-graph row degrees: BG1 {3..10, 19}, BG2 {3..10}.
template <bool FIRST, int ZT, int NT>
__device__ __forceinline__ void row_dispatch(int deg, int tid, int Z, int8_t* soft, const uint32_t* edge, int8_t* c2v_row,
                                             int8_t* mbuf)
{
  switch (deg) {
    case 3: row_update<3, FIRST, ZT>(tid, Z, soft, edge, c2v_row); break;
    case 4: row_update<4, FIRST, ZT>(tid, Z, soft, edge, c2v_row); break;
    case 5: row_update<5, FIRST, ZT>(tid, Z, soft, edge, c2v_row); break;
    case 6: row_update<6, FIRST, ZT>(tid, Z, soft, edge, c2v_row); break;
    case 7: row_update<7, FIRST, ZT>(tid, Z, soft, edge, c2v_row); break;
    case 8: row_update<8, FIRST, ZT>(tid, Z, soft, edge, c2v_row); break;
    case 9: row_update<9, FIRST, ZT>(tid, Z, soft, edge, c2v_row); break;
    case 10: row_update<10, FIRST, ZT>(tid, Z, soft, edge, c2v_row); break;
    default: row_update_wide<FIRST, ZT, NT>(deg, tid, Z, soft, edge, c2v_row, mbuf); break;
  }
}

// Shared memory of the one-lane decoder: NT threads, lifting sizes up to MAXZ (22 * MAXZ / 32 <= NT,
// so that one thread per 32-bit hard-decision word covers the message).
template <int NT, int MAXZ>
struct smem_scalar_t {
  __align__(16) int8_t soft[pg::kMaxNodes * MAXZ];
  uint32_t             edge[pg::kBg1Edges];
  uint32_t             hard[(22 * MAXZ) / 32];
  uint32_t             red[NT / 32];
  int8_t               mbuf[pg::kMaxRowDegree * NT]; // v2c staging of the degree-19 rows
  int                  s_last;
  int                  s_done;
};
using smem_t = smem_scalar_t<kThreads, pg::kMaxZ>;

// Decodes codeblock cb with check-to-variable slab `slab`, one lane per thread (NT threads, Z <=
// MAXZ); ZT > 0 specialises the lifting size at compile time.
template <int ZT, int NT, int MAXZ>
__device__ __forceinline__ void decode_codeblock(const pg_ldpc_cb& d, smem_scalar_t<NT, MAXZ>& sm,
                                                 const int8_t* __restrict__ llrs,
                                                 uint8_t* __restrict__ bits, int32_t* __restrict__ iterations,
                                                 int8_t* __restrict__ c2v_all, const uint32_t* __restrict__ crc_pow,
                                                 const int cb, const int slab)
{
  int8_t*   soft   = sm.soft;
  uint32_t* edge   = sm.edge;
  uint32_t* hard   = sm.hard;
  uint32_t* red    = sm.red;
  int&      s_last = sm.s_last;
  int&      s_done = sm.s_done;
  const int        tid = threadIdx.x;
  const int        bg  = d.base_graph;
  const int        Z   = ZT > 0 ? ZT : (int)d.lifting_size;
  const int        set = (Z >= 2 && Z <= MAXZ) ? dev_set_index(Z) : -1;
  if ((bg != 1 && bg != 2) || set < 0) {
    if (tid == 0) {
      iterations[cb] = -1;
    }
    return;
  }
  const int     g        = bg - 1;
  const int     Kb       = bg == 1 ? 22 : 10;
  const int     nrows    = bg == 1 ? pg::kBg1Rows : pg::kBg2Rows;
  const int     nedges   = bg == 1 ? pg::kBg1Edges : pg::kBg2Edges;
  const int     nfull    = bg == 1 ? 68 : 52;
  const int     msg_len  = Kb * Z;
  const int     n        = (int)d.nof_llrs;
  const int8_t* in       = llrs + d.llr_offset;
  int8_t*       c2v      = c2v_all + (size_t)slab * pg::kC2vStride;
  const int     nbytes   = (msg_len + 7) / 8;
  uint8_t*      out      = bits + d.out_offset;
  const int     crc_poly = d.crc_poly;
  const int     nwords   = (msg_len + 31) / 32;

  // Edge table of this lifting size: node offset (col * Z) and shift (V mod Z).
  for (int e = tid; e < nedges; e += NT) {
    const int col = c_edge_col[g][e];
    const int s   = c_edge_v[g][e][set] % Z;
    edge[e]       = ((uint32_t)(col * Z) << 16) | (uint32_t)s;
  }
  if (tid == 0) {
    s_last = 0;
    s_done = 0;
  }
  __syncthreads();

  // One pass over the input: soft bits (2Z punctured zeros, whole nodes clamped to +-64, a ragged
  // tail as is, ldpc_decoder_impl.cpp:147-188) and the last non-zero LLR (the trailing-zero trim,
  // ldpc_decoder_impl.cpp:66-71), four LLRs per thread step.
  const int nof_full = (n / Z) * Z;
  const int soft_len = nfull * Z;
  for (int i = tid; i < 2 * Z; i += NT) {
    soft[i] = 0;
  }
  for (int i = 2 * Z + n + tid; i < soft_len; i += NT) {
    soft[i] = 0;
  }
  int        last    = 0;
  const bool aligned = (reinterpret_cast<uintptr_t>(in) & 3u) == 0;
  for (int k0 = 4 * tid; k0 < n; k0 += 4 * NT) {
    int v[4];
    if (aligned && k0 + 3 < n) {
      const uint32_t w = pg::load_written(reinterpret_cast<const uint32_t*>(in + k0));
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[j] = (int)(int8_t)(w >> (8 * j));
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[j] = k0 + j < n ? pg::load_written(in + k0 + j) : 0;
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int k = k0 + j;
      if (k < n && 2 * Z + k < soft_len) {
        last = v[j] != 0 ? k + 1 : last;
        soft[2 * Z + k] = (int8_t)(k < nof_full ? max(-64, min(64, v[j])) : v[j]);
      }
    }
  }
  last = warp_max(last);
  if ((tid & 31) == 0 && last > 0) {
    atomicMax(&s_last, last);
  }
  __syncthreads();

  const int input_size = s_last;
  if (input_size < msg_len) {
    for (int b = tid; b < nbytes; b += NT) {
      out[b] = 0xff;
    }
    if (tid == 0) {
      iterations[cb] = 0;
    }
    return;
  }
  int cb_len = max(input_size + 2 * Z, (Kb + 4) * Z);
  cb_len     = ((cb_len + Z - 1) / Z) * Z;
  const int nof_layers = min(cb_len / Z - Kb, nrows);

  uint32_t g_poly = 0;
  int      order  = 24;
  if (crc_poly == PG_CRC16) {
    order = 16;
  }
  const uint32_t* pow_tab = crc_pow + (size_t)(crc_poly <= PG_CRC24B ? crc_poly : 0) * pg::kCrcPowLen;
  (void)g_poly;
  const int crc_len = msg_len - (int)d.nof_filler_bits;

  int result = 0;
  const int max_it = d.max_iterations;
  const int nsteps = steps_for_layers(g, nof_layers);
  // With at most a warp of lanes one warp runs the rows of an iteration and meets no other in between, and the
  // messages are in shared memory: a barrier of the whole CTA per step, with messages in L2, made a batch of 200
  // codeblocks of Z = 3 (BG2) take 325 us instead of 230.
  constexpr bool one_warp = MAXZ <= 32;
  for (int it = 0; it < max_it; ++it) {
    for (int st = 0; st < nsteps && (!one_warp || tid < 32); ++st) {
      // Messages are read from the second iteration on: prefetch the next step's.
      if (!one_warp && (it > 0 || st + 1 == nsteps)) {
        prefetch_step(g, st + 1 < nsteps ? st + 1 : 0, nof_layers, tid, reinterpret_cast<const char*>(c2v), Z);
      }
      const int r0 = c_step_row0[g][st];
      const int r1 = min(r0 + (int)c_step_nrows[g][st], nof_layers);
      if (tid < Z) {
        for (int r = r0; r < r1; ++r) {
          const int deg     = c_row_deg[g][r];
          const int e0      = c_row_e0[g][r];
          int8_t*   c2v_row = c2v + (size_t)e0 * Z + tid;
          if (it == 0) {
            row_dispatch<true, ZT, NT>(deg, tid, Z, soft, edge + e0, c2v_row, sm.mbuf);
          } else {
            row_dispatch<false, ZT, NT>(deg, tid, Z, soft, edge + e0, c2v_row, sm.mbuf);
          }
        }
      }
      if (one_warp) {
        __syncwarp();
      } else {
        __syncthreads();
      }
    }
    if (one_warp) {
      __syncthreads();
    }

    // Hard decisions, zero check and CRC over the significant bits.
    int      zero = 0;
    uint32_t crc  = 0;
    if (tid < nwords) {
      const int4* p = reinterpret_cast<const int4*>(soft + 32 * tid);
      const int4  a = p[0];
      const int4  b = p[1];
      const int   wv[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
      uint32_t    w     = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int idx = 32 * tid + 4 * k + j;
          const int x   = (int)(int8_t)((uint32_t)wv[k] >> (8 * j));
          if (idx < msg_len) {
            w |= (uint32_t)(x <= 0) << (31 - (4 * k + j));
            zero |= (x == 0);
          }
        }
      }
      hard[tid] = w;
      if (crc_poly != PG_CRC_NONE) {
        const int valid = crc_len - 32 * tid;
        uint32_t  wc    = w;
        if (valid <= 0) {
          wc = 0;
        } else if (valid < 32) {
          wc &= ~((1u << (32 - valid)) - 1u);
        }
        const int e_w = crc_len - 32 * tid - 32 + order;
        while (wc != 0) {
          const int q = __ffs(wc) - 1;
          crc ^= __ldg(pow_tab + e_w + q);
          wc &= wc - 1;
        }
      }
    }
    zero = __syncthreads_or(zero);
    crc  = warp_xor(crc);
    if ((tid & 31) == 0) {
      red[tid >> 5] = crc;
    }
    __syncthreads();
    if (tid == 0) {
      uint32_t t = 0;
      for (int w = 0; w < NT / 32; ++w) {
        t ^= red[w];
      }
      s_done = (crc_poly != PG_CRC_NONE && !zero && t == 0) ? 1 : 0;
    }
    __syncthreads();
    if (s_done) {
      result = it + 1;
      break;
    }
  }

  if (crc_poly == PG_CRC_NONE) {
    // Syndrome check over the processed rows (ldpc_decoder_impl.cpp:329-387).
    int bad = 0;
    if (tid < Z) {
      int e0 = 0;
      for (int r = 0; r < nof_layers; ++r) {
        const int deg    = c_row_deg[g][r];
        int       parity = 0;
        for (int e = 0; e < deg; ++e) {
          const uint32_t ed = edge[e0 + e];
          int            p  = tid + (int)(ed & 0xffffu);
          p                 = (p >= Z) ? p - Z : p;
          const int x       = soft[p + (int)(ed >> 16)];
          bad |= (x == 0);
          parity ^= (x <= 0);
        }
        bad |= parity;
        e0 += deg;
      }
    }
    bad = __syncthreads_or(bad);
    // The hard words of the last iteration are in hard[]; a zero soft bit also fails.
    int zero = 0;
    if (tid < nwords) {
      for (int k = 0; k < 32; ++k) {
        const int idx = 32 * tid + k;
        if (idx < msg_len && soft[idx] == 0) {
          zero = 1;
        }
      }
    }
    zero   = __syncthreads_or(zero);
    result = (!bad && !zero) ? max_it : 0;
  }

  for (int b = tid; b < nbytes; b += NT) {
    out[b] = (uint8_t)(hard[b >> 2] >> (24 - 8 * (b & 3)));
  }
  if (tid == 0) {
    iterations[cb] = result;
  }
}


// counter == nullptr: one CTA per codeblock (blockIdx.x), slab blockIdx.x. Otherwise a persistent
// grid: each CTA takes the next work index from *counter (zeroed before the launch), decodes
// codeblock order[w] (or w) with its own slab blockIdx.x, and stops when the n codeblocks are
// taken. Codeblocks are independent, so the order of work changes no result. With an order, counter[1] (the
// arrivals of the ordering launch) is left at zero.
__global__ void __launch_bounds__(kThreads, 2) ldpc_decode_kernel(const pg_ldpc_cb* __restrict__ descs,
                                                              const int8_t* __restrict__ llrs,
                                                              uint8_t* __restrict__ bits,
                                                              int32_t* __restrict__ iterations,
                                                              int8_t* __restrict__ c2v_all,
                                                              const uint32_t* __restrict__ crc_pow,
                                                              const uint32_t* __restrict__ order, int n,
                                                              int* __restrict__ counter)
{
  __shared__ smem_t sm;
  __shared__ int    s_work;
  if (counter == nullptr) {
    const pg_ldpc_cb d = descs[blockIdx.x];
    if (d.lifting_size == 384) {
      decode_codeblock<384, kThreads, pg::kMaxZ>(d, sm, llrs, bits, iterations, c2v_all, crc_pow, blockIdx.x, blockIdx.x);
    } else {
      decode_codeblock<0, kThreads, pg::kMaxZ>(d, sm, llrs, bits, iterations, c2v_all, crc_pow, blockIdx.x, blockIdx.x);
    }
    return;
  }
  for (;;) {
    if (threadIdx.x == 0) {
      s_work = atomicAdd(counter, 1);
    }
    __syncthreads();
    const int w = s_work;
    __syncthreads();
    if (w >= n) {
      if (order != nullptr && blockIdx.x == 0 && threadIdx.x == 0) {
        counter[1] = 0;
      }
      break;
    }
    const int        cb = order != nullptr ? (int)order[w] : w;
    const pg_ldpc_cb d  = descs[cb];
    if (d.lifting_size == 384) {
      decode_codeblock<384, kThreads, pg::kMaxZ>(d, sm, llrs, bits, iterations, c2v_all, crc_pow, cb, blockIdx.x);
    } else {
      decode_codeblock<0, kThreads, pg::kMaxZ>(d, sm, llrs, bits, iterations, c2v_all, crc_pow, cb, blockIdx.x);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Lane-pair decoder: even lifting sizes, H = Z / 2. A lane pair j (0 <= j < H) is check lanes j and
// j + H, carried as the two halves of one f16x2 register by T adjacent threads, which split the
// edges of every row.
//
// Soft bits: E[col][k] = (soft[col][k], soft[col][k + H]) as one f16x2 word, 0 <= k < H, in shared
// memory. For an edge of shift s, lane j reads variable lane (j + s) mod Z and lane j + H reads
// (j + H + s) mod Z: both are halves of the same word k = (j + s') mod H with s' = s mod H, swapped
// when (j + s' >= H) differs from (s >= H). The edge table in shared memory holds what pair_edge needs. Rows are
// padded to a multiple of T edges with an edge to a constant column of
// saturated positive soft bits, which changes no minimum, sign or message of the row.
//
// Arithmetic: the reference's int8 rules as exact f16x2 identities (every value that decides is an
// integer of magnitude at most 2,048):
//   soft x       finite when |x| <= 120; any larger magnitude is the reference's +-127. The promotion
//                of a sum above 120 is not done when the sum is stored but when it is read: the
//                stored sum (at most 120 + 96) is compared with 120 there.
//   v2c          v = min(max(clamp(x - c, +-120), 400x - 48128), 400x + 48128), fused multiply-adds: for
//                |x| <= 120 the bounds lie outside [-120, 120]; from |x| = 121 they are at least 272 in
//                magnitude with x's sign (or infinite). So a saturated v never is the row's minimum
//                (the search starts at 120), keeps its sign, and v + c is again above 120 (|c| <= 96):
//                a saturated soft bit stays saturated. Messages are finite, so no infinity meets its
//                negative.
//   min1/min2/sign: min.xorsign.abs keeps min(|.|) and accumulates the sign product in min1's sign.
//   scale        floor(m * 52428 / 2^16) for integer 0 <= m <= 120 is max(fma(m, f16(0.8), 1023.5) -
//                1024, 0): the fused multiply-add rounds once, to an integer (the spacing of f16 in
//                [1024, 2048)), and f16(0.8) = 0.7998046875 errs by at most 0.024 at m = 120, inside
//                the 0.1 margin of every rounding decision (checked for every m).
//   c2v          (|v| == min1 ? s2 : s1) with the sign product of the others by XOR of sign bits.
//   soft         c + v.
// Whole input nodes are clamped to +-64. In a ragged tail (fewer LLRs than the node) the values 121 to
// 126 are finite in the first iteration, which this reading rule cannot tell from a sum: a codeblock
// that holds one runs its first iteration through pair_row_ragged, which promotes when it stores.
//
// Check-to-variable messages are offset-binary byte pairs (value + 128: f16 bits 0x6400 | byte are
// 1024 + byte), two edges to a 32-bit word, one word column per thread; each thread reads only what
// it wrote. They stay in shared memory when the rows that the codeblock runs fit there (behind the
// columns that those rows use), else in the CTA's global slab.
constexpr uint32_t kH120     = 0x57805780u; // 120
constexpr uint32_t kHm120    = 0xd780d780u; // -120
constexpr uint32_t kH126p5   = 0x57e857e8u; // 126.5
constexpr uint32_t kH400     = 0x5e405e40u; // 400
constexpr uint32_t kH48128   = 0x79e079e0u; // 48128
constexpr uint32_t kHm48128  = 0xf9e0f9e0u; // -48128
constexpr uint32_t kH1152    = 0x64806480u; // 1152 = 1024 + 128
constexpr uint32_t kHm1152   = 0xe480e480u; // -1152
constexpr uint32_t kAbs      = 0x7fff7fffu;
constexpr uint32_t kSign     = 0x80008000u;
constexpr uint32_t kSat      = 0x60006000u; // the top two exponent bits
constexpr uint32_t kH8192    = 0x70007000u; // 8192 (the constant column)
constexpr uint32_t kH0       = 0x00000000u; // 0
constexpr uint32_t kH0p8     = 0x3a663a66u; // f16(0.8) = 0.7998046875
constexpr uint32_t kH1023p5  = 0x63ff63ffu; // 1023.5
constexpr uint32_t kHm1024   = 0xe400e400u; // -1024

__device__ __forceinline__ uint32_t h2_sub(uint32_t a, uint32_t b)
{
  uint32_t r;
  asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t h2_add(uint32_t a, uint32_t b)
{
  uint32_t r;
  asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t h2_fma(uint32_t a, uint32_t b, uint32_t c)
{
  uint32_t r;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}
__device__ __forceinline__ uint32_t h2_min(uint32_t a, uint32_t b)
{
  uint32_t r;
  asm("min.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t h2_max(uint32_t a, uint32_t b)
{
  uint32_t r;
  asm("max.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t h2_min_xs(uint32_t a, uint32_t b)
{
  uint32_t r;
  asm("min.xorsign.abs.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t h2_max_xs(uint32_t a, uint32_t b)
{
  uint32_t r;
  asm("max.xorsign.abs.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
// All ones in the halves where |a| > b, or |a| == b.
__device__ __forceinline__ uint32_t h2_abs_gt_mask(uint32_t a, uint32_t b)
{
  const __half2 x = __habs2(*reinterpret_cast<const __half2*>(&a));
  return __hgt2_mask(x, *reinterpret_cast<const __half2*>(&b));
}
__device__ __forceinline__ uint32_t h2_abs_eq_mask(uint32_t a, uint32_t b)
{
  const __half2 x = __habs2(*reinterpret_cast<const __half2*>(&a));
  return __heq2_mask(x, *reinterpret_cast<const __half2*>(&b));
}
// 1.0 in the halves where |a| != b, else 0.0.
__device__ __forceinline__ uint32_t h2_abs_ne(uint32_t a, uint32_t b)
{
  const __half2 r = __hne2(__habs2(*reinterpret_cast<const __half2*>(&a)), *reinterpret_cast<const __half2*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}

// Offset-binary byte pair -> f16x2 integers (low byte first).
__device__ __forceinline__ uint32_t bytes_to_h2(uint32_t b)
{
  return h2_add(__byte_perm(b, 0x6464u, 0x5140u), kHm1152);
}

__device__ __forceinline__ uint32_t pair_scale(uint32_t m)
{
  return h2_max(h2_add(h2_fma(m, kH0p8, kH1023p5), kHm1024), kH0);
}

// Shared-memory accesses by 32-bit shared address (the soft-bit addresses of the edge table are
// absolute, so that no base is added per edge).
__device__ __forceinline__ uint32_t lds_u32(uint32_t adr)
{
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(adr));
  return v;
}
__device__ __forceinline__ uint4 lds_v4(uint32_t adr)
{
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(adr));
  return v;
}
__device__ __forceinline__ void sts_u32(uint32_t adr, uint32_t v)
{
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(adr), "r"(v));
}

constexpr int kPairMaxEdges = 460; // padded edges of a graph, T <= 4 (316 + 3 * 46 at most)

// Tables of the base graphs, indexed by [graph], and of their rows padded to a multiple of T = 2 << lg
// edges ([lg][graph]): first padded edge and first message word (in units of the active
// threads) of each row. In global memory: threads read different entries.
struct pair_tables {
  uint16_t pad_v[2][2][kPairMaxEdges][8]; // shift of each padded edge, per lifting set
  uint8_t  pad_col[2][2][kPairMaxEdges];  // its column plus 1, 0 for an edge to the constant column
  uint8_t  row_sync[2][pg::kBg1Rows];     // the row is the last of its step
  uint16_t pad_e0[2][2][pg::kBg1Rows + 1];
  uint16_t msg0[2][2][pg::kBg1Rows + 1];
};
__device__ pair_tables g_pair_tables;

constexpr uint32_t kPairTabBytes = kPairMaxEdges * 16;
constexpr uint32_t kPairMinSmem  = kPairTabBytes + (pg::kMaxNodes + 1) * (pg::kMaxZ / 2) * 4; // every column
constexpr int      kOddMaxZ      = 16;   // odd lifting sizes are at most 15

constexpr int kPairThreads = 384;

// Descriptors of a batch passed in a launch's arguments.
template <int N>
struct desc_args {
  pg_ldpc_cb cb[N];
};
constexpr int kDecodeArgs = 260;  // of the decoder: batches of one CTA per codeblock
constexpr int kScoreArgs  = 1600; // of the ordering launch: 32,000 bytes of the 32,764 a launch takes
static_assert(sizeof(desc_args<kScoreArgs>) <= 32000, "arguments of a launch");

struct pair_shared {
  uint4    row[pg::kBg1Rows + 1]; // first padded edge, first message byte, edges per thread, threads to meet after it or 0
  uint32_t tb_crc;
  int      seen[kPairThreads / 32]; // per warp: twice the last non-zero LLR's end, plus 1 for a ragged value
  uint32_t crc[2];
  int      zero[2];
  int      work;
};

// Byte offset in E and byte-permute selector of edge table entry c for lane pair j. The decoder is
// bound by the ALU pipe (comparisons, selects, logic, byte permutes: 64 lanes a cycle on an SM), so
// both are formed on the FP32 pipe: w = 1 when the edge wraps (the saturated sum of j and 1 - (H - s')
// is 0 or 1), and the integers travel as the bits of denormal numbers, on which an FP32 multiply-add by
// w is exact: adr = (4 j + base) - w 4 H, sel = sel0 + w dsel.
__device__ __forceinline__ void pair_edge(const uint4 c, const float jf, const float j4d, const float nh4d,
                                          uint32_t& adr, uint32_t& sel)
{
  const float w = __saturatef(__fadd_rn(jf, __uint_as_float(c.y)));
  adr           = __float_as_uint(__fmaf_rn(w, nh4d, __fadd_rn(j4d, __uint_as_float(c.x))));
  sel           = __float_as_uint(__fmaf_rn(w, __uint_as_float(c.w), __uint_as_float(c.z)));
}

// The partial (min1, min2, sign) of the T threads of a lane pair meet through shuffles.
template <int T>
__device__ __forceinline__ void pair_reduce(uint32_t& min1, uint32_t& min2)
{
#pragma unroll
  for (int o = 1; o < T; o <<= 1) {
    const uint32_t o1 = __shfl_xor_sync(0xffffffffu, min1, o);
    const uint32_t o2 = __shfl_xor_sync(0xffffffffu, min2, o);
    min2              = h2_min_xs(h2_min_xs(min2, o2), h2_max_xs(min1, o1));
    min1              = h2_min_xs(min1, o1);
  }
}

// A thread's message words of one row: in shared memory (a 32-bit address) or in the global slab.
struct msg_shared {
  uint32_t a;
  __device__ __forceinline__ msg_shared at(uint32_t byte) const { return {a + byte}; }
  template <int NW>
  __device__ __forceinline__ void load(uint32_t* m) const
  {
    if constexpr (NW == 2) {
      asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(m[0]), "=r"(m[NW - 1]) : "r"(a));
    } else {
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        m[w] = lds_u32(a + 4 * w);
      }
    }
  }
  template <int NW>
  __device__ __forceinline__ void store(const uint32_t* m) const
  {
    if constexpr (NW == 2) {
      asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(a), "r"(m[0]), "r"(m[NW - 1]) : "memory");
    } else {
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        sts_u32(a + 4 * w, m[w]);
      }
    }
  }
};
struct msg_global {
  unsigned char* a;
  __device__ __forceinline__ msg_global at(uint32_t byte) const { return {a + byte}; }
  template <int NW>
  __device__ __forceinline__ void load(uint32_t* m) const
  {
    if constexpr (NW == 2) {
      const uint2 q = *reinterpret_cast<const uint2*>(a);
      m[0] = q.x, m[NW - 1] = q.y;
    } else {
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        m[w] = reinterpret_cast<const uint32_t*>(a)[w];
      }
    }
  }
  template <int NW>
  __device__ __forceinline__ void store(const uint32_t* m) const
  {
    if constexpr (NW == 2) {
      *reinterpret_cast<uint2*>(a) = make_uint2(m[0], m[NW - 1]);
    } else {
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        reinterpret_cast<uint32_t*>(a)[w] = m[w];
      }
    }
  }
};

// The end of a step: the rows before it have stored their soft bits. A row meets the step before it only when
// it reads soft bits; its edge table and messages, which no other thread writes, are read before that. nthreads: the threads of the rows, or 0.
__device__ __forceinline__ void step_sync(const uint32_t nthreads)
{
  if (nthreads != 0) {
    asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory");
  }
}

// One row for this thread's NE edges (table entries zt[0 .. NE - 1], message words msg[0], msg[nta],
// ...). FIRST: the first iteration, whose messages are still zero.
template <int NE, bool FIRST, int T, class M>
__device__ __forceinline__ void pair_row(const uint32_t zt, const float jf, const float j4d, const float nh4d,
                                         const M msg, const bool active, const uint32_t sync)
{
  constexpr int NW = (NE + 1) / 2;
  uint32_t      m[NW], v[NE], adr[NE], sel[NE];
  if (!FIRST) {
    msg.template load<NW>(m);
  }
#pragma unroll
  for (int e = 0; e < NE; ++e) {
    pair_edge(lds_v4(zt + 16 * e), jf, j4d, nh4d, adr[e], sel[e]);
  }
  step_sync(sync);
  uint32_t min1 = kH120, min2 = kH120;
#pragma unroll
  for (int e = 0; e < NE; ++e) {
    const uint32_t x = __byte_perm(lds_u32(adr[e]), 0, sel[e]);
    uint32_t       d = x;
    if (!FIRST) {
      const uint32_t c = h2_add(__byte_perm(m[e / 2], 0x64646464u, (e & 1) ? 0x4342u : 0x4140u), kHm1152);
      d                = h2_min(h2_max(h2_sub(x, c), kHm120), kH120);
    }
    v[e]             = h2_min(h2_max(d, h2_fma(x, kH400, kHm48128)), h2_fma(x, kH400, kH48128));
    const uint32_t t = h2_max_xs(min1, v[e]);
    min2             = h2_min_xs(min2, t);
    min1             = h2_min_xs(min1, v[e]);
  }
  pair_reduce<T>(min1, min2);
  const uint32_t m1  = min1 & kAbs;
  const uint32_t sgn = min1 & kSign; // sign product of every v2c of the row
  const uint32_t s1  = pair_scale(m1) ^ sgn;
  const uint32_t s2  = pair_scale(min2 & kAbs) ^ sgn;
  const uint32_t ds  = h2_sub(s1, s2);
#pragma unroll
  for (int e = 0; e < NE; ++e) {
    const uint32_t c = h2_fma(ds, h2_abs_ne(v[e], m1), s2) ^ (v[e] & kSign);
    if (active) {
      sts_u32(adr[e], __byte_perm(h2_add(c, v[e]), 0, sel[e]));
    }
    v[e] = h2_add(c, kH1152); // bytes 0 and 2 are the offset-binary messages
  }
#pragma unroll
  for (int w = 0; w < NW; ++w) {
    m[w] = __byte_perm(v[2 * w], v[2 * w + 1 < NE ? 2 * w + 1 : 2 * w], 0x6420u);
  }
  msg.template store<NW>(m);
}

// The first iteration's row with the promotion where the soft bit is stored, for codeblocks whose
// ragged tail holds magnitudes of 121 to 126: soft bits up to 126 are finite. Any ne; each edge's v2c is
// formed again in the second pass.
template <int T>
__device__ __noinline__ void pair_row_ragged(const int ne, const uint32_t zt, const float jf, const float j4d,
                                             const float nh4d, uint32_t* msg, const bool active, const uint32_t sync)
{
  step_sync(sync);
  uint32_t min1 = kH120, min2 = kH120, adr, sel;
#pragma unroll 1
  for (int e = 0; e < ne; ++e) {
    pair_edge(lds_v4(zt + 16 * e), jf, j4d, nh4d, adr, sel);
    const uint32_t x = __byte_perm(lds_u32(adr), 0, sel);
    const uint32_t v = x | (h2_abs_gt_mask(x, kH126p5) & kSat);
    const uint32_t t = h2_max_xs(min1, v);
    min2             = h2_min_xs(min2, t);
    min1             = h2_min_xs(min1, v);
  }
  pair_reduce<T>(min1, min2);
  const uint32_t m1  = min1 & kAbs;
  const uint32_t sgn = min1 & kSign;
  const uint32_t s1  = pair_scale(m1) ^ sgn;
  const uint32_t s2  = pair_scale(min2 & kAbs) ^ sgn;
  uint32_t       pack = 0;
#pragma unroll 1
  for (int e = 0; e < ne; ++e) {
    pair_edge(lds_v4(zt + 16 * e), jf, j4d, nh4d, adr, sel);
    const uint32_t x  = __byte_perm(lds_u32(adr), 0, sel);
    const uint32_t v  = x | (h2_abs_gt_mask(x, kH126p5) & kSat);
    const uint32_t eq = h2_abs_eq_mask(v, m1);
    const uint32_t c  = ((eq & s2) | (~eq & s1)) ^ (v & kSign);
    const uint32_t b  = h2_add(c, kH1152);
    pack              = (e & 1) ? __byte_perm(pack, b, 0x6420u) : b;
    if ((e & 1) != 0 || e + 1 == ne) {
      msg[e / 2] = (e & 1) ? pack : __byte_perm(pack, pack, 0x6420u);
    }
    const uint32_t u = h2_add(c, v);
    if (active) {
      sts_u32(adr, __byte_perm(u | (h2_abs_gt_mask(u, kH120) & kSat), 0, sel));
    }
  }
}

// The rows of one iteration.
template <bool FIRST, int T, class M>
__device__ __forceinline__ void pair_rows(const pair_shared& sh, const int nof_layers, const uint32_t tpart16,
                                          const float jf, const float j4d, const float nh4d, const M msg,
                                          const bool active)
{
  const uint32_t tid4 = 4u * threadIdx.x;
  uint32_t       sync = 0; // the step before this row
  uint4          rd   = sh.row[0];
#pragma unroll 1
  for (int r = 0; r < nof_layers; ++r) {
    const uint4 next = sh.row[r + 1];
    const int   ne   = (int)rd.z;
    const M     mr   = msg.at(rd.y);
    // Base-graph row degrees: BG1 {3..10, 19}, BG2 {3..10}.
#define PG_PAIR_ROW(n) \
  pair_row<n, FIRST, T>(rd.x + tpart16 * (n), jf, j4d, nh4d, mr.at(tid4 * (((n) + 1) / 2)), active, sync)
    if constexpr (T == 2) {
      if (ne < 4) {
        if (ne < 3) {
          PG_PAIR_ROW(2);
        } else {
          PG_PAIR_ROW(3);
        }
      } else if (ne < 5) {
        PG_PAIR_ROW(4);
      } else if (ne < 6) {
        PG_PAIR_ROW(5);
      } else {
        PG_PAIR_ROW(10);
      }
    } else {
      if (ne < 3) {
        if (ne < 2) {
          PG_PAIR_ROW(1);
        } else {
          PG_PAIR_ROW(2);
        }
      } else if (ne < 4) {
        PG_PAIR_ROW(3);
      } else {
        PG_PAIR_ROW(5);
      }
    }
#undef PG_PAIR_ROW
    sync = rd.w;
    rd   = next;
  }
}

// f16 soft bit -> hard bit: soft <= 0 (either zero counts as 0).
__device__ __forceinline__ bool pair_hard(uint32_t h)
{
  return (h & 0x8000u) != 0 || (h & 0x7fffu) == 0;
}

constexpr int kFetchBatch = 5; // pieces of eight lane pairs per thread step: 68 columns of Z = 384 in one

// Eight input LLRs from index k (any k; outside [0, n) they are zero) as soft bits in offset
// binary, four per word: whole nodes (index < nof_full) clamped to +-64, a ragged tail as is
// (ldpc_decoder_impl.cpp:147-188). last: one past the last non-zero LLR seen (the trailing-zero trim,
// ldpc_decoder_impl.cpp:66-71); ragged: a tail value of magnitude 121 to 126 was seen.
// q: the eight LLRs where fetch_whole holds.
__device__ __forceinline__ bool fetch_whole(int k, int nof_full, bool aligned)
{
  return aligned && k >= 0 && k + 8 <= nof_full;
}

__device__ __forceinline__ void fetch8(const int8_t* __restrict__ in, int k, int n, int nof_full, bool aligned, uint2 q,
                                       int& last, int& ragged, uint32_t& w0, uint32_t& w1)
{
  if (fetch_whole(k, nof_full, aligned)) {
    if ((q.x | q.y) != 0) {
      last = max(last, k + (q.y != 0 ? 8 - (__clz(q.y) >> 3) : 4 - (__clz(q.x) >> 3)));
    }
    w0 = __vmaxs4(__vmins4(q.x, 0x40404040u), 0xc0c0c0c0u) ^ 0x80808080u;
    w1 = __vmaxs4(__vmins4(q.y, 0x40404040u), 0xc0c0c0c0u) ^ 0x80808080u;
    return;
  }
  w0 = 0;
  w1 = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int kk = k + i;
    int       x  = (kk >= 0 && kk < n) ? pg::load_written(in + kk) : 0;
    last         = x != 0 ? max(last, kk + 1) : last;
    if (kk < nof_full) {
      x = max(-64, min(64, x));
    } else {
      ragged |= (abs(x) > 120 && abs(x) < 127) ? 1 : 0;
    }
    const uint32_t b = (uint32_t)(x + 128);
    if (i < 4) {
      w0 |= b << (8 * i);
    } else {
      w1 |= b << (8 * (i - 4));
    }
  }
}

// a(x) b(x) mod g(x) for a of degree below `order` (Horner over the bits of b).
__device__ __forceinline__ uint32_t gf2_mulmod_horner(uint32_t a, uint32_t b, uint32_t g, int order)
{
  uint32_t p = 0;
  for (int i = order - 1; i >= 0; --i) {
    p <<= 1;
    p ^= (p >> order) & 1u ? g : 0u;
    p ^= (b >> i) & 1u ? a : 0u;
  }
  return p;
}

// Transport-block join in the decoder (sink.tbs not null): codeblock cb's part of the TB is stored by its
// decoder, and the last codeblock of a TB to arrive forms the TB's result, so that nothing follows the
// decoder in a slot (a TB assembly and a result kernel after it, with two fills, took 16 to 20 us of a
// slot). First payload byte of the codeblock in the TB, and the bytes it stores.
__device__ __forceinline__ uint8_t* tb_part(const pg::ldpc_tb_sink& sink, const pg_tb_desc& t, const int cb, int& nb)
{
  const uint32_t off = (uint32_t)(cb - (int)t.cb_first) * t.cb_payload_bits / 8u; // whole bytes (checked by the host)
  const uint32_t all = t.tbs_bits / 8u;
  nb                 = (int)min((t.cb_payload_bits + 7u) / 8u, all > off ? all - off : 0u);
  return sink.tb_out + t.tb_out_offset + off;
}

// Called by the first warp when its thread 0 has stored iterations[cb] and added the codeblock's CRC.
__device__ __forceinline__ void tb_arrive(const pg::ldpc_tb_sink& sink, const pg_tb_desc& t, const uint32_t tb,
                                          const int32_t* iterations)
{
  const int lane = threadIdx.x & 31;
  int       last = 0;
  if (lane == 0) {
    __threadfence();
    last = atomicAdd(&sink.arrivals[tb], 1) == (int)t.nof_cbs - 1;
  }
  if (__shfl_sync(0xffffffffu, last, 0) == 0) {
    return;
  }
  __threadfence();
  // pusch_decoder_result: C == 1, the codeblock CRC is the TB CRC; C > 1, every codeblock CRC and the TB
  // CRC. A failed codeblock counts max_iterations (pusch_decoder_impl.cpp:612-710).
  const uint32_t maxit = sink.ues[tb].max_iterations;
  uint32_t       ok = 0, sum = 0, mx = 0;
  for (uint32_t c = lane; c < t.nof_cbs; c += 32) {
    const int32_t  it  = __ldcg(iterations + t.cb_first + c);
    const uint32_t run = it > 0 ? (uint32_t)it : maxit;
    ok += it > 0 ? 1u : 0u;
    sum += run;
    mx = max(mx, run);
  }
  ok  = __reduce_add_sync(0xffffffffu, ok);
  sum = __reduce_add_sync(0xffffffffu, sum);
  mx  = __reduce_max_sync(0xffffffffu, mx);
  if (lane == 0) {
    const uint32_t crc   = __ldcg(&sink.crc[tb]);
    pg_sch_result  r;
    r.tb_crc_ok          = (ok == t.nof_cbs && (t.nof_cbs == 1 || crc == 0)) ? 1u : 0u;
    r.nof_cbs            = t.nof_cbs;
    r.nof_cbs_crc_ok     = ok;
    r.mean_iterations    = (float)sum / (float)t.nof_cbs;
    r.max_iterations_run = mx;
    sink.results[tb]     = r;
  }
}

// Decodes codeblock cb (even Z <= 2 NT / T) with T threads per lane pair; smem: smem_bytes of dynamic
// shared memory (at least kPairMinSmem); slab: the CTA's global message slab.
template <int T, int NT>
__device__ __forceinline__ void decode_codeblock_pair(const pg_ldpc_cb& d, pair_shared& sh, unsigned char* smem,
                                                      const uint32_t smem_bytes, const int8_t* __restrict__ llrs,
                                                      uint8_t* __restrict__ bits, int32_t* __restrict__ iterations,
                                                      uint32_t* slab, const uint32_t* __restrict__ crc_pow,
                                                      const int cb, const pg::ldpc_tb_sink& sink)
{
  constexpr int LG  = T == 2 ? 0 : 1; // index of the T-dependent tables
  const int     tid = threadIdx.x;
  const int     bg  = d.base_graph;
  const int     Z   = (int)d.lifting_size;
  const int     H   = Z >> 1;
  const int     set = dev_set_index(Z);
  if ((bg != 1 && bg != 2) || set < 0) {
    if (tid == 0) {
      iterations[cb] = -1;
    }
    return;
  }
  const int          g        = bg - 1;
  const int          Kb       = bg == 1 ? 22 : 10;
  const int          nrows    = bg == 1 ? pg::kBg1Rows : pg::kBg2Rows;
  const int          nfull    = bg == 1 ? 68 : 52;
  const int          msg_len  = Kb * Z;
  const int          n        = (int)d.nof_llrs;
  const int8_t*      in       = llrs + d.llr_offset;
  int                nbytes   = (msg_len + 7) / 8;
  uint8_t*           out      = bits + d.out_offset;
  uint32_t           tbi      = 0; // TB of the codeblock
  pg_tb_desc         td       = {};
  if (sink.tbs != nullptr) {
    tbi = sink.cbs[cb].tb;
    td  = sink.tbs[tbi];
    out = tb_part(sink, td, cb, nbytes);
  }
  const int          crc_poly = d.crc_poly;
  const uint32_t     h4       = 4u * (uint32_t)H;
  const pair_tables& tb       = g_pair_tables;
  uint4*             tab      = reinterpret_cast<uint4*>(smem);
  unsigned char*     E        = smem + kPairTabBytes; // the constant column, then the graph's columns
  const uint32_t     tab_s    = (uint32_t)__cvta_generic_to_shared(tab);
  const uint32_t     E_s      = (uint32_t)__cvta_generic_to_shared(E);
  const int          nta      = (T * H + 31) & ~31;   // threads of the rows (whole warps)
  const bool         active   = tid < T * H;
  const uint32_t     jp       = (uint32_t)(active ? tid / T : H - 1);

  // Edge table of this lifting size, row list, constant column. Meets the soft bits' loads below at one
  // barrier.
  for (int p = tid; p < tb.pad_e0[LG][g][nrows]; p += NT) {
    const uint32_t c  = tb.pad_col[LG][g][p];
    const uint32_t s  = (uint32_t)tb.pad_v[LG][g][p][set] % (uint32_t)Z;
    const bool     up = s >= (uint32_t)H;
    const uint32_t sp = up ? s - (uint32_t)H : s;
    // {shared address of (col, s'), 1 - (H - s') as a float, selector 0x3210 or (swapped) 0x1032, its change when
    // the edge wraps (sign and magnitude)}; the constant column's edges never wrap.
    tab[p] = c == 0u ? make_uint4(E_s, __float_as_uint(-1024.f), 0x3210u, 0u)
                     : make_uint4(E_s + h4 * c + 4u * sp, __float_as_uint(1.f - (float)(H - (int)sp)),
                                  up ? 0x1032u : 0x3210u, up ? 0x21deu : 0x800021deu);
  }
  for (int r = tid; r < nrows; r += NT) {
    const int p0 = tb.pad_e0[LG][g][r], p1 = tb.pad_e0[LG][g][r + 1];
    sh.row[r] = make_uint4(tab_s + 16u * (uint32_t)p0, 4u * (uint32_t)(nta * tb.msg0[LG][g][r]), (uint32_t)((p1 - p0) / T),
                           tb.row_sync[g][r] != 0 ? (uint32_t)nta : 0u);
  }
  for (int k = tid; k < H; k += NT) {
    reinterpret_cast<uint32_t*>(E)[k] = kH8192;
  }
  if (tid == 0) {
    sh.tb_crc = 0;
    sh.crc[0] = sh.crc[1] = 0;
    sh.zero[0] = sh.zero[1] = 0;
  }

  // Everything above reads descriptors and tables that no kernel ahead in the stream writes.
  pg::wait_prerequisites();
  // Soft bits as f16 pairs (2Z punctured zeros, then the input): eight pairs per thread step when
  // the node halves are multiples of eight lanes, else one.
  {
    const int nof_full = (n / Z) * Z;
    const int ncols    = min(nfull, max((n + Z - 1) / Z + 2, Kb + 4)); // the columns that the rows can use
    int       last = 0, ragged = 0;
    uint32_t* E0 = reinterpret_cast<uint32_t*>(E) + H;
    if ((H & 7) == 0) {
      const int      per_col = H >> 3;
      const int      nchunks = ncols * per_col;
      const uint32_t inv     = 0xffffffffu / (uint32_t)per_col + 1u;
      const bool     aligned = (reinterpret_cast<uintptr_t>(in) & 7u) == 0;
      for (int q0 = tid; q0 < nchunks; q0 += kFetchBatch * NT) {
        // The batch's aligned whole-node loads are issued together; other pieces are read when they are used.
        uint2 raw[kFetchBatch][2];
        int   pos[kFetchBatch];
#pragma unroll
        for (int u = 0; u < kFetchBatch; ++u) {
          const int q   = q0 + u * NT;
          const int col = per_col == 1 ? q : (int)__umulhi((uint32_t)q, inv);
          const int k   = (col - 2) * Z + (q - col * per_col) * 8;
          pos[u]        = q < nchunks ? k : INT_MIN;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            raw[u][i] = make_uint2(0u, 0u);
            if (fetch_whole(k + i * H, nof_full, aligned) && q < nchunks) {
              raw[u][i] = pg::load_written(reinterpret_cast<const uint2*>(in + k + i * H));
            }
          }
        }
#pragma unroll
        for (int u = 0; u < kFetchBatch; ++u) {
          if (pos[u] == INT_MIN) {
            break;
          }
          const int q   = q0 + u * NT;
          const int col = per_col == 1 ? q : (int)__umulhi((uint32_t)q, inv);
          uint32_t  l0, l1, u0, u1;
          fetch8(in, pos[u], n, nof_full, aligned, raw[u][0], last, ragged, l0, l1);
          fetch8(in, pos[u] + H, n, nof_full, aligned, raw[u][1], last, ragged, u0, u1);
          const uint32_t p0 = __byte_perm(l0, u0, 0x5140), p1 = __byte_perm(l0, u0, 0x7362);
          const uint32_t p2 = __byte_perm(l1, u1, 0x5140), p3 = __byte_perm(l1, u1, 0x7362);
          uint32_t*      o = E0 + col * H + (q - col * per_col) * 8;
          *reinterpret_cast<uint4*>(o) =
              make_uint4(bytes_to_h2(p0), bytes_to_h2(p0 >> 16), bytes_to_h2(p1), bytes_to_h2(p1 >> 16));
          *reinterpret_cast<uint4*>(o + 4) =
              make_uint4(bytes_to_h2(p2), bytes_to_h2(p2 >> 16), bytes_to_h2(p3), bytes_to_h2(p3 >> 16));
        }
      }
    } else {
      const int      nwords = ncols * H;
      const uint32_t inv    = 0xffffffffu / (uint32_t)H + 1u;
#pragma unroll 4
      for (int q = tid; q < nwords; q += NT) {
        const int col = H == 1 ? q : (int)__umulhi((uint32_t)q, inv);
        const int k   = (col - 2) * Z + (q - col * H);
        int       x[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int kk = k + i * H;
          x[i]         = (kk >= 0 && kk < n) ? pg::load_written(in + kk) : 0;
          last         = x[i] != 0 ? max(last, kk + 1) : last;
          if (kk < nof_full) {
            x[i] = max(-64, min(64, x[i]));
          } else {
            ragged |= (abs(x[i]) > 120 && abs(x[i]) < 127) ? 1 : 0;
          }
        }
        E0[q] = bytes_to_h2((uint32_t)(x[0] + 128) | ((uint32_t)(x[1] + 128) << 8));
      }
    }
    last = __reduce_max_sync(0xffffffffu, last);
    ragged = __any_sync(0xffffffffu, ragged);
    if ((tid & 31) == 0) {
      sh.seen[tid >> 5] = 2 * last + (ragged != 0 ? 1 : 0);
    }
  }
  __syncthreads();

  int input_size = 0, ragged_any = 0;
#pragma unroll
  for (int w = 0; w < NT / 32; ++w) {
    input_size = max(input_size, sh.seen[w] >> 1);
    ragged_any |= sh.seen[w] & 1;
  }
  if (input_size < msg_len) {
    for (int b = tid; b < nbytes; b += NT) {
      out[b] = 0xff;
    }
    if (tid == 0) {
      iterations[cb] = 0;
    }
    if (sink.tbs != nullptr && tid < 32) {
      tb_arrive(sink, td, tbi, iterations);
    }
    return;
  }
  int cb_len = max(input_size + 2 * Z, (Kb + 4) * Z);
  cb_len     = ((cb_len + Z - 1) / Z) * Z;
  const int      nof_layers = min(cb_len / Z - Kb, nrows);
  const bool     ragged     = ragged_any != 0;
  const int      order      = crc_poly == PG_CRC16 ? 16 : 24;
  const uint32_t* pow_tab   = crc_pow + (size_t)(crc_poly <= PG_CRC24B ? crc_poly : 0) * pg::kCrcPowLen;
  const int      crc_len    = msg_len - (int)d.nof_filler_bits;

  // Messages: behind the columns of the rows that run (the columns past them hold only zeros).
  const uint32_t o_msg    = kPairTabBytes + ((h4 * (uint32_t)(1 + Kb + nof_layers) + 15u) & ~15u);
  const bool     in_smem  = o_msg + 4u * (uint32_t)nta * tb.msg0[LG][g][nof_layers] <= smem_bytes;
  const msg_shared msg_s{tab_s + o_msg};
  const msg_global msg_g{reinterpret_cast<unsigned char*>(slab)};

  int       result = 0;
  const int max_it = d.max_iterations;
  const int lane   = tid & 31;
  const int tpart  = tid % T;
  const int cgrp   = tid / H; // column group of the hard-decision phase
  const int ngrp   = NT / H;
  const uint32_t tpart16 = 16u * (uint32_t)tpart;
  const float jf   = (float)jp; // lane pair, its byte offset and -4 H as denormals (pair_edge)
  const float j4d  = __uint_as_float(4u * jp);
  const float nh4d = __uint_as_float(0x80000000u | h4);
  for (int it = 0; it < max_it; ++it) {
    if (tid < nta) {
      if (it > 0) {
        if (in_smem) {
          pair_rows<false, T>(sh, nof_layers, tpart16, jf, j4d, nh4d, msg_s, active);
        } else {
          pair_rows<false, T>(sh, nof_layers, tpart16, jf, j4d, nh4d, msg_g, active);
        }
      } else if (!ragged) {
        if (in_smem) {
          pair_rows<true, T>(sh, nof_layers, tpart16, jf, j4d, nh4d, msg_s, active);
        } else {
          pair_rows<true, T>(sh, nof_layers, tpart16, jf, j4d, nh4d, msg_g, active);
        }
      } else {
        uint32_t* const msg = in_smem ? reinterpret_cast<uint32_t*>(smem + o_msg) : slab;
        uint32_t        sync = 0;
        for (int r = 0; r < nof_layers; ++r) {
          const uint4 rd = sh.row[r];
          const int   ne = (int)rd.z;
          pair_row_ragged<T>(ne, rd.x + tpart16 * ne, jf, j4d, nh4d, msg + rd.y / 4 + tid * ((ne + 1) / 2), active, sync);
          sync = rd.w;
        }
      }
    }
    __syncthreads();

    // Hard decisions (soft <= 0), zero check and CRC: lane pair k of every ngrp-th message column; each
    // set bit within the CRC length adds x^e mod g.
    bool     zero = false;
    uint32_t crc  = 0;
    if (cgrp < ngrp) {
      const int       k  = tid - cgrp * H;
      const uint32_t* Ec = reinterpret_cast<const uint32_t*>(E) + H + k;
#pragma unroll 6
      for (int c = cgrp; c < Kb; c += ngrp) {
        const uint32_t x  = Ec[c * H];
        const int      i0 = c * Z + k, i1 = i0 + H;
        // The powers are loaded whatever the soft bits are, so that the loads of several columns overlap.
        const uint32_t q0 = crc_poly != PG_CRC_NONE && i0 < crc_len ? __ldg(pow_tab + (crc_len - 1 - i0 + order)) : 0u;
        const uint32_t q1 = crc_poly != PG_CRC_NONE && i1 < crc_len ? __ldg(pow_tab + (crc_len - 1 - i1 + order)) : 0u;
        zero |= (x & 0x7fffu) == 0 || (x & 0x7fff0000u) == 0;
        crc ^= pair_hard(x & 0xffffu) ? q0 : 0u;
        crc ^= pair_hard(x >> 16) ? q1 : 0u;
      }
    }
    crc  = __reduce_xor_sync(0xffffffffu, crc);
    zero = __any_sync(0xffffffffu, zero);
    if (lane == 0) {
      if (crc != 0) {
        atomicXor(&sh.crc[it & 1], crc);
      }
      if (zero) {
        sh.zero[it & 1] = 1;
      }
    }
    __syncthreads();
    const bool done = crc_poly != PG_CRC_NONE && sh.zero[it & 1] == 0 && sh.crc[it & 1] == 0;
    if (tid == 0) {
      sh.crc[(it + 1) & 1]  = 0; // last read before this iteration's rows
      sh.zero[(it + 1) & 1] = 0;
    }
    if (done) {
      result = it + 1;
      break;
    }
  }

  if (crc_poly == PG_CRC_NONE) {
    // Syndrome check over the processed rows (ldpc_decoder_impl.cpp:329-387), both lanes (the padding
    // edges read a positive soft bit). A zero soft bit of a row or of the message fails too.
    int bad = max_it > 0 ? sh.zero[(max_it - 1) & 1] : 1;
    if (active && tpart == 0) {
      for (int r = 0; r < nof_layers; ++r) {
        const uint4 rd     = sh.row[r];
        uint32_t    parity = 0;
        for (int e = 0; e < (int)rd.z * T; ++e) {
          uint32_t a, s;
          pair_edge(lds_v4(rd.x + 16 * e), jf, j4d, nh4d, a, s);
          const uint32_t x = __byte_perm(lds_u32(a), 0, s);
          bad |= ((x & 0x7fffu) == 0) | ((x & 0x7fff0000u) == 0);
          parity ^= (uint32_t)pair_hard(x & 0xffffu) | ((uint32_t)pair_hard(x >> 16) << 1);
        }
        bad |= parity != 0;
      }
    }
    bad    = __syncthreads_or(bad);
    result = !bad ? max_it : 0;
  }

  // Decoded bits: one 32-bit word per warp step, lane k holding bit 32 wi + k (MSB first after the
  // reversal); message bit i of column c = i / Z, lane w = i mod Z is half (w >= H) of E[c][w mod H].
  {
    const uint32_t inv = 0xffffffffu / (uint32_t)Z + 1u;
    for (int wi = tid >> 5; wi < (nbytes + 3) / 4; wi += NT / 32) {
      const int idx = 32 * wi + lane;
      bool      bit = false;
      if (idx < msg_len) {
        const int      col = (int)__umulhi((uint32_t)idx, inv);
        const int      w   = idx - col * Z;
        const uint32_t x   = reinterpret_cast<const uint32_t*>(E)[H + col * H + (w < H ? w : w - H)];
        bit                = pair_hard(w < H ? (x & 0xffffu) : (x >> 16));
      }
      const uint32_t wd = __brev(__ballot_sync(0xffffffffu, bit));
      if (lane < 4 && 4 * wi + lane < nbytes) {
        out[4 * wi + lane] = (uint8_t)(wd >> (24 - 8 * lane));
      }
    }
  }
  if (sink.tbs != nullptr && td.nof_cbs > 1 && result > 0) {
    // The payload's remainder, shifted to its place in the TB.
    const uint32_t* ptab = crc_pow + (size_t)td.crc_poly * pg::kCrcPowLen;
    const int       P    = (int)td.cb_payload_bits;
    uint32_t        crc  = 0;
    if (cgrp < ngrp) {
      const int       k  = tid - cgrp * H;
      const uint32_t* Ec = reinterpret_cast<const uint32_t*>(E) + H + k;
#pragma unroll 4
      for (int c = cgrp; c < Kb; c += ngrp) {
        const uint32_t x  = Ec[c * H];
        const int      i0 = c * Z + k, i1 = i0 + H;
        if (pair_hard(x & 0xffffu) && i0 < P) {
          crc ^= __ldg(ptab + (P - 1 - i0));
        }
        if (pair_hard(x >> 16) && i1 < P) {
          crc ^= __ldg(ptab + (P - 1 - i1));
        }
      }
    }
    crc = __reduce_xor_sync(0xffffffffu, crc);
    if (lane == 0 && crc != 0) {
      atomicXor(&sh.tb_crc, crc);
    }
    __syncthreads();
    if (tid == 0) {
      uint32_t gp;
      int      go;
      pg::crc_poly_params((int)td.crc_poly, &gp, &go);
      atomicXor(&sink.crc[tbi], gf2_mulmod_horner(sh.tb_crc, sink.cbs[cb].factor, gp, go));
    }
  }
  if (tid == 0) {
    iterations[cb] = result;
  }
  if (sink.tbs != nullptr && tid < 32) {
    __syncwarp();
    tb_arrive(sink, td, tbi, iterations);
  }
}

constexpr int kPairPerSm   = 2;
constexpr int kPairMaxSmem = 227 * 1024 - (((int)sizeof(pair_shared) + 15) & ~15); // dynamic, one CTA per SM

// Dynamic shared memory of a launch with per_sm CTAs on each SM (228 KB, 1 KB of it reserved per CTA).
int pair_smem(int per_sm)
{
  const int share = 228 * 1024 / per_sm - 1024 - (((int)sizeof(pair_shared) + 15) & ~15);
  return std::min(share, kPairMaxSmem) & ~127;
}
static_assert(kPairMinSmem + 2048 <= 228 * 1024 / kPairPerSm, "every column fits next to the other CTAs");

// Persistent decoder of a work list, every lifting size: each CTA takes codeblock order[w] (or w), w
// its own index first, then from *counter (zero before the launch when n exceeds the grid). Two
// threads per lane pair above Z = 192, four below; odd lifting sizes (Z <= 15) with the one-lane
// arithmetic.
//
// Bound: at 512 codeblocks instruction issue (71 % of the slots with 24 warps per SM), with few codeblocks
// latency (12 warps, 47 %). B200, against the kernel this one replaced (two lanes per thread, one thread per
// lane pair, Z = 384 only, messages in L2): 512 codeblocks BG1/BG2 Z = 384, 528 -> 327 us; 6 codeblocks BG1
// Z = 384, 257 -> 123 us; 200 codeblocks of many sizes, 302 -> 134 us. One thread per lane pair (192 threads,
// three CTAs per SM) took 415, 200 and 268 us where this split took 364, 155 and 190. From there: the step's
// barrier moved behind the next row's tables and messages 336, 138 and 156 us; message addresses of their
// space (shared or global) in place of generic ones 330, 128 and 137; the table and the soft bits loaded in one
// latency, the CRC powers by address alone 327, 123 and 134.
__global__ void __launch_bounds__(kPairThreads, kPairPerSm)
    ldpc_decode_pair_kernel(const pg_ldpc_cb* __restrict__ descs, const int8_t* __restrict__ llrs,
                            uint8_t* __restrict__ bits, int32_t* __restrict__ iterations, int8_t* __restrict__ c2v_all,
                            const uint32_t* __restrict__ crc_pow, const uint32_t* __restrict__ order, int n,
                            int* __restrict__ counter, uint32_t smem_bytes, const __grid_constant__ pg::ldpc_tb_sink sink,
                            const __grid_constant__ desc_args<kDecodeArgs> args)
{
  extern __shared__ __align__(16) unsigned char smem_pair[];
  __shared__ pair_shared sh;
  constexpr int NT   = kPairThreads;
  uint32_t*     slab = reinterpret_cast<uint32_t*>(c2v_all + (size_t)blockIdx.x * pg::kPairSlab);
  for (int w = blockIdx.x; w < n;) {
    const int        cb = order != nullptr ? (int)order[w] : w;
    const pg_ldpc_cb d  = descs != nullptr ? descs[cb] : args.cb[cb];
    const int        Z  = d.lifting_size;
    if ((Z & 1) != 0 || Z < 2 || Z > pg::kMaxZ) {
      pg::wait_prerequisites();
      if (Z < kOddMaxZ) {
        using odd_smem = smem_scalar_t<NT, kOddMaxZ>;
        static_assert(sizeof(odd_smem) + pg::kBg1Edges * kOddMaxZ <= kPairMinSmem, "messages behind the soft bits");
        decode_codeblock<0, NT, kOddMaxZ>(d, *reinterpret_cast<odd_smem*>(smem_pair), llrs, bits, iterations,
                                          reinterpret_cast<int8_t*>(smem_pair) + sizeof(odd_smem), crc_pow, cb, 0);
        if (sink.tbs != nullptr) {
          // A TB of one codeblock (checked by the host): its bytes are the first of the decoded bits.
          const uint32_t   tb = sink.cbs[cb].tb;
          const pg_tb_desc td = sink.tbs[tb];
          int              nb;
          uint8_t*         out = tb_part(sink, td, cb, nb);
          __syncthreads();
          for (int b = threadIdx.x; b < nb; b += NT) {
            out[b] = bits[d.out_offset + b];
          }
          if (threadIdx.x < 32) {
            tb_arrive(sink, td, tb, iterations);
          }
        }
      } else if (threadIdx.x == 0) {
        iterations[cb] = -1;
      }
    } else if (Z <= NT / 2) {
      decode_codeblock_pair<4, NT>(d, sh, smem_pair, smem_bytes, llrs, bits, iterations, slab, crc_pow, cb, sink);
    } else {
      decode_codeblock_pair<2, NT>(d, sh, smem_pair, smem_bytes, llrs, bits, iterations, slab, crc_pow, cb, sink);
    }
    if (n <= (int)gridDim.x) {
      break;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      sh.work = (int)gridDim.x + atomicAdd(counter, 1);
    }
    __syncthreads();
    w = sh.work;
  }
  // The arrivals of the ordering launch ahead of this one. Its last CTA clears them too, but knows that it is the
  // last from the count: cleared here, a count that was off (ordering launches that ran at the same time, from
  // replays of captured decodes) spoils no later batch.
  if (order != nullptr && blockIdx.x == 0 && threadIdx.x == 0) {
    counter[1] = 0;
  }
}

// Longest-first work order of a batch for the persistent decoders. A codeblock's expected decoding
// time is its work per iteration (the edges of the check rows its input reaches, as the decoder
// counts them from the last non-zero LLR, times Z) times the iterations it needs, which fall as its
// information per message bit rises: the sum of its LLR magnitudes over its K = Kb Z message bits
// (the mean LLR magnitude over the code rate; on the 512-codeblock BG1/BG2 batch the iterations
// correlate with it at -0.9 within each graph). Cost = edges Z K / sum |LLR|; the key is
// 255 - 16 log2(1 + cost), clamped to 0..255 (no non-zero LLR: 255), and the order lists the
// codeblocks by ascending key, so that the long decodes start first and the short ones fill the
// tail. The order only schedules: every codeblock's result is independent of it. One CTA per
// codeblock reads its whole input, 16 bytes per load in the aligned body.
constexpr int kScoreThreads = 512; // launch of 200 and 512 codeblocks, us: 128 threads 9.8 and 14.1, 256 6.8 and
                                   // 9.5, 512 5.9 and 9.5, 1024 6.2 and 10.9

__device__ __forceinline__ void score_word(uint32_t w, int idx, uint32_t& sum, uint32_t& cnt, int& last)
{
  const uint32_t a  = __vabsss4(w);                    // |x| per byte (saturating, -128 -> 127)
  const uint32_t nz = __vcmpne4(w, 0u) & 0x01010101u;  // 1 per non-zero byte
  sum               = __dp4a(a, 0x01010101u, sum);
  cnt               = __dp4a(nz, 0x01010101u, cnt);
  if (w != 0) {
    last = max(last, idx + 4 - (__clz(w) >> 3));     // one past the highest non-zero byte
  }
}

//
// The descriptors come from device memory (N = 1) or with the launch's arguments, and are then stored to
// `store` for the decoder. The last CTA to finish sorts the keys (a counting sort) into order[0 .. n) and
// leaves both counters (work counter, arrivals) at zero for the decoder and the next launch. Staging the
// descriptors by a copy, a sort launch and a memset of the work counter put the decoder 20 us behind the call
// instead of 10 (200 codeblocks).
template <int N>
__global__ void __launch_bounds__(kScoreThreads) ldpc_score_kernel(const pg_ldpc_cb* __restrict__ descs, int n,
                                                                  const int8_t* __restrict__ llrs, uint8_t* keys,
                                                                  uint32_t* __restrict__ order, int* counters,
                                                                  pg_ldpc_cb* __restrict__ store,
                                                                  const __grid_constant__ desc_args<N> args)
{
  __shared__ uint32_t s_red[3][kScoreThreads / 32];
  __shared__ int      s_last;
  const pg_ldpc_cb d    = N > 1 ? args.cb[blockIdx.x] : descs[blockIdx.x];
  const int8_t*    in   = llrs + d.llr_offset;
  if (N > 1 && threadIdx.x == 0) {
    store[blockIdx.x] = d;
  }
  const int        len  = (int)d.nof_llrs;
  const int        head = min(len, (int)((16u - (unsigned)(reinterpret_cast<uintptr_t>(in) & 15u)) & 15u));
  const int        nvec = (len - head) / 16;
  uint32_t         sum = 0, cnt = 0;
  int              last = 0;
  for (int k = threadIdx.x; k < head; k += kScoreThreads) {
    score_word((uint32_t)(uint8_t)__ldg(in + k), k, sum, cnt, last);
  }
  const uint4* body = reinterpret_cast<const uint4*>(in + head);
  for (int q = threadIdx.x; q < nvec; q += kScoreThreads) {
    const uint4 v  = __ldg(body + q);
    const int   k0 = head + 16 * q;
    score_word(v.x, k0, sum, cnt, last);
    score_word(v.y, k0 + 4, sum, cnt, last);
    score_word(v.z, k0 + 8, sum, cnt, last);
    score_word(v.w, k0 + 12, sum, cnt, last);
  }
  for (int k = head + 16 * nvec + threadIdx.x; k < len; k += kScoreThreads) {
    score_word((uint32_t)(uint8_t)__ldg(in + k), k, sum, cnt, last);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    last = max(last, __shfl_xor_sync(0xffffffffu, last, o));
  }
  if ((threadIdx.x & 31) == 0) {
    s_red[0][threadIdx.x >> 5] = sum;
    s_red[1][threadIdx.x >> 5] = cnt;
    s_red[2][threadIdx.x >> 5] = (uint32_t)last;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t ts = 0, tc = 0;
    int      tl = 0;
    for (int w = 0; w < kScoreThreads / 32; ++w) {
      ts += s_red[0][w];
      tc += s_red[1][w];
      tl = max(tl, (int)s_red[2][w]);
    }
    uint32_t key = 255u;
    if (tc > 0) {
      const int   Z    = max(1, (int)d.lifting_size);
      const int   Kb   = d.base_graph == 1 ? 22 : 10;
      const int   nr   = d.base_graph == 1 ? pg::kBg1Rows : pg::kBg2Rows;
      const int   rows  = min(max((tl + 2 * Z) / Z, Kb + 4) - Kb, nr);
      const int   edges = c_row_e0[d.base_graph == 2 ? 1 : 0][rows];
      const float cost  = (float)edges * (float)Z * (float)(Kb * Z) / (float)max(ts, 1u);
      key               = 255u - (uint32_t)min(255.f, 16.f * log2f(1.f + cost));
    }
    keys[blockIdx.x] = (uint8_t)key;
    __threadfence();
    s_last = atomicAdd(&counters[1], 1) == n - 1;
  }
  __syncthreads();
  if (!s_last) {
    return;
  }
  __threadfence();
  if (threadIdx.x == 0) {
    counters[0] = 0;
    counters[1] = 0;
  }
  __shared__ uint32_t bin[256];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) {
    bin[i] = 0;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    atomicAdd(&bin[__ldcg(keys + k)], 1u);
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    // Exclusive prefix sum of the 256 bins: eight per lane, then across the warp.
    uint32_t v[8], t = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      v[i] = bin[8 * threadIdx.x + i];
      t += v[i];
    }
    uint32_t inc = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
      inc += threadIdx.x >= (unsigned)o ? y : 0u;
    }
    uint32_t run = inc - t;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      bin[8 * threadIdx.x + i] = run;
      run += v[i];
    }
  }
  __syncthreads();
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    order[atomicAdd(&bin[__ldcg(keys + k)], 1u)] = (uint32_t)k;
  }
}

} // namespace

// Check-to-variable scratch of pg_ldpc_decode_batch_static_scratch (described with that entry).
static __device__ __align__(256) int8_t g_static_c2v[(size_t)PG_STATIC_SCRATCH_MAX_CODEBLOCKS * pg::kC2vStride];

namespace pg {

int lifting_set_index(int Z)
{
  static const int a_tab[8] = {2, 3, 5, 7, 9, 11, 13, 15};
  if (Z < 2 || Z > kMaxZ) {
    return -1;
  }
  for (int i = 0; i < 8; ++i) {
    int t = Z;
    while ((t % 2) == 0 && t > a_tab[i]) {
      t /= 2;
    }
    if (t == a_tab[i]) {
      return i;
    }
  }
  return -1;
}

int ldpc_upload_tables(pg_context* ctx)
{
  uint8_t  col[2][kBg1Edges] = {};
  uint16_t v[2][kBg1Edges][8] = {};
  uint8_t  deg[2][kBg1Rows]   = {};
  for (int e = 0; e < PG_BG1_EDGES; ++e) {
    col[0][e] = PG_BG1_EDGE_COL[e];
    for (int s = 0; s < 8; ++s) {
      v[0][e][s] = PG_BG1_EDGE_V[e][s];
    }
  }
  for (int e = 0; e < PG_BG2_EDGES; ++e) {
    col[1][e] = PG_BG2_EDGE_COL[e];
    for (int s = 0; s < 8; ++s) {
      v[1][e][s] = PG_BG2_EDGE_V[e][s];
    }
  }
  for (int r = 0; r < PG_BG1_ROWS; ++r) {
    deg[0][r] = PG_BG1_ROW_DEG[r];
  }
  for (int r = 0; r < PG_BG2_ROWS; ++r) {
    deg[1][r] = PG_BG2_ROW_DEG[r];
  }
  int rc = check_cuda(ctx, cudaMemcpyToSymbol(c_edge_col, col, sizeof(col)), "cudaMemcpyToSymbol(edge_col)");
  if (rc == PG_OK) {
    rc = check_cuda(ctx, cudaMemcpyToSymbol(c_edge_v, v, sizeof(v)), "cudaMemcpyToSymbol(edge_v)");
  }
  if (rc == PG_OK) {
    rc = check_cuda(ctx, cudaMemcpyToSymbol(c_row_deg, deg, sizeof(deg)), "cudaMemcpyToSymbol(row_deg)");
  }
  // Layer steps: greedy runs of consecutive rows with pairwise disjoint columns.
  uint8_t  step_row0[2][kBg1Rows] = {}, step_nrows[2][kBg1Rows] = {}, nsteps[2] = {};
  uint16_t row_e0[2][kBg1Rows + 1] = {};
  for (int gi = 0; gi < 2; ++gi) {
    const int rows = gi == 0 ? PG_BG1_ROWS : PG_BG2_ROWS;
    for (int r = 0; r < rows; ++r) {
      row_e0[gi][r + 1] = (uint16_t)(row_e0[gi][r] + deg[gi][r]);
    }
    uint64_t used[2] = {0, 0}; // columns 0..67 of the current step
    int      ns      = 0;
    for (int r = 0; r < rows; ++r) {
      uint64_t cols[2] = {0, 0};
      for (int e = row_e0[gi][r]; e < row_e0[gi][r + 1]; ++e) {
        cols[col[gi][e] >> 6] |= 1ull << (col[gi][e] & 63);
      }
      if (r == 0 || (cols[0] & used[0]) != 0 || (cols[1] & used[1]) != 0) {
        step_row0[gi][ns]  = (uint8_t)r;
        step_nrows[gi][ns] = 1;
        ++ns;
        used[0] = cols[0];
        used[1] = cols[1];
      } else {
        ++step_nrows[gi][ns - 1];
        used[0] |= cols[0];
        used[1] |= cols[1];
      }
    }
    nsteps[gi] = (uint8_t)ns;
  }
  if (rc == PG_OK) {
    rc = check_cuda(ctx, cudaMemcpyToSymbol(c_step_row0, step_row0, sizeof(step_row0)), "cudaMemcpyToSymbol(steps)");
  }
  if (rc == PG_OK) {
    rc = check_cuda(ctx, cudaMemcpyToSymbol(c_step_nrows, step_nrows, sizeof(step_nrows)), "cudaMemcpyToSymbol(steps)");
  }
  if (rc == PG_OK) {
    rc = check_cuda(ctx, cudaMemcpyToSymbol(c_nsteps, nsteps, sizeof(nsteps)), "cudaMemcpyToSymbol(steps)");
  }
  if (rc == PG_OK) {
    rc = check_cuda(ctx, cudaMemcpyToSymbol(c_row_e0, row_e0, sizeof(row_e0)), "cudaMemcpyToSymbol(row_e0)");
  }
  // Formed by the first call (the values are the same in every one), while calls of other threads wait.
  static const pair_tables tables = [&] {
    pair_tables pt = {};
    for (int gi = 0; gi < 2; ++gi) {
      const int rows = gi == 0 ? PG_BG1_ROWS : PG_BG2_ROWS;
      for (int r = 0; r < rows; ++r) {
        for (int lg = 0; lg < 2; ++lg) {
          const int t                = 2 << lg;
          const int ne               = (deg[gi][r] + t - 1) / t;
          pt.pad_e0[lg][gi][r + 1]   = (uint16_t)(pt.pad_e0[lg][gi][r] + ne * t);
          pt.msg0[lg][gi][r + 1]     = (uint16_t)(pt.msg0[lg][gi][r] + (ne + 1) / 2);
          for (int k = 0; k < deg[gi][r]; ++k) {
            const int e = row_e0[gi][r] + k, p = pt.pad_e0[lg][gi][r] + k;
            pt.pad_col[lg][gi][p] = (uint8_t)(col[gi][e] + 1);
            std::copy(v[gi][e], v[gi][e] + 8, pt.pad_v[lg][gi][p]);
          }
        }
      }
      for (int st = 0; st < nsteps[gi]; ++st) {
        pt.row_sync[gi][step_row0[gi][st] + step_nrows[gi][st] - 1] = 1;
      }
    }
    return pt;
  }();
  if (rc == PG_OK) {
    rc = check_cuda(ctx, cudaMemcpyToSymbol(g_pair_tables, &tables, sizeof(tables)), "cudaMemcpyToSymbol(pair tables)");
  }
  if (rc == PG_OK) {
    rc = check_cuda(ctx,
                    cudaFuncSetAttribute(ldpc_decode_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kPairMaxSmem),
                    "cudaFuncSetAttribute(ldpc_decode_pair_kernel)");
  }
  if (rc == PG_OK) {
    // Device address of the static scratch on this context's device (current here), looked up
    // once so that the static-scratch entry makes no runtime call besides its launch.
    rc = check_cuda(ctx, cudaGetSymbolAddress((void**)&ctx->static_c2v, g_static_c2v),
                    "cudaGetSymbolAddress(static check-to-variable scratch)");
  }
  return rc;
}

int ldpc_launch(pg_context* ctx, const pg_ldpc_cb* descs_dev, int n, const int8_t* llrs, uint8_t* bits,
                int32_t* iterations, cudaStream_t stream, const pg_ldpc_cb* descs_host)
{
  return ldpc_launch_scratch(ctx, descs_dev, n, llrs, bits, iterations, ctx->dev.c2v, stream, descs_host);
}

// CTAs of the decoder the context's batch decodes launch for n codeblocks: one per SM up to one and three
// quarter codeblocks per SM (their messages then stay in shared memory), two per SM above. One against two
// per SM, whole calls: 200 codeblocks of many sizes 196 and 231 us; BG1/BG2 mixed, Z = 384, 222 codeblocks
// 228 and 299, 260 238 and 308, 350 300 and 291, 512 399 and 353; Z = 96, 200 codeblocks 153 and 160, 296
// 182 and 166.
static int batch_ctas(const pg_context* ctx, int n)
{
  const int per_sm = ctx->ldpc_ctas_per_sm > 0 ? ctx->ldpc_ctas_per_sm : (4 * n <= 7 * ctx->sm_count ? 1 : kPairPerSm);
  return std::min(n, ldpc_max_ctas(ctx, per_sm, ctx->ldpc_kernel));
}

int ldpc_max_ctas(const pg_context* ctx, int per_sm, int kernel)
{
  return kernel == PG_LDPC_KERNEL_ONE_LANE ? std::min(per_sm * ctx->sm_count, ctx->ldpc_ctas)
                                           : std::min(per_sm, kPairPerSm) * ctx->sm_count;
}

// Whether the batch decodes run n codeblocks in longest-first order. With a CTA for every codeblock all start
// at once, and their order decides nothing.
static bool batch_ordered(const pg_context* ctx, int n)
{
  return ctx->ldpc_order_mode == PG_LDPC_ORDER_LONGEST_FIRST && n > batch_ctas(ctx, n) && n <= ctx->max_codeblocks;
}

bool ldpc_descs_by_value(const pg_context* ctx, int n)
{
  return batch_ordered(ctx, n) ? n <= kScoreArgs : n <= kDecodeArgs && ctx->ldpc_kernel != PG_LDPC_KERNEL_ONE_LANE;
}

int ldpc_launch_scratch(pg_context* ctx, const pg_ldpc_cb* descs_dev, int n, const int8_t* llrs, uint8_t* bits,
                        int32_t* iterations, int8_t* c2v, cudaStream_t stream, const pg_ldpc_cb* descs_host)
{
  const uint32_t* order = nullptr;
  if (batch_ordered(ctx, n)) {
    if (int rc = ldpc_order_launch(ctx, descs_dev, n, llrs, ctx->dev.ldpc_keys, ctx->dev.ldpc_order,
                                   ctx->dev.ldpc_counter, stream, descs_host)) {
      return rc;
    }
    order      = ctx->dev.ldpc_order;
    descs_host = nullptr; // the ordering launch has stored them
  }
  return ldpc_launch_persistent(ctx, descs_dev, n, llrs, bits, iterations, c2v, order, ctx->dev.ldpc_counter, stream,
                                batch_ctas(ctx, n), ctx->ldpc_kernel, nullptr, order != nullptr, descs_host);
}

template <int N>
static void score_launch(pg_context* ctx, pg_ldpc_cb* descs_dev, int n, const int8_t* llrs, uint8_t* keys, uint32_t* order,
                         int* counters, cudaStream_t stream, const pg_ldpc_cb* descs_host)
{
  desc_args<N> args;
  if (descs_host != nullptr) {
    std::memcpy(args.cb, descs_host, (size_t)n * sizeof(pg_ldpc_cb));
  }
  ldpc_score_kernel<N><<<n, kScoreThreads, 0, stream>>>(N > 1 ? nullptr : descs_dev, n, llrs, keys, order, counters,
                                                       N > 1 ? descs_dev : nullptr, args);
}

int ldpc_order_launch(pg_context* ctx, const pg_ldpc_cb* descs_dev, int n, const int8_t* llrs, uint8_t* keys,
                      uint32_t* order, int* counters, cudaStream_t stream, const pg_ldpc_cb* descs_host)
{
  if (n <= 0) {
    return PG_OK;
  }
  pg_ldpc_cb* dev = const_cast<pg_ldpc_cb*>(descs_dev); // written only when the descriptors come from the host
  if (descs_host == nullptr) {
    score_launch<1>(ctx, dev, n, llrs, keys, order, counters, stream, nullptr);
  } else if (n <= kScoreArgs / 4) {
    score_launch<kScoreArgs / 4>(ctx, dev, n, llrs, keys, order, counters, stream, descs_host);
  } else if (n <= kScoreArgs / 2) {
    score_launch<kScoreArgs / 2>(ctx, dev, n, llrs, keys, order, counters, stream, descs_host);
  } else {
    score_launch<kScoreArgs>(ctx, dev, n, llrs, keys, order, counters, stream, descs_host);
  }
  return check_cuda(ctx, cudaGetLastError(), "ldpc_score_kernel launch");
}

unsigned int timing_record_flags(pg_context* ctx, cudaStream_t s)
{
  // Under stream capture the timing events become event-record nodes of the graph (external
  // records); a plain record there would only mark a capture dependency.
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  if (ctx->timed && cudaStreamIsCapturing(s, &capturing) == cudaSuccess &&
      capturing == cudaStreamCaptureStatusActive) {
    return cudaEventRecordExternal;
  }
  return cudaEventRecordDefault;
}

int ldpc_resident_ctas(pg_context* ctx)
{
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ldpc_decode_kernel, kThreads, 0) != cudaSuccess ||
      per_sm < 1) {
    (void)cudaGetLastError();
    per_sm = 1;
  }
  return per_sm * ctx->sm_count;
}

int ldpc_launch_persistent(pg_context* ctx, const pg_ldpc_cb* descs_dev, int n, const int8_t* llrs, uint8_t* bits,
                           int32_t* iterations, int8_t* c2v, const uint32_t* order, int* counter,
                           cudaStream_t stream, int max_ctas, int kernel, const ldpc_tb_sink* sink, bool counter_zero,
                           const pg_ldpc_cb* descs_host, bool overlap)
{
  if (n == 0) {
    return PG_OK;
  }
  const int grid = std::max(1, std::min(n, max_ctas));
  if (!counter_zero && (n > grid || kernel == PG_LDPC_KERNEL_ONE_LANE)) {
    if (int rc = check_cuda(ctx, cudaMemsetAsync(counter, 0, sizeof(int), stream), "cudaMemsetAsync(ldpc counter)")) {
      return rc;
    }
  }
  const unsigned int rec_flags = timing_record_flags(ctx, stream);
  if (ctx->timed) {
    cudaEventRecordWithFlags(ctx->ev_start, stream, rec_flags);
  }
  int rc = PG_OK;
  if (kernel != PG_LDPC_KERNEL_ONE_LANE) {
    const int smem = pair_smem((grid + ctx->sm_count - 1) / ctx->sm_count);
    desc_args<kDecodeArgs> args;
    if (descs_host != nullptr) {
      std::memcpy(args.cb, descs_host, (size_t)n * sizeof(pg_ldpc_cb));
    }
    const pg_ldpc_cb*  dev = descs_host != nullptr ? nullptr : descs_dev;
    const ldpc_tb_sink snk = sink != nullptr ? *sink : ldpc_tb_sink{};
    // Only with one CTA per SM: two are placed on the SMs that the kernel ahead leaves first, and the others
    // stay idle (104 to 148 codeblocks: 4 us less; 200 codeblocks: 60 us instead of 48).
    if (overlap && grid <= ctx->sm_count) {
      rc = check_cuda(ctx,
                      launch_overlapped(ldpc_decode_pair_kernel, grid, kPairThreads, (size_t)smem, stream, dev, llrs, bits,
                                        iterations, c2v, ctx->dev.crc_pow, order, n, counter, (uint32_t)smem, snk, args),
                      "ldpc_decode_pair_kernel launch");
    } else {
      ldpc_decode_pair_kernel<<<grid, kPairThreads, smem, stream>>>(dev, llrs, bits, iterations, c2v, ctx->dev.crc_pow,
                                                                    order, n, counter, (uint32_t)smem, snk, args);
      rc = check_cuda(ctx, cudaGetLastError(), "ldpc_decode_pair_kernel launch");
    }
  } else {
    ldpc_decode_kernel<<<grid, kThreads, 0, stream>>>(descs_dev, llrs, bits, iterations, c2v, ctx->dev.crc_pow, order,
                                                      n, counter);
    rc = check_cuda(ctx, cudaGetLastError(), "ldpc_decode_kernel launch");
  }
  if (ctx->timed) {
    cudaEventRecordWithFlags(ctx->ev_stop, stream, rec_flags);
  }
  return rc;
}

} // namespace pg

// ---------------------------------------------------------------------------------------------
// Decoding with a module-static check-to-variable scratch (pg_ldpc_decode_batch_static_scratch).
//
// Some callers cannot allocate device memory while they decode: a PHY worker that has to finish
// each slot by its deadline (cudaMalloc / cudaFree take driver locks and may synchronise the whole
// device, so their latency has no useful bound), and a process that reserved its device memory
// when it started and must not run into out-of-memory in the middle of traffic. For them the
// scratch is a device array of this module, reserved by the driver when the module loads: room for
// PG_STATIC_SCRATCH_MAX_CODEBLOCKS codeblocks of the largest graph (BG1, Z = 384).
//
// Nothing in the array has to start at zero: the first layered iteration of each codeblock writes
// every check-to-variable message of the rows it processes before any later iteration reads one,
// so what an earlier call left behind is never read. Every call on a device uses the same array;
// kernels of two calls that run at the same time race on it. The array's device address is
// looked up once per context, in ldpc_upload_tables (called by pg_create).

extern "C" int pg_ldpc_decode_batch_static_scratch(pg_context* ctx, const pg_ldpc_cb* cbs_dev, int nof_cbs,
                                                   const int8_t* llrs, uint8_t* bits, int32_t* iterations,
                                                   void* stream)
{
  if (ctx == nullptr) {
    return PG_ERR_INVALID;
  }
  if (nof_cbs < 0) {
    return pg::set_error(ctx, PG_ERR_INVALID, "negative codeblock count");
  }
  if (nof_cbs > PG_STATIC_SCRATCH_MAX_CODEBLOCKS) {
    return pg::set_error(ctx, PG_ERR_CAPACITY,
                         "batch of " + std::to_string(nof_cbs) + " codeblocks exceeds the static scratch limit of " +
                             std::to_string(PG_STATIC_SCRATCH_MAX_CODEBLOCKS) + " codeblocks per call");
  }
  if (nof_cbs == 0) {
    return PG_OK;
  }
  if (cbs_dev == nullptr || llrs == nullptr || bits == nullptr || iterations == nullptr) {
    return pg::set_error(ctx, PG_ERR_INVALID, "null device buffer");
  }
  int prev = -1;
  if (int rc = pg::check_cuda(ctx, cudaGetDevice(&prev), "cudaGetDevice")) {
    return rc;
  }
  if (prev != ctx->device) {
    if (int rc = pg::check_cuda(ctx, cudaSetDevice(ctx->device), "cudaSetDevice")) {
      return rc;
    }
  }
  const cudaStream_t s          = static_cast<cudaStream_t>(stream);
  const unsigned int rec_flags  = pg::timing_record_flags(ctx, s);
  if (ctx->timed) {
    cudaEventRecordWithFlags(ctx->ev_start, s, rec_flags);
  }
  ldpc_decode_kernel<<<nof_cbs, kThreads, 0, s>>>(cbs_dev, llrs, bits, iterations, ctx->static_c2v, ctx->dev.crc_pow,
                                                  nullptr, nof_cbs, nullptr);
  int rc = pg::check_cuda(ctx, cudaGetLastError(), "ldpc_decode_kernel launch (static scratch)");
  if (ctx->timed) {
    cudaEventRecordWithFlags(ctx->ev_stop, s, rec_flags);
  }
  if (prev != ctx->device) {
    cudaSetDevice(prev);
  }
  return rc;
}
