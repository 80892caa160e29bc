// Polar-coded UCI on PUSCH (HARQ-ACK or CSI Part 1 of 12 to 1706 bits): the reference's
// uci_decoder_impl::decode_codeword_polar (lib/phy/upper/channel_processors/uci/uci_decoder_impl.cpp:25-99)
// with its polar code construction (lib/phy/upper/channel_coding/polar/polar_code_impl.cpp:330-480),
// rate dematcher (polar_rate_dematcher_impl.cpp), simplified successive-cancellation decoder
// (polar_decoder_impl.cpp) and deallocator (polar_deallocator_impl.cpp), on the GPU.
//
// The host builds each codeblock's code (N, the information and parity-check sub-channels) once
// per call; one CTA decodes one message (a message longer than 359 bits with at least 1088 soft bits,
// or of 1013 bits and more, has two codeblocks). The CTA runs channel de-interleaving, bit selection
// and sub-block de-interleaving into the decoder's input in shared memory; then one warp per codeblock
// walks the rate-0, rate-1 and rate-R nodes depth first, with the f / g steps spread over the 32 lanes
// and codewords and decoded bits held as bit words, one word a lane, and runs the deallocation and the
// codeblock CRC. Every LLR operation is the reference's int8 arithmetic
// (log_likelihood_ratio: saturated sum at +-120 with +-127 as infinity, soft_xor, hard bit v <= 0,
// promotion sum on repetition).
#include "pg_internal.h"

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

namespace {

#include "polar_tables.inc"

__constant__ uint8_t c_polar_subblock[32] = {PG_POLAR_SUBBLOCK_PATTERN};

constexpr int kPolarNMax   = 1024; // polar_code::NMAX
constexpr int kPolarEMax   = 8192; // polar_code::EMAX
constexpr int kPolarNMaxLg = 10;   // uplink nMax
constexpr int kPolarMaxA   = 1706; // uci_decoder_impl MAX_CODEBLOCK_SIZE (TS 38.212 5.2.1)

// One codeblock as the decoding warp reads it.
struct polar_cb {
  uint32_t llr_offset; // first soft bit of the codeblock
  uint32_t E;          // rate-matched length (0: no codeblock)
  uint32_t out_offset; // first output byte of the payload bits
  uint16_t K;          // polar K: filler + payload + CRC bits
  uint16_t nbits;      // payload bits
  uint8_t  n;          // log2 N
  uint8_t  crc_size;   // 6 or 11
  uint8_t  nof_filler; // leading zero bits of the first codeblock
  uint8_t  reserved;
  uint16_t pc[4];      // sorted parity-check sub-channels, terminated by kPolarNMax
  uint32_t info[kPolarNMax / 32]; // K_set: sub-channels that carry payload, CRC, filler or parity bits
};
static_assert(sizeof(polar_cb) == 156, "polar_cb layout");

// The code of one codeblock: polar_code_impl::set_code_params (polar_code_impl.cpp:330-421) and
// polar_code_impl::set (:432-480) for nMax = 10 (uplink).
struct polar_code_host {
  int      n = 0, N = 0, K = 0, E = 0, nPC = 0, nWmPC = 0;
  uint16_t pc[4]                 = {kPolarNMax, kPolarNMax, kPolarNMax, kPolarNMax};
  uint32_t info[kPolarNMax / 32] = {};
};

uint16_t subblock_index(int j, int N)
{
  const int b = N / 32;
  return (uint16_t)(kPolarSubblock[(32 * j) / N] * b + j % b);
}

std::string polar_code_build(unsigned K, unsigned E, polar_code_host& c)
{
  if (E > (unsigned)kPolarEMax) {
    return "E above 8192";
  }
  if (K < 18 || (K > 25 && K < 31) || K > 1023) {
    return "K out of the uplink range (18..25, 31..1023)";
  }
  c.K     = (int)K;
  c.E     = (int)E;
  c.nPC   = K <= 25 ? 3 : 0;
  c.nWmPC = (K <= 25 && E > K + 189) ? 1 : 0;
  if (!(K + (unsigned)c.nPC < E)) {
    return "E not above K + nPC";
  }
  unsigned e = 1;
  for (; e <= 13; ++e) {
    if ((1u << e) >= E) {
      break;
    }
  }
  const unsigned n1 = ((8 * E <= 9 * (1u << (e - 1))) && (16 * K < 9 * E)) ? e - 1 : e;
  unsigned       k  = 0;
  for (; k <= 10; ++k) {
    if ((1u << k) >= K) {
      break;
    }
  }
  unsigned n = std::min(n1, k + 3);
  n          = std::min(n, (unsigned)kPolarNMaxLg);
  n          = std::max(n, 5u);
  c.n        = (int)n;
  c.N        = 1 << n;
  const int N = c.N;
  if (!((int)K < N)) {
    return "K not below N";
  }
  // The sequence for N (ascending reliability).
  std::vector<uint16_t> mother;
  mother.reserve(N);
  for (int i = 0; i < kPolarNMax; ++i) {
    if (kPolarQ[i] < N) {
      mother.push_back(kPolarQ[i]);
    }
  }
  const int             nk = (int)K + c.nPC;
  std::vector<uint16_t> kset(mother.end() - nk, mother.end());
  if (N > (int)E) {
    // Sub-channels frozen by puncturing or shortening, then the stable set difference that also
    // drops every index <= T (polar_code_impl.cpp:443-467, setdiff_stable :284-313).
    unsigned              T  = 0;
    const int             nf = N - (int)E;
    std::vector<uint16_t> fset(nf);
    if (16 * K <= 7 * E) {
      const unsigned nth = 3u * (unsigned)N / 4u;
      T                  = E >= nth ? nth - (E >> 1) - 1 : 9u * (unsigned)N / 16u - (E >> 2);
      for (int i = 0; i < nf; ++i) {
        fset[i] = subblock_index(i, N);
      }
    } else {
      for (int i = 0; i < nf; ++i) {
        fset[i] = subblock_index((int)E + i, N);
      }
    }
    std::vector<uint8_t> frozen(N, 0);
    for (const uint16_t x : fset) {
      frozen[x] = 1;
    }
    std::vector<uint16_t> kept;
    for (const uint16_t x : mother) {
      if (x <= T || frozen[x] != 0) {
        continue;
      }
      kept.push_back(x);
    }
    if ((int)kept.size() < nk) {
      return "too few sub-channels left after puncturing or shortening";
    }
    kset.assign(kept.end() - nk, kept.end());
  }
  // Parity-check sub-channels: the nPC - nWmPC least reliable of K_set, and 252 (K <= 21) or 248
  // for the minimum-weight one (polar_code_impl.cpp:469-480).
  for (int i = 0; i < c.nPC - c.nWmPC; ++i) {
    c.pc[i] = kset[i];
  }
  if (c.nWmPC == 1) {
    c.pc[c.nPC - 1] = K <= 21 ? 252 : 248;
  }
  std::sort(c.pc, c.pc + c.nPC);
  for (const uint16_t x : kset) {
    c.info[x >> 5] |= 1u << (x & 31);
  }
  return std::string();
}

// UCI segmentation and CRC size (include/ocudu/ran/uci/uci_info.h:22-47).
int uci_nof_codeblocks(unsigned A, unsigned E)
{
  return ((A >= 360 && E >= 1088) || A >= 1013) ? 2 : 1;
}
int uci_crc_size(unsigned A)
{
  return A < 12 ? 0 : (A < 20 ? 6 : 11);
}

// ---------------------------------------------------------------------------------------------
// Device side.

constexpr int kLlrMax = 120;
constexpr int kLlrInf = 127;

// log_likelihood_ratio::operator+ (lib/phy/upper/log_likelihood_ratio.cpp:21-55): opposite values
// give 0, an infinite term wins, otherwise the sum saturated at +-120.
__device__ __forceinline__ int llr_sat_sum(int a, int b)
{
  if (a == -b) {
    return 0;
  }
  if (a > kLlrMax || a < -kLlrMax) {
    return a;
  }
  if (b > kLlrMax || b < -kLlrMax) {
    return b;
  }
  return max(-kLlrMax, min(kLlrMax, a + b));
}

// log_likelihood_ratio::promotion_sum (log_likelihood_ratio.cpp:57-70): as the saturated sum, but a
// finite sum above 120 in magnitude becomes infinite.
__device__ __forceinline__ int llr_promotion_sum(int a, int b)
{
  if (a == -b) {
    return 0;
  }
  if (a > kLlrMax || a < -kLlrMax) {
    return a;
  }
  if (b > kLlrMax || b < -kLlrMax) {
    return b;
  }
  const int t = a + b;
  return t > kLlrMax ? kLlrInf : (t < -kLlrMax ? -kLlrInf : t);
}

// log_likelihood_ratio::soft_xor: sign(x y) min(|x|, |y|).
__device__ __forceinline__ int llr_soft_xor(int x, int y)
{
  const int m = min(abs(x), abs(y));
  return x * y < 0 ? -m : m;
}

constexpr int kPolarThreads = 128;

struct polar_cb_smem {
  int8_t   e[kPolarEMax];          // de-interleaved soft bits
  uint32_t in[kPolarEMax / 4 + 1]; // the received soft bits, then the deallocated message bits
  int8_t   llr[2 * kPolarNMax];    // stage s (5 .. n) at offset 2^s, 2^s values
  int      valid;
};

// Bits of a word of sub-channels re-encoded by the polar transform: bit i ^= bit i + st for st = 1, 2, ...
__device__ __forceinline__ uint32_t polar_transform_word(uint32_t x)
{
  x ^= (x >> 1) & 0x55555555u;
  x ^= (x >> 2) & 0x33333333u;
  x ^= (x >> 4) & 0x0f0f0f0fu;
  x ^= (x >> 8) & 0x00ff00ffu;
  x ^= x >> 16;
  return x;
}

__device__ __forceinline__ int llr_f(int x, int y)
{
  return (int)(int8_t)llr_soft_xor(x, y);
}

__device__ __forceinline__ int llr_g(int x, int y, uint32_t bit)
{
  return (int)(int8_t)llr_sat_sum(y, bit == 0 ? x : -x);
}

// One node of stage S <= 5 (polar_decoder_impl.cpp:163-252) in registers: lane i < 2^S holds the LLR of the
// node's element i, info its sub-channels' K_set bits; returns the node's codeword (bit i: element i) and
// in u its decoded sub-channel bits. The two children share one copy of the code.
template <int S>
__device__ __forceinline__ uint32_t polar_node(int l, uint32_t info, uint32_t& u)
{
  constexpr uint32_t m = S == 5 ? 0xffffffffu : (1u << (1 << (S < 5 ? S : 0))) - 1u;
  if (info == 0u) { // rate 0: zeros (:163-178)
    u = 0u;
    return 0u;
  }
  if (info == m) { // rate 1: hard decisions, re-encoded into the message bits (:180-205)
    const uint32_t e = __ballot_sync(0xffffffffu, l <= 0) & m;
    u                = polar_transform_word(e);
    return e;
  }
  if constexpr (S > 0) {
    constexpr int      h  = 1 << (S - 1);
    constexpr uint32_t mh = (1u << h) - 1u;
    const int          y  = __shfl_down_sync(0xffffffffu, l, h);
    int                lc = llr_f(l, y); // left child (:214-218)
    uint32_t           e0 = 0u, u0 = 0u;
#pragma unroll 1
    for (int half = 0;; ++half) {
      uint32_t       uc;
      const uint32_t e = polar_node<S - 1>(lc, half == 0 ? info & mh : info >> h, uc);
      if (half == 1) {
        u = u0 | (uc << h);
        return (e0 ^ e) | (e << h); // (:240-252)
      }
      e0 = e;
      u0 = uc;
      lc = llr_g(l, y, (e0 >> (threadIdx.x & 31)) & 1u); // right child (:228-233)
    }
  }
  return 0u;
}

// Rate dematching of one codeblock by the CTA: the soft bits into shared memory, the channel
// de-interleaver, and bit selection with sub-block de-interleaving into the stage-n LLRs.
__device__ __forceinline__ void polar_rate_dematch(const polar_cb& d, polar_cb_smem& sm, const int8_t* __restrict__ llrs)
{
  const int     tid = threadIdx.x;
  const int     n   = d.n;
  const int     N   = 1 << n;
  const int     E   = (int)d.E;
  const int     K   = d.K;
  const int8_t* f   = llrs + d.llr_offset;

  // By aligned words that hold soft bits only; an unaligned stream is shifted into place. The few soft bits
  // before and behind come by bytes: nothing outside the stream is read.
  {
    const int       sh = (int)(reinterpret_cast<uintptr_t>(f) & 3u);
    const uint32_t* w  = reinterpret_cast<const uint32_t*>(f - sh);
    const int       i0 = sh != 0 ? 1 : 0;                         // words i0 .. i1 - 1 of the shared copy
    const int       i1 = max(i0, (E + sh) / 4 - (sh != 0 ? 1 : 0));
#pragma unroll 8
    for (int i = i0 + tid; i < i1; i += kPolarThreads) {
      const uint32_t lo = __ldg(w + i), hi = sh != 0 ? __ldg(w + i + 1) : 0u;
      sm.in[i]          = __funnelshift_r(lo, hi, 8 * sh);
    }
    int8_t* const in8 = reinterpret_cast<int8_t*>(sm.in);
    for (int b = tid; b < 4 * i0 + E - 4 * i1; b += kPolarThreads) {
      const int p = b < 4 * i0 ? b : b - 4 * i0 + 4 * i1;
      in8[p]      = __ldg(f + p);
    }
  }
  __syncthreads();
  const int8_t* const fin = reinterpret_cast<const int8_t*>(sm.in);

  // Channel de-interleaver (polar_rate_dematcher_impl.cpp:53-79): a triangle of T columns, T the smallest
  // with T (T + 1) / 2 >= E, column c of T - c entries. Position S(c) + r, S(c) = c T - c (c - 1) / 2, is
  // the entry (r, c); positions at or beyond E are missing: the last q columns whole and the last `rem`
  // entries of the column before them. The input fills the rows in turn, one thread a row (T <= 128).
  int T = (int)ceilf((sqrtf(8.0f * (float)E + 1.0f) - 1.0f) * 0.5f);
  while (T > 1 && (T - 1) * T / 2 >= E) {
    --T;
  }
  while (T * (T + 1) / 2 < E) {
    ++T;
  }
  const int miss = T * (T + 1) / 2 - E; // < T
  int       q    = (int)((sqrtf(8.0f * (float)miss + 1.0f) - 1.0f) * 0.5f);
  while (q * (q + 1) / 2 > miss) {
    --q;
  }
  while ((q + 1) * (q + 2) / 2 <= miss) {
    ++q;
  }
  const int rem = miss - q * (q + 1) / 2;
  for (int r = tid; r < T; r += kPolarThreads) {
    const int a     = min(r, q);
    const int cnt   = T - r - max(0, q - r) - (r <= q && r > q - rem ? 1 : 0);
    const int first = r * T - r * (r - 1) / 2 - (a * q - a * (a - 1) / 2) - max(0, min(r, q + 1) - (q + 1 - rem));
    int       i_in  = r;
    int       c     = 0;
    for (; c + 4 <= cnt; c += 4) {
      int8_t x[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        x[k] = fin[first + c + k];
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        sm.e[i_in] = x[k];
        i_in += T - c - k;
      }
    }
    for (; c < cnt; ++c) {
      sm.e[i_in] = fin[first + c];
      i_in += T - c;
    }
  }
  __syncthreads();

  // Bit selection (:21-50) and sub-block de-interleaving (:12-19) into the stage-n LLRs.
  int8_t* const ln    = sm.llr + N;
  const bool    rep   = E >= N;
  const bool    punct = !rep && 16 * K <= 7 * E;
  const int     b     = N >> 5;
  for (int j = tid; j < N; j += kPolarThreads) {
    int y;
    if (rep) {
      y = sm.e[j];
#pragma unroll 4
      for (int k = j + N; k < E; k += N) {
        y = llr_promotion_sum(y, sm.e[k]);
      }
    } else if (punct) {
      y = j < N - E ? 0 : sm.e[j - (N - E)];
    } else {
      y = j < E ? sm.e[j] : kLlrInf;
    }
    ln[c_polar_subblock[j >> (n - 5)] * b + (j & (b - 1))] = (int8_t)y;
  }
  __syncthreads();
}

// Simplified successive cancellation (polar_decoder_impl.cpp:163-316) of one codeblock by one warp, depth
// first, then deallocation and CRC. Lane w holds sub-channels 32 w .. 32 w + 31: their K_set bits, codeword
// estimates and decoded bits. Stages above 5 keep their LLRs in shared memory; a node of stage 5 is decoded
// in registers.
__device__ __forceinline__ void polar_decode_codeblock(const polar_cb& d, polar_cb_smem& sm, uint8_t* __restrict__ bits)
{
  const int      lane  = threadIdx.x & 31;
  const int      n     = d.n;
  const int      N     = 1 << n;
  const int      K     = d.K;
  const uint32_t info  = lane < (N >> 5) ? d.info[lane] : 0u;
  const uint32_t zeros = __ballot_sync(0xffffffffu, info == 0u); // words of rate 0 and of rate 1
  const uint32_t ones  = __ballot_sync(0xffffffffu, info == 0xffffffffu);
  uint32_t       cw = 0u, u = 0u;

  // The node: stage s, words w0 .. w0 + 2^(s-5) - 1. phases holds two bits per stage: 0 = node entered,
  // 1 = left child done, 2 = right child done.
  int      s = n, w0 = 0;
  uint32_t phases = 0;
  for (;;) {
    if (s == 5) {
      uint32_t       uc;
      const uint32_t e = polar_node<5>(sm.llr[32 + lane], __shfl_sync(0xffffffffu, info, w0), uc);
      if (lane == w0) {
        cw = e;
        u  = uc;
      }
    } else {
      const int      ph  = (int)((phases >> (2 * s)) & 3u);
      const int      h   = 1 << (s - 1);
      const int      cnt = 1 << (s - 5);
      const uint32_t m   = (cnt == 32 ? 0xffffffffu : (1u << cnt) - 1u) << w0;
      const int8_t*  ls  = sm.llr + (1 << s);
      int8_t*        lc  = sm.llr + h;
      const bool     in  = ((m >> lane) & 1u) != 0u;
      if (ph == 0 && (zeros & m) == m) {
        // rate 0: the words stay zero
      } else if (ph == 0 && (ones & m) == m) {
        for (int k = 0; k < cnt; ++k) {
          const uint32_t e = __ballot_sync(0xffffffffu, ls[32 * k + lane] <= 0);
          if (lane == w0 + k) {
            cw = e;
            u  = polar_transform_word(e);
          }
        }
        for (int st = 1; st < cnt; st <<= 1) {
          const uint32_t t = __shfl_down_sync(0xffffffffu, u, st);
          if (in && ((lane - w0) & st) == 0) {
            u ^= t;
          }
        }
      } else if (ph < 2) {
        __syncwarp();
        if (ph == 0) {
#pragma unroll 4
          for (int i = lane; i < h; i += 32) {
            lc[i] = (int8_t)llr_f(ls[i], ls[i + h]);
          }
        } else {
#pragma unroll 4
          for (int k = 0; k < (h >> 5); ++k) {
            const int      i  = 32 * k + lane;
            const uint32_t eb = __shfl_sync(0xffffffffu, cw, w0 + k);
            lc[i]             = (int8_t)llr_g(ls[i], ls[i + h], (eb >> lane) & 1u);
          }
        }
        __syncwarp();
        phases = (phases & ~(3u << (2 * s))) | ((uint32_t)(ph + 1) << (2 * s));
        w0 += ph == 0 ? 0 : cnt >> 1;
        --s;
        phases &= ~(3u << (2 * s));
        continue;
      } else {
        // Both children done: left codeword ^= right codeword (:240-252).
        const uint32_t t = __shfl_down_sync(0xffffffffu, cw, cnt >> 1);
        if (in && lane < w0 + (cnt >> 1)) {
          cw ^= t;
        }
      }
    }
    if (s == n) {
      break;
    }
    ++s;
    w0 &= ~((1 << (s - 5)) - 1);
  }

  // Deallocation (polar_deallocator_impl.cpp:10-24): a lane's first message index is the number of K_set
  // entries of the lower sub-channels less the parity ones among them.
  int8_t* const msg = reinterpret_cast<int8_t*>(sm.in);
  {
    uint32_t x = info;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t pc = d.pc[k];
      if ((pc >> 5) == (uint32_t)lane) {
        x &= ~(1u << (pc & 31u));
      }
    }
    const int cnt  = __popc(x);
    int       incl = cnt;
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) {
        incl += t;
      }
    }
    int iK = incl - cnt;
    while (x != 0u) {
      const int i = __ffs(x) - 1;
      x &= x - 1u;
      if (iK < K) {
        msg[iK] = (int8_t)((u >> i) & 1u);
      }
      ++iK;
    }
  }
  __syncwarp();
  // The codeblock CRC over the K bits (uci_decoder_impl.cpp:74-92): words of 32 bits by the warp, the
  // register by every lane alike.
  {
    const int      L    = d.crc_size;
    const uint32_t poly = L == 11 ? 0x621u : 0x21u; // CRC11 0xE21, CRC6 0x61 without the x^L term
    const uint32_t mask = (1u << L) - 1u;
    uint32_t       reg  = 0;
    for (int i0 = 0; i0 < K; i0 += 32) {
      const uint32_t w = __ballot_sync(0xffffffffu, i0 + lane < K && msg[i0 + lane] != 0);
      const int      m = min(32, K - i0);
      for (int i = 0; i < m; ++i) {
        const uint32_t top = ((reg >> (L - 1)) ^ (w >> i)) & 1u;
        reg                = ((reg << 1) & mask) ^ (top ? poly : 0u);
      }
    }
    if (lane == 0) {
      sm.valid = reg == 0u ? 1 : 0;
    }
  }
  for (int i = lane; i < d.nbits; i += 32) {
    bits[d.out_offset + i] = (uint8_t)msg[d.nof_filler + i];
  }
}

// One CTA per message: all its warps prepare the decoder's input, then one warp decodes each codeblock.
// Bound: latency, the chain of node steps. Six messages of 20 to 60 bits over up to 8192 soft bits took
// 90 us with the walk down to single sub-channels in shared memory, bytes for codewords and one warp that
// read its soft bits from global memory one by one; with stage 5 in registers and four warps that prepare the
// input 42 us.
__global__ void __launch_bounds__(kPolarThreads) uci_polar_kernel(const polar_cb* __restrict__ cbs, int n,
                                                                 const int8_t* __restrict__ llrs,
                                                                 uint8_t* __restrict__ bits,
                                                                 uint8_t* __restrict__ valid)
{
  __shared__ polar_cb_smem sm[2];
  __shared__ polar_cb      cb[2];
  const int msg  = blockIdx.x;
  const int warp = threadIdx.x >> 5;
  if (msg >= n) {
    return;
  }
  constexpr int kWords = (int)(2 * sizeof(polar_cb) / 4);
  static_assert(kWords <= kPolarThreads && alignof(polar_cb) == 4, "one word of the two descriptors per thread");
  if ((int)threadIdx.x < kWords) {
    reinterpret_cast<uint32_t*>(cb)[threadIdx.x] = reinterpret_cast<const uint32_t*>(cbs + 2 * (size_t)msg)[threadIdx.x];
  }
  __syncthreads();
  for (int c = 0; c < 2; ++c) {
    if (cb[c].E > 0) {
      polar_rate_dematch(cb[c], sm[c], llrs);
    }
  }
  if (warp < 2) {
    if (cb[warp].E > 0) {
      polar_decode_codeblock(cb[warp], sm[warp], bits);
    } else if ((threadIdx.x & 31) == 0) {
      sm[warp].valid = 1;
    }
  }
  __syncthreads();
  // uci_decoder_impl.cpp:40-57: valid when every codeblock passes its CRC.
  if (threadIdx.x == 0) {
    valid[msg] = (uint8_t)((sm[0].valid && sm[1].valid) ? 1 : 0);
  }
}

// The device blob of n messages: two polar_cb per message (the second with E = 0 when the message
// has one codeblock). Returns an error text for an invalid message.
std::string polar_blob_cbs(const pg_uci_polar* items, int n, std::vector<polar_cb>& cbs)
{
  cbs.assign((size_t)2 * n, polar_cb{});
  for (int i = 0; i < n; ++i) {
    const pg_uci_polar& it = items[i];
    const unsigned      A  = it.nof_bits;
    const unsigned      Et = it.nof_llrs;
    if (A < 12 || A > (unsigned)kPolarMaxA) {
      return "message " + std::to_string(i) + ": 12 to 1706 bits";
    }
    const int      C   = uci_nof_codeblocks(A, Et);
    const int      L   = uci_crc_size(A);
    const unsigned A0  = A / C, E0 = Et / C, F = A % C;
    for (int c = 0; c < C; ++c) {
      const unsigned  Ac = c == 0 ? A0 : (A + C - 1) / C;
      const unsigned  Ec = c == 0 ? E0 : Et - E0;
      const unsigned  Fc = c == 0 ? F : 0;
      polar_code_host pc;
      const std::string err = polar_code_build(Ac + L + Fc, Ec, pc);
      if (!err.empty()) {
        return "message " + std::to_string(i) + " codeblock " + std::to_string(c) + ": " + err;
      }
      polar_cb& d  = cbs[2 * (size_t)i + c];
      d.llr_offset = it.llr_offset + (c == 0 ? 0 : E0);
      d.E          = Ec;
      d.out_offset = it.out_offset + (c == 0 ? 0 : A0);
      d.K          = (uint16_t)pc.K;
      d.nbits      = (uint16_t)Ac;
      d.n          = (uint8_t)pc.n;
      d.crc_size   = (uint8_t)L;
      d.nof_filler = (uint8_t)Fc;
      std::memcpy(d.pc, pc.pc, sizeof(d.pc));
      std::memcpy(d.info, pc.info, sizeof(d.info));
    }
  }
  return std::string();
}

} // namespace

namespace pg {

std::string uci_polar_blob(const pg_uci_polar* items, int n, std::vector<uint8_t>& blob)
{
  std::vector<polar_cb> cbs;
  const std::string     err = polar_blob_cbs(items, n, cbs);
  blob.resize(cbs.size() * sizeof(polar_cb));
  std::memcpy(blob.data(), cbs.data(), blob.size());
  return err;
}

int uci_polar_launch_dev(pg_context* ctx, const void* cbs_dev, int n, const int8_t* llrs, uint8_t* bits,
                         uint8_t* valid, cudaStream_t s)
{
  if (n == 0) {
    return PG_OK;
  }
  uci_polar_kernel<<<(unsigned)n, kPolarThreads, 0, s>>>(static_cast<const polar_cb*>(cbs_dev), n, llrs, bits,
                                                         valid);
  return check_cuda(ctx, cudaGetLastError(), "uci_polar_kernel launch");
}

int uci_polar_launch(pg_context* ctx, const pg_uci_polar* items, int n, const int8_t* llrs, uint8_t* bits,
                     uint8_t* valid, cudaStream_t s)
{
  std::vector<uint8_t> blob;
  const std::string    err = uci_polar_blob(items, n, blob);
  if (!err.empty()) {
    return set_error(ctx, PG_ERR_INVALID, err);
  }
  void* dev = nullptr;
  if (int rc = stage_slot(ctx, SLOT_UCI_POLAR, blob.data(), blob.size(), s, &dev)) {
    return rc;
  }
  if (int rc = uci_polar_launch_dev(ctx, dev, n, llrs, bits, valid, s)) {
    return rc;
  }
  return release_slot_after(ctx, SLOT_UCI_POLAR, s);
}

} // namespace pg

using namespace pg;

extern "C" {

int pg_polar_code(uint32_t K, uint32_t E, pg_polar_code_info* out)
{
  if (out == nullptr) {
    return PG_ERR_INVALID;
  }
  polar_code_host c;
  if (!polar_code_build(K, E, c).empty()) {
    return PG_ERR_INVALID;
  }
  std::memset(out, 0, sizeof(*out));
  out->n     = (uint16_t)c.n;
  out->N     = (uint16_t)c.N;
  out->K     = (uint16_t)c.K;
  out->E     = (uint16_t)c.E;
  out->nPC   = (uint8_t)c.nPC;
  out->nWmPC = (uint8_t)c.nWmPC;
  std::memcpy(out->pc_set, c.pc, sizeof(out->pc_set));
  std::memcpy(out->k_set, c.info, sizeof(out->k_set));
  for (int j = 0; j < c.N; ++j) {
    out->subblock[j] = subblock_index(j, c.N);
  }
  return PG_OK;
}

int pg_uci_polar_decode_device(pg_context* ctx, const pg_uci_polar* items, int n, const int8_t* llrs, uint8_t* bits,
                               uint8_t* valid, void* stream)
{
  if (ctx == nullptr) {
    return PG_ERR_INVALID;
  }
  if (n < 0 || (n > 0 && (items == nullptr || llrs == nullptr || bits == nullptr || valid == nullptr))) {
    return set_error(ctx, PG_ERR_INVALID, "null argument");
  }
  if (n == 0) {
    return PG_OK;
  }
  // The codes are built and staged first, so that the kernel events time the kernel alone.
  cudaStream_t         s = static_cast<cudaStream_t>(stream);
  std::vector<uint8_t> blob;
  const std::string    err = uci_polar_blob(items, n, blob);
  if (!err.empty()) {
    return set_error(ctx, PG_ERR_INVALID, err);
  }
  void* dev = nullptr;
  if (int rc = stage_slot(ctx, SLOT_UCI_POLAR, blob.data(), blob.size(), s, &dev)) {
    return rc;
  }
  const unsigned int rec = timing_record_flags(ctx, s);
  if (ctx->timed) {
    cudaEventRecordWithFlags(ctx->ev_start, s, rec);
  }
  const int rc = uci_polar_launch_dev(ctx, dev, n, llrs, bits, valid, s);
  if (ctx->timed) {
    cudaEventRecordWithFlags(ctx->ev_stop, s, rec);
  }
  return rc != PG_OK ? rc : release_slot_after(ctx, SLOT_UCI_POLAR, s);
}

} // extern "C"
