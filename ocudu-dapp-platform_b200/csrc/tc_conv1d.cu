// 1-D convolution (kernel 5, 'same' padding) on the 5th-generation tensor cores: the layers of the
// learned channel estimator, forward and backward, as implicit GEMMs with tcgen05.mma (BF16
// operands from shared memory, FP32 accumulators in tensor memory).
//
// Activation layout: [C/8][R][8] bf16 - channel chunks of 8, each a column of R 16-byte rows
// (one row per resource element position of a batch of concatenated samples, with zero rows
// between samples). In this layout a row is a core-matrix row of the tensor cores' K-major
// no-swizzle operand format with 8-row groups 128 bytes apart, so row r of a chunk sits at
// r * 16 bytes. The five taps of the convolution are therefore the same shared-memory tile seen
// from five start addresses 16 bytes apart: no im2col copy.
//
//   forward:  Y[r][co] = sum_{t, ci} X[r + t - 2][ci] * W[co][ci][t]      (M = rows, N = co, K = 5 x ci)
//   input gradient: the same kernel with W'[ci][co][t] = W[co][ci][4 - t], plus a residual gradient and
//                   the ReLU mask of the forward activation in the epilogue
//   weight gradient: dW[t][ci][co] = sum_r X[r + t - 2][ci] * dY[r][co]   (M = (tap, ci), N = co, K = rows;
//                    both operands MN-major in the activation layout, the taps as row-shifted copies of
//                    the input tile)
//
// Every wait on an mbarrier has an iteration limit; on expiry the kernel records an error code,
// skips its epilogue, frees its tensor memory and returns.
#include "pg_internal.h"
#include "tc_common.cuh"

#include <cuda_bf16.h>

#include <algorithm>

namespace {

using namespace pg::tc;

constexpr int kTapCount    = 5;
constexpr int kTileRows    = 128;
constexpr int kHaloRows    = kTileRows + kTapCount - 1; // 132
constexpr int kConvThreads = 128;

// True for the bf16 values of the 8 lanes of v that are > 0 (ReLU outputs: +0 or positive).
__device__ __forceinline__ void positive_mask(const uint4 v, bool* m)
{
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t lo = w[j] & 0xffffu, hi = w[j] >> 16;
    m[2 * j]     = lo - 1u < 0x7fffu;
    m[2 * j + 1] = hi - 1u < 0x7fffu;
  }
}

// Forward convolution over row tiles of 128 (persistent CTAs). CIN, COUT in {16, 64}.
// Epilogue: + bias (if bias != null), + residual (if res != null), ReLU (if relu), zero where the
// ReLU output `mask` (same layout as y) is not positive (if mask != null), stored as bf16 on valid
// rows.
template <int CIN, int COUT>
__global__ void __launch_bounds__(kConvThreads) conv1d_fwd_kernel(const uint4* __restrict__ x, const uint4* __restrict__ w,
                                                                  const float* __restrict__ bias,
                                                                  const uint4* __restrict__ res,
                                                                  const uint4* __restrict__ mask, uint4* __restrict__ y,
                                                                  const uint8_t* __restrict__ row_valid, int R,
                                                                  int relu, int* __restrict__ err)
{
  constexpr int      kInChunks  = CIN / 8;
  constexpr uint32_t kXChunkB   = kHaloRows * 16;        // bytes per input chunk column in smem
  constexpr uint32_t kWTapB     = kInChunks * COUT * 16; // bytes per tap of packed weights
  constexpr uint32_t kCols      = tmem_cols<COUT>();
  extern __shared__ __align__(128) unsigned char smem[];
  uint4*              xs      = reinterpret_cast<uint4*>(smem);                          // [kInChunks][132]
  uint4*              ws      = reinterpret_cast<uint4*>(smem + kInChunks * kXChunkB);   // [5][kInChunks][COUT]
  uint64_t*           mbar    = reinterpret_cast<uint64_t*>(smem + kInChunks * kXChunkB + kTapCount * kWTapB);
  uint32_t*           tmem_sm = reinterpret_cast<uint32_t*>(mbar + 1);
  uint32_t*           ok_sm   = tmem_sm + 1;
  const int           tid     = threadIdx.x;
  const int           warp    = tid >> 5;

  // Weights once per CTA.
  for (int i = tid; i < kTapCount * kInChunks * COUT; i += kConvThreads) {
    ws[i] = w[i];
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(tmem_sm), kCols);
  }
  if (tid == 0) {
    mbar_init(smem_u32(mbar), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem   = *tmem_sm;
  const uint32_t idesc  = make_idesc(kTileRows, COUT, false, false);
  const int      ntiles = (R + kTileRows - 1) / kTileRows;
  uint32_t       phase  = 0;
  bool           ok     = true;

  for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
    const int m0 = tile * kTileRows;
    // Input rows m0 - 2 .. m0 + 129 of every chunk (zero outside [0, R)).
    for (int i = tid; i < kInChunks * kHaloRows; i += kConvThreads) {
      const int c  = i / kHaloRows;
      const int rr = i - c * kHaloRows;
      const int gr = m0 + rr - 2;
      xs[i]        = (gr >= 0 && gr < R) ? x[(size_t)c * R + gr] : make_uint4(0, 0, 0, 0);
    }
    fence_async_shared();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (tid == 0) {
      const uint32_t xb = smem_u32(xs);
      const uint32_t wb = smem_u32(ws);
      uint32_t       acc = 0;
#pragma unroll
      for (int t = 0; t < kTapCount; ++t) {
#pragma unroll
        for (int kc = 0; kc < CIN / 16; ++kc) {
          const uint64_t ad = make_desc(xb + (uint32_t)(2 * kc) * kXChunkB + (uint32_t)t * 16u, kXChunkB, 128);
          const uint64_t bd = make_desc(wb + (uint32_t)t * kWTapB + (uint32_t)(2 * kc) * (COUT * 16), COUT * 16, 128);
          mma_bf16(tmem, ad, bd, idesc, acc);
          acc = 1;
        }
      }
      mma_commit(smem_u32(mbar));
    }
    // One thread waits (bounded) and publishes the outcome, so that every thread takes the same
    // path.
    if (tid == 0) {
      const bool done = mbar_wait_bounded(smem_u32(mbar), phase);
      *ok_sm          = done ? 1u : 0u;
      if (!done) {
        atomicExch(err, 1);
      }
    }
    phase ^= 1u;
    __syncthreads();
    tc_fence_after();
    ok = *ok_sm != 0;
    if (!ok) {
      break;
    }
    // Epilogue: thread = row (warp w holds TMEM lanes 32w .. 32w + 31).
    const int      r   = warp * 32 + (tid & 31);
    const int      gr  = m0 + r;
    const bool     st  = gr < R && row_valid[gr] != 0;
    const uint32_t tad = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll
    for (int cc = 0; cc < COUT / 16; ++cc) {
      float v[16];
      tmem_ld16(tad + (uint32_t)(cc * 16), v);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int oc = 2 * cc + h; // output chunk of 8 channels
        float     o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          o[j] = v[8 * h + j] + (bias != nullptr ? bias[8 * oc + j] : 0.f);
        }
        if (st && res != nullptr) {
          const uint4          rv = res[(size_t)oc * R + gr];
          const __nv_bfloat16* rb = reinterpret_cast<const __nv_bfloat16*>(&rv);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            o[j] += __bfloat162float(rb[j]);
          }
        }
        if (relu) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            o[j] = fmaxf(o[j], 0.f);
          }
        }
        if (st && mask != nullptr) {
          bool m[8];
          positive_mask(mask[(size_t)oc * R + gr], m);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            o[j] = m[j] ? o[j] : 0.f;
          }
        }
        if (gr < R) {
          // Rows outside samples are written as zeros, so that a buffer reused with another row
          // layout keeps zero rows between its samples.
          uint4           pk = make_uint4(0, 0, 0, 0);
          __nv_bfloat162* pb = reinterpret_cast<__nv_bfloat162*>(&pk);
          if (st) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              pb[j] = __floats2bfloat162_rn(o[2 * j], o[2 * j + 1]);
            }
          }
          y[(size_t)oc * R + gr] = pk;
        }
      }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
  }
  __syncthreads();
  if (warp == 0) {
    tmem_dealloc(tmem, kCols);
  }
}

// ---------------------------------------------------------------------------------------------
// Weight and bias gradients of a list of layers, one launch. Per layer D[m][co] = sum_r A[m][r] * dY[r][co]
// over K tiles of 128 rows, with m = (tap, ci): the input tile is staged as `copies` row-shifted copies
// (copy k holds X[r0 - 2 + k + j]), so that the 16 eight-channel groups of one M tile of 128 sit at a
// uniform stride; M tile j adds j * copies rows to the start address. CIN = 64: 2 copies, 3 M tiles (taps
// 0-1, 2-3, 4 and a discarded 5th); CIN = 16: 8 copies, 1 M tile (taps 0-4 and three discarded). Both
// operands are MN-major without swizzle (SBO = stride of the 8-element MN groups, LBO = stride of the
// 8-row K groups).
//
// The tiles of all layers form one list that is split evenly over one CTA per SM (about 70 tiles each at
// 96,000 rows and 14 layers, so that few CTAs add to one layer's gradients), and a ring of four stages is
// filled by bulk copies (one per 8-channel column and copy) ahead of the MMAs. Warp 0 issues the MMAs,
// warp 1 the copies (and zeroes the rows outside [0, R)), warps 2 and 3 sum dY for the bias gradient from
// the same stage, and warps 4 to 7 add each group of four tiles' FP32 accumulators (two sets in tensor
// memory, one filled while the other is read) to FP32 sums in registers, so that no sum of more than 512
// rows is formed in the tensor cores. When a CTA's run of tiles of one layer ends, its sums are added to
// dw[t][ci][co] with vector atomics. At 96,000 rows the 14 layers take 100 us (722 us with one launch per
// layer, two synchronous stages and a second launch for the bias); bound by the MMAs' shared-memory operand
// reads and by the loads.
constexpr int      kWgTile     = 128;
constexpr int      kWgCopyRows = kWgTile + 8;
constexpr int      kWgStages   = 4;
constexpr uint32_t kWgABytes   = 16u * kWgCopyRows * 16u;
constexpr uint32_t kWgBBytes   = 8u * kWgTile * 16u;
constexpr uint32_t kWgStageB   = kWgABytes + kWgBBytes;
constexpr int      kWgThreads  = 256;
constexpr int      kWgGroup    = 4;   // tiles per accumulator set
constexpr uint32_t kWgCols     = 512; // two sets of up to 3 M tiles x 64 columns, 256 columns apart
constexpr size_t   kWgSmem     = kWgStages * (size_t)kWgStageB + 8 * (2 * kWgStages + 4) + 24;
static_assert(kWgStageB % 128 == 0 && kWgSmem <= 227 * 1024, "shared memory of the weight-gradient kernel");

struct wg_args {
  pg::wgrad_layer l[pg::kMaxWgradLayers];
  int             n;
};

// The MMAs of one stage: the descriptors are formed once and each MMA adds a constant to their
// start-address fields (16-byte units, below 2^14, so no carry reaches the next field). Formed per MMA by
// the one issuing thread they set the time of a tile (154 us for the 14 layers at 96,000 rows).
template <int CIN, int COUT>
__device__ __forceinline__ void wgrad_issue_tile(uint32_t go, uint32_t ab, uint32_t d, uint32_t acc)
{
  constexpr int      kCopies = 16 / (CIN / 8);
  constexpr int      kMTiles = (kTapCount + kCopies - 1) / kCopies;
  constexpr uint32_t idesc   = make_idesc(kTileRows, COUT, true, true);
  const uint64_t     a0      = make_desc(ab, 128, kWgCopyRows * 16);
  const uint64_t     b0      = make_desc(ab + kWgABytes, 128, kWgTile * 16);
#pragma unroll
  for (int ks = 0; ks < kWgTile / 16; ++ks) {
#pragma unroll
    for (int j = 0; j < kMTiles; ++j) {
      mma_bf16_warp(go, d + (uint32_t)(j * COUT), a0 + (uint64_t)(j * kCopies + ks * 16), b0 + (uint64_t)(ks * 16), idesc,
               ks > 0 ? 1u : acc);
    }
  }
}

__global__ void __launch_bounds__(kWgThreads, 1) conv1d_wgrad_kernel(const __grid_constant__ wg_args args, int R,
                                                                       int* __restrict__ err)
{
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t*          bars     = reinterpret_cast<uint64_t*>(smem + kWgStages * kWgStageB);
  uint32_t*          tmem_sm  = reinterpret_cast<uint32_t*>(bars + 2 * kWgStages + 4);
  volatile uint32_t* abort_sm = tmem_sm + 1;
  const uint32_t     bar_full = smem_u32(&bars[0]);             // + 8 stage: copies landed
  const uint32_t     bar_free = smem_u32(&bars[kWgStages]);     // + 8 stage: MMAs and bias sums done
  const uint32_t     bar_acc  = smem_u32(&bars[2 * kWgStages]);     // + 8 set: accumulators of a group complete
  const uint32_t     bar_read = smem_u32(&bars[2 * kWgStages + 2]); // + 8 set: they have been read
  const uint32_t     base     = smem_u32(smem);
  const int          tid      = threadIdx.x;
  const int          warp     = __shfl_sync(0xffffffffu, tid >> 5, 0); // uniform
  const int          lane     = tid & 31;
  if (warp == 0) {
    tmem_alloc(smem_u32(tmem_sm), kWgCols);
  }
  if (tid == 0) {
    for (int i = 0; i < kWgStages; ++i) {
      mbar_init(bar_full + 8u * i, 1);
      mbar_init(bar_free + 8u * i, 3); // the MMA commit and the two bias warps
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar_acc + 8u * i, 1);
      mbar_init(bar_read + 8u * i, 4); // the four accumulating warps
    }
    *abort_sm = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem   = __shfl_sync(0xffffffffu, *tmem_sm, 0);
  const int      ntiles = (R + kWgTile - 1) / kWgTile;
  const long     total  = (long)args.n * ntiles;
  const long     t_end  = total * (blockIdx.x + 1) / gridDim.x;
  auto wait = [&](uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < kWaitLimit; ++i) {
      if (mbar_try_wait(bar, parity)) {
        return true;
      }
      if (*abort_sm != 0) {
        return false;
      }
    }
    *abort_sm = 1;
    atomicExch(err, 1);
    return false;
  };
  uint32_t k0 = 0; // tiles of the earlier runs: tile k of this CTA goes to stage k mod kWgStages
  uint32_t g0 = 0; // groups of the earlier runs: group g uses accumulator set g mod 2
  for (long t = total * blockIdx.x / gridDim.x; t < t_end;) {
    const int              li     = (int)(t / ntiles);
    const int              tile0  = (int)(t - (long)li * ntiles);
    const int              nt     = (int)min((long)(ntiles - tile0), t_end - t);
    const pg::wgrad_layer& L      = args.l[li];
    const int              inch   = L.cin / 8;
    const int              copies = 16 / inch;
    const int              mt     = (kTapCount + copies - 1) / copies;
    const int              bch    = L.cout / 8;
    const int              ngrp   = (nt + kWgGroup - 1) / kWgGroup;
    if (warp == 0) {
      // The whole warp takes the same path (lane 0 polls, issues and commits).
      const uint32_t go = lane == 0 ? 1u : 0u;
      for (int i = 0; i < nt; ++i) {
        const uint32_t k = k0 + (uint32_t)i, st = k % kWgStages;
        const uint32_t grp = g0 + (uint32_t)(i / kWgGroup), set = grp & 1u;
        bool           ok = true;
        if (lane == 0) {
          ok = (i % kWgGroup != 0 || grp < 2 || wait(bar_read + 8u * set, (grp / 2 - 1u) & 1u)) &&
               wait(bar_full + 8u * st, (k / kWgStages) & 1u);
        }
        if (__all_sync(0xffffffffu, ok) == 0) {
          break;
        }
        tc_fence_after();
        const uint32_t ab = base + st * kWgStageB, acc = i % kWgGroup > 0 ? 1u : 0u, d = tmem + 256u * set;
        if (L.cin == 16) {
          wgrad_issue_tile<16, 64>(go, ab, d, acc);
        } else if (L.cout == 16) {
          wgrad_issue_tile<64, 16>(go, ab, d, acc);
        } else {
          wgrad_issue_tile<64, 64>(go, ab, d, acc);
        }
        if (lane == 0) {
          mma_commit(bar_free + 8u * st);
          if (i % kWgGroup == kWgGroup - 1 || i + 1 == nt) {
            mma_commit(bar_acc + 8u * set);
          }
        }
        __syncwarp();
      }
    } else if (warp == 1) {
      // Lane g: column g of A (copy g / inch, chunk g % inch), lane 16 + c: column c of B.
      const int    ak  = lane / inch;
      const int    col = lane < 16 ? lane - ak * inch : lane - 16;
      const bool   on  = lane < 16 || col < bch;
      const uint4* src = static_cast<const uint4*>(lane < 16 ? L.x : L.dy) + (size_t)(on ? col : 0) * R;
      const int    len = lane < 16 ? kWgCopyRows : kWgTile;
      for (int i = 0; i < nt; ++i) {
        const uint32_t k = k0 + (uint32_t)i, st = k % kWgStages;
        bool           ok = true;
        if (lane == 0 && k >= kWgStages) {
          ok = wait(bar_free + 8u * st, (k / kWgStages - 1u) & 1u);
        }
        if (__shfl_sync(0xffffffffu, ok ? 1 : 0, 0) == 0) {
          break;
        }
        const int      r0  = (tile0 + i) * kWgTile + (lane < 16 ? ak - 2 : 0); // first row of the column
        const int      lo  = on ? max(0, -r0) : 0;
        const int      hi  = on ? max(lo, min(len, R - r0)) : 0;
        const uint32_t dst = base + st * kWgStageB + (lane < 16 ? (uint32_t)lane * (kWgCopyRows * 16u)
                                                               : kWgABytes + (uint32_t)col * (kWgTile * 16u));
        if (on && hi - lo < len) {
          for (int r = 0; r < len; ++r) {
            if (r < lo || r >= hi) {
              *reinterpret_cast<uint4*>(smem + (dst - base) + 16 * r) = make_uint4(0, 0, 0, 0);
            }
          }
          fence_async_shared();
        }
        const uint32_t bytes = __reduce_add_sync(0xffffffffu, 16u * (uint32_t)(hi - lo));
        __syncwarp();
        if (lane == 0) {
          mbar_expect_tx(bar_full + 8u * st, bytes);
        }
        __syncwarp();
        if (hi > lo) {
          bulk_g2s(dst + 16u * (uint32_t)lo, src + r0 + lo, 16u * (uint32_t)(hi - lo), bar_full + 8u * st);
        }
      }
    } else if (warp < 4) {
      // Thread: rows bt % 8, + 8, ... of dY column bt / 8.
      float      bsum[8] = {};
      const int  bt = tid - 64, c = bt >> 3;
      const bool on = c < bch && L.db != nullptr;
      for (int i = 0; i < nt; ++i) {
        const uint32_t k = k0 + (uint32_t)i, st = k % kWgStages;
        bool           ok = true;
        if (lane == 0) {
          ok = wait(bar_full + 8u * st, (k / kWgStages) & 1u);
        }
        if (__shfl_sync(0xffffffffu, ok ? 1 : 0, 0) == 0) {
          break;
        }
        __syncwarp(); // the copies that lane 0 waited for are visible to the warp
        if (on) {
          const uint4* p = reinterpret_cast<const uint4*>(smem + st * kWgStageB + kWgABytes) + c * kWgTile + (bt & 7);
          float        tsum[8] = {}; // of the tile
#pragma unroll
          for (int r = 0; r < kWgTile / 8; ++r) {
            const uint4           v = p[8 * r];
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              tsum[2 * j] += __low2float(h[j]);
              tsum[2 * j + 1] += __high2float(h[j]);
            }
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            bsum[j] += tsum[j];
          }
        }
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(bar_free + 8u * st);
        }
      }
      const bool whole = __shfl_sync(0xffffffffu, *abort_sm == 0 ? 1 : 0, 0) != 0;
      if (on && whole) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float v = bsum[j];
          v += __shfl_xor_sync(0xffu << (lane & 24), v, 1);
          v += __shfl_xor_sync(0xffu << (lane & 24), v, 2);
          v += __shfl_xor_sync(0xffu << (lane & 24), v, 4);
          if ((bt & 7) == 0) {
            atomicAdd(L.db + 8 * c + j, v);
          }
        }
      }
    } else {
      // Thread = TMEM lane m of every M tile: group mg = m / 8 (copy ck, chunk), lane m % 8.
      const int      m  = tid - 128;
      const int      mg = m >> 3;
      const int      ck = mg / inch;
      const int      ci = 8 * (mg - ck * inch) + (m & 7);
      const int      nc = mt * L.cout / 16; // 16-column pieces
      float          acc[12][16];
#pragma unroll
      for (int p = 0; p < 12; ++p) {
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          acc[p][q] = 0.f;
        }
      }
      for (int i = 0; i < ngrp; ++i) {
        const uint32_t grp = g0 + (uint32_t)i, set = grp & 1u;
        bool           ok  = true;
        if (lane == 0) {
          ok = wait(bar_acc + 8u * set, (grp / 2) & 1u);
        }
        if (__shfl_sync(0xffffffffu, ok ? 1 : 0, 0) == 0) {
          break;
        }
        tc_fence_after();
        const uint32_t tad = tmem + 256u * set + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll
        for (int p = 0; p < 12; ++p) {
          if (p < nc) {
            float v[16];
            tmem_ld16(tad + 16u * (uint32_t)p, v);
#pragma unroll
            for (int q = 0; q < 16; ++q) {
              acc[p][q] += v[q];
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(bar_read + 8u * set);
        }
      }
      if (*abort_sm == 0) {
        const int per = L.cout / 16; // pieces per M tile
#pragma unroll
        for (int p = 0; p < 12; ++p) {
          const int j = p / per, tap = j * copies + ck;
          if (p < nc && tap < kTapCount) {
            float4* dst = reinterpret_cast<float4*>(L.dw + ((size_t)tap * L.cin + ci) * L.cout + (p - j * per) * 16);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              atomicAdd(dst + q, make_float4(acc[p][4 * q], acc[p][4 * q + 1], acc[p][4 * q + 2], acc[p][4 * q + 3]));
            }
          }
        }
      }
    }
    __syncthreads();
    if (*abort_sm != 0) {
      break;
    }
    g0 += (uint32_t)ngrp;
    k0 += (uint32_t)nt;
    t += nt;
  }
  // After a failure: wait (bounded) for the copies and MMAs that may be in flight (a barrier's phase in
  // flight is one of the two parities; the other returns at once).
  if (*abort_sm != 0) {
    if (tid == 0) {
      mma_commit(bar_acc);
    }
    if (tid < kWgStages + 2) {
      for (uint32_t ph = 0; ph < 2; ++ph) {
        (void)mbar_wait_bounded(tid < kWgStages ? bar_full + 8u * tid : bar_acc + 8u * (tid - kWgStages), ph);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tmem_dealloc(tmem, kWgCols);
  }
}

template <int CIN, int COUT>
size_t fwd_smem_bytes()
{
  return (size_t)(CIN / 8) * kHaloRows * 16 + (size_t)kTapCount * (CIN / 8) * COUT * 16 + 16;
}

template <int CIN, int COUT>
int fwd_setup()
{
  return cudaFuncSetAttribute(conv1d_fwd_kernel<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)fwd_smem_bytes<CIN, COUT>()) == cudaSuccess
             ? PG_OK
             : PG_ERR_CUDA;
}

template <int CIN, int COUT>
int fwd_launch(pg_context* ctx, const void* x, const void* w, const float* bias, const void* res, const void* mask,
               void* y, const uint8_t* row_valid, int R, int relu, int* err, cudaStream_t s)
{
  const int ntiles = (R + kTileRows - 1) / kTileRows;
  const int grid   = std::max(1, std::min(ntiles, ctx->sm_count * 2));
  conv1d_fwd_kernel<CIN, COUT><<<grid, kConvThreads, fwd_smem_bytes<CIN, COUT>(), s>>>(
      static_cast<const uint4*>(x), static_cast<const uint4*>(w), bias, static_cast<const uint4*>(res),
      static_cast<const uint4*>(mask), static_cast<uint4*>(y), row_valid, R, relu, err);
  return pg::check_cuda(ctx, cudaGetLastError(), "conv1d_fwd_kernel launch");
}

} // namespace

namespace pg {

int conv_setup(pg_context* ctx)
{
  int rc = fwd_setup<16, 64>();
  if (rc == PG_OK) {
    rc = fwd_setup<64, 64>();
  }
  if (rc == PG_OK) {
    rc = fwd_setup<64, 16>();
  }
  if (rc == PG_OK && cudaFuncSetAttribute(conv1d_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)kWgSmem) != cudaSuccess) {
    rc = PG_ERR_CUDA;
  }
  if (rc != PG_OK) {
    (void)cudaGetLastError();
    return set_error(ctx, PG_ERR_CUDA, "cudaFuncSetAttribute(conv1d kernels)");
  }
  return PG_OK;
}

int conv_forward_launch(pg_context* ctx, int cin, int cout, const void* x, const void* w, const float* bias,
                        const void* res, const void* mask, void* y, const uint8_t* row_valid, int R, int relu,
                        int* err, cudaStream_t s)
{
  if (R <= 0) {
    return PG_OK;
  }
  if (cin == 16 && cout == 64) {
    return fwd_launch<16, 64>(ctx, x, w, bias, res, mask, y, row_valid, R, relu, err, s);
  }
  if (cin == 64 && cout == 64) {
    return fwd_launch<64, 64>(ctx, x, w, bias, res, mask, y, row_valid, R, relu, err, s);
  }
  if (cin == 64 && cout == 16) {
    return fwd_launch<64, 16>(ctx, x, w, bias, res, mask, y, row_valid, R, relu, err, s);
  }
  return set_error(ctx, PG_ERR_INVALID, "conv1d: channel counts must be (16,64), (64,64) or (64,16)");
}

int conv_wgrad_launch(pg_context* ctx, const wgrad_layer* layers, int n, int R, int* err, cudaStream_t s)
{
  if (R <= 0 || n <= 0) {
    return PG_OK;
  }
  wg_args args{};
  for (int i = 0; i < n; ++i) {
    const int ci = layers[i].cin, co = layers[i].cout;
    if (n > kMaxWgradLayers || !((ci == 16 && co == 64) || (ci == 64 && co == 64) || (ci == 64 && co == 16))) {
      return set_error(ctx, PG_ERR_INVALID, "conv1d: channel counts must be (16,64), (64,64) or (64,16)");
    }
    args.l[i] = layers[i];
  }
  args.n = n;
  // At least four K tiles per CTA (fewer partial sums to add), at most one CTA per SM.
  const long tiles = (long)n * ((R + kWgTile - 1) / kWgTile);
  const int  grid  = (int)std::max(1l, std::min((long)ctx->sm_count, tiles / 4));
  conv1d_wgrad_kernel<<<grid, kWgThreads, kWgSmem, s>>>(args, R, err);
  return check_cuda(ctx, cudaGetLastError(), "conv1d_wgrad_kernel launch");
}

} // namespace pg

extern "C" int pg_conv1d_forward_device(pg_context* ctx, int cin, int cout, const void* x, const void* w,
                                        const float* bias, const void* res, void* y, const uint8_t* row_valid, int rows,
                                        int relu, int* err, void* stream)
{
  if (ctx == nullptr) {
    return PG_ERR_INVALID;
  }
  if (x == nullptr || w == nullptr || bias == nullptr || y == nullptr || row_valid == nullptr || err == nullptr ||
      rows < 0) {
    return pg::set_error(ctx, PG_ERR_INVALID, "conv1d: null buffer or negative row count");
  }
  return pg::conv_forward_launch(ctx, cin, cout, x, w, bias, res, nullptr, y, row_valid, rows, relu, err,
                                 static_cast<cudaStream_t>(stream));
}

extern "C" int pg_conv1d_backward_data_device(pg_context* ctx, int cin, int cout, const void* dy, const void* w_t,
                                              const void* res, const void* mask, void* dx, const uint8_t* row_valid,
                                              int rows, int* err, void* stream)
{
  if (ctx == nullptr) {
    return PG_ERR_INVALID;
  }
  if (dy == nullptr || w_t == nullptr || dx == nullptr || row_valid == nullptr || err == nullptr || rows < 0) {
    return pg::set_error(ctx, PG_ERR_INVALID, "conv1d backward: null buffer or negative row count");
  }
  // The input gradient of a (cin -> cout) layer is a (cout -> cin) convolution.
  return pg::conv_forward_launch(ctx, cout, cin, dy, w_t, nullptr, res, mask, dx, row_valid, rows, 0, err,
                                 static_cast<cudaStream_t>(stream));
}

extern "C" int pg_conv1d_backward_weights_device(pg_context* ctx, int cin, int cout, const void* x, const void* dy,
                                                 int rows, float* dw, float* db, int* err, void* stream)
{
  if (ctx == nullptr) {
    return PG_ERR_INVALID;
  }
  if (x == nullptr || dy == nullptr || dw == nullptr || err == nullptr || rows < 0) {
    return pg::set_error(ctx, PG_ERR_INVALID, "conv1d weight gradient: null buffer or negative row count");
  }
  const pg::wgrad_layer layer = {x, dy, dw, db, cin, cout};
  return pg::conv_wgrad_launch(ctx, &layer, 1, rows, err, static_cast<cudaStream_t>(stream));
}
