// tcgen05 GEMM kernels behind linear_forward / linear_dgrad / linear_wgrad.
//
// The kernels share one warp-specialised structure per CTA (320 threads and, where noted, a few warps more):
//   warp 0 (one lane)  TMA producer: fills a ring of shared-memory stages with 128-byte-swizzled
//                      tiles of 64 k-elements, one mbarrier per stage counting bytes;
//   warp 1 (one lane)  MMA issuer: four tcgen05.mma (K = 16 each) per stage into a TMEM
//                      accumulator, tcgen05.commit frees the stage and finally signals the epilogue;
//   warps 2-9          epilogue: two warps per TMEM lane quarter, each taking half of the tile's
//                      columns; tcgen05.ld the accumulator (one row per thread) and fuse bias + ReLU
//                      (+ a one-bit ReLU mask) in the forward pass, the ReLU mask in the input
//                      gradient, or a split-K TMA reduce-add into the fp32 gradient buffer.
// gemm_kernel computes one 128 x BN tile per CTA; gemm_bres_kernel and gemm_pair_kernel are
// persistent, keep their slice of the weights in shared memory and stream activation tiles past it
// with two TMEM accumulators (the pair variant runs tcgen05.mma.cta_group::2 on two CTAs);
// gemm_pair_wgrad_kernel is the weight gradient on CTA pairs, for large ones.
// Operands are K-major except in the weight gradient, which contracts over the batch and
// therefore reads both activations MN-major, as they sit in memory.
// Every mbarrier wait is bounded; on a give-up the CTA records kTimeout, lets its outstanding
// TMA copies land, frees its tensor memory and returns.  No TMA load uses cluster multicast.
#include <cuda_bf16.h>

#include <mutex>

#include "../core/types.h"
#include "common.cuh"
#include "mlp_gemm.h"
#include "tcgen05.cuh"

namespace kb {
namespace cu {

namespace {

constexpr int kBM = 128;         // rows of the output tile = TMEM lanes
constexpr int kBK = 64;          // k-elements per stage = one 128-byte swizzle atom of bf16
constexpr int kEpiWarps = 8;     // two warps per TMEM lane quarter, each taking half of the tile's columns
constexpr int kThreads = 64 + 32 * kEpiWarps;
constexpr uint32_t kWaitLimit = 1u << 22;
constexpr int kMaxStages = 8;

enum { EPI_BIAS_ACT = 0, EPI_RELU_MASK = 1, EPI_RED_F32 = 2 };

// Passed as a __grid_constant__: the slow path below takes its address, and a by-value parameter was copied to each
// thread's local memory for that, where every access of the epilogues then went (65536 x 400 x 432: 46 us a forward layer
// so, 37 us from constant memory).
struct GemmArgs {
  int M, N, K;            // output is M x N, contraction length K
  int BN;                 // tile width (multiple of 16; of 64 when B is MN-major)
  int stages;
  int kb_per_split;       // k-blocks per blockIdx.z, or per work item of the streaming variant
  int tiles_m, tiles_n;   // ... its grid of tiles, and the number of (tile, split) items
  int items;
  int relu;
  const float* bias;      // [N]            (EPI_BIAS_ACT)
  const __nv_bfloat16* H; // [M, ldh]       (EPI_RELU_MASK, when no bit mask is given)
  int ldh;
  const uint16_t* mask;   // [chunks, ldm] one bit per element: word (c, r) = columns [16c, 16c + 16) of row r
  uint16_t* mask_out;     // same layout, written by EPI_BIAS_ACT with relu: bit = output > 0
  int ldm;                // row pitch of the mask in words (>= M): a warp's 32 rows are 64 contiguous bytes
  int mask_chunks;        // number of 16-column words per row that the mask holds
  int out_v8;             // bf16 output rows and tile columns are 32-byte aligned: one 256-bit store per chunk
  int out_tma;            // gemm_pair_kernel: the output goes out in 32 x 32 boxes through the TMA unit (BN a multiple of 32)
  __nv_bfloat16* out;     // [M, ldo] bf16  (EPI_BIAS_ACT, EPI_RELU_MASK)
  int ldo;
  int zero_cols;          // columns behind the N of `out` that are cleared, a multiple of 8 (EPI_RELU_MASK)
  float* col_sums;        // [M] += column sums of A, or null (EPI_RED_F32 with an MN-major A: the bias gradient)
  int* status;
  int late;               // host: launched behind the kernel in front and not beside its end (what wrote the bias)
};

// Position in a ring of stages: the stage and the parity of the round through it.  The threads that issue copies and MMAs
// count along instead of dividing a running number (150 cycles for a division by a run-time number of stages, one to three of
// them in front of every k-block, whose MMAs take 512 for 128 x 256), and the MMA threads look at the next stage's barrier
// between two MMAs: the look takes 200 cycles, for which the tensor cores would stand still behind the last one.
struct Ring {
  int s = 0;
  uint32_t parity = 0;
  __device__ __forceinline__ void next(int stages) {
    if (++s == stages) s = 0, parity ^= 1;
  }
};

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}


// ------------------------------------------------------------------ epilogue
// Slow path for a 16-column chunk that straddles N: the whole warp calls it (the decision depends
// on the column only); it reads the chunk from tensor memory itself and writes element-wise with
// bounds checks, so the fast path never needs its registers in addressable memory.
template <int EPI>
__device__ __noinline__ void epilogue_tail(const GemmArgs& g, const float* s_bias, uint32_t taddr, int row, int col,
                                           int c) {
  uint32_t r[16];
  tc::tmem_ld16(taddr, r);
  tc::tmem_ld_wait();
  if (row >= g.M) return;
  uint32_t bits_out = 0;
  const uint32_t bits_in =
      (EPI == EPI_RELU_MASK && g.mask != nullptr) ? g.mask[static_cast<size_t>(col >> 4) * g.ldm + row] : 0xFFFFu;
  for (int j = 0; j < 16 && col + j < g.N; ++j) {
    float v = __uint_as_float(r[j]);
    if (EPI == EPI_BIAS_ACT) {
      v += s_bias[c + j];
      if (g.relu) v = fmaxf(v, 0.f);
      if (v > 0.f) bits_out |= 1u << j;
    }
    if (EPI == EPI_RELU_MASK && g.mask != nullptr && !((bits_in >> j) & 1u)) v = 0.f;
    if (EPI == EPI_RELU_MASK && g.mask == nullptr && g.H != nullptr &&
        !(__bfloat162float(g.H[static_cast<size_t>(row) * g.ldh + col + j]) > 0.f))
      v = 0.f;
    g.out[static_cast<size_t>(row) * g.ldo + col + j] = __float2bfloat16(v);
  }
  if (EPI == EPI_BIAS_ACT && g.mask_out != nullptr)
    g.mask_out[static_cast<size_t>(col >> 4) * g.ldm + row] = static_cast<uint16_t>(bits_out);
}

// Fast path: all 16 columns valid.  Everything is unrolled with constant indices so the
// accumulator chunk stays in registers.
template <int EPI, bool RELU>
__device__ __forceinline__ void epilogue_full(const GemmArgs& g, const float* s_bias, int row, int col, int c,
                                              const uint32_t (&r)[16], uint32_t keep_bits) {
  float v[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
  if (EPI == EPI_BIAS_ACT) {
    uint32_t bits = 0;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      v[j] += s_bias[c + j];
      if (RELU) v[j] = fmaxf(v[j], 0.f);
      bits |= (v[j] > 0.f ? 1u : 0u) << j;
    }
    if (g.mask_out != nullptr) g.mask_out[static_cast<size_t>(col >> 4) * g.ldm + row] = static_cast<uint16_t>(bits);
  }
  if (EPI == EPI_RELU_MASK) {
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (!((keep_bits >> j) & 1u)) v[j] = 0.f;
  }
  __nv_bfloat16* o = g.out + static_cast<size_t>(row) * g.ldo + col;
  uint4 w0, w1;
  w0.x = pack_bf16(v[0], v[1]);   w0.y = pack_bf16(v[2], v[3]);
  w0.z = pack_bf16(v[4], v[5]);   w0.w = pack_bf16(v[6], v[7]);
  w1.x = pack_bf16(v[8], v[9]);   w1.y = pack_bf16(v[10], v[11]);
  w1.z = pack_bf16(v[12], v[13]); w1.w = pack_bf16(v[14], v[15]);
  if (g.out_v8) {
    // one 32-byte sector per request: the L2 write-request rate, not bytes, bounds this epilogue
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(o), "r"(w0.x), "r"(w0.y), "r"(w0.z),
                 "r"(w0.w), "r"(w1.x), "r"(w1.y), "r"(w1.z), "r"(w1.w)
                 : "memory");
  } else {
    *reinterpret_cast<uint4*>(o) = w0;
    *reinterpret_cast<uint4*>(o + 8) = w1;
  }
}

// 16 keep-bits from 16 bf16 activations: bf16 > 0  <=>  sign bit clear and not zero.
__device__ __forceinline__ uint32_t keep_bits_of(const uint4& h0, const uint4& h1) {
  const uint32_t hw[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
  uint32_t bits = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t lo = hw[j] & 0xFFFFu, hi = hw[j] >> 16;
    bits |= ((lo != 0u && !(lo & 0x8000u)) ? 1u : 0u) << (2 * j);
    bits |= ((hi != 0u && !(hi & 0x8000u)) ? 1u : 0u) << (2 * j + 1);
  }
  return bits;
}

// The mask words of one row for up to eight 16-column chunks starting at chunk `cb`, packed into
// 128 bits.  Issued before the accumulator wait, so the loads fly while the MMAs run.
struct RowMask {
  unsigned long long lo, hi;
  __device__ __forceinline__ uint32_t chunk(int i) const {
    return static_cast<uint32_t>((i < 4 ? lo >> (16 * i) : hi >> (16 * (i - 4))) & 0xFFFFull);
  }
};

// As they are loaded: packing them waits for the loads.
struct MaskWords {
  uint16_t w[8];
  __device__ __forceinline__ void load(const GemmArgs& g, int row, int cb, int nchunks) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      w[i] = g.mask != nullptr && row < g.M && i < nchunks && cb + i < g.mask_chunks
                 ? __ldg(g.mask + row + static_cast<size_t>(cb + i) * g.ldm) : 0xFFFFu;
  }
  __device__ __forceinline__ RowMask packed() const {
    RowMask m{0, 0};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      m.lo |= static_cast<unsigned long long>(w[i]) << (16 * i);
      m.hi |= static_cast<unsigned long long>(w[i + 4]) << (16 * i);
    }
    return m;
  }
};

__device__ __forceinline__ RowMask load_row_mask(const GemmArgs& g, int row, int cb, int nchunks) {
  MaskWords words;
  words.load(g, row, cb, nchunks);
  return words.packed();
}

// One epilogue warp's share of a 128 x BN accumulator: TMEM lanes of its quarter (one row per
// thread) and the column range [c_begin, c_end).  Two 16-column chunks are in flight per wait.
template <int EPI, bool RELU>
__device__ __forceinline__ void store_rows(const GemmArgs& g, const float* s_bias, uint32_t t_row, int row, int n0,
                                           int c_begin, int c_end, const RowMask& rm) {
  const bool in_rows = row < g.M;
  // ReLU keep-bits come from the bit mask when there is one (already in registers), else from H
  const bool from_h = EPI == EPI_RELU_MASK && g.mask == nullptr && g.H != nullptr;
  int c = c_begin;
  // pairs of full chunks: both loads are issued before the single wait
  for (; c + 32 <= c_end && n0 + c + 32 <= g.N; c += 32) {
    const int col = n0 + c;
    uint32_t r0[16], r1[16];
    tc::tmem_ld16(t_row + c, r0);
    tc::tmem_ld16(t_row + c + 16, r1);
    uint32_t k0 = rm.chunk((c - c_begin) >> 4), k1 = rm.chunk(((c - c_begin) >> 4) + 1);
    if (from_h && in_rows) {
      const __nv_bfloat16* h = g.H + static_cast<size_t>(row) * g.ldh + col;
      k0 = keep_bits_of(*reinterpret_cast<const uint4*>(h), *reinterpret_cast<const uint4*>(h + 8));
      k1 = keep_bits_of(*reinterpret_cast<const uint4*>(h + 16), *reinterpret_cast<const uint4*>(h + 24));
    }
    tc::tmem_ld_wait();
    if (in_rows) {
      epilogue_full<EPI, RELU>(g, s_bias, row, col, c, r0, k0);
      epilogue_full<EPI, RELU>(g, s_bias, row, col + 16, c + 16, r1, k1);
    }
  }
  // what is left: single chunks, full or straddling N (all conditions are warp-uniform)
  for (; c < c_end && n0 + c < g.N; c += 16) {
    const int col = n0 + c;
    if (col + 16 <= g.N) {
      uint32_t r0[16];
      tc::tmem_ld16(t_row + c, r0);
      uint32_t k0 = rm.chunk((c - c_begin) >> 4);
      if (from_h && in_rows) {
        const __nv_bfloat16* h = g.H + static_cast<size_t>(row) * g.ldh + col;
        k0 = keep_bits_of(*reinterpret_cast<const uint4*>(h), *reinterpret_cast<const uint4*>(h + 8));
      }
      tc::tmem_ld_wait();
      if (in_rows) epilogue_full<EPI, RELU>(g, s_bias, row, col, c, r0, k0);
    } else {
      epilogue_tail<EPI>(g, s_bias, t_row + c, row, col, c);
    }
  }
}

// The columns behind an input gradient, cleared by the warps that hold its last column: a launch of its own for these zeros
// took 4 to 6.5 us of the backward chain.
__device__ __forceinline__ void clear_behind(const GemmArgs& g, int row, int n0, int c_begin, int c_end) {
  if (g.zero_cols > 0 && row < g.M && n0 + c_begin < g.N && n0 + c_end >= g.N)
    for (int j = 0; j < g.zero_cols; j += 8)
      *reinterpret_cast<uint4*>(g.out + static_cast<size_t>(row) * g.ldo + g.N + j) = make_uint4(0, 0, 0, 0);
}

// (the choice once and not per element: a branch on it inside took 500 cycles of 780 per 32 columns)
template <int EPI>
__device__ __forceinline__ void epilogue_rows(const GemmArgs& g, const float* s_bias, uint32_t t_row, int row, int n0,
                                              int c_begin, int c_end, const RowMask& rm) {
  if (EPI == EPI_BIAS_ACT && g.relu)
    store_rows<EPI, true>(g, s_bias, t_row, row, n0, c_begin, c_end, rm);
  else
    store_rows<EPI, false>(g, s_bias, t_row, row, n0, c_begin, c_end, rm);
  if (EPI == EPI_RELU_MASK) clear_behind(g, row, n0, c_begin, c_end);
}

// The same for EPI_RED_F32: 32 x 32 boxes of the accumulator go through two 4 KB buffers of the warp in shared memory
// (128-byte swizzle: a lane holds a row, and 8 lanes' 16-byte chunks fall into 8 different columns of banks) and are
// added to dW by the TMA unit, in whole lines.  As 16-byte red.global.add from every lane's own row each warp instruction
// touched 32 lines, half a sector each, and that, not the MMAs, set the time: the three layers 784-4096-4096-4096 at
// batch 1024 took 173 us, 142 us so.
__device__ __forceinline__ void epilogue_reduce(const GemmArgs& g, const CUtensorMap* tmD, uint8_t* buf, uint32_t t_row,
                                                int row0, int n0, int c_begin, int c_end, int& turn) {
  const int lane = threadIdx.x & 31;
  if (row0 >= g.M) return;  // the same for the whole warp
  for (int c = c_begin; c < c_end && n0 + c < g.N; c += 32, ++turn) {
    uint8_t* const b = buf + (turn & 1) * 4096;
    uint32_t r0[16], r1[16];
    tc::tmem_ld16(t_row + c, r0);
    tc::tmem_ld16(t_row + c + 16, r1);
    if (turn >= 2 && lane == 0) tc::bulk_wait_read<1>();
    __syncwarp();
    tc::tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      *reinterpret_cast<uint4*>(b + lane * 128 + ((j ^ (lane & 7)) << 4)) =
          make_uint4(r0[4 * j], r0[4 * j + 1], r0[4 * j + 2], r0[4 * j + 3]);
      *reinterpret_cast<uint4*>(b + lane * 128 + (((j + 4) ^ (lane & 7)) << 4)) =
          make_uint4(r1[4 * j], r1[4 * j + 1], r1[4 * j + 2], r1[4 * j + 3]);
    }
    tc::fence_async_shared();
    __syncwarp();
    if (lane == 0) tc::tma_reduce_add_2d(tmD, b, n0 + c, row0);
  }
}

// epilogue_rows for outputs that leave as 32 x 32 boxes: a lane writes its row's 64 bytes into one of the warp's two 2 KB
// buffers (64-byte swizzle: 8 lanes' 16-byte chunks fall into 8 different columns of banks) and the TMA unit stores the box;
// what lies outside the matrix it leaves out.  Stored from the registers, every warp instruction touched 32 rows, one sector
// each.  The epilogue is what bounds the persistent kernel (of 7900 cycles a tile of 256 x 208 x 432 it took 6600, the MMAs
// 2900): forward 65536 x 400 x 432 34.3 us and input gradient 35.1 before, 30.4 and 28.5 with these boxes, the choice of ReLU
// outside the loop over elements, the mask words of the next tile loaded ahead, and no release at cluster scope behind a tile.
// gemm_kernel, one tile per CTA, stores from the registers: it would wait for its boxes at its end.
template <int EPI, bool RELU>
__device__ __forceinline__ void store_boxes(const GemmArgs& g, const CUtensorMap* tmD, uint8_t* buf, const float* s_bias,
                                            uint32_t t_row, int row0, int n0, int c_begin, int c_end, const RowMask& rm, int& turn) {
  const int lane = threadIdx.x & 31;
  if (row0 >= g.M) return;  // the same for the whole warp
  const int row = row0 + lane;
  for (int c = c_begin; c < c_end && n0 + c < g.N; c += 32, ++turn) {
    uint8_t* const b = buf + (turn & 1) * 2048;
    uint32_t r0[16], r1[16];
    tc::tmem_ld16(t_row + c, r0);
    tc::tmem_ld16(t_row + c + 16, r1);
    const uint32_t keep = EPI == EPI_RELU_MASK
                              ? rm.chunk((c - c_begin) >> 4) | (rm.chunk(((c - c_begin) >> 4) + 1) << 16) : 0;
    if (turn >= 2 && lane == 0) tc::bulk_wait_read<1>();
    __syncwarp();
    tc::tmem_ld_wait();
    uint32_t bits = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {  // eight columns, 16 bytes
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(q < 2 ? r0[8 * q + j] : r1[8 * (q - 2) + j]);
      if (EPI == EPI_BIAS_ACT) {
        const float4 ba = *reinterpret_cast<const float4*>(s_bias + c + 8 * q);
        const float4 bb = *reinterpret_cast<const float4*>(s_bias + c + 8 * q + 4);
        const float bias[8] = {ba.x, ba.y, ba.z, ba.w, bb.x, bb.y, bb.z, bb.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          v[j] += bias[j];
          if (RELU) v[j] = fmaxf(v[j], 0.f);
          bits |= (v[j] > 0.f ? 1u : 0u) << (8 * q + j);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (!((keep >> (8 * q + j)) & 1u)) v[j] = 0.f;
      }
      *reinterpret_cast<uint4*>(b + lane * 64 + ((q ^ ((lane >> 1) & 3)) << 4)) =
          make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
    }
    if (EPI == EPI_BIAS_ACT && g.mask_out != nullptr && row < g.M) {
      uint16_t* const m = g.mask_out + static_cast<size_t>((n0 + c) >> 4) * g.ldm + row;
      m[0] = static_cast<uint16_t>(bits);
      if (n0 + c + 16 < g.N) m[g.ldm] = static_cast<uint16_t>(bits >> 16);
    }
    tc::fence_async_shared();
    __syncwarp();
    if (lane == 0) tc::tma_store_2d(tmD, b, n0 + c, row0);
  }
}

template <int EPI>
__device__ __forceinline__ void epilogue_store(const GemmArgs& g, const CUtensorMap* tmD, uint8_t* buf, const float* s_bias,
                                               uint32_t t_row, int row0, int n0, int c_begin, int c_end, const RowMask& rm,
                                               int& turn) {
  if (EPI == EPI_BIAS_ACT && g.relu)
    store_boxes<EPI, true>(g, tmD, buf, s_bias, t_row, row0, n0, c_begin, c_end, rm, turn);
  else
    store_boxes<EPI, false>(g, tmD, buf, s_bias, t_row, row0, n0, c_begin, c_end, rm, turn);
  if (EPI == EPI_RELU_MASK) clear_behind(g, row0 + (threadIdx.x & 31), n0, c_begin, c_end);
}

// Column range of epilogue warp `ew` (0 .. kEpiWarps - 1): the tile's chunks of `unit` columns are split
// between the two warps that share a TMEM lane quarter.
__device__ __forceinline__ void epi_cols(int bn, int ew, int* c_begin, int* c_end, int unit = 16) {
  const int chunks = bn / unit;
  const int first = (chunks + 1) / 2;
  if (ew < 4) {
    *c_begin = 0;
    *c_end = first * unit;
  } else {
    *c_begin = first * unit;
    *c_end = bn;
  }
}

// Adds one stage of an MN-major A tile (two boxes of 64 rows x 64 columns, 128-byte swizzle) to the column sums that the
// 256 epilogue threads keep: a thread owns 8 columns of a box and 4 of its rows, 16-byte reads.
__device__ __forceinline__ void add_stage_columns(const uint8_t* a, int t, float (&acc)[8]) {
  const uint8_t* box = a + (t >> 7) * 8192;
  const int chunk = t & 7, r0 = (t >> 3) & 15;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int r = r0 + 16 * j;
    const uint4 v = *reinterpret_cast<const uint4*>(box + r * 128 + ((chunk ^ (r & 7)) << 4));
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      acc[2 * q] += __uint_as_float(w[q] << 16);
      acc[2 * q + 1] += __uint_as_float(w[q] & 0xFFFF0000u);
    }
  }
}

// Bias of the tile's columns into shared memory (zeros where there is none).
__device__ __forceinline__ void stage_bias(const GemmArgs& g, float* s_bias, int n0, int tid, int nthreads) {
  for (int j = tid; j < 256; j += nthreads) s_bias[j] = (g.bias && j < g.BN && n0 + j < g.N) ? g.bias[n0 + j] : 0.f;
}

// Descriptor of the first k-step of an operand's tile at `tile`; a stage further adds its bytes / 16, a k-step `k_step`.
template <bool MN>
__device__ __forceinline__ uint64_t stage_desc(const uint8_t* tile) {
  return MN ? tc::smem_desc(tc::smem_u32(tile), 8192, 1024) : tc::smem_desc(tc::smem_u32(tile), 16, 1024);
}
template <bool MN>
constexpr uint32_t k_step = (MN ? 2048 : 32) >> 4;

// Threads of gemm_kernel: the four boxes of an MN-major B are issued by a warp of their own (10), beside the two of A.  One
// thread took 600 cycles for the six, more than their MMAs: batch 8192 of 400 x 400 11.6 us, 11.1 so.
template <bool B_MN>
constexpr int kTileThreads = kThreads + (B_MN ? 32 : 0);

template <bool A_MN, bool B_MN, int EPI>
__global__ void __launch_bounds__(kTileThreads<B_MN>)
gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
            const __grid_constant__ CUtensorMap tmD, const __grid_constant__ GemmArgs g) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t a_bytes = kBM * 128;
  const uint32_t b_bytes = static_cast<uint32_t>(g.BN) * 128;
  const uint32_t stage_bytes = a_bytes + b_bytes;

  __shared__ uint64_t full_bar[kMaxStages];
  __shared__ uint64_t empty_bar[kMaxStages];
  __shared__ uint64_t acc_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  __shared__ __align__(16) float s_bias[256];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * kBM;
  const int n0 = blockIdx.y * g.BN;
  const int total_kb = (g.K + kBK - 1) / kBK;
  const int kb_begin = blockIdx.z * g.kb_per_split;
  const int kb_end = min(total_kb, kb_begin + g.kb_per_split);
  const int num_kb = max(0, kb_end - kb_begin);
  uint32_t tmem_cols = 32;
  while (tmem_cols < static_cast<uint32_t>(g.BN)) tmem_cols <<= 1;

  // The epilogue warps are idle until the accumulator is complete: in one column of tiles they sum the columns of A as
  // it passes through shared memory, which is the bias gradient of the layer.  A kernel of its own read all of dY again:
  // three layers of 65536 x 400 took 125 us of the stream that the weight gradients share with the backward chain.
  const bool sums = A_MN && EPI == EPI_RED_F32 && g.col_sums != nullptr && blockIdx.y == 0;
  if (threadIdx.x == 0) {
    for (int s = 0; s < g.stages; ++s) {
      tc::mbar_init(&full_bar[s], 1);
      tc::mbar_init(&empty_bar[s], sums ? 1 + kEpiWarps : 1);  // the MMAs that read the stage, and the summing warps
    }
    tc::mbar_init(&acc_bar, 1);
    abort_flag = 0;
    tc::fence_barrier_init();
    tc::prefetch_tmap(&tmA);
    tc::prefetch_tmap(&tmB);
  }
  if (warp == 1) tc::tmem_alloc(&tmem_slot, tmem_cols);
  if (EPI == EPI_BIAS_ACT) stage_bias(g, s_bias, n0, threadIdx.x, blockDim.x);
  if (EPI == EPI_RED_F32 && threadIdx.x < kBM) s_bias[threadIdx.x] = 0.f;  // the column sums meet here
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  pdl_enter();  // everything above touches nothing the kernel in front of this one writes
  const uint32_t tmem_base = tmem_slot;

  const bool b_producer = B_MN && warp == 2 + kEpiWarps;
  if ((warp == 0 || b_producer) && lane == 0) {
    // ---------------- TMA producer
    bool ok = true;
    Ring ring;
    for (int i = 0; i < num_kb; ++i, ring.next(g.stages)) {
      const int s = ring.s;
      ok = tc::mbar_wait(&empty_bar[s], ring.parity ^ 1, kWaitLimit);  // the first round finds the stages free
      if (!ok) break;
      uint8_t* a_dst = smem + static_cast<size_t>(s) * stage_bytes;
      uint8_t* b_dst = a_dst + a_bytes;
      const int k0 = (kb_begin + i) * kBK;
      if (b_producer) {  // the bytes may arrive before warp 0 expects them: the phase waits for its arrival
        for (int j = 0; j < g.BN / 64; ++j) tc::tma_load_2d(b_dst + j * 8192, &tmB, &full_bar[s], n0 + 64 * j, k0);
        continue;
      }
      tc::mbar_expect_tx(&full_bar[s], stage_bytes);
      if (A_MN) {
        for (int j = 0; j < kBM / 64; ++j) tc::tma_load_2d(a_dst + j * 8192, &tmA, &full_bar[s], m0 + 64 * j, k0);
      } else {
        tc::tma_load_2d(a_dst, &tmA, &full_bar[s], k0, m0);
      }
      if (!B_MN) tc::tma_load_2d(b_dst, &tmB, &full_bar[s], k0, n0);
    }
    if (!ok) {
      atomicCAS(g.status, 0, err::kTimeout);
      abort_flag = 1;
    }
  } else if (warp == 1 && lane == 0) {
    // ---------------- MMA issuer
    const uint32_t idesc = tc::instr_desc_bf16(kBM, g.BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
    bool ok = true, ready = false;
    Ring ring;
    const uint64_t ad0 = stage_desc<A_MN>(smem), bd0 = stage_desc<B_MN>(smem + a_bytes);
    for (int i = 0; i < num_kb; ++i, ring.next(g.stages)) {
      const int s = ring.s;
      if (!ready) ok = tc::mbar_wait(&full_bar[s], ring.parity, kWaitLimit);
      if (!ok) break;
      tc::fence_after_sync();
      const uint32_t at = s * (stage_bytes >> 4);
      Ring ahead = ring;
      ahead.next(g.stages);
#pragma unroll
      for (int k = 0; k < kBK / 16; ++k) {
        if (k == 2) ready = tc::mbar_test(&full_bar[ahead.s], ahead.parity);  // see Ring
        tc::mma_bf16(tmem_base, ad0 + at + k * k_step<A_MN>, bd0 + at + k * k_step<B_MN>, idesc, (i > 0 || k > 0) ? 1u : 0u);
      }
      tc::mma_commit(&empty_bar[s]);  // the stage is free again once these MMAs have read it
    }
    if (ok) {
      tc::mma_commit(&acc_bar);
    } else {
      atomicCAS(g.status, 0, err::kTimeout);
      abort_flag = 1;
      tc::mbar_arrive(&acc_bar);  // release the epilogue warps; they see abort_flag and skip
    }
  } else if (warp >= 2 && warp < 2 + kEpiWarps) {
    // ---------------- epilogue: thread = one accumulator row, warp = one column half
    const int quarter = warp & 3;  // a warp may only read TMEM lanes [32 * (warp % 4), +32)
    const int row = m0 + quarter * 32 + lane;
    int c_begin, c_end;
    epi_cols(g.BN, warp - 2, &c_begin, &c_end);
    RowMask rm{~0ull, ~0ull};
    if (EPI == EPI_RELU_MASK) rm = load_row_mask(g, row, (n0 + c_begin) >> 4, (c_end - c_begin + 15) >> 4);
    if (A_MN && EPI == EPI_RED_F32 && sums) {
      const int t = threadIdx.x - 64;
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      bool fine = true;
      Ring ring;
      for (int i = 0; i < num_kb && fine; ++i, ring.next(g.stages)) {
        const int s = ring.s;
        fine = tc::mbar_wait(&full_bar[s], ring.parity, kWaitLimit);
        fine = __all_sync(0xffffffffu, fine);
        if (!fine) break;
        add_stage_columns(smem + static_cast<size_t>(s) * stage_bytes, t, acc);
        // The stage may be refilled once the warp has arrived, so what was read must be in registers by then: which lane
        // arrives depends on a vote over values that all of the lanes' reads went into.  (An arrival behind a mere
        // __syncwarp overtook reads that other kernels' memory traffic on the SM had held up.)
        const unsigned landed = __ballot_sync(0xffffffffu, __float_as_uint(acc[0]) != 0x7FFFDEADu);
        if (lane == (landed ? __ffs(landed) - 1 : 0)) tc::mbar_arrive(&empty_bar[s]);
      }
      if (!fine && lane == 0) atomicCAS(g.status, 0, err::kTimeout);
#pragma unroll
      for (int q = 0; q < 8; ++q) {  // lanes 8 apart hold other rows of the same columns
        acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], 8);
        acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], 16);
      }
      if (lane < 8) {
#pragma unroll
        for (int q = 0; q < 8; ++q) atomicAdd(&s_bias[(t >> 7) * 64 + lane * 8 + q], acc[q]);
      }
      asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpiWarps) : "memory");  // the epilogue warps only
      if (fine && t < kBM && m0 + t < g.M) atomicAdd(g.col_sums + m0 + t, s_bias[t]);
    }
    const bool ok = tc::mbar_wait(&acc_bar, 0, kWaitLimit);
    tc::fence_after_sync();
    if (!ok && lane == 0) atomicCAS(g.status, 0, err::kTimeout);
    if (EPI == EPI_RED_F32) {
      // every stage has been read by then: by the MMAs (acc_bar) and by the summing warps (their barrier)
      int turn = 0;
      if (ok && abort_flag == 0 && num_kb > 0)
        epilogue_reduce(g, &tmD, smem + (warp - 2) * 8192, tmem_base + (static_cast<uint32_t>(quarter * 32) << 16),
                        m0 + quarter * 32, n0, c_begin, c_end, turn);
      if (lane == 0) tc::bulk_wait_all();
    } else if (ok && abort_flag == 0 && num_kb > 0)
      epilogue_rows<EPI>(g, s_bias, tmem_base + (static_cast<uint32_t>(quarter * 32) << 16), row, n0, c_begin, c_end, rm);
  }

  // ---------------- teardown: let the copies that were issued land, then free tensor memory
  if (warp == 0 && lane == 0) {
    const int first = max(0, num_kb - g.stages);
    for (int i = first; i < num_kb; ++i)
      tc::mbar_wait(&full_bar[i % g.stages], static_cast<uint32_t>(i / g.stages) & 1, kWaitLimit);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 1) tc::tmem_dealloc(tmem_base, tmem_cols);
}

// ------------------------------------------------------------------ weight-resident persistent variant
// Forward and input-gradient GEMMs of an MLP are tall and skinny: M = batch (tens of thousands),
// N and K a few hundred.  With one output tile per CTA every CTA re-reads its 128 x K slice of the
// weights from L2, and that traffic, not the tensor cores, sets the time.  Here a CTA (one per SM)
// loads its BN x K slice of the weight matrix ONCE, keeps it in shared memory, and then streams
// activation tiles for many 128-row tiles through a small ring, with two TMEM accumulators so the
// epilogue of tile j overlaps the MMAs of tile j + 1.
template <int EPI>
__global__ void __launch_bounds__(kThreads, 1)
gemm_bres_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ GemmArgs g) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int total_kb = (g.K + kBK - 1) / kBK;
  const uint32_t a_bytes = kBM * 128;
  const uint32_t b_bytes = static_cast<uint32_t>(g.BN) * 128;  // one k-block of the resident weights
  uint8_t* b_res = smem;
  uint8_t* a_ring = smem + static_cast<size_t>(total_kb) * b_bytes;

  __shared__ uint64_t b_full, a_full[kMaxStages], a_empty[kMaxStages], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  __shared__ __align__(16) float s_bias[256];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int n0 = blockIdx.y * g.BN;
  const int m_tiles = (g.M + kBM - 1) / kBM;
  const int my_tiles = (m_tiles - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
  constexpr uint32_t kAccCols = 256;  // column stride between the two accumulators

  if (threadIdx.x == 0) {
    tc::mbar_init(&b_full, 1);
    for (int s = 0; s < g.stages; ++s) {
      tc::mbar_init(&a_full[s], 1);
      tc::mbar_init(&a_empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&acc_full[b], 1);
      tc::mbar_init(&acc_empty[b], kEpiWarps);  // one arrival per epilogue warp
    }
    abort_flag = 0;
    tc::fence_barrier_init();
    tc::prefetch_tmap(&tmA);
    tc::prefetch_tmap(&tmB);
  }
  if (warp == 1) tc::tmem_alloc(&tmem_slot, 512);
  if (EPI == EPI_BIAS_ACT) stage_bias(g, s_bias, n0, threadIdx.x, blockDim.x);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  pdl_enter();  // everything above touches nothing the kernel in front of this one writes
  const uint32_t tmem_base = tmem_slot;
  const int total_it = my_tiles * total_kb;

  if (warp == 0 && lane == 0) {
    // ---------------- producer: the weights once, then the activation stream
    tc::mbar_expect_tx(&b_full, static_cast<uint32_t>(total_kb) * b_bytes);
    for (int kb = 0; kb < total_kb; ++kb)
      tc::tma_load_2d(b_res + static_cast<size_t>(kb) * b_bytes, &tmB, &b_full, kb * kBK, n0);
    bool ok = true;
    Ring ring;
    for (int tile = blockIdx.x; tile < m_tiles && ok; tile += gridDim.x) {
      for (int kb = 0; kb < total_kb; ++kb, ring.next(g.stages)) {
        const int s = ring.s;
        ok = tc::mbar_wait(&a_empty[s], ring.parity ^ 1, kWaitLimit);  // the first round finds the stages free
        if (!ok) break;
        tc::mbar_expect_tx(&a_full[s], a_bytes);
        tc::tma_load_2d(a_ring + static_cast<size_t>(s) * a_bytes, &tmA, &a_full[s], kb * kBK, tile * kBM);
      }
    }
    if (!ok) {
      atomicCAS(g.status, 0, err::kTimeout);
      abort_flag = 1;
    }
  } else if (warp == 1 && lane == 0) {
    // ---------------- MMA issuer
    const uint32_t idesc = tc::instr_desc_bf16(kBM, g.BN, 0, 0);
    bool ready = false;
    bool ok = tc::mbar_wait(&b_full, 0, kWaitLimit);
    tc::fence_after_sync();
    const uint64_t bd0 = stage_desc<false>(b_res), ad0 = stage_desc<false>(a_ring);
    Ring ring;
    for (int j = 0; j < my_tiles && ok; ++j) {
      const int buf = j & 1;
      const uint32_t use = static_cast<uint32_t>(j >> 1);
      if (use > 0) {
        ok = tc::mbar_wait(&acc_empty[buf], (use - 1) & 1, kWaitLimit);  // epilogue has drained this buffer
        if (!ok) break;
        tc::fence_after_sync();
      }
      const uint32_t d_tmem = tmem_base + buf * kAccCols;
      for (int kb = 0; kb < total_kb; ++kb, ring.next(g.stages)) {
        const int s = ring.s;
        if (!ready) ok = tc::mbar_wait(&a_full[s], ring.parity, kWaitLimit);
        if (!ok) break;
        tc::fence_after_sync();
        const uint64_t ad = ad0 + s * (a_bytes >> 4), bd = bd0 + kb * (b_bytes >> 4);
        Ring ahead = ring;
        ahead.next(g.stages);
#pragma unroll
        for (int k = 0; k < kBK / 16; ++k) {
          if (k == 2) ready = tc::mbar_test(&a_full[ahead.s], ahead.parity);  // see Ring
          tc::mma_bf16(d_tmem, ad + k * k_step<false>, bd + k * k_step<false>, idesc, (kb > 0 || k > 0) ? 1u : 0u);
        }
        tc::mma_commit(&a_empty[s]);
      }
      if (ok) tc::mma_commit(&acc_full[buf]);
    }
    if (!ok) {
      atomicCAS(g.status, 0, err::kTimeout);
      abort_flag = 1;
      tc::mbar_arrive(&acc_full[0]);
      tc::mbar_arrive(&acc_full[1]);
    }
  } else if (warp >= 2) {
    // ---------------- epilogue
    const int quarter = warp & 3;
    int c_begin, c_end;
    epi_cols(g.BN, warp - 2, &c_begin, &c_end);
    bool ok = true;
    for (int j = 0; j < my_tiles && ok; ++j) {
      const int buf = j & 1;
      const int tile = blockIdx.x + j * gridDim.x;
      const int row = tile * kBM + quarter * 32 + lane;
      RowMask rm{~0ull, ~0ull};
      if (EPI == EPI_RELU_MASK) rm = load_row_mask(g, row, (n0 + c_begin) >> 4, (c_end - c_begin + 15) >> 4);
      ok = tc::mbar_wait(&acc_full[buf], static_cast<uint32_t>(j >> 1) & 1, kWaitLimit);
      tc::fence_after_sync();
      if (!ok || abort_flag != 0) {
        if (!ok && lane == 0) atomicCAS(g.status, 0, err::kTimeout);
        ok = false;
        break;
      }
      epilogue_rows<EPI>(g, s_bias, tmem_base + buf * kAccCols + (static_cast<uint32_t>(quarter * 32) << 16), row, n0,
                         c_begin, c_end, rm);
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&acc_empty[buf]);
    }
  }

  // ---------------- teardown
  if (warp == 0 && lane == 0) {
    tc::mbar_wait(&b_full, 0, kWaitLimit);
    const int first = max(0, total_it - g.stages);
    for (int it = first; it < total_it; ++it)
      tc::mbar_wait(&a_full[it % g.stages], static_cast<uint32_t>(it / g.stages) & 1, kWaitLimit);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 1) tc::tmem_dealloc(tmem_base, 512);
}

// ------------------------------------------------------------------ weight-resident CTA-pair variant
// The single-CTA resident kernel above is bound by what one SM can take in: every MMA reads
// (128 + BN) x 32 bytes of operands from shared memory, which keeps the shared-memory port busy
// for most of the MMA's duration and stalls the TMA stream that shares it, and a column tile
// narrow enough to leave room for a deep activation ring makes every activation tile cross the
// L2-to-SM fabric once per column tile.  A pair of CTAs on one TPC running tcgen05.mma with
// cta_group::2 fixes both: each CTA keeps only half of the column tile's weights (so the same
// shared memory holds a wider tile AND a deeper ring) and reads only half of the B bytes per MMA.
//
//   cluster = 2 CTAs; pair tile = 256 rows x BN columns; CTA r loads rows [r * 128, +128) of A and
//   weight rows [n0 + r * BN / 2, +BN / 2); the even CTA's warp 1 issues every MMA; the byte
//   counts of both CTAs' loads complete on the even CTA's barriers; tcgen05.commit with a CTA
//   mask frees ring stages and publishes accumulators in both CTAs; epilogue warps of both CTAs
//   release an accumulator buffer by arriving on the even CTA's barrier.
template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmD, const __grid_constant__ GemmArgs g) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int total_kb = (g.K + kBK - 1) / kBK;
  const int half_bn = g.BN / 2;
  const uint32_t a_bytes = kBM * 128;
  const uint32_t b_bytes = static_cast<uint32_t>(half_bn) * 128;  // one k-block of this CTA's half of the weights
  uint8_t* b_res = smem;
  uint8_t* a_ring = smem + static_cast<size_t>(total_kb) * b_bytes;
  uint8_t* const staging = a_ring + static_cast<size_t>(g.stages) * a_bytes;  // boxes of the output on their way out

  __shared__ uint64_t b_full, a_full[kMaxStages], a_empty[kMaxStages], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  __shared__ __align__(16) float s_bias[256];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = tc::cluster_ctarank();  // 0 = the CTA that issues the MMAs
  const int pair = blockIdx.x >> 1;
  const int pairs = gridDim.x >> 1;
  const int n0 = blockIdx.y * g.BN;
  const int m_tiles = (g.M + 2 * kBM - 1) / (2 * kBM);  // pair tiles of 256 rows
  const int my_tiles = (m_tiles - pair + pairs - 1) / pairs;
  constexpr uint32_t kAccCols = 256;

  if (threadIdx.x == 0) {
    tc::mbar_init(&b_full, 1);
    for (int s = 0; s < g.stages; ++s) {
      tc::mbar_init(&a_full[s], 1);
      tc::mbar_init(&a_empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&acc_full[b], 1);
      tc::mbar_init(&acc_empty[b], 2 * kEpiWarps);  // every epilogue warp of both CTAs
    }
    abort_flag = 0;
    tc::fence_barrier_init();
    tc::prefetch_tmap(&tmA);
    tc::prefetch_tmap(&tmB);
  }
  if (warp == 1) tc::tmem_alloc_pair(&tmem_slot, 512);
  if (EPI == EPI_BIAS_ACT) stage_bias(g, s_bias, n0, threadIdx.x, blockDim.x);
  tc::fence_before_sync();
  __syncthreads();
  tc::cluster_sync_all();  // the other CTA's barriers exist before anything arrives on them
  tc::fence_after_sync();
  pdl_enter();  // everything above touches nothing the kernel in front of this one writes
  const uint32_t tmem_base = tmem_slot;
  const int total_it = my_tiles * total_kb;

  if (warp == 0 && lane == 0) {
    // ---------------- producer (both CTAs): own half of the weights once, then own rows of the stream
    const uint32_t lead_b_full = tc::map_to_cta(tc::smem_u32(&b_full), 0);
    if (rank == 0) tc::mbar_expect_tx(&b_full, 2u * static_cast<uint32_t>(total_kb) * b_bytes);
    for (int kb = 0; kb < total_kb; ++kb)
      tc::tma_load_2d_pair(b_res + static_cast<size_t>(kb) * b_bytes, &tmB, lead_b_full, kb * kBK,
                           n0 + static_cast<int>(rank) * half_bn);
    bool ok = true;
    Ring ring;
    const uint32_t lead_a_full = tc::map_to_cta(tc::smem_u32(&a_full[0]), 0);
    for (int tile = pair; tile < m_tiles && ok; tile += pairs) {
      for (int kb = 0; kb < total_kb; ++kb, ring.next(g.stages)) {
        const int s = ring.s;
        ok = tc::mbar_wait(&a_empty[s], ring.parity ^ 1, kWaitLimit);  // the first round finds the stages free
        if (!ok) break;
        if (rank == 0) tc::mbar_expect_tx(&a_full[s], 2u * a_bytes);
        tc::tma_load_2d_pair(a_ring + static_cast<size_t>(s) * a_bytes, &tmA, lead_a_full + s * 8, kb * kBK,
                             tile * 2 * kBM + static_cast<int>(rank) * kBM);
      }
    }
    if (!ok) {
      atomicCAS(g.status, 0, err::kTimeout);
      abort_flag = 1;
    }
  } else if (warp == 1 && lane == 0 && rank == 0) {
    // ---------------- MMA issuer (even CTA only)
    const uint32_t idesc = tc::instr_desc_bf16(2 * kBM, g.BN, 0, 0);
    bool ready = false;
    bool ok = tc::mbar_wait(&b_full, 0, kWaitLimit);
    tc::fence_after_sync();
    const uint64_t bd0 = stage_desc<false>(b_res), ad0 = stage_desc<false>(a_ring);
    Ring ring;
    for (int j = 0; j < my_tiles && ok; ++j) {
      const int buf = j & 1;
      const uint32_t use = static_cast<uint32_t>(j >> 1);
      if (use > 0) {
        ok = tc::mbar_wait(&acc_empty[buf], (use - 1) & 1, kWaitLimit);
        if (!ok) break;
        tc::fence_after_sync();
      }
      const uint32_t d_tmem = tmem_base + buf * kAccCols;
      for (int kb = 0; kb < total_kb; ++kb, ring.next(g.stages)) {
        const int s = ring.s;
        if (!ready) ok = tc::mbar_wait(&a_full[s], ring.parity, kWaitLimit);
        if (!ok) break;
        tc::fence_after_sync();
        const uint64_t ad = ad0 + s * (a_bytes >> 4), bd = bd0 + kb * (b_bytes >> 4);
        Ring ahead = ring;
        ahead.next(g.stages);
#pragma unroll
        for (int k = 0; k < kBK / 16; ++k) {
          if (k == 2) ready = tc::mbar_test(&a_full[ahead.s], ahead.parity);  // see Ring
          tc::mma_bf16_pair(d_tmem, ad + k * k_step<false>, bd + k * k_step<false>, idesc, (kb > 0 || k > 0) ? 1u : 0u);
        }
        tc::mma_commit_pair(&a_empty[s], 3);  // the stage is free in both CTAs
      }
      if (ok) tc::mma_commit_pair(&acc_full[buf], 3);
    }
    if (!ok) {
      atomicCAS(g.status, 0, err::kTimeout);
      abort_flag = 1;
    }
  } else if (warp >= 2) {
    // ---------------- epilogue (both CTAs, each on its own 128 rows)
    const int quarter = warp & 3;
    const uint32_t lead_acc_empty[2] = {tc::map_to_cta(tc::smem_u32(&acc_empty[0]), 0),
                                        tc::map_to_cta(tc::smem_u32(&acc_empty[1]), 0)};
    int c_begin, c_end;
    epi_cols(g.BN, warp - 2, &c_begin, &c_end, g.out_tma ? 32 : 16);
    int turn = 0;
    bool ok = true;
    const int chunk0 = (n0 + c_begin) >> 4, chunks = (c_end - c_begin + 15) >> 4;
    int row = pair * 2 * kBM + static_cast<int>(rank) * kBM + quarter * 32 + lane;
    MaskWords words;  // of the tile that comes next: a tile's own would be waited for
    if (EPI == EPI_RELU_MASK) words.load(g, row, chunk0, chunks);
    for (int j = 0; j < my_tiles && ok; ++j, row += pairs * 2 * kBM) {
      const int buf = j & 1;
      RowMask rm{~0ull, ~0ull};
      if (EPI == EPI_RELU_MASK) {
        rm = words.packed();
        words.load(g, row + pairs * 2 * kBM, chunk0, chunks);  // none behind the last row
      }
      ok = tc::mbar_wait(&acc_full[buf], static_cast<uint32_t>(j >> 1) & 1, kWaitLimit);
      tc::fence_after_sync();
      if (!ok) {
        if (lane == 0) atomicCAS(g.status, 0, err::kTimeout);
        break;
      }
      const uint32_t t_row = tmem_base + buf * kAccCols + (static_cast<uint32_t>(quarter * 32) << 16);
      if (g.out_tma)
        epilogue_store<EPI>(g, &tmD, staging + (warp - 2) * 4096, s_bias, t_row, row - lane, n0, c_begin, c_end, rm, turn);
      else
        epilogue_rows<EPI>(g, s_bias, t_row, row, n0, c_begin, c_end, rm);
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive_cluster(lead_acc_empty[buf]);
    }
    if (lane == 0) tc::bulk_wait_all();
  }

  // ---------------- teardown: the even CTA's barriers count both CTAs' copies
  if (warp == 0 && lane == 0 && rank == 0) {
    tc::mbar_wait(&b_full, 0, kWaitLimit);
    const int first = max(0, total_it - g.stages);
    for (int it = first; it < total_it; ++it)
      tc::mbar_wait(&a_full[it % g.stages], static_cast<uint32_t>(it / g.stages) & 1, kWaitLimit);
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::cluster_sync_all();  // neither CTA leaves while the other may still touch its memory or barriers
  if (warp == 1) tc::tmem_dealloc_pair(tmem_base, 512);
}

// ------------------------------------------------------------------ weight gradients on CTA pairs
// dW [N, K] += dY^T X: both operands MN-major, the contraction is the batch, and both stream through a ring past 256-row
// tiles of a CTA pair (cta_group::2; CTA r holds dY columns [m0 + r * 128, +128) and its half of the X columns of a sub-tile).
// What bounded gemm_kernel here was its producer: a k-block of a 128 x 256 tile is six boxes of 64 x 64, 100 cycles each to
// issue, and with the wait for the stage that is 800 cycles where the MMAs take 512; and it brings 48 KB in for them, which
// is 10 TB/s over all SMs.  A pair needs 32 KB per CTA for the same products, and with two sub-tiles of 256 columns - 512 in
// ONE tile, all of tensor memory - 24 KB: dY crosses the fabric once and X once per 256 rows.  The boxes are issued by three warps:
// dY, and each sub-tile's half of X.  Batch 65536 of 400 x 432: 38.1 us there, 31.2 here, of which 16 are MMAs; 4096 x 4096 at
// batch 1024 51 and 39.5.  What is left is the start, and the reductions of 37 partial sums into L2.
//
// A work item is a tile and a range of k-blocks; a pair takes items pair, pair + pairs, ...  Warps 10-13 exist where the bias
// gradient is wanted: they add up the columns of the dY tiles of the items in the first column of tiles.  The byte counts of
// both CTAs' copies complete on the even CTA's barriers, which only that CTA can wait on, so the summing warps of both take a
// stage when its MMAs have read it (`landed`: the commit arrives in both CTAs), and they, not the commit, free it.  (Passing
// the even CTA's barrier on by a remote arrival took 1500 cycles of its MMA thread per k-block.)
constexpr int kSumWarps = 4;
constexpr int kProducers = 3;                              // warps 0, 14 and 15
constexpr int kPairWgradThreads = kThreads + 32 * (kSumWarps + kProducers - 1);

constexpr int kSubs = 2, kSubCols = 256;  // a tile: two MMAs of 256 rows x 256 columns

struct Item {
  int m0, n0, kb0, kb1;
  bool first_col;
};

__device__ __forceinline__ Item item_at(const GemmArgs& g, int i, int total_kb) {
  Item t;
  const int tm = i % g.tiles_m, rest = i / g.tiles_m;
  const int tn = rest % g.tiles_n, split = rest / g.tiles_n;
  t.m0 = tm * 2 * kBM;
  t.n0 = tn * kSubs * kSubCols;
  t.kb0 = split * g.kb_per_split;
  t.kb1 = min(total_kb, t.kb0 + g.kb_per_split);
  t.first_col = tn == 0;
  return t;
}

// 64-element boxes of an operand that lie inside the matrix; the others are not loaded (what their part of the stage holds
// only reaches accumulator rows or columns outside the output).
__device__ __forceinline__ int boxes_inside(int begin, int width, int limit) {
  const int inside = min(width, limit - begin);
  return inside <= 0 ? 0 : (inside + 63) / 64;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairWgradThreads, 2)
gemm_pair_wgrad_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                       const __grid_constant__ CUtensorMap tmD, const __grid_constant__ GemmArgs g) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int half_bn = kSubCols / 2;
  constexpr uint32_t a_bytes = kBM * 128;
  constexpr uint32_t b_bytes = half_bn * 128;  // this CTA's half of one sub-tile
  constexpr uint32_t stage_bytes = a_bytes + kSubs * b_bytes;
  // boxes of the epilogue's TMA reductions: behind the ring, or, where every pair has one item, in it
  const bool in_ring = g.items <= static_cast<int>(gridDim.x >> 1);
  uint8_t* const staging = smem + (in_ring ? 0 : static_cast<size_t>(g.stages) * stage_bytes);

  __shared__ uint64_t full_bar[kMaxStages], empty_bar[kMaxStages], landed_bar[kMaxStages], acc_full, acc_empty;
  __shared__ uint32_t tmem_slot;
  __shared__ float s_sum[kBM];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = tc::cluster_ctarank();
  const int pair = blockIdx.x >> 1;
  const int pairs = gridDim.x >> 1;
  const int total_kb = (g.K + kBK - 1) / kBK;
  const bool sums = g.col_sums != nullptr;

  if (threadIdx.x == 0) {
    for (int s = 0; s < g.stages; ++s) {
      tc::mbar_init(&full_bar[s], 1);
      tc::mbar_init(&empty_bar[s], sums ? kSumWarps : 1);
      tc::mbar_init(&landed_bar[s], 1);
    }
    tc::mbar_init(&acc_full, 1);
    tc::mbar_init(&acc_empty, 2 * kEpiWarps);
    tc::fence_barrier_init();
    tc::prefetch_tmap(&tmA);
    tc::prefetch_tmap(&tmB);
  }
  if (warp == 1) tc::tmem_alloc_pair(&tmem_slot, 512);
  if (threadIdx.x < kBM) s_sum[threadIdx.x] = 0.f;
  tc::fence_before_sync();
  __syncthreads();
  tc::cluster_sync_all();  // the other CTA's barriers exist before anything arrives on them
  tc::fence_after_sync();
  pdl_enter();  // everything above touches nothing the kernel in front of this one writes
  const uint32_t tmem_base = tmem_slot;

  const int producer = warp == 0 ? 0 : warp - (2 + kEpiWarps + kSumWarps) + 1;  // 0: dY, 1 and 2: sub-tiles of X
  if ((warp == 0 || producer > 0) && lane == 0) {
    // ---------------- producers (both CTAs)
    bool ok = true;
    int it = 0;
    Ring ring;
    const uint32_t lead_full = tc::map_to_cta(tc::smem_u32(&full_bar[0]), 0);
    for (int i = pair; i < g.items && ok; i += pairs) {
      const Item t = item_at(g, i, total_kb);
      uint32_t bytes = 0;  // of both CTAs' copies of a k-block
      for (int r = 0; r < 2; ++r) {
        bytes += boxes_inside(t.m0 + r * kBM, kBM, g.M) * 8192;
        for (int u = 0; u < kSubs; ++u) bytes += boxes_inside(t.n0 + u * kSubCols + r * half_bn, half_bn, g.N) * 8192;
      }
      const CUtensorMap* const tm = producer == 0 ? &tmA : &tmB;
      const int x0 = producer == 0 ? t.m0 + static_cast<int>(rank) * kBM
                                   : t.n0 + (producer - 1) * kSubCols + static_cast<int>(rank) * half_bn;
      const int boxes = producer == 0 ? boxes_inside(x0, kBM, g.M) : boxes_inside(x0, half_bn, g.N);
      uint8_t* const base = smem + (producer == 0 ? 0 : a_bytes + (producer - 1) * b_bytes);
      for (int kb = t.kb0; kb < t.kb1; ++kb, ++it, ring.next(g.stages)) {
        const int s = ring.s;
        ok = tc::mbar_wait(&empty_bar[s], ring.parity ^ 1, kWaitLimit);  // the first round finds the stages free
        if (!ok) break;
        if (producer == 0 && rank == 0) tc::mbar_expect_tx(&full_bar[s], bytes);
        uint8_t* const dst = base + static_cast<size_t>(s) * stage_bytes;
        for (int j = 0; j < boxes; ++j) tc::tma_load_2d_pair(dst + j * 8192, tm, lead_full + s * 8, x0 + 64 * j, kb * kBK);
      }
    }
    if (!ok) atomicCAS(g.status, 0, err::kTimeout);
    if (producer == 0 && rank == 0) {  // the even CTA's barriers count both CTAs' copies: let the last of them land
      for (int k = max(0, it - g.stages); k < it; ++k)
        tc::mbar_wait(&full_bar[k % g.stages], static_cast<uint32_t>(k / g.stages) & 1, kWaitLimit);
    }
  } else if (warp == 1 && lane == 0 && rank == 0) {
    // ---------------- MMA issuer (even CTA only)
    const uint32_t idesc = tc::instr_desc_bf16(2 * kBM, kSubCols, 1, 1);
    bool ok = true, ready = false;
    int j = 0;
    Ring ring;
    const uint64_t ad0 = stage_desc<true>(smem), bd0 = stage_desc<true>(smem + a_bytes);
    uint64_t* const read_bar = sums ? landed_bar : empty_bar;
    for (int i = pair; i < g.items && ok; i += pairs, ++j) {
      const Item t = item_at(g, i, total_kb);
      if (j > 0) {
        ok = tc::mbar_wait(&acc_empty, static_cast<uint32_t>(j - 1) & 1, kWaitLimit);
        if (!ok) break;
        tc::fence_after_sync();
      }
      for (int kb = t.kb0; kb < t.kb1; ++kb, ring.next(g.stages)) {
        const int s = ring.s;
        if (!ready) ok = tc::mbar_wait(&full_bar[s], ring.parity, kWaitLimit);
        if (!ok) break;
        tc::fence_after_sync();
        const uint32_t at = s * (stage_bytes >> 4);
        Ring ahead = ring;
        ahead.next(g.stages);
#pragma unroll
        for (int k = 0; k < kBK / 16; ++k) {
          if (k == 2) ready = tc::mbar_test(&full_bar[ahead.s], ahead.parity);  // see Ring
          const uint64_t ad = ad0 + at + k * k_step<true>, bd = bd0 + at + k * k_step<true>;
          const uint32_t more = (kb > t.kb0 || k > 0) ? 1u : 0u;
          tc::mma_bf16_pair(tmem_base, ad, bd, idesc, more);
          tc::mma_bf16_pair(tmem_base + kSubCols, ad, bd + (b_bytes >> 4), idesc, more);
        }
        tc::mma_commit_pair(&read_bar[s], 3);  // the stage has been read in both CTAs
      }
      if (ok) tc::mma_commit_pair(&acc_full, 3);
    }
    if (!ok) atomicCAS(g.status, 0, err::kTimeout);
  } else if (warp >= 2 && warp < 2 + kEpiWarps) {
    // ---------------- epilogue (both CTAs, each on its own 128 rows)
    const int quarter = warp & 3;
    const uint32_t lead_acc_empty = tc::map_to_cta(tc::smem_u32(&acc_empty), 0);
    int j = 0, turn = 0;
    for (int i = pair; i < g.items; i += pairs, ++j) {
      const Item t = item_at(g, i, total_kb);
      const int row0 = t.m0 + static_cast<int>(rank) * kBM + quarter * 32;
      int c_begin, c_end;
      epi_cols(min(kSubs * kSubCols, (g.N - t.n0 + 63) / 64 * 64), warp - 2, &c_begin, &c_end);
      const bool ok = __all_sync(0xffffffffu, tc::mbar_wait(&acc_full, static_cast<uint32_t>(j) & 1, kWaitLimit));
      tc::fence_after_sync();
      if (in_ring && sums)  // the MMAs have read every stage, and so must the summing warps have
        asm volatile("bar.sync 3, %0;" ::"n"(32 * (kEpiWarps + kSumWarps)) : "memory");
      if (!ok) {
        if (lane == 0) atomicCAS(g.status, 0, err::kTimeout);
        break;
      }
      epilogue_reduce(g, &tmD, staging + (warp - 2) * 8192,
                      tmem_base + (static_cast<uint32_t>(quarter * 32) << 16), row0, t.n0, c_begin, c_end,
                      turn);
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive_cluster(lead_acc_empty);
    }
    if (lane == 0) tc::bulk_wait_all();
  } else if (warp >= 2 + kEpiWarps && warp < 2 + kEpiWarps + kSumWarps && sums) {
    // ---------------- column sums of dY
    const int th = threadIdx.x - kThreads;
    bool fine = true;
    Ring ring;
    for (int i = pair; i < g.items; i += pairs) {
      const Item t = item_at(g, i, total_kb);
      float acc0[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, acc1[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int kb = t.kb0; kb < t.kb1; ++kb, ring.next(g.stages)) {
        const int s = ring.s;
        if (fine) fine = __all_sync(0xffffffffu, tc::mbar_wait(&landed_bar[s], ring.parity, kWaitLimit));
        if (!fine) break;
        if (t.first_col) {
          tc::fence_async_shared();  // what the copies of this CTA wrote, read by plain loads
          add_stage_columns(smem + static_cast<size_t>(s) * stage_bytes, th, acc0);
          add_stage_columns(smem + static_cast<size_t>(s) * stage_bytes, th + 128, acc1);
        }
        // as in gemm_kernel: the arrival depends on values that all of the lanes' reads went into
        const unsigned read =
            __ballot_sync(0xffffffffu, __float_as_uint(acc0[0]) != 0x7FFFDEADu && __float_as_uint(acc1[0]) != 0x7FFFDEADu);
        if (lane == (read ? __ffs(read) - 1 : 0)) tc::mbar_arrive(&empty_bar[s]);
      }
      if (in_ring) asm volatile("bar.arrive 3, %0;" ::"n"(32 * (kEpiWarps + kSumWarps)) : "memory");
      if (!fine && lane == 0) atomicCAS(g.status, 0, err::kTimeout);
      if (!t.first_col) continue;  // a warp that has given up still meets the others at the barriers below
#pragma unroll
      for (int q = 0; q < 8; ++q) {  // lanes 8 apart hold other rows of the same columns
        acc0[q] += __shfl_xor_sync(0xffffffffu, acc0[q], 8);
        acc0[q] += __shfl_xor_sync(0xffffffffu, acc0[q], 16);
        acc1[q] += __shfl_xor_sync(0xffffffffu, acc1[q], 8);
        acc1[q] += __shfl_xor_sync(0xffffffffu, acc1[q], 16);
      }
      if (lane < 8) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          atomicAdd(&s_sum[lane * 8 + q], acc0[q]);
          atomicAdd(&s_sum[64 + lane * 8 + q], acc1[q]);
        }
      }
      asm volatile("bar.sync 2, %0;" ::"n"(32 * kSumWarps) : "memory");
      const int row = t.m0 + static_cast<int>(rank) * kBM + th;
      if (fine && row < g.M) atomicAdd(g.col_sums + row, s_sum[th]);
      s_sum[th] = 0.f;
      asm volatile("bar.sync 2, %0;" ::"n"(32 * kSumWarps) : "memory");
    }
  }

  tc::fence_before_sync();
  __syncthreads();
  tc::cluster_sync_all();  // neither CTA leaves while the other may still touch its memory or barriers
  if (warp == 1) tc::tmem_dealloc_pair(tmem_base, 512);
}

// ------------------------------------------------------------------ column sums
__global__ void __launch_bounds__(256)
colsum_bf16_kernel(const __nv_bfloat16* __restrict__ x, int ld, int M, int N, int rows_per_block, float* out) {
  pdl_enter();
  // block = 256 threads: 32 column pairs x 8 row lanes over a 64-column strip
  const int cpair = threadIdx.x & 31;
  const int rlane = threadIdx.x >> 5;
  const int col = blockIdx.x * 64 + cpair * 2;
  const int r0 = blockIdx.y * rows_per_block;
  const int r1 = min(M, r0 + rows_per_block);
  float s0 = 0.f, s1 = 0.f;
  if (col < N) {
    for (int r = r0 + rlane; r < r1; r += 8) {
      const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(x + static_cast<size_t>(r) * ld + col);
      s0 += __bfloat162float(v.x);
      s1 += __bfloat162float(v.y);
    }
  }
  __shared__ float sh[8][64];
  sh[rlane][cpair * 2] = s0;
  sh[rlane][cpair * 2 + 1] = s1;
  __syncthreads();
  if (threadIdx.x < 64) {
    float t = 0.f;
    for (int k = 0; k < 8; ++k) t += sh[k][threadIdx.x];
    const int c = blockIdx.x * 64 + threadIdx.x;
    if (c < N) atomicAdd(out + c, t);
  }
}

// ------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// 2-D bf16 row-major tensor [rows, cols] with pitch ld (elements); box = box_cols x box_rows,
// 128-byte swizzle, out-of-range elements read as zero.
bool make_tmap(CUtensorMap* m, const __nv_bfloat16* base, int rows, int cols, int ld, int box_cols, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || (ld % 8) != 0 || box_cols != 64 || box_rows > 256) return false;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(box_cols), static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// 2-D fp32 row-major tensor [rows, cols] with pitch ld (elements), for 32 x 32 boxes in the 128-byte swizzle.
bool make_tmap_f32(CUtensorMap* m, float* base, int rows, int cols, int ld) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || (ld % 4) != 0) return false;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 4};
  cuuint32_t box[2] = {32, 32};
  cuuint32_t estr[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// 2-D bf16 row-major output [rows, cols] with pitch ld (elements), for 32 x 32 boxes in the 64-byte swizzle.
bool make_tmap_out(CUtensorMap* m, __nv_bfloat16* base, int rows, int cols, int ld) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || (ld % 8) != 0) return false;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
  cuuint32_t box[2] = {32, 32};
  cuuint32_t estr[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int pick_bn(int n, int granule) {
  // fewest tiles first, then the narrowest tile that still covers n with that many tiles
  const int tiles = (n + 255) / 256;
  int bn = (n + tiles - 1) / tiles;
  bn = (bn + granule - 1) / granule * granule;
  return bn < granule ? granule : bn;
}

// Tile width of gemm_kernel for an m x n output.  Where wide tiles leave
// SMs idle, the narrowest width that is still one wave: a k-block takes its 99 cycles an MMA and the trip to L2 whatever the
// width, but the epilogue gets shorter (forward, us at the fewest tiles / so: 512 x 256 x 224 6.0 / 4.0, 1789 x 400 x 432
// 6.8 / 5.4, 1024 x 1024 x 1024 10.2 / 8.8, 100 x 4096 x 4096 27.6 / 23.5, 8192 x 400 x 400 the same width).
int tile_bn(int m, int n) {
  const int rows = (m + kBM - 1) / kBM;
  const int widest = pick_bn(n, 16);
  for (int bn = 32; bn < widest; bn += 32)
    if (rows * ((n + bn - 1) / bn) <= 148) return bn;
  return widest;
}

// With at most one CTA per SM there is no second CTA to hide a short pipeline behind: as many stages as fit (and as there are
// k-blocks) when the whole grid fits in one wave, else 2 stages and two CTAs per SM.
int one_wave_stages(int m, int n, int k, int bn) {
  const int tiles = ((m + kBM - 1) / kBM) * ((n + bn - 1) / bn);
  if (tiles > 148) return 2;
  const int fit = 199 * 1024 / ((kBM + bn) * 128), total_kb = (k + kBK - 1) / kBK;
  const int stages = fit < kMaxStages ? fit : kMaxStages;
  return stages < total_kb ? stages : total_kb < 2 ? 2 : total_kb;
}

template <bool A_MN, bool B_MN, int EPI>
int launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, GemmArgs g, int splits, cudaStream_t stream) {
  const size_t smem = static_cast<size_t>(g.stages) * (kBM + g.BN) * 128 + 1024;
  static bool attr_set = false;
  if (!attr_set) {
    cudaFuncSetAttribute(gemm_kernel<A_MN, B_MN, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    attr_set = true;
  }
  dim3 grid((g.M + kBM - 1) / kBM, (g.N + g.BN - 1) / g.BN, splits);
  launch_pdl_if(g.late == 0, gemm_kernel<A_MN, B_MN, EPI>, grid, dim3(kTileThreads<B_MN>), smem, stream, ta, tb, td, g);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int g_variant = 0;           // 0 = choose; 1 = CTA pair; 2 = single-CTA resident; 3 = one tile per CTA
int g_resident_n_tiles = 0;  // 0 = choose; otherwise the number of column tiles of the resident variant

// Plan of the resident-weight variant for an M x N output contracting over K: tile width and depth
// of the activation ring.  The ring's depth decides how many bytes a CTA keeps in flight from L2,
// and that, not the tensor cores, bounds these tall-and-skinny products; so the plan takes the
// fewest column tiles whose weight slice leaves room for at least four 16 KB activation stages
// (more column tiles re-read the activations from L2 once more each, which costs less than a
// starved ring).  Returns false when the variant does not apply.
bool plan_resident(int M, int N, int K, int* bn_out, int* stages_out) {
  const int total_kb = (K + kBK - 1) / kBK;
  const int m_tiles = (M + kBM - 1) / kBM;
  const size_t budget = 225 * 1024 - 1024;
  int best_bn = 0, best_stages = 0;
  for (int n_tiles = (N + 255) / 256; n_tiles <= 8; ++n_tiles) {
    if (g_resident_n_tiles > 0 && n_tiles != g_resident_n_tiles) continue;
    int bn = (N + n_tiles - 1) / n_tiles;
    bn = (bn + 15) / 16 * 16;
    if (bn < 16) bn = 16;
    const size_t weights = static_cast<size_t>(total_kb) * bn * 128;
    if (weights + 2 * kBM * 128 > budget) continue;
    int stages = static_cast<int>((budget - weights) / (kBM * 128));
    if (stages > kMaxStages) stages = kMaxStages;
    if (stages > best_stages) best_bn = bn, best_stages = stages;
    if (stages >= 4) break;
  }
  if (best_bn == 0) return false;
  const int n_tiles = (N + best_bn - 1) / best_bn;
  if (n_tiles > 148 || m_tiles * n_tiles < 2 * 148) return false;
  *bn_out = best_bn;
  *stages_out = best_stages;
  return true;
}

// Plan of the CTA-pair variant: the widest column tile (fewest activation re-reads) whose half
// slice of the weights leaves at least four ring stages.
bool plan_pair(int M, int N, int K, bool out_tma, int* bn_out, int* stages_out) {
  const int total_kb = (K + kBK - 1) / kBK;
  const int m_tiles = (M + 2 * kBM - 1) / (2 * kBM);
  const size_t budget = 225 * 1024 - 1024 - (out_tma ? kEpiWarps * 4096 : 0);
  for (int n_tiles = (N + 255) / 256; n_tiles <= 4; ++n_tiles) {
    if (g_resident_n_tiles > 0 && n_tiles != g_resident_n_tiles) continue;
    int bn = (N + n_tiles - 1) / n_tiles;
    const int unit = out_tma ? 32 : 16;  // the MMA's N is a multiple of 16; each half is then whole 8-row swizzle groups
    bn = (bn + unit - 1) / unit * unit;
    const size_t weights = static_cast<size_t>(total_kb) * (bn / 2) * 128;
    if (weights + 4 * kBM * 128 > budget) continue;
    int stages = static_cast<int>((budget - weights) / (kBM * 128));
    if (stages > kMaxStages) stages = kMaxStages;
    if (m_tiles * n_tiles < 2 * 74) return false;  // too few tiles to amortise loading the weights
    *bn_out = bn;
    *stages_out = stages;
    return true;
  }
  return false;
}

template <int EPI>
int launch_pair(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, GemmArgs g, cudaStream_t stream) {
  const int total_kb = (g.K + kBK - 1) / kBK;
  const int n_tiles = (g.N + g.BN - 1) / g.BN;
  const int m_tiles = (g.M + 2 * kBM - 1) / (2 * kBM);
  const size_t smem = static_cast<size_t>(total_kb) * (g.BN / 2) * 128 + static_cast<size_t>(g.stages) * kBM * 128 +
                      (g.out_tma ? kEpiWarps * 4096 : 0) + 1024;
  static size_t attr_smem = 0;
  if (smem > attr_smem) {
    if (cudaFuncSetAttribute(gemm_pair_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(smem)) != cudaSuccess) {
      cudaGetLastError();
      return -2;
    }
    attr_smem = smem;
  }
  int pairs = 74 / n_tiles;
  if (pairs > m_tiles) pairs = m_tiles;
  launch_pdl_if(g.late == 0, gemm_pair_kernel<EPI>, dim3(2 * pairs, n_tiles), dim3(kThreads), smem, stream, ta, tb, td, g);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

template <int EPI>
int launch_resident(const CUtensorMap& ta, const CUtensorMap& tb, GemmArgs g, cudaStream_t stream) {
  const int total_kb = (g.K + kBK - 1) / kBK;
  const int n_tiles = (g.N + g.BN - 1) / g.BN;
  const int m_tiles = (g.M + kBM - 1) / kBM;
  const size_t smem = static_cast<size_t>(total_kb) * g.BN * 128 + static_cast<size_t>(g.stages) * kBM * 128 + 1024;
  static size_t attr_smem = 0;  // static + dynamic shared memory share the 227 KB limit: ask for what is needed
  if (smem > attr_smem) {
    if (cudaFuncSetAttribute(gemm_bres_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(smem)) != cudaSuccess) {
      cudaGetLastError();
      return -2;
    }
    attr_smem = smem;
  }
  int per_n = 148 / n_tiles;
  if (per_n > m_tiles) per_n = m_tiles;
  launch_pdl_if(g.late == 0, gemm_bres_kernel<EPI>, dim3(per_n, n_tiles), dim3(kThreads), smem, stream, ta, tb, g);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// Plan of the CTA-pair weight gradient of an M x N matrix (N inputs): tiles of 256 x 512 and as many ranges of the batch
// as give every pair one.  True where it is the faster one: rows and columns enough for the
// traffic that a pair saves, and tiles for every pair or ranges that are worth its longer start and its reductions.  Measured,
// us as tiles per CTA / on pairs: batch 65536 of 400 x 432 38.0 / 30.9, 32768 (14 k-blocks) 22.8 / 20.9, 16384 (7) 15.1 / 15.7,
// 65536 of 256 x 512 23.4 / 26.8; 4096 x 4096 at batch 1024 51.8 / 41.6, at 100 25.0 / 20.5; 1024 x 6416 at 1000 26.8 / 23.3;
// 2048 x 2048 at 1024 (8) 15.0 / 16.4.
bool plan_pair_wgrad(int M, int N, int K, GemmArgs* g, int* splits) {
  const int total_kb = (K + kBK - 1) / kBK;
  constexpr int kCols = kSubs * kSubCols;
  const int tiles = ((M + 2 * kBM - 1) / (2 * kBM)) * ((N + kCols - 1) / kCols);
  int n = tiles < 74 ? 74 / tiles : 1;
  if (n > total_kb) n = total_kb;
  g->kb_per_split = (total_kb + n - 1) / n;
  *splits = (total_kb + g->kb_per_split - 1) / g->kb_per_split;
  return M > 2 * kBM && N > 256 && (tiles >= 74 || g->kb_per_split >= 14);
}

int launch_pair_wgrad(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, GemmArgs g, int splits,
                      cudaStream_t stream) {
  constexpr size_t stage = kBM * 128 + kSubs * (kSubCols / 2) * 128;
  g.tiles_m = (g.M + 2 * kBM - 1) / (2 * kBM);
  g.tiles_n = (g.N + kSubs * kSubCols - 1) / (kSubs * kSubCols);
  g.items = g.tiles_m * g.tiles_n * splits;
  const size_t limit = 225 * 1024;
  const size_t staging = g.items <= 74 ? 0 : kEpiWarps * 8192;  // one item a pair: the epilogue uses the ring (64 KB or more)
  g.stages = static_cast<int>((limit - 1024 - staging) / stage);  // 4, or 3
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(gemm_pair_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(limit)) != cudaSuccess) {
      cudaGetLastError();
      return -2;
    }
    attr_set = true;
  }
  const int pairs = g.items < 74 ? g.items : 74;
  launch_pdl(gemm_pair_wgrad_kernel, dim3(2 * pairs), dim3(kPairWgradThreads), g.stages * stage + staging + 1024, stream, ta,
             tb, td, g);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace

// 256-bit stores need 32-byte aligned rows; tile columns are multiples of 16 elements already.
static int can_store_v8(const void* out, int ld) {
  return (reinterpret_cast<uintptr_t>(out) % 32 == 0 && ld % 16 == 0) ? 1 : 0;
}

int linear_forward(const __nv_bfloat16* X, int ldx, const __nv_bfloat16* W, int ldw, const float* bias,
                   __nv_bfloat16* Y, int ldy, int M, int N, int K, bool relu, uint16_t* mask_out, int ldm, int* status,
                   bool late, cudaStream_t stream) {
  GemmArgs g{};
  g.late = late ? 1 : 0;
  g.M = M, g.N = N, g.K = K;
  g.BN = pick_bn(N, 16);
  g.stages = 2;
  g.kb_per_split = (K + kBK - 1) / kBK;
  g.relu = relu ? 1 : 0;
  g.bias = bias;
  g.out = Y, g.ldo = ldy;
  g.mask_out = mask_out, g.ldm = ldm, g.mask_chunks = (N + 15) / 16;
  g.out_v8 = can_store_v8(Y, ldy);
  if (mask_out != nullptr && ldm < M) return -1;
  g.status = status;
  CUtensorMap ta, tb, td;
  g.out_tma = g_variant < 2 && (reinterpret_cast<uintptr_t>(Y) & 15) == 0 && (ldy % 8) == 0 ? 1 : 0;
  const bool pair = (g_variant == 0 || g_variant == 1) && plan_pair(M, N, K, g.out_tma != 0, &g.BN, &g.stages);
  const bool resident = !pair && (g_variant == 0 || g_variant == 2) && plan_resident(M, N, K, &g.BN, &g.stages);
  if (!pair && !resident) g.BN = tile_bn(M, N);
  if (!pair) g.out_tma = 0;
  if ((ldy % 8) != 0 || !make_tmap(&ta, X, M, K, ldx, 64, kBM) ||
      !make_tmap(&tb, W, N, K, ldw, 64, pair ? g.BN / 2 : g.BN))
    return -1;
  if (g.out_tma ? !make_tmap_out(&td, Y, M, N, ldy) : (td = ta, false)) return -1;  // or a map that nothing reads
  if (pair) return launch_pair<EPI_BIAS_ACT>(ta, tb, td, g, stream);
  if (resident) return launch_resident<EPI_BIAS_ACT>(ta, tb, g, stream);
  g.stages = one_wave_stages(M, N, K, g.BN);
  return launch<false, false, EPI_BIAS_ACT>(ta, tb, ta, g, 1, stream);  // no third map is read
}

int linear_dgrad(const __nv_bfloat16* dY, int lddy, const __nv_bfloat16* Wt, int ldwt, const __nv_bfloat16* H,
                 int ldh, const uint16_t* mask, int ldm, __nv_bfloat16* dX, int lddx, int M, int N, int K, int zero_cols,
                 int* status, cudaStream_t stream) {
  // out dX is [M, K]; the contraction runs over the layer's N outputs
  GemmArgs g{};
  g.M = M, g.N = K, g.K = N;
  g.BN = pick_bn(K, 16);
  g.stages = 2;
  g.kb_per_split = (N + kBK - 1) / kBK;
  g.H = H, g.ldh = ldh;
  g.mask = mask, g.ldm = ldm, g.mask_chunks = (K + 15) / 16;
  g.out_v8 = can_store_v8(dX, lddx);
  if (mask != nullptr && ldm < M) return -1;
  g.out = dX, g.ldo = lddx;
  g.zero_cols = zero_cols;
  if (zero_cols % 8 != 0 || (zero_cols > 0 && (K % 8 != 0 || K + zero_cols > lddx || (reinterpret_cast<uintptr_t>(dX) & 15) != 0)))
    return -1;
  g.status = status;
  CUtensorMap ta, tb, td;
  // (with the activations instead of their bits the epilogue reads 16 columns of a row at a time and stores as it goes)
  g.out_tma = g_variant < 2 && (H == nullptr || mask != nullptr) && (reinterpret_cast<uintptr_t>(dX) & 15) == 0 && (lddx % 8) == 0 ? 1 : 0;
  const bool pair = (g_variant == 0 || g_variant == 1) && plan_pair(M, K, N, g.out_tma != 0, &g.BN, &g.stages);
  const bool resident = !pair && (g_variant == 0 || g_variant == 2) && plan_resident(M, K, N, &g.BN, &g.stages);
  if (!pair && !resident) g.BN = tile_bn(M, K);
  if (!pair) g.out_tma = 0;
  if ((lddx % 8) != 0 || (H && (ldh % 8) != 0) || !make_tmap(&ta, dY, M, N, lddy, 64, kBM) ||
      !make_tmap(&tb, Wt, K, N, ldwt, 64, pair ? g.BN / 2 : g.BN))
    return -1;
  if (g.out_tma ? !make_tmap_out(&td, dX, M, K, lddx) : (td = ta, false)) return -1;  // or a map that nothing reads
  if (pair) return launch_pair<EPI_RELU_MASK>(ta, tb, td, g, stream);
  if (resident) return launch_resident<EPI_RELU_MASK>(ta, tb, g, stream);
  g.stages = one_wave_stages(M, K, N, g.BN);
  return launch<false, false, EPI_RELU_MASK>(ta, tb, ta, g, 1, stream);
}

int linear_wgrad(const __nv_bfloat16* dY, int lddy, const __nv_bfloat16* X, int ldx, float* dW, int lddw, float* db, int M,
                 int N, int K, int* status, cudaStream_t stream) {
  // out dW is [N, K]; the contraction runs over the M batch rows, split across blockIdx.z
  GemmArgs g{};
  g.M = N, g.N = K, g.K = M;
  g.BN = pick_bn(K, 64);
  g.stages = 4;
  const int total_kb = (M + kBK - 1) / kBK;
  const int tiles = ((N + kBM - 1) / kBM) * ((K + g.BN - 1) / g.BN);
  int splits = 148 / (tiles > 0 ? tiles : 1);
  if (splits < 1) splits = 1;
  if (splits > total_kb) splits = total_kb;
  g.kb_per_split = (total_kb + splits - 1) / splits;
  splits = (total_kb + g.kb_per_split - 1) / g.kb_per_split;  // no empty split
  g.col_sums = db;
  g.status = status;
  CUtensorMap ta, tb, td;
  if ((lddw % 4) != 0 || (reinterpret_cast<uintptr_t>(dW) & 15) != 0 || !make_tmap(&ta, dY, M, N, lddy, 64, 64) ||
      !make_tmap(&tb, X, M, K, ldx, 64, 64) || !make_tmap_f32(&td, dW, N, K, lddw))
    return -1;
  GemmArgs paired = g;
  int paired_splits = 1;
  if ((plan_pair_wgrad(N, K, M, &paired, &paired_splits) && g_variant != 3) || g_variant == 4)
    return launch_pair_wgrad(ta, tb, td, paired, paired_splits, stream);
  return launch<true, true, EPI_RED_F32>(ta, tb, td, g, splits, stream);
}

void gemm_set_tuning(int variant, int n_tiles) {
  g_variant = variant;
  g_resident_n_tiles = n_tiles;
}

void colsum_bf16(const __nv_bfloat16* dY, int lddy, int M, int N, float* db, cudaStream_t stream) {
  const int strips = (N + 63) / 64;
  int row_blocks = (148 * 4 + strips - 1) / strips;
  int rows_per_block = (M + row_blocks - 1) / row_blocks;
  if (rows_per_block < 64) rows_per_block = 64;
  row_blocks = (M + rows_per_block - 1) / rows_per_block;
  launch_pdl(colsum_bf16_kernel, dim3(strips, row_blocks), dim3(256), 0, stream, dY, lddy, M, N, rows_per_block, db);
}

}  // namespace cu
}  // namespace kb
