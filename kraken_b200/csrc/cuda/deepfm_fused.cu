// DeepFM front end fused around the sparse exchange.
//
// Two table layouts are accepted: a dim-D embedding table plus a separate dim-1 first-order
// table, or ONE table whose rows are RD >= D + 1 floats wide with the first-order weight in
// column D (rows1 / ugrad1 null): the second costs one exchange per step instead of two.
//
// Forward: reads the UNIQUE rows that the pull left in the receive buffers (second-order
// table [U2, D] and first-order table [U1, 1]) through the occurrence -> unique maps and, in
// one pass per sample, writes the bf16 MLP input [emb | dense | 0-pad] and the fp32 FM logit
//   sum_f w_f + 0.5 * sum_d ((sum_f e_fd)^2 - sum_f e_fd^2).
// Backward: from d(MLP input) and d(logit) forms each occurrence's embedding gradient
//   dlogit * (S_d - e_fd) + dX[f, d]   and   dlogit (first order)
// and red-adds it straight into the per-unique gradient buffers that push_dispatch sends, so
// the expanded [B, F, D] tensors of the unfused path never exist.
// Reference model math: examples/DeepFM/model/DeepFM.py:87-125 (torch CPU ops).
#include <cuda_bf16.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace kb {
namespace cu {

namespace {

constexpr int kThreads = 256;
constexpr int kForwardBlocks = 4;   // a multiprocessor: 64 registers a thread
// Row loads of a lane in flight in the forward pass.  With FM the 64 registers hold them for rows of 4, 8, 16 and 128 floats;
// for 32 and 64 they spill 40 and 56 bytes.  Six there spill nothing and are better for 39 fields of 32 floats (32768 samples:
// 39.4 us for 44.1), worse for 26 (29.9 for 28.9), the same within 5 % for 64 floats.
constexpr int kBatch = 7;
constexpr int kBackwardBlocks = 5;

// Row index of unique entry `u`: the entry itself when the rows were gathered into a receive
// buffer, or the table slot the owner resolved for it when the kernel reads the table in place
// (single-GPU jobs: no copy of the rows is made).  A failed lookup (slot < 0) reads row 0; the
// status word already carries the error.
__device__ __forceinline__ size_t row_of(const int* __restrict__ slots, int u) {
  if (slots == nullptr) return static_cast<size_t>(u);
  const int s = __ldg(slots + u);
  return static_cast<size_t>(s < 0 ? 0 : s);
}

// Field groups per sample: as many as keep (D / 4) x G lanes within half a warp; rows of 128 floats take a whole one.
constexpr int field_groups(int chunks) {
  int g = 1;
  while (chunks * g * 2 <= 16) g <<= 1;
  return g;
}

// P2 and P1 are the pitches of rows2 and rows1 in floats: the row width for gathered rows, the tables' pitch in place.
// Lanes per sample = (D / 4) x G: lane (g, c) owns dims [4c, 4c + 4) of the fields g, g + G, ...
// Splitting the fields over G lane groups (a power of two) multiplies the number of independent
// row loads in flight; the per-sample sums are combined with shuffles and the forward pass leaves
// S[b, :] = sum_f e_f for the backward pass, whose lanes then need nothing from each other.
// The forward pass is bound by the latency of its loads, entry -> slot -> row, not by bandwidth.  So a lane fetches the entries
// of two of 2 x lpr fields, reads their first-order weights, and the lane groups get theirs by shuffles: kBatch rows of each
// lane are in flight together.  65536 samples of 26 fields of dim 16, rows in L2: 36.8 us (5.2 TB/s of rows and x); 50.2 us
// with the entries loaded where they are used, four fields unrolled and the rest one after the other.  Four rows in flight
// take 39.1 us, eight 42.5 (they spill), seven with 5 blocks and spills 64; with the sizes as arguments of the kernel 43.8.
// FM false (Wide&Deep): the logit is sum_f w_f alone, and the backward pass needs neither the rows nor ssum.
template <bool FM, int chunks>
__global__ void __launch_bounds__(kThreads, kForwardBlocks)
deepfm_pack_forward_kernel(const float* __restrict__ rows2, const int* __restrict__ inv2,
                           const int* __restrict__ slots2, const float* __restrict__ rows1,
                           const int* __restrict__ inv1, const int* __restrict__ slots1,
                           const float* __restrict__ dense, int B, int F, int P2, int P1, int ND,
                           __nv_bfloat16* __restrict__ x, int ldx, float* __restrict__ fm_logit,
                           float* __restrict__ ssum) {
  pdl_enter();
  constexpr int D = 4 * chunks, G = field_groups(chunks), lpr = chunks * G;
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = gtid % lpr;
  const int stride = (gridDim.x * blockDim.x) / lpr;
  const unsigned group_mask = (lpr == 32 ? 0xffffffffu : ((1u << lpr) - 1u)) << ((threadIdx.x & 31) / lpr * lpr);
  const int c = lane % chunks;   // chunks * G == lpr
  const int fg = lane / chunks;
  const int rounds = (B + stride - 1) / stride;
  for (int it = 0; it < rounds; ++it) {
    const int b = gtid / lpr + it * stride;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f), q = s;
    float part = 0.f;
    const int fields = b < B ? F : 0;
    __nv_bfloat16* xr = x + static_cast<size_t>(b) * ldx;
    for (int base = 0; base < F; base += 2 * lpr) {
      const int f0 = base + lane, f1 = f0 + lpr;
      const int* i2 = inv2 + static_cast<size_t>(b) * F;
      int r0 = 0, r1 = 0;
      if (f0 < fields) r0 = i2[f0];
      if (f1 < fields) r1 = i2[f1];
      float w0 = 0.f, w1 = 0.f;
      if (rows1 != nullptr) {
        const int* i1 = inv1 + static_cast<size_t>(b) * F;
        int u0 = 0, u1 = 0;
        if (f0 < fields) u0 = i1[f0];
        if (f1 < fields) u1 = i1[f1];
        if (f0 < fields) w0 = __ldcg(rows1 + row_of(slots1, u0) * P1);
        if (f1 < fields) w1 = __ldcg(rows1 + row_of(slots1, u1) * P1);
      }
      if (slots2 != nullptr) {
        if (f0 < fields) r0 = static_cast<int>(row_of(slots2, r0));
        if (f1 < fields) r1 = static_cast<int>(row_of(slots2, r1));
      }
      if (rows1 == nullptr) {
        // folded layout: column D of the same row is the field's first-order weight
        if (f0 < fields) w0 = __ldcg(rows2 + static_cast<size_t>(r0) * P2 + D);
        if (f1 < fields) w1 = __ldcg(rows2 + static_cast<size_t>(r1) * P2 + D);
      }
      for (int j = 0; j < 2 * chunks && base + j * G < F; j += kBatch) {
        float4 e[kBatch];
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
          const int k = (j + i) * G + fg;  // field of the 2 x lpr
          const int row = __shfl_sync(group_mask, j + i < chunks ? r0 : r1, k & (lpr - 1), lpr);
          e[i] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (j + i < 2 * chunks && base + k < fields)
            e[i] = __ldcg(reinterpret_cast<const float4*>(rows2 + static_cast<size_t>(row) * P2) + c);
        }
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
          const int k = (j + i) * G + fg;
          if (FM) {
            s.x += e[i].x, s.y += e[i].y, s.z += e[i].z, s.w += e[i].w;
            q.x += e[i].x * e[i].x, q.y += e[i].y * e[i].y, q.z += e[i].z * e[i].z, q.w += e[i].w * e[i].w;
          }
          __nv_bfloat162 lo = __floats2bfloat162_rn(e[i].x, e[i].y), hi = __floats2bfloat162_rn(e[i].z, e[i].w);
          uint2 packed;
          packed.x = *reinterpret_cast<uint32_t*>(&lo);
          packed.y = *reinterpret_cast<uint32_t*>(&hi);
          if (j + i < 2 * chunks && base + k < fields) *reinterpret_cast<uint2*>(xr + (base + k) * D + c * 4) = packed;
        }
      }
      part += w0 + w1;
    }
    if (b < B) {
      // dense features and the zero pad, spread over the sample's lanes
      const int base = F * D;
      for (int j = lane; base + j < ldx; j += lpr)
        xr[base + j] = __float2bfloat16(j < ND ? dense[static_cast<size_t>(b) * ND + j] : 0.f);
    }
    // sums over the field groups of the same chunk (lanes c, c + chunks, c + 2 chunks, ...)
    for (int o = chunks; FM && o < lpr; o <<= 1) {
      s.x += __shfl_xor_sync(group_mask, s.x, o), s.y += __shfl_xor_sync(group_mask, s.y, o);
      s.z += __shfl_xor_sync(group_mask, s.z, o), s.w += __shfl_xor_sync(group_mask, s.w, o);
      q.x += __shfl_xor_sync(group_mask, q.x, o), q.y += __shfl_xor_sync(group_mask, q.y, o);
      q.z += __shfl_xor_sync(group_mask, q.z, o), q.w += __shfl_xor_sync(group_mask, q.w, o);
    }
    if (FM && b < B && fg == 0) {
      part += 0.5f * (s.x * s.x - q.x + s.y * s.y - q.y + s.z * s.z - q.z + s.w * s.w - q.w);
      if (ssum != nullptr) *reinterpret_cast<float4*>(ssum + static_cast<size_t>(b) * D + c * 4) = s;
    }
    for (int o = lpr >> 1; o > 0; o >>= 1) part += __shfl_xor_sync(group_mask, part, o);
    if (b < B && lane == 0) fm_logit[b] = part;
  }
}

// Bound by the reductions: those on one row are serialised in L2 (about 2.6 ns each), and the top id of a skewed field has
// thousands.  65536 samples of 26 fields of dim 16: 52.1 us for uniform ids, 90.0 for Zipf(1.1) ids, whose top ids come 5550
// times; 52.1 and 92.9 us with the sizes as arguments.  Over 500 .. 32768 samples of 10 .. 39 fields of 4 .. 64 floats it
// takes 0.93 of the time of that form; with 4, 6 or 7 blocks a multiprocessor 0.96 to 0.97.  With the forward pass's batches
// uniform ids took 70 us: the blocks in flight matter more.  Sums of the block's repeated ids first (counts and lists in
// shared memory) took 83 us for Zipf ids, but 70 for uniform ones.
template <bool FM, int chunks>
__global__ void __launch_bounds__(kThreads, kBackwardBlocks)
deepfm_pack_backward_kernel(const float* __restrict__ rows2, const int* __restrict__ inv2,
                            const int* __restrict__ slots2, const int* __restrict__ inv1,
                            const __nv_bfloat16* __restrict__ dx, int lddx, const float* __restrict__ dlogit,
                            const float* __restrict__ ssum, int B, int F, int P2, int RD,
                            float* ugrad2, float* ugrad1) {
  pdl_enter();
  constexpr int D = 4 * chunks, G = field_groups(chunks), lpr = chunks * G;
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = gtid % lpr;
  const int stride = (gridDim.x * blockDim.x) / lpr;
  const int c = lane % chunks;
  const int fg = lane / chunks;
  for (int b = gtid / lpr; b < B; b += stride) {
    const int* i2 = inv2 + static_cast<size_t>(b) * F;
    const float g = dlogit[b];
    const __nv_bfloat16* dxr = dx ? dx + static_cast<size_t>(b) * lddx : nullptr;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (FM) s = *reinterpret_cast<const float4*>(ssum + static_cast<size_t>(b) * D + c * 4);
#pragma unroll 4
    for (int f = fg; f < F; f += G) {
      const int u = i2[f];
      float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
      if (FM) {
        const float4 e = __ldcg(reinterpret_cast<const float4*>(rows2 + row_of(slots2, u) * P2) + c);
        d = make_float4(g * (s.x - e.x), g * (s.y - e.y), g * (s.z - e.z), g * (s.w - e.w));
      }
      if (dxr) {
        const uint2 p = *reinterpret_cast<const uint2*>(dxr + f * D + c * 4);
        const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&p.x);
        const __nv_bfloat162 hi = *reinterpret_cast<const __nv_bfloat162*>(&p.y);
        d.x += __bfloat162float(lo.x), d.y += __bfloat162float(lo.y);
        d.z += __bfloat162float(hi.x), d.w += __bfloat162float(hi.y);
      }
      red_add_v4(ugrad2 + static_cast<size_t>(u) * RD + c * 4, d);
    }
    if (ugrad1 != nullptr) {
      const int* i1 = inv1 + static_cast<size_t>(b) * F;
      for (int f = lane; f < F; f += lpr) atomicAdd(ugrad1 + i1[f], g);
    } else {
      for (int f = lane; f < F; f += lpr) atomicAdd(ugrad2 + static_cast<size_t>(i2[f]) * RD + D, g);
    }
  }
}

Sym to_sym(const SymHost& h) {
  Sym s;
  for (int i = 0; i < kMaxWorld; ++i) s.base[i] = static_cast<char*>(h.base[i]);
  s.rank = h.rank;
  s.world = h.world;
  return s;
}

int grid_for(long long rows, int lpr) {
  long long g = (rows * lpr + kThreads - 1) / kThreads;
  if (g < 1) g = 1;
  if (g > 148 * 16) g = 148 * 16;
  return static_cast<int>(g);
}

// Calls f with the chunk count as a compile-time constant; D is 4 .. 128, D / 4 a power of two (the bindings check it).
template <typename Fn>
void by_chunks(int D, Fn f) {
  switch (D / 4) {
    case 1: return f(std::integral_constant<int, 1>());
    case 2: return f(std::integral_constant<int, 2>());
    case 4: return f(std::integral_constant<int, 4>());
    case 8: return f(std::integral_constant<int, 8>());
    case 16: return f(std::integral_constant<int, 16>());
    case 32: return f(std::integral_constant<int, 32>());
  }
}

}  // namespace

void deepfm_pack_forward(const float* rows2, const int* inv2, const int* slots2, const float* rows1, const int* inv1,
                         const int* slots1, const float* dense, int B, int F, int D, int P2, int P1, int ND, __nv_bfloat16* x,
                         int ldx, float* fm_logit, float* ssum, bool fm, cudaStream_t stream) {
  if (B <= 0) return;
  by_chunks(D, [&](auto n) {
    constexpr int chunks = decltype(n)::value;
    auto kernel = fm ? deepfm_pack_forward_kernel<true, chunks> : deepfm_pack_forward_kernel<false, chunks>;
    launch_pdl(kernel, dim3(grid_for(B, chunks * field_groups(chunks))), dim3(kThreads), 0, stream, rows2, inv2, slots2,
               rows1, inv1, slots1, dense, B, F, P2, P1, ND, x, ldx, fm_logit, ssum);
  });
}

void deepfm_pack_backward(const float* rows2, const int* inv2, const int* slots2, const int* inv1,
                          const __nv_bfloat16* dx, int lddx,
                          const float* dlogit, const float* ssum, int B, int F, int D, int P2, int RD, float* ugrad2,
                          float* ugrad1, cudaStream_t stream) {
  if (B <= 0) return;
  by_chunks(D, [&](auto n) {
    constexpr int chunks = decltype(n)::value;
    auto kernel = ssum != nullptr ? deepfm_pack_backward_kernel<true, chunks> : deepfm_pack_backward_kernel<false, chunks>;
    launch_pdl(kernel, dim3(grid_for(B, chunks * field_groups(chunks))), dim3(kThreads), 0, stream, rows2, inv2, slots2,
               inv1, dx, lddx, dlogit, ssum, B, F, P2, RD, ugrad2, ugrad1);
  });
}

}  // namespace cu
}  // namespace kb
