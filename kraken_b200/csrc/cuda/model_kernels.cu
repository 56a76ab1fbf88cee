// Memory-bound model kernels: jagged (bag) pooling, FM second-order
// interaction and binary cross entropy with logits.  Each makes one pass over
// its input at HBM speed with the reduction done in registers / shuffles.
//
// Counterparts in the reference: kraken/pytorch/py/jagged_ops.cc:14-420 (CPU,
// OpenMP), examples/DeepFM/model/DeepFM.py:96-107 (FM as torch expressions)
// and :140 (BCEWithLogits).
#include <cuda_bf16.h>

#include "common.cuh"
#include "kernels.h"

namespace kb {
namespace cu {

namespace {

constexpr int kThreads = 256;

int lanes_for(int dim) {
  int l = 1;
  while (l < dim && l < 32) l <<= 1;
  return l;
}

int grid_rows(long long rows, int lpr, int cap = 148 * 16) {
  long long g = (rows * lpr + kThreads - 1) / kThreads;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return static_cast<int>(g);
}

__global__ void __launch_bounds__(kThreads)
jagged_forward_kernel(const float* __restrict__ values, const float* __restrict__ weights,
                      const int64_t* __restrict__ offsets, int k, int dim, int lpr, int mean, float patch_value,
                      float* __restrict__ out) {
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = gtid % lpr;
  const int stride = (gridDim.x * blockDim.x) / lpr;
  for (int b = gtid / lpr; b < k; b += stride) {
    const int64_t lo = offsets[b], hi = offsets[b + 1];
    for (int j = lane; j < dim; j += lpr) {
      float acc = 0.f;
      for (int64_t r = lo; r < hi; ++r) acc += (weights ? weights[r] : 1.f) * values[r * dim + j];
      if (hi <= lo)
        acc = patch_value;
      else if (mean)
        acc /= static_cast<float>(hi - lo);
      out[static_cast<size_t>(b) * dim + j] = acc;
    }
  }
}

__global__ void __launch_bounds__(kThreads)
jagged_backward_kernel(const float* __restrict__ grads, const float* __restrict__ weights,
                       const int64_t* __restrict__ offsets, int k, int dim, int lpr, int mean,
                       float* __restrict__ out) {
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = gtid % lpr;
  const int stride = (gridDim.x * blockDim.x) / lpr;
  for (int b = gtid / lpr; b < k; b += stride) {
    const int64_t lo = offsets[b], hi = offsets[b + 1];
    if (hi <= lo) continue;
    const float scale = mean ? 1.f / static_cast<float>(hi - lo) : 1.f;
    for (int j = lane; j < dim; j += lpr) {
      const float g = grads[static_cast<size_t>(b) * dim + j] * scale;
      for (int64_t r = lo; r < hi; ++r) out[r * dim + j] = weights ? g * weights[r] : g;
    }
  }
}

__global__ void __launch_bounds__(kThreads)
fm_forward_kernel(const float* __restrict__ emb, int B, int F, int D, int lpr, float* __restrict__ out) {
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = gtid % lpr;
  const int stride = (gridDim.x * blockDim.x) / lpr;
  const unsigned group_mask = (lpr == 32 ? 0xffffffffu : ((1u << lpr) - 1u)) << ((threadIdx.x & 31) / lpr * lpr);
  const int rounds = (B + stride - 1) / stride;
  for (int it = 0; it < rounds; ++it) {
    const int b = gtid / lpr + it * stride;
    float part = 0.f;
    if (b < B) {
      const float* e = emb + static_cast<size_t>(b) * F * D;
      for (int j = lane; j < D; j += lpr) {
        float s = 0.f, q = 0.f;
        for (int f = 0; f < F; ++f) {
          const float v = e[f * D + j];
          s += v;
          q += v * v;
        }
        part += 0.5f * (s * s - q);
      }
    }
    for (int o = lpr >> 1; o > 0; o >>= 1) part += __shfl_xor_sync(group_mask, part, o);
    if (b < B && lane == 0) out[b] = part;
  }
}

__global__ void __launch_bounds__(kThreads)
fm_backward_kernel(const float* __restrict__ emb, const float* __restrict__ gout, int B, int F, int D, int lpr,
                   float* __restrict__ gemb) {
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = gtid % lpr;
  const int stride = (gridDim.x * blockDim.x) / lpr;
  for (int b = gtid / lpr; b < B; b += stride) {
    const float* e = emb + static_cast<size_t>(b) * F * D;
    float* g = gemb + static_cast<size_t>(b) * F * D;
    const float go = gout[b];
    for (int j = lane; j < D; j += lpr) {
      float s = 0.f;
      for (int f = 0; f < F; ++f) s += e[f * D + j];
      for (int f = 0; f < F; ++f) g[f * D + j] = go * (s - e[f * D + j]);
    }
  }
}

__global__ void __launch_bounds__(kThreads)
bce_kernel(const float* __restrict__ logits, const float* __restrict__ labels, int n, float inv_n, float* loss,
           float* __restrict__ grad) {
  pdl_enter();
  float acc = 0.f;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float x = logits[i], y = labels[i];
    const float ax = fabsf(x);
    const float t = expf(-ax);
    acc += fmaxf(x, 0.f) - x * y + log1pf(t);
    if (grad) {
      const float sig = x >= 0.f ? 1.f / (1.f + t) : t / (1.f + t);
      grad[i] = (sig - y) * inv_n;
    }
  }
  __shared__ float warp_sum[kThreads / 32];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = threadIdx.x < kThreads / 32 ? warp_sum[threadIdx.x] : 0.f;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) atomicAdd(loss, v * inv_n);
  }
}

// ---- Linear layer with a single output (the MLP's logit head): y[m] = x[m, :] . w + b
// Bound by memory: x is read once, 65536 x 400 in 16.5 us (3.2 TB/s, from L2 and DRAM).  Four rows a warp with 16-byte loads
// took 18.2 us (a row of 400 fills 50 lanes of 64), and 3.2 us for 2.7 at 4096 rows, which leave such warps too few.
__global__ void __launch_bounds__(kThreads)
rowdot_forward_kernel(const __nv_bfloat16* __restrict__ x, int ldx, const float* __restrict__ w,
                      const float* __restrict__ bias, const float* __restrict__ addend, int M, int K,
                      float* __restrict__ y) {
  pdl_enter();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int m = warp; m < M; m += nwarps) {
    const __nv_bfloat16* row = x + static_cast<size_t>(m) * ldx;
    float acc = 0.f;
    for (int k = lane * 2; k < K; k += 64) {
      const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(row + k);
      acc += __bfloat162float(v.x) * w[k];
      if (k + 1 < K) acc += __bfloat162float(v.y) * w[k + 1];
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) y[m] = acc + (bias ? bias[0] : 0.f) + (addend ? addend[m] : 0.f);
  }
}

__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    f[2 * q] = __uint_as_float(w[q] << 16);
    f[2 * q + 1] = __uint_as_float(w[q] & 0xFFFF0000u);
  }
}

// ---- Linear layer with a few outputs (a 10-class head) on bf16 activations: fp32 weights, products and sums.
// y[m, c] = x[m, :] . w[c, :] + b[c].  A block takes four rows, its warps share K, a lane reads 16 bytes of each row and the
// C weights of those columns (from L2: 160 KB for 10 x 4096, read once per four rows), and the warps' sums meet in shared
// memory.  C is a compile-time bound, rounded up to a multiple of 4, so that the sums stay in registers.  In library calls
// (float copy, fp32 GEMM of 64 x 64 tiles, split reduction; for the backward two GEMMs, two copies, mask, product, rounding
// and a row sum) the head of an MLP 784-4096-4096-4096-10 at batch 1024 took 105 us of a step of 604 us; the step takes
// 520 us with this kernel and the next.
constexpr int kHeadRows = 4;

template <int C>
__global__ void __launch_bounds__(kThreads)
head_forward_kernel(const __nv_bfloat16* __restrict__ x, int ldx, const float* __restrict__ w,
                    const float* __restrict__ bias, int M, int K, int classes, float* __restrict__ y) {
  pdl_enter();
  __shared__ float s_acc[kThreads / 32][kHeadRows * C];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * kHeadRows;
  float acc[kHeadRows][C];
#pragma unroll
  for (int r = 0; r < kHeadRows; ++r)
#pragma unroll
    for (int c = 0; c < C; ++c) acc[r][c] = 0.f;
  for (int k = threadIdx.x * 8; k < K; k += kThreads * 8) {
    float f[kHeadRows][8];
#pragma unroll
    for (int r = 0; r < kHeadRows; ++r)
      unpack8(m0 + r < M ? __ldcg(reinterpret_cast<const uint4*>(x + static_cast<size_t>(m0 + r) * ldx + k))
                         : make_uint4(0, 0, 0, 0), f[r]);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      if (c >= classes) break;
      const float4 wa = *reinterpret_cast<const float4*>(w + static_cast<size_t>(c) * K + k);
      const float4 wb = *reinterpret_cast<const float4*>(w + static_cast<size_t>(c) * K + k + 4);
#pragma unroll
      for (int r = 0; r < kHeadRows; ++r) {
        acc[r][c] += f[r][0] * wa.x + f[r][1] * wa.y + f[r][2] * wa.z + f[r][3] * wa.w;
        acc[r][c] += f[r][4] * wb.x + f[r][5] * wb.y + f[r][6] * wb.z + f[r][7] * wb.w;
      }
    }
  }
#pragma unroll
  for (int r = 0; r < kHeadRows; ++r)
#pragma unroll
    for (int c = 0; c < C; ++c) {
      float a = acc[r][c];
      for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      if (lane == 0) s_acc[warp][r * C + c] = a;
    }
  __syncthreads();
  for (int i = threadIdx.x; i < kHeadRows * C; i += kThreads) {
    const int r = i / C, c = i - r * C;
    if (m0 + r >= M || c >= classes) continue;
    float a = 0.f;
#pragma unroll
    for (int v = 0; v < kThreads / 32; ++v) a += s_acc[v][i];
    y[static_cast<size_t>(m0 + r) * classes + c] = a + (bias ? bias[c] : 0.f);
  }
}

// Its backward in one pass over the activations: dw[c, k] += sum_m g[m, c] x[m, k], db[c] += sum_m g[m, c] and
// dx[m, k] = (sum_c g[m, c] w[c, k]) * (x[m, k] > 0 if relu_mask), rounded to bf16.  A thread owns four columns - their C
// weights and C weight gradients live in its registers - and walks the rows of its block's range, whose g pass through
// shared memory.  The sums of the ranges are left in `part` [ranges][classes * K], behind them [ranges][classes] of db, and
// head_sum_kernel adds them up in the order of the ranges: reductions into dw added them in the order in which blocks
// arrived, and a training step that starts from the same state did not repeat bit for bit.  A single range (null part) adds
// to dw and db itself.  1024 rows of 4096 columns, 10 classes: 14.3 us with reductions, 16.8 so, 2.5 of them the second
// kernel; 65536 x 1024: 161 and 120 us; 65536 x 4096: 596 and 425.
constexpr int kHeadThreads = 128;
constexpr int kHeadStep = 64;   // rows of g in shared memory
constexpr int kHeadRange = 32;  // rows of a range at least

// Blocks of a multiprocessor: as many as 59, 92, 126 and 161 registers a thread leave room for.
constexpr int head_blocks(int classes) { return classes <= 4 ? 8 : classes <= 8 ? 5 : classes <= 12 ? 4 : 3; }

template <int C>
__global__ void __launch_bounds__(kHeadThreads, head_blocks(C))
head_backward_kernel(const __nv_bfloat16* __restrict__ x, int ldx, const float* __restrict__ w,
                     const float* __restrict__ g, int M, int K, int classes, int relu_mask, int range,
                     __nv_bfloat16* __restrict__ dx, int lddx, float* dw, float* db, float* __restrict__ part) {
  pdl_enter();
  __shared__ float s_g[kHeadStep][C];
  const int k = (blockIdx.y * kHeadThreads + threadIdx.x) * 4;
  float wk[C][4], acc[C][4], sum_g = 0.f;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const float4 v = k < K && c < classes ? *reinterpret_cast<const float4*>(w + static_cast<size_t>(c) * K + k)
                                          : make_float4(0.f, 0.f, 0.f, 0.f);
    wk[c][0] = v.x, wk[c][1] = v.y, wk[c][2] = v.z, wk[c][3] = v.w;
    acc[c][0] = acc[c][1] = acc[c][2] = acc[c][3] = 0.f;
  }
  const int begin = static_cast<int>(blockIdx.x) * range, end = min(M - begin, range) + begin;
  for (int r0 = begin; r0 < end; r0 += kHeadStep) {
    const int rows = min(kHeadStep, end - r0);
    __syncthreads();  // the rows before these have been used
    for (int i = threadIdx.x; i < rows * C; i += kHeadThreads) {
      const int r = i / C, c = i - r * C;
      s_g[r][c] = c < classes ? g[static_cast<size_t>(r0 + r) * classes + c] : 0.f;
    }
    __syncthreads();
    if (blockIdx.y == 0 && threadIdx.x < classes)
      for (int r = 0; r < rows; ++r) sum_g += s_g[r][threadIdx.x];
    if (k >= K) continue;
    constexpr int kAhead = 4;  // rows requested together
    for (int r = 0; r < rows; r += kAhead) {
      uint2 v[kAhead];
#pragma unroll
      for (int q = 0; q < kAhead; ++q)
        v[q] = r + q < rows ? __ldcg(reinterpret_cast<const uint2*>(x + static_cast<size_t>(r0 + r + q) * ldx + k))
                            : make_uint2(0, 0);
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        if (r + q >= rows) break;
        const float f[4] = {__uint_as_float(v[q].x << 16), __uint_as_float(v[q].x & 0xFFFF0000u),
                            __uint_as_float(v[q].y << 16), __uint_as_float(v[q].y & 0xFFFF0000u)};
        float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < C; ++c) {
          if (c >= classes) break;  // nothing of a class that is not there: 0 times infinity is not 0
          const float gc = s_g[r + q][c];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            d[e] += gc * wk[c][e];
            acc[c][e] += gc * f[e];
          }
        }
        if (dx == nullptr) continue;
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (relu_mask && !(f[e] > 0.f)) d[e] = 0.f;
        const __nv_bfloat162 lo = __floats2bfloat162_rn(d[0], d[1]), hi = __floats2bfloat162_rn(d[2], d[3]);
        *reinterpret_cast<uint2*>(dx + static_cast<size_t>(r0 + r + q) * lddx + k) =
            make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
      }
    }
  }
  const size_t n = static_cast<size_t>(classes) * K;
  if (k < K) {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      if (c >= classes) break;
      float4 v = make_float4(acc[c][0], acc[c][1], acc[c][2], acc[c][3]);
      float4* const to = reinterpret_cast<float4*>((part ? part + blockIdx.x * n : dw) + static_cast<size_t>(c) * K + k);
      if (part == nullptr) {
        const float4 o = *to;
        v = make_float4(o.x + v.x, o.y + v.y, o.z + v.z, o.w + v.w);
      }
      *to = v;
    }
  }
  if (blockIdx.y == 0 && threadIdx.x < classes) {
    if (part == nullptr)
      db[threadIdx.x] += sum_g;
    else
      part[gridDim.x * n + static_cast<size_t>(blockIdx.x) * classes + threadIdx.x] = sum_g;
  }
}

// dw += and db += the sums of the ranges.  A block takes 32 times four floats of dw, its warps the ranges in turn (eight loads
// of a lane in flight), and the first warp adds up what they have; the last block does db.
constexpr int kHeadSumWarps = 32;  // of a block where there are many ranges, else a quarter of them

__global__ void __launch_bounds__(32 * kHeadSumWarps)
head_sum_kernel(const float* __restrict__ part, int ranges, size_t n, int classes, float* dw, float* db) {
  pdl_enter();
  __shared__ float4 s_sum[kHeadSumWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const bool bias = blockIdx.x == gridDim.x - 1;
  const size_t at = (static_cast<size_t>(blockIdx.x) * 32 + lane) * 4;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  if (bias) {
    if (lane < classes)
      for (int r = warp; r < ranges; r += warps) a.x += part[ranges * n + static_cast<size_t>(r) * classes + lane];
  } else if (at < n) {
#pragma unroll 8
    for (int r = warp; r < ranges; r += warps) {
      const float4 v = *reinterpret_cast<const float4*>(part + r * n + at);
      a.x += v.x, a.y += v.y, a.z += v.z, a.w += v.w;
    }
  }
  s_sum[warp][lane] = a;
  __syncthreads();
  if (warp != 0) return;
  for (int v = 1; v < warps; ++v) {
    const float4 o = s_sum[v][lane];
    a.x += o.x, a.y += o.y, a.z += o.z, a.w += o.w;
  }
  if (bias) {
    if (lane < classes) db[lane] += a.x;
  } else if (at < n) {
    float4* const to = reinterpret_cast<float4*>(dw + at);
    const float4 o = *to;
    *to = make_float4(o.x + a.x, o.y + a.y, o.z + a.z, o.w + a.w);
  }
}

// dx[m, k] = dy[m] * w[k] * (x[m, k] > 0 if relu_mask), dw[k] += sum_m dy[m] x[m, k], db += sum_m dy[m]
__global__ void __launch_bounds__(kThreads)
rowdot_backward_kernel(const __nv_bfloat16* __restrict__ x, int ldx, const float* __restrict__ w,
                       const float* __restrict__ dy, int M, int K, int rows_per_block, int relu_mask,
                       __nv_bfloat16* __restrict__ dx, int lddx, float* dw, float* db) {
  pdl_enter();
  const int r0 = blockIdx.x * rows_per_block;
  const int r1 = min(M, r0 + rows_per_block);
  for (int k = threadIdx.x * 2; k < K; k += 2 * blockDim.x) {
    const float w0 = w[k], w1 = (k + 1 < K) ? w[k + 1] : 0.f;
    float a0 = 0.f, a1 = 0.f;
    for (int m = r0; m < r1; ++m) {
      const float g = dy[m];
      const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(x + static_cast<size_t>(m) * ldx + k);
      const float x0 = __bfloat162float(v.x), x1 = __bfloat162float(v.y);
      a0 += g * x0;
      a1 += g * x1;
      if (dx) {
        const float d0 = (!relu_mask || x0 > 0.f) ? g * w0 : 0.f;
        const float d1 = (!relu_mask || x1 > 0.f) ? g * w1 : 0.f;
        *reinterpret_cast<__nv_bfloat162*>(dx + static_cast<size_t>(m) * lddx + k) = __floats2bfloat162_rn(d0, d1);
      }
    }
    atomicAdd(dw + k, a0);
    if (k + 1 < K) atomicAdd(dw + k + 1, a1);
  }
  if (db && threadIdx.x == 0) {
    float s = 0.f;
    for (int m = r0; m < r1; ++m) s += dy[m];
    atomicAdd(db, s);
  }
}

// Same contract, for K % 8 == 0 and 16-byte aligned rows: a thread owns 8 columns (one 16-byte
// load and store per row), the block's threads are split into row lanes, and every thread keeps
// two rows in flight, so the kernel streams x and dx at memory speed instead of waiting on one
// 4-byte load at a time.
__global__ void __launch_bounds__(kThreads)
rowdot_backward_wide_kernel(const __nv_bfloat16* __restrict__ x, int ldx, const float* __restrict__ w,
                            const float* __restrict__ dy, int M, int K, int rows_per_block, int relu_mask,
                            __nv_bfloat16* __restrict__ dx, int lddx, float* dw, float* db) {
  pdl_enter();
  extern __shared__ float s_dw[];  // [K] partial sums of this block
  const int groups = K / 8;                       // 16-byte column groups per row
  const int lanes = blockDim.x / groups;          // row lanes (>= 1: the launcher guarantees groups <= blockDim.x)
  const int cg = threadIdx.x % groups;
  const int rl = threadIdx.x / groups;
  const int r0 = blockIdx.x * rows_per_block;
  const int r1 = min(M, r0 + rows_per_block);
  for (int k = threadIdx.x; k < K; k += blockDim.x) s_dw[k] = 0.f;
  __syncthreads();
  if (rl < lanes) {
    float wk[8], acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) wk[j] = w[cg * 8 + j], acc[j] = 0.f;
    for (int m = r0 + rl; m < r1; m += 2 * lanes) {
      const int m2 = m + lanes;
      const bool two = m2 < r1;
      const uint4 va = *reinterpret_cast<const uint4*>(x + static_cast<size_t>(m) * ldx + cg * 8);
      const uint4 vb = two ? *reinterpret_cast<const uint4*>(x + static_cast<size_t>(m2) * ldx + cg * 8) : va;
      const float ga = dy[m], gb = two ? dy[m2] : 0.f;
      const uint32_t wa[4] = {va.x, va.y, va.z, va.w}, wb[4] = {vb.x, vb.y, vb.z, vb.w};
      uint32_t oa[4], ob[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const __nv_bfloat162 pa = *reinterpret_cast<const __nv_bfloat162*>(&wa[j]);
        const __nv_bfloat162 pb = *reinterpret_cast<const __nv_bfloat162*>(&wb[j]);
        const float a0 = __bfloat162float(pa.x), a1 = __bfloat162float(pa.y);
        const float b0 = __bfloat162float(pb.x), b1 = __bfloat162float(pb.y);
        acc[2 * j] += ga * a0 + gb * b0;
        acc[2 * j + 1] += ga * a1 + gb * b1;
        const __nv_bfloat162 da = __floats2bfloat162_rn((!relu_mask || a0 > 0.f) ? ga * wk[2 * j] : 0.f,
                                                        (!relu_mask || a1 > 0.f) ? ga * wk[2 * j + 1] : 0.f);
        const __nv_bfloat162 dbv = __floats2bfloat162_rn((!relu_mask || b0 > 0.f) ? gb * wk[2 * j] : 0.f,
                                                         (!relu_mask || b1 > 0.f) ? gb * wk[2 * j + 1] : 0.f);
        oa[j] = *reinterpret_cast<const uint32_t*>(&da);
        ob[j] = *reinterpret_cast<const uint32_t*>(&dbv);
      }
      if (dx) {
        *reinterpret_cast<uint4*>(dx + static_cast<size_t>(m) * lddx + cg * 8) = make_uint4(oa[0], oa[1], oa[2], oa[3]);
        if (two)
          *reinterpret_cast<uint4*>(dx + static_cast<size_t>(m2) * lddx + cg * 8) = make_uint4(ob[0], ob[1], ob[2], ob[3]);
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) atomicAdd(&s_dw[cg * 8 + j], acc[j]);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < K; k += blockDim.x) atomicAdd(dw + k, s_dw[k]);
  if (db && threadIdx.x == 0) {
    float sum = 0.f;
    for (int m = r0; m < r1; ++m) sum += dy[m];
    atomicAdd(db, sum);
  }
}

// Buffers of a step's inputs, one launch for all of them: as copies of their own, each of two microseconds and its gap, they
// stood in front of every replay of a captured step (three of a DeepFM batch of 8192: 6.7 us, 3.3 so; of 65536: 12.4 and
// 8.2).  Thread t takes piece t of the buffers laid end to end; a buffer goes in pieces of the 16, 8 or 4 bytes that both of
// its addresses are aligned to (a batch sliced out of a larger tensor may start on any float), the rest of it by bytes.
__global__ void __launch_bounds__(kThreads)
copy_batch_kernel(CopyBatch b, long long pieces) {
  pdl_enter();
  constexpr int kUnroll = 4;
  const long long stride = static_cast<long long>(gridDim.x) * kThreads;
  for (long long p0 = blockIdx.x * static_cast<long long>(kThreads) + threadIdx.x; p0 < pieces; p0 += stride * kUnroll) {
    uint4 v[kUnroll];
    const char* s[kUnroll];
    char* d[kUnroll];
    int size[kUnroll], left[kUnroll];  // bytes of a whole piece and of this one, 0 for none
#pragma unroll
    for (int q = 0; q < kUnroll; ++q) {
      const long long p = p0 + q * stride;
      left[q] = 0;
      if (p >= pieces) continue;
      int l = 0;
      while (l + 1 < b.n && p >= b.first[l + 1]) ++l;
      const long long at = (p - b.first[l]) << b.shift[l];
      s[q] = b.src[l] + at;
      d[q] = b.dst[l] + at;
      size[q] = 1 << b.shift[l];
      left[q] = static_cast<int>(min(static_cast<long long>(size[q]), b.bytes[l] - at));
      if (left[q] < size[q]) continue;
      if (size[q] == 16)
        v[q] = __ldcs(reinterpret_cast<const uint4*>(s[q]));
      else if (size[q] == 8)
        *reinterpret_cast<uint2*>(&v[q]) = __ldcs(reinterpret_cast<const uint2*>(s[q]));
      else
        v[q].x = __ldcs(reinterpret_cast<const uint32_t*>(s[q]));
    }
#pragma unroll
    for (int q = 0; q < kUnroll; ++q) {
      if (left[q] == 0) continue;
      if (left[q] < size[q])
        for (int j = 0; j < left[q]; ++j) d[q][j] = s[q][j];
      else if (size[q] == 16)
        *reinterpret_cast<uint4*>(d[q]) = v[q];
      else if (size[q] == 8)
        *reinterpret_cast<uint2*>(d[q]) = make_uint2(v[q].x, v[q].y);
      else
        *reinterpret_cast<uint32_t*>(d[q]) = v[q].x;
    }
  }
}

// fp32 weight [N, K] -> bf16 copy [N, K] and bf16 transpose [K, N] in one pass (the forward and
// the input-gradient GEMMs want the two layouts).
__global__ void __launch_bounds__(256)
cast_w_wt_kernel(const float* __restrict__ w, int N, int K, __nv_bfloat16* __restrict__ w16,
                 __nv_bfloat16* __restrict__ wt16) {
  pdl_enter();
  __shared__ float tile[32][33];
  const int n0 = blockIdx.y * 32, k0 = blockIdx.x * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
  for (int r = ty; r < 32; r += 8) {
    const int n = n0 + r, k = k0 + tx;
    const float v = (n < N && k < K) ? w[static_cast<size_t>(n) * K + k] : 0.f;
    tile[r][tx] = v;
    if (n < N && k < K) w16[static_cast<size_t>(n) * K + k] = __float2bfloat16(v);
  }
  __syncthreads();
  for (int r = ty; r < 32; r += 8) {
    const int k = k0 + r, n = n0 + tx;
    if (k < K && n < N) wt16[static_cast<size_t>(k) * N + n] = __float2bfloat16(tile[tx][r]);
  }
}

// The same for all layers of an MLP in one launch, 64 x 64 tiles: 16-byte loads, 8-byte stores of the copy, 16-byte stores
// of the transpose (which is left out where no backward pass will want it).  Bound by HBM: 4 bytes read, 2 or 4 written
// per weight.  The 32 x 32 kernel above, with its 2-byte stores, takes 110 us for 784-4096-4096-4096, 48 us this
// one, of 45 us at the copy rate.
__global__ void __launch_bounds__(256)
cast_weights_kernel(CastBatch b) {
  pdl_enter();
  constexpr int kPitch = 66;  // columns of the tile are read 8 rows apart: 33 words of pitch spread them over the banks
  __shared__ __nv_bfloat16 tile[64 * kPitch];
  int l = 0;
  while (l + 1 < b.layers && static_cast<int>(blockIdx.x) >= b.first[l + 1]) ++l;
  const int N = b.N[l], K = b.K[l];
  const int at = blockIdx.x - b.first[l];
  const int tiles_k = (K + 63) / 64;
  const int n0 = at / tiles_k * 64, k0 = at % tiles_k * 64;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float4 v[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int n = n0 + ty + 16 * j, k = k0 + tx * 4;
    v[j] = n < N && k < K ? __ldcs(reinterpret_cast<const float4*>(b.w[l] + static_cast<size_t>(n) * K + k))
                          : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int n = n0 + ty + 16 * j, k = k0 + tx * 4;
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v[j].x, v[j].y), hi = __floats2bfloat162_rn(v[j].z, v[j].w);
    uint2 packed;
    packed.x = *reinterpret_cast<const uint32_t*>(&lo);
    packed.y = *reinterpret_cast<const uint32_t*>(&hi);
    if (n < N && k < K) *reinterpret_cast<uint2*>(b.w16[l] + static_cast<size_t>(n) * K + k) = packed;
    uint32_t* t = reinterpret_cast<uint32_t*>(tile + (ty + 16 * j) * kPitch + tx * 4);
    t[0] = packed.x;
    t[1] = packed.y;
  }
  if (b.wt16[l] == nullptr) return;  // the same for the whole block
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int kk = (threadIdx.x >> 3) + 32 * j, nn = (threadIdx.x & 7) * 8;
    const int k = k0 + kk, n = n0 + nn;
    if (k >= K || n >= N) continue;
    __align__(16) __nv_bfloat16 col[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) col[i] = tile[(nn + i) * kPitch + kk];
    *reinterpret_cast<uint4*>(b.wt16[l] + static_cast<size_t>(k) * N + n) = *reinterpret_cast<const uint4*>(col);
  }
}

}  // namespace

void copy_batch(CopyBatch b, cudaStream_t stream) {
  long long pieces = 0;
  for (int l = 0; l < b.n; ++l) {
    const uintptr_t both = reinterpret_cast<uintptr_t>(b.src[l]) | reinterpret_cast<uintptr_t>(b.dst[l]);
    b.shift[l] = both % 16 == 0 ? 4 : both % 8 == 0 ? 3 : 2;
    b.first[l] = pieces;
    pieces += (b.bytes[l] + (1 << b.shift[l]) - 1) >> b.shift[l];
  }
  if (pieces <= 0) return;
  long long grid = (pieces + 4 * kThreads - 1) / (4 * kThreads);
  if (grid > 148 * 8) grid = 148 * 8;
  launch_pdl(copy_batch_kernel, dim3(static_cast<unsigned>(grid)), dim3(kThreads), 0, stream, b, pieces);
}

void cast_weights(CastBatch b, cudaStream_t stream) {
  int tiles = 0;
  for (int l = 0; l < b.layers; ++l) {
    b.first[l] = tiles;
    tiles += ((b.N[l] + 63) / 64) * ((b.K[l] + 63) / 64);
  }
  if (tiles > 0) launch_pdl(cast_weights_kernel, dim3(tiles), dim3(256), 0, stream, b);
}

void jagged_forward(const float* values, const float* weights, const int64_t* offsets, int k, int dim, bool mean,
                    float patch_value, float* out, cudaStream_t stream) {
  if (k <= 0) return;
  const int lpr = lanes_for(dim);
  jagged_forward_kernel<<<grid_rows(k, lpr), kThreads, 0, stream>>>(values, weights, offsets, k, dim, lpr, mean ? 1 : 0,
                                                                    patch_value, out);
}

void jagged_backward(const float* grads, const float* weights, const int64_t* offsets, int k, int dim, bool mean,
                     float* out, cudaStream_t stream) {
  if (k <= 0) return;
  const int lpr = lanes_for(dim);
  jagged_backward_kernel<<<grid_rows(k, lpr), kThreads, 0, stream>>>(grads, weights, offsets, k, dim, lpr, mean ? 1 : 0,
                                                                     out);
}

void fm_forward(const float* emb, int B, int F, int D, float* out, cudaStream_t stream) {
  if (B <= 0) return;
  const int lpr = lanes_for(D);
  fm_forward_kernel<<<grid_rows(B, lpr), kThreads, 0, stream>>>(emb, B, F, D, lpr, out);
}

void fm_backward(const float* emb, const float* gout, int B, int F, int D, float* gemb, cudaStream_t stream) {
  if (B <= 0) return;
  const int lpr = lanes_for(D);
  fm_backward_kernel<<<grid_rows(B, lpr), kThreads, 0, stream>>>(emb, gout, B, F, D, lpr, gemb);
}

void bce_forward_backward(const float* logits, const float* labels, int n, float* loss, float* grad,
                          cudaStream_t stream) {
  if (n <= 0) return;
  int grid = (n + kThreads - 1) / kThreads;
  if (grid > 148 * 4) grid = 148 * 4;
  launch_pdl(bce_kernel, dim3(grid), dim3(kThreads), 0, stream, logits, labels, n, 1.f / static_cast<float>(n), loss, grad);
}

void rowdot_forward(const __nv_bfloat16* x, int ldx, const float* w, const float* bias, const float* addend, int M,
                    int K, float* y, cudaStream_t stream) {
  if (M <= 0) return;
  int grid = (M * 32 + kThreads - 1) / kThreads;
  if (grid > 148 * 8) grid = 148 * 8;
  launch_pdl(rowdot_forward_kernel, dim3(grid), dim3(kThreads), 0, stream, x, ldx, w, bias, addend, M, K, y);
}

void rowdot_backward(const __nv_bfloat16* x, int ldx, const float* w, const float* dy, int M, int K, bool relu_mask,
                     __nv_bfloat16* dx, int lddx, float* dw, float* db, cudaStream_t stream) {
  if (M <= 0) return;
  int blocks = 148 * 4;
  int rows_per_block = (M + blocks - 1) / blocks;
  if (rows_per_block < 16) rows_per_block = 16;
  blocks = (M + rows_per_block - 1) / rows_per_block;
  const bool wide = K % 8 == 0 && K / 8 <= kThreads && ldx % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 &&
                    (dx == nullptr || (lddx % 8 == 0 && (reinterpret_cast<uintptr_t>(dx) & 15) == 0));
  if (wide) {
    launch_pdl(rowdot_backward_wide_kernel, dim3(blocks), dim3(kThreads), K * sizeof(float), stream, x, ldx, w, dy, M, K,
               rows_per_block, relu_mask ? 1 : 0, dx, lddx, dw, db);
    return;
  }
  launch_pdl(rowdot_backward_kernel, dim3(blocks), dim3(kThreads), 0, stream, x, ldx, w, dy, M, K, rows_per_block,
             relu_mask ? 1 : 0, dx, lddx, dw, db);
}

bool head_supported(const void* x, int ldx, const void* w, int K, int classes) {
  return classes >= 1 && classes <= kMaxHead && K % 8 == 0 && ldx % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 &&
         (reinterpret_cast<uintptr_t>(w) & 15) == 0;
}

void head_forward(const __nv_bfloat16* x, int ldx, const float* w, const float* bias, int M, int K, int classes, float* y,
                  cudaStream_t stream) {
  if (M <= 0) return;
  auto kernel = classes <= 4 ? head_forward_kernel<4> : classes <= 8 ? head_forward_kernel<8>
                : classes <= 12 ? head_forward_kernel<12> : head_forward_kernel<16>;
  launch_pdl(kernel, dim3((M + kHeadRows - 1) / kHeadRows), dim3(kThreads), 0, stream, x, ldx, w, bias, M, K, classes, y);
}

// Rows of a range and how many there are: two waves of blocks, or as many as there are rows for.  (65536 x 1024, 3 classes:
// 68 us; 81 with whole steps of rows a range, whose blocks are 1.15 waves; 91 with half a wave.)
static int head_range(int M, int K, int classes, int* ranges) {
  const int columns = (K / 4 + kHeadThreads - 1) / kHeadThreads, blocks = 148 * 2 * head_blocks(classes);
  const int most = blocks < columns ? 1 : blocks / columns;
  int range = ((M - 1) / most + 4) / 4 * 4;
  if (range < kHeadRange) range = kHeadRange;
  *ranges = (M - 1) / range + 1;
  return range;
}

size_t head_part_floats(int M, int K, int classes) {
  if (M <= 0) return 0;
  int ranges;
  head_range(M, K, classes, &ranges);
  return ranges > 1 ? static_cast<size_t>(ranges) * classes * (static_cast<size_t>(K) + 1) : 0;
}

void head_backward(const __nv_bfloat16* x, int ldx, const float* w, const float* g, int M, int K, int classes,
                   bool relu_mask, __nv_bfloat16* dx, int lddx, float* dw, float* db, float* part, cudaStream_t stream) {
  if (M <= 0) return;
  auto kernel = classes <= 4 ? head_backward_kernel<4> : classes <= 8 ? head_backward_kernel<8>
                : classes <= 12 ? head_backward_kernel<12> : head_backward_kernel<16>;
  int ranges;
  const int range = head_range(M, K, classes, &ranges);
  if (ranges == 1) part = nullptr;
  const dim3 grid(ranges, (K / 4 + kHeadThreads - 1) / kHeadThreads);  // y ends at 65535
  launch_pdl(kernel, grid, dim3(kHeadThreads), 0, stream, x, ldx, w, g, M, K, classes, relu_mask ? 1 : 0, range, dx, lddx, dw,
             db, part);
  if (part != nullptr) {
    const size_t n = static_cast<size_t>(classes) * K;
    const int warps = ranges > 64 ? kHeadSumWarps : kHeadSumWarps / 4;
    launch_pdl(head_sum_kernel, dim3(static_cast<unsigned>((n / 4 + 31) / 32 + 1)), dim3(32 * warps), 0, stream, part, ranges,
               n, classes, dw, db);
  }
}

void cast_w_wt(const float* w, int N, int K, __nv_bfloat16* w16, __nv_bfloat16* wt16, cudaStream_t stream) {
  if (N <= 0 || K <= 0) return;
  launch_pdl(cast_w_wt_kernel, dim3((K + 31) / 32, (N + 31) / 32), dim3(256), 0, stream, w, N, K, w16, wt16);
}

}  // namespace cu
}  // namespace kb
