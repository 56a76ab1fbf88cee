// The sparse exchange of a job on ONE GPU.
//
// With one rank there is nobody to exchange with: the rank that looks ids up owns every row.  The
// kernels of sparse.cu would still move every row through the channel's inboxes, because that is what
// peers read and write; these move each row once.
#include "sparse_common.cuh"

namespace kb {
namespace cu {

using namespace sparse_detail;

namespace {

// Early residency (launch_pdl) pays for a launch that leaves room on the chip.  The waiting blocks of a grid that
// fills it hold the registers and threads that the kernels of another stream - in a training step the weight
// gradients beside the sparse backward - could use: a DeepFM step of 8192 samples takes 237 us with an early
// update grid and 226 us with one in plain stream order, one of 65536 samples 980 and 963 us.
constexpr int kFullGrid = 148 * 4;

// Optimizer update straight from the segment-sum buffer: entry u of `ugrad` is the gradient of the row
// in slot_cache[u], and is zeroed here for the next step's segment-sum.
//
// Bound by HBM: per row it must read the gradient, read and write value and state rows and write the
// zeros.  The two-kernel form (push_dispatch into the inbox, push_update out of it) wrote and read
// every gradient row once more.  Measured for 2.3 M rows of 64 floats with Adagrad: 853 us before (310 + 543), 590 us
// now, of 543 us at the copy rate; 0.55 M rows of 20 floats with Adam: 245 us before, 214 us now.  A row is handled by `chunks` neighbouring threads of a block, one
// 16-byte chunk each (a row width like 20 floats leaves no lane idle, as a power-of-two group per row
// would); the threads of a row may sit in two warps, so its step counter is read by all of them before
// the block barrier and written behind it.
template <int VEC, int OPT>
__global__ void __launch_bounds__(kThreads, 4)
local_update_kernel(TableView t, float* __restrict__ ugrad, const int* __restrict__ off,
                    const int* __restrict__ slot_cache, OptimPOD optim_in, const float* __restrict__ lr_ptr, int cap_s,
                    int chunks, int tpr) {
  pdl_enter();
  using V = Vec<VEC>;
  OptimPOD optim = optim_in;
  optim.type = OPT;
  const float lr = *lr_ptr;
  const int U = off[1];
  const int rows = kThreads / tpr;             // rows of one block and pass
  const int r = threadIdx.x / tpr;
  const int c0 = threadIdx.x - r * tpr;
  const int stride = gridDim.x * rows;
  const int limit = min(U, cap_s);
  const bool counts = t.steps != nullptr;
  const bool active = r < rows;
  int u = blockIdx.x * rows + r;
  int slot = active && u < limit ? slot_cache[u] : -1;
  for (int base = blockIdx.x * rows; base < U; base += stride, u += stride) {
    const int next = active && u + stride < limit ? slot_cache[u + stride] : -1;
    const bool mine = active && u < U;
    float* const gu = ugrad + static_cast<size_t>(u) * t.dim;
    const size_t row = static_cast<size_t>(slot < 0 ? 0 : slot) * t.dim;
    // an id that was not found (reported by the lookup) has no row: its gradient is dropped
    const bool found = mine && slot >= 0;
    int step_i = 1;
    if (counts && found) step_i = t.steps[slot] + 1;
    float g[VEC], w[VEC], a0[VEC], a1[VEC], a2[VEC];
    auto load = [&](int c) {
      *reinterpret_cast<typename V::T*>(g) = V::ldcg(gu + c * VEC);
      *reinterpret_cast<typename V::T*>(w) = V::ld(t.val + row + c * VEC);
      if (t.s[0]) *reinterpret_cast<typename V::T*>(a0) = V::ld(t.s[0] + row + c * VEC);
      if (t.s[1]) *reinterpret_cast<typename V::T*>(a1) = V::ld(t.s[1] + row + c * VEC);
      if (t.s[2]) *reinterpret_cast<typename V::T*>(a2) = V::ld(t.s[2] + row + c * VEC);
    };
    if (found) load(c0);  // in flight across the barrier
    if (counts) {
      __syncthreads();
      if (found && c0 == 0) t.steps[slot] = step_i;
    }
    if (found) {
      const int64_t step = step_i;
      const AdamBias ab = optim.type == 1 ? AdamBiasAt(optim, step) : AdamBias{1.f, 1.f};
      for (int c = c0; c < chunks; c += tpr) {
        if (c != c0) load(c);
#pragma unroll
        for (int e = 0; e < VEC; ++e) UpdateElem(optim, lr, g[e], step, ab, w[e], a0[e], a1[e], a2[e]);
        V::st(t.val + row + c * VEC, *reinterpret_cast<typename V::T*>(w));
        if (t.s[0]) V::st(t.s[0] + row + c * VEC, *reinterpret_cast<typename V::T*>(a0));
        if (t.s[1]) V::st(t.s[1] + row + c * VEC, *reinterpret_cast<typename V::T*>(a1));
        if (t.s[2]) V::st(t.s[2] + row + c * VEC, *reinterpret_cast<typename V::T*>(a2));
      }
    }
    if (mine)
      for (int c = c0; c < chunks; c += tpr) V::st(gu + c * VEC, V::zero());
    slot = next;
  }
}

template <int VEC>
void launch_local_update(int grid, cudaStream_t stream, const TableView& t, float* ugrad, const int* off,
                         const int* slot_cache, const OptimPOD& optim, const float* lr, int cap_s, int chunks, int tpr) {
  auto go = [&](auto kernel) {
    launch_pdl_if(grid < kFullGrid, kernel, dim3(grid), dim3(kThreads), 0, stream, t, ugrad, off, slot_cache, optim, lr,
                  cap_s, chunks, tpr);
  };
  switch (optim.type) {
    case 0: go(local_update_kernel<VEC, 0>); break;
    case 1: go(local_update_kernel<VEC, 1>); break;
    case 2: go(local_update_kernel<VEC, 2>); break;
    default: go(local_update_kernel<VEC, 3>); break;
  }
}

}  // namespace

void local_push_update(TableHost table, float* ugrad, const int* off, const int* slot_cache, int max_n, int cap_s,
                       OptimPOD optim, const float* lr, cudaStream_t stream) {
  const RowGeom g = row_geom(table.dim);
  const int tpr = g.chunks < kThreads ? g.chunks : kThreads;
  const int rows = kThreads / tpr;
  const int grid = grid_for(max_n, rows);
  if (g.vec == 4)
    launch_local_update<4>(grid, stream, to_view(table), ugrad, off, slot_cache, optim, lr, cap_s, g.chunks, tpr);
  else
    launch_local_update<1>(grid, stream, to_view(table), ugrad, off, slot_cache, optim, lr, cap_s, g.chunks, tpr);
}

}  // namespace cu
}  // namespace kb
