// The sparse exchange of a job on ONE GPU.
//
// With one rank there is nobody to exchange with: the rank that looks ids up owns every row.  The
// kernels of sparse.cu would still move every row through the channel's inboxes, because that is what
// peers read and write; these move each row once.
#include <cuda_bf16.h>

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

// Rows of less than a sector (8 floats) are summed in any case: telling the update where a gradient is takes as much
// traffic as the gradient.
constexpr int kDirectDim = 8;

// Where the update finds the gradient of every id's first occurrence.
struct DirectSource {
  const float* grads;          // [n, dim], or [bags, dim]
  const __nv_bfloat16* grads16;  // of bags that were pooled into an MLP input: bag b = field b % fields of row b / fields
  int ld16, fields;
  const int64_t* bag_offsets;  // null: one gradient row per occurrence
  int nbags;
  const float* weights;        // per occurrence of a bag, or null
  const uint8_t* bag_mean;
  int mean;
  const int* win;              // unique id -> its first occurrence
  // Unique id -> {bag of its first occurrence, factor of that bag's gradient as bits of a float} (null without bags); bag -1
  // where the occurrence lies outside every bag (offsets that start behind the first id or end before the last).  Every push
  // writes the entries of all of its unique ids.
  const int2* bag_of;
  const uint32_t* multi;       // == *epoch: the id occurs more than once
  const uint32_t* epoch;       // number of the lookup
  __device__ __forceinline__ float bag_scale(int b) const {
    const int64_t len = bag_offsets[b + 1] - bag_offsets[b];
    const bool is_mean = bag_mean ? bag_mean[b] != 0 : mean != 0;
    return is_mean && len > 0 ? 1.f / static_cast<float>(len) : 1.f;
  }
  // where the gradient of row `i` begins, and VEC elements of it
  template <bool B16>
  __device__ __forceinline__ size_t row(int i, int dim) const {
    if (!B16) return static_cast<size_t>(i) * dim;
    const int sample = i / fields;
    return static_cast<size_t>(sample) * ld16 + (i - sample * fields) * dim;
  }
  template <int VEC, bool B16>
  __device__ __forceinline__ typename Vec<VEC>::T ldcg(size_t at) const {
    if constexpr (B16) {
      static_assert(VEC == 4, "bf16 gradients go by four");
      const uint2 v = __ldcg(reinterpret_cast<const uint2*>(grads16 + at));
      return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xFFFF0000u), __uint_as_float(v.y << 16),
                         __uint_as_float(v.y & 0xFFFF0000u));
    } else {
      return Vec<VEC>::ldcg(grads + at);
    }
  }
};

// Optimizer update straight from the segment-sum buffer: entry u of `ugrad` is the gradient of the row
// in slot_cache[u], and is zeroed here for the next step's segment-sum.
//
// Bound by HBM: per row it must read the gradient, read and write value and state rows and write the zeros.  The
// two-kernel form (push_dispatch into the inbox, push_update out of it) wrote and read every gradient row once more.
// Measured for 0.55 M rows of 20 floats with Adam: 245 us before, 194 us so, 99 us since a row's state lies beside its
// value.  A row is handled by `chunks` neighbouring
// threads of a block, one 16-byte chunk each (a row width like 20 floats leaves no lane idle, as a power-of-two group
// per row would); the threads of a row may sit in two warps, so its step counter is read by all of them before the
// block barrier and written behind it.  What is known of the next row is fetched one pass ahead.  Nine blocks of 128
// threads per SM leave 56 registers a thread, which holds every variant but those of 4-float chunks with direct gradients for
// Adam (4 bytes spilled with rows, 20 with bags, 16 with bf16 ones) and RMSprop (4 with bags); eight of them were 3 to 6 % slower, four or five blocks of 256 threads up to
// 25 %.
//
// FROM: with kFromRows and kFromBags the gradient of every id's first occurrence is read from the caller's gradients
// (`so`); `ugrad` holds the sum of the others, which is not read where there are none.  2.3 M rows of 64 floats,
// Adagrad: 853 us with two kernels, 590 us with one that reads and clears every sum, 500 us so, of 460 us at the copy
// rate.  A first occurrence outside every bag has no gradient: the row is updated with the sum of the others, or with
// zeros.
constexpr int kUpdateThreads = 128;
enum GradSource { kFromSum = 0, kFromRows = 1, kFromBags = 2, kFromBags16 = 3 };

template <int VEC, int OPT, int FROM>
__global__ void __launch_bounds__(kUpdateThreads, 9)
local_update_kernel(TableView t, float* __restrict__ ugrad, const int* __restrict__ off,
                    const int* __restrict__ slot_cache, DirectSource so, OptimPOD optim_in,
                    const float* __restrict__ lr_ptr, int cap_s, int chunks, int tpr) {
  pdl_enter();
  using V = Vec<VEC>;
  constexpr bool kBags = FROM == kFromBags || FROM == kFromBags16, kHalf = FROM == kFromBags16;
  const uint32_t now = FROM != kFromSum ? *so.epoch : 0;
  OptimPOD optim = optim_in;
  optim.type = OPT;
  const float lr = *lr_ptr;
  const int U = off[1];
  const int rows = kUpdateThreads / tpr;             // rows of one block and pass
  const int r = threadIdx.x / tpr;
  const int c0 = threadIdx.x - r * tpr;
  const int stride = gridDim.x * rows;
  const int limit = min(U, cap_s);
  const bool counts = t.steps != nullptr;
  const bool active = r < rows;
  int u = blockIdx.x * rows + r;
  // what is known of a row before its data: its slot, the row of `grads`, whether there is a sum of others
  auto slot_of = [&](int v) { return active && v < limit ? slot_cache[v] : -1; };
  // (one 8-byte entry: from win, the offsets, the means and the weights it was seven loads of each of a row's threads, and the
  // multi-hot step, 3.2 M rows of 64 floats, took 2590 us instead of 2345)
  auto src_of = [&](int v) {
    if (FROM == kFromSum || !active || v >= U) return make_int2(0, 0);
    return kBags ? so.bag_of[v] : make_int2(so.win[v], 0);
  };
  auto many_of = [&](int v) { return active && v < U && (FROM == kFromSum || so.multi[v] == now); };
  int slot = slot_of(u);
  int2 from = src_of(u);
  bool many = many_of(u);
  for (int base = blockIdx.x * rows; base < U; base += stride, u += stride) {
    const int next = slot_of(u + stride);
    const int2 next_from = src_of(u + stride);
    const bool next_many = many_of(u + stride);
    const bool mine = active && u < U;
    float* const gu = ugrad + static_cast<size_t>(u) * t.dim;
    const bool direct = FROM == kFromRows || (kBags && static_cast<unsigned>(from.x) < static_cast<unsigned>(so.nbags));
    const size_t gd = FROM != kFromSum && direct ? so.template row<kHalf>(from.x, t.dim) : 0;
    const float scale = __int_as_float(from.y);
    const size_t row = static_cast<size_t>(slot < 0 ? 0 : slot) * t.pitch;
    int* const counter = t.steps + static_cast<size_t>(slot < 0 ? 0 : slot) * t.step_pitch;
    // an id that was not found (reported by the lookup) has no row: its gradient is dropped
    const bool found = mine && slot >= 0;
    int step_i = 1;
    if (counts && found) step_i = *counter + 1;
    float g[VEC], d[VEC], w[VEC], a0[VEC], a1[VEC], a2[VEC];
    auto load = [&](int c) {
      *reinterpret_cast<typename V::T*>(g) = many ? V::ldcg(gu + c * VEC) : V::zero();
      if (FROM != kFromSum) *reinterpret_cast<typename V::T*>(d) = direct ? so.template ldcg<VEC, kHalf>(gd + c * VEC) : V::zero();
      *reinterpret_cast<typename V::T*>(w) = V::ld(t.val + row + c * VEC);
      if (t.s[0]) *reinterpret_cast<typename V::T*>(a0) = V::ld(t.s[0] + row + c * VEC);
      if (t.s[1]) *reinterpret_cast<typename V::T*>(a1) = V::ld(t.s[1] + row + c * VEC);
      if (t.s[2]) *reinterpret_cast<typename V::T*>(a2) = V::ld(t.s[2] + row + c * VEC);
    };
    if (found) load(c0);  // in flight across the barrier
    if (counts) {
      __syncthreads();
      if (found && c0 == 0) *counter = step_i;
    }
    if (found) {
      const int64_t step = step_i;
      const AdamBias ab = optim.type == 1 ? AdamBiasAt(optim, step) : AdamBias{1.f, 1.f};
      for (int c = c0; c < chunks; c += tpr) {
        if (c != c0) load(c);
        if (FROM != kFromSum && direct) {
#pragma unroll
          for (int e = 0; e < VEC; ++e) g[e] += kBags ? d[e] * scale : d[e];
        }
#pragma unroll
        for (int e = 0; e < VEC; ++e) UpdateElem(optim, lr, g[e], step, ab, w[e], a0[e], a1[e], a2[e]);
        V::st(t.val + row + c * VEC, *reinterpret_cast<typename V::T*>(w));
        if (t.s[0]) V::st(t.s[0] + row + c * VEC, *reinterpret_cast<typename V::T*>(a0));
        if (t.s[1]) V::st(t.s[1] + row + c * VEC, *reinterpret_cast<typename V::T*>(a1));
        if (t.s[2]) V::st(t.s[2] + row + c * VEC, *reinterpret_cast<typename V::T*>(a2));
      }
    }
    if (many)
      for (int c = c0; c < chunks; c += tpr) V::st(gu + c * VEC, V::zero());
    slot = next, from = next_from, many = next_many;
  }
}

template <int VEC, int FROM>
void launch_local_update(int grid, cudaStream_t stream, const TableView& t, float* ugrad, const int* off,
                         const int* slot_cache, const DirectSource& so, const OptimPOD& optim, const float* lr, int cap_s,
                         int chunks, int tpr) {
  auto go = [&](auto kernel) {
    launch_pdl_if(grid < 2 * kFullGrid, kernel, dim3(grid), dim3(kUpdateThreads), 0, stream, t, ugrad, off, slot_cache, so,
                  optim, lr, cap_s, chunks, tpr);
  };
  switch (optim.type) {
    case 0: go(local_update_kernel<VEC, 0, FROM>); break;
    case 1: go(local_update_kernel<VEC, 1, FROM>); break;
    case 2: go(local_update_kernel<VEC, 2, FROM>); break;
    default: go(local_update_kernel<VEC, 3, FROM>); break;
  }
}

// Segment-sum of the gradients of all but every id's first occurrence; `first` < 0 names that one, and its gradient is
// left to the update, which for a bag is told the bag.  Bound by the 16-byte reductions in L2 and by the HBM traffic of
// reductions into rows that are not there: an id that occurs once has its row neither read and written here nor read
// and cleared in the update.  3.4 M rows of 64 floats: 490 us with every row summed, 245 us now.  The ids with a sum are
// marked here, by plain stores: marking them in the dedup, with a look at the mark first, took 84 us for 240 k ids instead
// of 7 - lines that are read and written from both dies move to and fro.
template <int VEC>
__global__ void __launch_bounds__(kThreads)
local_scatter_kernel(const int* __restrict__ inv, const int* __restrict__ first, DirectSource so, uint32_t* multi, int n,
                     int dim, int chunks, int tpr, float* ugrad) {
  pdl_enter();
  using V = Vec<VEC>;
  constexpr int kUnroll = 4;
  const uint32_t now = *so.epoch;
  const int rows = kThreads / tpr;
  const int r = threadIdx.x / tpr, c0 = threadIdx.x - r * tpr;
  if (r >= rows) return;
  const int stride = gridDim.x * rows;
  for (int i0 = blockIdx.x * rows + r; i0 < n; i0 += stride * kUnroll) {
    int u[kUnroll];
#pragma unroll
    for (int q = 0; q < kUnroll; ++q) {
      const int i = i0 + q * stride;
      u[q] = i < n && first[i] >= 0 ? inv[i] : -1;
    }
    for (int c = c0; c < chunks; c += tpr) {
      typename V::T v[kUnroll];
#pragma unroll
      for (int q = 0; q < kUnroll; ++q)
        if (u[q] >= 0) v[q] = V::ld(so.grads + static_cast<size_t>(i0 + q * stride) * dim + c * VEC);
#pragma unroll
      for (int q = 0; q < kUnroll; ++q)
        if (u[q] >= 0) {
          V::red(ugrad + static_cast<size_t>(u[q]) * dim + c * VEC, v[q]);
          if (c == 0) multi[u[q]] = now;
        }
    }
  }
}

template <int VEC, bool B16>
__global__ void __launch_bounds__(kThreads)
local_bag_scatter_kernel(const int* __restrict__ inv, const int* __restrict__ first, DirectSource so, uint32_t* multi,
                         int2* __restrict__ bag_of, int n, int nbags, int dim, int chunks, int tpr, float* ugrad) {
  pdl_enter();
  using V = Vec<VEC>;
  constexpr int kUnroll = 4;
  const uint32_t now = *so.epoch;
  const int rows = kThreads / tpr;
  const int g = threadIdx.x / tpr, c0 = threadIdx.x - g * tpr;
  // ids in front of the first bag and behind the last: their first occurrences have no gradient
  const int head = static_cast<int>(min(static_cast<int64_t>(n), so.bag_offsets[0]));
  const int tail = static_cast<int>(max(static_cast<int64_t>(0), so.bag_offsets[nbags]));
  for (int j = blockIdx.x * kThreads + threadIdx.x; j < head || j < n - tail; j += gridDim.x * kThreads) {
    if (j < head && first[j] < 0) bag_of[inv[j]] = make_int2(-1, 0);
    if (j < n - tail && first[tail + j] < 0) bag_of[inv[tail + j]] = make_int2(-1, 0);
  }
  if (g >= rows) return;
  for (int b = blockIdx.x * rows + g; b < nbags; b += gridDim.x * rows) {
    const int lo = static_cast<int>(so.bag_offsets[b]), hi = static_cast<int>(so.bag_offsets[b + 1]);
    const float scale = so.bag_scale(b);
    for (int c = c0; c < chunks; c += tpr) {
      const typename V::T v = V::scale(so.template ldcg<VEC, B16>(so.template row<B16>(b, dim) + c * VEC), scale);
      for (int i0 = lo; i0 < hi; i0 += kUnroll) {
        int u[kUnroll], f[kUnroll];
#pragma unroll
        for (int q = 0; q < kUnroll; ++q) {
          u[q] = i0 + q < hi ? inv[i0 + q] : -1;
          f[q] = i0 + q < hi ? first[i0 + q] : 0;
        }
#pragma unroll
        for (int q = 0; q < kUnroll; ++q) {
          if (u[q] < 0) continue;
          if (f[q] >= 0) {
            V::red(ugrad + static_cast<size_t>(u[q]) * dim + c * VEC, so.weights ? V::scale(v, so.weights[i0 + q]) : v);
            if (c == 0) multi[u[q]] = now;
          } else if (c == 0) {
            bag_of[u[q]] = make_int2(b, __float_as_int(so.weights ? scale * so.weights[i0 + q] : scale));
          }
        }
      }
    }
  }
}

// ------------------------------------------------------------------ lookup
// The id that marks a free slot is not available as a key; it is treated as its neighbour.
__device__ __forceinline__ uint64_t canonical_id(uint64_t id) { return id == kEmptyKey ? kEmptyKey - 1 : id; }

// Dedup without an exchange.  The scratch set holds 4-byte OCCURRENCE INDEXES instead of keys: entry h is the index of
// the occurrence that claimed it (the winner of its id), and a probe compares ids[entry].  What is accessed at random is
// then the set (4 bytes a slot) and the ids themselves, both of which stay in L2 at millions of ids, where the 16-byte
// {key, position} entries of the multi-rank dedup cost a sector of HBM each on the way in, at the number's read-back and
// at the clearing.  Measured for 3.4 M ids of which 2.3 M are distinct: insert + finalize + probe 260 us
// before, 185 us now; 1.7 M ids, 0.55 M distinct: 102 and 58 us.

// First kernel: every occurrence finds or claims its id's entry; the winner numbers the id.  first[i] = the winner's
// index for the others, ~entry for the winner itself; pos[i] = the number, written by winners only, like the unique list
// and win.  One id per thread:
// two or four were slower (3.4 M ids: 80, 85 and 107 us), the claims of a thread wait for one another.  The first look
// at an entry may be a stale one from L1, where the entries of frequent ids stay: an entry only ever goes from free to
// claimed within a launch, and a claim is made by compare-and-swap.
__global__ void __launch_bounds__(kThreads)
local_insert_kernel(const int64_t* __restrict__ ids, int n, int* set, uint32_t hbits, int* __restrict__ first,
                    int* __restrict__ pos, int* cnt, int64_t* __restrict__ uniq, int* __restrict__ win, int cap_u,
                    int* status) {
  pdl_enter();
  constexpr int kWarps = kThreads / 32;
  __shared__ int s_cnt[kWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x * kThreads + threadIdx.x;
  const uint32_t mask = static_cast<uint32_t>((1ull << hbits) - 1);
  bool won = false;
  uint64_t id = 0;
  if (i < n) {
    id = static_cast<uint64_t>(ids[i]);
    if (id == kEmptyKey) set_status(status, err::kBadArgument);  // reserved: reported, then treated as its neighbour
    id = canonical_id(id);
    uint32_t slot = static_cast<uint32_t>(SlotHash(id ^ kDedupSalt, hbits));
    int e = __ldca(&set[slot]);
    for (uint32_t probe = 0; probe <= mask; ++probe) {
      if (e < 0) {
        e = atomicCAS(&set[slot], -1, i);
        if (e < 0) {
          won = true;
          break;
        }
      }
      if (canonical_id(static_cast<uint64_t>(__ldg(ids + e))) == id) break;
      slot = (slot + 1) & mask;
      e = __ldca(&set[slot]);
    }
    first[i] = won ? static_cast<int>(~slot) : e;
  }
  const unsigned winners = __ballot_sync(0xffffffffu, won);
  if (lane == 0) s_cnt[warp] = __popc(winners);
  __syncthreads();
  if (threadIdx.x == 0) {
    int total = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const int c = s_cnt[w];
      s_cnt[w] = total;
      total += c;
    }
    const int start = total > 0 ? atomicAdd(cnt, total) : 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) s_cnt[w] += start;
  }
  __syncthreads();
  if (won) {
    const int u = s_cnt[warp] + __popc(winners & ((1u << lane) - 1u));
    pos[i] = u;
    if (u < cap_u) {
      uniq[u] = static_cast<int64_t>(id);
      win[u] = i;
    }
  }
}

// Rows that the warp's lanes have just created (bit set in `todo`, slot and id per lane), initialised by the whole
// warp: `lpr` lanes per row, so that the Philox draws and the stores of a row are spread over lanes.
template <int VEC>
__device__ __forceinline__ void init_created(const TableView& t, unsigned todo, int slot, uint64_t id, int chunks, int lpr) {
  const int lane = threadIdx.x & 31;
  const int rows_per_pass = 32 / lpr;
  while (todo) {
    int src = -1;
    for (int g = 0; g < rows_per_pass && todo; ++g) {
      const int l = __ffs(todo) - 1;
      todo &= todo - 1;
      if (g == lane / lpr) src = l;
    }
    const int r_slot = __shfl_sync(0xffffffffu, slot, src < 0 ? 0 : src);
    const uint64_t r_id = __shfl_sync(0xffffffffu, id, src < 0 ? 0 : src);
    if (src < 0) continue;
    float* row = t.val + static_cast<size_t>(r_slot) * t.pitch;
    for (int c = lane % lpr; c < chunks; c += lpr) {
      float q[4];
      if (VEC == 4) {
        InitQuad(t.init, t.seed_key, r_id, c, t.dim, q);
        *reinterpret_cast<float4*>(row + c * 4) = make_float4(q[0], q[1], q[2], q[3]);
      } else {
        InitQuad(t.init, t.seed_key, r_id, c >> 2, t.dim, q);
        row[c] = q[c & 3];
      }
    }
  }
}

// Second kernel, with the table probe: every occurrence learns its unique id's number, a winner empties its entry of the
// set, and thread u finds (or, with `insert`, claims and initialises) the row of unique id u.  The probe is the long chain
// of this kernel, a random access to HBM or more; as the winner's own work it held every warp with a winner among its lanes
// (nearly all of them, where a third of the occurrences win), over unique ids it is done by full warps and by no more of
// them than there are ids: 8.6 M ids, 3.2 M distinct, 211 us before and 167 us so; 3.4 M, 2.3 M distinct, 112 and 103 us.
// The block that finishes last zeroes `cnt` for the next call and counts the lookup.  The ids do not pass through the inbox,
// and no block ends on a system-scope fence.
template <int VEC>
__global__ void __launch_bounds__(kThreads)
local_resolve_kernel(int n, int* __restrict__ set, const int* __restrict__ first, const int* __restrict__ pos, int* cnt,
                     int* off, const int64_t* __restrict__ uniq, int* __restrict__ inv, int cap_u, TableView t, int* __restrict__ slot_cache, int cap_s, int insert,
                     uint32_t* epoch, uint32_t* done, int* status, int chunks, int lpr) {
  pdl_enter();
  const int U = *cnt;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    // more unique ids than the channel's buffers hold: reported and clamped, so that no later kernel indexes
    // past a buffer (the step's result is then invalid, not its memory)
    if (U > cap_u || U > cap_s) set_status(status, err::kInboxOverflow);
    off[0] = 0;
    off[1] = min(U, cap_u);
  }
  const int i = blockIdx.x * kThreads + threadIdx.x;
  bool created = false;
  int slot = -1;
  uint64_t id = 0;
  if (i < n) {
    const int f = first[i];
    const int u = pos[f < 0 ? i : f];
    inv[i] = u < cap_u ? u : 0;
    if (f < 0) set[~f] = -1;  // leave the set empty for the next call
  }
  if (i < min(U, min(cap_u, cap_s))) {
    id = static_cast<uint64_t>(uniq[i]);
    slot = table_find_or_insert(t, id, insert != 0, &created);
    if (slot < 0 && !insert) set_status(status, err::kSparseIdNotExist);
    slot_cache[i] = slot;
  }
  const unsigned todo = __ballot_sync(0xffffffffu, created);
  if (todo) {
    if ((threadIdx.x & 31) == __ffs(todo) - 1) atomicAdd(t.size, __popc(todo));
    init_created<VEC>(t, todo, slot, id, chunks, lpr);
  }
  __syncthreads();  // every thread of the block has read the count, so the last block to arrive may clear it
  if (threadIdx.x == 0) {
    if (atomicAdd(done, 1u) == gridDim.x - 1) {
      *done = 0;
      *cnt = 0;
      *epoch += 1;
    }
  }
}

// The lookup of unique ids that another channel has just deduplicated (the first-order table beside the embedding
// table): only the probe is left.
template <int VEC>
__global__ void __launch_bounds__(kThreads)
local_probe_kernel(const int64_t* __restrict__ uniq, const int* __restrict__ off, TableView t, int* __restrict__ slot_cache,
                   int cap_s, int insert, int* status, int chunks, int lpr) {
  pdl_enter();
  const int U = off[1];
  if (blockIdx.x == 0 && threadIdx.x == 0 && U > cap_s) set_status(status, err::kInboxOverflow);
  const int limit = min(U, cap_s);
  for (int base = blockIdx.x * blockDim.x; base < limit; base += gridDim.x * blockDim.x) {
    const int u = base + threadIdx.x;
    bool created = false;
    int slot = -1;
    uint64_t id = 0;
    if (u < limit) {
      id = static_cast<uint64_t>(uniq[u]);
      slot = table_find_or_insert(t, id, insert != 0, &created);
      if (slot < 0 && !insert) set_status(status, err::kSparseIdNotExist);
      slot_cache[u] = slot;
    }
    const unsigned todo = __ballot_sync(0xffffffffu, created);
    if (todo) {
      if ((threadIdx.x & 31) == __ffs(todo) - 1) atomicAdd(t.size, __popc(todo));
      init_created<VEC>(t, todo, slot, id, chunks, lpr);
    }
  }
}

// Row of unique entry u: its slot in the table, or -1 for one that was not found (its row reads as zeros).
__device__ __forceinline__ int slot_at(const int* __restrict__ slot_cache, int u, int cap_s) {
  return u < cap_s ? slot_cache[u] : -1;
}

// Unique rows into a compact buffer, for consumers that visit every occurrence of small rows (the DeepFM pack
// kernels): `tpr` threads per row, four rows of a thread in flight.
template <int VEC>
__global__ void __launch_bounds__(kThreads)
local_gather_kernel(TableView t, const int* __restrict__ off, const int* __restrict__ slot_cache, int cap_s, int chunks,
                    int tpr, float* __restrict__ rows_out) {
  pdl_enter();
  using V = Vec<VEC>;
  constexpr int kUnroll = 4;
  const int U = off[1];
  const int rows = kThreads / tpr;
  const int r = threadIdx.x / tpr, c0 = threadIdx.x - r * tpr;
  if (r >= rows) return;
  const int stride = gridDim.x * rows;
  for (int u0 = blockIdx.x * rows + r; u0 < U; u0 += stride * kUnroll) {
    int slot[kUnroll];
#pragma unroll
    for (int q = 0; q < kUnroll; ++q) slot[q] = u0 + q * stride < U ? slot_at(slot_cache, u0 + q * stride, cap_s) : -1;
    for (int c = c0; c < chunks; c += tpr) {
      typename V::T v[kUnroll];
#pragma unroll
      for (int q = 0; q < kUnroll; ++q)
        v[q] = slot[q] < 0 ? V::zero() : V::ld(t.val + static_cast<size_t>(slot[q]) * t.pitch + c * VEC);
#pragma unroll
      for (int q = 0; q < kUnroll; ++q)
        if (u0 + q * stride < U) V::st(rows_out + static_cast<size_t>(u0 + q * stride) * t.dim + c * VEC, v[q]);
    }
  }
}

// out[i] = row of occurrence i, read from the table where it is.
template <int VEC>
__global__ void __launch_bounds__(kThreads)
local_expand_kernel(TableView t, const int* __restrict__ inv, const int* __restrict__ slot_cache, int cap_s, int n,
                    int chunks, int tpr, float* __restrict__ out) {
  pdl_enter();
  using V = Vec<VEC>;
  constexpr int kUnroll = 4;
  const int rows = kThreads / tpr;
  const int r = threadIdx.x / tpr, c0 = threadIdx.x - r * tpr;
  if (r >= rows) return;
  const int stride = gridDim.x * rows;
  for (int i0 = blockIdx.x * rows + r; i0 < n; i0 += stride * kUnroll) {
    int slot[kUnroll];
#pragma unroll
    for (int q = 0; q < kUnroll; ++q) slot[q] = i0 + q * stride < n ? inv[i0 + q * stride] : -1;
#pragma unroll
    for (int q = 0; q < kUnroll; ++q) slot[q] = slot[q] < 0 ? -1 : slot_at(slot_cache, slot[q], cap_s);
    for (int c = c0; c < chunks; c += tpr) {
      typename V::T v[kUnroll];
#pragma unroll
      for (int q = 0; q < kUnroll; ++q)
        v[q] = slot[q] < 0 ? V::zero() : V::ld(t.val + static_cast<size_t>(slot[q]) * t.pitch + c * VEC);
#pragma unroll
      for (int q = 0; q < kUnroll; ++q)
        if (i0 + q * stride < n) V::st(out + static_cast<size_t>(i0 + q * stride) * t.dim + c * VEC, v[q]);
    }
  }
}

// out[b] = pooled rows of bag b, read from the table where they are; four rows of a bag in flight per thread.  The
// sum runs in the order of the occurrences, as in pull_combine_kernel.  What it waits for is rows, so six blocks of it
// are resident; five were a quarter slower (8.6 M rows of 64 floats: 305 and 392 us).
//
// INPUT: the pooled rows go out as what the first layer of an MLP reads (`in`), rounded here as its own conversion would
// round them; the threads of a sample's last field also write its dense features and the zeros behind them.
template <int VEC, bool INPUT>
__global__ void __launch_bounds__(kThreads, VEC == 4 ? 6 : 8)
local_pool_kernel(TableView t, const int* __restrict__ inv, const int* __restrict__ slot_cache, int cap_s, int chunks,
                  int tpr, const int64_t* __restrict__ bag_offsets, int nbags, const float* __restrict__ weights, int mean,
                  const uint8_t* __restrict__ bag_mean, float patch_value, float* __restrict__ out, PooledInput in) {
  pdl_enter();
  using V = Vec<VEC>;
  constexpr int kUnroll = 4;
  const int rows = kThreads / tpr;
  const int g = threadIdx.x / tpr, c0 = threadIdx.x - g * tpr;
  if (g >= rows) return;
  for (int b = blockIdx.x * rows + g; b < nbags; b += gridDim.x * rows) {
    const int lo = static_cast<int>(bag_offsets[b]), hi = static_cast<int>(bag_offsets[b + 1]);  // ids of a call: an int
    const bool is_mean = bag_mean ? bag_mean[b] != 0 : mean != 0;
    for (int c = c0; c < chunks; c += tpr) {
      typename V::T acc = V::zero();
      for (int r = lo; r < hi; r += kUnroll) {
        int slot[kUnroll];
        typename V::T v[kUnroll];
#pragma unroll
        for (int q = 0; q < kUnroll; ++q) slot[q] = r + q < hi ? inv[r + q] : -1;
#pragma unroll
        for (int q = 0; q < kUnroll; ++q) slot[q] = slot[q] < 0 ? -1 : slot_at(slot_cache, slot[q], cap_s);
#pragma unroll
        for (int q = 0; q < kUnroll; ++q)
          v[q] = slot[q] < 0 ? V::zero() : V::ld(t.val + static_cast<size_t>(slot[q]) * t.pitch + c * VEC);
#pragma unroll
        for (int q = 0; q < kUnroll; ++q)
          if (r + q < hi) V::fma(acc, weights ? weights[r + q] : 1.f, v[q]);
      }
      if (hi <= lo)
        acc = V::fill(patch_value);
      else if (is_mean)
        acc = V::scale(acc, 1.f / static_cast<float>(hi - lo));
      if constexpr (INPUT) {
        const int sample = b / in.fields;
        const __nv_bfloat162 lo2 = __floats2bfloat162_rn(acc.x, acc.y), hi2 = __floats2bfloat162_rn(acc.z, acc.w);
        uint2 packed;
        packed.x = *reinterpret_cast<const uint32_t*>(&lo2);
        packed.y = *reinterpret_cast<const uint32_t*>(&hi2);
        *reinterpret_cast<uint2*>(in.x + static_cast<size_t>(sample) * in.ldx + (b - sample * in.fields) * t.dim + c * VEC) =
            packed;
      } else {
        V::st(out + static_cast<size_t>(b) * t.dim + c * VEC, acc);
      }
    }
    if (INPUT && b % in.fields == in.fields - 1) {
      const int sample = b / in.fields, base = in.fields * t.dim;
      for (int j = c0; base + j < in.ldx; j += tpr)
        in.x[static_cast<size_t>(sample) * in.ldx + base + j] =
            __float2bfloat16(j < in.nd ? in.dense[static_cast<size_t>(sample) * in.nd + j] : 0.f);
    }
  }
}

}  // namespace

void local_lookup(const int64_t* ids, int n, LocalScratch sc, int* cnt, int* off, int64_t* uniq, int* inv, int cap_u,
                  TableHost table, int* slot_cache, int cap_s, bool insert, Ctrl* ctrl, cudaStream_t stream) {
  if (n <= 0) {
    cudaMemsetAsync(off, 0, 2 * sizeof(int), stream);
    return;
  }
  const RowGeom g = row_geom(table.dim);
  const dim3 grid((n + kThreads - 1) / kThreads);
  const bool early = grid.x < kFullGrid;
  launch_pdl_if(early, local_insert_kernel, grid, dim3(kThreads), 0, stream, ids, n, sc.set, sc.hbits, sc.first, sc.pos, cnt,
                uniq, sc.win, cap_u, &ctrl->status);
  auto kernel = g.vec == 4 ? local_resolve_kernel<4> : local_resolve_kernel<1>;
  launch_pdl_if(early, kernel, grid, dim3(kThreads), 0, stream, n, sc.set, static_cast<const int*>(sc.first),
                static_cast<const int*>(sc.pos), cnt, off, static_cast<const int64_t*>(uniq), inv, cap_u, to_view(table), slot_cache, cap_s,
                insert ? 1 : 0, &ctrl->pull_epoch, &ctrl->done[0], &ctrl->status, g.chunks, g.lpr);
}

void local_probe(const int64_t* uniq, const int* off, int max_n, TableHost table, int* slot_cache, int cap_s, bool insert,
                 Ctrl* ctrl, cudaStream_t stream) {
  const RowGeom g = row_geom(table.dim);
  const int grid = grid_for(max_n);
  auto kernel = g.vec == 4 ? local_probe_kernel<4> : local_probe_kernel<1>;
  launch_pdl_if(grid < kFullGrid, kernel, dim3(grid), dim3(kThreads), 0, stream, uniq, off, to_view(table), slot_cache,
                cap_s, insert ? 1 : 0, &ctrl->status, g.chunks, g.lpr);
}

void local_gather(TableHost table, const int* off, const int* slot_cache, int max_n, int cap_s, float* rows_out,
                  cudaStream_t stream) {
  const RowGeom g = row_geom(table.dim);
  const int tpr = g.chunks < kThreads ? g.chunks : kThreads;
  const int grid = grid_for(max_n, kThreads / tpr);
  auto kernel = g.vec == 4 ? local_gather_kernel<4> : local_gather_kernel<1>;
  launch_pdl_if(grid < kFullGrid, kernel, dim3(grid), dim3(kThreads), 0, stream, to_view(table), off, slot_cache, cap_s,
                g.chunks, tpr, rows_out);
}

void local_combine(TableHost table, const int* inv, const int* slot_cache, int n, int cap_s, const int64_t* bag_offsets,
                   int k, const float* weights, bool mean, const uint8_t* bag_mean, float patch_value, float* out,
                   cudaStream_t stream) {
  const RowGeom g = row_geom(table.dim);
  const int tpr = g.chunks < kThreads ? g.chunks : kThreads;
  const int grid = grid_for(bag_offsets ? k : n, kThreads / tpr, 148 * 16);
  if ((bag_offsets ? k : n) <= 0) return;
  const bool early = grid < kFullGrid;
  if (bag_offsets == nullptr) {
    auto kernel = g.vec == 4 ? local_expand_kernel<4> : local_expand_kernel<1>;
    launch_pdl_if(early, kernel, dim3(grid), dim3(kThreads), 0, stream, to_view(table), inv, slot_cache, cap_s, n, g.chunks,
                  tpr, out);
  } else {
    auto kernel = g.vec == 4 ? local_pool_kernel<4, false> : local_pool_kernel<1, false>;
    launch_pdl_if(early, kernel, dim3(grid), dim3(kThreads), 0, stream, to_view(table), inv, slot_cache, cap_s, g.chunks, tpr,
                  bag_offsets, k, weights, mean ? 1 : 0, bag_mean, patch_value, out, PooledInput{});
  }
}

void local_combine_input(TableHost table, const int* inv, const int* slot_cache, int cap_s, const int64_t* bag_offsets, int k,
                         const uint8_t* bag_mean, float patch_value, const PooledInput& in, cudaStream_t stream) {
  if (k <= 0) return;
  const RowGeom g = row_geom(table.dim);
  const int tpr = g.chunks < kThreads ? g.chunks : kThreads;
  const int grid = grid_for(k, kThreads / tpr, 148 * 16);
  launch_pdl_if(grid < kFullGrid, local_pool_kernel<4, true>, dim3(grid), dim3(kThreads), 0, stream, to_view(table), inv,
                slot_cache, cap_s, g.chunks, tpr, bag_offsets, k, static_cast<const float*>(nullptr), 0, bag_mean,
                patch_value, static_cast<float*>(nullptr), in);
}

namespace {
template <int FROM>
void update_all(TableHost table, float* ugrad, const int* off, const int* slot_cache, const DirectSource& so, int max_n,
                int cap_s, OptimPOD optim, const float* lr, cudaStream_t stream) {
  const RowGeom g = row_geom(table.dim);
  const int tpr = g.chunks < kUpdateThreads ? g.chunks : kUpdateThreads;
  const int grid = grid_for(max_n, kUpdateThreads / tpr, 148 * 80);
  const TableView t = to_view(table);
  if (FROM == kFromBags16 || g.vec == 4)
    launch_local_update<4, FROM>(grid, stream, t, ugrad, off, slot_cache, so, optim, lr, cap_s, g.chunks, tpr);
  else
    launch_local_update<FROM == kFromBags16 ? 4 : 1, FROM>(grid, stream, t, ugrad, off, slot_cache, so, optim, lr, cap_s, g.chunks, tpr);
}
}  // namespace

void local_push_update(TableHost table, float* ugrad, const int* off, const int* slot_cache, int max_n, int cap_s,
                       OptimPOD optim, const float* lr, cudaStream_t stream) {
  update_all<kFromSum>(table, ugrad, off, slot_cache, DirectSource{}, max_n, cap_s, optim, lr, stream);
}

void local_push(TableHost table, const LocalPush& p, float* ugrad, const int* off, const int* slot_cache, int n, int cap_s,
                OptimPOD optim, const float* lr, cudaStream_t stream) {
  if (n <= 0) return;
  const bool bags = p.bag_offsets != nullptr;
  if (table.dim < kDirectDim) {
    push_scatter(p.grads, p.inv, n, table.dim, p.bag_offsets, p.nbags, p.weights, p.mean, p.bag_mean, ugrad, stream);
    update_all<kFromSum>(table, ugrad, off, slot_cache, DirectSource{}, n, cap_s, optim, lr, stream);
    return;
  }
  DirectSource so{};
  so.grads = p.grads, so.grads16 = p.grads16, so.ld16 = p.ld16, so.fields = p.fields;
  so.bag_offsets = p.bag_offsets, so.nbags = p.nbags;
  so.weights = p.weights, so.bag_mean = p.bag_mean, so.mean = p.mean ? 1 : 0;
  so.win = p.win, so.multi = p.multi, so.epoch = &p.lookup->pull_epoch;
  so.bag_of = reinterpret_cast<const int2*>(p.bag_of);
  const RowGeom g = row_geom(table.dim);
  const int tpr = g.chunks < kThreads ? g.chunks : kThreads;
  const int grid = grid_for(bags ? p.nbags : n, kThreads / tpr, 148 * 16);
  if (bags) {
    auto kernel = p.grads16 != nullptr ? local_bag_scatter_kernel<4, true>
                  : g.vec == 4         ? local_bag_scatter_kernel<4, false>
                                       : local_bag_scatter_kernel<1, false>;
    if (p.nbags > 0)
      launch_pdl_if(grid < kFullGrid, kernel, dim3(grid), dim3(kThreads), 0, stream, p.inv, p.first, so, p.multi,
                    reinterpret_cast<int2*>(p.bag_of), n, p.nbags, table.dim, g.chunks, tpr, ugrad);
  } else {
    auto kernel = g.vec == 4 ? local_scatter_kernel<4> : local_scatter_kernel<1>;
    launch_pdl_if(grid < kFullGrid, kernel, dim3(grid), dim3(kThreads), 0, stream, p.inv, p.first, so, p.multi, n, table.dim,
                  g.chunks, tpr, ugrad);
  }
  if (p.grads16 != nullptr)
    update_all<kFromBags16>(table, ugrad, off, slot_cache, so, n, cap_s, optim, lr, stream);
  else if (bags)
    update_all<kFromBags>(table, ugrad, off, slot_cache, so, n, cap_s, optim, lr, stream);
  else
    update_all<kFromRows>(table, ugrad, off, slot_cache, so, n, cap_s, optim, lr, stream);
}

}  // namespace cu
}  // namespace kb
