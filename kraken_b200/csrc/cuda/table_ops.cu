// Maintenance kernels of a hash-table shard: clear, bulk import (checkpoint
// load, rehash, resharding receive), lookup without insert, and filtered
// export (checkpoint save, rehash, resharding send, eviction).
//
// The reference walks its skip lists on the host for all of these
// (kraken/ps/ps.cc:60-118,236-333; kraken/checkpoint/checkpoint.cc:494-507,628-646);
// here a full-table scan is one pass over the key array at HBM speed.
#include "common.cuh"
#include "kernels.h"

namespace kb {
namespace cu {

namespace {

constexpr int kThreads = 256;

TableView to_view(const TableHost& h) {
  TableView t;
  t.keys = static_cast<unsigned long long*>(h.keys);
  t.val = h.val;
  for (int i = 0; i < 3; ++i) t.s[i] = h.s[i];
  t.steps = h.steps;
  t.lead = static_cast<unsigned long long*>(h.lead);
  t.size = h.size;
  t.status = h.status;
  t.bits = h.bits;
  t.dim = h.dim;
  t.pitch = h.pitch;
  t.step_pitch = h.step_pitch;
  t.init = h.init;
  t.seed_key = h.seed_key;
  return t;
}

// Records of `pitch` floats, zeros but for columns [at, at + dim) of each, which take `value`: one pass over the memory (8.6 GB
// in 1.4 ms).  Zeros first and then a strided fill of the accumulators took 3.3 ms.  Thread i takes every stride-th four
// floats; where in its record these start is carried along, a division for each would cost more than the store.
__global__ void __launch_bounds__(kThreads)
fill_records_kernel(float* __restrict__ records, long long floats, int pitch, int at, int dim, float value) {
  const long long stride = static_cast<long long>(gridDim.x) * kThreads * 4;
  const int advance = static_cast<int>(stride % pitch);
  long long i = (blockIdx.x * static_cast<long long>(kThreads) + threadIdx.x) * 4;
  int column = static_cast<int>(i % pitch);
  for (; i < floats; i += stride) {
    float v[4];
    int c = column;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      v[e] = static_cast<unsigned>(c - at) < static_cast<unsigned>(dim) ? value : 0.f;
      if (++c == pitch) c = 0;
    }
    if (i + 4 <= floats) {
      *reinterpret_cast<float4*>(records + i) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
      for (int e = 0; i + e < floats; ++e) records[i + e] = v[e];
    }
    column += advance;
    if (column >= pitch) column -= pitch;
  }
}

// Calls move(dst + j, src + j) for the floats of every lane's row (`mine`); the warp must be converged.  Rows go in
// turn to the groups of 8, 16 or 32 lanes that a warp is divided into.  600 k rows with one state, us to export and to
// import: of 64 floats 857 and 1666 with a thread a row, a sector for each float, 311 and 310 so; of 8 floats 160 and 109 with
// a thread a row, 212 and 125 with a warp a row, 146 and 83 so.
constexpr int kGroupRow = 8;

template <typename Move>
__device__ __forceinline__ void move_rows(bool mine, size_t dst, size_t src, int dim, Move move) {
  if (dim < kGroupRow) {
    if (mine)
      for (int j = 0; j < dim; ++j) move(dst + j, src + j);
    return;
  }
  const int lane = threadIdx.x & 31, group = dim < 16 ? 8 : dim < 32 ? 16 : 32;
  const int groups = 32 / group;
  unsigned left = __ballot_sync(0xffffffffu, mine);
  int rows = __popc(left);
  for (int k = lane / group; k > 0; --k) left &= left - 1;
  for (; rows > 0; rows -= groups) {
    const int l = left ? __ffs(left) - 1 : 0;
    const size_t d = __shfl_sync(0xffffffffu, dst, l), s = __shfl_sync(0xffffffffu, src, l);
    if (left)
      for (int j = lane & (group - 1); j < dim; j += group) move(d + j, s + j);
    for (int k = 0; k < groups; ++k) left &= left - 1;
  }
}

__global__ void table_clear_kernel(TableView t) {
  const uint64_t cap = 1ull << t.bits;
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < cap;
       i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    t.keys[i] = kEmptyKey;
    if (t.steps) t.steps[i * t.step_pitch] = 0;
    if (t.lead) t.lead[i] = 0;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *t.size = 0;
}

__global__ void table_import_kernel(TableView t, const int64_t* __restrict__ ids, const float* __restrict__ vals,
                                    const float* __restrict__ s0, const float* __restrict__ s1,
                                    const float* __restrict__ s2, const int* __restrict__ steps, int n) {
  const bool on0 = t.s[0] && s0, on1 = t.s[1] && s1, on2 = t.s[2] && s2;
  for (int base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
    const int i = base + threadIdx.x;
    bool created = false;
    int found = -1;
    if (i < n) {
      const uint64_t id = static_cast<uint64_t>(ids[i]);
      // find-or-claim without running the initializer: the row is overwritten below
      const uint64_t mask = (1ull << t.bits) - 1;
      uint64_t slot = SlotHash(id, t.bits);
      const uint32_t max_probe = t.bits >= 13 ? 8192u : (1u << t.bits);
      for (uint32_t p = 0; p < max_probe && found < 0; ++p) {
        const unsigned long long k = __ldcg(&t.keys[slot]);
        if (k == id) {
          found = static_cast<int>(slot);
        } else if (k == kEmptyKey) {
          const unsigned long long old = atomicCAS(&t.keys[slot], kEmptyKey, static_cast<unsigned long long>(id));
          if (old == kEmptyKey) {
            created = true;
            found = static_cast<int>(slot);
          } else if (old == id) {
            found = static_cast<int>(slot);
          }
        }
        if (found < 0) slot = (slot + 1) & mask;
      }
      if (found < 0)
        set_status(t.status, err::kTableFull);
      else if (t.steps && steps)
        t.steps[static_cast<size_t>(found) * t.step_pitch] = steps[i];
    }
    move_rows(found >= 0, static_cast<size_t>(found < 0 ? 0 : found) * t.pitch, static_cast<size_t>(i) * t.dim, t.dim,
              [&](size_t d, size_t s) {
                const float v = vals[s], a = on0 ? s0[s] : 0.f, b = on1 ? s1[s] : 0.f, c = on2 ? s2[s] : 0.f;
                t.val[d] = v;
                if (on0) t.s[0][d] = a;
                if (on1) t.s[1][d] = b;
                if (on2) t.s[2][d] = c;
              });
    count_created(t, created);
  }
}

__global__ void table_lookup_kernel(TableView t, const int64_t* __restrict__ ids, int n, float* rows, uint8_t* found) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  bool created;
  const int slot = table_find_or_insert(t, static_cast<uint64_t>(ids[i]), false, &created);
  found[i] = slot >= 0;
  for (int j = 0; j < t.dim; ++j)
    rows[static_cast<size_t>(i) * t.dim + j] = slot >= 0 ? t.val[static_cast<size_t>(slot) * t.pitch + j] : 0.f;
}

__global__ void table_export_kernel(TableView t, int filter_mode, uint64_t salt, int world, int rank, int min_steps,
                                    int64_t* out_ids, float* out_vals, float* out_s0, float* out_s1, float* out_s2,
                                    int* out_steps, int* out_count, int out_cap) {
  const uint64_t cap = 1ull << t.bits;
  const bool on0 = out_s0 && t.s[0], on1 = out_s1 && t.s[1], on2 = out_s2 && t.s[2];
  for (uint64_t base = blockIdx.x * static_cast<uint64_t>(blockDim.x); base < cap;
       base += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const uint64_t slot = base + threadIdx.x;
    bool take = false;
    unsigned long long k = kEmptyKey;
    if (slot < cap) {
      k = t.keys[slot];
      if (k != kEmptyKey) {
        switch (filter_mode) {
          case 1: take = static_cast<int>(OwnerOf(salt, k, world)) == rank; break;
          case 2: take = static_cast<int>(OwnerOf(salt, k, world)) != rank; break;
          case 3: take = t.steps ? t.steps[slot * t.step_pitch] >= min_steps : true; break;
          case 4: take = static_cast<int>(k % static_cast<unsigned long long>(world)) == rank; break;  // id % world == rank
          default: take = true;
        }
      }
    }
    // one atomic per warp, then lane-ranked positions
    const unsigned m = __ballot_sync(0xffffffffu, take);
    int warp_base = 0;
    const int lane = threadIdx.x & 31;
    if (m != 0 && lane == __ffs(m) - 1) warp_base = atomicAdd(out_count, __popc(m));
    warp_base = __shfl_sync(0xffffffffu, warp_base, m ? __ffs(m) - 1 : 0);
    const int pos = warp_base + __popc(m & ((1u << lane) - 1));
    const bool fits = take && pos < out_cap;
    if (fits) {
      out_ids[pos] = static_cast<int64_t>(k);
      if (out_steps) out_steps[pos] = t.steps ? t.steps[slot * t.step_pitch] : 0;
    }
    move_rows(fits, static_cast<size_t>(fits ? pos : 0) * t.dim, slot * t.pitch, t.dim, [&](size_t d, size_t s) {
      const float v = t.val[s], a = on0 ? t.s[0][s] : 0.f, b = on1 ? t.s[1][s] : 0.f, c = on2 ? t.s[2][s] : 0.f;
      out_vals[d] = v;
      if (on0) out_s0[d] = a;
      if (on1) out_s1[d] = b;
      if (on2) out_s2[d] = c;
    });
  }
}

__global__ void owner_of_kernel(const int64_t* __restrict__ ids, int n, uint64_t salt, int world, int* owners) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) owners[i] = static_cast<int>(OwnerOf(salt, static_cast<uint64_t>(ids[i]), world));
}

}  // namespace

void owner_of(const int64_t* ids, int n, uint64_t salt, int world, int* owners, cudaStream_t stream) {
  if (n <= 0) return;
  owner_of_kernel<<<(n + kThreads - 1) / kThreads, kThreads, 0, stream>>>(ids, n, salt, world, owners);
}

void fill_records(float* records, long long floats, int pitch, int at, int dim, float value, cudaStream_t stream) {
  if (floats <= 0) return;
  const long long blocks = (floats + 4 * kThreads - 1) / (4 * kThreads);
  fill_records_kernel<<<static_cast<unsigned>(blocks < 148 * 8 ? blocks : 148 * 8), kThreads, 0, stream>>>(records, floats,
                                                                                                       pitch, at, dim, value);
}

void table_clear(TableHost table, cudaStream_t stream) {
  table_clear_kernel<<<148 * 4, kThreads, 0, stream>>>(to_view(table));
}

void table_import(TableHost table, const int64_t* ids, const float* vals, const float* s0, const float* s1,
                  const float* s2, const int* steps, int n, cudaStream_t stream) {
  if (n <= 0) return;
  int grid = (n + kThreads - 1) / kThreads;
  if (grid > 148 * 8) grid = 148 * 8;
  table_import_kernel<<<grid, kThreads, 0, stream>>>(to_view(table), ids, vals, s0, s1, s2, steps, n);
}

void table_lookup(TableHost table, const int64_t* ids, int n, float* rows, uint8_t* found, cudaStream_t stream) {
  if (n <= 0) return;
  table_lookup_kernel<<<(n + kThreads - 1) / kThreads, kThreads, 0, stream>>>(to_view(table), ids, n, rows, found);
}

void table_export(TableHost table, int filter_mode, uint64_t salt, int world, int rank, int min_steps,
                  int64_t* out_ids, float* out_vals, float* out_s0, float* out_s1, float* out_s2, int* out_steps,
                  int* out_count, int out_cap, cudaStream_t stream) {
  cudaMemsetAsync(out_count, 0, sizeof(int), stream);
  table_export_kernel<<<148 * 8, kThreads, 0, stream>>>(to_view(table), filter_mode, salt, world, rank, min_steps,
                                                        out_ids, out_vals, out_s0, out_s1, out_s2, out_steps, out_count,
                                                        out_cap);
}

}  // namespace cu
}  // namespace kb
