// Exact merging of identical rows between plain layers (SNICIT mode).
//
// Every row is computed independently of the others, in a fixed FP32 order
// (the same slots, the same FMA sequence, whatever tile or kernel instance
// holds it), so two rows that are bitwise equal after layer l stay bitwise
// equal through every later layer and end in the same category.  On the SDGC
// workloads the surviving rows collapse onto a handful of fixed points well
// before the threshold layer; SNICIT's clustering finds them at the threshold
// (zero residues), this step finds them as soon as they appear and drops all
// but one copy from the row list, with no approximation:
//
//  1. dedup_hash_kernel: a team of 1, 4 or 16 warps per listed row (by width)
//     hashes the row's bits (two 32-bit streams, fixed thread order) and
//     inserts the key into an open-addressed table (linear probing with
//     atomicCAS; the table has at least twice as many entries as rows, so a
//     probe always ends); the smallest row id per key wins the slot
//     (atomicMin), which makes the kept row -- and so everything downstream --
//     independent of thread timing.  Keys and winners carry the merge step's
//     number, so what earlier steps left counts as empty and the table is
//     cleared once per inference;
//  2. dedup_verify_kernel: a row whose slot names another row compares the
//     two rows bit for bit; equal -> alias[r] = that row and r leaves the
//     list; unequal (a hash collision) -> r stays.  The rows that stay go to
//     the next layer's list, one atomic per 16 rows or fewer.
//
// Both wait for memory: a merge of a few rows is two round trips over a row.
// A whole merge step (us, in the stream of an inference): 160 rows of 65536
// neurons 80 with one warp per row and three launches -> 19; one row of 1024
// neurons 9 -> 6.
//
// At the end of the inference resolve_alias_kernel points every merged row at
// the root of its chain and copies the root's category; activations and head
// outputs of merged rows are read through alias (materialize, head).
#include <cstdint>

#include "sdnn_internal.h"

namespace sdnn {

namespace {

// MurmurHash3's 32-bit finaliser (Appleby, public domain).
__device__ __forceinline__ uint32_t fmix32(uint32_t h) {
  h ^= h >> 16;
  h *= 0x85EBCA6Bu;
  h ^= h >> 13;
  h *= 0xC2B2AE35u;
  h ^= h >> 16;
  return h;
}

__device__ __forceinline__ void mix_in(uint32_t& h1, uint32_t& h2, uint32_t v) {
  h1 = (h1 ^ v) * 0x9E3779B1u;
  h2 = (h2 + v) * 0x85EBCA77u;
  h2 ^= h2 >> 15;
}

constexpr int kDedupWarps = 16;

template <int TEAM>
__global__ void __launch_bounds__(kDedupWarps * 32) dedup_hash_kernel(const DedupArgs a) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  constexpr int kRows = kDedupWarps / TEAM;  // rows of a block at a time
  constexpr int kThreads = TEAM * 32;        // of a row
  __shared__ uint2 s_h[kDedupWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int team = warp / TEAM, me = threadIdx.x % kThreads;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int n = *a.count_in;
  if (n <= 1) return;  // nothing to merge: no slot is looked at
  const uint32_t mask = dedup_table_mask(*a.nrows, a.mask);
  const bool vec = (a.N & 3) == 0;
  for (int base = blockIdx.x * kRows; base < n; base += gridDim.x * kRows) {
    const int i = base + team;
    uint32_t h1 = 0x243F6A88u, h2 = 0xB7E15162u;
    const int r = i < n ? a.list_in[i] : -1;
    if (r >= 0) {
      const float* row = a.y + (size_t)r * a.N;
      if (vec) {
        // eight 16-byte loads in flight per thread, then the mixing
        const uint4* p = reinterpret_cast<const uint4*>(row);
        const int n4 = a.N >> 2;
        int j = me;
        for (; j + 7 * kThreads < n4; j += 8 * kThreads) {
          uint4 v[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) v[k] = __ldcg(p + j + k * kThreads);
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            mix_in(h1, h2, v[k].x);
            mix_in(h1, h2, v[k].y);
            mix_in(h1, h2, v[k].z);
            mix_in(h1, h2, v[k].w);
          }
        }
        for (; j < n4; j += kThreads) {
          const uint4 v = __ldcg(p + j);
          mix_in(h1, h2, v.x);
          mix_in(h1, h2, v.y);
          mix_in(h1, h2, v.z);
          mix_in(h1, h2, v.w);
        }
      } else {
        const uint32_t* p = reinterpret_cast<const uint32_t*>(row);
        for (int j = me; j < a.N; j += kThreads) mix_in(h1, h2, __ldcg(p + j));
      }
    }
    uint32_t v1 = fmix32(h1 + (uint32_t)me * 0x27D4EB2Fu);
    uint32_t v2 = fmix32(h2 ^ ((uint32_t)me * 0x165667B1u + 1u));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      v1 ^= __shfl_xor_sync(0xffffffffu, v1, o);
      v2 ^= __shfl_xor_sync(0xffffffffu, v2, o);
    }
    if constexpr (TEAM > 1) {
      if (lane == 0) s_h[warp] = make_uint2(v1, v2);
      __syncthreads();
      if (me == 0) {
#pragma unroll
        for (int w = 1; w < TEAM; ++w) {
          v1 ^= s_h[warp + w].x;
          v2 ^= s_h[warp + w].y;
        }
      }
      __syncthreads();
    }
    if (me == 0 && r >= 0) {
      const unsigned long long step = (unsigned long long)(a.step & 0x7fff) + 1ull;
      const unsigned long long key =
          (step << 48) | ((unsigned long long)(v1 & 0xffffu) << 32) | v2;
      uint32_t slot = (v2 ^ (v1 << 7)) & mask;
      // at most mask + 1 probes; the table holds >= 2x the listed rows
      for (uint32_t probe = 0; probe <= mask; ++probe) {
        unsigned long long cur = __ldcg(a.table + slot);
        while ((cur >> 48) != step) {  // empty, or left by an earlier step
          const unsigned long long old = atomicCAS(a.table + slot, cur, key);
          cur = old == cur ? key : old;
        }
        if (cur == key) break;
        slot = (slot + 1u) & mask;
      }
      a.pos_slot[i] = (int32_t)slot;
      // a later step's value is smaller than any earlier one's
      const unsigned long long mine =
          ((unsigned long long)(0x7fffffffu - (uint32_t)a.step) << 32) | (uint32_t)r;
      atomicMin(a.slot_rep + slot, mine);
    }
  }
}

template <int TEAM>
__global__ void __launch_bounds__(kDedupWarps * 32) dedup_verify_kernel(const DedupArgs a) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  constexpr int kRows = kDedupWarps / TEAM;
  constexpr int kThreads = TEAM * 32;
  __shared__ int32_t s_diff[kRows], s_keep[kRows];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int team = warp / TEAM, me = threadIdx.x % kThreads;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int n = *a.count_in;
  const bool vec = (a.N & 3) == 0;
  for (int base = blockIdx.x * kRows; base < n; base += gridDim.x * kRows) {
    const int i = base + team;
    const int r = i < n ? a.list_in[i] : -1;
    const int rep =
        i < n && n > 1 ? (int)(uint32_t)__ldcg(a.slot_rep + __ldcg(a.pos_slot + i)) : r;
    if (me == 0) s_diff[team] = 0;
    __syncthreads();
    if (rep != r) {
      bool same = true;
      if (vec) {
        const uint4* p = reinterpret_cast<const uint4*>(a.y + (size_t)r * a.N);
        const uint4* q = reinterpret_cast<const uint4*>(a.y + (size_t)rep * a.N);
        const int n4 = a.N >> 2;
        int j = me;
        for (; j + 3 * kThreads < n4; j += 4 * kThreads) {
          uint4 u[4], v[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            u[k] = __ldcg(p + j + k * kThreads);
            v[k] = __ldcg(q + j + k * kThreads);
          }
#pragma unroll
          for (int k = 0; k < 4; ++k)
            same &= u[k].x == v[k].x && u[k].y == v[k].y && u[k].z == v[k].z && u[k].w == v[k].w;
        }
        for (; j < n4; j += kThreads) {
          const uint4 u = __ldcg(p + j), v = __ldcg(q + j);
          same &= u.x == v.x && u.y == v.y && u.z == v.z && u.w == v.w;
        }
      } else {
        const uint32_t* p = reinterpret_cast<const uint32_t*>(a.y + (size_t)r * a.N);
        const uint32_t* q = reinterpret_cast<const uint32_t*>(a.y + (size_t)rep * a.N);
        for (int j = me; j < a.N; j += kThreads) same &= __ldcg(p + j) == __ldcg(q + j);
      }
      if (!__all_sync(0xffffffffu, same) && lane == 0) s_diff[team] = 1;
    }
    __syncthreads();
    if (me == 0) {
      const bool merged = rep != r && !s_diff[team];
      if (merged) a.alias[r] = rep;
      s_keep[team] = i < n && !merged ? r : -1;
    }
    __syncthreads();
    if (warp == 0) {
      const int row = lane < kRows ? s_keep[lane] : -1;
      const uint32_t w = __ballot_sync(0xffffffffu, row >= 0);
      int at = 0;
      if (lane == 0 && w) at = atomicAdd(a.count_out, __popc(w));
      at = __shfl_sync(0xffffffffu, at, 0) + __popc(w & ((1u << lane) - 1u));
      if (row >= 0) a.list_out[at] = row;
    }
  }
}

__global__ void resolve_alias_kernel(const int32_t* nrows, int32_t* alias, int32_t* flags,
                                     int32_t max_depth) {
  pdl_prologue();
  const int n = *nrows;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    int x = alias[r];
    if (x < 0) continue;
    // chains only point at smaller row ids, one link per merge step
    for (int d = 0; d < max_depth; ++d) {
      const int y = alias[x];
      if (y < 0) break;
      x = y;
    }
    alias[r] = x;
    if (flags) flags[r] = flags[x];
  }
}

}  // namespace

cudaError_t launch_dedup(const DedupArgs& a, int num_sms, cudaStream_t s) {
  // a row's bytes over its team: 4 KB by one warp, 16 KB by 4, more by 16
  auto hash = a.N <= 2048   ? dedup_hash_kernel<1>
              : a.N <= 8192 ? dedup_hash_kernel<4>
                            : dedup_hash_kernel<16>;
  auto verify = a.N <= 2048   ? dedup_verify_kernel<1>
                : a.N <= 8192 ? dedup_verify_kernel<4>
                              : dedup_verify_kernel<16>;
  cudaError_t rc = launch_pdl(hash, num_sms * 4, kDedupWarps * 32, 0, s, a);
  if (rc == cudaSuccess) rc = launch_pdl(verify, num_sms * 4, kDedupWarps * 32, 0, s, a);
  return rc;
}

void launch_resolve_alias(const int32_t* nrows, int32_t* alias, int32_t* flags, int32_t max_depth,
                          cudaStream_t s) {
  launch_pdl(resolve_alias_kernel, 264, 256, 0, s, nrows, alias, flags, max_depth);
}

}  // namespace sdnn
