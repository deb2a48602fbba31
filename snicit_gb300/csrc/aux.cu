// Row-list utilities, category identification, the SNICIT threshold stage
// (candidate pick, pruning, nearest-centroid residue conversion) and recovery.
#include <climits>
#include "sdnn_internal.h"

namespace sdnn {

__host__ __device__ inline uint64_t mix64(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

static int grid_for(long work, int per_block, int cap = 4096) {
  long g = (work + per_block - 1) / per_block;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return (int)g;
}

// ---------------------------------------------------------------- row lists

// Rows of the current inference come from a device scalar (set just before a
// captured graph is launched), so one graph serves every row count.
__global__ void set_scalar_kernel(int32_t* p, int32_t v) { *p = v; }
__global__ void set_rows_kernel(int32_t* p, int32_t rows, int32_t share) {
  p[0] = rows;
  p[1] = share;
}
void launch_set_rows(int32_t* p, int32_t rows, int32_t share, cudaStream_t s) {
  set_rows_kernel<<<1, 1, 0, s>>>(p, rows, share);
}
void launch_set_scalar(int32_t* p, int32_t v, cudaStream_t s) { set_scalar_kernel<<<1, 1, 0, s>>>(p, v); }

__global__ void post_choice_kernel(const PostChoiceArgs a, cudaGraphConditionalHandle h) {
  const int residues = *a.rcount + (a.scount ? *a.scount : 0), centroids = *a.ccount;
  int body = 0;
  if (!a.no_chain && residues == 0 && centroids >= 1) {
    int i = 0, kc = 1;
    while (kc < centroids) {
      kc *= 2;
      ++i;
    }
    if (i < 4) {
      // the cluster kernel where the rows fit shared memory, else the grid kernel
      if (centroids <= a.chain_cap && a.has_body[1 + 2 * i]) body = 1 + 2 * i;
      else if (centroids <= a.grid_cap && a.has_body[2 + 2 * i]) body = 2 + 2 * i;
    }
  }
  cudaGraphSetConditional(h, (unsigned)body);
  *a.choice = body;
}
void launch_post_choice(const PostChoiceArgs& a, cudaGraphConditionalHandle h, cudaStream_t s) {
  post_choice_kernel<<<1, 1, 0, s>>>(a, h);
}

__global__ void sum_piece_counts_kernel(const int32_t* pc, int pieces, int stride, int layers,
                                        int32_t* counts) {
  for (int l = threadIdx.x; l < layers; l += blockDim.x) {
    int32_t t = 0;
    for (int p = 0; p < pieces; ++p) t += pc[(size_t)p * stride + l];
    counts[l] = t;
  }
}
void launch_sum_piece_counts(const int32_t* piece_counts, int pieces, int stride, int layers,
                             int32_t* counts, cudaStream_t s) {
  sum_piece_counts_kernel<<<1, 256, 0, s>>>(piece_counts, pieces, stride, layers, counts);
}

__global__ void begin_kernel(const BeginArgs a) {
  const int n = *a.nrows;
  const int at = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  for (int i = at; i < n; i += stride) {
    a.list[i] = i;
#pragma unroll
    for (int k = 0; k < 5; ++k) a.zero[k][i] = 0;
    a.alias[i] = -1;
  }
  for (int i = at; i < a.counts_n; i += stride) a.counts[i] = i == 0 ? n : 0;
  for (int i = at; i < a.extra_n; i += stride) a.extra[i] = 0;
  if (a.tile_state)
    for (int i = at; i < (n + 31) / 32; i += stride) a.tile_state[i] = 0;
  if (a.mask) {
    const uint32_t mask = dedup_table_mask(n, a.mask);
    for (uint32_t i = at; i <= mask; i += stride) {
      a.table[i] = 0ull;
      a.slot_rep[i] = ~0ull;
    }
  }
}
void launch_begin(const BeginArgs& a, cudaStream_t s) { begin_kernel<<<264, 256, 0, s>>>(a); }

__global__ void copy_rows_kernel(const int32_t* nrows, const float4* src, float4* dst, int32_t n4) {
  const size_t total = (size_t)(*nrows) * (size_t)n4;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (size_t)gridDim.x * blockDim.x)
    dst[i] = src[i];
}
void launch_copy_rows(const int32_t* nrows, const float* src, float* dst, int32_t N, cudaStream_t s) {
  copy_rows_kernel<<<1024, 256, 0, s>>>(nrows, reinterpret_cast<const float4*>(src),
                                        reinterpret_cast<float4*>(dst), N / 4);
}

// A copy per batch and direction costs 4 us of the stream, however small, and
// the host's time to issue it, in which the GPU waits for the first layer: 7
// batches, 9000 rows of 4096 in all, 1114 us -> 1068 with one launch each way.
__device__ __forceinline__ int batch_of(const BatchTable& t, int row) {
  int lo = 0, hi = t.n - 1;  // the last batch that begins at or before the row
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (t.first[mid] <= row) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}
__global__ void __launch_bounds__(256) gather_batches_kernel(const __grid_constant__ BatchTable t,
                                                             float4* rows, int32_t n4) {
  // units of 1024 quads of one row
  const int per_row = (n4 + 1023) / 1024;
  const long first = (long)t.first[0] * per_row, end = (long)t.first[t.n] * per_row;
  for (long u = first + blockIdx.x; u < end; u += gridDim.x) {
    const int row = (int)(u / per_row), b = batch_of(t, row);
    const float4* src = reinterpret_cast<const float4*>(t.in[b]) + (size_t)(row - t.first[b]) * n4;
    float4* dst = rows + (size_t)row * n4;
    const int q0 = (int)(u % per_row) * 1024 + threadIdx.x;
    float4 v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (q0 + k * 256 < n4) v[k] = __ldcs(src + q0 + k * 256);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (q0 + k * 256 < n4) dst[q0 + k * 256] = v[k];
  }
}
__global__ void scatter_flags_kernel(const __grid_constant__ BatchTable t, const int32_t* flags) {
  for (int r = t.first[0] + blockIdx.x * blockDim.x + threadIdx.x; r < t.first[t.n];
       r += gridDim.x * blockDim.x) {
    const int b = batch_of(t, r);
    t.flags[b][r - t.first[b]] = flags[r];
  }
}
void launch_gather_batches(const BatchTable& t, float* rows, int32_t N, int num_sms, cudaStream_t s) {
  gather_batches_kernel<<<num_sms * 8, 256, 0, s>>>(t, reinterpret_cast<float4*>(rows), N / 4);
}
void launch_scatter_flags(const BatchTable& t, const int32_t* flags, cudaStream_t s) {
  scatter_flags_kernel<<<64, 256, 0, s>>>(t, flags);
}

// Whether any of at(0) .. at(N - 1) is positive (one warp; 8 loads of a lane in
// flight, ending with the round that finds one).
template <typename At>
__device__ __forceinline__ bool any_positive(int N, int lane, At at) {
  for (int j0 = 0; j0 < N; j0 += 256) {
    bool any = false;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int j = j0 + 32 * t + lane;
      if (j < N) any |= at(j) > 0.f;
    }
    if (__any_sync(0xffffffffu, any)) return true;
  }
  return false;
}

// identify (src/SDGC/utility.hpp:194-212): category = 1 if the row has an
// activation > 0.  (The reference sums the row with thrust::reduce and an int
// initial value; see the oracle for that variant.)  One warp per listed row.
__global__ void identify_kernel(const float* y, const int32_t* list,
                                const int32_t* count, int32_t N, int32_t* flags, int32_t* state) {
  pdl_prologue();
  const int n = *count;
  const int lane = threadIdx.x & 31;
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  for (int i = wid; i < n; i += nw) {
    const int r = list[i];
    const float* row = y + (size_t)r * N;
    const bool any = any_positive(N, lane, [&](int j) { return row[j]; });
    if (lane == 0) {
      flags[r] = any ? 1 : 0;
      state[r] = 1;
    }
  }
}
void launch_identify(const float* y, const int32_t* list, const int32_t* count, int32_t N,
                     int32_t* flags, int32_t* state, int num_sms, cudaStream_t s) {
  launch_pdl(identify_kernel, num_sms * 4, 256, 0, s, y, list, count, N, flags, state);
}

// ------------------------------------------------------- SNICIT threshold stage
//
// Reference: reduction + centroid_sel (src/SDGC/SNICIT/kernel.hpp:138-194),
// host y* compaction (src/SDGC/SNICIT/SNICIT.hpp:457-462), coarse_cluster
// (kernel.hpp:8-69) and the host ne_record -> rowsY pass (SNICIT.hpp:505-509).
// Differences, by design: candidates are a seeded pick of K live rows (the
// reference takes the first 32 rows of the batch); the 16 downsampling bins
// are disjoint N/16-neuron ranges for every N; the centroid pick and the
// residue list are built on the device.

constexpr int kHistBins = 4096;
constexpr int kCandCap = 2048;

__global__ void __launch_bounds__(1024) cand_select_kernel(ClusterArgs a) {
  pdl_prologue();
  __shared__ int hist[kHistBins];
  __shared__ unsigned long long skey[kCandCap];
  __shared__ int srow[kCandCap];
  __shared__ int s_cut, s_n;
  const int tid = threadIdx.x;
  const int n = *a.live_count;
  const int K = a.K;
  for (int i = tid; i < kHistBins; i += blockDim.x) hist[i] = 0;
  if (tid == 0) s_n = 0;
  __syncthreads();
  for (int i = tid; i < n; i += blockDim.x) {
    const uint64_t key = mix64(a.seed ^ mix64((uint64_t)a.live[i]));
    atomicAdd(&hist[key >> 52], 1);
  }
  __syncthreads();
  if (tid < 32) {
    // first bin whose cumulative count reaches K: lane i sums bins
    // [128 i, 128 i + 128), a warp scan finds the lane, that lane walks its bins
    constexpr int per = kHistBins / 32;
    int part = 0;
    for (int b = 0; b < per; ++b) part += hist[tid * per + b];
    int incl = part;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (tid >= o) incl += v;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, incl >= K);
    if (hit == 0u) {
      if (tid == 0) s_cut = kHistBins - 1;  // fewer live rows than K: all are candidates
    } else if (tid == __ffs(hit) - 1) {
      int cum = incl - part, cut = (tid + 1) * per - 1;
      for (int b = 0; b < per; ++b) {
        cum += hist[tid * per + b];
        if (cum >= K) {
          cut = tid * per + b;
          break;
        }
      }
      s_cut = cut;
    }
  }
  __syncthreads();
  for (int i = tid; i < n; i += blockDim.x) {
    const int r = a.live[i];
    const uint64_t key = mix64(a.seed ^ mix64((uint64_t)r));
    if ((int)(key >> 52) <= s_cut) {
      const int pos = atomicAdd(&s_n, 1);
      if (pos < kCandCap) {
        skey[pos] = key;
        srow[pos] = r;
      }
    }
  }
  __syncthreads();
  const int m = min(s_n, kCandCap);
  int M = 1;
  while (M < m) M <<= 1;
  for (int i = m + tid; i < M; i += blockDim.x) {
    skey[i] = ~0ull;
    srow[i] = INT_MAX;
  }
  __syncthreads();
  // bitonic sort on (key, row)
  for (int k = 2; k <= M; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = tid; i < M; i += blockDim.x) {
        const int ixj = i ^ j;
        if (ixj > i) {
          const bool up = (i & k) == 0;
          const unsigned long long ki = skey[i], kj = skey[ixj];
          const int ri = srow[i], rj = srow[ixj];
          const bool gt = (ki > kj) || (ki == kj && ri > rj);
          if (gt == up) {
            skey[i] = kj;
            skey[ixj] = ki;
            srow[i] = rj;
            srow[ixj] = ri;
          }
        }
      }
      __syncthreads();
    }
  }
  const int nc = min(K, m);
  for (int i = tid; i < nc; i += blockDim.x) a.cand[i] = srow[i];
  if (tid == 0) *a.ncand = nc;
}

// 16 disjoint bin sums per candidate; one warp per bin, fixed reduction order.
__global__ void cand_bins_kernel(ClusterArgs a) {
  pdl_prologue();
  const int k = blockIdx.x;
  if (k >= *a.ncand) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float* row = a.y + (size_t)a.cand[k] * a.N;
  const int w = a.N / 16;
  for (int b = warp; b < 16; b += blockDim.x >> 5) {
    float s = 0.f;
    for (int j = b * w + lane; j < (b + 1) * w; j += 32) s += row[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) a.bins[k * 16 + b] = s;
  }
}

// Greedy pruning (paper Alg. 1; centroid_sel, src/SDGC/SNICIT/kernel.hpp:156-194):
// candidate k is dropped when an earlier kept candidate has every one of the 16
// bins within 0.03 (the reference drops when fewer than 16*0.03 bins differ by
// more than 0.03, i.e. when none does).
__global__ void __launch_bounds__(256) prune_kernel(ClusterArgs a) {
  pdl_prologue();
  __shared__ int keep[256];
  __shared__ float sb[256 * 16];
  const int tid = threadIdx.x;
  const int nc = min(*a.ncand, 256);
  for (int i = tid; i < nc * 16; i += blockDim.x) sb[i] = a.bins[i];
  if (tid < nc) keep[tid] = 1;
  __syncthreads();
  for (int k = 1; k < nc; ++k) {
    bool similar = false;
    if (tid < k && keep[tid]) {
      similar = true;
      for (int b = 0; b < 16; ++b)
        if (fabsf(sb[k * 16 + b] - sb[tid * 16 + b]) > 0.03f) {
          similar = false;
          break;
        }
    }
    const int any = __syncthreads_or(similar);
    if (tid == 0 && any) keep[k] = 0;
    __syncthreads();
  }
  if (tid == 0) {
    int ci = 0;
    for (int k = 0; k < nc; ++k) {
      if (!keep[k]) continue;
      const int r = a.cand[k];
      a.clist[ci] = r;
      a.cslot[r] = ci;
      a.is_centroid[r] = 1;
      ++ci;
    }
    *a.ccount = ci;
  }
}

// Nearest centroid by L0 distance (count of differing entries), ties to the
// lowest centroid index, residue written in place: y[r] <- y[r] - c.  Rows at
// distance 0 get no residue and are left out of the residue list.
// One CTA per row, its warps taking the centroids in turn: with one warp per
// row 150 rows of 4096 neurons against 32 centroids took 244 us, 32 reads of a
// row one after the other; now 30.
constexpr int kAssignWarps = 8;
__global__ void __launch_bounds__(kAssignWarps * 32) assign_kernel(ClusterArgs a) {
  pdl_prologue();
  __shared__ unsigned long long s_best;  // (distance, centroid), the smallest so far
  const int n = *a.live_count;
  const int nc = *a.ccount;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int N = a.N;
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const int r = a.live[i];
    if (a.is_centroid[r]) continue;
    if (tid == 0) s_best = ((unsigned long long)INT_MAX << 32);
    __syncthreads();
    float* yr = a.y + (size_t)r * N;
    const float4* yr4 = reinterpret_cast<const float4*>(yr);
    for (int k = warp; k < nc; k += kAssignWarps) {
      const float4* yc4 = reinterpret_cast<const float4*>(a.y + (size_t)a.clist[k] * N);
      unsigned dt = 0;
      bool lost = false;
      // 1024 entries per step, all 16 loads of a lane in flight before the
      // comparisons; stop as soon as this centroid cannot be the nearest
      for (int j0 = 0; j0 < N; j0 += 1024) {
        const unsigned long long best = *(volatile unsigned long long*)&s_best;
        lost = (((unsigned long long)dt << 32) | (unsigned)k) > best;
        if (__any_sync(0xffffffffu, lost)) {
          lost = true;
          break;
        }
        float4 u[8], v[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          const int j = j0 + 128 * t + 4 * lane;
          u[t] = j < N ? yr4[j >> 2] : make_float4(0.f, 0.f, 0.f, 0.f);
          v[t] = j < N ? yc4[j >> 2] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        unsigned dl = 0;
#pragma unroll
        for (int t = 0; t < 8; ++t)
          dl += (u[t].x != v[t].x) + (u[t].y != v[t].y) + (u[t].z != v[t].z) + (u[t].w != v[t].w);
        dt += __reduce_add_sync(0xffffffffu, dl);
      }
      if (!lost && lane == 0) atomicMin(&s_best, ((unsigned long long)dt << 32) | (unsigned)k);
    }
    __syncthreads();
    const int best = (int)(s_best >> 32), bk = (int)(uint32_t)s_best;
    if (best > 0) {
      const float* yc = a.y + (size_t)a.clist[bk] * N;
      for (int j = tid; j < N; j += blockDim.x) yr[j] = yr[j] - yc[j];
    }
    if (tid == 0) {
      a.cslot[r] = bk;
      if (best > 0) a.rlist[atomicAdd(a.rcount, 1)] = r;
    }
    __syncthreads();
  }
}

void launch_cluster(const ClusterArgs& a, int num_sms, cudaStream_t s) {
  launch_pdl(cand_select_kernel, 1, 1024, 0, s, a);
  launch_pdl(cand_bins_kernel, a.K, 512, 0, s, a);
  launch_pdl(prune_kernel, 1, 256, 0, s, a);
  launch_pdl(assign_kernel, num_sms * 8, kAssignWarps * 32, 0, s, a);
}

// ------------------------------------------------------------------ recovery

// recover (src/SDGC/SNICIT/kernel.hpp:197-218): flags[r] = any((delta + c) > 0).
__global__ void recover_kernel(const float* y, const int32_t* live,
                               const int32_t* live_count, const int32_t* cslot,
                               const int32_t* clist, const int32_t* is_centroid,
                               const int32_t* res_flag, int32_t N, int32_t* flags,
                               int32_t* state) {
  pdl_prologue();
  const int n = *live_count;
  const int lane = threadIdx.x & 31;
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  for (int i = wid; i < n; i += nw) {
    const int r = live[i];
    const float* yr = y + (size_t)r * N;
    bool any;
    if (is_centroid[r]) {
      any = any_positive(N, lane, [&](int j) { return yr[j]; });
    } else {
      const float* yc = y + (size_t)clist[cslot[r]] * N;
      if (res_flag[r]) any = any_positive(N, lane, [&](int j) { return yr[j] + yc[j]; });
      else any = any_positive(N, lane, [&](int j) { return yc[j]; });
    }
    if (lane == 0) {
      flags[r] = any ? 1 : 0;
      state[r] = 2;
    }
  }
}
void launch_recover(const float* y, const int32_t* live, const int32_t* live_count,
                    const int32_t* cslot, const int32_t* clist, const int32_t* is_centroid,
                    const int32_t* res_flag, int32_t N, int32_t* flags, int32_t* state, int num_sms,
                    cudaStream_t s) {
  launch_pdl(recover_kernel, num_sms * 4, 256, 0, s, y, live, live_count, cslot, clist, is_centroid,
             res_flag, N, flags, state);
}

// Final activations per row, in neuron order (out[r][c] reads position perm[c]):
// state 0 -> zeros (dead), 1 -> copy of the final buffer (plain modes),
// 2 -> SNICIT recovery (centroid, or centroid + residue).
__global__ void materialize_kernel(const float* __restrict__ y, const int32_t* state,
                                   const int32_t* cslot, const int32_t* clist,
                                   const int32_t* is_centroid, const int32_t* res_flag,
                                   const int32_t* alias, const int32_t* perm, int32_t N,
                                   int32_t rows, float* out) {
  for (int ro = blockIdx.x; ro < rows; ro += gridDim.x) {
    float* o = out + (size_t)ro * N;
    const int r = alias && alias[ro] >= 0 ? alias[ro] : ro;
    const int st = state[r];
    const float* yr = y + (size_t)r * N;
    if (st == 0) {
      for (int j = threadIdx.x; j < N; j += blockDim.x) o[j] = 0.f;
      continue;
    }
    const bool plain = st == 1 || is_centroid[r];
    const float* yc = plain ? yr : y + (size_t)clist[cslot[r]] * N;
    const bool has_res = !plain && res_flag[r];
    for (int j = threadIdx.x; j < N; j += blockDim.x) {
      const int p = perm ? perm[j] : j;
      o[j] = plain ? yr[p] : (has_res ? yr[p] + yc[p] : yc[p]);
    }
  }
}

void launch_materialize(const float* y, const int32_t* state, const int32_t* cslot,
                        const int32_t* clist, const int32_t* is_centroid, const int32_t* res_flag,
                        const int32_t* alias, const int32_t* perm, int32_t N, float* out,
                        int32_t rows, cudaStream_t s) {
  materialize_kernel<<<grid_for(rows, 1, 8192), 256, 0, s>>>(y, state, cslot, clist, is_centroid,
                                                             res_flag, alias, perm, N, rows, out);
}

// Dense output head on the final activations (dense_output,
// src/beyond/general.hpp:74-102: logits = y . H + b, no activation), one warp
// per row, rows read the way materialize_kernel reads them (dead rows are
// zero, SNICIT rows are recovered).  Hp is the head stored by final position
// (Hp[p][k] = H[neuron at p][k]); lane-strided sums over positions, then a
// fixed xor-shuffle tree: deterministic.  argmax: first maximal logit.
template <int H>
__global__ void head_kernel(const float* __restrict__ y, const int32_t* state, const int32_t* cslot,
                            const int32_t* clist, const int32_t* is_centroid,
                            const int32_t* res_flag, const int32_t* alias,
                            const float* __restrict__ Hp, const float* __restrict__ hb, int32_t N,
                            int32_t rows, float* logits, int32_t* argmax) {
  const int lane = threadIdx.x & 31;
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  for (int ro = wid; ro < rows; ro += nw) {
    float acc[H];
#pragma unroll
    for (int k = 0; k < H; ++k) acc[k] = 0.f;
    const int r = alias && alias[ro] >= 0 ? alias[ro] : ro;
    const int st = state[r];
    if (st != 0) {
      const float* yr = y + (size_t)r * N;
      const bool plain = st == 1 || is_centroid[r];
      const float* yc = plain ? yr : y + (size_t)clist[cslot[r]] * N;
      const bool has_res = !plain && res_flag[r];
      for (int p = lane; p < N; p += 32) {
        const float v = plain ? yr[p] : (has_res ? yr[p] + yc[p] : yc[p]);
        if (v != 0.f) {
#pragma unroll
          for (int k = 0; k < H; ++k) acc[k] = fmaf(v, __ldg(Hp + (size_t)p * H + k), acc[k]);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < H; ++k) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
    }
    if (lane == 0) {
      int best = 0;
      float bv = 0.f;
#pragma unroll
      for (int k = 0; k < H; ++k) {
        const float v = acc[k] + hb[k];
        logits[(size_t)ro * H + k] = v;
        if (k == 0 || v > bv) {
          bv = v;
          best = k;
        }
      }
      argmax[ro] = best;
    }
  }
}

bool launch_head(const float* y, const int32_t* state, const int32_t* cslot, const int32_t* clist,
                 const int32_t* is_centroid, const int32_t* res_flag, const int32_t* alias,
                 const float* Hp, const float* hb, int32_t H, int32_t N, int32_t rows,
                 float* logits, int32_t* argmax, cudaStream_t s) {
  const int grid = grid_for(rows, 8, 2048);
#define SDNN_HEAD(K)                                                                           \
  case K:                                                                                     \
    head_kernel<K><<<grid, 256, 0, s>>>(y, state, cslot, clist, is_centroid, res_flag, alias, Hp, \
                                        hb, N, rows, logits, argmax);                         \
    return true;
  switch (H) {
    SDNN_HEAD(1)
    SDNN_HEAD(2)
    SDNN_HEAD(4)
    SDNN_HEAD(8)
    SDNN_HEAD(10)
    SDNN_HEAD(16)
    SDNN_HEAD(32)
    default: return false;
  }
#undef SDNN_HEAD
}

}  // namespace sdnn

namespace sdnn {

// One-bit input rows (entry j in bit j % 64 of word j / 64, ceil(N / 64) words
// per row) to FP32 0/1 rows; one thread writes four consecutive entries.
__global__ void expand_bits_kernel(const unsigned long long* __restrict__ bits, int64_t rows,
                                   int32_t N, float4* out) {
  const int32_t W = (N + 63) / 64, n4 = N / 4;
  const int64_t total = rows * n4;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / n4;
    const int32_t j = (int32_t)(i % n4) * 4;
    const unsigned long long w = __ldg(bits + r * W + (j >> 6));
    const uint32_t b = (uint32_t)(w >> (j & 63)) & 15u;
    out[i] = make_float4(b & 1u ? 1.f : 0.f, b & 2u ? 1.f : 0.f, b & 4u ? 1.f : 0.f,
                         b & 8u ? 1.f : 0.f);
  }
}

void launch_expand_bits(const uint64_t* bits, int64_t rows, int32_t N, float* out, cudaStream_t s) {
  expand_bits_kernel<<<4096, 256, 0, s>>>(reinterpret_cast<const unsigned long long*>(bits), rows,
                                          N, reinterpret_cast<float4*>(out));
}

}  // namespace sdnn
