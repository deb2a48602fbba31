// Sparse residue rows of the SNICIT post-threshold stage.
//
// After the threshold every live row is a centroid row or centroid + residue
// Delta (src/SDGC/SNICIT/kernel.hpp:8-69).  As rows saturate towards their
// centroid, Delta keeps only a few nonzeros; the reference's post_spMM then
// skips the zero entries of the residue (kernel.hpp:71-102, `if (val != 0)`),
// but its post_minus still walks every output (kernel.hpp:104-136).  Here a
// residue row with at most SC nonzeros (N/32, at least 32: a sparse row's
// scatter runs on one warp, so longer lists would stretch the layer) is kept as
// a sorted (position, value) list and its update touches only what it must:
//
//   split_residue_kernel   residue conversion: a CTA of 4 warps per dense
//                          residue row, each warp a quarter of it (with many
//                          rows a warp per row); the nonzeros are compacted
//                          into the row's list (ascending positions), or the
//                          row stays dense when it has more than SC of them;
//   sparse_residue_kernel  a CTA per sparse row: W * Delta by scattering each
//                          nonzero along its input's out-edges (the transposed
//                          layer, one edge per lane, entries in ascending
//                          order by one warp, so every output adds its terms in
//                          a fixed order: deterministic, no atomics on values)
//                          into a shared-memory row; then
//                          Delta' = f(pre_c + W Delta) - f(pre_c) by all warps
//                          (an output no entry reaches has W Delta = 0, so
//                          Delta' = 0 there exactly), 32 neighbouring outputs
//                          at a time, compacted again -- or written as a dense
//                          row when it grew past SC, or dropped from the lists
//                          when it is all zero (the row has converged to its
//                          centroid);
//   finish_rows_kernel     the final sparse rows written densely into the last
//                          layer's buffer, so recovery reads every residue row
//                          the same way, and every residue row marked.
//
// A layer has tens of such rows at most, so these wait for memory, row by row.
// With one warp per row, a bitmap of the outputs reached kept with shared
// atomics and each lane walking 32 outputs of its own (a load of pre_c, 32
// lines apart, per output), a layer of 30 sparse rows of 4096 neurons took 75 -
// 110 us; now 20.
#include "sdnn_internal.h"

namespace sdnn {
namespace {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ float clamp_hi(float v, float hi) { return fminf(hi, fmaxf(0.f, v)); }

constexpr int kRowWarps = 4;  // warps of a CTA that share a residue row
constexpr int kStage = kRowWarps * 32;   // entries whose edges are staged at a time
constexpr int kNoOutput = 0xffff;        // (rows here have at most 32768 outputs)

// Exclusive sum of the warps' counts before this one and the total; the
// caller's s_cnt is free again after the next barrier.
__device__ __forceinline__ int warps_before(const int* s_cnt, int warp, int& total) {
  int before = 0;
  total = 0;
#pragma unroll
  for (int w = 0; w < kRowWarps; ++w) {
    if (w < warp) before += s_cnt[w];
    total += s_cnt[w];
  }
  return before;
}

// Appends the nonzeros of 128 entries to a row's list, `base` of whose (at most
// `cap`) entries are taken, and returns how many are then.  Lane L holds entries
// j .. j + 3, j = j0 + 4 L; a lane's nonzeros go after those of the lanes below
// it, so the list comes out in ascending position.
__device__ __forceinline__ int append_nonzeros(float4 v, int j, int base, int cap, int32_t* oi,
                                               float* ov, int lane) {
  const float e[4] = {v.x, v.y, v.z, v.w};
  const int mine = (e[0] != 0.f) + (e[1] != 0.f) + (e[2] != 0.f) + (e[3] != 0.f);
  if (!__any_sync(kFull, mine != 0)) return base;
  int incl = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int u = __shfl_up_sync(kFull, incl, d);
    if (lane >= d) incl += u;
  }
  int k = base + incl - mine;
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    if (e[t] != 0.f) {
      if (k < cap) {
        oi[k] = j + t;
        ov[k] = e[t];
      }
      ++k;
    }
  }
  return base + __shfl_sync(kFull, incl, 31);
}

__global__ void __launch_bounds__(kRowWarps * 32)
    split_residue_kernel(const float* y, const int32_t* list, const int32_t* count, SparseRows out,
                         int32_t* dense_list, int32_t* dense_count, int32_t* sparse_list,
                         int32_t* sparse_count, int32_t N) {
  __shared__ int s_cnt[kRowWarps];
  pdl_prologue();
  const int n = *count;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int SC = out.cap;
  // the warp's part of a row, a multiple of 128 entries
  const int part = ((N + kRowWarps * 128 - 1) / (kRowWarps * 128)) * 128;
  const int j_begin = min(N, warp * part), j_end = min(N, j_begin + part);
  if (n > 4 * (int)gridDim.x) {
    // Many rows: most stay dense, and a row is decided once SC + 1 nonzeros are
    // seen, in its first few hundred entries.  So a warp per row, with no barrier
    // and no more of a dense row read than that (14 post layers of some 21000
    // residue rows of 1024 neurons 2.85 -> 2.47 ms).
    for (int i = blockIdx.x * kRowWarps + warp; i < n; i += gridDim.x * kRowWarps) {
      const int r = list[i];
      const float4* yr = reinterpret_cast<const float4*>(y + (size_t)r * N);
      int32_t* oi = out.idx + (size_t)r * SC;
      float* ov = out.val + (size_t)r * SC;
      int base = 0;
      for (int j0 = 0; j0 < N && base <= SC; j0 += 256) {
        float4 v[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int j = j0 + 128 * h + 4 * lane;
          v[h] = j < N ? yr[j >> 2] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
          base = append_nonzeros(v[h], j0 + 128 * h + 4 * lane, base, SC, oi, ov, lane);
      }
      if (lane == 0) {
        if (base <= SC) {
          out.cnt[r] = base;
          sparse_list[atomicAdd(sparse_count, 1)] = r;
        } else {
          dense_list[atomicAdd(dense_count, 1)] = r;
        }
      }
    }
    return;
  }
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const int r = list[i];
    const float4* yr = reinterpret_cast<const float4*>(y + (size_t)r * N);
    int nz = 0;
    for (int j0 = j_begin; j0 < j_end; j0 += 8 * 128) {
      float4 v[8];
#pragma unroll
      for (int h = 0; h < 8; ++h) {
        const int j = j0 + 128 * h + 4 * lane;
        v[h] = j < j_end ? yr[j >> 2] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int h = 0; h < 8; ++h)
        nz += (v[h].x != 0.f) + (v[h].y != 0.f) + (v[h].z != 0.f) + (v[h].w != 0.f);
    }
    nz = (int)__reduce_add_sync(kFull, (unsigned)nz);
    if (lane == 0) s_cnt[warp] = nz;
    __syncthreads();
    int total;
    int base = warps_before(s_cnt, warp, total);
    if (total <= SC) {
      int32_t* oi = out.idx + (size_t)r * SC;
      float* ov = out.val + (size_t)r * SC;
      for (int j0 = j_begin; j0 < j_end && nz > 0; j0 += 128) {
        const int j = j0 + 4 * lane;
        const float4 v = j < j_end ? yr[j >> 2] : make_float4(0.f, 0.f, 0.f, 0.f);
        base = append_nonzeros(v, j, base, SC, oi, ov, lane);
      }
    }
    if (threadIdx.x == 0) {
      if (total <= SC) {
        out.cnt[r] = total;
        sparse_list[atomicAdd(sparse_count, 1)] = r;
      } else {
        dense_list[atomicAdd(dense_count, 1)] = r;
      }
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kRowWarps * 32) sparse_residue_kernel(const SparseResArgs a) {
  extern __shared__ __align__(16) float acc[];  // [N]
  __shared__ int s_cnt[kRowWarps];
  __shared__ uint16_t s_out[kStage * 32];
  __shared__ float s_w[kStage * 32];
  __shared__ float s_v[kStage];
  __shared__ int s_t0[kStage], s_deg[kStage];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int N = a.N, nwords = N >> 5, SC = a.in.cap;
  pdl_prologue();
  const int n = *a.count_in;
  if ((int)blockIdx.x >= n) return;  // no row for this CTA (often no row at all)
  for (int j = tid; j < N; j += blockDim.x) acc[j] = 0.f;
  __syncthreads();
  const float hi = a.clampv;
  // the warp's part of the outputs, in groups of 32
  const int part = (nwords + kRowWarps - 1) / kRowWarps;
  const int w_begin = min(nwords, warp * part), w_end = min(nwords, w_begin + part);
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const int r = a.list_in[i];
    const int cnt = a.in.cnt[r];
    const int32_t* ei = a.in.idx + (size_t)r * SC;
    const float* ev = a.in.val + (size_t)r * SC;
    // W * Delta: entries in ascending position, each along its out-edges.  All
    // warps fetch the entries' edges into shared memory, 128 entries at a time
    // (a chain of three loads, 32 entries of a warp in flight), then one warp
    // applies them in entry order.
    for (int c0 = 0; c0 < cnt; c0 += kStage) {
      const int ne = min(kStage, cnt - c0);
      const int e = warp * 32 + lane;
      int t0 = 0, deg = 0;
      if (e < ne) {
        const int j = ei[c0 + e];
        s_v[e] = ev[c0 + e];
        t0 = __ldg(a.tr_off + j);
        deg = __ldg(a.tr_off + j + 1) - t0;
        s_t0[e] = t0;
        s_deg[e] = deg;
      }
#pragma unroll 8
      for (int u = 0; u < 32; ++u) {
        const int tu = __shfl_sync(kFull, t0, u), du = __shfl_sync(kFull, deg, u);
        const int at = (warp * 32 + u) * 32 + lane;
        s_out[at] = lane < du ? __ldg(a.tr_out + tu + lane) : kNoOutput;
        if (a.tr_val && lane < du) s_w[at] = __ldg(a.tr_val + tu + lane);
      }
      __syncthreads();
      if (warp == 0) {
#pragma unroll 4
        for (int k = 0; k < ne; ++k) {
          const int o = s_out[k * 32 + lane];
          const float v = s_v[k];
          const float w = a.tr_val ? s_w[k * 32 + lane] : a.wconst;
          if (o != kNoOutput) acc[o] = fmaf(w, v, acc[o]);
          // out-degrees above 32 (general layers): the rest of the edges
          for (int t = s_t0[k] + 32 + lane; t < s_t0[k] + s_deg[k]; t += 32) {
            const int oo = __ldg(a.tr_out + t);
            const float ww = a.tr_val ? __ldg(a.tr_val + t) : a.wconst;
            acc[oo] = fmaf(ww, v, acc[oo]);
          }
          __syncwarp();
        }
      }
      __syncthreads();
    }
    const float* pre = a.pre + (size_t)a.cslot[r] * N;
    __syncthreads();
    // Delta' into acc
    int nz = 0;
    for (int w0 = w_begin; w0 < w_end; w0 += 8) {
      float pc[8];
#pragma unroll
      for (int h = 0; h < 8; ++h) pc[h] = w0 + h < w_end ? pre[(w0 + h) * 32 + lane] : 0.f;
#pragma unroll
      for (int h = 0; h < 8; ++h) {
        if (w0 + h < w_end) {
          // (not computed where W Delta = 0: with no clamp, pre_c may be infinite)
          float* at = acc + (w0 + h) * 32 + lane;
          const float d = *at;
          const float y = d != 0.f ? clamp_hi(pc[h] + d, hi) - clamp_hi(pc[h], hi) : 0.f;
          *at = y;
          nz += y != 0.f;
        }
      }
    }
    nz = (int)__reduce_add_sync(kFull, (unsigned)nz);
    if (lane == 0) s_cnt[warp] = nz;
    __syncthreads();
    int total;
    int base = warps_before(s_cnt, warp, total);
    int32_t* oi = a.out.idx + (size_t)r * SC;
    float* ov = a.out.val + (size_t)r * SC;
    float* dst = a.y_out + (size_t)r * N;
    // past the list capacity: a dense row; else the list in ascending position;
    // acc cleared for the next row
    for (int w = w_begin; w < w_end; ++w) {
      float* at = acc + w * 32 + lane;
      const float y = *at;
      const uint32_t m = __ballot_sync(kFull, y != 0.f);
      if (total > SC) {
        dst[w * 32 + lane] = y;
      } else if (y != 0.f) {
        const int k = base + __popc(m & ((1u << lane) - 1u));
        oi[k] = w * 32 + lane;
        ov[k] = y;
      }
      base += __popc(m);
      *at = 0.f;
    }
    if (tid == 0) {
      if (total > SC) {
        a.dense_list[atomicAdd(a.dense_count, 1)] = r;
      } else if (total > 0) {
        a.out.cnt[r] = total;
        a.sparse_list[atomicAdd(a.sparse_count, 1)] = r;
      }
    }
    __syncthreads();
  }
}

__global__ void finish_rows_kernel(const int32_t* dense_list, const int32_t* dense_count,
                                   const int32_t* sparse_list, const int32_t* sparse_count,
                                   SparseRows rows, float* y, int32_t* res_flag, int32_t N) {
  pdl_prologue();
  const int nd = *dense_count, n = sparse_list ? *sparse_count : 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nd; i += gridDim.x * blockDim.x)
    res_flag[dense_list[i]] = 1;
  const int lane = threadIdx.x & 31;
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  for (int i = wid; i < n; i += nw) {
    const int r = sparse_list[i];
    float* dst = y + (size_t)r * N;
    for (int c = lane; c < N; c += 32) dst[c] = 0.f;
    __syncwarp();
    const int cnt = rows.cnt[r];
    const int32_t* ei = rows.idx + (size_t)r * rows.cap;
    const float* ev = rows.val + (size_t)r * rows.cap;
    for (int e = lane; e < cnt; e += 32) dst[ei[e]] = ev[e];
    if (lane == 0) res_flag[r] = 1;
    __syncwarp();
  }
}

}  // namespace

size_t sparse_residue_smem(int N) { return (size_t)N * sizeof(float); }

bool sparse_residue_fits(int N) { return N <= 32768; }

cudaError_t sparse_residue_prepare(int N) {
  if (!sparse_residue_fits(N)) return cudaErrorInvalidValue;
  return allow_smem((const void*)sparse_residue_kernel);
}

void launch_split_residue(const float* y, const int32_t* list, const int32_t* count,
                          const SparseRows& out, int32_t* dense_list, int32_t* dense_count,
                          int32_t* sparse_list, int32_t* sparse_count, int32_t N, int num_sms,
                          cudaStream_t s) {
  launch_pdl(split_residue_kernel, num_sms * 8, kRowWarps * 32, 0, s, y, list, count, out, dense_list,
             dense_count, sparse_list, sparse_count, N);
}

cudaError_t launch_sparse_residue(const SparseResArgs& a, int num_sms, cudaStream_t s) {
  const size_t smem = sparse_residue_smem(a.N);
  int per_sm = (int)((227 * 1024) / (smem + 28 * 1024));
  per_sm = per_sm < 1 ? 1 : (per_sm > 8 ? 8 : per_sm);
  return launch_pdl(sparse_residue_kernel, num_sms * per_sm, kRowWarps * 32, smem, s, a);
}

void launch_finish_rows(const int32_t* dense_list, const int32_t* dense_count,
                        const int32_t* sparse_list, const int32_t* sparse_count,
                        const SparseRows& rows, float* y, int32_t* res_flag, int32_t N, int num_sms,
                        cudaStream_t s) {
  launch_pdl(finish_rows_kernel, num_sms * 2, 256, 0, s, dense_list, dense_count, sparse_list,
             sparse_count, rows, y, res_flag, N);
}

}  // namespace sdnn
