// Plain / centroid / residue layer kernel (the sparse-W x dense-Y step).
//
// Computes, for each row r of a row list and each output neuron c,
//     acc = sum over in-edges (j -> c) of w_jc * Y_in[r][j]
// and applies one of three epilogues (sdnn_internal.h).  The reference's
// forms of this step are bf_inference (src/SDGC/BF/kernel.hpp:26-89),
// snig_inference (src/SDGC/SNIG/kernel.hpp:24-114), the XY pre-threshold
// kernels (src/SDGC/XY/kernel.hpp:12-149) and post_spMM + post_minus
// (src/SDGC/SNICIT/kernel.hpp:71-136).  Those scatter Y*W into a shared row
// with shared-memory atomics; this kernel gathers instead:
//
//  * a CTA owns a tile of T rows; one thread issues 1-D TMA bulk copies
//    (cp.async.bulk + mbarrier) of the T input rows (or one input chunk of
//    them) into shared memory, row stride RS = chunk + 32 floats; the last 32
//    floats of every row are zero and serve the padding slots;
//  * a warp takes output groups of 32 neurons, lane i owns output 32g+i and
//    keeps T accumulators in registers (one per row of the tile);
//  * the in-edges of a group are pre-arranged into slots whose 32 indices hit
//    32 distinct banks, so every shared load of a slot is one wavefront;
//  * the summation order of an output is its slot order, fixed at packing
//    time, so results are bitwise reproducible (no atomics on values);
//  * bias + ReLU + clamp (or the residue update) are fused in the epilogue;
//    the CTA compacts surviving rows into the next row list with one atomic
//    per tile (and a mark per row when several CTAs share a tile).
#pragma once
#include "sdnn_internal.h"

namespace sdnn {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Waits for an mbarrier phase for at most limit_ns (default 2 s); on timeout
// records DEV_TIMEOUT in the error word and returns false.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, int32_t* err,
                                                  uint64_t limit_ns = 2000000000ull) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = global_ns();
  while (!mbar_try_wait(bar, parity)) {
    if (global_ns() - t0 > limit_ns) {
      atomicExch(err, DEV_TIMEOUT);
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
// This CTA's share of the lists that the next launch reads, into L2 (one
// thread): a layer's weights are read once per inference, far apart.
__device__ __forceinline__ void fetch_next_lists(const LayerArgs& a) {
  if (!a.next) return;
  const uint32_t share = (a.next_bytes / gridDim.x + 16) & ~15u, from = blockIdx.x * share;
  if (from < a.next_bytes)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"((const char*)a.next + from),
                 "r"(min(share, a.next_bytes - from))
                 : "memory");
}
__device__ __forceinline__ float clampf(float v, float hi) { return fminf(hi, fmaxf(0.f, v)); }


// Adds one slot (index j of the packed word, weight w) to acc[T].
template <int T, int RSW>
__device__ __forceinline__ void apply_slot(float (&acc)[T], uint32_t j, float w,
                                           const float* __restrict__ ys, int RS) {
  // byte offset or float index, fixed by the packer for this row stride
  const float* p = rsw_in_bytes(RSW)
                       ? reinterpret_cast<const float*>(reinterpret_cast<const char*>(ys) + j)
                       : ys + j;
#pragma unroll
  for (int t = 0; t < T; ++t) {
    const int off = (RSW > 0 ? RSW : RS) * t;
    acc[t] = fmaf(w, p[off], acc[t]);
  }
}

// Applies the first n slots of a block (1 <= n <= 4, the same for the whole
// warp); n is a compile-time 4 for full blocks.
template <int T, int RSW, bool CONSTW>
__device__ __forceinline__ void apply_block(float (&acc)[T], uint2 iv, const float4& vv, float wc,
                                            const float* __restrict__ ys, int RS, int n) {
  apply_slot<T, RSW>(acc, iv.x & 0xffffu, CONSTW ? wc : vv.x, ys, RS);
  if (n > 1) apply_slot<T, RSW>(acc, iv.x >> 16, CONSTW ? wc : vv.y, ys, RS);
  if (n > 2) apply_slot<T, RSW>(acc, iv.y & 0xffffu, CONSTW ? wc : vv.z, ys, RS);
  if (n > 3) apply_slot<T, RSW>(acc, iv.y >> 16, CONSTW ? wc : vv.w, ys, RS);
}

// Blocks of a list held in registers ahead of their use (per lane 2 registers
// a block, 4 more for per-edge values); tiles of one or two rows.
template <bool CONSTW>
constexpr int kAhead = CONSTW ? 4 : 2;

// The groups gbeg + warp, + nwarps, ... below gend of a tile in shared memory:
// accumulates each group's list and hands (acc, group) to done().  The slot
// lists are walked as one stream: a block's registers are refilled with the
// block NB further on -- of this group or the next -- as soon as it has been
// applied, so a warp never waits for a round trip to L2 between batches or
// groups.  That costs registers (64 a thread against 32 to 64 in batches): it
// pays where a CTA has its SM to itself and a list is few gathers, tiles of one
// or two rows (choose_kernel has the times).  A list ends at its last used slot,
// not at the end of its last block of 4 (1.5 of 38 slots).
template <int T, int RSW, bool CONSTW, typename Done>
__device__ __forceinline__ void walk_groups(const LayerDev& wl, const float* __restrict__ ys, int RS,
                                            int gbeg, int gend, int warp, int nwarps, int lane,
                                            Done done) {
  constexpr int NB = kAhead<CONSTW>;
  const float wc = wl.wconst;
  const uint2* __restrict__ idx = wl.idx + lane;
  const float4* __restrict__ val = CONSTW ? nullptr : wl.val + lane;
  for (int base = gbeg + warp; base < gend; base += 32 * nwarps) {
    // lane i holds the list (first block, slots) of the warp's i-th group
    int2 mine = make_int2(0, 0);
    if (base + lane * nwarps < gend) mine = __ldg(wl.lists + base + lane * nwarps);
    const int n = min(32, (gend - base + nwarps - 1) / nwarps);
    int b = __shfl_sync(0xffffffffu, mine.x, 0), slots = __shfl_sync(0xffffffffu, mine.y, 0);
    uint2 iv[NB];
    float4 vv[CONSTW ? 1 : NB];
#pragma unroll
    for (int k = 0; k < NB; ++k) {
      if (4 * k < slots) {
        iv[k] = __ldg(idx + (size_t)(b + k) * 32);
        if constexpr (!CONSTW) vv[k] = __ldg(val + (size_t)(b + k) * 32);
      }
    }
    for (int i = 0; i < n; ++i) {
      float acc[T];
#pragma unroll
      for (int t = 0; t < T; ++t) acc[t] = 0.f;
      bool last;
      do {
        last = slots <= 4 * NB;
        // where the refills come from: the rest of this list, or the next one
        const int fb = last ? __shfl_sync(0xffffffffu, mine.x, (i + 1) & 31) : b + NB;
        int fs = slots - 4 * NB;
        if (last) fs = i + 1 < n ? __shfl_sync(0xffffffffu, mine.y, (i + 1) & 31) : 0;
        if (slots >= 4 * NB) {  // a whole batch: one straight run of gathers
#pragma unroll
          for (int k = 0; k < NB; ++k) {
            apply_block<T, RSW, CONSTW>(acc, iv[k], vv[CONSTW ? 0 : k], wc, ys, RS, 4);
            if (4 * k < fs) {
              iv[k] = __ldg(idx + (size_t)(fb + k) * 32);
              if constexpr (!CONSTW) vv[k] = __ldg(val + (size_t)(fb + k) * 32);
            }
          }
        } else {
          const int full = slots >> 2, part = slots & 3;
          uint2 ti = iv[0];
          float4 tv = vv[0];
#pragma unroll
          for (int k = 0; k < NB; ++k) {
            if (k > 0 && k == full) {
              ti = iv[k];
              if constexpr (!CONSTW) tv = vv[k];
            }
            if (k < full)
              apply_block<T, RSW, CONSTW>(acc, iv[k], vv[CONSTW ? 0 : k], wc, ys, RS, 4);
            if (4 * k < fs) {
              iv[k] = __ldg(idx + (size_t)(fb + k) * 32);
              if constexpr (!CONSTW) vv[k] = __ldg(val + (size_t)(fb + k) * 32);
            }
          }
          if (part) apply_block<T, RSW, CONSTW>(acc, ti, tv, wc, ys, RS, part);
        }
        b = fb;
        slots = fs;
      } while (!last);
      done(acc, base + i * nwarps);
    }
  }
}

// Applies one block of slots of an input chunk to acc[T].
template <int T, int RSW, bool CONSTW, int NB>
__device__ __forceinline__ void apply_blocks(float (&acc)[T], const uint2 (&iv)[NB],
                                             const float4 (&vv)[CONSTW ? 1 : NB], float wc,
                                             const float* __restrict__ ys, int RS) {
#pragma unroll
  for (int k = 0; k < NB; ++k)
    apply_block<T, RSW, CONSTW>(acc, iv[k], vv[CONSTW ? 0 : k], wc, ys, RS, 4);
}

// Loads NB blocks starting at block b (indices and, for general layers, values).
template <bool CONSTW, int NB>
__device__ __forceinline__ void load_blocks(uint2 (&iv)[NB], float4 (&vv)[CONSTW ? 1 : NB],
                                            const uint2* __restrict__ ip,
                                            const float4* __restrict__ vp, int b) {
#pragma unroll
  for (int k = 0; k < NB; ++k) {
    iv[k] = __ldg(ip + (size_t)(b + k) * 32);
    if constexpr (!CONSTW) vv[k] = __ldg(vp + (size_t)(b + k) * 32);
  }
}

// Accumulates the in-edges of group g from input chunk q into acc[T].
// Slot blocks are fetched in batches of 8, then 2, then 1 (no predicated
// tail): all indices of a batch are in registers before the first is used,
// so a warp waits for one memory round trip per batch.
template <int T, int RSW, bool CONSTW>
__device__ __forceinline__ void accumulate_group(float (&acc)[T], const LayerDev& wl, int nq,
                                                 const float* __restrict__ ys, int RS, int g,
                                                 int q, int lane) {
  const int32_t b0 = __ldg(wl.grp_blk + g * nq + q);
  const int32_t b1 = __ldg(wl.grp_blk + g * nq + q + 1);
  const uint2* __restrict__ ip = wl.idx + (size_t)b0 * 32 + lane;
  const float4* __restrict__ vp = CONSTW ? nullptr : wl.val + (size_t)b0 * 32 + lane;
  const float wc = wl.wconst;
  const int nb = b1 - b0;
  int b = 0;
  for (; b + 8 <= nb; b += 8) {
    uint2 iv[8];
    float4 vv[CONSTW ? 1 : 8];
    load_blocks<CONSTW, 8>(iv, vv, ip, vp, b);
    apply_blocks<T, RSW, CONSTW, 8>(acc, iv, vv, wc, ys, RS);
  }
  for (; b + 2 <= nb; b += 2) {
    uint2 iv[2];
    float4 vv[CONSTW ? 1 : 2];
    load_blocks<CONSTW, 2>(iv, vv, ip, vp, b);
    apply_blocks<T, RSW, CONSTW, 2>(acc, iv, vv, wc, ys, RS);
  }
  if (b < nb) {
    uint2 iv[1];
    float4 vv[1];
    load_blocks<CONSTW, 1>(iv, vv, ip, vp, b);
    apply_blocks<T, RSW, CONSTW, 1>(acc, iv, vv, wc, ys, RS);
  }
}

// Input chunks: the KG groups of a warp (gbeg + warp + kk * nwarps) over
// chunk q.  Their lists are short (about 8 slots per lane and chunk), so
// fetching them group by group costs a memory round trip per group; here the
// KG offsets come in one load (lane kk holds group kk's), and the first
// CHUNK_NB blocks of group kk + 1 are loaded while group kk is applied.  The
// FMA order of every group is unchanged (blocks, then slots, in order).
constexpr int CHUNK_NB = 4;
template <int T, int RSW, bool CONSTW, int KG>
__device__ __forceinline__ void accumulate_chunk(float (&acc)[KG][T], const LayerDev& wl, int nq,
                                                 const float* __restrict__ ys, int RS, int gbeg,
                                                 int gend, int warp, int nwarps, int q, int lane) {
  int32_t my_b0 = 0, my_b1 = 0;
  if (lane < KG) {
    const int g = gbeg + warp + lane * nwarps;
    if (g < gend) {
      my_b0 = __ldg(wl.grp_blk + g * nq + q);
      my_b1 = __ldg(wl.grp_blk + g * nq + q + 1);
    }
  }
  const float wc = wl.wconst;
  uint2 iv[2][CHUNK_NB];
  float4 vv[2][CONSTW ? 1 : CHUNK_NB];
  auto fetch = [&](int kk, uint2 (&i)[CHUNK_NB], float4 (&v)[CONSTW ? 1 : CHUNK_NB]) {
    const int32_t b0 = __shfl_sync(0xffffffffu, my_b0, kk);
    const int nb = __shfl_sync(0xffffffffu, my_b1, kk) - b0;
    const uint2* ip = wl.idx + (size_t)b0 * 32 + lane;
#pragma unroll
    for (int k = 0; k < CHUNK_NB; ++k) {
      if (k < nb) {
        i[k] = __ldg(ip + (size_t)k * 32);
        if constexpr (!CONSTW) v[k] = __ldg(wl.val + (size_t)(b0 + k) * 32 + lane);
      }
    }
  };
  fetch(0, iv[0], vv[0]);
#pragma unroll
  for (int kk = 0; kk < KG; ++kk) {
    const int cur = kk & 1;
    if (kk + 1 < KG) fetch(kk + 1, iv[cur ^ 1], vv[cur ^ 1]);
    const int32_t b0 = __shfl_sync(0xffffffffu, my_b0, kk);
    const int nb = __shfl_sync(0xffffffffu, my_b1, kk) - b0;
    // the first CHUNK_NB blocks (prefetched), one at a time in order
#pragma unroll
    for (int k = 0; k < CHUNK_NB; ++k) {
      if (k < nb) {
        uint2 one[1] = {iv[cur][k]};
        float4 onev[1];
        if constexpr (!CONSTW) onev[0] = vv[cur][k];
        apply_blocks<T, RSW, CONSTW, 1>(acc[kk], one, onev, wc, ys, RS);
      }
    }
    // the rest of a long list, in exact-size batches
    if (nb > CHUNK_NB) {
      const uint2* ip = wl.idx + (size_t)b0 * 32 + lane;
      const float4* vp = CONSTW ? nullptr : wl.val + (size_t)b0 * 32 + lane;
      int b = CHUNK_NB;
      for (; b + 4 <= nb; b += 4) {
        uint2 i4[4];
        float4 v4[CONSTW ? 1 : 4];
        load_blocks<CONSTW, 4>(i4, v4, ip, vp, b);
        apply_blocks<T, RSW, CONSTW, 4>(acc[kk], i4, v4, wc, ys, RS);
      }
      for (; b < nb; ++b) {
        uint2 i1[1];
        float4 v1[1];
        load_blocks<CONSTW, 1>(i1, v1, ip, vp, b);
        apply_blocks<T, RSW, CONSTW, 1>(acc[kk], i1, v1, wc, ys, RS);
      }
    }
  }
}

// Epilogue of one group for the rows of the tile; returns this lane's mask of
// flagged rows (alive for PLAIN, non-empty for RESIDUE), merged over the warp
// once per tile.
template <int T>
__device__ __forceinline__ uint32_t epilogue_group(const float (&acc)[T], const LayerArgs& a,
                                                   const int32_t* s_rows, int nrows, int g,
                                                   int lane) {
  const int c = g * 32 + lane;
  const float bc = a.w.bias_vec ? __ldg(a.w.bias_vec + c) : a.w.bias;
  const float hi = a.clampv;
  uint32_t m = 0;
#pragma unroll
  for (int t = 0; t < T; ++t) {
    if (t < nrows) {
      const int row = s_rows[t];
      float* dst = a.y_out + (size_t)row * a.N + c;
      if (a.epi == EPI_PLAIN) {
        const float v = acc[t] + bc;
        *dst = clampf(v, hi);
        if (v > 0.f) m |= 1u << t;
      } else if (a.epi == EPI_CENTROID) {
        const int k = a.cslot[row];
        const float v = acc[t] + bc;
        a.pre_out[(size_t)k * a.N + c] = v;
        *dst = clampf(v, hi);
      } else {
        const int k = a.cslot[row];
        const float pc = a.pre_in[(size_t)k * a.N + c];
        const float y = clampf(pc + acc[t], hi) - clampf(pc, hi);
        *dst = y;
        if (y != 0.f) m |= 1u << t;
      }
    }
  }
  return m;
}

// Issues the TMA bulk copies of the rows of one tile (one input chunk) into a
// shared buffer and arms its mbarrier; called by one thread.
__device__ __forceinline__ void load_tile(const LayerArgs& a, float* buf, int RS,
                                          const int32_t* rows, int nrows, int q, uint64_t* bar) {
  const uint32_t row_bytes = (uint32_t)a.Q * 4u;
  mbar_expect_tx(bar, row_bytes * (uint32_t)nrows);
  for (int t = 0; t < nrows; ++t) {
    const char* src =
        reinterpret_cast<const char*>(a.y_in + (size_t)rows[t] * a.N + (size_t)q * a.Q);
    char* dst = reinterpret_cast<char*>(buf + (size_t)t * RS);
    for (uint32_t off = 0; off < row_bytes; off += 32768u)
      bulk_g2s(dst + off, src + off, min(32768u, row_bytes - off), bar);
  }
}

// Appends the rows of a finished piece of a tile that are flagged in m to the
// next list (called by one warp).  When other CTAs hold the tile's other
// groups, a row may be found by several of them: the first to put this
// launch's mark on the row appends it (a.stamp; marks differ between the
// launches of an inference and are cleared at its start).
__device__ __forceinline__ void publish_rows(const LayerArgs& a, uint32_t m, bool shared,
                                             const int32_t* rows, int lane) {
  if (a.epi == EPI_CENTROID || m == 0) return;
  bool mine = (m >> lane) & 1u;
  const int row = mine ? rows[lane] : 0;
  if (shared && mine) mine = atomicExch(a.stamp + row, a.stamp_id) != a.stamp_id;
  const uint32_t w = __ballot_sync(0xffffffffu, mine);
  if (!w) return;
  int at = 0;
  if (lane == 0) at = atomicAdd(a.count_out, __popc(w));
  at = __shfl_sync(0xffffffffu, at, 0) + __popc(w & ((1u << lane) - 1u));
  if (mine) a.list_out[at] = row;
}

// ---------------------------------------------------------------------------
// Whole rows in shared memory (N <= 32768).
//
// Split of the work: the tiles' groups are cut into units of one group per
// warp, and the units of all tiles, in order, are divided evenly over the
// CTAs, so a CTA gets a contiguous run of units that may begin and end inside
// a tile.  With one item per (tile, part) the last wave was nearly empty for
// row counts between the grid's size and a few times that: 329 rows of 16384
// neurons took two rounds of half-tile items, 104 us, for 21 us of gathers.
// With fewer units than CTAs the tiles are cut finer, at most one piece per
// CTA.  Small row counts use smaller tiles (TE < T): what bounds them is the
// time to fetch rows and lists, which the CTAs then share.
//
// A CTA's run is worked out by one warp, in 32 bits (rows in memory times
// groups stay far below 2^32 units): done by every warp in 64 bits it took
// longer than the copy of a row.
struct Cut {
  int count, TE, unit, per_tile;  // rows, rows per tile, groups per unit, units per tile
  int tile, first, left;          // the CTA's run: first tile and unit in it, units
};
// Largest tile size <= T, then halved from the power of 2 below it, that
// still gives every CTA a unit.
template <int T>
__device__ __forceinline__ Cut make_cut(int count, int G, int nwarps) {
  Cut c;
  c.count = count;
  c.unit = nwarps;
  c.per_tile = (G + nwarps - 1) / nwarps;
  c.TE = T;
  int p2 = 1;
  while (2 * p2 < T) p2 *= 2;
  const unsigned grid = gridDim.x, rows = (unsigned)count;
  unsigned tiles = (rows + T - 1) / T;
  while (c.TE > 1 && tiles * c.per_tile < grid) {
    c.TE = c.TE == T ? p2 : c.TE / 2;
    tiles = (rows + c.TE - 1) / (unsigned)c.TE;
  }
  if (tiles * c.per_tile < grid && tiles > 0) {
    const unsigned parts = grid / tiles;
    c.unit = (int)(((unsigned)G + parts - 1) / parts);
    c.per_tile = (int)(((unsigned)G + c.unit - 1) / (unsigned)c.unit);
  }
  const unsigned units = tiles * c.per_tile, share = units / grid, more = units % grid;
  const unsigned lo = share * blockIdx.x + min(blockIdx.x, more);
  c.left = (int)(share + (blockIdx.x < more ? 1 : 0));
  c.tile = (int)(lo / (unsigned)c.per_tile);
  c.first = (int)(lo % (unsigned)c.per_tile);
  return c;
}

// One piece of a tile: groups [gbeg, gend) of the rows in shared memory.
template <int T, int RSW, bool CONSTW, bool AHEAD>
__device__ __forceinline__ uint32_t run_piece(const LayerArgs& a, const float* ys, int RS,
                                              const int32_t* rows, int nrows, int gbeg, int gend,
                                              int warp, int nwarps, int lane) {
  uint32_t m = 0;
  if constexpr (AHEAD) {
    walk_groups<T, RSW, CONSTW>(a.w, ys, RS, gbeg, gend, warp, nwarps, lane,
                                [&](const float (&acc)[T], int g) {
                                  m |= epilogue_group<T>(acc, a, rows, nrows, g, lane);
                                });
  } else {
    for (int g = gbeg + warp; g < gend; g += nwarps) {
      float acc[T];
#pragma unroll
      for (int t = 0; t < T; ++t) acc[t] = 0.f;
      accumulate_group<T, RSW, CONSTW>(acc, a.w, 1, ys, RS, g, 0, lane);
      m |= epilogue_group<T>(acc, a, rows, nrows, g, lane);
    }
  }
  return m;
}
// ... with the code of the smallest tile size that holds TE rows.
template <int T, int P2, int RSW, bool CONSTW, bool AHEAD>
__device__ __forceinline__ uint32_t run_sized(int TE, const LayerArgs& a, const float* ys, int RS,
                                              const int32_t* rows, int nrows, int gbeg, int gend,
                                              int warp, int nwarps, int lane) {
  if constexpr (P2 >= 1) {
    if (TE <= P2)
      return run_sized<P2, P2 / 2, RSW, CONSTW, AHEAD>(TE, a, ys, RS, rows, nrows, gbeg, gend, warp,
                                                       nwarps, lane);
  }
  return run_piece<T, RSW, CONSTW, AHEAD>(a, ys, RS, rows, nrows, gbeg, gend, warp, nwarps, lane);
}
__host__ __device__ constexpr int pow2_below(int t) {
  int p = 1;
  while (2 * p < t) p *= 2;
  return t > 1 ? p : 0;
}

template <int T, int RSW, bool CONSTW, bool AHEAD>
__device__ __forceinline__ void layer_rows(const LayerArgs& a) {
  extern __shared__ __align__(128) float ys[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ int32_t s_rows[2][32];
  __shared__ uint32_t s_mask[2];
  __shared__ int32_t s_fail;
  __shared__ Cut s_cut;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int RS = RSW > 0 ? RSW : a.Q + 32;
  // Launched with programmatic stream serialization: the next launch may be
  // scheduled now, and this one may have started before its predecessor
  // ended -- so only CTA-local setup comes before griddepcontrol.wait, which
  // returns once the predecessor has completed and its writes are visible.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (tid == (int)blockDim.x - 32) fetch_next_lists(a);
  // One tile buffer, reloaded per tile: the load of one CTA overlaps the
  // compute of the other CTAs on the SM (up to four).
  for (int i = tid; i < T * 32; i += blockDim.x) ys[(i >> 5) * RS + a.Q + (i & 31)] = 0.f;
  if (tid == 0) {
    mbar_init(&bar, 1);
    s_mask[0] = s_mask[1] = 0;
    s_fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (warp == 0) {
    const Cut c = make_cut<T>(__ldcg(a.count_in), a.G, nwarps);
    if (lane == 0) s_cut = c;
  }
  __syncthreads();
  const Cut cut = s_cut;
  int tile = cut.tile, first = cut.first, left = cut.left;
  if (left == 0) return;
  // the row ids of the tile after the current one are fetched while it runs
  int next_row = -1;
  if (warp == 0 && lane < cut.TE && tile * cut.TE + lane < cut.count)
    next_row = a.list_in[tile * cut.TE + lane];
  uint32_t phase = 0;
  int buf = 0;
  bool pending = false, pending_shared = false;
  while (left > 0) {
    const int take = min(left, cut.per_tile - first);
    const int nrows = min(cut.TE, cut.count - tile * cut.TE);
    const int gbeg = first * cut.unit, gend = min(a.G, (first + take) * cut.unit);
    __syncthreads();  // every warp is done with the previous tile
    if (warp == 0) {
      s_rows[buf][lane] = next_row;
      // one lane per row issues its copies (a long row in pieces of 32 KB)
      const uint32_t row_bytes = (uint32_t)a.Q * 4u;
      if (lane == 0) mbar_expect_tx(&bar, row_bytes * (uint32_t)nrows);
      __syncwarp();
      if (lane < nrows) {
        const char* src = reinterpret_cast<const char*>(a.y_in + (size_t)next_row * a.N);
        char* dst = reinterpret_cast<char*>(ys + (size_t)lane * RS);
        for (uint32_t off = 0; off < row_bytes; off += 32768u)
          bulk_g2s(dst + off, src + off, min(32768u, row_bytes - off), &bar);
      }
      const int nt = tile + 1;
      next_row = -1;
      if (take < left && lane < cut.TE && nt * cut.TE + lane < cut.count)
        next_row = a.list_in[nt * cut.TE + lane];
      if (lane == 0 && !mbar_wait_bounded(&bar, phase, a.err)) s_fail = 1;
    }
    // the rows of the previous piece are published while this tile loads
    if (warp == nwarps - 1 && pending) {
      publish_rows(a, s_mask[buf ^ 1], pending_shared, s_rows[buf ^ 1], lane);
      __syncwarp();
      if (lane == 0) s_mask[buf ^ 1] = 0;
    }
    __syncthreads();
    if (s_fail) return;
    mbar_try_wait(&bar, phase);
    phase ^= 1u;
    uint32_t m = run_sized<T, pow2_below(T), RSW, CONSTW, AHEAD>(
        cut.TE, a, ys, RS, s_rows[buf], nrows, gbeg, gend, warp, nwarps, lane);
    m = __reduce_or_sync(0xffffffffu, m);
    if (lane == 0 && m) atomicOr(&s_mask[buf], m);
    pending = true;
    pending_shared = take < cut.per_tile;
    left -= take;
    first = 0;
    ++tile;
    buf ^= 1;
  }
  __syncthreads();
  if (warp == nwarps - 1)
    publish_rows(a, s_mask[buf ^ 1], pending_shared, s_rows[buf ^ 1], lane);
}

// Registers.  Where rows are short several CTAs share an SM, and half of them
// at 64 registers a thread cost up to 1.7 times the time (60000 rows of 1024 with
// values, 24 x 256: 447 -> 769 us; of 96: 142 -> 218); the compiler, left alone,
// takes 32 to 64.  With one value and tiles of 4 to 8 rows it takes 32 and spills,
// or leaves too few loads in flight: those have 48 (600 rows of 992, 8 x 512:
// 16.5 -> 14.2 us; 20000 of 8192: 928 -> 895), or 32 without its spills at the
// stride of 1024 (60000 rows, 8 x 1024: 373 -> 358).
template <int T, int RSW, bool CONSTW, bool AHEAD>
__global__ void __launch_bounds__(1024, AHEAD ? 1 : 0) layer_rows_kernel(const LayerArgs a) {
  layer_rows<T, RSW, CONSTW, AHEAD>(a);
}
template <int T, int RSW, bool CONSTW>
__global__ void __maxnreg__(RSW == 1056 ? 32 : 48) layer_rows_regs_kernel(const LayerArgs a) {
  layer_rows<T, RSW, CONSTW, false>(a);
}

// ---------------------------------------------------------------------------
// Input chunks (rows too wide for shared memory): an item is (tile, part of
// the groups), parts sized to the registers that hold the accumulators.
struct Split {
  int count, n_tiles, spl;
  int items;
};
template <int T>
__device__ __forceinline__ Split make_split(const LayerArgs& a) {
  Split sp;
  sp.count = *a.count_in;
  sp.n_tiles = (sp.count + T - 1) / T;
  int spl = sp.n_tiles > 0 ? (int)((gridDim.x + sp.n_tiles - 1) / sp.n_tiles) : 1;
  spl = max(spl, a.min_split);
  spl = min(spl, a.max_split);
  sp.spl = max(spl, 1);
  sp.items = sp.n_tiles * sp.spl;
  return sp;
}

template <int T, int RSW, int KG, bool CONSTW>
// (instances with up to 8 groups per warp may run 1024 threads; 16 groups per
// warp keep 512 so their KG x T accumulators stay in registers)
__global__ void __launch_bounds__(KG <= 8 ? 1024 : 512, 1) layer_chunk_kernel(const LayerArgs a) {
  extern __shared__ __align__(128) float ys[];
  __shared__ __align__(8) uint64_t bar[1];
  __shared__ int32_t s_rows[2][T];
  __shared__ int32_t s_next[T];
  __shared__ uint32_t s_mask, s_pmask;
  __shared__ int32_t s_ppending, s_pbuf;
  __shared__ int32_t s_fail;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int RS = RSW > 0 ? RSW : a.Q + 32;
  // (programmatic stream serialization, see layer_rows_kernel)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (tid == (int)blockDim.x - 32) fetch_next_lists(a);
  for (int i = tid; i < T * 32; i += blockDim.x) ys[(i >> 5) * RS + a.Q + (i & 31)] = 0.f;
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    s_mask = 0;
    s_fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const Split sp = make_split<T>(a);
  if (sp.count <= 0 || (int)blockIdx.x >= sp.items) return;
  __syncthreads();

  // Per item: row ids of the item after it are fetched while it runs, and the
  // rows it flags are published (a chain of global atomics) during the next
  // item, while the other warps already work on it -- both by the CTA's last
  // warp; s_rows is double-buffered, and the pending state lives in shared
  // memory so that it costs the compute warps no registers.
  const bool last_warp = warp == nwarps - 1;
  auto item_row = [&](int it, int t) -> int {
    const int r0 = (int)(it / sp.spl) * T;
    return t < min(T, sp.count - r0) ? a.list_in[r0 + t] : -1;
  };
  if (last_warp && lane < T) s_next[lane] = item_row(blockIdx.x, lane);
  if (last_warp && lane == 31) s_ppending = 0;
  uint32_t phase = 0;
  int b = 0;
  for (int item = blockIdx.x; item < sp.items; item += gridDim.x, b ^= 1) {
    const int tile = (int)(item / sp.spl), part = (int)(item % sp.spl);
    const int row0 = tile * T;
    const int nrows = min(T, sp.count - row0);
    const int gbeg = (int)((long)a.G * part / sp.spl), gend = (int)((long)a.G * (part + 1) / sp.spl);
    __syncthreads();  // s_rows[b] is free: the item that used it was published
    if (tid < T) s_rows[b][tid] = s_next[tid];
    __syncthreads();
    if (last_warp) {
      if (lane < T && item + gridDim.x < sp.items) s_next[lane] = item_row(item + gridDim.x, lane);
      if (s_ppending) publish_rows(a, s_pmask, sp.spl > 1, s_rows[s_pbuf], lane);
    }
    uint32_t m = 0;
    // accumulators of KG groups per warp live across chunks
    float acc[KG][T];
#pragma unroll
    for (int kk = 0; kk < KG; ++kk)
#pragma unroll
      for (int t = 0; t < T; ++t) acc[kk][t] = 0.f;
    for (int q = 0; q < a.nq; ++q) {
      if (q > 0) __syncthreads();
      if (tid == 0) {
        load_tile(a, ys, RS, s_rows[b], nrows, q, &bar[0]);
        s_fail = mbar_wait_bounded(&bar[0], phase, a.err) ? 0 : 1;
      }
      __syncthreads();
      if (s_fail) return;
      mbar_try_wait(&bar[0], phase);
      phase ^= 1u;
      accumulate_chunk<T, RSW, CONSTW, KG>(acc, a.w, a.nq, ys, RS, gbeg, gend, warp, nwarps, q,
                                           lane);
    }
#pragma unroll
    for (int kk = 0; kk < KG; ++kk) {
      const int g = gbeg + warp + kk * nwarps;
      if (g < gend) m |= epilogue_group<T>(acc[kk], a, s_rows[b], nrows, g, lane);
    }
    m = __reduce_or_sync(0xffffffffu, m);
    if (lane == 0 && m) atomicOr(&s_mask, m);
    __syncthreads();
    if (last_warp && lane == 31) {
      s_pmask = s_mask;
      s_mask = 0;
      s_ppending = 1;
      s_pbuf = b;
    }
    __syncwarp();
  }
  if (last_warp && s_ppending) publish_rows(a, s_pmask, sp.spl > 1, s_rows[s_pbuf], lane);
}

#define SDNN_CHUNK_INSTANCE(T, RSW, KG, CW) \
  template __global__ void layer_chunk_kernel<T, RSW, KG, CW>(const LayerArgs);

// Registry entry used by the dispatcher.
struct LayerInstance {
  int T, rsw, kg;
  bool constw, ahead;
  const void* fn;
};

template <int T, int RSW, bool CONSTW, bool AHEAD>
LayerInstance rows_instance() {
  if constexpr (CONSTW && !AHEAD && T >= 4 && T <= 8)
    return {T, RSW, 1, CONSTW, AHEAD, (const void*)&layer_rows_regs_kernel<T, RSW, CONSTW>};
  else
    return {T, RSW, 1, CONSTW, AHEAD, (const void*)&layer_rows_kernel<T, RSW, CONSTW, AHEAD>};
}
// ... for layers with a value per edge and with one value.
#define SDNN_ROWS_INSTANCES(v, T, RSW, AHEAD)          \
  v.push_back(rows_instance<T, RSW, false, AHEAD>()); \
  v.push_back(rows_instance<T, RSW, true, AHEAD>())

}  // namespace sdnn
