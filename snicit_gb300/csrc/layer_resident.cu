// Layer kernel with the slot lists resident in tensor memory (N <= 4096).
//
// The same step, epilogues, slots and summation order as layer_rows_kernel
// (layer_kernel.cuh): bitwise the same rows.  What bounds both is the shared
// memory port (a gather of 32 operands is one wavefront); layer_rows_kernel
// fetches every slot list again for every tile, through the same port: two
// wavefronts to fill L1 and two to read a block of 4 slots, for 4 T wavefronts
// of gathers -- 17 % at T = 6 rows of 4096 neurons, twice that with a value
// per edge.  Here a CTA keeps its groups' lists for the whole launch in tensor
// memory (256 KB per SM, its own read path, no use of the port), 128 columns
// per warp, and streams row tiles past them:
//
//  * one CTA of 16 warps per SM; a warp owns up to 4 groups of 32 outputs (2
//    when the layer has a value per edge: 6 bytes per slot instead of 2), deep
//    ones and shallow ones together so that the warps stay level; layers of
//    more groups than a CTA holds are split over `split` CTAs that read the
//    same rows;
//  * row tiles arrive by TMA bulk copies in a ring of stages; a warp waits for
//    its stage's copies only, and the last warp to finish a tile lists the
//    tile's surviving rows and reloads the stage, so no barrier ties the warps
//    together and the copies run a few tiles ahead;
//  * the lists are loaded before griddepcontrol.wait (weights do not depend on
//    the previous launch), so their latency hides behind its end;
//  * a launch of few rows -- most layers of an inference, once rows have died
//    and merged -- is a chain of round trips: count, row ids and rows, lists.
//    There more CTAs share a tile than must, each with a group or so per warp,
//    one warp per CTA reads the count (all of them at one address took 1 us),
//    all blocks of a list are asked for at once, and the launch before has
//    fetched the lists into L2.  One row of 1024 neurons 8.0 -> 5.5 us in the
//    stream of an inference, of 4096 12.0 -> 5.4; 60 layers of 2048 with 600
//    rows at first 717 -> 573.
//
// One layer through the one-layer entry point, us with lists streamed per tile
// (best tile) -> kept: 60000 rows of 1024 neurons 307 -> 299, of 4096 1240 ->
// 1116, of 2048 651 -> 531 (the gathers alone need 239, 956 and 478 at one
// wavefront per clock).  The port is then 85 % busy, tile copies and stores
// included.  With a value per edge the two are level for many rows (1024: 333 ->
// 346, 4096: 1427 -> 1457) and the kept lists ahead in layer after layer of a few
// hundred (40 of 300 rows of 1536: 416 -> 301).
#include <algorithm>
#include <climits>
#include <cstdint>
#include "layer_kernel.cuh"

namespace sdnn {

namespace {

constexpr int kWarps = 16;
constexpr int kCols = 128;  // tensor memory columns of a warp
constexpr int kMaxStages = 6;
// groups a warp owns and the blocks of 4 slots it keeps of each: 2 words of
// indices a block, then 4 words of values a block in general layers
template <bool CONSTW>
constexpr int kGroups = CONSTW ? 4 : 2;
template <bool CONSTW>
constexpr int kResBlocks = CONSTW ? 16 : 10;
template <bool CONSTW>
constexpr int kGroupCols = kCols / kGroups<CONSTW>;
constexpr size_t kResSmem = 225 * 1024;

__device__ __forceinline__ void tmem_free(uint32_t base) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(base) : "memory");
}
__device__ __forceinline__ void tmem_st2(uint32_t addr, uint2 v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(v.x), "r"(v.y)
               : "memory");
}
__device__ __forceinline__ void tmem_st4(uint32_t addr, float4 v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr),
               "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)),
               "r"(__float_as_uint(v.w))
               : "memory");
}
__device__ __forceinline__ void tmem_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void tmem_ld8(uint32_t (&r)[8], uint32_t addr) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                 "=r"(r[7])
               : "r"(addr));
}
// The registers of the loads before it are valid after this wait (they are
// operands so that their uses stay behind it).
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]),
                 "+r"(r[7])::"memory");
}
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[4], uint32_t (&v)[8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(v[0]), "+r"(v[1]), "+r"(v[2]),
                 "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7])::"memory");
}

// A batch of a list in registers: 16 slots of a layer with one weight value,
// or 8 slots and their values.
template <bool CONSTW>
struct Batch;
template <>
struct Batch<true> {
  static constexpr int kSlots = 16;
  uint32_t w[8];
  // block words from column `col` on, b the first block
  __device__ __forceinline__ void load(uint32_t col, int b) { tmem_ld8(w, col + 2 * b); }
  __device__ __forceinline__ void wait() { tmem_wait_ld(w); }
  __device__ __forceinline__ float val(int, float wc) const { return wc; }
  __device__ __forceinline__ void drop(int pairs) {  // the first pairs are used up
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k + pairs < 8) w[k] = w[k + pairs];
  }
};
template <>
struct Batch<false> {
  static constexpr int kSlots = 8;
  uint32_t w[4], v[8];
  __device__ __forceinline__ void load(uint32_t col, int b) {
    tmem_ld4(w, col + 2 * b);
    tmem_ld8(v, col + 2 * kResBlocks<false> + 4 * b);
  }
  __device__ __forceinline__ void wait() { tmem_wait_ld(w, v); }
  __device__ __forceinline__ float val(int slot, float) const { return __uint_as_float(v[slot]); }
  __device__ __forceinline__ void drop(int pairs) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k + pairs < 4) w[k] = w[k + pairs];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k + 2 * pairs < 8) v[k] = v[k + 2 * pairs];
  }
};

template <int PAIRS, int T, int RSW, bool CONSTW>
__device__ __forceinline__ void apply_pairs(float (&acc)[T], const Batch<CONSTW>& b, float wc,
                                            const float* ys, int RS) {
#pragma unroll
  for (int k = 0; k < PAIRS; ++k) {
    apply_slot<T, RSW>(acc, b.w[k] & 0xffffu, b.val(2 * k, wc), ys, RS);
    apply_slot<T, RSW>(acc, b.w[k] >> 16, b.val(2 * k + 1, wc), ys, RS);
  }
}

// acc[T] over the first `slots` slots of the list in tensor memory from column
// `col` on.  cur holds the list's first batch on entry and that of the list at
// `next` on return: the next batch is always on its way while one is applied.
// The last batch is taken in runs of 8, 4, 2 and 1 slots.
template <int T, int RSW, bool CONSTW>
__device__ __forceinline__ void gather(float (&acc)[T], Batch<CONSTW>& cur, uint32_t col,
                                       uint32_t next, int slots, float wc, const float* ys, int RS) {
  constexpr int S = Batch<CONSTW>::kSlots;
  Batch<CONSTW> nxt;
  int b = 0;
  while (slots > S) {
    b += S / 4;
    nxt.load(col, b);
    apply_pairs<S / 2, T, RSW, CONSTW>(acc, cur, wc, ys, RS);
    nxt.wait();
    cur = nxt;
    slots -= S;
  }
  nxt.load(next, 0);
  if (slots == S) {
    apply_pairs<S / 2, T, RSW, CONSTW>(acc, cur, wc, ys, RS);
  } else {
    if (S == 16 && (slots & 8)) {
      apply_pairs<4, T, RSW, CONSTW>(acc, cur, wc, ys, RS);
      cur.drop(4);
    }
    if (slots & 4) {
      apply_pairs<2, T, RSW, CONSTW>(acc, cur, wc, ys, RS);
      cur.drop(2);
    }
    if (slots & 2) {
      apply_pairs<1, T, RSW, CONSTW>(acc, cur, wc, ys, RS);
      cur.drop(1);
    }
    if (slots & 1) apply_slot<T, RSW>(acc, cur.w[0] & 0xffffu, cur.val(0, wc), ys, RS);
  }
  nxt.wait();
  cur = nxt;
}

// Outputs of one group for a full tile in plain mode: no per-row tests.
template <int T>
__device__ __forceinline__ uint32_t plain_outputs(const float (&acc)[T], const LayerArgs& a,
                                                  float* const (&dst)[T], int g, int lane) {
  const int c = g * 32 + lane;
  const float bc = a.w.bias_vec ? __ldg(a.w.bias_vec + c) : a.w.bias;
  uint32_t m = 0;
#pragma unroll
  for (int t = 0; t < T; ++t) {
    const float v = acc[t] + bc;
    dst[t][c] = clampf(v, a.clampv);
    if (v > 0.f) m |= 1u << t;
  }
  return m;
}

// ... in residue mode: every row's pre-activation is on its way before the first
// is used (each is two loads, one after the other, and a CTA has its SM's only
// 16 warps).  14 post layers of some 21000 residue rows of 1024 neurons
// 2533 -> 1955 us (2416 with lists streamed per tile, of which 48 warps share an
// SM).
template <int T>
__device__ __forceinline__ uint32_t residue_outputs(const float (&acc)[T], const LayerArgs& a,
                                                    const int32_t* rows, int nrows, int g, int lane) {
  const int c = g * 32 + lane;
  float pc[T];
#pragma unroll
  for (int t = 0; t < T; ++t)
    pc[t] = t < nrows ? a.pre_in[(size_t)a.cslot[rows[t]] * a.N + c] : 0.f;
  uint32_t m = 0;
#pragma unroll
  for (int t = 0; t < T; ++t) {
    if (t < nrows) {
      const float y = clampf(pc[t] + acc[t], a.clampv) - clampf(pc[t], a.clampv);
      a.y_out[(size_t)rows[t] * a.N + c] = y;
      if (y != 0.f) m |= 1u << t;
    }
  }
  return m;
}

// One warp's groups over the rows of a stage; returns the lane's row mask.  (A
// loop of its own in residue mode: as a branch in the one loop it cost plain
// layers 1 %.)
template <int T, int RSW, bool CONSTW, bool RESIDUE>
__device__ __forceinline__ uint32_t run_groups(const LayerArgs& a, const float* ys, int RS,
                                               const int32_t* rows, int nrows, uint32_t col,
                                               Batch<CONSTW>& cur, const int2* lists, int first_grp,
                                               int step0, int step1, int n, int lane) {
  constexpr int kHeld = 4 * kResBlocks<CONSTW>;
  const bool plain = !RESIDUE && a.epi == EPI_PLAIN && nrows == T;
  float* dst[T];
#pragma unroll
  for (int t = 0; t < T; ++t) dst[t] = plain ? a.y_out + (size_t)rows[t] * a.N : nullptr;
  uint32_t m = 0;
  int g = first_grp;
#pragma unroll 1
  for (int i = 0; i < n; ++i) {
    const int2 list = lists[i];
    float acc[T];
#pragma unroll
    for (int t = 0; t < T; ++t) acc[t] = 0.f;
    const uint32_t here = col + i * kGroupCols<CONSTW>;
    gather<T, RSW, CONSTW>(acc, cur, here, i + 1 < n ? here + kGroupCols<CONSTW> : col,
                           min(list.y, kHeld), a.w.wconst, ys, RS);
    // slots past the resident ones (few groups of a layer, if any)
    for (int s = kHeld; s < list.y; s += 4) {
      const size_t at = (size_t)(list.x + (s >> 2)) * 32 + lane;
      const uint2 iv = __ldg(a.w.idx + at);
      float4 vv = make_float4(0.f, 0.f, 0.f, 0.f);
      if constexpr (!CONSTW) vv = __ldg(a.w.val + at);
      apply_block<T, RSW, CONSTW>(acc, iv, vv, a.w.wconst, ys, RS, min(4, list.y - s));
    }
    if constexpr (RESIDUE)
      m |= residue_outputs<T>(acc, a, rows, nrows, g, lane);
    else
      m |= plain ? plain_outputs<T>(acc, a, dst, g, lane)
                 : epilogue_group<T>(acc, a, rows, nrows, g, lane);
    g += (i & 1) ? step1 : step0;
  }
  return m;
}

// ... with the code of the smallest tile size that holds TE rows.
template <int T, int RSW, bool CONSTW>
__device__ __forceinline__ uint32_t run_stage(int TE, const LayerArgs& a, const float* ys, int RS,
                                              const int32_t* rows, int nrows, uint32_t col,
                                              Batch<CONSTW>& cur, const int2* lists, int first_grp,
                                              int step0, int step1, int n, int lane) {
  if constexpr (T > 1) {
    if (TE <= pow2_below(T))
      return run_stage<pow2_below(T), RSW, CONSTW>(TE, a, ys, RS, rows, nrows, col, cur, lists, first_grp,
                                           step0, step1, n, lane);
  }
  if (a.epi == EPI_RESIDUE)
    return run_groups<T, RSW, CONSTW, true>(a, ys, RS, rows, nrows, col, cur, lists, first_grp, step0,
                                            step1, n, lane);
  return run_groups<T, RSW, CONSTW, false>(a, ys, RS, rows, nrows, col, cur, lists, first_grp, step0,
                                           step1, n, lane);
}

template <int T, int RSW, bool CONSTW>
__global__ void __launch_bounds__(kWarps * 32, 1)
    layer_resident_kernel(const LayerArgs a, const int plan_split, int stages, const FewRows f) {
  extern __shared__ __align__(128) float ring[];  // [stages][T][RS]
  __shared__ __align__(8) uint64_t full[kMaxStages];
  __shared__ int32_t s_rows[kMaxStages][T];
  __shared__ uint32_t s_mask[kMaxStages];
  __shared__ int32_t s_done[kMaxStages];
  __shared__ uint32_t s_tmem;
  __shared__ int32_t s_count, s_share;
  __shared__ bool s_many;
  __shared__ int2 s_lists[kWarps][kGroups<CONSTW>];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int RS = RSW;  // (the zero columns are at a.Q, whatever the stride)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (tid == kWarps * 32 - 32) fetch_next_lists(a);
  // Engines that work side by side take a share of the SMs each: a CTA fills
  // its SM, and of launches over all SMs one waits for the other, round trips
  // and all.  (The number is set before the inference's first launch.)  A
  // server of 4 slots at 2000 requests a second: median latency 12.2 -> 7.8 ms
  // with merging, 11.9 -> 5.8 without.
  auto grid_of = [&](unsigned share) { return max((unsigned)f.teams / share, 1u) * plan_split; };
  // ---- before the previous launch has ended: nothing it writes is relied on.
  // Each warp sets up a part, the loads beside the taking of tensor memory (0.8
  // us): one after the other, a layer that no row reaches -- every one after the
  // last row has died -- took 2.65 us, now 1.9; the kernel with lists streamed
  // per tile takes 1.55.  (Taking it only once rows are known to come: 1.8, but
  // 0.8 more where they do.  A warp more to read the count meanwhile: 1.75, but
  // 96 registers a thread, 2 % of a layer of many rows.)
  if (warp == 0) {
    // Where there are many rows, the lists are kept before the previous launch
    // has ended.  That is then known only roughly (the counts may still grow): a
    // wrong guess costs time, not results.
    int rows = a.rows, share = 1;
    if (a.hint) rows = max(__ldcg(a.hint), __ldcg(a.count_in));
    if (a.share) share = __ldcg(a.share);
    if (lane == 0) {
      s_many = rows > f.few / share;
      s_share = share;
    }
  } else if (warp == 1) {
    if (!a.share || blockIdx.x < grid_of(__ldcg(a.share))) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                       smem_u32(&s_tmem))
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
  } else if (warp == 2) {
    if (lane < kMaxStages) {
      mbar_init(&full[lane], 1);
      s_mask[lane] = 0;
      s_done[lane] = 0;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  } else {
    for (int i = warp - 3; i < T * stages; i += kWarps - 3) ring[(size_t)i * RS + a.Q + lane] = 0.f;
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_tmem;
  const unsigned share = (unsigned)s_share, grid = grid_of(share);
  if (blockIdx.x >= grid) return;
  const unsigned few = (unsigned)f.few / share;
  // the warp's columns: its quarter of the lanes, 128 of the 512 columns
  const uint32_t col = tmem + ((uint32_t)(warp & 3) << 21) + (uint32_t)(warp >> 2) * kCols;
  // The CTAs of a tile (its "split"), and with it the groups of this warp.
  int split = 0, part, team, teams, first_grp, step0, step1, n = 0;
  Batch<CONSTW> cur;
  auto assign = [&](int sp) {
    split = sp;
    part = blockIdx.x % sp, team = blockIdx.x / sp, teams = grid / sp;
    // Groups come in order of depth (degree order), so the warps take them
    // there and back: warp w the w-th, the (31 - w)-th, the (32 + w)-th, ...
    first_grp = warp * sp + part;
    step0 = (2 * kWarps - 1 - 2 * warp) * sp, step1 = (2 * warp + 1) * sp;
  };
  // (every load of a group in flight before the first is stored: a list is two
  // round trips, not one for every few blocks)
  auto keep_lists = [&]() {
    constexpr int NB = kResBlocks<CONSTW>;
    int2 list[kGroups<CONSTW>];
    int g = first_grp;
    n = 0;
#pragma unroll
    for (int i = 0; i < kGroups<CONSTW>; ++i) {
      if (g < a.G) {
        list[i] = __ldg(a.w.lists + g);
        if (lane == 0) s_lists[warp][i] = list[i];
        n = i + 1;
      }
      g += (i & 1) ? step1 : step0;
    }
#pragma unroll
    for (int i = 0; i < kGroups<CONSTW>; ++i) {
      if (i < n) {
        const int nb = (list[i].y + 3) >> 2;
        const size_t at = (size_t)list[i].x * 32 + lane;
        const uint32_t to = col + i * kGroupCols<CONSTW>;
        uint2 iv[NB];
#pragma unroll
        for (int b = 0; b < NB; ++b)
          if (b < nb) iv[b] = __ldg(a.w.idx + at + (size_t)b * 32);
        if constexpr (!CONSTW) {
          float4 vv[NB];
#pragma unroll
          for (int b = 0; b < NB; ++b)
            if (b < nb) vv[b] = __ldg(a.w.val + at + (size_t)b * 32);
#pragma unroll
          for (int b = 0; b < NB; ++b)
            if (b < nb) tmem_st4(to + 2 * NB + 4 * b, vv[b]);
        }
#pragma unroll
        for (int b = 0; b < NB; ++b)
          if (b < nb) tmem_st2(to + 2 * b, iv[b]);
      }
    }
    tmem_wait_st();
    __syncwarp();
    cur.load(col, 0);
    cur.wait();
  };
  if (s_many) {
    assign(plan_split);
    keep_lists();
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (tid == 0) s_count = __ldcg(a.count_in);
  __syncthreads();
  const unsigned count = (unsigned)s_count;
  if (count == 0) {
    if (warp == 1) tmem_free(tmem);
    return;
  }
  unsigned TE, tiles;
  int sp = plan_split;
  if (count > few) {
    // Rows per tile: as many as still give every team a tile, the last round of
    // tiles full (TE = 1 .. T).
    const unsigned all = grid / plan_split;
    const unsigned rounds = max(1u, (count + T * all - 1) / (T * all));
    TE = min((unsigned)T, max(1u, (count + rounds * all - 1) / (rounds * all)));
    tiles = (count + TE - 1) / TE;
  } else {
    // Few rows: one tile per CTA, and as many CTAs to a tile as there are, so
    // that a CTA fetches few lists (few_rows() has the sizes).
    const unsigned like = count * share;
    TE = like <= (unsigned)f.cap[0] ? 1 : like <= (unsigned)f.cap[1] ? 2 : like <= (unsigned)f.cap[2] ? 4 : T;
    tiles = (count + TE - 1) / TE;
    sp = max((unsigned)plan_split, min(grid / max(1u, tiles), (unsigned)f.most));
  }
  const bool late = sp != split;
  if (late) assign(sp);
  const int mine =
      team < (int)min((unsigned)teams, tiles) ? (int)((tiles - team + teams - 1) / (unsigned)teams) : 0;
  // Lists the rows of this CTA's k-th tile and starts their copies into stage s
  // (one warp).
  auto load = [&](int k, int s) {
    const long long r0 = (long long)(team + (long long)k * teams) * TE;
    const int nrows = (int)min((long long)TE, (long long)count - r0);
    const int row = lane < nrows ? a.list_in[r0 + lane] : -1;
    if (lane < T) s_rows[s][lane] = row;
    __syncwarp();
    const uint32_t bytes = (uint32_t)a.N * 4u;
    if (lane == 0) mbar_expect_tx(&full[s], bytes * (uint32_t)nrows);
    __syncwarp();
    if (lane < nrows)
      bulk_g2s(ring + (size_t)(s * T + lane) * RS, a.y_in + (size_t)row * a.N, bytes, &full[s]);
  };
  if (warp < stages && warp < mine) load(warp, warp);
  if (late && mine > 0) keep_lists();
  int s = 0;
  uint32_t phase = 0;
  bool ok = true;
  for (int k = 0; k < mine; ++k) {
    ok = mbar_wait_bounded(&full[s], phase, a.err);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) break;
    const long long r0 = (long long)(team + (long long)k * teams) * TE;
    const int nrows = (int)min((long long)TE, (long long)count - r0);
    uint32_t m = run_stage<T, RSW, CONSTW>(TE, a, ring + (size_t)s * T * RS, RS, s_rows[s], nrows,
                                           col, cur, s_lists[warp], first_grp, step0, step1, n, lane);
    m = __reduce_or_sync(0xffffffffu, m);
    int before = 0;
    if (lane == 0) {
      if (m) atomicOr(&s_mask[s], m);
      __threadfence_block();
      before = atomicAdd(&s_done[s], 1);
    }
    before = __shfl_sync(0xffffffffu, before, 0);
    if (before == kWarps - 1) {
      // every warp is done with the tile
      __threadfence_block();
      const uint32_t mask = s_mask[s];
      publish_rows(a, mask, split > 1, s_rows[s], lane);
      __syncwarp();
      if (lane == 0) {
        s_mask[s] = 0;
        s_done[s] = 0;
      }
      __syncwarp();
      if (k + stages < mine) load(k + stages, s);
    }
    if (++s == stages) {
      s = 0;
      phase ^= 1u;
    }
  }
  __syncthreads();
  if (warp == 1) tmem_free(tmem);
}

// Row strides of the widths without one of their own (their indices are in
// floats), each for the widths that it holds with the zero columns.
constexpr int kStride1536 = 1568, kStride2368 = 2400, kStride4064 = 4096;

struct Instance {
  int T, rsw;
  bool constw;
  const void* fn;
};
#define SDNN_RESIDENT(T, RSW) \
  {T, RSW, true, (const void*)&layer_resident_kernel<T, RSW, true>}, \
      {T, RSW, false, (const void*)&layer_resident_kernel<T, RSW, false>}
const Instance kInstances[] = {SDNN_RESIDENT(8, 1056), SDNN_RESIDENT(8, kStride1536),
                               SDNN_RESIDENT(8, kStride2368), SDNN_RESIDENT(6, kStride4064),
                               SDNN_RESIDENT(6, 4128)};

const void* find_instance(int T, int rsw, bool constw) {
  for (const Instance& e : kInstances)
    if (e.T == T && e.rsw == rsw && e.constw == constw) return e.fn;
  return nullptr;
}

}  // namespace

// A launch of few rows is the time to fetch the lists, so up to `few` rows (a
// tile for every other team) more CTAs share a tile than must.  Of the tile
// sizes, the one with the fewest bytes to fetch per CTA, rows and lists
// together; at least 4 groups are left to a CTA, one for each scheduler.  A list
// counts as 44 slots whatever it holds: what it costs is round trips more than
// bytes.  With the layer's own list sizes 40 layers took 212 -> 293 us (55 rows
// of 4096, 4 edges an input), 306 -> 383 (120 of 1024, 80 edges), and the same
// within 2 % at 32 edges.
static FewRows few_rows(const ResidentPlan& p, int N, bool constw, int num_sms) {
  FewRows f{};
  const int G = N / 32, list_bytes = 44 * 32 * (constw ? 2 : 6);
  f.teams = std::max(1, num_sms / p.split);
  f.most = std::max(p.split, G / 4);
  f.few = p.T * f.teams / 2;
  const int grid = f.teams * p.split;
  for (int count = 1; count <= f.few; ++count) {
    long least = LONG_MAX;
    int best = 3;
    for (int i = 3; i >= 0; --i) {
      const int te = i == 3 ? p.T : 1 << i, tiles = (count + te - 1) / te;
      const int split = std::min(grid / tiles, f.most);
      const long bytes = (long)te * N * 4 + (long)((G + split - 1) / std::max(1, split)) * list_bytes;
      if (split >= p.split && bytes < least) {
        least = bytes;
        best = i;
      }
    }
    for (int i = best; i < 3; ++i) f.cap[i] = count;
  }
  return f;
}

ResidentPlan resident_plan(int N, bool constw, int max_depth, int num_sms) {
  ResidentPlan p{};
  const int G = N / 32;
  const int per_cta = kWarps * (constw ? kGroups<true> : kGroups<false>);
  const int held = 4 * (constw ? kResBlocks<true> : kResBlocks<false>);
  if (N % 32 != 0 || N < 1024 || N > 4096 || max_depth > 2 * held) return p;
  p.split = (G + per_cta - 1) / per_cta;
  // Strides are known when compiling: every gather then has its row's offset as
  // an immediate (60000 rows, us, stride N + 32 at run time -> one of these:
  // 2048 neurons 563 -> 531, 4064 1168 -> 1094, with values 1509 -> 1380; 3072
  // with values 1147 -> 1040, where lists streamed per tile took 1084).
  p.rsw = N == 1024 ? 1056
          : N == 4096 ? 4128
          : N <= kStride1536 - 32 ? kStride1536
          : N <= kStride2368 - 32 ? kStride2368
                                  : kStride4064;
  const size_t row = (size_t)p.rsw * 4;
  // 8 rows where three stages of them fit, else two stages of 6: at N = 4096
  // three stages of 4 rows took 1208 us for 60000 rows, two of 6 1119 (fewer
  // list words and group turns per row); at N = 1024 16 rows are no faster than
  // 8 (285 against 290 us) and leave more of the last round empty (10000 rows:
  // 76 against 64 us).
  p.T = 3 * 8 * row <= kResSmem ? 8 : 6;
  p.stages = (int)std::min<size_t>(kMaxStages, kResSmem / (p.T * row));
  p.smem = p.stages * p.T * row;
  p.fn = find_instance(p.T, p.rsw, constw);
  // A warp with one group more than the others holds up its CTA: just past a
  // width that fills the warps' turns, lists streamed per tile are faster for
  // many rows (60000 rows, us, streamed against kept: 1056 neurons with values
  // 411 against 507, 1088 429 against 477; 2080 with one value 660 against 707,
  // with values 719 against 751; 1056 with one value 361 against 363, but its
  // residue layers 2543 against 2631).  Up to 4096 rows they are level or slower
  // (300 rows, 40 layers: 366 against 303).
  const int turns = p.split * kWarps * ((G + p.split * kWarps - 1) / (p.split * kWarps));
  if (G < 0.7 * turns) p.most_rows = 4096;
  p.few = few_rows(p, N, constw, num_sms);
  return p;
}

cudaError_t resident_prepare(const ResidentPlan& p) { return allow_smem(p.fn); }

cudaError_t launch_layer_resident(const ResidentPlan& p, const LayerArgs& a, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.few.teams * p.split);
  cfg.blockDim = dim3(kWarps * 32);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = a.share ? 0 : 1;  // (CTAs that wait would hold another engine's SMs)
  int split = p.split, stages = p.stages;
  FewRows f = p.few;
  void* args[] = {const_cast<LayerArgs*>(&a), &split, &stages, &f};
  return cudaLaunchKernelExC(&cfg, p.fn, args);
}

}  // namespace sdnn
