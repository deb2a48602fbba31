// First-layer kernel for binary inputs (the SDGC input images are 0/1).
//
// When every input of a row is 0 or 1 and the layer has one common weight
// value w, the pre-activation of output c is S(k) + b, where k is the number
// of active in-edges of c and S(k) is w added k times in FP32 -- exactly what
// the float gather (the layer kernels, which add w * 1 or w * 0 slot by slot)
// computes.  This kernel therefore counts instead of multiplying:
//
//  * bits_transpose_kernel turns tiles of 32 rows into one 32-bit word per input
//    (bit t is input j of row t), 1024 inputs a unit, coalesced 16-byte loads, 8
//    rows in flight per lane; the words go to global memory (1/32 of the rows),
//    and a tile that holds any value other than 0 or 1 is flagged;
//  * bits_count_kernel (whole rows) and bits_count_chunked_kernel (input chunks)
//    take (tile, part of the groups) items: the tile's words come into shared
//    memory by TMA (N + 32 words, the last 32 zero for the padding slots), and
//    lane i of a warp owns output 32g + i and walks the same bank-scheduled
//    slots as the layer kernels, loading one word per slot (one wavefront per slot
//    for all 32 rows) and adding it into bit-sliced counters with a Harley-Seal
//    carry-save tree (15 full adders per 16 slots);
//  * the epilogue extracts each row's count, looks up S(k) (a 128-entry table
//    built on the host with the same FP32 additions), adds the bias, clamps,
//    stores row t coalesced and lists the surviving rows.
//
// The rows of a flagged tile are not computed here: they go to a fallback list
// that the float kernel processes right after.
//
// Both passes move bytes: the rows in, the rows out.  One kernel for both, a
// CTA per tile, kept neither DRAM direction busy (its CTAs alternated between
// reading, counting and writing) and left SMs without a tile when there were
// few: 60000 rows of 4096 neurons 486 us, 6001 of 16384 299; now 400 and 202
// (the transposes 179 and 83 of them, at 5.5 TB/s; the rows in and out take 290
// and 116 at the copy rate).
#include <algorithm>
#include <cstdint>
#include "layer_kernel.cuh"

namespace sdnn {

__device__ __forceinline__ void csa(uint32_t& h, uint32_t& l, uint32_t a, uint32_t b, uint32_t c) {
  const uint32_t u = a ^ b;
  h = (a & b) | (u & c);
  l = u ^ c;
}

// Bit-sliced counters c[0..6] (c[i] bit t = bit i of row t's count) plus 16,
// 8 or 4 words, each word adding 1 to the rows whose bit is set: Harley-Seal
// carry-save trees, the carry out of the tree rippled into the higher planes.
__device__ __forceinline__ void ripple(uint32_t (&c)[7], int from, uint32_t cy) {
#pragma unroll
  for (int i = 0; i < 7; ++i) {
    if (i < from) continue;
    const uint32_t t = c[i] & cy;
    c[i] ^= cy;
    cy = t;
  }
}
__device__ __forceinline__ void add16(uint32_t (&c)[7], const uint32_t (&w)[16]) {
  uint32_t twosA, twosB, foursA, foursB, eightsA, eightsB, c16;
  csa(twosA, c[0], c[0], w[0], w[1]);
  csa(twosB, c[0], c[0], w[2], w[3]);
  csa(foursA, c[1], c[1], twosA, twosB);
  csa(twosA, c[0], c[0], w[4], w[5]);
  csa(twosB, c[0], c[0], w[6], w[7]);
  csa(foursB, c[1], c[1], twosA, twosB);
  csa(eightsA, c[2], c[2], foursA, foursB);
  csa(twosA, c[0], c[0], w[8], w[9]);
  csa(twosB, c[0], c[0], w[10], w[11]);
  csa(foursA, c[1], c[1], twosA, twosB);
  csa(twosA, c[0], c[0], w[12], w[13]);
  csa(twosB, c[0], c[0], w[14], w[15]);
  csa(foursB, c[1], c[1], twosA, twosB);
  csa(eightsB, c[2], c[2], foursA, foursB);
  csa(c16, c[3], c[3], eightsA, eightsB);
  ripple(c, 4, c16);
}
__device__ __forceinline__ void add8(uint32_t (&c)[7], const uint32_t* w) {
  uint32_t twosA, twosB, foursA, foursB, eights;
  csa(twosA, c[0], c[0], w[0], w[1]);
  csa(twosB, c[0], c[0], w[2], w[3]);
  csa(foursA, c[1], c[1], twosA, twosB);
  csa(twosA, c[0], c[0], w[4], w[5]);
  csa(twosB, c[0], c[0], w[6], w[7]);
  csa(foursB, c[1], c[1], twosA, twosB);
  csa(eights, c[2], c[2], foursA, foursB);
  ripple(c, 3, eights);
}
__device__ __forceinline__ void add4(uint32_t (&c)[7], const uint32_t* w) {
  uint32_t twosA, twosB, fours;
  csa(twosA, c[0], c[0], w[0], w[1]);
  csa(twosB, c[0], c[0], w[2], w[3]);
  csa(fours, c[1], c[1], twosA, twosB);
  ripple(c, 2, fours);
}

// Index words of K blocks (block b0 onwards; indices ip, lane-strided).
template <int K>
__device__ __forceinline__ void load_slots(uint2* iv, const uint2* __restrict__ ip, int b0) {
#pragma unroll
  for (int k = 0; k < K; ++k) iv[k] = __ldg(ip + (size_t)(b0 + k) * 32);
}
// Bit words of their slots from the shared row `bits` (BYTES: indices are byte
// offsets).
template <bool BYTES, int K>
__device__ __forceinline__ void gather_words(uint32_t* w, const uint2* iv, const uint32_t* bits) {
#pragma unroll
  for (int k = 0; k < K; ++k) {
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const uint32_t j = ((s < 2 ? iv[k].x : iv[k].y) >> ((s & 1) * 16)) & 0xffffu;
      w[k * 4 + s] = BYTES ? *reinterpret_cast<const uint32_t*>(
                                 reinterpret_cast<const char*>(bits) + j)
                           : bits[j];
    }
  }
}

// Adds the slots of a list of nb blocks into the counters: 4 blocks at a
// time, then 2, then 1 (no adder work on blocks past the list's end).  head
// holds the list's first four blocks (those it has).
template <bool BYTES>
__device__ __forceinline__ void count_list(uint32_t (&c)[7], const uint2 (&head)[4],
                                           const uint2* __restrict__ ip, int nb,
                                           const uint32_t* bits) {
  uint2 iv[4];
  int b = 0;
  if (nb >= 4) {
    uint32_t w[16];
    if (nb >= 8) load_slots<4>(iv, ip, 4);
    gather_words<BYTES, 4>(w, head, bits);
    add16(c, w);
    for (b = 4; b + 4 <= nb; b += 4) {
      gather_words<BYTES, 4>(w, iv, bits);
      if (b + 8 <= nb) load_slots<4>(iv, ip, b + 4);
      add16(c, w);
    }
    if (b + 2 <= nb) load_slots<2>(iv, ip, b);
    if ((nb - b) & 1) load_slots<1>(iv + 2, ip, nb - 1);
  } else {
    iv[0] = head[0];
    iv[1] = head[1];
    iv[2] = nb == 3 ? head[2] : head[0];
  }
  if (b + 2 <= nb) {
    uint32_t w[8];
    gather_words<BYTES, 2>(w, iv, bits);
    add8(c, w);
  }
  if ((nb - b) & 1) {
    uint32_t w[4];
    gather_words<BYTES, 1>(w, iv + 2, bits);
    add4(c, w);
  }
}
// The same for the lists of an input chunk (float indices; about four blocks,
// nothing fetched ahead: the counters of four groups fill the registers).
__device__ __forceinline__ void count_short_list(uint32_t (&c)[7], const uint2* __restrict__ ip,
                                                 int nb, const uint32_t* bits) {
  uint2 iv[4];
  int b = 0;
  for (; b + 4 <= nb; b += 4) {
    uint32_t w[16];
    load_slots<4>(iv, ip, b);
    gather_words<false, 4>(w, iv, bits);
    add16(c, w);
  }
  if (b + 2 <= nb) {
    uint32_t w[8];
    load_slots<2>(iv, ip, b);
    gather_words<false, 2>(w, iv, bits);
    add8(c, w);
    b += 2;
  }
  if (b < nb) {
    uint32_t w[4];
    load_slots<1>(iv, ip, b);
    gather_words<false, 1>(w, iv, bits);
    add4(c, w);
  }
}
// The first blocks of a list of nb.
__device__ __forceinline__ void load_head(uint2 (&head)[4], const uint2* __restrict__ ip, int nb) {
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (k < nb) head[k] = __ldg(ip + (size_t)k * 32);
}

// ---- epilogue: per-row counts out of the bit-sliced counters ----------------
//
// Rows of a tile are bits of the counter planes P[0..6] (P[i] bit t = bit i of
// row t's count).  With a scalar bias the output of a row depends on its count
// only, through a 128-entry table, and the rows that survive are those whose
// count lies in an interval, so:
//  * the survivor mask of all 32 rows comes from bitwise comparisons of the
//    planes with the interval's end (no per-row vote);
//  * the counts come out of one 8 x 8 bit-matrix transpose of the eight plane
//    registers, all four bytes of them at once (the block-swap transpose of
//    Hacker's Delight, section 7-3): register r then holds, in byte b, the
//    count of row 8 b + r.  Where no output has 64 in-edges or more, six planes
//    go in at bits 2 .. 7 and a byte is the table's byte offset.
// What bounds the counting pass is the ALU: with a transpose per byte of the
// planes it took 491 of its instructions per (tile, group), now 330, and a row's
// offset is an immediate since the rows of layer 0 are consecutive.

// Rows whose count is >= k0 (k0 in 0..128).
__device__ __forceinline__ uint32_t count_ge(const uint32_t (&P)[7], uint32_t k0) {
  if (k0 >= 128u) return 0u;
  uint32_t gt = 0u, eq = 0xffffffffu;
#pragma unroll
  for (int i = 6; i >= 0; --i) {
    if ((k0 >> i) & 1u) eq &= P[i];
    else gt |= eq & P[i];
  }
  return gt | eq;
}

// Bit i of byte b of R[r] <- bit r of byte b of R[i], for every byte b.
__device__ __forceinline__ void transpose8(uint32_t (&R)[8]) {
#pragma unroll
  for (int step = 4; step > 0; step >>= 1) {
    const uint32_t mask = step == 4 ? 0x0f0f0f0fu : step == 2 ? 0x33333333u : 0x55555555u;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (i & step) continue;
      const uint32_t t = ((R[i] >> step) ^ R[i + step]) & mask;
      R[i + step] ^= t;
      R[i] ^= t << step;
    }
  }
}

// Survivor interval of the counts for a scalar bias: kind 1 = [k0, 127],
// kind 2 = [0, k1]; kind 0 = per-neuron bias or no interval (generic path).
struct CountInterval {
  int kind;
  uint32_t lo, hi;
};

__device__ CountInterval count_interval(const float* s_sum, float bias, bool per_neuron) {
  __shared__ uint32_t s_alive[4];
  __shared__ CountInterval s_iv;
  const int tid = threadIdx.x;
  if (tid < 128) {
    const uint32_t m = __ballot_sync(0xffffffffu, s_sum[tid] + bias > 0.f);
    if ((tid & 31) == 0) s_alive[tid >> 5] = m;
  }
  __syncthreads();
  if (tid == 0) {
    CountInterval iv{0, 0u, 0u};
    if (!per_neuron) {
      // alive counts as a 128-bit set; suffix [k0, 127] or prefix [0, k1]?
      int first = -1, last = -1;
      for (int k = 0; k < 128; ++k)
        if ((s_alive[k >> 5] >> (k & 31)) & 1u) {
          if (first < 0) first = k;
          last = k;
        }
      int n = 0;
      for (int w = 0; w < 4; ++w) n += __popc(s_alive[w]);
      if (first < 0) {
        iv = {1, 128u, 0u};  // nothing survives: k >= 128 never holds
      } else if (n == last - first + 1 && last == 127) {
        iv = {1, (uint32_t)first, 0u};
      } else if (n == last - first + 1 && first == 0) {
        iv = {2, 0u, (uint32_t)last};
      }
    }
    s_iv = iv;
  }
  __syncthreads();
  return s_iv;
}

// Outputs row 8 b + r of the tile <- the table entry of byte b of R[r], rows
// below nrows.  NC: neurons when known (the rows' offsets are then immediate).
template <int NC, bool FEW, bool FULL>
__device__ __forceinline__ void store_counts(const uint32_t (&R)[8], const float* s_val, float* out,
                                             int N, int nrows) {
#pragma unroll
  for (int b = 0; b < 4; ++b) {
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int t = 8 * b + r;
      if (FULL || t < nrows) {
        const uint32_t k = __byte_perm(R[r], 0u, 0x4440 | b);
        const float v = FEW ? *reinterpret_cast<const float*>(reinterpret_cast<const char*>(s_val) + k)
                            : s_val[k];
        out[(size_t)t * (NC > 0 ? NC : N)] = v;
      }
    }
  }
}

// Outputs of one group for the rows of a tile (row0 onwards) from its counters.
template <int NC>
__device__ __forceinline__ uint32_t bits_epilogue(const uint32_t (&P)[7], const Layer0Args& a,
                                                  const float* s_sum, const float* s_val,
                                                  const CountInterval& iv, int row0, int nrows,
                                                  int c_out) {
  const int N = NC > 0 ? NC : a.N;
  float* out = a.y_out + (size_t)row0 * N + c_out;
  uint32_t m = 0;
  if (iv.kind != 0) {
    const uint32_t rows_mask = nrows >= 32 ? 0xffffffffu : ((1u << nrows) - 1u);
    uint32_t alive = iv.kind == 1 ? count_ge(P, iv.lo) : ~count_ge(P, iv.hi + 1u);
    m = alive & rows_mask;
    const bool few = a.max_count < 64;  // counts fit six planes
    uint32_t R[8];
    R[0] = few ? 0u : P[0];
    R[1] = few ? 0u : P[1];
#pragma unroll
    for (int i = 2; i < 8; ++i) R[i] = few ? P[i - 2] : (i < 7 ? P[i] : 0u);
    transpose8(R);
    if (few && nrows == 32) store_counts<NC, true, true>(R, s_val, out, N, nrows);
    else if (few) store_counts<NC, true, false>(R, s_val, out, N, nrows);
    else store_counts<NC, false, false>(R, s_val, out, N, nrows);
    return m;
  }
  const float bc = a.bias_vec ? __ldg(a.bias_vec + c_out) : a.bias;
  for (int t = 0; t < nrows; ++t) {
    uint32_t k = 0;
#pragma unroll
    for (int i = 0; i < 7; ++i) k |= ((P[i] >> t) & 1u) << i;
    const float v = s_sum[k] + bc;
    out[(size_t)t * N] = clampf(v, a.clampv);
    if (v > 0.f) m |= 1u << t;
  }
  return m;
}

constexpr int kChunkGroupsPerWarp = 4;
constexpr int kChunkWarps = 16;
constexpr int kTransposeThreads = 256;
constexpr int kTransposeInputs = 4 * kTransposeThreads;  // inputs of a unit

__global__ void __launch_bounds__(kTransposeThreads) bits_transpose_kernel(const Layer0Args a) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int tid = threadIdx.x, lane = tid & 31;
  const int N = a.N;
  const int count = *a.count_in;
  const int n_tiles = (count + 31) / 32;
  const int per_tile = (N + kTransposeInputs - 1) / kTransposeInputs;
  const long units = (long)n_tiles * per_tile;
  for (long unit = blockIdx.x; unit < units; unit += gridDim.x) {
    const int tile = (int)(unit / per_tile), block = (int)(unit % per_tile);
    const int row0 = tile * 32;
    const int nrows = min(32, count - row0);
    const int j = block * kTransposeInputs + tid * 4;
    const float* in = a.y_in + (size_t)(a.first_row + row0) * N + j;
    bool nonbin = false;
    if (j < N) {
      uint32_t w0 = 0, w1 = 0, w2 = 0, w3 = 0;
#pragma unroll 1
      for (int t0 = 0; t0 < nrows; t0 += 8) {
        float4 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (t0 + u < nrows)
            v[u] = __ldg(reinterpret_cast<const float4*>(in + (size_t)(t0 + u) * N));
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          if (t0 + u < nrows) {
            const float x[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
            for (int q = 0; q < 4; ++q) nonbin |= (x[q] != 0.f) && (x[q] != 1.f);
            const uint32_t bit = 1u << (t0 + u);
            w0 |= x[0] != 0.f ? bit : 0u;
            w1 |= x[1] != 0.f ? bit : 0u;
            w2 |= x[2] != 0.f ? bit : 0u;
            w3 |= x[3] != 0.f ? bit : 0u;
          }
        }
      }
      *reinterpret_cast<uint4*>(a.bits + (size_t)tile * N + j) = make_uint4(w0, w1, w2, w3);
    }
    if (__any_sync(0xffffffffu, nonbin) && lane == 0) a.tile_state[tile] = 1;
  }
}

// The same words from rows that came as bits: a warp takes 64 inputs of a tile,
// a word per row and lane, and transposes two squares of 32 x 32 bits.  It moves
// 1/4 of a byte per input, bits in and words out; expanding 60000 rows of 1024
// inputs to floats and reading those back took 102 us (the whole call 1829 ->
// 1722).
__global__ void __launch_bounds__(kTransposeThreads) bit_rows_transpose_kernel(const Layer0Args a) {
  pdl_prologue();
  const int lane = threadIdx.x & 31, N = a.N;
  const int count = *a.count_in, n_tiles = (count + 31) / 32, W = (N + 63) / 64;
  const long units = (long)n_tiles * W;
  const long warps = (long)gridDim.x * (kTransposeThreads / 32);
  for (long unit = blockIdx.x * (long)(kTransposeThreads / 32) + (threadIdx.x >> 5); unit < units;
       unit += warps) {
    const int tile = (int)(unit / W), w = (int)(unit % W), row = tile * 32 + lane;
    const auto* rows = reinterpret_cast<const unsigned long long*>(a.bit_rows);
    const uint64_t word = row < count ? __ldcg(rows + (size_t)(a.first_row + row) * W + w) : 0ull;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      uint32_t x = (uint32_t)(word >> (32 * half));
#pragma unroll
      for (int k = 16; k > 0; k >>= 1) {
        // the low k bits of every 2k
        const uint32_t low = k == 16  ? 0x0000ffffu
                             : k == 8 ? 0x00ff00ffu
                             : k == 4 ? 0x0f0f0f0fu
                             : k == 2 ? 0x33333333u
                                      : 0x55555555u;
        const uint32_t y = __shfl_xor_sync(0xffffffffu, x, k);
        x = lane & k ? (x & ~low) | ((y & ~low) >> k) : (x & low) | ((y & low) << k);
      }
      const int j = w * 64 + half * 32 + lane;
      if (j < N) a.bits[(size_t)tile * N + j] = x;
    }
  }
}

// Rows of a tile that are flagged in m to the next list (one warp); parts of a
// tile run on other CTAs when it is shared, and the first to mark a row lists it.
__device__ __forceinline__ void list_rows(const Layer0Args& a, uint32_t m, bool shared, int row0,
                                          int lane) {
  bool mine = (m >> lane) & 1u;
  const int row = a.first_row + row0 + lane;
  if (shared && mine) mine = atomicExch(a.stamp + row, a.stamp_id) != a.stamp_id;
  const uint32_t w = __ballot_sync(0xffffffffu, mine);
  if (!w) return;
  int at = 0;
  if (lane == 0) at = atomicAdd(a.count_out, __popc(w));
  at = __shfl_sync(0xffffffffu, at, 0) + __popc(w & ((1u << lane) - 1u));
  if (mine) a.list_out[at] = row;
}

// A flagged tile: its rows to the fallback list (by the CTA of its first part).
__device__ __forceinline__ void list_fallback(const Layer0Args& a, int row0, int nrows, int lane) {
  int at = 0;
  if (lane == 0) at = atomicAdd(a.fallback_count, nrows);
  at = __shfl_sync(0xffffffffu, at, 0);
  if (lane < nrows) a.fallback_list[at + lane] = a.first_row + row0 + lane;
}

// Whole rows of words in shared memory.  256 threads, up to four CTAs per SM:
// one CTA's load and stores overlap another's counting.
constexpr int kCountWarps = 8;
// Buffers of words: the next item's are copied while one is counted, unless
// that would cost CTAs.
__host__ __device__ constexpr int count_buffers(int N) { return N <= 4096 ? 2 : 1; }
template <int RSW>
__global__ void __launch_bounds__(kCountWarps * 32, 4) bits_count_kernel(const Layer0Args a) {
  extern __shared__ __align__(128) uint32_t bits[];  // [bufs][RSW] words
  constexpr int bufs = count_buffers(RSW - 32);
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ float s_sum[128];
  __shared__ float s_val[128];  // output of a row with count k (scalar bias)
  __shared__ uint32_t s_mask;
  __shared__ int32_t s_fail;

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int N = a.N;
  if (tid < 128) {
    s_sum[tid] = a.sums[tid];
    s_val[tid] = clampf(a.sums[tid] + a.bias, a.clampv);
  }
  if (tid < 32 * bufs) bits[(tid >> 5) * RSW + N + lane] = 0u;
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    s_mask = 0;
    s_fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  const CountInterval iv = count_interval(s_sum, a.bias, a.bias_vec != nullptr);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int count = *a.count_in;
  const int n_tiles = (count + 31) / 32;
  if (n_tiles == 0) return;
  // parts of a tile: about four items per CTA, a group per warp at least
  const int parts = max(1, min((a.G + kCountWarps - 1) / kCountWarps,
                               (int)((4 * gridDim.x + n_tiles - 1) / n_tiles)));
  const long items = (long)n_tiles * parts;
  // copies the words of an item's tile into buffer s (one thread)
  auto start = [&](long it, int s) {
    const uint32_t bytes = (uint32_t)N * 4u;
    mbar_expect_tx(&bar[s], bytes);
    const char* src = reinterpret_cast<const char*>(a.bits + (size_t)(it / parts) * N);
    char* dst = reinterpret_cast<char*>(bits + (size_t)s * RSW);
    for (uint32_t off = 0; off < bytes; off += 32768u)
      bulk_g2s(dst + off, src + off, min(32768u, bytes - off), &bar[s]);
  };
  uint32_t phases = 0;  // bit s: phase of bar[s]
  int buf = 0;
  bool started = false;
  for (long item = blockIdx.x; item < items; item += gridDim.x) {
    const int tile = (int)(item / parts), part = (int)(item % parts);
    const int row0 = tile * 32;
    const int nrows = min(32, count - row0);
    if (a.tile_state[tile]) {  // (the same for every thread)
      if (part == 0 && warp == 0) list_fallback(a, row0, nrows, lane);
      continue;
    }
    const int gbeg = (int)((long)a.G * part / parts), gend = (int)((long)a.G * (part + 1) / parts);
    // the first list of the warp's groups, on its way while the words are
    int32_t b0 = 0, nb = 0;
    uint2 head[4];
    auto fetch = [&](int g) {
      b0 = __ldg(a.grp_blk + g);
      nb = __ldg(a.grp_blk + g + 1) - b0;
      load_head(head, a.idx + (size_t)b0 * 32 + lane, nb);
    };
    if (gbeg + warp < gend) fetch(gbeg + warp);
    __syncthreads();  // every warp is done with the item before
    if (tid == 0) {
      // this item's words unless the item before has started them, and the
      // next one's where there are two buffers
      if (!started) start(item, buf);
      started = false;
      if (bufs == 2) {
        long next = item + gridDim.x;
        while (next < items && a.tile_state[next / parts]) next += gridDim.x;
        if (next < items) {
          start(next, buf ^ 1);
          started = true;
        }
      }
      if (!mbar_wait_bounded(&bar[buf], (phases >> buf) & 1u, a.err)) s_fail = 1;
    }
    __syncthreads();
    if (s_fail) return;
    mbar_try_wait(&bar[buf], (phases >> buf) & 1u);
    phases ^= 1u << buf;
    const uint32_t* words = bits + (size_t)buf * RSW;
    if (bufs == 2) buf ^= 1;
    uint32_t m = 0;
    for (int g = gbeg + warp; g < gend; g += kCountWarps) {
      uint32_t P[7] = {0u, 0u, 0u, 0u, 0u, 0u, 0u};
      count_list<rsw_in_bytes(RSW)>(P, head, a.idx + (size_t)b0 * 32 + lane, nb, words);
      // the next group's list is fetched while this one's outputs are stored
      if (g + kCountWarps < gend) fetch(g + kCountWarps);
      m |= bits_epilogue<RSW - 32>(P, a, s_sum, s_val, iv, a.first_row + row0, nrows, g * 32 + lane);
    }
    m = __reduce_or_sync(0xffffffffu, m);
    if (lane == 0 && m) atomicOr(&s_mask, m);
    __syncthreads();
    if (warp == 0) {
      list_rows(a, s_mask, parts > 1, row0, lane);
      __syncwarp();
      if (lane == 0) s_mask = 0;
    }
  }
}

// ---------------------------------------------------------------------------
// Input chunks (N > 16384: a row of bit words does not fit shared memory): an
// item is (tile, subset of groups); for each input chunk the CTA copies the
// chunk's Q words into shared memory (TMA bulk copy) and every warp adds the
// slots of its groups into bit-sliced counters that stay in registers across
// the chunks; after the last chunk the epilogue is the one of bits_count_kernel.
__global__ void __launch_bounds__(kChunkWarps * 32) bits_count_chunked_kernel(const Layer0Args a) {
  extern __shared__ __align__(128) uint32_t cbits[];  // Q + 32 words
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  __shared__ __align__(8) uint64_t bar;
  __shared__ float s_sum[128];
  __shared__ uint32_t s_mask;
  __shared__ int32_t s_fail;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int N = a.N, Q = a.Q, nq = a.nq;
  const int count = *a.count_in;
  const int n_tiles = (count + 31) / 32;
  constexpr int per_item = kChunkWarps * kChunkGroupsPerWarp;
  const int subsets = (a.G + per_item - 1) / per_item;
  const long items = (long)n_tiles * subsets;
  __shared__ float s_val[128];
  if (tid < 128) {
    s_sum[tid] = a.sums[tid];
    s_val[tid] = clampf(a.sums[tid] + a.bias, a.clampv);
  }
  for (int i = tid; i < 32; i += blockDim.x) cbits[Q + i] = 0u;
  if (tid == 0) {
    mbar_init(&bar, 1);
    s_mask = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  const CountInterval iv = count_interval(s_sum, a.bias, a.bias_vec != nullptr);
  uint32_t phase = 0;
  for (long item = blockIdx.x; item < items; item += gridDim.x) {
    const int tile = (int)(item / subsets), sub = (int)(item % subsets);
    const int row0 = tile * 32;
    const int nrows = min(32, count - row0);
    if (a.tile_state[tile]) {  // non-binary tile: the float kernel runs it
      if (sub == 0 && warp == 0) list_fallback(a, row0, nrows, lane);
      continue;
    }
    uint32_t c[kChunkGroupsPerWarp][7];
#pragma unroll
    for (int k = 0; k < kChunkGroupsPerWarp; ++k)
#pragma unroll
      for (int i = 0; i < 7; ++i) c[k][i] = 0u;
    for (int q = 0; q < nq; ++q) {
      __syncthreads();  // every warp is done with the previous chunk
      if (tid == 0) {
        const uint32_t bytes = (uint32_t)Q * 4u;
        mbar_expect_tx(&bar, bytes);
        const char* src = reinterpret_cast<const char*>(a.bits + (size_t)tile * N + (size_t)q * Q);
        char* dst = reinterpret_cast<char*>(cbits);
        for (uint32_t off = 0; off < bytes; off += 32768u)
          bulk_g2s(dst + off, src + off, min(32768u, bytes - off), &bar);
        s_fail = mbar_wait_bounded(&bar, phase, a.err) ? 0 : 1;
      }
      __syncthreads();
      if (s_fail) return;
      mbar_try_wait(&bar, phase);
      phase ^= 1u;
#pragma unroll
      for (int k = 0; k < kChunkGroupsPerWarp; ++k) {
        const int g = sub * per_item + k * kChunkWarps + warp;
        if (g < a.G) {
          const int32_t b0 = __ldg(a.grp_blk + g * nq + q), b1 = __ldg(a.grp_blk + g * nq + q + 1);
          count_short_list(c[k], a.idx + (size_t)b0 * 32 + lane, b1 - b0, cbits);
        }
      }
    }
    uint32_t m = 0;
#pragma unroll
    for (int k = 0; k < kChunkGroupsPerWarp; ++k) {
      const int g = sub * per_item + k * kChunkWarps + warp;
      if (g >= a.G) continue;
      m |= bits_epilogue<0>(c[k], a, s_sum, s_val, iv, a.first_row + row0, nrows, g * 32 + lane);
    }
    m = __reduce_or_sync(0xffffffffu, m);
    if (lane == 0 && m) atomicOr(&s_mask, m);
    __syncthreads();
    if (warp == 0) {
      list_rows(a, s_mask, subsets > 1, row0, lane);
      __syncwarp();
      if (lane == 0) s_mask = 0;
    }
  }
}

namespace {

cudaError_t launch_pdl(const void* fn, int grid, int threads, size_t smem, const Layer0Args& a,
                       cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void* args[] = {const_cast<Layer0Args*>(&a)};
  return cudaLaunchKernelExC(&cfg, fn, args);
}

const void* count_fn(int N) {
  switch (N) {
    case 1024: return (const void*)&bits_count_kernel<1056>;
    case 4096: return (const void*)&bits_count_kernel<4128>;
    case 16384: return (const void*)&bits_count_kernel<16416>;
    default: return nullptr;
  }
}

}  // namespace

bool layer0_bits_chunked_supported(int N, int Q) {
  return Q == 16384 && N % Q == 0 && N / Q > 1 && N % 128 == 0;
}

bool layer0_bits_supported(int N) { return count_fn(N) != nullptr; }

cudaError_t launch_layer0_bits(const Layer0Args& a, int num_sms, cudaStream_t s) {
  const bool chunked = a.nq > 1;
  const void* fn = chunked ? (const void*)&bits_count_chunked_kernel : count_fn(a.N);
  if (!fn || (chunked && !layer0_bits_chunked_supported(a.N, a.Q))) return cudaErrorInvalidValue;
  const int threads = chunked ? kChunkWarps * 32 : kCountWarps * 32;
  const size_t smem = (size_t)((chunked ? a.Q : a.N) + 32) * 4 * (chunked ? 1 : count_buffers(a.N));
  cudaError_t rc = allow_smem(fn);
  if (rc != cudaSuccess) return rc;
  int per_sm = 0;
  rc = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem);
  if (rc != cudaSuccess) return rc;
  rc = a.bit_rows
           ? launch_pdl((const void*)&bit_rows_transpose_kernel, num_sms * 8, kTransposeThreads, 0, a, s)
           : launch_pdl((const void*)&bits_transpose_kernel, num_sms * 6, kTransposeThreads, 0, a, s);
  if (rc != cudaSuccess) return rc;
  return launch_pdl(fn, num_sms * std::max(1, per_sm), threads, smem, a, s);
}

}  // namespace sdnn
