// Post-threshold layers once no residue row is left.
//
// After the threshold clustering, a row whose activations equal its centroid's
// has no residue and never gets one again (a zero residue updates to zero), so
// when the residue list is empty the rest of the inference is the K centroid
// rows alone, carried through the remaining layers (SNICIT's post_spMM +
// post_minus with nerow = K, src/SDGC/SNICIT/kernel.hpp:71-136).  Run as one
// launch per layer, that is 2 launches of a few microseconds each for a few
// rows.  Here one thread-block cluster runs all of those layers in one launch:
//
//  * every CTA of the cluster keeps all K rows in shared memory (two buffers,
//    this layer's input and the next layer's);
//  * CTA r computes the outputs of its share of the 32-neuron groups for all K
//    rows, with the same bank-scheduled slots and FP32 order as the layer kernels
//    (so the rows are bitwise equal to the per-layer path), applies bias and
//    clamp, and stores each output into the next-layer buffer of every CTA of
//    the cluster (distributed shared memory);
//  * a cluster barrier separates layers; after the last layer the rows go to
//    the final activation buffer for recovery.
#include <algorithm>
#include <map>
#include <mutex>
#include <utility>

#include <cooperative_groups.h>

#include "layer_kernel.cuh"

namespace cg = cooperative_groups;

namespace sdnn {

constexpr int kChainCluster = 8;

template <int RSW, int KC>
__global__ void __launch_bounds__(1024, 1) chain_kernel(const ChainArgs a) {
  extern __shared__ __align__(128) float rows[];  // [2][KC][RSW]
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int csize = (int)cluster.num_blocks();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int N = a.N;
  const int K = min(*a.ccount, KC);
  // zero columns of both buffers, then this layer's rows from the threshold buffer
  for (int i = tid; i < 2 * KC * 32; i += blockDim.x) rows[(i >> 5) * RSW + N + (i & 31)] = 0.f;
  for (int t = 0; t < K; ++t) {
    const float* src = a.y_in + (size_t)a.clist[t] * N;
    for (int j = tid; j < N; j += blockDim.x) rows[t * RSW + j] = src[j];
  }
  cluster.sync();
  const int gbeg = (int)((long)a.G * rank / csize), gend = (int)((long)a.G * (rank + 1) / csize);
  // this CTA's slot blocks of layer l are contiguous: prefetch them into L2 a
  // few layers ahead so the per-layer loads hit L2 instead of HBM
  auto prefetch = [&](int l) {
    if (tid != 0 || l >= a.last) return;
    const LayerDev wp = a.layers[l];
    const int32_t b0 = wp.grp_blk[gbeg], b1 = wp.grp_blk[gend];
    const uint32_t bytes = (uint32_t)(b1 - b0) * 32u * (uint32_t)sizeof(uint2);
    if (bytes > 0)
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(wp.idx + (size_t)b0 * 32),
                   "r"(bytes)
                   : "memory");
    if (wp.val && bytes > 0)
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(wp.val + (size_t)b0 * 32),
                   "r"(bytes * 2u)
                   : "memory");
  };
  for (int d = 0; d < 4; ++d) prefetch(a.first + d);
  for (int l = a.first; l < a.last; ++l) {
    prefetch(l + 4);
    const LayerDev wl = a.layers[l];
    const float* cur = rows + (size_t)((l - a.first) & 1) * KC * RSW;
    float* nxt = rows + (size_t)(((l - a.first) & 1) ^ 1) * KC * RSW;
    const bool last = l + 1 == a.last;
    for (int g = gbeg + warp; g < gend; g += nwarps) {
      float acc[KC];
#pragma unroll
      for (int t = 0; t < KC; ++t) acc[t] = 0.f;
      if (wl.val == nullptr)
        accumulate_group<KC, RSW, true>(acc, wl, 1, cur, RSW, g, 0, lane);
      else
        accumulate_group<KC, RSW, false>(acc, wl, 1, cur, RSW, g, 0, lane);
      const int c = g * 32 + lane;
      const float bc = wl.bias_vec ? __ldg(wl.bias_vec + c) : wl.bias;
#pragma unroll
      for (int t = 0; t < KC; ++t) {
        if (t < K) {
          const float y = clampf(acc[t] + bc, a.clampv);
          for (int p = 0; p < csize; ++p) cluster.map_shared_rank(nxt, p)[t * RSW + c] = y;
          if (last) a.y_out[(size_t)a.clist[t] * N + c] = y;
        }
      }
    }
    cluster.sync();
  }
}

// ---------------------------------------------------------------------------
// chain2_kernel: the same computation with the weights streamed into shared
// memory and point-to-point row exchange.  A layer of one row is a few hundred
// gathers, so a layer costs what its longest wait costs:
//
//  * one producer warp (the last warp of the CTA) keeps a ring of weight
//    buffers (2 to 8, as many as fit) filled with this CTA's lists and slot
//    blocks of the next layers, by 1-D TMA bulk copies.  It knows the address
//    and size of 32 layers at a time (one per lane; the next 32 are looked up
//    and fetched into L2 meanwhile), so a refill is one lane issuing two or
//    three copies, and with three buffers or more its round trip is covered by
//    the layers in between.  (With two buffers and the table and offsets read
//    from memory per layer, that chain of loads was the layer time.)
//  * a compute warp takes a layer's slots into registers before it waits for
//    the layer's inputs: from the last input on, a layer is one run of
//    gathers, the stores, and their way to the other CTAs;
//  * outputs go to every CTA of the cluster with 16-byte st.async, each
//    signalling the receiving CTA's mbarrier for its next row buffer; a CTA
//    starts layer l + 1 when all N x K values of its next buffer have
//    arrived -- no cluster-wide barrier per layer;
//  * two row buffers suffice: a CTA that starts layer l has received every
//    CTA's layer l - 1 outputs, which each CTA sends only after it has read
//    all of its layer l - 1 inputs -- the buffer that layer l's outputs
//    overwrite everywhere.
// What is left is the exchange (an all-to-all of a row takes 660 cycles at
// N = 1024 and 1350 at N = 4096, where a CTA takes in 18 bytes per clock) and
// the deepest list's gathers (13 blocks: 500-600 cycles).  One row: 90 layers
// of 1024 neurons 115 -> 74 us, 450 layers of 4096 699 -> 458.
// Same slots, same FMA order as the layer kernels and chain_kernel: bitwise
// equal.
constexpr int kChain2ComputeWarps = 16;  // at most (one per group)
constexpr int kChain2MaxGroups = 64;     // groups per CTA (G / cluster size)
constexpr int kChain2MaxBufs = 8;        // weight buffers
constexpr size_t kChain2Static = 1024;    // static shared memory, at most

// The lists' part of a weight buffer.
__host__ __device__ constexpr uint32_t chain2_list_bytes(int groups) {
  return ((uint32_t)groups * 8u + 127u) / 128u * 128u;
}

__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_async_v4(uint32_t raddr, float4 v, uint32_t rbar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, "
      "[%5];" ::"r"(raddr),
      "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(rbar)
      : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
  if (bytes > 0)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// Blocks of a list in registers.  Blocks past the list's end gather the zero
// column with weight 0: they change no sum.
template <bool CONSTW>
struct ChainSlots {
  static constexpr int NB = CONSTW ? 16 : 8;
  uint2 iv[NB];
  float4 vv[CONSTW ? 1 : NB];
  __device__ __forceinline__ void load(const uint2* sidx, const float4* sval, int nb, uint32_t pad,
                                       int lane) {
#pragma unroll
    for (int k = 0; k < NB; ++k) {
      iv[k] = make_uint2(pad, pad);
      if (k < nb) iv[k] = sidx[k * 32 + lane];
      if constexpr (!CONSTW) {
        vv[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (k < nb) vv[k] = sval[k * 32 + lane];
      }
    }
  }
  // a straight run over B blocks, of which the list has B - 1 or more (or none)
  template <int B, int KC, int RSW>
  __device__ __forceinline__ void run(float (&acc)[KC], int nb, float wc, const float* ys) const {
#pragma unroll
    for (int k = 0; k < B; ++k)
      apply_block<KC, RSW, CONSTW>(acc, iv[k], vv[CONSTW ? 0 : k], (B > 2 && k < B - 1) || k < nb ? wc : 0.f, ys, RSW, 4);
  }
  // ... over the list's blocks, rounded up to a pair
  template <int B, int KC, int RSW>
  __device__ __forceinline__ void apply(float (&acc)[KC], int nb, float wc, const float* ys) const {
    if constexpr (B > 2) {
      if (nb <= B - 2) return apply<B - 2, KC, RSW>(acc, nb, wc, ys);
    }
    run<B, KC, RSW>(acc, nb, wc, ys);
  }
};

// One group: its first slots are taken before ready() (the wait for the
// layer's inputs), the rest of a longer list after.
template <int KC, int RSW, bool CONSTW, typename Ready>
__device__ __forceinline__ void chain_group(float (&acc)[KC], const uint2* sidx, const float4* sval,
                                            int nb, float wc, const float* ys, int lane,
                                            Ready ready) {
  using Slots = ChainSlots<CONSTW>;
  const uint32_t zero = (uint32_t)(RSW - 32 + lane) * (rsw_in_bytes(RSW) ? 4u : 1u);
  const uint32_t pad = zero | (zero << 16);
#pragma unroll
  for (int t = 0; t < KC; ++t) acc[t] = 0.f;
  Slots s;
  s.load(sidx, sval, nb, pad, lane);
  ready();
  s.template apply<Slots::NB, KC, RSW>(acc, nb, wc, ys);
#pragma unroll 1
  for (int b = Slots::NB; b < nb; b += Slots::NB) {
    s.load(sidx + b * 32, CONSTW ? nullptr : sval + b * 32, nb - b, pad, lane);
    s.template apply<Slots::NB, KC, RSW>(acc, nb - b, wc, ys);
  }
}

// What the compute warps need of a layer besides its lists and blocks.
struct ChainLayer {
  const float* bias_vec;
  float bias, wconst;
  int32_t b0;       // first slot block of this CTA's groups
  int32_t nblk;     // ... and how many
  int32_t general;  // a value per edge
};

template <int RSW, int KC>
__global__ void __launch_bounds__((kChain2ComputeWarps + 1) * 32, 1) chain2_kernel(const ChainArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  float* rows = reinterpret_cast<float*>(smem);  // [2][KC][RSW]
  // [nbuf][wcap]: lists, slot blocks, values
  unsigned char* wbase = smem + (size_t)2 * KC * RSW * 4;
  __shared__ __align__(8) uint64_t rb[2];               // row buffer b complete
  __shared__ __align__(8) uint64_t wb[kChain2MaxBufs];  // weight buffer b loaded
  __shared__ __align__(8) uint64_t wd[kChain2MaxBufs];  // ... and read by every compute warp
  __shared__ ChainLayer s_layer[kChain2MaxBufs];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int csize = (int)cluster.num_blocks();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nwarps = (blockDim.x >> 5) - 1;  // compute warps
  const bool producer = warp == nwarps;
  const int N = a.N;
  const int K = min(*a.ccount, KC);
  // (G is a multiple of twice the cluster size: lists start on 16 bytes)
  const int ng = a.G / csize, gbeg = rank * ng;
  const uint32_t row_bytes = (uint32_t)K * (uint32_t)N * 4u;
  const uint32_t wcap = a.wcap, list_bytes = chain2_list_bytes(ng);
  const int nbuf = a.nbuf, layers = a.last - a.first;
  const uint32_t base = smem_u32(smem);

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) mbar_init(&rb[i], 1);
    for (int i = 0; i < nbuf; ++i) {
      mbar_init(&wb[i], 1);
      mbar_init(&wd[i], nwarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = tid; i < 2 * KC * 32; i += blockDim.x) rows[(i >> 5) * RSW + N + (i & 31)] = 0.f;
  for (int t = 0; t < K; ++t) {
    const float* src = a.y_in + (size_t)a.clist[t] * N;
    for (int j = tid; j < N; j += blockDim.x) rows[t * RSW + j] = src[j];
  }
  cluster.sync();  // every CTA's barriers exist before any remote store

  if (producer) {
    // lane i: layers i, i + 32, ... (this window's, and the next one's)
    LayerDev cur{}, nxt{};
    int2 f = make_int2(0, 0), t = make_int2(0, 0);
    int32_t b0 = 0, nblk = 0, nb0 = 0, nnblk = 0;
    auto look_up = [&](int l) {
      if (l < layers) nxt = a.layers[a.first + l];
    };
    auto ends = [&](int l) {
      if (l < layers) {
        f = __ldg(nxt.lists + gbeg);
        t = __ldg(nxt.lists + gbeg + ng - 1);
      }
    };
    auto sizes = [&](int l) {
      nb0 = f.x;
      nnblk = l < layers ? t.x + ((t.y + 3) >> 2) - f.x : 0;
    };
    auto fetch = [&](int l) {  // into L2
      if (l < layers) {
        prefetch_l2(nxt.lists + gbeg, (uint32_t)ng * 8u);
        prefetch_l2(nxt.idx + (size_t)nb0 * 32, (uint32_t)nnblk * 256u);
        if (nxt.val) prefetch_l2(nxt.val + (size_t)nb0 * 32, (uint32_t)nnblk * 512u);
      }
    };
    look_up(lane);
    ends(lane);
    sizes(lane);
    int buf = 0, filled = 0;
    uint32_t wdpar = 1u;  // the first round of buffers is free
    for (int l = 0; l < layers; ++l) {
      if ((l & 31) == 0) {
        cur = nxt;
        b0 = nb0;
        nblk = nnblk;
      }
      if (l >= nbuf) {
        bool ok = mbar_wait_bounded(&wd[buf], wdpar, a.err);
        if (!__all_sync(0xffffffffu, ok)) break;
      }
      if (lane == (l & 31)) {
        s_layer[buf] = ChainLayer{cur.bias_vec, cur.bias, cur.wconst, b0, nblk, cur.val != nullptr};
        const uint32_t bl = (uint32_t)ng * 8u, bi = (uint32_t)nblk * 256u;
        const uint32_t bv = cur.val ? (uint32_t)nblk * 512u : 0u;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(&wb[buf], bl + bi + bv);
        unsigned char* dst = wbase + (size_t)buf * wcap;
        bulk_g2s(dst, cur.lists + gbeg, bl, &wb[buf]);
        dst += list_bytes;
        if (bi) bulk_g2s(dst, cur.idx + (size_t)b0 * 32, bi, &wb[buf]);
        if (bv) bulk_g2s(dst + bi, cur.val + (size_t)b0 * 32, bv, &wb[buf]);
      }
      __syncwarp();
      ++filled;
      if (++buf == nbuf) {
        buf = 0;
        wdpar ^= 1u;
      }
      // the steps of the next window, a layer's time or more apart
      if (l == nbuf - 1 || (layers <= nbuf && l == layers - 1)) {
        // (the rest of the first window, once its first buffers are on their way)
        if (lane >= nbuf && (l & ~31) == 0) {
          fetch(lane);
        }
      }
      const int step = l & 31, next = (l & ~31) + 32 + lane;
      if (step == 12) look_up(next);
      if (step == 16) ends(next);
      if (step == 20) {
        sizes(next);
        fetch(next);
      }
    }
    if (lane == 0 && *reinterpret_cast<volatile int32_t*>(a.err) != 0) {
      // after a timeout the compute warps stop waiting: let the last copy
      // issued into each buffer land before the CTA exits
      for (int b = 0; b < nbuf; ++b) {
        const int fills = (filled + nbuf - 1 - b) / nbuf;
        if (fills > 0 && !mbar_wait_bounded(&wb[b], (uint32_t)(fills - 1) & 1u, a.err)) break;
      }
    }
  } else {
    // A warp sends its 32 outputs of a row as 8 quads to each CTA: lane i quad
    // i & 7 to the CTAs i >> 3, + 4, ... (where their shared memory is seen)
    uint32_t seen[4];
#pragma unroll
    for (int p = 0; p < 4; ++p)
      seen[p] = mapa_u32(base, (uint32_t)min((lane >> 3) + 4 * p, csize - 1));
    const int quad = (lane & 7) * 4;
    int buf = 0;
    uint32_t wpar = 0;
    bool failed = false;
    for (int l = 0; l < layers; ++l) {
      const int cur = l & 1, nxt = cur ^ 1;
      const bool last = l + 1 == layers;
      const bool ok = mbar_wait_bounded(&wb[buf], wpar, a.err);
      if (!__all_sync(0xffffffffu, ok)) break;  // no lists: nothing to read rows with
      const ChainLayer wl = s_layer[buf];
      const float* ys = rows + (size_t)cur * KC * RSW;
      const int2* slists = reinterpret_cast<const int2*>(wbase + (size_t)buf * wcap);
      const uint2* sidx = reinterpret_cast<const uint2*>(wbase + (size_t)buf * wcap + list_bytes);
      const float4* sval = reinterpret_cast<const float4*>(sidx + (size_t)wl.nblk * 32);
      bool waited = l == 0;
      auto ready = [&]() {
        if (!waited) {
          // the inputs of layer l are the ((l - 1) / 2)-th use of their buffer
          if (!failed && !mbar_wait_bounded(&rb[cur], (uint32_t)((l - 1) >> 1) & 1u, a.err))
            failed = true;
          __syncwarp();
          waited = true;
        }
      };
      // its first use is free; later ones after the buffer's last inputs (of
      // layer l - 1) were waited for, which this thread did before
      if (!last && tid == 0) mbar_expect_tx(&rb[nxt], row_bytes);
      const uint32_t nbuf_off = smem_u32(rows + (size_t)nxt * KC * RSW) - base;
      const uint32_t nbar_off = smem_u32(&rb[nxt]) - base;
      for (int g = warp; g < ng; g += nwarps) {
        const int c = (gbeg + g) * 32 + lane;
        const float bc = wl.bias_vec ? __ldg(wl.bias_vec + c) : wl.bias;
        const int2 list = slists[g];
        const int o = list.x - wl.b0, nb = (list.y + 3) >> 2;
        float acc[KC];
        if (!wl.general)
          chain_group<KC, RSW, true>(acc, sidx + (size_t)o * 32, nullptr, nb, wl.wconst, ys, lane,
                                     ready);
        else
          chain_group<KC, RSW, false>(acc, sidx + (size_t)o * 32, sval + (size_t)o * 32, nb,
                                      wl.wconst, ys, lane, ready);
#pragma unroll
        for (int t = 0; t < KC; ++t) {
          if (t < K) {
            const float y = clampf(acc[t] + bc, a.clampv);
            if (last) {
              a.y_out[(size_t)a.clist[t] * N + c] = y;
            } else {
              float4 v;
              v.x = __shfl_sync(0xffffffffu, y, quad);
              v.y = __shfl_sync(0xffffffffu, y, quad + 1);
              v.z = __shfl_sync(0xffffffffu, y, quad + 2);
              v.w = __shfl_sync(0xffffffffu, y, quad + 3);
              const uint32_t off = nbuf_off + (uint32_t)(t * RSW + c - lane + quad) * 4u;
              st_async_v4(seen[0] + off, v, seen[0] + nbar_off);
              st_async_v4(seen[1] + off, v, seen[1] + nbar_off);
              if (csize > 8) {
                st_async_v4(seen[2] + off, v, seen[2] + nbar_off);
                st_async_v4(seen[3] + off, v, seen[3] + nbar_off);
              }
            }
          }
        }
      }
      ready();  // (a warp with no group)
      __syncwarp();
      if (lane == 0 && l + nbuf < layers) mbar_arrive(&wd[buf]);
      if (++buf == nbuf) {
        buf = 0;
        wpar ^= 1u;
      }
    }
  }
  cluster.sync();  // no CTA leaves while another may still store into it
}

template __global__ void chain2_kernel<1056, 1>(const ChainArgs);
template __global__ void chain2_kernel<1056, 2>(const ChainArgs);
template __global__ void chain2_kernel<1056, 4>(const ChainArgs);
template __global__ void chain2_kernel<1056, 8>(const ChainArgs);
template __global__ void chain2_kernel<4128, 1>(const ChainArgs);
template __global__ void chain2_kernel<4128, 2>(const ChainArgs);
template __global__ void chain2_kernel<4128, 4>(const ChainArgs);
template __global__ void chain2_kernel<16416, 1>(const ChainArgs);

template __global__ void chain_kernel<1056, 1>(const ChainArgs);
template __global__ void chain_kernel<1056, 2>(const ChainArgs);
template __global__ void chain_kernel<1056, 4>(const ChainArgs);
template __global__ void chain_kernel<1056, 8>(const ChainArgs);
template __global__ void chain_kernel<4128, 1>(const ChainArgs);
template __global__ void chain_kernel<4128, 2>(const ChainArgs);
template __global__ void chain_kernel<4128, 4>(const ChainArgs);
template __global__ void chain_kernel<16416, 1>(const ChainArgs);

static const void* chain_fn(int rsw, int kc) {
#define SDNN_PICK(R, K) \
  if (rsw == R && kc == K) return (const void*)&chain_kernel<R, K>;
  SDNN_PICK(1056, 1)
  SDNN_PICK(1056, 2)
  SDNN_PICK(1056, 4)
  SDNN_PICK(1056, 8)
  SDNN_PICK(4128, 1)
  SDNN_PICK(4128, 2)
  SDNN_PICK(4128, 4)
  SDNN_PICK(16416, 1)
#undef SDNN_PICK
  return nullptr;
}

static const void* chain2_fn(int rsw, int kc) {
#define SDNN_PICK(R, K) \
  if (rsw == R && kc == K) return (const void*)&chain2_kernel<R, K>;
  SDNN_PICK(1056, 1)
  SDNN_PICK(1056, 2)
  SDNN_PICK(1056, 4)
  SDNN_PICK(1056, 8)
  SDNN_PICK(4128, 1)
  SDNN_PICK(4128, 2)
  SDNN_PICK(4128, 4)
  SDNN_PICK(16416, 1)
#undef SDNN_PICK
  return nullptr;
}

uint32_t chain_slice_bytes(const int32_t* grp_blk, int G, bool general, int cluster) {
  uint32_t best = 0;
  for (int r = 0; r < cluster; ++r) {
    const int gb = (int)((long)G * r / cluster), ge = (int)((long)G * (r + 1) / cluster);
    const uint32_t nblk = (uint32_t)(grp_blk[ge] - grp_blk[gb]);
    best = std::max(best, nblk * 32u * (general ? 24u : 8u));
  }
  return best;
}

int chain_capacity(int N) {
  const int rsw = N + 32;
  int best = 0;
  for (int kc : {1, 2, 4, 8})
    if (chain_fn(rsw, kc)) best = kc;
  return best;
}

static int chain_kc_for(int rsw, int kc_needed) {
  for (int k : {1, 2, 4, 8})
    if (k >= kc_needed && chain_fn(rsw, k)) return k;
  return 0;
}

// Whether clusters of 16 CTAs (non-portable size) of this kernel fit the
// current device, at the largest shared memory; asked once per device.
static bool cluster16_ok(const void* fn, int threads) {
  static std::mutex mutex;
  static std::map<std::pair<int, const void*>, bool> known;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  std::lock_guard<std::mutex> lock(mutex);
  const auto at = known.find({dev, fn});
  if (at != known.end()) return at->second;
  cudaFuncAttributes attrs;
  int n = 0;
  bool ok = allow_smem(fn) == cudaSuccess && cudaFuncGetAttributes(&attrs, fn) == cudaSuccess &&
            cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
  if (ok) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = (size_t)attrs.maxDynamicSharedSizeBytes;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 16;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    ok = cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess && n > 0;
  }
  if (!ok) cudaGetLastError();
  known[{dev, fn}] = ok;
  return ok;
}

ChainPlan chain_plan(const ChainArgs& a, int kc_needed) {
  ChainPlan p{};
  const int rsw = a.N + 32;
  const int kc = chain_kc_for(rsw, kc_needed);
  if (!kc) return p;
  p.kc = kc;
  p.variant = 1;
  p.cluster = kChainCluster;
  p.threads = 512;
  p.smem = (size_t)2 * kc * rsw * sizeof(float);
  // wide rows (many groups per CTA): a cluster of 16 and 1024 threads, one
  // group per warp at N = 16384
  if (a.G / kChainCluster > 32 && cluster16_ok(chain_fn(rsw, kc), 1024)) {
    p.cluster = 16;
    p.threads = 1024;
  }
  if (!a.stream) return p;
  // Streamed weights.  Where a cluster of 8 has more than 8 groups per CTA, 16
  // CTAs share the gathers better (N = 4096: 1.02 us a layer against 1.34; at
  // N = 1024, 4 groups, 0.80 against 0.82, so the portable size stays).  Two
  // weight buffers at least; wide rows are taken with one too.
  const size_t room = 227 * 1024 - kChain2Static;
  struct Option { int cluster, least; uint32_t wcap; };
  const bool wide = a.G / kChainCluster > 8;
  const Option opts[] = {{wide ? 16 : 8, 2, wide ? a.wcap16 : a.wcap8},
                         {wide ? 8 : 16, 2, wide ? a.wcap8 : a.wcap16},
                         {16, 1, a.wcap16},
                         {8, 1, a.wcap8}};
  for (const auto& o : opts) {
    if (o.least == 1 && rsw != 16416) break;
    if (o.wcap == 0 || a.G % (2 * o.cluster) != 0 || a.G / o.cluster > kChain2MaxGroups) continue;
    const void* fn = chain2_fn(rsw, kc);
    const uint32_t wcap = o.wcap + chain2_list_bytes(a.G / o.cluster);
    const int fits = p.smem < room ? (int)std::min<size_t>(kChain2MaxBufs, (room - p.smem) / wcap) : 0;
    if (!fn || fits < o.least) continue;
    const int threads = (std::min(kChain2ComputeWarps, a.G / o.cluster) + 1) * 32;
    const size_t smem = p.smem + (size_t)fits * wcap;
    if (o.cluster == 16 && !cluster16_ok(fn, threads)) continue;
    p.variant = 2;
    p.cluster = o.cluster;
    p.nbuf = fits;
    p.wcap = wcap;
    p.threads = threads;
    p.smem = smem;
    return p;
  }
  return p;
}

cudaError_t launch_chain(const ChainArgs& a0, int kc_needed, cudaStream_t s) {
  const ChainPlan p = chain_plan(a0, kc_needed);
  if (!p.variant) return cudaErrorInvalidValue;
  const int rsw = a0.N + 32;
  ChainArgs a = a0;
  a.wcap = p.wcap;
  a.nbuf = p.nbuf;
  const void* fn = p.variant == 2 ? chain2_fn(rsw, p.kc) : chain_fn(rsw, p.kc);
  cudaError_t rc = allow_smem(fn);
  if (rc != cudaSuccess) return rc;
  if (p.cluster > 8) {
    rc = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (rc != cudaSuccess) return rc;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.cluster);
  cfg.blockDim = dim3(p.threads);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void* args[] = {&a};
  return cudaLaunchKernelExC(&cfg, fn, args);
}

}  // namespace sdnn
