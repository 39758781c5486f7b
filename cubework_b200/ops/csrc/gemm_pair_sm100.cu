// GEMM on pairs of SMs (cta_group::2): TMA -> shared memory -> tcgen05.mma of 256 x 256 x 16 -> TMEM -> epilogue.
//
// The single-CTA kernel of gemm_sm100.cu lets every SM fetch its own copy of a 256-column B tile: 48 KB through L2 for
// 128 x 256 x 64 of the product, 0.42 us a k-block at 8192^3.  Here a cluster of two CTAs shares a 256 x 256 tile: each
// loads its own 128 rows of A and half of B (32 KB), one thread of the leading CTA issues the MMAs for both SMs, and each
// CTA keeps the accumulator of its 128 rows: 0.39 us, of which the tensor cores need 0.36 at the clock that the power cap
// leaves them.  8192^3: 751 -> 694 us (cuBLAS 648); 32768 x 1600 x 6400: 527 -> 492 (468); 50432 x 2304 x 768: 146 -> 126
// (140); 6400 x 1600 x 32768 with fp32 output: 564 -> 511 (548).
// Narrower tiles were measured and do not pay: an MMA takes the same time whatever its N below 256 (8192^3 at a width of
// 192: 835 us, at 128: 1324, at 64: 2390), so a k-block does, and 32768 x 1600 is cheaper as seven tiles of 256 (126 us)
// than as ten of 160 (171).
//
// Roles per CTA as in gemm_sm100.cu: warp 0 loads, warp 1 owns TMEM and (leader) issues, warps 2-9 write tiles out.
//   full_bar    leader only: both CTAs' loads of a stage complete on it (expect_tx of both halves by the leader)
//   empty_bar   each CTA its own: the leader's commit arrives on both, the stage is free in both
//   tfull_bar   each CTA its own, same commit; tempty_bar: leader only, the epilogue warps of both CTAs arrive on it
// All waits are bounded; both CTAs meet in a cluster barrier before either leaves, because the partner's copies,
// commits and arrivals land in their shared memory.
#include <cmath>

#include "gemm_sm100.cuh"

namespace cw {

constexpr int kPairBN = 256;
constexpr int kPairStageBytes = 32768;            // A half: 128 x 64; B half: 128 x 64
constexpr int kPairStages = 6;
constexpr int kPairBarBytes = (2 * kPairStages + 4) * 8 + 16;
constexpr int kPairSmemBytes = kPairStages * kPairStageBytes + kEpiWarps * kEpiBlockBytes + kPairBarBytes + 1024;
static_assert(kPairSmemBytes <= 227 * 1024, "GEMM exceeds the shared memory of one SM");
constexpr int kPairGroup = 8;                     // row blocks (of 256) that are walked together, for reuse in L2

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_rank(const void* p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Load into this CTA's shared memory that completes on a barrier of either CTA of the pair (a shared::cluster address).
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tc_mma_f16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                                uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives on the barrier at this offset in both CTAs once the MMAs issued so far have finished.
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"(static_cast<uint16_t>(3))
               : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

struct PairWork {
  int tiles_m, tiles_n, num_tiles, kb_total, per, splits;
  __device__ __forceinline__ void decode(int w, int& tile_m, int& tile_n, int& kb0, int& kb1) const {
    const int split = splits > 1 ? fast_div(w, num_tiles) : 0;
    const int t = w - split * num_tiles;
    const int group = fast_div(t, kPairGroup * tiles_n);
    const int first_m = group * kPairGroup;
    const int gsz = min(tiles_m - first_m, kPairGroup);
    const int in_group = t - group * kPairGroup * tiles_n;
    tile_n = gsz == kPairGroup ? in_group / kPairGroup : fast_div(in_group, gsz);
    tile_m = first_m + in_group - tile_n * gsz;
    kb0 = split * per;
    kb1 = min(kb0 + per, kb_total);
  }
};

template <bool A_KMAJOR, bool B_KMAJOR, typename InT, bool OUT_F32>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreadsV2, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                 const __grid_constant__ CUtensorMap tma_out, const __grid_constant__ CUtensorMap tma_z, GemmParams p) {
  constexpr int kHalfN = kPairBN / 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* stage_out = smem + kPairStages * kPairStageBytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(stage_out + kEpiWarps * kEpiBlockBytes);
  uint64_t* empty_bar = full_bar + kPairStages;
  uint64_t* tfull_bar = empty_bar + kPairStages;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const bool leader = rank == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kPairStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], 2 * kEpiWarps);
    }
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_b);
    if (p.tma_store) {
      tma_prefetch_desc(&tma_out);
      if (p.z_out != nullptr) tma_prefetch_desc(&tma_z);
    }
  }
  if (warp == 1) {
    __syncwarp();
    tmem_alloc_pair(tmem_slot, 512);
  }
  tc_fence_before();
  __syncthreads();
  __syncwarp();
  cluster_sync_all();                     // the partner's barriers are initialised before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  PairWork work;
  work.tiles_m = (p.M + 2 * kBM - 1) / (2 * kBM);
  work.tiles_n = (p.N + kPairBN - 1) / kPairBN;
  work.num_tiles = work.tiles_m * work.tiles_n;
  work.kb_total = (p.K + kBK - 1) / kBK;
  work.splits = p.splits;
  work.per = (work.kb_total + p.splits - 1) / p.splits;
  const int total_work = work.num_tiles * p.splits;
  const int first = blockIdx.x >> 1, stride = gridDim.x >> 1;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int w = first; w < total_work && !*abort_flag; w += stride) {
        int tile_m, tile_n, kb0, kb1;
        work.decode(w, tile_m, tile_n, kb0, kb1);
        const int row = tile_m * 2 * kBM + static_cast<int>(rank) * kBM;
        const int col = tile_n * kPairBN + static_cast<int>(rank) * kHalfN;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.status, kErrEmptyBarrierTimeout, w)) break;
          if (leader) mbar_expect_tx(&full_bar[stage], 2 * kPairStageBytes);
          const uint32_t bar = map_to_rank(&full_bar[stage], 0);
          uint8_t* sa = smem + stage * kPairStageBytes;
          uint8_t* sb = sa + kBM * kBK * 2;
          if (A_KMAJOR) {
            tma_load_2d_pair(sa, &tma_a, bar, kb * kBK, row);
          } else {
#pragma unroll
            for (int g = 0; g < kBM / 64; ++g) tma_load_2d_pair(sa + g * 8192, &tma_a, bar, row + g * 64, kb * kBK);
          }
          if (B_KMAJOR) {
            tma_load_2d_pair(sb, &tma_b, bar, kb * kBK, col);
          } else {
#pragma unroll
            for (int g = 0; g < kHalfN / 64; ++g) tma_load_2d_pair(sb + g * 8192, &tma_b, bar, col + g * 64, kb * kBK);
          }
          if (++stage == kPairStages) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader)
    if (leader && lane == 0) {
      const uint32_t idesc = make_idesc_f16(2 * kBM, kPairBN, !A_KMAJOR, !B_KMAJOR, p.is_bf16);
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      for (int w = first; w < total_work && !*abort_flag; w += stride, ++it) {
        int tile_m, tile_n, kb0, kb1;
        work.decode(w, tile_m, tile_n, kb0, kb1);
        const int acc = it & 1;
        const uint32_t acc_phase = (it >> 1) & 1;
        if (!mbar_wait(&tempty_bar[acc], acc_phase ^ 1, abort_flag, p.status, kErrTmemEmptyTimeout, w)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * 256;
        bool ok = true;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&full_bar[stage], phase, abort_flag, p.status, kErrFullBarrierTimeout, w)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * kPairStageBytes);
          const uint32_t sb = sa + kBM * kBK * 2;
#pragma unroll
          for (int k16 = 0; k16 < kBK / 16; ++k16) {
            const uint64_t da = A_KMAJOR ? make_smem_desc(sa + k16 * 32, 16, 1024)
                                         : make_smem_desc(sa + k16 * 2048, kGemmMnLbo, kGemmMnSbo);
            const uint64_t db = B_KMAJOR ? make_smem_desc(sb + k16 * 32, 16, 1024)
                                         : make_smem_desc(sb + k16 * 2048, kGemmMnLbo, kGemmMnSbo);
            tc_mma_f16_pair(d_tmem, da, db, idesc, (kb > kb0 || k16 > 0) ? 1u : 0u);
          }
          tc_commit_pair(&empty_bar[stage]);
          if (++stage == kPairStages) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        tc_commit_pair(&tfull_bar[acc]);
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (8 warps of each CTA, its 128 rows)
    using OutT = typename OutType<InT, OUT_F32>::type;
    const int ew = warp - 2;
    const int quarter = warp & 3;            // TMEM lanes [32*quarter, 32*quarter + 32) (fixed by the hardware)
    const int half = ew >> 2;                // the two warps of a quarter take the 128-byte column chunks in turn
    constexpr int kChunk = 128 / static_cast<int>(sizeof(OutT));
    constexpr int kChunks = kPairBN / kChunk;
    uint8_t* sbuf = stage_out + ew * kEpiBlockBytes;
    OutT* out = reinterpret_cast<OutT*>(p.out);
    InT* zout = reinterpret_cast<InT*>(p.z_out);
    int it = 0;
    for (int w = first; w < total_work && !*abort_flag; w += stride, ++it) {
      int tile_m, tile_n, kb0, kb1;
      work.decode(w, tile_m, tile_n, kb0, kb1);
      const int acc = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1;
      if (!mbar_wait(&tfull_bar[acc], acc_phase, abort_flag, p.status, kErrTmemFullTimeout, w)) break;
      tc_fence_after();
      const int row0 = tile_m * 2 * kBM + static_cast<int>(rank) * kBM + quarter * 32;
      const int row = row0 + lane;
      const bool add_bias = p.bias != nullptr && kb0 == 0;   // split-K: only the first split adds it
      const uint32_t t_addr = tmem_base + acc * 256 + (static_cast<uint32_t>(quarter * 32) << 16);
      const uint32_t release = map_to_rank(&tempty_bar[acc], 0);
      const int colbase = tile_n * kPairBN;
      const int live_chunks = min(kChunks, (p.N - colbase + kChunk - 1) / kChunk);
      if (half >= live_chunks) {             // no column for this warp
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(release);
        continue;
      }
#pragma unroll 1
      for (int c = half; c < live_chunks; c += 2) {
        const int col0 = colbase + c * kChunk;
        const bool last = c + 2 >= live_chunks;
        if (!p.tma_store) {
          // direct stores: row pitch or base not 16-byte aligned
#pragma unroll 1
          for (int s = 0; s < kChunk; s += 32) {
            uint32_t r[32];
            tmem_ld_32x32(t_addr + c * kChunk + s, r);
            tmem_wait_ld();
            const int left = p.N - col0 - s;
            if (row < p.M && left > 0) {
              float v[32];
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
              if (add_bias) {
#pragma unroll
                for (int j = 0; j < 32; ++j)
                  if (j < left) v[j] += __ldg(p.bias + col0 + s + j);
              }
              const size_t at = static_cast<size_t>(row) * p.ldo + col0 + s;
              if (p.z_out != nullptr) store_row<InT>(zout + at, v, false, left);
              if (p.act == kActGelu) {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = gelu_fast(v[j]);
              } else if (p.act == kActRelu) {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.f);
              }
              if (OUT_F32 && p.splits > 1) red_row(reinterpret_cast<float*>(out + at), v, false, left);
              else store_row<OutT>(out + at, v, false, left);
            }
          }
          if (last) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(release);
          }
          continue;
        }
        float v[kChunk];
        {
          uint32_t r0[32];
          tmem_ld_32x32(t_addr + c * kChunk, r0);
          if constexpr (kChunk == 64) {
            uint32_t r1[32];
            tmem_ld_32x32(t_addr + c * kChunk + 32, r1);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; ++j) v[32 + j] = __uint_as_float(r1[j]);
          } else {
            tmem_wait_ld();
          }
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r0[j]);
        }
        if (last) {
          // every column of this warp's part has been read: the leader may overwrite the accumulator
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(release);
        }
        if (add_bias) {
#pragma unroll
          for (int j = 0; j < kChunk; ++j) v[j] += (col0 + j < p.N) ? __ldg(p.bias + col0 + j) : 0.f;
        }
        if constexpr (!OUT_F32) {
          if (p.z_out != nullptr) {
            if (lane == 0) bulk_wait_group_read0();
            __syncwarp();
            stage_row_16bit<InT>(sbuf, lane, v);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
              tma_store_2d(&tma_z, sbuf, col0, row0);
              bulk_commit_group();
            }
          }
        }
        if (p.act == kActGelu) {
#pragma unroll
          for (int j = 0; j < kChunk; ++j) v[j] = gelu_fast(v[j]);
        } else if (p.act == kActRelu) {
#pragma unroll
          for (int j = 0; j < kChunk; ++j) v[j] = fmaxf(v[j], 0.f);
        }
        if (lane == 0) bulk_wait_group_read0();       // the previous store of this warp has finished reading sbuf
        __syncwarp();
        if constexpr (OUT_F32) stage_row_f32(sbuf, lane, v);
        else stage_row_16bit<InT>(sbuf, lane, v);
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
          if (OUT_F32 && p.splits > 1) tma_reduce_add_2d(&tma_out, sbuf, col0, row0);
          else tma_store_2d(&tma_out, sbuf, col0, row0);
          bulk_commit_group();
        }
      }
    }
    if (lane == 0) bulk_wait_group0();     // the tile stores must have left shared memory (and landed) before exit
  }

  // ---------------------------------------------------------------------- teardown
  if (*abort_flag) {
    // give copies that are still in flight time to land before shared memory and TMEM are released
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  __syncwarp();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

template <bool AK, bool BK_, typename InT, bool OUT_F32>
static void launch_pair(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& to, const CUtensorMap& tz,
                        const GemmParams& p, int pairs, cudaStream_t stream) {
  auto kern = gemm_pair_kernel<AK, BK_, InT, OUT_F32>;
  static bool configured = false;
  if (!configured) {
    C10_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmemBytes));
    configured = true;
  }
  kern<<<2 * pairs, kGemmThreadsV2, kPairSmemBytes, stream>>>(ta, tb, to, tz, p);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
}

template <typename InT, bool OUT_F32>
static void dispatch_pair(bool ak, bool bk, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& to,
                          const CUtensorMap& tz, const GemmParams& p, int pairs, cudaStream_t s) {
  if (ak && bk) launch_pair<true, true, InT, OUT_F32>(ta, tb, to, tz, p, pairs, s);
  else if (ak && !bk) launch_pair<true, false, InT, OUT_F32>(ta, tb, to, tz, p, pairs, s);
  else if (!ak && bk) launch_pair<false, true, InT, OUT_F32>(ta, tb, to, tz, p, pairs, s);
  else launch_pair<false, false, InT, OUT_F32>(ta, tb, to, tz, p, pairs, s);
}

// k-blocks from which a 16-bit product is faster in pairs, by its waves over 74 pairs.  Pairs win 7 to 10 % of the MMAs' time and
// lose 1.6 us at the start (cluster barriers) and some of a short tile's epilogue, most with GELU.  Time in pairs over time in single
// CTAs, 2172 shapes in turn; K-major B (forward) / MN-major B (data gradient):
//   one wave    32 k-blocks 1.09 / 1.06, 48 1.07 / 1.04, 80 1.02 / 1.00, 128 1.00 / 0.98
//   two waves   16 k-blocks 1.04 / 0.99, 25 1.03 / 1.00, 40 0.99 / 0.97, 80 0.92 / 0.93
//   three       12 k-blocks 1.01 / 0.97, 20 1.01 / 0.98, 25 0.99 / 0.97; with a pre-activation copy 0.97 from 12 on
//   more        8 k-blocks 1.06 / 0.99, 12 0.96 / 0.93, 16 0.94 / 0.92; with GELU 12 1.07, 16 1.02, 20 0.97, 25 0.97
static int pair_min_kb(const GemmArgs& g, int64_t waves) {
  const bool kmajor = g.trans_b;
  const int kb = waves == 1 ? (kmajor ? 128 : 72) : waves == 2 ? (kmajor ? 40 : 24) : waves == 3 && kmajor && g.z_out == nullptr ? 24 : 12;
  return g.act == kActGelu ? std::max(kb, 20) : kb;
}

// Split-K factor for pairs, or 0 where the single-CTA kernel stays: products with an extent that half a tile covers, those
// of too few k-blocks, and those that take more waves of pairs than of single CTAs (333 x 10240 x 2560: two waves instead of one,
// 33.9 us and 20.3).
// A weight gradient has few, very long tiles (K = tokens), so K is split to fill the waves: a wave costs the k-blocks of a
// tile plus about 3 for what does not overlap, a split about 2 k-blocks per million outputs for its partial sums.  Best of
// a sweep: 6400 x 1600 x 32768 two splits, 1600 x 1600 three, 768 x 768 x 50432 eight, 4800 x 1600 x 32768 one.  With fp32
// outputs pairs pay from 32 k-blocks over all waves (2048 x 2048 x 2000: 18.4 and 17.9 us), of at least 8 each (50304 x 768, 6
// k-blocks: 42.9 and 47.4; 8: 51.6 and 50.7); with split K from 28 (768 x 768 x 2000, 4 splits of 8: 10.9 and 12.0; 2304 x 768 x
// 3000, 2 of 24: 17.9 and 18.1; x 4096, 2 of 32: 21.1 and 20.8).
int gemm_pair_splits(const GemmArgs& g) {
  if (g.M <= kBM || g.N <= kPairBN / 2 || (g.out_f32 && g.z_out != nullptr)) return 0;
  const int kb = (g.K + kBK - 1) / kBK, pairs = g.num_sms / 2;
  const int64_t tiles = static_cast<int64_t>((g.M + 2 * kBM - 1) / (2 * kBM)) * ((g.N + kPairBN - 1) / kPairBN);
  const int64_t waves1 = (tiles + pairs - 1) / pairs;
  const int64_t single = (static_cast<int64_t>((g.M + kBM - 1) / kBM) * ((g.N + kPairBN - 1) / kPairBN) + g.num_sms - 1) / g.num_sms;
  const bool more_waves = waves1 * 14 > single * 15;
  if (!g.out_f32) return more_waves || kb < pair_min_kb(g, waves1) ? 0 : 1;
  const int max_split = g.allow_split_k ? std::min(32, std::max(1, kb / 8)) : 1;
  int best = 1, best_per = kb;
  int64_t best_waves = waves1;
  double best_time = 0.0;
  for (int sp = 1; sp <= max_split; ++sp) {
    const int per = (kb + sp - 1) / sp;
    if ((kb + per - 1) / per != sp) continue;              // no split may be empty: its accumulator would be stale TMEM
    const int64_t waves = (tiles * sp + pairs - 1) / pairs;
    double t = static_cast<double>(waves) * (per + 3.0);
    if (sp > 1) t += 2e-6 * sp * g.M * static_cast<double>(g.N) + 4.0;       // 4: the memset
    if (sp == 1 || t < best_time) { best = sp; best_time = t; best_per = per; best_waves = waves; }
  }
  if (best > 1) return best_waves * best_per >= 28 ? best : 0;
  return more_waves || kb < 8 || waves1 * kb < 32 ? 0 : 1;
}

void gemm_pair_launch(const GemmArgs& g, int splits, cudaStream_t stream) {
  const bool ak = !g.trans_a, bk = g.trans_b;
  const int64_t tiles = static_cast<int64_t>((g.M + 2 * kBM - 1) / (2 * kBM)) * ((g.N + kPairBN - 1) / kPairBN);
  if (splits > 1) C10_CUDA_CHECK(cudaMemsetAsync(g.out, 0, static_cast<size_t>(g.M) * g.N * sizeof(float), stream));
  CUtensorMap ta = ak ? make_tma_2d(g.a, g.M, g.K, g.K, kBM) : make_tma_2d(g.a, g.K, g.M, g.M, 64);
  CUtensorMap tb = bk ? make_tma_2d(g.b, g.N, g.K, g.K, kPairBN / 2) : make_tma_2d(g.b, g.K, g.N, g.N, 64);
  GemmParams p;
  p.M = g.M; p.N = g.N; p.K = g.K;
  p.out = g.out; p.z_out = g.z_out; p.bias = g.bias; p.ldo = g.N;
  p.act = g.act; p.splits = splits; p.is_bf16 = g.is_bf16 ? 1 : 0;
  p.status = g.status;
  const int out_bytes = g.out_f32 ? 4 : 2;
  const bool out_ok = (reinterpret_cast<uintptr_t>(g.out) & 15) == 0 && (static_cast<size_t>(g.N) * out_bytes) % 16 == 0;
  const bool z_ok = g.z_out == nullptr || ((reinterpret_cast<uintptr_t>(g.z_out) & 15) == 0 && (static_cast<size_t>(g.N) * 2) % 16 == 0);
  p.tma_store = (out_ok && z_ok) ? 1 : 0;
  CUtensorMap to = ta, tz = ta;      // placeholders when unused
  if (p.tma_store) {
    to = make_tma_2d_store(g.out, g.M, g.N, g.N, out_bytes, g.is_bf16);
    if (g.z_out != nullptr) tz = make_tma_2d_store(g.z_out, g.M, g.N, g.N, 2, g.is_bf16);
  }
  const int pairs = static_cast<int>(std::min<int64_t>(tiles * splits, g.num_sms / 2));
  if (g.is_bf16) {
    if (g.out_f32) dispatch_pair<__nv_bfloat16, true>(ak, bk, ta, tb, to, tz, p, pairs, stream);
    else dispatch_pair<__nv_bfloat16, false>(ak, bk, ta, tb, to, tz, p, pairs, stream);
  } else {
    if (g.out_f32) dispatch_pair<__half, true>(ak, bk, ta, tb, to, tz, p, pairs, stream);
    else dispatch_pair<__half, false>(ak, bk, ta, tb, to, tz, p, pairs, stream);
  }
}

}  // namespace cw
