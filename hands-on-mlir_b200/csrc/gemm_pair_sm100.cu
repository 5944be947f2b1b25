// fp16 GEMM on CTA pairs (tcgen05 cta_group::2): a cluster of two CTAs on neighbouring SMs
// computes a 256 x BN2 output tile.  Each CTA loads its own 128 rows of A and its own BN2/2
// columns of B per K block (plain per-CTA TMA loads whose byte counts complete on the even
// CTA's mbarrier), one thread of the even CTA issues tcgen05.mma for the whole 256 x BN2 x 16
// step, and each CTA drains its 128 accumulator rows from its own tensor memory.  Compared
// with one CTA per 128 x 256 tile this halves the B bytes every SM pulls through L2 and
// shared memory for the same MMA time, which is what the TMA ring needs to keep the tensor
// pipe fed; the freed shared memory holds five stages and the epilogue staging.
//
//   warps 0, 2  TMA producers of A and of B
//   warp 1      tensor-memory allocation (both CTAs) and MMA issue (even CTA only)
//   warps 3-18  epilogue: four warps per tensor-memory lane quarter, each draining one
//               64-column group of the tile: tcgen05.ld, fp32 alpha/beta/bias/erf-GELU, fp16
//               results staged in swizzled shared memory and written out by TMA stores
//
// Hand-offs: full[s] lives in the even CTA (armed by its producer for the bytes of both CTAs);
// empty[s] and acc_full[a] exist in both CTAs and are signalled by tcgen05.commit addressed to
// both; acc_empty[a] lives in the even CTA (32 arrivals: 16 epilogue warps x 2 CTAs).
// A work unit is a 256 x BN2 tile or one of the `split_k` K ranges of a tile (SplitK,
// gemm_epilogue.cuh).
#include <cstdio>
#include <cstdlib>

#include "gemm_epilogue.cuh"
#include "gemm_sm100.cuh"
#include "ptx_sm100.cuh"

namespace hom {
namespace gemm {

using namespace hom::ptx;

namespace {

constexpr int BK = 64;
constexpr int kPairThreads = 32 * (kControlWarps + kEpilogueWarps);
constexpr uint32_t kABytes = 128 * BK * 2;

template <int BN2>
struct PairCfg {
  static constexpr int kHalfN = BN2 / 2;
  static constexpr uint32_t kBBytes = kHalfN * BK * 2;
  static constexpr uint32_t kStageBytes = kABytes + kBBytes;
  static constexpr int kStages = BN2 == 256 ? 5 : 8;
  static constexpr uint32_t kTmemCols = 2 * BN2;  // two accumulators; 512 or 256
  static constexpr uint32_t kStagingBytes = BN2 / 64 * 4 * kEpilogueStageBytes;
  static constexpr uint32_t kBarrierBytes = 8 * (2 * kStages + 4) + 16;
  static constexpr uint32_t kSmemBytes = kStages * kStageBytes + kStagingBytes + kBarrierBytes + 1024;
};

struct PairParams {
  EpilogueParams ep;
  int K;
  int n_blocks, num_tiles, num_kb;
  int b_grouped;  // B [K,N] is fetched through the grouped 3-D tensor map (N % 64 == 0)
  int b_early;    // B is a declared constant: request its first tiles before griddepcontrol.wait
  // Split-K: every tile is cut into `split_k` work units (K-block ranges); num_units = num_tiles
  // * split_k.  Workspace: per (tile, CTA of the pair, epilogue warp) `split_k` fp32 slots and a
  // pair of counters (see SplitK in gemm_epilogue.cuh).
  int split_k, num_units;
  float *ws_slots;
  int *ws_counters;
  int *status;
  HOM_DIAG(long long *prof;)  // optional per-role cycle counters of CTA 0, else null
  HOM_DIAG(long long *tl;)    // optional launch-timeline slot, else null
};

// After an expired wait: gives copies already in flight time to land (about 2 ms) before the
// CTA's shared memory is released.
__device__ __forceinline__ void drain_copies() {
  const long long t0 = clock64();
  while (clock64() - t0 < 4000000LL) {
  }
}

template <int BN2, bool B_NK, bool SPLIT = false, int FORMS = 0, int EPI = 0>
__global__ void __launch_bounds__(kPairThreads, 1)
gemm_f16_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ CUtensorMap tmD, const PairParams p) {
  using Cfg = PairCfg<BN2>;
  constexpr int STAGES = Cfg::kStages;
  constexpr int HALF = Cfg::kHalfN;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t smem_base = (raw_addr + 1023u) & ~1023u;
  uint8_t *smem_gen = smem_raw + (smem_base - raw_addr);

  const uint32_t staging_base = smem_base + STAGES * Cfg::kStageBytes;
  const uint32_t bar_base = staging_base + Cfg::kStagingBytes;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + a); };
  auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + 2 + a); };
  volatile uint32_t *tmem_slot =
      reinterpret_cast<volatile uint32_t *>(smem_gen + STAGES * Cfg::kStageBytes + Cfg::kStagingBytes +
                                            8 * (2 * STAGES + 4));
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();  // 0: even CTA (issues the MMAs), 1: odd CTA
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;

  HOM_DIAG(unsigned long long g_entry = 0; if (p.tl) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(g_entry));
           if (p.tl && threadIdx.x == 0) timeline_stamp(p.tl, 0);)
  // The first TMA instruction stalls until its descriptor has been fetched: start those
  // fetches before anything else so that they overlap the barrier and tensor-memory set-up.
  if (threadIdx.x == 64) {
    prefetch_tensormap(&tmB);
    prefetch_tensormap(&tmA);
    prefetch_tensormap(&tmD);
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull_bar(a), 1);
      mbar_init(tempty_bar(a), 2 * kEpilogueWarps);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(const_cast<uint32_t *>(tmem_slot)), Cfg::kTmemCols);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  cluster_sync_all();  // barriers of both CTAs are initialised before anyone signals them
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  // Dependents may be scheduled only now that this grid's CTAs hold their tensor memory.
  pdl_launch_dependents();
  // longest set-up (entry -> barriers, tensor memory and cluster barrier done) over the CTAs, ns
  HOM_DIAG(if (p.tl && threadIdx.x == 0) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    atomicMax(p.tl + 480, static_cast<long long>(t - g_entry));
  })

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer, A
    // One elected lane runs the whole loop; A and B come from two warps (see gemm_sm100.cu).
    if (elect_one()) {
      // Copies of both CTAs complete on the even CTA's barriers, which the even CTA's A producer
      // arms for the bytes of all four (copies may land first: the phase needs the arrival).
      const uint32_t full_even = map_to_cta(full_bar(0), 0);
      uint32_t dst = smem_base, slot = 0, ph = 0;
      bool ok = true;
      HOM_DIAG(long long t_wait = 0; const long long t_begin = clock64();)
      auto advance = [&]() {
        dst += Cfg::kStageBytes;
        slot += 8;
        if (slot == 8 * STAGES) {
          dst = smem_base;
          slot = 0;
          ph ^= 1u;
        }
      };
      // The first ring is armed before the wait for the previous kernel (gemm_sm100.cu).
      int ready = 0;
      if (pair < p.num_units) {
        const int part0 = pair % p.split_k;
        ready = min(STAGES, (part0 + 1) * p.num_kb / p.split_k - part0 * p.num_kb / p.split_k);
        if (rank == 0)
          for (int i = 0; i < ready; ++i) mbar_arrive_expect_tx(full_bar(i), 2 * Cfg::kStageBytes);
      }
      pdl_wait();
      HOM_DIAG(if (p.tl) timeline_stamp(p.tl, 2);)
      for (int unit = pair; unit < p.num_units && ok; unit += num_pairs) {
        const int tile = unit / p.split_k, part = unit % p.split_k;
        const int m0 = (tile / p.n_blocks) * 256 + static_cast<int>(rank) * 128;
        const int k_end = (part + 1) * p.num_kb / p.split_k * BK;
        int k = part * p.num_kb / p.split_k * BK;
        for (; ready > 0; --ready, k += BK) {
          tma_load_2d_pair(dst, &tmA, full_even + slot, k, m0);
          advance();
        }
        for (; k < k_end; k += BK) {
          HOM_DIAG(const long long tw = p.prof ? clock64() : 0;)
          ok = mbar_wait(empty_bar(0) + slot, ph ^ 1u, abort_flag, p.status, kDevWaitTimeoutProducer);
          if (!ok) break;
          HOM_DIAG(if (p.prof) t_wait += clock64() - tw;)
          if (rank == 0) mbar_arrive_expect_tx(full_bar(0) + slot, 2 * Cfg::kStageBytes);
          tma_load_2d_pair(dst, &tmA, full_even + slot, k, m0);
          advance();
        }
      }
      HOM_DIAG(if (p.prof && blockIdx.x < 2) {
        p.prof[0 + 8 * blockIdx.x] = clock64() - t_begin;
        p.prof[1 + 8 * blockIdx.x] = t_wait;
      })
      if (!ok) drain_copies();
    }
    __syncwarp();
  } else if (warp == 2) {
    // ------------------------------------------------------------ TMA producer, B
    if (elect_one()) {
      const uint32_t full_even = map_to_cta(full_bar(0), 0);
      uint32_t dst = smem_base + kABytes, slot = 0, ph = 0;
      bool ok = true;
      const bool b_grouped = p.b_grouped != 0;
      // A declared constant is requested without waiting for the previous kernel (gemm_sm100.cu).
      if (!p.b_early) pdl_wait();
      for (int unit = pair; unit < p.num_units && ok; unit += num_pairs) {
        const int tile = unit / p.split_k, part = unit % p.split_k;
        const int nb0 = (tile % p.n_blocks) * BN2 + static_cast<int>(rank) * HALF;
        const int k_end = (part + 1) * p.num_kb / p.split_k * BK;
        for (int k = part * p.num_kb / p.split_k * BK; k < k_end; k += BK) {
          ok = mbar_wait(empty_bar(0) + slot, ph ^ 1u, abort_flag, p.status, kDevWaitTimeoutProducer);
          if (!ok) break;
          if (B_NK) {
            tma_load_2d_pair(dst, &tmB, full_even + slot, k, nb0);
          } else if (b_grouped) {
            tma_load_3d_pair(dst, &tmB, full_even + slot, 0, k, nb0 / 64);
          } else {
#pragma unroll
            for (int g = 0; g < HALF / 64; ++g)
              tma_load_2d_pair(dst + g * (BK * 128), &tmB, full_even + slot, nb0 + g * 64, k);
          }
          dst += Cfg::kStageBytes;
          slot += 8;
          if (slot == 8 * STAGES) {
            dst = smem_base + kABytes;
            slot = 0;
            ph ^= 1u;
          }
        }
      }
      if (!ok) drain_copies();
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------- MMA issuer (even CTA only)
    // One elected lane runs the whole loop (see gemm_sm100.cu).
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = make_idesc_f16(256, BN2, false, !B_NK);
      const uint64_t da0 = make_smem_desc_sw128(smem_base, 16, 1024);
      const uint64_t db0 = make_smem_desc_sw128(smem_base + kABytes, B_NK ? 16 : BK * 128, 1024);
      uint64_t da = da0, db = db0;
      uint32_t bar = full_bar(0), ph = 0;
      bool ok = true;
      int it = 0;
      HOM_DIAG(long long t_full = 0, t_acc = 0; const long long t_begin = clock64();)
      for (int unit = pair; unit < p.num_units && ok; unit += num_pairs, ++it) {
        const int part = unit % p.split_k;
        const int num_kb = (part + 1) * p.num_kb / p.split_k - part * p.num_kb / p.split_k;
        const int acc = it & 1;
        const uint32_t acc_ph = (it >> 1) & 1;
        HOM_DIAG(const long long ta = p.prof ? clock64() : 0;)
        ok = mbar_wait(tempty_bar(acc), acc_ph ^ 1u, abort_flag, p.status, kDevWaitTimeoutMma);
        if (!ok) break;
        HOM_DIAG(if (p.prof) t_acc += clock64() - ta;)
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + acc * BN2;
        for (int kb = 0; kb < num_kb; ++kb) {
          HOM_DIAG(const long long tw = p.prof ? clock64() : 0;)
          ok = mbar_wait(bar, ph, abort_flag, p.status, kDevWaitTimeoutMma);
          if (!ok) break;
          HOM_DIAG(if (p.prof) t_full += clock64() - tw;)
          tc_fence_after_sync();
          HOM_DIAG(if (p.tl && it == 0 && kb == 0) timeline_stamp(p.tl, 6);)
          tc_mma_f16_ss_pair(d_tmem, da, db, idesc, kb != 0 ? 1u : 0u);
#pragma unroll
          for (int k = 1; k < BK / 16; ++k)
            tc_mma_f16_ss_pair(d_tmem, smem_desc_advance(da, k * 32), smem_desc_advance(db, B_NK ? k * 32 : k * 2048),
                               idesc, 1u);
          tc_commit_pair(bar + 8u * STAGES, 0x3);  // frees the stage in both CTAs
          da = smem_desc_advance(da, Cfg::kStageBytes);
          db = smem_desc_advance(db, Cfg::kStageBytes);
          bar += 8;
          if (bar == full_bar(STAGES)) {
            da = da0;
            db = db0;
            bar = full_bar(0);
            ph ^= 1u;
          }
        }
        if (ok) tc_commit_pair(tfull_bar(acc), 0x3);  // accumulator ready in both CTAs
      }
      HOM_DIAG(if (p.prof && blockIdx.x == 0) {
        p.prof[2] = clock64() - t_begin;
        p.prof[3] = t_full;
        p.prof[4] = t_acc;
      })
    }
    __syncwarp();
  } else if (warp >= kControlWarps) {
    // --------------------------------------------------------------- epilogue
    const int quarter = warp & 3;       // tensor-memory lanes [32*quarter, +32)
    const int group = (warp - kControlWarps) >> 2;  // which 64-column group of the tile
    const int col_begin = group * 64;
    const bool active = col_begin < BN2;
    const uint32_t stage_smem = staging_base + (warp - kControlWarps) * kEpilogueStageBytes;
    int it = 0;
    HOM_DIAG(long long t_wait = 0; const long long t_begin = clock64();)
    pdl_wait();  // C may be produced, and D still read, by the previous kernel
    float2 next_col_sums = make_float2(0.f, 0.f);
    if constexpr ((FORMS & kFormLnA) != 0) {
      if (active && pair < p.num_units)
        next_col_sums = epilogue_load_col_sums(p.ep, (pair % p.n_blocks) * BN2 + col_begin, lane);
    }
    for (int unit = pair; unit < p.num_units; unit += num_pairs, ++it) {
      const int tile = unit / p.split_k;
      const int acc = it & 1;
      const uint32_t acc_ph = (it >> 1) & 1;
      const int m0 = (tile / p.n_blocks) * 256 + static_cast<int>(rank) * 128;
      const int n0 = (tile % p.n_blocks) * BN2 + col_begin;
      uint4 cval[8];
      SplitK sk;
      if constexpr (SPLIT) {
        // this warp's block of the tile: (tile, CTA of the pair, epilogue warp)
        const size_t block = (static_cast<size_t>(tile) * 2 + rank) * kEpilogueWarps + (warp - kControlWarps);
        sk.parts = p.split_k;
        sk.part = unit % p.split_k;
        sk.slot = p.ws_slots + block * kSplitSlotFloats;
        sk.counter = p.ws_counters + block;
      } else {
        if constexpr (EPI == kEpiGeneric || EPI == kEpiAddC) {
          if (active) epilogue_load_c<0, 8, EPI != kEpiGeneric || FORMS != 0>(p.ep, m0 + quarter * 32 + lane, n0, cval);
        }
      }
      RowAffine ra;
      float2 col_sums = make_float2(0.f, 0.f);
      if constexpr ((FORMS & (kFormLnA | kFormLnR)) != 0) {
        if (active) ra = epilogue_row_affine(p.ep, m0 + quarter * 32 + lane);
      }
      if constexpr ((FORMS & kFormLnA) != 0) {
        col_sums = next_col_sums;
        const int next = unit + num_pairs;
        if (active && next < p.num_units)
          next_col_sums = epilogue_load_col_sums(p.ep, (next % p.n_blocks) * BN2 + col_begin, lane);
      }
      HOM_DIAG(const long long tw = p.prof ? clock64() : 0;)
      bool ok = mbar_wait(tfull_bar(acc), acc_ph, abort_flag, p.status, kDevWaitTimeoutEpilogue);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      HOM_DIAG(if (p.prof) t_wait += clock64() - tw;)
      HOM_DIAG(if (p.tl && warp == kControlWarps && lane == 0 && unit + num_pairs >= p.num_units)
                   timeline_stamp(p.tl, 8);)
      tc_fence_after_sync();
      auto release = [&]() {
        if (lane == 0) {
          if (rank == 0) mbar_arrive(tempty_bar(acc));
          else mbar_arrive_cluster(map_to_cta(tempty_bar(acc), 0));
        }
      };
      const uint32_t t_row =
          tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * BN2 + col_begin;
      if (!epilogue_warp_block<SPLIT, FORMS, EPI>(p.ep, &tmD, t_row, m0 + quarter * 32, n0, active, stage_smem, lane,
                                             cval, release, sk, abort_flag, p.status, ra, col_sums))
        break;
    }
    // A store still in flight reads this warp's staging tile: let it finish reading.
    if (lane == 0) bulk_wait_group_read_0();
    __syncwarp();
    HOM_DIAG(if (p.prof && blockIdx.x == 0 && threadIdx.x == 32 * kControlWarps) {
      p.prof[5] = clock64() - t_begin;
      p.prof[6] = t_wait;
    })
  }

  // Nobody leaves while the other CTA may still read this CTA's shared memory (MMA operand
  // fetch) or signal its barriers.
  tc_fence_before_sync();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, Cfg::kTmemCols);
  }
  HOM_DIAG(if (p.tl && threadIdx.x == 0) timeline_stamp(p.tl, 4);)
}

template <int BN2, bool B_NK>
bool launch_pair_variant(const Problem &pb, int split_k, cudaStream_t stream) {
  using Cfg = PairCfg<BN2>;
  static bool attr_set[64] = {};
  static int max_clusters[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  // the whole-K kernel without LayerNorm forms: generic, or one of the three specialised epilogues
  const int epi = epilogue_kind(pb);
  auto kernel = epi == kEpiPlain  ? gemm_f16_pair_kernel<BN2, B_NK, false, 0, kEpiPlain>
                : epi == kEpiGelu ? gemm_f16_pair_kernel<BN2, B_NK, false, 0, kEpiGelu>
                : epi == kEpiAddC ? gemm_f16_pair_kernel<BN2, B_NK, false, 0, kEpiAddC>
                                  : gemm_f16_pair_kernel<BN2, B_NK>;
  auto kernel_split = gemm_f16_pair_kernel<BN2, B_NK, true>;
  // the LayerNorm forms of the epilogue: on A only / on the residual + statistics / any mix
  const int forms = layernorm_forms(pb);
  auto kernel_forms = forms == kFormLnA ? gemm_f16_pair_kernel<BN2, B_NK, false, kFormLnA>
                      : (forms & kFormLnA) == 0 ? gemm_f16_pair_kernel<BN2, B_NK, false, kFormLnR | kFormStats>
                                                : gemm_f16_pair_kernel<BN2, B_NK, false, kFormLnA | kFormLnR | kFormStats>;

  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  cfg.blockDim = dim3(kPairThreads);
  cfg.dynamicSmemBytes = Cfg::kSmemBytes;
  cfg.stream = stream;

  if (!attr_set[dev]) {
    if (!check_cuda(cudaFuncSetAttribute(gemm_f16_pair_kernel<BN2, B_NK>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         Cfg::kSmemBytes),
                    "cudaFuncSetAttribute(gemm pair)") ||
        !check_cuda(cudaFuncSetAttribute(gemm_f16_pair_kernel<BN2, B_NK, false, 0, kEpiPlain>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes),
                    "cudaFuncSetAttribute(gemm pair, plain)") ||
        !check_cuda(cudaFuncSetAttribute(gemm_f16_pair_kernel<BN2, B_NK, false, 0, kEpiGelu>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes),
                    "cudaFuncSetAttribute(gemm pair, GELU)") ||
        !check_cuda(cudaFuncSetAttribute(gemm_f16_pair_kernel<BN2, B_NK, false, 0, kEpiAddC>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes),
                    "cudaFuncSetAttribute(gemm pair, + C)") ||
        !check_cuda(cudaFuncSetAttribute(gemm_f16_pair_kernel<BN2, B_NK, false, kFormLnA>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes),
                    "cudaFuncSetAttribute(gemm pair, LayerNorm on A)") ||
        !check_cuda(cudaFuncSetAttribute(gemm_f16_pair_kernel<BN2, B_NK, false, kFormLnR | kFormStats>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes),
                    "cudaFuncSetAttribute(gemm pair, LayerNorm on the residual)") ||
        !check_cuda(cudaFuncSetAttribute(gemm_f16_pair_kernel<BN2, B_NK, false, kFormLnA | kFormLnR | kFormStats>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes),
                    "cudaFuncSetAttribute(gemm pair, LayerNorm forms)") ||
        !check_cuda(cudaFuncSetAttribute(kernel_split, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         Cfg::kSmemBytes),
                    "cudaFuncSetAttribute(gemm pair, split-K)"))
      return false;
    // How many CTA pairs the device can hold at once (pairs need neighbouring SMs).
    cfg.gridDim = dim3(2 * (sm_count() / 2));
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      n = sm_count() / 2;
    }
    HOM_DIAG(if (const char *env = std::getenv("HOM_GEMM_PAIRS")) {  // experiment knob
      const int v = std::atoi(env);
      if (v >= 1) n = v;
    }
    if (std::getenv("HOM_DEBUG"))
      fprintf(stderr, "[hom] gemm pair BN2=%d nk=%d: %d co-resident CTA pairs\n", BN2, int(B_NK), n);)
    max_clusters[dev] = n;
    attr_set[dev] = true;
  }

  CUtensorMap tmA, tmB, tmD;
  if (!make_tensor_map_2d(pb.A, pb.K, pb.M, BK, 128, &tmA)) return false;
  if (pb.N % 8 == 0) {
    if (!make_tensor_map_2d(pb.D, pb.N, pb.M, 64, 32, &tmD)) return false;
  } else {
    tmD = tmA;  // never dereferenced: the epilogue stores without TMA when N % 8 != 0
  }
  const bool grouped = !B_NK && pb.N % 64 == 0;
  if (B_NK) {
    if (!make_tensor_map_2d(pb.B, pb.K, pb.N, BK, Cfg::kHalfN, &tmB)) return false;
  } else if (grouped) {
    if (!make_tensor_map_grouped(pb.B, pb.N, pb.K, BK, Cfg::kHalfN / 64, &tmB)) return false;
  } else {
    if (!make_tensor_map_2d(pb.B, pb.N, pb.K, 64, BK, &tmB, pb.ldb)) return false;
  }
  PairParams p;
  p.b_grouped = grouped ? 1 : 0;
  p.b_early = pb.b_const ? 1 : 0;
  p.ep.C = pb.C;
  p.ep.ldc = pb.N;
  p.ep.c_mode = pb.c_mode;
  p.ep.D = pb.D;
  p.ep.ldd = pb.N;
  p.ep.alpha = pb.alpha;
  p.ep.beta = pb.beta;
  p.ep.act = pb.act;
  p.ep.row_scale = pb.row_scale;
  p.ep.row_shift = pb.row_shift;
  p.ep.col_sum = pb.col_sum;
  p.ep.a_partials = pb.a_partials;
  p.ep.r_partials = pb.r_partials;
  p.ep.a_groups = pb.a_groups;
  p.ep.r_groups = pb.r_groups;
  p.ep.a_inv_n = pb.K > 0 ? 1.f / static_cast<float>(pb.K) : 0.f;
  p.ep.r_inv_n = pb.N > 0 ? 1.f / static_cast<float>(pb.N) : 0.f;
  p.ep.ln_eps = pb.ln_eps;
  p.ep.unaligned_n = pb.N % 8 != 0 ? 1 : 0;
  p.ep.row_partials = pb.row_partials;
  p.ep.M = static_cast<int>(pb.M);
  p.ep.N = static_cast<int>(pb.N);
  p.K = static_cast<int>(pb.K);
  const int m_blocks = static_cast<int>((pb.M + 255) / 256);
  p.n_blocks = static_cast<int>((pb.N + BN2 - 1) / BN2);
  p.num_tiles = m_blocks * p.n_blocks;
  p.num_kb = static_cast<int>((pb.K + BK - 1) / BK);
  p.status = device_status_word();
  HOM_DIAG(p.prof = profile_buffer(); p.tl = launch_timeline_slot();)
  p.split_k = split_k < 1 || has_layernorm_form(pb) ? 1 : split_k > 16 ? 16 : split_k;
  if (p.split_k > p.num_kb) p.split_k = p.num_kb;
  p.num_units = p.num_tiles * p.split_k;
  p.ws_slots = nullptr;
  p.ws_counters = nullptr;
  if (p.split_k > 1) {
    const size_t blocks = static_cast<size_t>(p.num_tiles) * 2 * kEpilogueWarps;
    SplitWorkspace ws;
    if (!split_workspace(blocks * kSplitSlotFloats, blocks, stream, &ws)) return false;
    p.ws_slots = ws.slots;
    p.ws_counters = ws.counters;
  }
  const int pairs = p.num_units < max_clusters[dev] ? p.num_units : max_clusters[dev];
  cfg.gridDim = dim3(2 * pairs);
  const double flops = 2.0 * pb.M * pb.N * pb.K;
  const double bytes = 2.0 * (static_cast<double>(pb.M) * pb.K + static_cast<double>(pb.K) * pb.N +
                              static_cast<double>(pb.M) * pb.N) +
                       (pb.c_mode == 1 ? 2.0 * pb.M * pb.N : pb.c_mode == 2 ? 2.0 * pb.N : 0.0);
  LaunchScope scope(kOpGemm, flops, bytes);
  if (!check_cuda(cudaLaunchKernelEx(&cfg, forms != 0 ? kernel_forms : p.split_k > 1 ? kernel_split : kernel,
                                     tmA, tmB, tmD, p),
                  "gemm pair kernel launch"))
    return false;
  HOM_DIAG(if (p.prof) profile_report("gemm CTA-pair", p.num_tiles, 2 * pairs, p.num_kb, stream);)
  return check_cuda(cudaGetLastError(), "gemm pair kernel launch");
}

}  // namespace

bool run_pair(const Problem &pb, int bn2, int split_k, cudaStream_t stream) {
  if (pb.b_is_nk) {
    return bn2 == 128 ? launch_pair_variant<128, true>(pb, split_k, stream)
                      : launch_pair_variant<256, true>(pb, split_k, stream);
  }
  return bn2 == 128 ? launch_pair_variant<128, false>(pb, split_k, stream)
                    : launch_pair_variant<256, false>(pb, split_k, stream);
}

}  // namespace gemm
}  // namespace hom
