// fp16 GEMM for few output tiles: one 128 x BN tile per thread-block cluster, its K range cut
// over the CTAs of the cluster and reduced through distributed shared memory.
//
// With the rows of one to a few sequences (M up to about a thousand) a layer's GEMMs have 12 to
// 100 output tiles, and what a launch costs is the chain one CTA goes through: the 64-deep K
// blocks of its tile one after the other, as fast as a single SM can pull them (a 128 x 64 tile
// of K = 3072 is 1.2 MB), on a chip that is mostly idle.  Here S = 2..8 CTAs share a tile, each
// accumulates its K blocks in its own tensor memory (the first six, with 128-column tiles four, are
// requested at once, their weights even before the previous kernel has finished; a longer share
// goes round the ring), and the
// partial tiles are exchanged SM to SM: CTA r of the cluster owns rows [r, r + 1) * ceil(rows / S)
// of the tile, every CTA stores the rows of its partial accumulator straight into their owner's
// shared memory, and after one cluster barrier the owner adds the S parts in part order (the sum
// does not depend on timing: bit-identical from run to run), applies the epilogue and writes full
// rows.  Nothing goes through global scratch, and no CTA waits for another launch's counter.
//
// 320 threads: warp 0 TMA producer, warp 1 MMA issuer, warps 2-9 accumulator exchange + epilogue.
#include <atomic>

#include <cuda_fp16.h>

#include "gemm_epilogue.cuh"
#include "gemm_sm100.cuh"
#include "ptx_sm100.cuh"

namespace hom {
namespace gemm {

using namespace hom::ptx;

namespace {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int kExchangeWarps = 8;
constexpr int kClusterThreads = 32 * (2 + kExchangeWarps);
constexpr uint32_t kABytes = BM * BK * 2;
// sm_100: shared memory of an SM, what each resident CTA takes of it besides its own request, and
// the largest request.
constexpr uint32_t kSmSmem = 228 * 1024, kCtaReservedSmem = 1024, kMaxCtaSmem = 227 * 1024;
// S * ceil(128 / S) rows for S = 2..8 (largest: 7 x 19)
constexpr uint32_t kRecvRows = 136;

template <int BN>
struct ClusterCfg {
  static constexpr uint32_t kBBytes = BN * BK * 2;
  static constexpr uint32_t kStageBytes = kABytes + kBBytes;
  static constexpr int kStages = BN == 64 ? 6 : 4;  // the ring, beside the receive buffer
  static constexpr uint32_t kRecvBytes = kRecvRows * BN * 4;
  static constexpr uint32_t kBarrierBytes = 8 * (2 * kStages + 1) + 16;
  // What the kernel uses (183 / 200 KB), and what it asks for: all that a CTA can have.  Its 320
  // threads leave half of an SM's registers and threads free, and no CTA of this kernel may sit
  // beside a CTA of the previous kernel that it depends on (or of the next one): with all of the
  // shared memory taken nothing else fits, whatever the other kernel needs.
  static constexpr uint32_t kUsedBytes = kStages * kStageBytes + kRecvBytes + kBarrierBytes + 1024;
  static constexpr uint32_t kSmemBytes = kMaxCtaSmem;
  static_assert(kUsedBytes <= kSmemBytes, "ring and receive buffer exceed a CTA's shared memory");
  static_assert(kSmemBytes + 2 * kCtaReservedSmem > kSmSmem, "another CTA would fit beside this one");
};

struct ClusterParams {
  const __half *C;
  __half *D;
  float alpha, beta;
  int c_mode, act;
  int M, N, num_kb, n_blocks;
  int b_early;  // B is a declared constant: request its tiles before griddepcontrol.wait
  int *status;
};

__device__ __forceinline__ uint32_t cluster_nctas() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}

__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d)
               : "memory");
}

template <int BN, bool B_NK>
__global__ void __launch_bounds__(kClusterThreads, 1)
gemm_f16_cluster_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                        const ClusterParams p) {
  using Cfg = ClusterCfg<BN>;
  constexpr int STAGES = Cfg::kStages;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t smem_base = (raw_addr + 1023u) & ~1023u;
  uint8_t *smem_gen = smem_raw + (smem_base - raw_addr);
  constexpr uint32_t kRecvOff = STAGES * Cfg::kStageBytes;
  constexpr uint32_t kBarOff = kRecvOff + Cfg::kRecvBytes;
  auto full_bar = [&](int s) { return smem_base + kBarOff + 8u * s; };
  auto empty_bar = [&](int s) { return smem_base + kBarOff + 8u * (STAGES + s); };
  const uint32_t acc_bar = smem_base + kBarOff + 8u * (2 * STAGES);
  volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(smem_gen + kBarOff + 8 * (2 * STAGES + 1));
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int parts = static_cast<int>(cluster_nctas());
  const int part = static_cast<int>(cluster_ctarank());
  const int tile = static_cast<int>(blockIdx.x) / parts;
  const int m0 = (tile / p.n_blocks) * BM, n0 = (tile % p.n_blocks) * BN;
  const int kb_begin = part * p.num_kb / parts, kb_end = (part + 1) * p.num_kb / parts;
  const int num_kb = kb_end - kb_begin;  // >= 1: the launcher keeps parts <= num_kb

  if (threadIdx.x == 64) {
    prefetch_tensormap(&tmB);
    prefetch_tensormap(&tmA);
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(acc_bar, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t *>(tmem_slot)), BN);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  // (after the tensor-memory allocation, like every kernel of the library that has one)
  pdl_launch_dependents();
  // Cluster barrier, phase 1: "this CTA runs"; its shared memory may be written by its peers.
  // Every thread of every CTA arrives and waits exactly once per phase, on error paths too.
  cluster_arrive();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    auto load_b = [&](uint32_t dst, uint32_t bar, int k) {
      if (B_NK) {
        tma_load_2d(dst, &tmB, bar, k, n0);
      } else {
#pragma unroll
        for (int g = 0; g < BN / 64; ++g) tma_load_2d(dst + g * (BK * 128), &tmB, bar, n0 + g * 64, k);
      }
    };
    if (elect_one()) {
      int pre = 0;
      if (p.b_early) {
        pre = num_kb < STAGES ? num_kb : STAGES;
        for (int i = 0; i < pre; ++i) {
          mbar_arrive_expect_tx(full_bar(i), Cfg::kStageBytes);
          load_b(smem_base + i * Cfg::kStageBytes + kABytes, full_bar(i), (kb_begin + i) * BK);
        }
      }
      pdl_wait();
      uint32_t dst = smem_base, bar = full_bar(0), ph = 0;
      bool ok = true;
      int armed = 0;
      for (int i = 0; i < num_kb; ++i) {
        const int k = (kb_begin + i) * BK;
        if (i >= pre) {
          ok = mbar_wait(bar + 8u * STAGES, ph ^ 1u, abort_flag, p.status, kDevWaitTimeoutProducer);
          if (!ok) break;
          mbar_arrive_expect_tx(bar, Cfg::kStageBytes);
          load_b(dst + kABytes, bar, k);
        }
        tma_load_2d(dst, &tmA, bar, k, m0);
        ++armed;
        dst += Cfg::kStageBytes;
        bar += 8;
        if (bar == full_bar(STAGES)) {
          dst = smem_base;
          bar = full_bar(0);
          ph ^= 1u;
        }
      }
      if (!ok) {
        // Let every copy this thread started land before the CTA gives its shared memory back.
        const long long t0 = clock64();
        for (int st = 0; st < STAGES; ++st) {
          const int n_st = armed / STAGES + (st < armed % STAGES ? 1 : 0);
          if (n_st > 0)
            while (!mbar_try_wait(full_bar(st), (n_st - 1) & 1) && clock64() - t0 < 400000000LL) {
            }
        }
      }
    }
    __syncwarp();
    cluster_wait();
    cluster_arrive();
    cluster_wait();
  } else if (warp == 1) {
    // ------------------------------------------------------------- MMA issuer
    constexpr uint32_t idesc = make_idesc_f16(BM, BN, false, !B_NK);
    if (elect_one()) {
      const uint64_t da0 = make_smem_desc_sw128(smem_base, 16, 1024);
      const uint64_t db0 = make_smem_desc_sw128(smem_base + kABytes, B_NK ? 16 : BK * 128, 1024);
      uint64_t da = da0, db = db0;
      uint32_t bar = full_bar(0), ph = 0;
      bool ok = true;
      for (int i = 0; i < num_kb; ++i) {
        ok = mbar_wait(bar, ph, abort_flag, p.status, kDevWaitTimeoutMma);
        if (!ok) break;
        tc_fence_after_sync();
        tc_mma_f16_ss(tmem_base, da, db, idesc, i != 0 ? 1u : 0u);
#pragma unroll
        for (int k = 1; k < BK / 16; ++k)
          tc_mma_f16_ss(tmem_base, smem_desc_advance(da, k * 32), smem_desc_advance(db, B_NK ? k * 32 : k * 2048),
                        idesc, 1u);
        tc_commit(bar + 8u * STAGES);
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
      if (ok) tc_commit(acc_bar);
    }
    __syncwarp();
    cluster_wait();
    cluster_arrive();
    cluster_wait();
  } else {
    // ------------------------------------------- accumulator exchange and epilogue
    const int rows = min(BM, p.M - m0);             // rows of the tile inside the matrix
    const int rows_per = (rows + parts - 1) / parts;  // rows each CTA of the cluster finishes
    const int row_first = part * rows_per;
    const int my_rows = max(0, min(rows_per, rows - row_first));
    constexpr int kChunks = BN / 8;  // 8-column pieces of an output row
    constexpr int kMaxTasks = (BM / 2) * kChunks / (32 * kExchangeWarps);
    const int t = threadIdx.x - 64;
    const int tasks = my_rows * kChunks;

    pdl_wait();  // C may be produced, and D still read, by the previous kernel
    uint4 cval[kMaxTasks];
#pragma unroll
    for (int i = 0; i < kMaxTasks; ++i) {
      cval[i] = make_uint4(0, 0, 0, 0);
      const int task = t + i * 32 * kExchangeWarps;
      const int col = n0 + (task % kChunks) * 8;
      if (p.c_mode != 0 && task < tasks && col < p.N) {
        const long long row = m0 + row_first + task / kChunks;
        cval[i] = *reinterpret_cast<const uint4 *>(p.C + (p.c_mode == 1 ? row * p.N : 0) + col);
      }
    }

    bool ok = mbar_wait(acc_bar, 0, abort_flag, p.status, kDevWaitTimeoutEpilogue);
    ok = __all_sync(0xffffffffu, ok);
    cluster_wait();  // phase 1: every CTA of the cluster runs
    if (ok) {
      tc_fence_after_sync();
      const int quarter = warp & 3;
      const int row = quarter * 32 + lane;
      const int col_begin = ((warp - 2) >> 2) * (BN / 2);
      if (quarter * 32 < rows) {  // warp-uniform: the accumulator read is warp-collective
        const int owner = row / rows_per;
        const int local = row - owner * rows_per;
        const uint32_t dst = map_to_cta(
            smem_base + kRecvOff + static_cast<uint32_t>(part * rows_per + local) * (BN * 4), static_cast<uint32_t>(min(owner, parts - 1)));
#pragma unroll
        for (int h = 0; h < BN / 64; ++h) {
          uint32_t acc[32];
          tmem_ld_32x32(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + col_begin + h * 32, acc);
          tmem_ld_wait();
          if (row < rows) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              // 16-byte chunks of a row are XOR-swizzled by the row: conflict-free stores
              const uint32_t chunk = static_cast<uint32_t>((col_begin + h * 32) / 4 + j) ^ (local & 7);
              st_cluster_v4(dst + chunk * 16, acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]);
            }
          }
        }
        tc_fence_before_sync();
      }
    }
    cluster_arrive();  // phase 2: the parts are delivered
    cluster_wait();
    if (ok) {
#pragma unroll
      for (int i = 0; i < kMaxTasks; ++i) {
        const int task = t + i * 32 * kExchangeWarps;
        if (task >= tasks) break;
        const int local = task / kChunks, piece = task % kChunks;
        const int col = n0 + piece * 8;
        if (col >= p.N) continue;
        float2 v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = make_float2(0.f, 0.f);
        for (int q = 0; q < parts; ++q) {
          const uint32_t src = smem_base + kRecvOff + static_cast<uint32_t>(q * rows_per + local) * (BN * 4);
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const uint32_t chunk = static_cast<uint32_t>(2 * piece + j) ^ (local & 7);
            float4 f;
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(f.x), "=f"(f.y), "=f"(f.z), "=f"(f.w)
                         : "r"(src + chunk * 16)
                         : "memory");
            v[2 * j].x += f.x;
            v[2 * j].y += f.y;
            v[2 * j + 1].x += f.z;
            v[2 * j + 1].y += f.w;
          }
        }
        const __half2 *c2 = reinterpret_cast<const __half2 *>(&cval[i]);
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float2 x = __fmul2_rn(make_float2(p.alpha, p.alpha), v[j]);
          if (p.c_mode != 0) x = __ffma2_rn(make_float2(p.beta, p.beta), __half22float2(c2[j]), x);
          if (p.act == 1) x = gelu_erf_fast2(x);
          const __half2 h = __floats2half2_rn(x.x, x.y);
          w[j] = *reinterpret_cast<const uint32_t *>(&h);
        }
        const long long row = m0 + row_first + local;
        *reinterpret_cast<uint4 *>(p.D + row * p.N + col) = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, BN);
  }
}

template <int BN, bool B_NK>
bool launch_cluster(const Problem &pb, int parts, cudaStream_t stream) {
  using Cfg = ClusterCfg<BN>;
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  auto kernel = gemm_f16_cluster_kernel<BN, B_NK>;
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    if (!check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes),
                    "cudaFuncSetAttribute(gemm, cluster split-K)"))
      return false;
    attr_set[dev] = true;
  }
  CUtensorMap tmA, tmB;
  if (!make_tensor_map_2d(pb.A, pb.K, pb.M, BK, BM, &tmA)) return false;
  if (B_NK) {
    if (!make_tensor_map_2d(pb.B, pb.K, pb.N, BK, BN, &tmB)) return false;
  } else {
    if (!make_tensor_map_2d(pb.B, pb.N, pb.K, 64, BK, &tmB, pb.ldb)) return false;
  }
  ClusterParams p;
  p.C = pb.C;
  p.D = pb.D;
  p.alpha = pb.alpha;
  p.beta = pb.beta;
  p.c_mode = pb.c_mode;
  p.act = pb.act;
  p.M = static_cast<int>(pb.M);
  p.N = static_cast<int>(pb.N);
  p.num_kb = static_cast<int>((pb.K + BK - 1) / BK);
  p.n_blocks = static_cast<int>((pb.N + BN - 1) / BN);
  p.b_early = pb.b_const ? 1 : 0;
  p.status = device_status_word();
  const int tiles = static_cast<int>((pb.M + BM - 1) / BM) * p.n_blocks;
  const double flops = 2.0 * pb.M * pb.N * pb.K;
  const double bytes = 2.0 * (static_cast<double>(pb.M) * pb.K + static_cast<double>(pb.K) * pb.N +
                              static_cast<double>(pb.M) * pb.N) +
                       (pb.c_mode == 1 ? 2.0 * pb.M * pb.N : pb.c_mode == 2 ? 2.0 * pb.N : 0.0);
  LaunchScope scope(kOpGemm, flops, bytes);
  return check_cuda(launch_pdl(kernel, dim3(tiles * parts), dim3(kClusterThreads), Cfg::kSmemBytes, stream,
                               static_cast<unsigned>(parts), tmA, tmB, p),
                    "gemm kernel launch (cluster split-K)");
}

}  // namespace

bool cluster_supported(const Problem &pb, int parts) {
  return parts >= 2 && parts <= kMaxClusterParts && pb.N % 8 == 0 && parts <= (pb.K + BK - 1) / BK &&
         !has_layernorm_form(pb);
}

// A split that a caller or a tuned entry asks for may have many more tiles than clusters run at
// once.  Every further wave of clusters is a kernel start of its own, while the serial form runs on
// persistent CTAs; its parts of a tile wait for one another, though, which is only short when they
// run in the same round, that is when the number of SMs is a multiple of the factor (2 and 4 of
// 148).  Measured, serial against cluster form in us: with 2 parts 128 tiles (2048 x 1024 x 1024,
// 128 wide) 15.3 / 15.5, 192 tiles (4096 x 768 x 3072, 128 wide) 27.9 / 36.7, 768 tiles
// (4096 x 3072 x 768, 128 wide) 54 / 81; with 4 parts 128 tiles 33.6 / 31.6, 192 tiles 50 / 61, 768
// tiles 117 / 181; but with 3 parts 768 tiles 156 / 130, with 8 parts 714 / 381.  So the line for 2
// and 4 is where the tiles alone fill the chip once.
bool cluster_pays(const Problem &pb, int bn, int parts) {
  const int64_t tiles = ((pb.M + BM - 1) / BM) * ((pb.N + bn - 1) / bn);
  return sm_count() % parts != 0 || tiles <= parts * cluster_capacity(bn, parts);
}

int cluster_capacity(int bn, int parts) {
  // Clusters of more than two CTAs need SMs of one GPC; how many fit depends on which SMs of each
  // GPC the device has.  Asked once per device; the fallback is a 148-SM part (and what a build
  // machine without a GPU answers).
  constexpr int kFallback[kMaxClusterParts + 1] = {0, 148, 74, 45, 33, 24, 18, 16, 14};
  if (parts < 2 || parts > kMaxClusterParts) return 0;
  static std::atomic<int> cache[64][2][kMaxClusterParts + 1] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    cudaGetLastError();
    return kFallback[parts];
  }
  std::atomic<int> &slot = cache[dev][bn == 64 ? 0 : 1][parts];
  int n = slot.load(std::memory_order_relaxed);
  if (n > 0) return n;
  auto query = [&](auto kernel, size_t smem) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = static_cast<unsigned>(parts);
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.gridDim = dim3(parts);
    cfg.blockDim = dim3(kClusterThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int count = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&count, kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return count;
  };
  n = bn == 64 ? query(gemm_f16_cluster_kernel<64, false>, ClusterCfg<64>::kSmemBytes)
               : query(gemm_f16_cluster_kernel<128, false>, ClusterCfg<128>::kSmemBytes);
  if (n <= 0) n = kFallback[parts];
  slot.store(n, std::memory_order_relaxed);
  return n;
}

bool run_cluster(const Problem &pb, int bn, int parts, cudaStream_t stream) {
  if (bn == 64)
    return pb.b_is_nk ? launch_cluster<64, true>(pb, parts, stream) : launch_cluster<64, false>(pb, parts, stream);
  return pb.b_is_nk ? launch_cluster<128, true>(pb, parts, stream) : launch_cluster<128, false>(pb, parts, stream);
}

}  // namespace gemm
}  // namespace hom
