// Packed-QKV padded bidirectional attention for sequences longer than one 128-key tile,
// head_dim 64: a persistent, warp-specialised kernel in which one CTA owns TWO 128-row query
// tiles of one (batch, head) at a time so that the tensor pipe and the softmax arithmetic of
// the two overlap.
//
//   warp 0       TMA producer: the two Q tiles of a work item and a three-stage ring of K / V
//                tiles (128 x 64 fp16 boxes lifted out of the packed [bs*seq, 3*heads*64]
//                tensor into 128-byte-swizzled shared memory);
//   warp 1       issues every tcgen05.mma: S_t = Q_t.K_j^T (128 x 128 x 64) into the tile's S
//                columns of tensor memory and O_t += P_t.V_j (128 x 64 x 128) into its O
//                columns, and hands buffers on with tcgen05.commit;
//   warps 4-7    softmax of tile A, one query row per thread: the 128 scores of a KV step are
//   warps 8-11   softmax of tile B  read from tensor memory once, into registers, and the S
//                columns are given back at once, so that the product of the next KV tile is
//                computed while the exponentials of this one are; P goes back to tensor memory as
//                fp16, two keys per column, and is the A operand of the second MMA from there.
// (Warps 2 and 3 complete the control warpgroup, which gives registers to the softmax ones.)
//
// O accumulates in tensor memory over the KV steps.  The exponentials of a row are taken relative
// to a reference that only follows the row's running maximum when that has grown by more than
// 2^8 (kLazyGrowth): until then P is at most 256 (fp16 keeps its relative precision there, the
// row sum is fp32), and the threads neither rescale O nor wait for the product before.
// (Two query tiles per CTA, the lazily followed maximum and P as a tensor-memory operand are steps
// of the published FlashAttention-4 algorithm.)
//
// What bounds it: the exponentials.  ex2 runs on the special-function unit at 16 per clock and
// SM, 2,048 clk for one KV step of both tiles.  (Evaluating one, two or three pairs of eight by a
// polynomial on the FMA pipes instead gave 112.9 / 115.6 / 121.4 us against 113.9 on the case
// below: the issue slots are the next limit.)
// A step of both tiles takes 3,300 clk: 800-1,000 until the scores are in registers and their
// maximum is known, 2,100-2,200 for the exponentials, the rest waits; an item's output adds 1,500.
// Starting one tile half a step late does not last: the tiles fall back into step at the next item.
// Measured, 16 heads, lengths U{256..512}, 64 x 512: 155 -> 114 us (one query row per thread
// reading S twice, P through shared memory, O folded into registers at every step); 6 x 384,
// lengths U{150..384}: 18.5 -> 10.7 us.
//
// Work items are (pair of query tiles, batch, head), the pair being the slowest index: the
// second pair of a ragged sequence has less or nothing to do, and the shorter items come last.  A
// CTA walks items blockIdx.x, blockIdx.x + gridDim.x, ... and the K / V ring runs across item
// boundaries, so the loads of the next item overlap the arithmetic of the current one.  KV tiles
// beyond a sequence's valid length are skipped, the ragged tile is masked, query tiles that are
// all padding are not computed, and padded query rows are written as zeros.
//
// Same contract as the reference's cuDNN fused attention behind TransformerEngine
// (include/NVGPUKernels/BertAttentionRunner.h:52-136: layout BS3HD, no bias, padding mask,
// no dropout, inference).
#include <atomic>
#include <cstdio>
#include <cstdlib>

#include "attention_sm100.cuh"
#include "gemm_sm100.cuh"
#include "hom_diag.cuh"
#include "ptx_sm100.cuh"

namespace hom {
namespace attention {

using namespace hom::ptx;

namespace {

constexpr int kTile = 128;
constexpr int kHeadDim = 64;
constexpr uint32_t kTileBytes = kTile * kHeadDim * 2;  // 16 KB
constexpr int kThreadsPP = 384;                        // control warpgroup, softmax of tile A, of tile B
constexpr int kKvStages = 3;

// shared-memory map (offsets from the 1024-byte aligned base)
constexpr uint32_t kOffQ = 0;                                   // 2 tiles x 2 buffers (item i, item i + 1)
constexpr uint32_t kOffK = kOffQ + 4 * kTileBytes;              // kKvStages tiles
constexpr uint32_t kOffV = kOffK + kKvStages * kTileBytes;      // kKvStages tiles
constexpr uint32_t kOffO = kOffV + kKvStages * kTileBytes;      // output staging, 2 tiles
constexpr uint32_t kOffBar = kOffO + 2 * kTileBytes;
constexpr uint32_t kSmemBytesPP = kOffBar + 256 + 1024;
// Tensor memory, columns: S_A, S_B 128 each; O_A, O_B 64 each; P_A, P_B 64 each.
constexpr uint32_t kTmemO = 2 * kTile, kTmemP = kTmemO + 2 * kHeadDim;
constexpr uint32_t kTmemColsPP = 512;

constexpr float kLazyGrowth = 8.0f;

// Registers per thread after the hand-over between the warpgroups.  The shares of the three must not
// add up to more than what the launch gave them, or the increase would wait for good.  How many a
// thread of the launch has is the compiler's choice, at most 65,536 / 384 rounded down to a multiple
// of 8 (168), so pingpong_available() looks at the compiled count before the kernel is ever run.
constexpr int kControlRegs = 72, kSoftmaxRegs = 216;
constexpr bool hand_over_fits(int launch_regs) { return kControlRegs + 2 * kSoftmaxRegs <= 3 * launch_regs; }
static_assert(hand_over_fits(168) && !hand_over_fits(160), "the shares use all that a launch can have");

struct ParamsPP {
  const int *cu_seqlens;
  __half *out;
  int seq, heads, bs;
  int tiles_per_item;  // 2, or 1 when that still leaves every CTA at most one item
  int num_items;       // query-tile groups * bs * heads
  int step_batch, step_head;  // the grid size as (batch, head) steps
  float scale_log2;
  int *status;
  HOM_DIAG(long long *prof;)  // phase cycle counters of CTA 0 (HOM_ATTN_PROFILE), else null
};

__device__ __forceinline__ float ex2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float y;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}

// The items of a CTA in order: (group of query tiles, batch, head), head fastest.  Stepping by the
// grid size is an addition with carries (an index division costs a hundred clocks, and an item's
// start is on the critical path of both tiles).
struct Walk {
  int item, group, batch, head;
};
__device__ __forceinline__ Walk walk_begin(const ParamsPP &p) {
  Walk w;
  w.item = blockIdx.x;
  w.head = w.item % p.heads;
  const int rest = w.item / p.heads;
  w.batch = rest % p.bs;
  w.group = rest / p.bs;
  return w;
}
__device__ __forceinline__ void walk_next(const ParamsPP &p, Walk &w) {
  w.item += gridDim.x;
  w.head += p.step_head;
  w.batch += p.step_batch;
  if (w.head >= p.heads) {
    w.head -= p.heads;
    ++w.batch;
  }
  while (w.batch >= p.bs) {
    w.batch -= p.bs;
    ++w.group;
  }
}

// What every role derives from an item.
struct Item {
  int batch, head, q0;  // q0: first query row of tile A
  int len, n_kv;        // valid length, KV tiles that hold valid keys
  bool act[2];          // tile t has at least one valid query row
};

__device__ __forceinline__ Item make_item(const ParamsPP &p, const Walk &w, int start, int end) {
  Item it;
  it.batch = w.batch;
  it.head = w.head;
  it.q0 = w.group * p.tiles_per_item * kTile;
  it.len = max(0, min(end - start, p.seq));
  it.n_kv = (it.len + kTile - 1) / kTile;
  it.act[0] = it.q0 < it.len;
  it.act[1] = p.tiles_per_item == 2 && it.q0 + kTile < it.len;
  return it;
}
__device__ __forceinline__ Item decode_item(const ParamsPP &p, const Walk &w) {
  return make_item(p, w, p.cu_seqlens[w.batch], p.cu_seqlens[w.batch + 1]);
}

__global__ void __launch_bounds__(kThreadsPP, 1)
attention_f16_pingpong_kernel(const __grid_constant__ CUtensorMap tmQKV, const __grid_constant__ CUtensorMap tmOut,
                              const ParamsPP p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t smem_base = (raw_addr + 1023u) & ~1023u;
  uint8_t *smem_gen = smem_raw + (smem_base - raw_addr);

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;

  // barriers, 8 bytes each
  const uint32_t bar0 = smem_base + kOffBar;
  auto q_full = [&](int t, int b) { return bar0 + 8u * (2 * t + b); };        // Q_t buffer b loaded
  auto q_empty = [&](int t, int b) { return bar0 + 8u * (4 + 2 * t + b); };   // ... and consumed
  auto k_full = [&](int s) { return bar0 + 8u * (8 + s); };
  auto k_empty = [&](int s) { return bar0 + 8u * (8 + kKvStages + s); };
  auto v_full = [&](int s) { return bar0 + 8u * (8 + 2 * kKvStages + s); };
  auto v_empty = [&](int s) { return bar0 + 8u * (8 + 3 * kKvStages + s); };
  constexpr int kBarTile = 8 + 4 * kKvStages;
  auto s_full = [&](int t) { return bar0 + 8u * (kBarTile + t); };       // S_t computed
  auto s_empty = [&](int t) { return bar0 + 8u * (kBarTile + 2 + t); };  // ... and read into registers
  auto p_full = [&](int t) { return bar0 + 8u * (kBarTile + 4 + t); };   // P_t written (and O_t ready to be added to)
  auto o_full = [&](int t) { return bar0 + 8u * (kBarTile + 6 + t); };   // P_t.V of the step added to O_t
  volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(smem_gen + kOffBar + 8 * (kBarTile + 8));
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

  if (tid == 64) {
    prefetch_tensormap(&tmQKV);
    prefetch_tensormap(&tmOut);
  }
  if (tid == 0) {
    for (int i = 0; i < kKvStages; ++i) {
      mbar_init(k_full(i), 1);
      mbar_init(k_empty(i), 1);
      mbar_init(v_full(i), 1);
      mbar_init(v_empty(i), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(s_full(i), 1);
      mbar_init(s_empty(i), kTile);  // every softmax thread of the tile arrives
      mbar_init(p_full(i), kTile);
      mbar_init(o_full(i), 1);
      for (int b = 0; b < 2; ++b) {
        mbar_init(q_full(i, b), 1);
        mbar_init(q_empty(i, b), 1);
      }
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t *>(tmem_slot)), kTmemColsPP);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  // Dependents may be scheduled only now that this CTA holds its tensor memory.
  pdl_launch_dependents();
  pdl_wait();  // cu_seqlens and the packed QKV come from earlier kernels of the stream

  const int hidden = p.heads * kHeadDim;

  if (warp < 4) {
    reg_dealloc<kControlRegs>();
    if (warp == 0) {
      // ------------------------------------------------------------ TMA producer
      // One elected lane runs the whole loop: see the MMA issuer.
      if (elect_one()) {
        uint32_t q_uses[2] = {0, 0};  // completed loads into each Q buffer
        uint32_t kv_uses = 0;         // K / V tiles loaded so far (stage = kv_uses % kKvStages)
        bool ok = true;
        for (Walk w = walk_begin(p); w.item < p.num_items && ok; walk_next(p, w)) {
          const Item it = decode_item(p, w);
          if (!it.act[0]) continue;  // tile B cannot be active without tile A
          const int row_base = it.batch * p.seq;
          for (int t = 0; t < 2 && ok; ++t) {
            if (!it.act[t]) continue;
            // the buffer is free once every S MMA of the item that used it last has completed
            const int b = q_uses[t] & 1u;
            ok = mbar_wait(q_empty(t, b), ((q_uses[t] >> 1) & 1u) ^ 1u, abort_flag, p.status, kDevWaitTimeoutAttention);
            if (!ok) break;
            mbar_arrive_expect_tx(q_full(t, b), kTileBytes);
            tma_load_2d(smem_base + kOffQ + (2 * t + b) * kTileBytes, &tmQKV, q_full(t, b), it.head * kHeadDim,
                        row_base + it.q0 + t * kTile);
            ++q_uses[t];
          }
          for (int j = 0; j < it.n_kv && ok; ++j) {
            const int s = kv_uses % kKvStages;
            const uint32_t ph = (kv_uses / kKvStages) & 1u;
            ok = mbar_wait(k_empty(s), ph ^ 1u, abort_flag, p.status, kDevWaitTimeoutAttention);
            if (!ok) break;
            mbar_arrive_expect_tx(k_full(s), kTileBytes);
            tma_load_2d(smem_base + kOffK + s * kTileBytes, &tmQKV, k_full(s), hidden + it.head * kHeadDim,
                        row_base + j * kTile);
            ok = mbar_wait(v_empty(s), ph ^ 1u, abort_flag, p.status, kDevWaitTimeoutAttention);
            if (!ok) break;
            mbar_arrive_expect_tx(v_full(s), kTileBytes);
            tma_load_2d(smem_base + kOffV + s * kTileBytes, &tmQKV, v_full(s), 2 * hidden + it.head * kHeadDim,
                        row_base + j * kTile);
            ++kv_uses;
          }
        }
        if (!ok) {
          // Give copies already in flight time to land before shared memory is released.
          const long long t0 = clock64();
          while (clock64() - t0 < 4000000LL) {
          }
        }
      }
      __syncwarp();
    } else if (warp == 1) {
      // ------------------------------------------------------------- MMA issuer
      // One lane, elected once around the whole loop, so that an MMA costs an issue slot and not a
      // vote, a re-election and a reconvergence of the warp (about 100 clk each).
      if (elect_one()) {
        constexpr uint32_t idesc_s = make_idesc_f16(kTile, kTile, false, false);
        constexpr uint32_t idesc_o = make_idesc_f16(kTile, kHeadDim, false, true);
        bool ok = true;
        auto wait = [&](uint32_t bar, uint32_t parity) {
          ok = mbar_wait(bar, parity, abort_flag, p.status, kDevWaitTimeoutAttention);
          tc_fence_after_sync();
          return ok;
        };
        // Two cursors walk the (item, KV tile) steps of this CTA: S is issued one step ahead of P.V,
        // across item boundaries, so that neither an item's first S nor its last P.V is waited for
        // with the other tile's threads idle.
        struct Cursor {
          Walk w;
          int j;
          Item it;
        };
        auto settle = [&](Cursor &c) {  // skip items without a valid key
          for (; c.w.item < p.num_items; walk_next(p, c.w)) {
            c.it = decode_item(p, c.w);
            if (c.it.act[0]) return;
          }
        };
        auto advance = [&](Cursor &c) {
          if (++c.j < c.it.n_kv) return;
          c.j = 0;
          walk_next(p, c.w);
          settle(c);
        };
        uint32_t q_uses[2] = {0, 0}, s_uses[2] = {0, 0}, p_uses[2] = {0, 0};
        uint32_t k_stage = 0, k_ph = 0, v_stage = 0, v_ph = 0;
        auto issue_s = [&](Cursor &c) {
          if (!wait(k_full(k_stage), k_ph)) return;
          const uint64_t db = make_smem_desc_sw128(smem_base + kOffK + k_stage * kTileBytes, 16, 1024);
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            if (!c.it.act[t]) break;
            const uint32_t qb = q_uses[t] & 1u;
            if (c.j == 0 && !wait(q_full(t, qb), (q_uses[t] >> 1) & 1u)) return;
            // the threads have read the S_t before this one
            if (!wait(s_empty(t), (s_uses[t] & 1u) ^ 1u)) return;
            ++s_uses[t];
            const uint64_t da = make_smem_desc_sw128(smem_base + kOffQ + (2 * t + qb) * kTileBytes, 16, 1024);
#pragma unroll
            for (int k = 0; k < kHeadDim / 16; ++k)
              tc_mma_f16_ss(tmem_base + t * kTile, smem_desc_advance(da, k * 32), smem_desc_advance(db, k * 32),
                            idesc_s, k != 0 ? 1u : 0u);
            tc_commit(s_full(t));
            if (c.j + 1 == c.it.n_kv) {  // the item's last S: its Q buffer is free once that completes
              tc_commit(q_empty(t, qb));
              ++q_uses[t];
            }
          }
          tc_commit(k_empty(k_stage));
          if (++k_stage == kKvStages) {
            k_stage = 0;
            k_ph ^= 1u;
          }
          advance(c);
        };
        auto issue_pv = [&](Cursor &c) {
          const int valid = min(kTile, c.it.len - c.j * kTile);
          const int k_steps = (valid + 15) >> 4;  // key groups that hold a valid key
          if (!wait(v_full(v_stage), v_ph)) return;
          // V tile: 128 kv rows of 128 B; N (= d) contiguous, 16 kv rows = 2048 B.
          const uint64_t db = make_smem_desc_sw128(smem_base + kOffV + v_stage * kTileBytes, kTileBytes, 1024);
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            if (!c.it.act[t]) break;
            // P_t of this step is in tensor memory, O_t holds the steps before it
            if (!wait(p_full(t), p_uses[t] & 1u)) return;
            ++p_uses[t];
            const uint32_t o_tmem = tmem_base + kTmemO + t * kHeadDim, p_tmem = tmem_base + kTmemP + t * kHeadDim;
            if (k_steps == kTile / 16) {
#pragma unroll
              for (int k = 0; k < kTile / 16; ++k)  // 16 keys of P = 8 columns
                tc_mma_f16_ts(o_tmem, p_tmem + k * 8, smem_desc_advance(db, k * 2048), idesc_o,
                              (c.j | k) != 0 ? 1u : 0u);
            } else {
              for (int k = 0; k < k_steps; ++k)
                tc_mma_f16_ts(o_tmem, p_tmem + k * 8, smem_desc_advance(db, k * 2048), idesc_o,
                              (c.j | k) != 0 ? 1u : 0u);
            }
            tc_commit(o_full(t));
          }
          tc_commit(v_empty(v_stage));
          if (++v_stage == kKvStages) {
            v_stage = 0;
            v_ph ^= 1u;
          }
          advance(c);
        };
        Cursor ahead{walk_begin(p), 0, {}};
        settle(ahead);
        Cursor cur = ahead;
        if (ahead.w.item < p.num_items) issue_s(ahead);
        while (ok && cur.w.item < p.num_items) {
          if (ahead.w.item < p.num_items) issue_s(ahead);
          if (ok) issue_pv(cur);
        }
      }
      __syncwarp();
    }
  } else {
    // ------------------------------------------------ softmax, one query row per thread
    reg_alloc<kSoftmaxRegs>();
    const int t = (warp - 4) >> 2;             // which query tile of the pair
    const int quarter = warp & 3;              // the warp's tensor-memory lane quarter
    const int row = quarter * 32 + lane;       // row of the tile
    const uint32_t lane_sel = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t tmem_s = tmem_base + t * kTile + lane_sel;
    const uint32_t tmem_o = tmem_base + kTmemO + t * kHeadDim + lane_sel;
    const uint32_t tmem_p = tmem_base + kTmemP + t * kHeadDim + lane_sel;
    const uint32_t o_stage = smem_base + kOffO + t * kTileBytes + quarter * 32 * 128;  // this warp's 32 rows
    const float2 scale2 = make_float2(p.scale_log2, p.scale_log2);
    uint32_t steps = 0;  // KV steps of this tile so far: phase of s_full, and of o_full one behind
    bool ok = true;
    HOM_DIAG(long long c_wait_s = 0, c_max = 0, c_exp = 0, c_wait_o = 0, c_store = 0, c_steps = 0;
             const long long c_begin = clock64(); long long c_t = 0;)
    auto wait = [&](uint32_t bar, uint32_t parity) {
      ok = mbar_wait(bar, parity, abort_flag, p.status, kDevWaitTimeoutAttention);
      ok = __all_sync(0xffffffffu, ok);
      tc_fence_after_sync();
      return ok;
    };
    // The finished tile of an item is written out during the first step of the next one, when its
    // last product has had that step's scores to complete.
    bool pending = false;
    int out_batch = 0, out_head = 0, out_row = 0;
    float out_scale = 0.f;
    // ---- O / l as fp16, staged in this warp's 32 rows of the tile's buffer, written by TMA (which
    // clips rows beyond the sequence)
    auto write_out = [&]() {
      HOM_DIAG(const long long t_out = clock64();)
      if (!wait(o_full(t), (steps & 1u) ^ 1u)) return false;
      // the item before handed its tile to TMA from these rows
      if (lane == 0) bulk_wait_group_read_0();
      __syncwarp();
      const float2 inv2 = make_float2(out_scale, out_scale);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t o[32];
        tmem_ld_32x32(tmem_o + c * 32, o);
        tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint32_t w[4] = {0u, 0u, 0u, 0u};
          if (out_scale != 0.f) {  // 0: a padded row
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
              const int i0 = g * 8 + 2 * jj;
              const float2 v = __fmul2_rn(make_float2(__uint_as_float(o[i0]), __uint_as_float(o[i0 + 1])), inv2);
              const __half2 h = __floats2half2_rn(v.x, v.y);
              w[jj] = *reinterpret_cast<const uint32_t *>(&h);
            }
          }
          const uint32_t chunk = static_cast<uint32_t>(c * 4 + g) ^ (lane & 7);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(o_stage + lane * 128 + (chunk << 4)),
                       "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3])
                       : "memory");
        }
      }
      fence_proxy_async_smem();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        if (out_row < p.seq) tma_store_3d(&tmOut, o_stage, out_head * kHeadDim, out_row, out_batch);
        bulk_commit_group();
      }
      pending = false;
      HOM_DIAG(c_store += clock64() - t_out;)
      return true;
    };
    // The lengths of the next item are requested while the current one is worked on.
    Walk w = walk_begin(p);
    int next_start = 0, next_end = 0;
    if (w.item < p.num_items) {
      next_start = p.cu_seqlens[w.batch];
      next_end = p.cu_seqlens[w.batch + 1];
    }
    while (w.item < p.num_items && ok) {
      const Item it = make_item(p, w, next_start, next_end);
      walk_next(p, w);
      if (w.item < p.num_items) {
        next_start = p.cu_seqlens[w.batch];
        next_end = p.cu_seqlens[w.batch + 1];
      }
      if (!it.act[t]) {
        // the whole query tile is padding (or beyond the sequence): zeros
        const int q_idx = it.q0 + t * kTile + row;
        if (q_idx < p.seq && t < p.tiles_per_item) {
          uint4 *out_row = reinterpret_cast<uint4 *>(
              p.out + (static_cast<long long>(it.batch) * p.seq + q_idx) * hidden + it.head * kHeadDim);
#pragma unroll
          for (int g = 0; g < 8; ++g) out_row[g] = make_uint4(0, 0, 0, 0);
        }
        continue;
      }
      float m_ref = -INFINITY;  // what the exponentials of this row are relative to
      float l_run = 0.f;
      for (int j = 0; j < it.n_kv && ok; ++j) {
        const int valid = min(kTile, it.len - j * kTile);  // columns [0, valid) are real keys
        HOM_DIAG(c_t = clock64();)
        if (!wait(s_full(t), steps & 1u)) break;
        HOM_DIAG(c_wait_s += clock64() - c_t; c_t = clock64(); ++c_steps;)
        uint32_t r[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_32x32(tmem_s + c * 32, r[c]);
        tmem_ld_wait();
        tc_fence_before_sync();
        mbar_arrive(s_empty(t));
        if (valid < kTile) {  // the last KV tile: keys beyond the sequence drop out of maximum and sum
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (c * 32 + i >= valid) r[c][i] = 0xff800000u;
        }
        float m4[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          m4[c] = fmaxf(__uint_as_float(r[c][0]), __uint_as_float(r[c][1]));
#pragma unroll
          for (int i = 2; i < 32; i += 2)
            m4[c] = max3(m4[c], __uint_as_float(r[c][i]), __uint_as_float(r[c][i + 1]));
        }
        // scale > 0, so the maximum of the scaled scores is the scaled maximum
        const float m_tile = max3(fmaxf(m4[0], m4[1]), m4[2], m4[3]) * p.scale_log2;
        HOM_DIAG(c_max += clock64() - c_t; c_t = clock64();)
        if (j == 0) {
          m_ref = m_tile;
          if (pending && !write_out()) break;
        } else {
          // The product of the step before has been added to O_t and has read P_t: it was queued one
          // step ago, so this wait is normally over.
          if (!wait(o_full(t), (steps & 1u) ^ 1u)) break;
          HOM_DIAG(c_wait_o += clock64() - c_t; c_t = clock64();)
          const bool grown = m_tile - m_ref > kLazyGrowth;
          if (__any_sync(0xffffffffu, grown)) {
            // tcgen05.ld / st are warp-collective: rows that keep their reference multiply by one
            const float m_new = grown ? m_tile : m_ref;
            const float corr = grown ? ex2_fast(m_ref - m_new) : 1.f;
            const float2 corr2 = make_float2(corr, corr);
            l_run *= corr;
            m_ref = m_new;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              uint32_t o[32];
              tmem_ld_32x32(tmem_o + c * 32, o);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; i += 2) {
                const float2 v = __fmul2_rn(make_float2(__uint_as_float(o[i]), __uint_as_float(o[i + 1])), corr2);
                o[i] = __float_as_uint(v.x);
                o[i + 1] = __float_as_uint(v.y);
              }
              tmem_st_32x32(tmem_o + c * 32, o);
            }
          }
        }
        // ---- P = exp2(scale * S - m_ref) as fp16 into tensor memory, row sum in fp32
        float2 l2a = make_float2(0.f, 0.f), l2b = make_float2(0.f, 0.f);
        const float2 neg_m2 = make_float2(-m_ref, -m_ref);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          // Chunks that lie entirely beyond the valid keys are never read by the second MMA (it stops
          // at the last 16-key group that holds a valid key).
          if (c * 32 < valid) {
            uint32_t w[16];
#pragma unroll
            for (int jj = 0; jj < 16; ++jj) {
              const float2 x = __ffma2_rn(make_float2(__uint_as_float(r[c][2 * jj]), __uint_as_float(r[c][2 * jj + 1])),
                                          scale2, neg_m2);
              const float2 e = make_float2(ex2_fast(x.x), ex2_fast(x.y));
              if (jj & 1) l2a = __fadd2_rn(l2a, e);
              else l2b = __fadd2_rn(l2b, e);
              const __half2 h = __floats2half2_rn(e.x, e.y);
              w[jj] = *reinterpret_cast<const uint32_t *>(&h);
            }
            tmem_st_32x16(tmem_p + c * 16, w);
          }
        }
        l_run += (l2a.x + l2b.x) + (l2a.y + l2b.y);
        // P is complete: hand it (and O_t, possibly rescaled) to the MMA warp
        tmem_st_wait();
        tc_fence_before_sync();
        mbar_arrive(p_full(t));
        ++steps;
        HOM_DIAG(c_exp += clock64() - c_t;)
      }
      if (!ok) break;
      pending = true;
      out_batch = it.batch;
      out_head = it.head;
      out_row = it.q0 + t * kTile + quarter * 32;
      out_scale = out_row + lane < it.len && l_run > 0.f ? 1.f / l_run : 0.f;
    }
    if (ok && pending) write_out();
    // A store still in flight reads this warp's staging rows: let it finish reading.
    if (lane == 0) bulk_wait_group_read_0();
    __syncwarp();
    HOM_DIAG(if (p.prof && blockIdx.x == 0 && lane == 0 && (warp == 4 || warp == 8)) {
      long long *o = p.prof + (warp == 4 ? 0 : 8);
      o[0] = clock64() - c_begin; o[1] = c_wait_s; o[2] = c_max; o[3] = c_exp; o[4] = c_wait_o; o[5] = 0;
      o[6] = c_store; o[7] = c_steps;
    })
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemColsPP);
  }
}

}  // namespace

bool pingpong_available() {
  static std::atomic<int> launch_regs[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  int regs = launch_regs[dev].load(std::memory_order_relaxed);
  if (regs == 0) {
    cudaFuncAttributes fa;
    if (!check_cuda(cudaFuncGetAttributes(&fa, attention_f16_pingpong_kernel), "cudaFuncGetAttributes(attention)"))
      return false;
    regs = fa.numRegs;
    launch_regs[dev].store(regs, std::memory_order_relaxed);
  }
  return hand_over_fits(regs);
}

bool run_pingpong(const Problem &pb, cudaStream_t stream) {
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    if (!check_cuda(cudaFuncSetAttribute(attention_f16_pingpong_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytesPP),
                    "cudaFuncSetAttribute(attention, two query tiles per CTA)"))
      return false;
    attr_set[dev] = true;
  }
  CUtensorMap tm;
  const uint64_t rows = static_cast<uint64_t>(pb.bs) * pb.seq;
  const uint64_t cols = 3ull * pb.heads * kHeadDim;
  if (!gemm::make_tensor_map_2d(pb.qkv, cols, rows, kHeadDim, kTile, &tm)) return false;
  CUtensorMap tm_out;  // a warp stores its 32 query rows
  if (!make_out_map(pb.out, pb.heads * kHeadDim, pb.seq, pb.bs, 32, &tm_out)) return false;
  ParamsPP p;
  p.cu_seqlens = pb.cu_seqlens;
  p.out = pb.out;
  p.seq = static_cast<int>(pb.seq);
  p.heads = static_cast<int>(pb.heads);
  p.bs = static_cast<int>(pb.bs);
  // Two query tiles per item hide each other's waits; with so few of them that every tile can have
  // a CTA to itself, the shorter chain of one tile wins.
  const int64_t q_tiles = (pb.seq + kTile - 1) / kTile;
  p.tiles_per_item = pb.bs * pb.heads * q_tiles <= sm_count() ? 1 : 2;
  const int64_t items = pb.bs * pb.heads * ((q_tiles + p.tiles_per_item - 1) / p.tiles_per_item);
  if (items > INT32_MAX) {
    set_error(HOM_ERR_UNSUPPORTED, "attention: too many (batch, head, query tile) work items");
    return false;
  }
  p.num_items = static_cast<int>(items);
  const int grid = p.num_items < sm_count() ? p.num_items : sm_count();
  p.step_batch = grid / p.heads;
  p.step_head = grid % p.heads;
  p.scale_log2 = pb.scale * 1.44269504088896340736f;
  p.status = device_status_word();
  HOM_DIAG(p.prof = std::getenv("HOM_ATTN_PROFILE") ? gemm::profile_buffer() : nullptr;)
  const double d = kHeadDim;
  const double flops = 4.0 * d * pb.heads * pb.bs * static_cast<double>(pb.seq) * pb.seq;
  const double bytes = 2.0 * rows * cols + 2.0 * rows * pb.heads * d + 4.0 * (pb.bs + 1);
  LaunchScope scope(kOpAttention, flops, bytes);
  const bool launched = check_cuda(launch_pdl(attention_f16_pingpong_kernel, dim3(grid), dim3(kThreadsPP),
                                              kSmemBytesPP, stream, 1, tm, tm_out, p),
                                   "attention kernel launch");
#if HOM_DIAG_ENABLED
  if (p.prof) {
    long long h[16];
    cudaStreamSynchronize(stream);
    cudaMemcpy(h, p.prof, sizeof(h), cudaMemcpyDeviceToHost);
    for (int w = 0; w < 2; ++w)
      fprintf(stderr,
              "[hom] attention CTA 0 tile %c: total %lld | wait S %lld | read + max %lld | exp %lld | wait O %lld | "
              "- %lld | store %lld cycles over %lld steps\n",
              w ? 'B' : 'A', h[8 * w], h[8 * w + 1], h[8 * w + 2], h[8 * w + 3], h[8 * w + 4], h[8 * w + 5],
              h[8 * w + 6], h[8 * w + 7]);
  }
#endif
  return launched;
}

}  // namespace attention
}  // namespace hom
