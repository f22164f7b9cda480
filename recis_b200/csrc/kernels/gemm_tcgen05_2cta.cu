// bf16 GEMM on pairs of SMs (tcgen05 cta_group::2): D[MM, NN] = act( A[MM, KK] * B[NN, KK]^T + bias + residual ).
//
// Two CTAs of a cluster, on the two SMs of one pair, compute one 256 x 256 tile of D together. Each CTA stages ITS half of the
// operands - 128 rows of A and 128 rows of B per 64-wide reduction step, 32 KB - with plain TMA loads of its own, and keeps its
// 128 rows of the fp32 accumulator (256 columns) in its own tensor memory; one thread of the leader CTA (cluster rank 0) issues
// tcgen05.mma.cta_group::2 for both, the hardware reading each CTA's A half from that CTA's shared memory and sharing the two
// B halves between the pair. A 128 x 128 tile per SM (the one-CTA kernel in gemm_tcgen05.cu) needs 256 bytes of shared-memory
// traffic per clock at full tensor rate - operand reads plus the TMA fill of the next stage - against the 128 an SM has; the
// pair needs half of that per SM for the same math, which is what lifts the ceiling of the one-CTA kernel.
//
// The grid is persistent, one pair per two SMs: the accumulator is double buffered in tensor memory, so a tile's epilogue and stores run
// under the loads and MMAs of the next tile.
//
// Protocol per reduction step (ring of stages, counted over all tiles; the barriers live at the same shared-memory offsets in both CTAs):
//   * both producers (warp 0) wait for their own empty[s]; the leader arms ITS full[s] with the bytes of both CTAs;
//     both issue their loads with the leader's full[s] as the completion barrier (no load is multicast);
//   * the leader's MMA warp (warp 1) waits for full[s], issues four 256 x 256 x 16 MMAs and commits them to empty[s] of
//     both CTAs (tcgen05.commit with a two-CTA mask), and after a tile's last step to accumulator_full of both CTAs;
//   * the epilogue warps (2..9) of each CTA drain their own accumulator, two warps per lane quarter with 128 columns each, box by box
//     (32 rows x 128 bytes): tcgen05.ld, bias / residual / ReLU / mask, conversion, staging in the 128-byte swizzle, TMA store
//     (add-reduction for a split reduction). A warp has its own staging slot, or with a residual or mask a ring of three, into which its boxes
//     travel two boxes ahead. Each warp reports to the leader's accumulator_empty when it has read its part.
//
// Every wait is bounded: on a timeout the CTA records kStatusWaitTimeout, gives outstanding copies time to land, joins the cluster
// barrier, frees its tensor memory and returns.
//
// Operands may be K-major or MN-major as in the one-CTA kernel.
//
// Measured on a B200 (L2 cold; before: one tile per CTA, two CTAs to an SM, a row per lane and conditions per element in the epilogue):
//   269000 x 1024 x 256, bias + ReLU, bf16 out:   325 -> 141 us (its 551 MB of output alone take 145 us to fill)
//   the same with mask and column sums:           510 -> 246 us (1.24 GB: 5.0 TB/s)
//   269000 x 256 x 1024, fp32 residual in / out:  343 -> 186 us (1.1 GB: 5.9 TB/s)
//   16384 x 2048 x 3200, bias + ReLU:             174 -> 131 us (1.64 PFLOP/s; the tensor pipe is busy 95 % of the cycles)
//   dW 2048 x 3200 of 16384 rows:                 178 -> 186 us (104 tiles of the whole reduction are two rounds however they are dealt)
// Tiles are dealt out before the start. Where a kernel of another stream holds SMs, as the exchange of a step on several GPUs may, a pair that
// starts late still has its whole share; what that costs has not been measured.
// What bounded the short reductions was the epilogue: first its instructions (finish_box), then the arrival on the leader's
// accumulator_empty, which with release semantics at cluster scope waited for the warp's stores (206 -> 141 us in the first case).
//
// The reference has no GEMM kernel of its own: its dense layers are nn.Linear (cuBLAS), examples/deepfm/deepfm_model.py:49-52.
#include "../common/rb_common.cuh"
#include "../common/rb_launch.h"
#include "../common/rb_tcgen05.cuh"
#include "rb_dense.h"
#include "rb_gemm_store.cuh"
#include <cuda.h>
#include <cuda_bf16.h>
#include <algorithm>
#include <cstdlib>

namespace {

using namespace rb::tc;
using rb::gemm::Store;

constexpr int TM = 128;        // rows of D per CTA (the pair covers 256)
constexpr int TN = 256;        // columns of D per pair; each CTA stages 128 rows of B
constexpr int BK = 64;
constexpr int UK = 16;
constexpr int kPairs = 74;      // pairs of SMs
constexpr int kThreads = 320;     // producer warp, MMA warp, 8 epilogue warps (two per tensor-memory lane quarter)
constexpr uint32_t kHalfBytes = 128 * BK * 2;                   // 16 KB: one operand half of one stage
constexpr uint32_t kStageBytes = 2 * kHalfBytes;                // this CTA's A half + B half
constexpr int kGroup = 8;                                       // column tiles per group of the walk
// Shared memory per CTA: a ring of operand stages and, for each of the eight epilogue warps, 4 KB staging slots. A second input of the
// epilogue needs three slots, so that its boxes can travel two boxes ahead; then two stages less fit. (Without one, two slots and five
// stages: 54.3 instead of 47.1 us at 8192 x 1024 x 3200, and nothing gained where the epilogue is what takes the time.)
template <bool kSrc> struct Ring {
  static constexpr int kStages = kSrc ? 4 : 6, kSlots = kSrc ? 3 : 1;
  static constexpr uint32_t kBytes = kStages * kStageBytes + 8 * kSlots * 4096 + 1024;
};
constexpr uint32_t kPeerMask = 0xFEFFFFFFu;                     // clears the CTA-rank bit of a shared::cluster address: rank 0's copy

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// TMA load into this CTA's shared memory that reports its bytes to the barrier at `bar_cluster_addr` (the leader's full barrier)
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, int x, int y, uint32_t bar_cluster_addr) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(x), "r"(y), "r"(bar_cluster_addr) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// completion of all MMAs issued so far arrives once on the barrier at this offset in both CTAs of the pair
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}

// one arrival on the barrier at this offset in the leader CTA (it hands back tensor memory that was only read: nothing to make visible)
__device__ __forceinline__ void arrive_leader(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(smem_u32(bar) & kPeerMask) : "memory");
}

// Tile t of the walk: this CTA's rows, the pair's columns, and its share of the reduction (may be empty when the reduction is split).
// Tiles are walked in groups of kGroup column tiles, columns fastest: the pairs at work read the same rows of A at the same time and the
// group's rows of B stay in L2. (Rows fastest, A came from DRAM once per column tile: 1055 instead of 690 MB at 269000 x 1024 x 256.)
struct PairTile {
  int m0, n0, kb_begin, num_kb;
  bool first_split;
  __device__ __forceinline__ PairTile(int t, int mt, int nt, int splits, int total_kb, uint32_t rank) {
    const int z = t / (mt * nt), tile = t - z * mt * nt;
    const int group = tile / (kGroup * mt), in_group = tile - group * kGroup * mt, width = min(kGroup, nt - group * kGroup);
    const int kb_per = (total_kb + splits - 1) / splits;
    m0 = in_group / width * 2 * TM + (int)rank * TM;
    n0 = (group * kGroup + in_group % width) * TN;
    kb_begin = z * kb_per;
    num_kb = max(0, min(total_kb, kb_begin + kb_per) - kb_begin);
    first_split = z == 0;
  }
};

template <bool A_MN, bool B_MN, bool kSrc, typename OutT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_bf16_tcgen05_2cta_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                              const __grid_constant__ CUtensorMap map_o, const __grid_constant__ CUtensorMap map_src,
                              const float* __restrict__ bias, float* __restrict__ colsum, int MM, int NN, int KK, int relu, int splits,
                              int reduce_out, int64_t* __restrict__ status) {
  constexpr int kStages = Ring<kSrc>::kStages, kSlots = Ring<kSrc>::kSlots;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kStages];
  __shared__ __align__(8) uint64_t empty_bar[kStages];
  __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2];
  __shared__ __align__(8) uint64_t src_bar[8 * kSlots];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();                        // 0 = leader
  const int mt = (MM + 2 * TM - 1) / (2 * TM), nt = (NN + TN - 1) / TN;
  const int total_kb = (KK + BK - 1) / BK;
  const int n_tiles = mt * nt * splits, first = (int)(blockIdx.x >> 1), stride = (int)(gridDim.x >> 1);

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < kStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 16); }     // 8 epilogue warps of both CTAs
    for (int s = 0; s < 8 * kSlots; ++s) mbar_init(&src_bar[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"((uint32_t)(2 * TN)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  __syncwarp();
  cluster_sync();                            // the peer's barriers exist before anything of ours signals them
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_base_slot;

  if (warp == 0 && lane == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
    bool ok = true;
    uint32_t s = 0, ph = 1;                                    // stage and the parity of its next release
    for (int t = first; t < n_tiles && ok; t += stride) {
      const PairTile tile(t, mt, nt, splits, total_kb, rank);
      const int m0 = tile.m0, nb0 = tile.n0 + (int)rank * 128;                 // this CTA's rows of A and of B
      for (int kb = 0; kb < tile.num_kb; ++kb) {
        ok = mbar_wait(&empty_bar[s], ph, &abort_flag);
        if (!ok) break;
        uint8_t* sa = smem + s * kStageBytes;
        uint8_t* sb = sa + kHalfBytes;
        if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * kStageBytes);        // both CTAs' loads complete on the leader's barrier
        const uint32_t bar = smem_u32(&full_bar[s]) & kPeerMask;
        const int k0 = (tile.kb_begin + kb) * BK;
        if (!A_MN) tma_load_2d_pair(sa, &map_a, k0, m0, bar);                                   // box {BK, 128}
        else { tma_load_2d_pair(sa, &map_a, m0, k0, bar); tma_load_2d_pair(sa + kHalfBytes / 2, &map_a, m0 + 64, k0, bar); }   // 2 x box {64, BK}
        if (!B_MN) tma_load_2d_pair(sb, &map_b, k0, nb0, bar);
        else { tma_load_2d_pair(sb, &map_b, nb0, k0, bar); tma_load_2d_pair(sb + kHalfBytes / 2, &map_b, nb0 + 64, k0, bar); }
        if (++s == (uint32_t)kStages) { s = 0; ph ^= 1u; }
      }
    }
  } else if (warp == 1 && rank == 0) {
    // ------------------------------------------------------------------ MMA issuer (leader only; the whole warp, one lane issues)
    // One issuer serves the SM pair, so a stage's four MMAs and commit must take less to issue than the 512 cycles they run: elect_one, and
    // descriptors that advance by adding to the 16-byte address field. (Issued from a branch of lane 0, with descriptors built for each:
    // 723 instead of 672 us at 8192^3, 143 instead of 130 at 16384 x 2048 x 3200.)
    // instruction descriptor: D = f32, A = B = bf16, majors, N >> 3, M >> 4 with M = 256 (both CTAs' rows)
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((A_MN ? 1u : 0u) << 15) | ((B_MN ? 1u : 0u) << 16) |
                           ((uint32_t)(TN >> 3) << 17) | ((uint32_t)((2 * TM) >> 4) << 24);
    const uint32_t base = smem_u32(smem);
    const uint64_t d_a = A_MN ? make_desc(base, BK * 128, 1024) : make_desc(base, 16, 1024);
    const uint64_t d_b = B_MN ? make_desc(base + kHalfBytes, BK * 128, 1024) : make_desc(base + kHalfBytes, 16, 1024);
    constexpr uint64_t kStepA = (A_MN ? 2048 : 32) >> 4, kStepB = (B_MN ? 2048 : 32) >> 4;        // 16 reduction elements further
    const bool leader = elect_one();
    auto wait_all = [&](uint64_t* bar, uint32_t parity) -> bool {               // one outcome for the whole warp
      return __all_sync(0xffffffffu, mbar_wait(bar, parity, &abort_flag) ? 1 : 0) != 0;
    };
    bool ok = true;
    uint32_t s = 0, ph = 0;
    int ti = 0;                                                // tiles since the start
    for (int t = first; t < n_tiles && ok; t += stride) {
      const PairTile tile(t, mt, nt, splits, total_kb, rank);
      if (tile.num_kb == 0) continue;
      const int buf = ti & 1;
      ok = wait_all(&acc_empty[buf], (uint32_t)((ti >> 1) & 1) ^ 1u);      // the epilogues of tile ti - 2 have read it
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t acc = tmem_base + (uint32_t)(buf * TN);
      for (int kb = 0; kb < tile.num_kb; ++kb) {
        ok = wait_all(&full_bar[s], ph);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t da = d_a + (uint64_t)(s * (kStageBytes >> 4)), db = d_b + (uint64_t)(s * (kStageBytes >> 4));
        if (leader) {
#pragma unroll
          for (int k = 0; k < BK / UK; ++k) umma_bf16_pair(acc, da + k * kStepA, db + k * kStepB, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          umma_commit_pair(&empty_bar[s]);
        }
        __syncwarp();
        if (++s == (uint32_t)kStages) { s = 0; ph ^= 1u; }
      }
      if (ok && leader) umma_commit_pair(&acc_full[buf]);
      __syncwarp();
      ++ti;
    }
  } else if (warp >= 2) {
    // ------------------------------------------------------------------ epilogue (8 warps: lane quarter warp & 3, column half (warp - 2) / 4)
    constexpr int kCols = Store<OutT>::kBoxCols, kBoxes = 128 / kCols;
    const int q = warp & 3, half = (warp - 2) >> 2;
    uint8_t* slots = smem + kStages * kStageBytes + (warp - 2) * kSlots * 4096;
    uint64_t* bars = src_bar + (warp - 2) * kSlots;
    const rb::gemm::EpilogueWork work{&map_o, MM, relu != 0, reduce_out != 0, colsum != nullptr};
    // Column sums stay in registers while the column tile stays the same (with the grid a multiple of the column tiles: always). Added to
    // global memory box by box they cost more than the rest of the epilogue.
    float sums[kBoxes][kCols / 32];
#pragma unroll
    for (int b = 0; b < kBoxes; ++b)
#pragma unroll
      for (int e = 0; e < kCols / 32; ++e) sums[b][e] = 0.f;
    int sums_n0 = -1;
    auto flush_sums = [&]() {
      const int at = sums_n0 + half * 128 + rb::gemm::column_of<kCols>(lane);
#pragma unroll
      for (int b = 0; b < kBoxes; ++b)
#pragma unroll
        for (int e = 0; e < kCols / 32; ++e) {
          if (at + b * kCols + e < NN) atomicAdd(colsum + at + b * kCols + e, sums[b][e]);
          sums[b][e] = 0.f;
        }
    };
    // Boxes are counted over all tiles: box g of this warp uses slot g % kSlots. `ahead` walks the boxes whose second input is fetched.
    int g = 0, ti = 0;
    int ahead_t = first, ahead_b = 0, ahead_g = 0;
    auto fetch_next = [&]() {                                  // lane 0: the next box's second input into its slot
      while (ahead_t < n_tiles) {
        const PairTile tile(ahead_t, mt, nt, splits, total_kb, rank);
        const int row0 = tile.m0 + q * 32, col = tile.n0 + half * 128 + ahead_b * kCols;
        if (row0 >= MM || col >= NN) { ahead_t += stride; ahead_b = 0; continue; }
        const int slot = ahead_g % kSlots;
        mbar_expect_tx(&bars[slot], 4096);
        tma_load_2d(slots + slot * 4096, &map_src, col, row0, &bars[slot]);
        ++ahead_g;
        if (++ahead_b == kBoxes) { ahead_t += stride; ahead_b = 0; }
        return;
      }
    };
    if (kSrc && lane == 0) { fetch_next(); fetch_next(); }
    bool ok = true;
    for (int t = first; t < n_tiles && ok; t += stride) {
      const PairTile tile(t, mt, nt, splits, total_kb, rank);
      if (tile.num_kb == 0) continue;
      const int row0 = tile.m0 + q * 32, buf = ti & 1;
      ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[buf], (uint32_t)((ti >> 1) & 1), &abort_flag) ? 1 : 0) != 0;
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t acc = tmem_base + (uint32_t)(buf * TN) + ((uint32_t)(q * 32) << 16);
      if (colsum != nullptr && tile.n0 != sums_n0) {
        if (sums_n0 >= 0) flush_sums();
        sums_n0 = tile.n0;
      }
      bool released = false;
#pragma unroll 1
      for (int b = 0; b < kBoxes; ++b, ++g) {
        const int c0 = half * 128 + b * kCols, col = tile.n0 + c0;
        if (row0 >= MM || col >= NN) break;
        const int slot = g % kSlots;
        float v[kCols];
        rb::gemm::load_box<kCols>(acc + (uint32_t)c0, v);
        if (b == kBoxes - 1) {                                 // the accumulator has been read: the tile after next may overwrite it
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) arrive_leader(&acc_empty[buf]);
          released = true;
        }
        if (kSrc) {
          ok = __all_sync(0xffffffffu, mbar_wait(&bars[slot], (uint32_t)(g / kSlots) & 1u, &abort_flag) ? 1 : 0) != 0;
          if (!ok) break;
          if (lane == 0) {
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");    // the box before this one has left its slot
            fetch_next();
          }
        } else {
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");      // the box before this one has left the slot
          __syncwarp();
        }
        const float* bias_at = bias != nullptr && tile.first_split ? bias + col : nullptr;
        if (bias_at != nullptr && (col + kCols > NN || (reinterpret_cast<uintptr_t>(bias_at) & 7))) {      // edge or odd address: one by one
#pragma unroll
          for (int j = 0; j < kCols; ++j) {
            const int c = 8 * ((j & (kCols / 2 - 1)) >> 2) + 2 * (lane & 3) + (j & 1);
            if (col + c < NN) v[j] += bias_at[c];
          }
          bias_at = nullptr;
        }
        float sum[kCols / 32];
#pragma unroll
        for (int e = 0; e < kCols / 32; ++e) sum[e] = 0.f;
        rb::gemm::finish_box<OutT>(work, v, bias_at, kSrc, slots + slot * 4096, row0, col, lane, sum);
#pragma unroll
        for (int k = 0; k < kBoxes; ++k)
#pragma unroll
          for (int e = 0; e < kCols / 32; ++e) sums[k][e] += k == b ? sum[e] : 0.f;
      }
      if (ok && !released) {                                   // nothing, or not everything, of this part lies inside D
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) arrive_leader(&acc_empty[buf]);
      }
      ++ti;
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");       // the slots must stay until the copies have read them
    if (colsum != nullptr) {
      // what is left, summed over the four row quarters first: a quarter of the additions to the same few addresses, whole lines of them
      float* part = reinterpret_cast<float*>(smem + kStages * kStageBytes);
      asm volatile("bar.sync 1, 256;" ::: "memory");             // every warp's boxes have left the slots
#pragma unroll
      for (int b = 0; b < kBoxes; ++b)
#pragma unroll
        for (int e = 0; e < kCols / 32; ++e) part[q * TN + half * 128 + b * kCols + rb::gemm::column_of<kCols>(lane) + e] = sums[b][e];
      asm volatile("bar.sync 1, 256;" ::: "memory");
      const int c = (int)threadIdx.x - 64;
      if (sums_n0 >= 0 && sums_n0 + c < NN) atomicAdd(colsum + sums_n0 + c, (part[c] + part[TN + c]) + (part[2 * TN + c] + part[3 * TN + c]));
    }
  }
  if (abort_flag) {
    // a wait ran out: copies of this pair may still be on their way into shared memory; give them time before it goes away
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  __syncwarp();
  cluster_sync();                            // both epilogues are done and nothing of the peer's is in flight towards this CTA
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)(2 * TN)) : "memory");
  }
  if (threadIdx.x == 0 && abort_flag) rb::set_status(status, rb::kStatusWaitTimeout);
}

template <bool A_MN, bool B_MN, bool kSrc, typename OutT>
int launch_pair(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mo, const CUtensorMap& ms, const float* bias, float* colsum,
                int MM, int NN, int KK, int relu, int splits, int reduce_out, int64_t* status, cudaStream_t st) {
  auto kern = gemm_bf16_tcgen05_2cta_kernel<A_MN, B_MN, kSrc, OutT>;
  constexpr uint32_t smem = Ring<kSrc>::kBytes;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 3;
    attr_set = true;
  }
  const int64_t tiles = (int64_t)((MM + 2 * TM - 1) / (2 * TM)) * ((NN + TN - 1) / TN) * splits;
  if (tiles > (int64_t)1 << 30) return 7;
  // As many pairs as share the tiles evenly in the rounds that they take: with a tile more or less each, the last round would run for a few, and
  // those of the rounds before would share the bandwidth of L2 with pairs that finish no earlier (24576 x 256 x 3200, 96 tiles: 42.9 us with
  // 74 pairs, 39.8 with 48; dW 2048 x 3200 of 65536 rows: 733 and 706). A second input or column sums are limited by memory rather than
  // by operands, and every SM helps (19200 x 256 x 256 with a residual, 75 tiles: 18.3 us with 74 pairs, 23.2 with 38).
  const bool operands_only = !kSrc && colsum == nullptr;
  const int64_t rounds = (tiles + kPairs - 1) / kPairs;
  int pairs = (int)(operands_only ? (tiles + rounds - 1) / rounds : std::min<int64_t>(tiles, kPairs));
  // with column sums a pair stays with one column tile where there are at most kGroup of them
  const int width = std::min((NN + TN - 1) / TN, kGroup);
  if (colsum != nullptr && pairs > width) pairs -= pairs % width;
  kern<<<2 * pairs, kThreads, smem, st>>>(ma, mb, mo, ms, bias, colsum, MM, NN, KK, relu, splits, reduce_out, status);
  rb::note_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

}  // namespace

// Same contract as rb_gemm_bf16 (rb_dense.h), for outputs that can leave through TMA stores (base and row pitch 16-byte aligned); `reduce_out`:
// the output is added to, by `splits` parts of the reduction.
// Returns 7 when the problem does not suit the pair kernel (the caller then uses the one-CTA kernel).
extern "C" int rb_gemm_bf16_pair(const void* a, int64_t lda, int a_mn, const void* b, int64_t ldb, int b_mn, void* out, int64_t ldo,
                                 int out_fp32, const float* bias, const float* beta_src, const RbGemmEpilogue* epi_in, int MM, int NN, int KK,
                                 int relu, int splits, int reduce_out, int64_t* status, cudaStream_t st) {
  RbGemmEpilogue epi{nullptr, 0, nullptr, 0};
  if (epi_in != nullptr) epi = *epi_in;
  if ((epi.mask_src != nullptr || epi.colsum != nullptr) && reduce_out) return 6;
  if (MM < 192 || NN < 192 || KK <= 0) return 7;
  if ((reinterpret_cast<uintptr_t>(a) & 15) || (reinterpret_cast<uintptr_t>(b) & 15) || (lda % 8) || (ldb % 8)) return 1;
  const int es = out_fp32 ? 4 : 2;
  if ((reinterpret_cast<uintptr_t>(out) & 15) || (ldo * es) % 16) return 7;
  if (reduce_out && (!out_fp32 || relu)) return 6;
  // the second input of the epilogue comes as boxes in the layout of the output: a residual (fp32 output) or a mask (bf16 output)
  const bool mask = epi.mask_src != nullptr;
  if ((mask && (out_fp32 || beta_src != nullptr)) || (beta_src != nullptr && !out_fp32)) return 7;
  const void* src = mask ? epi.mask_src : beta_src;
  const int64_t src_ld = mask ? epi.mask_ld : ldo;
  if (src != nullptr && (reduce_out || (reinterpret_cast<uintptr_t>(src) & 15) || (src_ld * es) % 16)) return 7;
  CUtensorMap ma, mb, mo, ms;
  // boxes: K-major operands {BK, 128 rows}; MN-major operands {64, BK}; output {32 or 64 columns, 32 rows}
  const int ra = a_mn ? rb_tensor_map_2d(&ma, a, KK, MM, lda, 64, BK, 0) : rb_tensor_map_2d(&ma, a, MM, KK, lda, BK, 128, 0);
  const int rbm = b_mn ? rb_tensor_map_2d(&mb, b, KK, NN, ldb, 64, BK, 0) : rb_tensor_map_2d(&mb, b, NN, KK, ldb, BK, 128, 0);
  const int ro = rb_tensor_map_2d(&mo, out, MM, NN, ldo, out_fp32 ? 32 : 64, 32, out_fp32);
  const int rs = src != nullptr ? rb_tensor_map_2d(&ms, src, MM, NN, src_ld, out_fp32 ? 32 : 64, 32, out_fp32) : 0;
  if (src == nullptr) ms = mo;
  if (ra || rbm || ro || rs) return 2;
#define RB_PAIR_CASE(AM, BMJ)                                                                                                    \
  if ((a_mn != 0) == AM && (b_mn != 0) == BMJ)                                                                                   \
    return out_fp32 ? (src != nullptr ? launch_pair<AM, BMJ, true, float> : launch_pair<AM, BMJ, false, float>)(ma, mb, mo, ms, bias, epi.colsum, MM, NN, KK, relu, splits, reduce_out, status, st)    \
                    : (src != nullptr ? launch_pair<AM, BMJ, true, __nv_bfloat16> : launch_pair<AM, BMJ, false, __nv_bfloat16>)(ma, mb, mo, ms, bias, epi.colsum, MM, NN, KK, relu, 1, 0, status, st);
  RB_PAIR_CASE(false, false)
  RB_PAIR_CASE(false, true)
  RB_PAIR_CASE(true, false)
  RB_PAIR_CASE(true, true)
#undef RB_PAIR_CASE
  return 5;
}
