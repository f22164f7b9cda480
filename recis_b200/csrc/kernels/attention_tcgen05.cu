// Ragged (unpadded) multi-head self-attention on the 5th-generation tensor cores, head width 64.
//
// Input is the packed projection output qkv [T, 3 * H * 64] (bf16) of all sequences of a batch back to back, plus the
// sequence boundaries offsets [B + 1]; no padding exists anywhere. A work item of the forward is one (sequence, head, 128-query tile); it
// walks the sequence's keys in steps of 128 with an online softmax:
//
//   S  = Q K^T        tcgen05.mma, A = Q tile, B = K tile, both K-major; the tiles arrive by TMA straight from the packed matrix
//                     in the 128-byte swizzle; fp32 result in tensor memory
//   P  = exp2(S * scale * log2 e - m)   each thread owns one query row: it reads its row of S with tcgen05.ld, keeps the maximum m and the
//                     sum l in registers and writes P (bf16) into shared memory
//   O += P V          tcgen05.mma, A = P, B = the V tile read as an MN-major operand (N = head column, K = key row); each step's product is
//                     added to O in registers. (Rescaling only from some growth on saves a tenth of the time, but then the largest P
//                     of a row is not exactly one: up to 12 % more error.)
//
// and finally writes O / l (bf16) and the log-sum-exp (base 2) of the row. Persistent CTAs with separate roles: four softmax warps, one
// that fetches work and issues the TMA loads, one that issues the MMAs. S of the next step is multiplied as soon as this one's has been read,
// under P V. Keys past the end of a sequence are masked in the softmax; query rows past the end are computed on whatever is there and not
// stored; of a partial tile only the 32-row boxes that hold a row are loaded.
//
// What bounds it is the latency of a step - score, exponentials, product, in sequence for a query tile - with two query tiles to an SM (tensor
// memory holds no more): no unit is near its limit (first case below: tensor pipe 21 %, special-function units 40 %, issue slots 38 %).
// Measured on a B200 with cold L2 (before: the kernel with a CTA per item below, which small batches still use):
//   256 sequences of 50..1000 tokens, 4 heads:  311 -> 235 us (93 GFLOP in existing elements: 395 TFLOP/s)
//   3000 sequences of 1..90 tokens, 8 heads:    425 -> 230 us; under a bound of 1000 instead of 90: 1319 -> 235 us
//   37 sequences of 1..1000 tokens, 4 heads:     58 -> 57 us;  one sequence of 1000 tokens, 8 heads: 27 -> 24.6 us
//
// The reference has no attention kernel; its sequence example pads to the longest sequence and calls the library SDPA
// (examples/seq2seq/transformer.py:36-38). Waits are bounded; a timeout sets the status word and the CTA frees its tensor
// memory and returns. These kernels are what ops/attention.py runs on CUDA for head width 64 (RECIS_ATTENTION=padded selects
// the padded library path).
#include "../common/rb_common.cuh"
#include "../common/rb_launch.h"
#include "../common/rb_tcgen05.cuh"
#include "rb_dense.h"
#include <cuda.h>
#include <cuda_bf16.h>
#include <algorithm>
#include <cstring>

namespace {

using namespace rb::tc;

constexpr int kTile = 128;                 // queries of a work item = keys per step = tensor-memory lanes
constexpr int kHead = 64;                  // head width (one 128-byte swizzle row)
constexpr int kBlk = kTile * 128;          // bytes of one [128 rows x 64 bf16] swizzled block

// 2^x on the special-function unit: one instruction, flushes denormals, 2^-inf = 0 (which is how masked entries become zero)
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// two floats -> packed bf16x2 (round to nearest even), first argument in the low half
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// ---------------------------------------------------------------------------------------------- forward
struct AttnItem { int s0, len, head, kt; };          // len < 0: no more work; kt: the item's tile (of queries here, of keys in the backward)

// 128 keys a step and the rows of O in registers, whatever the batch: an output depends on its sequence alone, to the bit. (64 keys a step and
// O in tensor memory let four CTAs share an SM, 166 against 235 us at 3000 sequences of 1..90 tokens, 8 heads, and 207 against 225 at
// 256 sequences of 50..1000 tokens, 4 heads. But P is then rounded against the maxima of half as many keys and O rescaled and summed in
// another order: 6e-4 of the first case's outputs by norm, and a sequence's outputs would depend on how many others are in its batch.)
constexpr int kFwdCtas = 2;                                      // per SM
constexpr uint32_t kFwdS = 0, kFwdO = kTile;                     // tensor-memory columns: S and O, fp32
constexpr uint32_t kFwdTmemCols = 256;
constexpr size_t kFwdSmem = 1024 + 5 * (size_t)kBlk;             // Q, two blocks of [128 q x 64 keys] of P, K, V
constexpr int kFwdThreads = 192;                                 // four softmax warps, producer, MMA

// 8 columns of tensor memory, one row per lane
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void fma_f32x2(float& x0, float& x1, float a0, float a1, float b, float c) {      // x = a * b + c
  asm("{\n\t.reg .b64 u, w, z;\n\tmov.b64 u, {%2, %3};\n\tmov.b64 w, {%4, %4};\n\tmov.b64 z, {%5, %5};\n\tfma.rn.f32x2 u, u, w, z;\n\tmov.b64 {%0, %1}, u;\n\t}"
      : "=f"(x0), "=f"(x1) : "f"(a0), "f"(a1), "f"(b), "f"(c));
}
__device__ __forceinline__ void add_f32x2(float& x0, float& x1, float a0, float a1) {
  asm("{\n\t.reg .b64 u, w;\n\tmov.b64 u, {%0, %1};\n\tmov.b64 w, {%2, %3};\n\tadd.rn.f32x2 u, u, w;\n\tmov.b64 {%0, %1}, u;\n\t}"
      : "+f"(x0), "+f"(x1) : "f"(a0), "f"(a1));
}

// N columns of one row of S: P = 2^(S * scale_log2 - m) as bf16 pairs; the sums go to four chains
template <int N>
__device__ __forceinline__ void exp_chunk(const uint32_t (&s)[N], float scale_log2, float neg_m, float (&sum)[4], uint32_t (&pk)[N / 2]) {
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {
    float x, y;
    fma_f32x2(x, y, __uint_as_float(s[2 * i]), __uint_as_float(s[2 * i + 1]), scale_log2, neg_m);
    x = fast_exp2(x);
    y = fast_exp2(y);
    add_f32x2(sum[(i & 1) * 2], sum[(i & 1) * 2 + 1], x, y);
    pk[i] = pack_bf16x2(x, y);
  }
}

// 16 bytes to shared memory. 32-bit addresses, and the swizzle as one exclusive-or per 16-byte column on a row base (bits 4..6 of
// the base already hold the row's part): the address arithmetic of all tiles shares eight registers.
__device__ __forceinline__ void st_shared16(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// One thread's row of a 128-key tile of S (tensor memory at `trow`): new running maximum and sum, P = 2^(S * scale_log2 - m)
// written as bf16 into the two K-major blocks of `ptile`. Returns the factor by which what was accumulated under the old
// maximum shrinks. kMask selects whether key columns >= valid are masked: a full tile pays for no compare or select.
// The row is read from tensor memory once (four 32-column reads in flight) and stays in registers for both passes; the
// maximum and the sum run as four independent chains each, since one warp per scheduler hides no dependent latency.
template <bool kMask>
__device__ __forceinline__ float softmax_row(uint32_t trow, int valid, float scale_log2, int t, uint8_t* ptile, float& m, float& l) {
  uint32_t s0[32], s1[32], s2[32], s3[32];
  __syncwarp();
  tmem_ld32(trow, s0);
  tmem_ld32(trow + 32u, s1);
  tmem_ld32(trow + 64u, s2);
  tmem_ld32(trow + 96u, s3);
  tmem_ld_wait();
  // masking is a select on the value (no branch per element): a masked key becomes -inf here and an exact zero after the
  // exponential; scale_log2 > 0, so the maximum can be taken before scaling
  if (kMask) {
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      if (i >= valid) s0[i] = 0xff800000u;
      if (32 + i >= valid) s1[i] = 0xff800000u;
      if (64 + i >= valid) s2[i] = 0xff800000u;
      if (96 + i >= valid) s3[i] = 0xff800000u;
    }
  }
  float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    mx0 = fmaxf(mx0, __uint_as_float(s0[i]));
    mx1 = fmaxf(mx1, __uint_as_float(s1[i]));
    mx2 = fmaxf(mx2, __uint_as_float(s2[i]));
    mx3 = fmaxf(mx3, __uint_as_float(s3[i]));
  }
  const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
  const float m_new = fmaxf(m, mx * scale_log2);
  const float alpha = (m == -INFINITY) ? 0.f : fast_exp2(m - m_new);
  float sum0 = 0.f, sum1 = 0.f, sum2 = 0.f, sum3 = 0.f;
#pragma unroll
  for (int q4 = 0; q4 < 4; ++q4) {                 // 32 key columns per quarter; two quarters per 64-wide K-major block
    uint8_t* blk = ptile + (q4 >> 1) * kBlk;
    uint32_t pk[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const uint32_t ua = q4 == 0 ? s0[2 * i] : q4 == 1 ? s1[2 * i] : q4 == 2 ? s2[2 * i] : s3[2 * i];
      const uint32_t ub = q4 == 0 ? s0[2 * i + 1] : q4 == 1 ? s1[2 * i + 1] : q4 == 2 ? s2[2 * i + 1] : s3[2 * i + 1];
      // -inf * scale_log2 - m_new = -inf (m_new is finite whenever the tile has one existing key): 2^-inf = 0
      const float p0 = fast_exp2(fmaf(__uint_as_float(ua), scale_log2, -m_new));
      const float p1 = fast_exp2(fmaf(__uint_as_float(ub), scale_log2, -m_new));
      if (i & 1) { sum1 += p0; sum3 += p1; } else { sum0 += p0; sum2 += p1; }
      pk[i] = pack_bf16x2(p0, p1);
    }
#pragma unroll
    for (int cq = 0; cq < 4; ++cq)
      *reinterpret_cast<uint4*>(blk + swizzle128_offset(t, (q4 & 1) * 32 + cq * 8)) =
          make_uint4(pk[cq * 4], pk[cq * 4 + 1], pk[cq * 4 + 2], pk[cq * 4 + 3]);
  }
  l = l * alpha + ((sum0 + sum1) + (sum2 + sum3));
  m = m_new;
  return alpha;
}

// Small batches: one CTA of 128 threads per work item (blockIdx: query tile, sequence, head), its loads, MMAs and exponentials one after the other,
// and two to an SM. There is no counter to clear, no work to fetch and one role to wake, which is what a few hundred short items take longest
// for; with the same steps, sums and roundings as in the persistent kernel below, every output is the same to the bit.
__global__ void __launch_bounds__(128, 2)
ragged_attention_fwd_item_kernel(const __grid_constant__ CUtensorMap map_qkv, const int32_t* __restrict__ offsets, int64_t T, int H, float scale_log2,
                            __nv_bfloat16* __restrict__ out, float* __restrict__ lse2, int64_t* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_q, bar_k, bar_v, bar_s, bar_o;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int b = blockIdx.y, h = blockIdx.z, qt = blockIdx.x;
  const int s0 = offsets[b], L = offsets[b + 1] - s0;
  // Rows that no tile computes read as zeros: tokens in front of and behind the sequences, and those of a sequence that is longer than the
  // bound the grid was sized with.
  const bool edge0 = qt == 0 && b == 0 && s0 > 0, edge1 = qt == 0 && b == (int)gridDim.y - 1 && s0 + L < T;
  const bool edge2 = qt == (int)gridDim.x - 1 && L > (qt + 1) * kTile;
  if (edge0 || edge1 || edge2) {
#pragma unroll 1
    for (int e = 0; e < 3; ++e) {
      if (!(e == 0 ? edge0 : e == 1 ? edge1 : edge2)) continue;
      const int64_t from = e == 0 ? 0 : e == 1 ? s0 + L : s0 + (qt + 1) * kTile, to = e == 0 ? (int64_t)s0 : e == 1 ? T : (int64_t)s0 + L;
#pragma unroll 1
      for (int64_t row = from + (threadIdx.x >> 3); row < to; row += 16) {
        reinterpret_cast<uint4*>(out + (row * H + h) * kHead)[threadIdx.x & 7] = make_uint4(0u, 0u, 0u, 0u);
        if (lse2 && (threadIdx.x & 7) == 0) lse2[row * H + h] = 0.f;
      }
    }
  }
  if (qt * kTile >= L) return;                                   // uniform for the CTA, before any barrier or allocation

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* qtile = smem;                  // [128 q][64 d]      K-major A of S = Q K^T
  uint8_t* ktile = smem + kBlk;           // [128 keys][64 d]   K-major B of S
  uint8_t* vtile = smem + 2 * kBlk;       // [128 keys][64 d]   MN-major B of PV (N = d, K = key)
  uint8_t* ptile = smem + 3 * kBlk;       // 2 x [128 q][64 keys] K-major A of PV
  const int t = threadIdx.x, warp = t >> 5;
  // Q, K and V tiles arrive by TMA straight from the packed [T, 3 * H * 64] matrix (box of 128 rows x 64 columns, 128-byte
  // swizzle). Rows past the end of the sequence belong to the next sequence (or read as zeros past the end of the matrix):
  // surplus query rows are computed and never stored, surplus keys are masked in the softmax, and the surplus rows of the V
  // tile are zeroed in shared memory, so that a zero probability never meets a non-finite value.
  const int xq = h * kHead, xk = (H + h) * kHead, xv = (2 * H + h) * kHead;
  if (t == 0) {
    abort_flag = 0;
    mbar_init(&bar_q, 1); mbar_init(&bar_k, 1); mbar_init(&bar_v, 1); mbar_init(&bar_s, 1); mbar_init(&bar_o, 1);
    mbar_fence_init();
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_qkv) : "memory");
    mbar_expect_tx(&bar_q, kBlk); tma_load_2d(qtile, &map_qkv, xq, s0 + qt * kTile, &bar_q);
    mbar_expect_tx(&bar_k, kBlk); tma_load_2d(ktile, &map_qkv, xk, s0, &bar_k);
    mbar_expect_tx(&bar_v, kBlk); tma_load_2d(vtile, &map_qkv, xv, s0, &bar_v);
  }
  if (warp == 0) tmem_alloc(&tmem_slot, kFwdTmemCols);

  const int q = qt * kTile + t;
  const bool q_ok = q < L;
  float o[kHead];
#pragma unroll
  for (int d = 0; d < kHead; ++d) o[d] = 0.f;
  float m = -INFINITY, l = 0.f;
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = tmem_slot;
  const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
  const uint32_t idesc_s = make_idesc_bf16(kTile, kTile, false, false);
  const uint32_t idesc_o = make_idesc_bf16(kTile, kHead, false, true);
  bool ok = true;

  const int n_kv = (L + kTile - 1) / kTile;
  for (int j = 0; j < n_kv && ok; ++j) {
    const uint32_t ph = (uint32_t)(j & 1);
    if (t == 0) {
      bool got = (j > 0 || mbar_wait(&bar_q, 0, &abort_flag)) && mbar_wait(&bar_k, ph, &abort_flag);
      if (got) {
        fence_after_sync();
        const uint32_t sq = smem_u32(qtile), sk = smem_u32(ktile);
#pragma unroll
        for (int k = 0; k < kHead / 16; ++k)
          umma_bf16(tmem, make_desc(sq + k * 32, 16, 1024), make_desc(sk + k * 32, 16, 1024), idesc_s, k > 0 ? 1u : 0u);
        umma_commit(&bar_s);
      }
    }
    // the outcome of a bounded wait is made uniform for the CTA: every thread takes the same path through the barriers below
    ok = __syncthreads_and(mbar_wait(&bar_s, ph, &abort_flag) ? 1 : 0) != 0;
    fence_after_sync();
    if (!ok) break;
    // S is complete, so the K tile is free: the next one travels while this tile's softmax and P V run
    if (t == 0 && j + 1 < n_kv) { mbar_expect_tx(&bar_k, kBlk); tma_load_2d(ktile, &map_qkv, xk, s0 + (j + 1) * kTile, &bar_k); }

    // ---- online softmax on this thread's row of S; only the sequence's last key tile can hold keys that do not exist
    const int valid = min(kTile, L - j * kTile);                 // key columns of this tile that exist
    const int steps = (valid + 15) >> 4;                         // 16-key steps of the product with V
    float alpha = 1.f;
    if (qt * kTile + warp * 32 >= L) { /* none of this warp's rows exist: what their P holds only reaches rows that are not stored */ }
    else if (valid == kTile) alpha = softmax_row<false>(tmem + lane_base, kTile, scale_log2, t, ptile, m, l);
    else alpha = softmax_row<true>(tmem + lane_base, valid, scale_log2, t, ptile, m, l);

    if (valid < kTile) {
      // last, partial tile: the V rows past the end of the sequence become zeros (this thread's row, once V has landed)
      ok = mbar_wait(&bar_v, ph, &abort_flag);
      if (ok && t >= valid && t < steps * 16) {
#pragma unroll
        for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4*>(vtile + swizzle128_offset(t, c * 8)) = make_uint4(0u, 0u, 0u, 0u);
      }
    }
    fence_smem_to_async();
    fence_before_sync();
    ok = __syncthreads_and(ok ? 1 : 0) != 0;
    fence_after_sync();
    if (!ok) break;
    if (t == 0) {
      if (mbar_wait(&bar_v, ph, &abort_flag)) {
        fence_after_sync();
        const uint32_t sp = smem_u32(ptile), sv = smem_u32(vtile);
        for (int k = 0; k < steps; ++k)
          umma_bf16(tmem + kFwdO, make_desc(sp + (k >> 2) * kBlk + (k & 3) * 32, 16, 1024), make_desc(sv + k * 2048, kBlk, 1024), idesc_o,
                    k > 0 ? 1u : 0u);
        umma_commit(&bar_o);
      }
    }
    ok = __syncthreads_and(mbar_wait(&bar_o, ph, &abort_flag) ? 1 : 0) != 0;
    fence_after_sync();
    if (!ok) break;
    // P V is complete, so the V tile is free
    if (t == 0 && j + 1 < n_kv) { mbar_expect_tx(&bar_v, kBlk); tma_load_2d(vtile, &map_qkv, xv, s0 + (j + 1) * kTile, &bar_v); }
    {
      uint32_t r0[32], r1[32];
      __syncwarp();
      tmem_ld32(tmem + lane_base + kFwdO, r0);
      tmem_ld32(tmem + lane_base + kFwdO + 32u, r1);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 32; ++i) {           // O = O * alpha + P V, one multiply-add per element
        o[i] = fmaf(o[i], alpha, __uint_as_float(r0[i]));
        o[32 + i] = fmaf(o[32 + i], alpha, __uint_as_float(r1[i]));
      }
    }
  }

  if (ok && q_ok) {
    const float inv = l > 0.f ? 1.f / l : 0.f;
    __nv_bfloat16* dst = out + (int64_t)(s0 + q) * H * kHead + h * kHead;
#pragma unroll
    for (int c = 0; c < 8; ++c)
      reinterpret_cast<uint4*>(dst)[c] = make_uint4(pack_bf16x2(o[c * 8] * inv, o[c * 8 + 1] * inv), pack_bf16x2(o[c * 8 + 2] * inv, o[c * 8 + 3] * inv),
                                                    pack_bf16x2(o[c * 8 + 4] * inv, o[c * 8 + 5] * inv), pack_bf16x2(o[c * 8 + 6] * inv, o[c * 8 + 7] * inv));
    if (lse2) lse2[(int64_t)(s0 + q) * H + h] = m + log2f(l);
  }
  if (abort_flag) {
    // a wait ran out: a copy may still be on its way into shared memory; give it time before the memory goes away
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) { __syncwarp(); fence_after_sync(); tmem_dealloc(tmem, kFwdTmemCols); }
  if (t == 0 && abort_flag) rb::set_status(status, rb::kStatusWaitTimeout);
}

// Rows [from, to) of out and lse become zeros; `threads` threads, this one is `t`.
__device__ __forceinline__ void clear_rows(int64_t from, int64_t to, int H, __nv_bfloat16* out, float* lse2, int64_t t, int64_t threads) {
  for (int64_t i = from * H * 8 + t; i < to * H * 8; i += threads) {
    reinterpret_cast<uint4*>(out)[i] = make_uint4(0u, 0u, 0u, 0u);
    if (lse2 && (i & 7) == 0) lse2[i >> 3] = 0.f;
  }
}

__global__ void __launch_bounds__(kFwdThreads, kFwdCtas)
ragged_attention_fwd_kernel(const __grid_constant__ CUtensorMap map_qkv, const __grid_constant__ CUtensorMap map_rows,
                            const int32_t* __restrict__ offsets, int64_t T, int B, int H, int tiles, int chunk, float scale_log2,
                            __nv_bfloat16* __restrict__ out, float* __restrict__ lse2, unsigned* __restrict__ counter,
                            int64_t* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t q_full[2], k_full, v_full;
  __shared__ __align__(8) uint64_t s_full, p_full, o_full, o_empty;
  __shared__ AttnItem slot[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* qtile = smem;                             // [128 q][64 d]   K-major A of S = Q K^T
  uint8_t* ptile = smem + kBlk;                      // 2 x [128 q][64 keys]   K-major A of P V; then the rows of O on their way out
  uint8_t* ktile = smem + 3 * kBlk;                  // [128 keys][64 d]       K-major B of S
  uint8_t* vtile = smem + 4 * kBlk;                  // [128 keys][64 d]       MN-major B of P V (N = d, K = key)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kProducer = 4, kMma = 5;

  // Rows that no item computes read as zeros: tokens in front of and behind the sequences, and those of a sequence that is longer than
  // the bound. Work of one warp.
  auto clear_uncovered = [&]() {
    const int64_t every = (int64_t)gridDim.x * 32, me = (int64_t)blockIdx.x * 32 + lane;
    clear_rows(0, offsets[0], H, out, lse2, me, every);
    clear_rows(offsets[B], T, H, out, lse2, me, every);
    for (int64_t b0 = (int64_t)blockIdx.x * 32; b0 < B; b0 += every) {
      const int b = (int)min(b0 + lane, (int64_t)B - 1), s0 = offsets[b], s1 = offsets[b + 1];
      unsigned todo = __ballot_sync(0xffffffffu, b0 + lane < B && s1 - s0 > tiles * kTile);
      for (; todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1;
        clear_rows((int64_t)__shfl_sync(0xffffffffu, s0, src) + tiles * kTile, __shfl_sync(0xffffffffu, s1, src), H, out, lse2, lane, 32);
      }
    }
  };
  // Without a counter every CTA has one item, the highest query tiles - those of the longest sequences - first; most may be empty.
  const bool dealt = counter == nullptr;
  const unsigned pairs = (unsigned)B * (unsigned)H;
  if (dealt) {
    const int b = (int)(blockIdx.x % pairs) / H;
    if ((tiles - 1 - (int)(blockIdx.x / pairs)) * kTile >= offsets[b + 1] - offsets[b]) {          // uniform for the CTA, before any barrier or allocation
      if (warp == kProducer) clear_uncovered();
      return;
    }
  }
  if (threadIdx.x == 0) {
    abort_flag = 0;
    mbar_init(&q_full[0], 1); mbar_init(&q_full[1], 1); mbar_init(&k_full, 1); mbar_init(&v_full, 1);
    mbar_init(&s_full, 1); mbar_init(&o_full, 1);
    mbar_init(&p_full, 4); mbar_init(&o_empty, 4);
    mbar_fence_init();
  }
  if (warp == kMma) tmem_alloc(&tmem_slot, kFwdTmemCols);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = tmem_slot;
  auto wait_all = [&](uint64_t* bar, uint32_t parity) -> bool {               // one outcome for the whole warp
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, &abort_flag) ? 1 : 0) != 0;
  };

  if (warp >= kProducer) {
    if (warp == kProducer) {
      // ------------------------------------------------------------------ work fetch + TMA producer
      const unsigned total = (unsigned)tiles * (unsigned)B * (unsigned)H;
      // With a counter the first items are dealt out and the others fetched; the tiles of a sequence are neighbours, so that its keys are
      // read from L2.
      unsigned next = blockIdx.x * (unsigned)chunk;
      int it = 0, g = 0;
      bool ok = true;
      // `rows` rows of 64 columns from row `row`: whole tiles as one box, shorter ones in boxes of 32 rows (what lies behind is not read, or
      // only by rows and columns that are masked or not stored)
      auto load = [&](uint8_t* dst, int x, int row, int rows, uint64_t* bar) {
        if (rows > kTile - 32) tma_load_2d(dst, &map_qkv, x, row, bar);
        else for (int i = 0; i * 32 < rows; ++i) tma_load_2d(dst + i * 4096, &map_rows, x, row + i * 32, bar);
      };
      while (ok) {
        const unsigned base = __shfl_sync(0xffffffffu, next, 0);
        if (base >= total) break;
        if (dealt) next = total;
        else if (lane == 0) next = (gridDim.x + atomicAdd(counter, 1u)) * (unsigned)chunk;        // needed only after these items: its latency is hidden
        AttnItem mine{0, 0, 0, 0};
        const unsigned idx = base + (unsigned)lane;
        bool have = lane < chunk && idx < total;
        if (have) {
          const unsigned bh = dealt ? idx % pairs : idx / (unsigned)tiles;
          const int b = (int)(bh / (unsigned)H);
          mine.kt = dealt ? tiles - 1 - (int)(idx / pairs) : (int)(idx - bh * (unsigned)tiles);
          mine.head = (int)(bh - (unsigned)b * (unsigned)H);
          mine.s0 = offsets[b];
          mine.len = offsets[b + 1] - mine.s0;
          have = mine.kt * kTile < mine.len;
        }
        unsigned todo = __ballot_sync(0xffffffffu, have);
        while (todo && ok) {
          const int src = __ffs(todo) - 1;
          todo &= todo - 1;
          AttnItem item;
          item.s0 = __shfl_sync(0xffffffffu, mine.s0, src); item.len = __shfl_sync(0xffffffffu, mine.len, src);
          item.head = __shfl_sync(0xffffffffu, mine.head, src); item.kt = __shfl_sync(0xffffffffu, mine.kt, src);
          if (lane == 0) {
            const int xq = item.head * kHead, xk = (H + item.head) * kHead, xv = (2 * H + item.head) * kHead;
            // A buffer is free when the MMAs that read it are complete: Q and K with S, V with P V of the step before.
            for (int j = 0; j * kTile < item.len; ++j, ++g) {
              const int rows = min(kTile, item.len - j * kTile);
              ok = g == 0 || mbar_wait(&s_full, (uint32_t)((g - 1) & 1), &abort_flag);
              if (!ok) break;
              if (j == 0) {
                const int q_rows = min(kTile, item.len - item.kt * kTile);
                slot[it & 1] = item;
                mbar_expect_tx(&q_full[it & 1], (uint32_t)((q_rows + 31) & ~31) * 128u);
                load(qtile, xq, item.s0 + item.kt * kTile, q_rows, &q_full[it & 1]);
                ++it;
              }
              mbar_expect_tx(&k_full, (uint32_t)((rows + 31) & ~31) * 128u);
              load(ktile, xk, item.s0 + j * kTile, rows, &k_full);
              ok = g == 0 || mbar_wait(&o_full, (uint32_t)((g - 1) & 1), &abort_flag);
              if (!ok) break;
              mbar_expect_tx(&v_full, (uint32_t)((rows + 31) & ~31) * 128u);
              load(vtile, xv, item.s0 + j * kTile, rows, &v_full);
            }
          }
          ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
        }
      }
      if (lane == 0 && ok && (g == 0 || mbar_wait(&s_full, (uint32_t)((g - 1) & 1), &abort_flag))) {
        slot[it & 1] = AttnItem{0, -1, 0, 0};
        mbar_arrive(&q_full[it & 1]);
      }
      clear_uncovered();
    } else {
      // ------------------------------------------------------------------ MMA issuer (the whole warp; one lane issues)
      // Descriptors advance by adding to the 16-byte address field.
      const uint64_t d_q = make_desc(smem_u32(qtile), 16, 1024), d_k = make_desc(smem_u32(ktile), 16, 1024);
      const uint64_t d_p = make_desc(smem_u32(ptile), 16, 1024), d_v = make_desc(smem_u32(vtile), kBlk, 1024);
      const uint32_t idesc_o = make_idesc_bf16(kTile, kHead, false, true);
      const bool leader = elect_one();
      int g = 0;
      bool ok = true;
      auto issue_s = [&](int keys) {                     // S of a step whose tiles have landed
        fence_after_sync();
        const uint32_t idesc_s = make_idesc_bf16(kTile, (keys + 15) & ~15, false, false);
        if (leader) {
#pragma unroll
          for (int k = 0; k < kHead / 16; ++k) umma_bf16(tmem + kFwdS, d_q + (uint64_t)(k * 2), d_k + (uint64_t)(k * 2), idesc_s, k > 0 ? 1u : 0u);
          umma_commit(&s_full);
        }
        __syncwarp();
      };
      for (int it = 0; ok; ++it) {
        ok = wait_all(&q_full[it & 1], (uint32_t)((it >> 1) & 1));
        if (!ok) break;
        const int len = __shfl_sync(0xffffffffu, slot[it & 1].len, 0);
        if (len < 0) break;
        ok = wait_all(&k_full, (uint32_t)(g & 1));
        if (!ok) break;
        issue_s(min(kTile, len));
        for (int j = 0; j * kTile < len; ++j, ++g) {
          const int left = len - j * kTile, steps = (min(kTile, left) + 15) >> 4;      // of 16 keys
          // everything else is waited for before P, which comes last: between P and the next S lies only their issue
          ok = wait_all(&v_full, (uint32_t)(g & 1)) && (j > 0 || it == 0 || wait_all(&o_empty, (uint32_t)((it - 1) & 1))) &&
               (left <= kTile || wait_all(&k_full, (uint32_t)((g + 1) & 1))) && wait_all(&p_full, (uint32_t)(g & 1));
          if (!ok) break;
          if (left > kTile) issue_s(min(kTile, left - kTile));                         // (S of this step has been read)
          else fence_after_sync();
          if (leader) {
            umma_bf16(tmem + kFwdO, d_p, d_v, idesc_o, 0u);
            if (steps == kTile / 16) {
#pragma unroll
              for (int k = 1; k < kTile / 16; ++k) umma_bf16(tmem + kFwdO, d_p + (uint64_t)((k >> 2) * (kBlk >> 4) + (k & 3) * 2), d_v + (uint64_t)(k * 128), idesc_o, 1u);
            } else {
#pragma unroll 1
              for (int k = 1; k < steps; ++k) umma_bf16(tmem + kFwdO, d_p + (uint64_t)((k >> 2) * (kBlk >> 4) + (k & 3) * 2), d_v + (uint64_t)(k * 128), idesc_o, 1u);
            }
            umma_commit(&o_full);
          }
          __syncwarp();
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax: thread = query row
    const int row = warp * 32 + lane;
    const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
    const uint32_t box = smem_u32(ptile) + (uint32_t)(warp * 4096), prow = box + (uint32_t)(lane * 128 + ((lane & 7) << 4));     // (with the row's swizzle)
    int g = 0;
    bool ok = true;
    for (int it = 0; ok; ++it) {
      ok = wait_all(&q_full[it & 1], (uint32_t)((it >> 1) & 1));
      if (!ok) break;
      const AttnItem item = slot[it & 1];
      if (item.len < 0) break;
      const int rows = item.len - item.kt * kTile - warp * 32;                // rows of this warp that exist (may be <= 0, or more than 32)
      float m = -INFINITY, l = 0.f, alpha = 0.f;                              // maximum so far (in powers of two), sum of P, the last step's rescale
      float o[kHead];                                                         // the row of O: each step's P V is added to it
#pragma unroll
      for (int d = 0; d < kHead; ++d) o[d] = 0.f;
      auto add_pv = [&]() {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          uint32_t r[32];
          tmem_ld32(trow + kFwdO + (uint32_t)(e * 32), r);
          tmem_ld_wait();
#pragma unroll
          for (int d = 0; d < 32; ++d) o[e * 32 + d] = fmaf(o[e * 32 + d], alpha, __uint_as_float(r[d]));
        }
      };
      for (int j = 0; j * kTile < item.len; ++j, ++g) {
        const int valid = min(kTile, item.len - j * kTile);                   // key columns of this step that exist
        ok = wait_all(&s_full, (uint32_t)(g & 1));
        if (!ok) break;
        fence_after_sync();
        if (rows > 0) {                                                       // (otherwise P of this warp only reaches rows that are not stored)
          // Read twice, for the maximum and for P, 32 columns at a time in rolled loops, and 8 at a time behind the last whole 32: only columns
          // that hold a key or complete a 16-key step, and code that stays in the instruction cache (spelt out for a whole row, waiting for
          // instructions was the largest stall). A masked key is -inf in the maximum and an exact zero in P.
          const int whole = valid & ~31, end = (valid + 15) & ~15;
          float m_new = m;
#pragma unroll 1
          for (int c = 0; c < whole; c += 32) {
            uint32_t s[32];
            tmem_ld32(trow + kFwdS + (uint32_t)c, s);
            tmem_ld_wait();
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int i = 0; i < 32; i += 8)
#pragma unroll
              for (int e = 0; e < 4; ++e) mx[e] = fmaxf(fmaxf(mx[e], __uint_as_float(s[i + e])), __uint_as_float(s[i + 4 + e]));
            m_new = fmaxf(m_new, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * scale_log2);
          }
#pragma unroll 1
          for (int c = whole; c < valid; c += 8) {
            uint32_t s[8];
            tmem_ld8(trow + kFwdS + (uint32_t)c, s);
            tmem_ld_wait();
            float mx = -INFINITY;
#pragma unroll
            for (int i = 0; i < 8; ++i) mx = fmaxf(mx, c + i < valid ? __uint_as_float(s[i]) : -INFINITY);
            m_new = fmaxf(m_new, mx * scale_log2);
          }
          if (g > 0) {                                                        // P V of the step before has read P and is in O
            ok = wait_all(&o_full, (uint32_t)((g - 1) & 1));
            if (!ok) break;
          }
          if (j > 0) {
            fence_after_sync();
            add_pv();
            alpha = fast_exp2(m - m_new);
          }
          m = m_new;
          const float neg_m = -m;
          float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
          for (int c = 0; c < whole; c += 32) {
            uint32_t s[32], pk[16];
            tmem_ld32(trow + kFwdS + (uint32_t)c, s);
            tmem_ld_wait();
            exp_chunk<32>(s, scale_log2, neg_m, sum, pk);
#pragma unroll
            for (int e = 0; e < 4; ++e)
              st_shared16((prow ^ (uint32_t)((((c >> 3) & 4) + e) << 4)) + (uint32_t)((c >> 6) * kBlk), pk[4 * e], pk[4 * e + 1], pk[4 * e + 2], pk[4 * e + 3]);
          }
#pragma unroll 1
          for (int c = whole; c < end; c += 8) {
            uint32_t s[8], pk[4];
            tmem_ld8(trow + kFwdS + (uint32_t)c, s);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 8; ++i) s[i] = c + i < valid ? s[i] : 0xff800000u;
            exp_chunk<8>(s, scale_log2, neg_m, sum, pk);
            st_shared16((prow ^ (uint32_t)(((c >> 3) & 7) << 4)) + (uint32_t)((c >> 6) * kBlk), pk[0], pk[1], pk[2], pk[3]);
          }
          l = fmaf(l, alpha, (sum[0] + sum[2]) + (sum[1] + sum[3]));
        }
        if (valid & 15) {
          // V rows between the last key and the end of the last 16-key step become zeros, so that the zeros of P never meet a non-finite value
          ok = wait_all(&v_full, (uint32_t)(g & 1));
          if (!ok) break;
          if (row >= valid && row < ((valid + 15) & ~15)) {
#pragma unroll
            for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4*>(vtile + swizzle128_offset(row, c * 8)) = make_uint4(0u, 0u, 0u, 0u);
          }
        }
        fence_smem_to_async();
        fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full);
      }
      if (!ok) break;
      // ---- the item's O. A warp without rows has not waited for the products before the last one, and where the last but one still runs, this wait
      // passes on the phase before that, which has the same parity. Such a warp reads nothing of O, and what it then arrives on, o_empty, is the
      // phase of this item all the same: the second S of an item is multiplied only after the o_empty of the item before is complete, and
      // the first S of the next item only after this item's last product is issued. The hand-back itself waits for warp 0, which always has
      // rows. (Following every phase cost 17.0 -> 18.2 us at 590 sequences of 1..40 tokens, 2 heads.)
      ok = wait_all(&o_full, (uint32_t)((g - 1) & 1));
      if (!ok) break;
      fence_after_sync();
      // through this warp's rows of the P tile, which the item no longer needs: eight lanes store a row, so that every store is whole lines
      const float inv = l > 0.f ? 1.f / l : 0.f;
      if (rows > 0) {
        add_pv();
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint32_t u[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) u[e] = pack_bf16x2(o[c * 8 + 2 * e] * inv, o[c * 8 + 2 * e + 1] * inv);
          st_shared16(prow ^ (uint32_t)(c << 4), u[0], u[1], u[2], u[3]);
        }
      }
      fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&o_empty);
      if (rows > 0) {
        const int64_t first = (int64_t)item.s0 + item.kt * kTile + warp * 32;
        if (lse2 && lane < rows) lse2[(first + lane) * H + item.head] = m + log2f(l);
        __syncwarp();
        __nv_bfloat16* dst = out + (first * H + item.head) * kHead;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = i * 4 + (lane >> 3);
          if (r < rows) {
            uint4 u;
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w)
                         : "r"(box + (uint32_t)(r * 128) + (uint32_t)(((lane & 7) ^ (r & 7)) << 4)) : "memory");
            reinterpret_cast<uint4*>(dst + (int64_t)r * H * kHead)[lane & 7] = u;
          }
        }
        __syncwarp();                                                         // read before the next item's P is written
      }
    }
  }
  if (abort_flag) {
    // a wait ran out: a tile may still be on its way into shared memory; give it time before the memory goes away
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  fence_before_sync();
  __syncthreads();
  if (warp == kMma) { fence_after_sync(); tmem_dealloc(tmem, kFwdTmemCols); }
  if (threadIdx.x == 0 && abort_flag) rb::set_status(status, rb::kStatusWaitTimeout);
}

// ---------------------------------------------------------------------------------------------- backward
// delta[t, h] = sum_d dO[t, h, d] * O[t, h, d] (the row-wise correction term of the softmax backward): eight lanes per (t, h), one
// 16-byte load of each operand per lane. The pass also zeroes what the main kernel needs zeroed: its work counter, and the
// gradient rows of tokens that belong to no sequence (in front of offsets[0] or behind offsets[B]).
__global__ void __launch_bounds__(256)
attention_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o, int64_t T, int H, int B,
                       const int32_t* __restrict__ offsets, float* __restrict__ delta, unsigned* __restrict__ counter,
                       __nv_bfloat16* __restrict__ dqkv) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *counter = 0u;
  const int sub = threadIdx.x & 7;
  const int64_t rows = T * H, step = (int64_t)gridDim.x * 32;
  const int t_first = offsets[0], t_last = offsets[B];
  for (int64_t r0 = (int64_t)blockIdx.x * 32; r0 < rows; r0 += step) {          // 32 rows per block and pass: uniform trip count
    const int64_t r = r0 + (threadIdx.x >> 3);
    float v = 0.f;
    if (r < rows) {
      const uint4 a = reinterpret_cast<const uint4*>(o + r * kHead)[sub];
      const uint4 b = reinterpret_cast<const uint4*>(d_o + r * kHead)[sub];
      const __nv_bfloat162* ap = reinterpret_cast<const __nv_bfloat162*>(&a);
      const __nv_bfloat162* bp = reinterpret_cast<const __nv_bfloat162*>(&b);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 x = __bfloat1622float2(ap[j]), y = __bfloat1622float2(bp[j]);
        v = fmaf(x.x, y.x, fmaf(x.y, y.y, v));
      }
    }
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if (r < rows) {
      if (sub == 0) delta[r] = v;
      const int64_t t = r / H;
      if (t < t_first || t >= t_last) {
        __nv_bfloat16* g = dqkv + t * 3 * H * kHead + (r - t * H) * kHead + sub * 8;
#pragma unroll
        for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(g + (int64_t)p * H * kHead) = make_uint4(0u, 0u, 0u, 0u);
      }
    }
  }
}

// dq_acc fp32 [T, H * 64] -> the q part of dqkv (bf16); eight columns per thread.
__global__ void __launch_bounds__(256)
attention_dq_store_kernel(const float* __restrict__ dq_acc, int64_t T, int cols, __nv_bfloat16* __restrict__ dqkv) {
  const int per_row = cols >> 3;
  const int64_t total = T * per_row;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = i / per_row;
    const int c = (int)(i - t * per_row) * 8;
    const float4 a = *reinterpret_cast<const float4*>(dq_acc + t * cols + c), b = *reinterpret_cast<const float4*>(dq_acc + t * cols + c + 4);
    *reinterpret_cast<uint4*>(dqkv + t * 3 * cols + c) =
        make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w));
  }
}

// A work item is one (sequence, head, 128-key tile); it walks the sequence's queries in tiles of 128. Per query tile:
//   S  = Q K^T, dP = dO V^T                          (two MMA chains, 128 x 128 x 64 each, results in tensor memory)
//   P  = exp2(S * scale * log2 e - lse2[q]),  dS = P * (dP - delta[q]) * scale        (written to shared memory as bf16 tiles [q][key])
//   dV += P^T dO, dK += dS^T Q                       (the [q][key] tiles read as MN-major A operands, dO / Q as MN-major B;
//                                                     accumulated in tensor memory over all query tiles)
//   dQ  = dS K                                       (the dS tile read as a K-major A operand, K as an MN-major B)
//
// One persistent CTA per SM with separate roles: warps 0..7 compute (two threads per query row, each with two of the four chunks of 32
// key columns), warp 8 fetches work and issues the TMA loads, warp 9 issues the MMAs. Work items come from a counter, so that sequences of very different length balance; K / V and Q / dO are double buffered across items, so the loads of the
// next item run under this one. The S and dP of step g + 1 are multiplied as soon as step g has them in registers, and the three
// products of step g - 1 run while step g computes its exponentials. No unit is near its limit (256 sequences of 50..1000 tokens, 4 heads:
// tensor pipe 26 %, L1 and shared memory 33 %, special-function units 19 %, issue slots 36 %): what bounds it is the chain load -> S, dP ->
// exponentials -> products -> results of a step, with eight compute warps on an SM to cover it.
// Parts of a tile that lie outside the sequence cost nothing: chunks of columns and warps of rows without an existing element are
// neither computed nor written, and the reductions stop at the last 16 rows that hold one. (Left-over values in unwritten parts only
// reach rows of the results that are not stored.)
//
// kSingle: the caller's bound on the length is at most 128, so every query that the forward computed is in one tile: dQ leaves as bf16
// from the registers. Otherwise dQ is added to an fp32 buffer with TMA add-reductions (other key tiles add theirs) and converted by
// attention_dq_store_kernel.
//
// A sequence may be longer than the bound. The forward then computes the queries in the `tiles` tiles of the bound, over all keys, and
// leaves zeros for the others. The same queries are walked here, for all key tiles (those past the bound belong to the item of the key tile
// `tiles` below); the others get a zero dQ. With kSingle that is query tile 0 with one key tile after the other, whose dQ add up in
// tensor memory until the last of them.
//
// Measured on a B200 with cold L2 (this kernel alone; before: one CTA of 128 threads per item, loads / MMAs / exponentials one after the other; in
// brackets with the MMAs issued from a branch of one lane):
//   256 sequences of 50..1000 tokens, 4 heads:  807 -> 489 us (528; 232 GFLOP in existing elements: 475 TFLOP/s)
//   3000 sequences of 1..90 tokens, 8 heads:   1288 -> 385 us (405; 0.84 GB read and written: 2.2 TB/s; fixed cost per item)
// and no zeroed fp32 gradient of q, k and v (413 MB resp. 826 MB of it) nor its conversion to bf16 around it any more.
constexpr uint32_t kColS = 0, kColDP = 128, kColDV = 256, kColDK = 320, kColDQ = 384;
constexpr int kBwdCompute = 8;                       // compute warps
constexpr int kBwdThreads = (kBwdCompute + 4) * 32;  // and one warpgroup of control warps, two of them idle (register split below)
// Work items fetched at a time: four where an item is one step and a fetch would not hide behind it, one where items are up to many steps
// long and a group of four made some SMs finish a sixth later than the rest (256 sequences of 50..1000 tokens, before the MMA warp ran converged:
// 585 -> 523 us). Which of the two is chosen by the caller's bound. Under a loose bound most items are empty and a single fetch costs more
// (3000 sequences of 1..90 tokens, 8 heads: 385 us under a bound of 90, 1191 under 1000).
constexpr int kBwdChunkShort = 4, kBwdChunkLong = 1;

// N key columns of one query row: pk = bf16 pairs of P, dk = bf16 pairs of dS. kMask: columns >= valid give exact zeros (S and dP
// of rows and keys that do not exist can be anything, so both results are selected, not multiplied to zero).
template <bool kMask, int N>
__device__ __forceinline__ void p_ds_chunk(const uint32_t (&rs)[N], const uint32_t (&rp)[N], int c0, int valid, float scale, float scale_log2,
                                           float lse_q, float nds, uint32_t (&pk)[N / 2], uint32_t (&dk)[N / 2]) {
#pragma unroll
  for (int e = 0; e < N / 2; ++e) {
    float p[2], ds[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      p[u] = fast_exp2(fmaf(__uint_as_float(rs[2 * e + u]), scale_log2, -lse_q));
      ds[u] = p[u] * fmaf(__uint_as_float(rp[2 * e + u]), scale, nds);
      if (kMask && c0 + 2 * e + u >= valid) { p[u] = 0.f; ds[u] = 0.f; }
    }
    pk[e] = pack_bf16x2(p[0], p[1]);
    dk[e] = pack_bf16x2(ds[0], ds[1]);
  }
}

// 32 columns (16 registers of bf16 pairs) of one row, starting at 16-byte column c16 (0 or 4) of the tile at byte `tile`
__device__ __forceinline__ void store_chunk(uint32_t rowbase, uint32_t tile, int c16, const uint32_t (&v)[16]) {
#pragma unroll
  for (int cq = 0; cq < 4; ++cq) st_shared16((rowbase ^ (uint32_t)((c16 + cq) << 4)) + tile, v[cq * 4], v[cq * 4 + 1], v[cq * 4 + 2], v[cq * 4 + 3]);
}

__device__ __forceinline__ void zero_half_row(uint32_t rowbase, uint32_t tile, int half) {
#pragma unroll
  for (int c = 0; c < 4; ++c) st_shared16((rowbase ^ (uint32_t)((half * 4 + c) << 4)) + tile, 0u, 0u, 0u, 0u);
}

template <bool kSingle>
__global__ void __launch_bounds__(kBwdThreads, 1)
ragged_attention_bwd_kernel(const __grid_constant__ CUtensorMap map_qkv, const __grid_constant__ CUtensorMap map_do,
                            const float* __restrict__ lse2, const float* __restrict__ delta, const int32_t* __restrict__ offsets, int B, int H,
                            int tiles, float scale, float scale_log2, __nv_bfloat16* __restrict__ dqkv, const __grid_constant__ CUtensorMap map_dq,
                            unsigned* __restrict__ counter, int64_t* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t kv_full[2], kv_empty[2], in_full[2], in_empty[2];
  __shared__ __align__(8) uint64_t s_full, s_empty, p_full, m2_full, post_empty;
  __shared__ AttnItem slot[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* kvtiles = smem;                 // 2 x (K [128 keys][64 d], V)
  uint8_t* qotiles = smem + 4 * kBlk;      // 2 x (Q [128 q][64 d], dO)
  uint8_t* ptile = smem + 8 * kBlk;        // 2 x [128 q][64 keys]
  uint8_t* dstile = smem + 10 * kBlk;      // 2 x [128 q][64 keys]
  uint8_t* outstage = smem + 12 * kBlk;    // 4 KB per compute warp: results on their way out
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kProducer = kBwdCompute, kMma = kProducer + 1;
  constexpr int kChunk = kSingle ? kBwdChunkShort : kBwdChunkLong;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < 2; ++s) {
      mbar_init(&kv_full[s], 1);
      mbar_init(&kv_empty[s], 1); mbar_init(&in_full[s], 1); mbar_init(&in_empty[s], 1);
    }
    mbar_init(&s_full, 1); mbar_init(&m2_full, 1);
    mbar_init(&s_empty, kBwdCompute); mbar_init(&p_full, kBwdCompute); mbar_init(&post_empty, kBwdCompute);
    mbar_fence_init();
  }
  if (warp == kMma) tmem_alloc(&tmem_slot, 512);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = tmem_slot;
  auto query_tiles = [&](int len) { return kSingle ? 1 : min((len + kTile - 1) / kTile, tiles); };        // as many as the forward computed
  auto wait_all = [&](uint64_t* bar, uint32_t parity) -> bool {               // one outcome for the whole warp
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, &abort_flag) ? 1 : 0) != 0;
  };

  // 12 warps launch with 168 registers a thread, 64512 in all: 256 x 232 + 128 x 40 = 64512
  if (warp >= kProducer) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == kProducer) {
      // ------------------------------------------------------------------ work fetch + TMA producer
      const unsigned total = (unsigned)tiles * (unsigned)B * (unsigned)H;
      unsigned next = 0;
      if (lane == 0) next = atomicAdd(counter, (unsigned)kChunk);
      int it = 0, g = 0;
      bool ok = true;
      while (ok) {
        const unsigned base = __shfl_sync(0xffffffffu, next, 0);
        if (base >= total) break;
        if (lane == 0) next = atomicAdd(counter, (unsigned)kChunk);       // needed only after these items: its latency is hidden
        AttnItem mine{0, 0, 0, 0};
        const unsigned idx = base + (unsigned)lane;
        bool have = lane < kChunk && idx < total;
        if (have) {
          const unsigned bh = idx / (unsigned)tiles;
          const int b = (int)(bh / (unsigned)H);
          mine.kt = (int)(idx - bh * (unsigned)tiles);
          mine.head = (int)(bh - (unsigned)b * (unsigned)H);
          mine.s0 = offsets[b];
          mine.len = offsets[b + 1] - mine.s0;
          have = mine.kt * kTile < mine.len;
        }
        unsigned todo = __ballot_sync(0xffffffffu, have);
        while (todo && ok) {
          const int src = __ffs(todo) - 1;
          todo &= todo - 1;
          AttnItem item;
          item.s0 = __shfl_sync(0xffffffffu, mine.s0, src); item.len = __shfl_sync(0xffffffffu, mine.len, src);
          item.head = __shfl_sync(0xffffffffu, mine.head, src); item.kt = __shfl_sync(0xffffffffu, mine.kt, src);
          if (lane == 0) {
            const int xq = item.head * kHead, xk = (H + item.head) * kHead, xv = (2 * H + item.head) * kHead;
            // (this item also takes the key tiles past the caller's bound)
            for (; item.kt * kTile < item.len && ok; item.kt += tiles, ++it) {
              const int st = it & 1;
              ok = mbar_wait(&kv_empty[st], (uint32_t)((it >> 1) & 1) ^ 1u, &abort_flag);
              if (!ok) break;
              slot[st] = item;
              mbar_expect_tx(&kv_full[st], 2 * kBlk);
              tma_load_2d(kvtiles + st * 2 * kBlk, &map_qkv, xk, item.s0 + item.kt * kTile, &kv_full[st]);
              tma_load_2d(kvtiles + st * 2 * kBlk + kBlk, &map_qkv, xv, item.s0 + item.kt * kTile, &kv_full[st]);
              const int n_q = query_tiles(item.len);
              for (int i = 0; i < n_q && ok; ++i, ++g) {
                const int buf = g & 1;
                ok = mbar_wait(&in_empty[buf], (uint32_t)((g >> 1) & 1) ^ 1u, &abort_flag);
                if (!ok) break;
                const int row0 = item.s0 + i * kTile;
                mbar_expect_tx(&in_full[buf], 2 * kBlk);
                tma_load_2d(qotiles + buf * 2 * kBlk, &map_qkv, xq, row0, &in_full[buf]);
                tma_load_2d(qotiles + buf * 2 * kBlk + kBlk, &map_do, xq, row0, &in_full[buf]);
              }
            }
          }
          ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
        }
      }
      if (lane == 0 && ok) {
        const int st = it & 1;
        if (mbar_wait(&kv_empty[st], (uint32_t)((it >> 1) & 1) ^ 1u, &abort_flag)) {
          slot[st] = AttnItem{0, -1, 0, 0};
          mbar_arrive(&kv_full[st]);
        }
      }
    } else if (warp == kMma) {
      // ------------------------------------------------------------------ MMA issuer (the whole warp; one lane issues)
      const uint32_t idesc_kk = make_idesc_bf16(kTile, kTile, false, false);    // S, dP: both operands K-major
      const uint32_t idesc_mm = make_idesc_bf16(kTile, kHead, true, true);      // dV, dK: both operands MN-major
      const uint32_t idesc_km = make_idesc_bf16(kTile, kHead, false, true);     // dQ: A K-major, B MN-major
      // Descriptors advance by adding to the 16-byte address field: they stay in a few registers.
      // A = P^T / dS^T: [q][key] tiles read MN-major (M = key: two 64-wide blocks kBlk apart, 16 q rows = 2048 bytes per step)
      // B = dO / Q:     [q][d] tiles read MN-major (N = d, one 64-wide block)
      const uint64_t d_qk = make_desc(smem_u32(qotiles), 16, 1024), d_kk = make_desc(smem_u32(kvtiles), 16, 1024);      // read K-major
      const uint64_t d_qm = make_desc(smem_u32(qotiles), kBlk, 1024), d_km = make_desc(smem_u32(kvtiles), kBlk, 1024);  // read MN-major
      const uint64_t d_p = make_desc(smem_u32(ptile), kBlk, 1024), d_ds = make_desc(smem_u32(dstile), kBlk, 1024), d_dsk = make_desc(smem_u32(dstile), 16, 1024);
      const bool leader = elect_one();
      int g = 0;
      int p_st = 0, p_kq = 0, p_kk = 0;                 // the previous step: K / V stage, 16-row reduction steps over queries and keys
      bool p_first = false, p_last = false, p_dq_acc = false;
      auto products = [&](int gs) -> bool {             // dV, dK, dQ of step gs
        if (gs > 0 && !wait_all(&post_empty, (uint32_t)((gs - 1) & 1))) return false;
        if (!wait_all(&p_full, (uint32_t)(gs & 1))) return false;
        fence_after_sync();
        const uint64_t q = d_qm + (uint64_t)((gs & 1) * (2 * kBlk >> 4)), d_o = q + (uint64_t)(kBlk >> 4), kt = d_km + (uint64_t)(p_st * (2 * kBlk >> 4));
        const uint32_t acc = p_first ? 0u : 1u, acc_q = p_dq_acc ? 1u : 0u;
        if (leader) {
          if (p_kq == kTile / 16) {                     // (a whole tile is spelt out: built in a loop, the 24 MMAs took 2400 cycles to issue)
#pragma unroll
            for (int k = 0; k < kTile / 16; ++k) {      // reduction over the queries of the tile, 16 rows per step
              umma_bf16(tmem + kColDV, d_p + (uint64_t)(k * 128), d_o + (uint64_t)(k * 128), idesc_mm, k > 0 ? 1u : acc);
              umma_bf16(tmem + kColDK, d_ds + (uint64_t)(k * 128), q + (uint64_t)(k * 128), idesc_mm, k > 0 ? 1u : acc);
            }
          } else {
#pragma unroll 1
            for (int k = 0; k < p_kq; ++k) {
              umma_bf16(tmem + kColDV, d_p + (uint64_t)(k * 128), d_o + (uint64_t)(k * 128), idesc_mm, k > 0 ? 1u : acc);
              umma_bf16(tmem + kColDK, d_ds + (uint64_t)(k * 128), q + (uint64_t)(k * 128), idesc_mm, k > 0 ? 1u : acc);
            }
          }
          if (p_kk == kTile / 16) {
#pragma unroll
            for (int k = 0; k < kTile / 16; ++k)        // reduction over the keys of the tile: dS read K-major, K read MN-major
              umma_bf16(tmem + kColDQ, d_dsk + (uint64_t)((k >> 2) * (kBlk >> 4) + (k & 3) * 2), kt + (uint64_t)(k * 128), idesc_km, k > 0 ? 1u : acc_q);
          } else {
#pragma unroll 1
            for (int k = 0; k < p_kk; ++k)
              umma_bf16(tmem + kColDQ, d_dsk + (uint64_t)((k >> 2) * (kBlk >> 4) + (k & 3) * 2), kt + (uint64_t)(k * 128), idesc_km, k > 0 ? 1u : acc_q);
          }
          umma_commit(&m2_full);
          umma_commit(&in_empty[gs & 1]);
          if (p_last) umma_commit(&kv_empty[p_st]);
        }
        __syncwarp();
        return true;
      };
      bool ok = true;
      for (int it = 0; ok; ++it) {
        const int st = it & 1;
        ok = wait_all(&kv_full[st], (uint32_t)((it >> 1) & 1));
        if (!ok) break;
        const int len = __shfl_sync(0xffffffffu, slot[st].len, 0), kt0 = __shfl_sync(0xffffffffu, slot[st].kt, 0);
        if (len < 0) break;
        const uint64_t d_k = d_kk + (uint64_t)(st * (2 * kBlk >> 4));
        const int n_q = query_tiles(len);
        for (int i = 0; i < n_q; ++i, ++g) {
          ok = wait_all(&in_full[g & 1], (uint32_t)((g >> 1) & 1)) && (g == 0 || wait_all(&s_empty, (uint32_t)((g - 1) & 1)));
          if (!ok) break;
          fence_after_sync();
          const uint64_t d_q = d_qk + (uint64_t)((g & 1) * (2 * kBlk >> 4));
          if (leader) {
#pragma unroll
            for (int k = 0; k < kHead / 16; ++k)
              umma_bf16(tmem + kColS, d_q + (uint64_t)(k * 2), d_k + (uint64_t)(k * 2), idesc_kk, k > 0 ? 1u : 0u);
#pragma unroll
            for (int k = 0; k < kHead / 16; ++k)         // dP = dO V^T: dO and V lie one block behind Q and K
              umma_bf16(tmem + kColDP, d_q + (uint64_t)((kBlk >> 4) + k * 2), d_k + (uint64_t)((kBlk >> 4) + k * 2), idesc_kk, k > 0 ? 1u : 0u);
            umma_commit(&s_full);
          }
          __syncwarp();
          if (g > 0) { ok = products(g - 1); if (!ok) break; }
          p_st = st; p_first = i == 0; p_last = i == n_q - 1; p_dq_acc = kSingle && kt0 > 0;
          p_kq = (min(kTile, len - i * kTile) + 15) >> 4;
          p_kk = (min(kTile, len - kt0 * kTile) + 15) >> 4;
        }
      }
      if (ok && g > 0) products(g - 1);
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
    // ------------------------------------------------------------------ compute: thread = (query row, two chunks of 32 key columns)
    const int quarter = warp & 3, half = warp >> 2;
    const int row = quarter * 32 + lane;
    const uint32_t trow = tmem + ((uint32_t)(quarter * 32) << 16);
    const int64_t ld = (int64_t)3 * H * kHead;
    const uint32_t rowbase = smem_u32(smem) + (uint32_t)((row >> 3) * 1024 + (row & 7) * 128 + ((row & 7) << 4));
    const uint32_t box = smem_u32(outstage) + (uint32_t)(warp * 4096);
    // The step whose products are still running: where its dQ goes, and (after the last step of an item) its keys. Row counts are
    // those of this warp's 32 rows and may be <= 0. A warp takes 32 of the 64 columns of each result.
    int p_row0 = 0, p_vq = 0, p_head = 0, p_key0 = 0, p_vk = 0;
    bool p_last = false, p_zero_q = false;                // p_zero_q: the key rows are no query rows of this pass (kSingle past the first tile)
    // 32 bf16 columns of the warp's first `valid` rows to global memory through a 2 KB corner of its box, four lanes per row and
    // eight rows per store instruction (a thread per row would touch 32 lines with each).
    auto stage16 = [&](uint32_t at, const uint32_t (&r)[32]) {
#pragma unroll
      for (int c = 0; c < 4; ++c)
        st_shared16(at + (uint32_t)(lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)), pack_bf16x2(__uint_as_float(r[c * 8]), __uint_as_float(r[c * 8 + 1])),
                    pack_bf16x2(__uint_as_float(r[c * 8 + 2]), __uint_as_float(r[c * 8 + 3])),
                    pack_bf16x2(__uint_as_float(r[c * 8 + 4]), __uint_as_float(r[c * 8 + 5])),
                    pack_bf16x2(__uint_as_float(r[c * 8 + 6]), __uint_as_float(r[c * 8 + 7])));
    };
    auto copy_out = [&](uint32_t at, __nv_bfloat16* dst, int valid) {
      const int c = lane & 3;
#pragma unroll 1
      for (int r = lane >> 2; r < 32; r += 8) {
        if (r < valid) {
          uint4 v;
          asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                       : "r"(at + (uint32_t)(r * 64 + ((c ^ ((r >> 1) & 3)) << 4))) : "memory");
          reinterpret_cast<uint4*>(dst + (int64_t)r * ld)[c] = v;
        }
      }
    };
    // everything the previous step left in tensor memory (its products are complete)
    auto post = [&]() {
      const bool kv = p_last && p_vk > 0;
      uint32_t r[32];
      if (!kSingle && lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");     // the previous box has been read
      __syncwarp();
      if (kv) {
        tmem_ld32(trow + kColDK + (uint32_t)(half * 32), r);
        tmem_ld_wait();
        stage16(box, r);
        tmem_ld32(trow + kColDV + (uint32_t)(half * 32), r);
        tmem_ld_wait();
        stage16(box + 2048u, r);
      }
      if (p_vq > 0) { tmem_ld32(trow + kColDQ + (uint32_t)(half * 32), r); tmem_ld_wait(); }
      fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&post_empty);
      if (kv) {
        __nv_bfloat16* kdst = dqkv + (int64_t)p_key0 * ld + (H + p_head) * kHead + half * 32;
        copy_out(box, kdst, p_vk);
        copy_out(box + 2048u, kdst + H * kHead, p_vk);
        if (kSingle && p_zero_q)
          for (int row = lane >> 2; row < min(p_vk, 32); row += 8)
            reinterpret_cast<uint4*>(kdst - H * kHead + (int64_t)row * ld)[lane & 3] = make_uint4(0u, 0u, 0u, 0u);
        __syncwarp();
      }
      if (p_vq <= 0) return;
      if (kSingle) {
        stage16(box, r);
        __syncwarp();
        copy_out(box, dqkv + (int64_t)p_row0 * ld + p_head * kHead + half * 32, p_vq);
      } else {
        // Rows past the end of this sequence leave as exact zeros, so adding them onto the next sequence's rows changes nothing;
        // rows past the end of the buffer are clipped by the copy.
        const bool on = lane < p_vq;
#pragma unroll
        for (int e = 0; e < 8; ++e)
          st_shared16((box + (uint32_t)(lane * 128 + ((lane & 7) << 4))) ^ (uint32_t)(e << 4), on ? r[4 * e] : 0u, on ? r[4 * e + 1] : 0u,
                      on ? r[4 * e + 2] : 0u, on ? r[4 * e + 3] : 0u);
        fence_smem_to_async();
        __syncwarp();
        if (lane == 0) {
          asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.bulk_group [%0, {%2, %3}], [%1];"
                       ::"l"(&map_dq), "r"(box), "r"(p_head * kHead + half * 32), "r"(p_row0) : "memory");
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      }
    };
    // One flat loop over the steps of all items, so that every part of the body exists once: with one step per item each part runs
    // once per item on eight warps, and fetching instructions was what bounded the kernel while the body was spelt out (the largest
    // stall reason by far; 610 us against the 407 of then at 3000 sequences of up to 90 tokens x 8 heads).
    AttnItem item{0, 0, 0, 0};
    int it = 0, g = 0, i = 0, n_q = 0, valid_k = 0;
    float lse_next = 0.f, delta_next = 0.f;                                   // this row's lse and delta, fetched one step ahead
    bool ok = true, more = true;
    while (ok && more) {
      if (i == n_q) {
        const int st = it & 1;
        ok = wait_all(&kv_full[st], (uint32_t)((it >> 1) & 1));
        if (!ok) break;
        item = slot[st];
        ++it;
        i = 0;
        more = item.len >= 0;
        if (more) {
          n_q = query_tiles(item.len);
          valid_k = min(kTile, item.len - item.kt * kTile);
          if (row < item.len) {
            const int64_t at = (int64_t)(item.s0 + row) * H + item.head;
            lse_next = lse2[at];
            delta_next = delta[at];
          }
        }
      }
      const int q0 = i * kTile;
      const int valid_q = min(kTile, item.len - q0);
      if (more) {
        const int read_k = (valid_k + 15) & ~15;                              // keys that the reduction of dQ reads
        const int read_q = (valid_q + 15) & ~15;                              // queries that the reductions of dV and dK read
        const bool q_ok = row < valid_q;
        ok = wait_all(&s_full, (uint32_t)(g & 1));
        if (!ok) break;
        fence_after_sync();
        // Rows past the end of the sequence belong to the next one (or read as zeros past the end of the matrix). Those that the
        // reductions below read become zeros, so that the zeros of P and dS never meet a non-finite value. S and dP of this step are
        // complete, the next step's read other Q / dO buffers, and the K tile is not read again before s_empty.
        if (i == 0 && row >= valid_k && row < read_k) zero_half_row(rowbase, (uint32_t)(((it - 1) & 1) * 2 * kBlk), half);
        if (row >= valid_q && row < read_q) {
          zero_half_row(rowbase, (uint32_t)((4 + (g & 1) * 2) * kBlk), half);
          zero_half_row(rowbase, (uint32_t)((5 + (g & 1) * 2) * kBlk), half);
        }
        __syncwarp();                                                         // the zeros above are some lanes' work, tcgen05.ld the warp's
        const bool rows_on = quarter * 32 < valid_q, rows_full = quarter * 32 + 32 <= valid_q;      // uniform for the warp
        const float lse_q = lse_next, nds = -delta_next * scale;              // (dP - delta) * scale = dP * scale + nds
        if constexpr (kSingle) {
          // 16 columns at a time, written as they come: short sequences fill few of them
          if (g > 0) {
            ok = wait_all(&m2_full, (uint32_t)((g - 1) & 1));                 // P and dS of the previous step have been read
            if (!ok) break;
            fence_after_sync();
          }
          if (rows_on) {
#pragma unroll 1
            for (int u = half; u * 16 < valid_k; u += 2) {
              uint32_t rs[16], rd[16], pk[8], dk[8];
              tmem_ld16(trow + kColS + (uint32_t)(u * 16), rs);
              tmem_ld16(trow + kColDP + (uint32_t)(u * 16), rd);
              tmem_ld_wait();
              p_ds_chunk<true>(rs, rd, u * 16, q_ok ? valid_k : 0, scale, scale_log2, lse_q, nds, pk, dk);
              const uint32_t at = rowbase + (uint32_t)((8 + (u >> 2)) * kBlk), c0 = (uint32_t)(((u & 3) * 2) << 4), c1 = c0 + 16u;
              st_shared16(at ^ c0, pk[0], pk[1], pk[2], pk[3]);
              st_shared16(at ^ c1, pk[4], pk[5], pk[6], pk[7]);
              st_shared16((at ^ c0) + 2u * kBlk, dk[0], dk[1], dk[2], dk[3]);
              st_shared16((at ^ c1) + 2u * kBlk, dk[4], dk[5], dk[6], dk[7]);
            }
          }
          fence_smem_to_async();
          fence_before_sync();
          __syncwarp();
          if (lane == 0) { mbar_arrive(&p_full); mbar_arrive(&s_empty); }
        } else {
          if (i + 1 < n_q && q0 + kTile + row < item.len) {
            const int64_t at = (int64_t)(item.s0 + q0 + kTile + row) * H + item.head;
            lse_next = lse2[at];
            delta_next = delta[at];
          }
          if (valid_k < read_k || valid_q < read_q) fence_smem_to_async();
          // Two chunks of 32 columns, one after the other: both in registers at once would not fit beside the results.
          uint32_t pk[2][16], dk[2][16];
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int c0 = (half + 2 * c) * 32;
            const bool on = rows_on && c0 < valid_k;                          // uniform for the warp
            uint32_t rs[32], rd[32];
            if (on) { tmem_ld32(trow + kColS + (uint32_t)c0, rs); tmem_ld32(trow + kColDP + (uint32_t)c0, rd); }
            tmem_ld_wait();
            if (c == 1) {
              fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive(&s_empty);
            }
            if (on) {
              if (rows_full && c0 + 32 <= valid_k) p_ds_chunk<false>(rs, rd, c0, kTile, scale, scale_log2, lse_q, nds, pk[c], dk[c]);
              else p_ds_chunk<true>(rs, rd, c0, q_ok ? valid_k : 0, scale, scale_log2, lse_q, nds, pk[c], dk[c]);
            }
          }
          if (g > 0) {
            ok = wait_all(&m2_full, (uint32_t)((g - 1) & 1));                 // P and dS of the previous step have been read
            if (!ok) break;
            fence_after_sync();
          }
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            if (rows_on && (half + 2 * c) * 32 < valid_k) {                   // chunk half + 2 c: block c, 16-byte columns 4 half ..
              store_chunk(rowbase, (uint32_t)((8 + c) * kBlk), half * 4, pk[c]);
              store_chunk(rowbase, (uint32_t)((10 + c) * kBlk), half * 4, dk[c]);
            }
          }
          fence_smem_to_async();
          __syncwarp();
          if (lane == 0) mbar_arrive(&p_full);
        }
      } else if (g > 0) {
        ok = wait_all(&m2_full, (uint32_t)((g - 1) & 1));
        if (!ok) break;
        fence_after_sync();
      }
      if (g > 0) post();
      p_row0 = item.s0 + q0 + quarter * 32; p_vq = valid_q - quarter * 32; p_head = item.head; p_last = i == n_q - 1;
      if (kSingle) {
        p_zero_q = item.kt > 0;
        if ((item.kt + 1) * kTile < item.len) p_vq = 0;                       // dQ goes on with the next key tile
      }
      p_key0 = item.s0 + item.kt * kTile + quarter * 32; p_vk = valid_k - quarter * 32;
      ++i; ++g;
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // shared memory must outlive the copies that read it
  }
  if (abort_flag) {
    // a wait ran out: a tile may still be on its way into shared memory; give it time before the memory goes away
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  fence_before_sync();
  __syncthreads();
  if (warp == kMma) { fence_after_sync(); tmem_dealloc(tmem, 512); }
  if (threadIdx.x == 0 && abort_flag) rb::set_status(status, rb::kStatusWaitTimeout);
}

}  // namespace

// qkv: bf16 [T, 3 * H * 64] packed (q | k | v, each H heads of 64), T tokens, offsets: int32 [B + 1] on the device, max_len: an upper bound
// of the sequence lengths, out: bf16 [T, H * 64], lse2: fp32 [T, H] or null (log2-domain log-sum-exp), counter: one word of scratch.
// Returns 0 on launch, 1 when the arguments are outside the kernel's range (alignment), > 1 on a launch error.
extern "C" int rb_ragged_attention_fwd(const void* qkv, const int32_t* offsets, int64_t T, int B, int H, int max_len, float scale, void* out,
                                       float* lse2, unsigned* counter, int64_t* status, cudaStream_t st) {
  if (B <= 0 || H <= 0 || max_len <= 0 || T <= 0) return 0;
  if ((reinterpret_cast<uintptr_t>(qkv) & 15) || (reinterpret_cast<uintptr_t>(out) & 15)) return 1;
  int tiles = (int)(((int64_t)max_len + kTile - 1) / kTile);
  if ((int64_t)tiles * B * H > (int64_t)1 << 31) return 1;
  tiles = (int)std::min<int64_t>(tiles, (T + kTile - 1) / kTile);      // no sequence is longer: row numbers of the last tile stay in 32 bits
  const int64_t items = (int64_t)tiles * B * H;
  CUtensorMap map_qkv, map_rows;
  if (rb_tensor_map_2d(&map_qkv, qkv, T, (int64_t)3 * H * kHead, (int64_t)3 * H * kHead, kHead, kTile, 0) != 0 ||
      rb_tensor_map_2d(&map_rows, qkv, T, (int64_t)3 * H * kHead, (int64_t)3 * H * kHead, kHead, 32, 0) != 0)
    return 1;
  static bool attr = false;
  if (!attr) {
    if (cudaFuncSetAttribute(ragged_attention_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFwdSmem) != cudaSuccess ||
        cudaFuncSetAttribute(ragged_attention_fwd_item_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFwdSmem) != cudaSuccess)
      return 3;
    attr = true;
  }
  const float scale_log2 = scale * 1.4426950408889634f;
  const int slots = kFwdCtas * 148;
  const int64_t most = (T / kTile + B) * H;          // items that hold a token, at most
  // Sequences of one tile and a half on average or less run on a CTA per item up to three rounds of items with a token and eight rounds of them in
  // all (100 sequences of 128 tokens, 4 heads: 11.4 us, persistent 14.4; 64 of 1..128 tokens under four times that: 12.6 and 16.5; 590 of
  // 1..90, one head: 12.9 and 14.5; the other way round 590 of 1..40, 2 heads, 1180 items: 21.3 and 16.8; 200 of 1..100, 2 heads, under eight
  // times that, 2800 items: 22.5 and 20.5; longer ones: 100 of 1..500, one head: 17.0 and 16.3).
  if (T <= (int64_t)(kTile * 3 / 2) * B && most <= 3 * slots && items <= 8 * slots) {
    ragged_attention_fwd_item_kernel<<<dim3(tiles, B, H), 128, kFwdSmem, st>>>(map_qkv, offsets, T, H, scale_log2, reinterpret_cast<__nv_bfloat16*>(out),
                                                                             lse2, status);
    rb::note_launch();
    return cudaGetLastError() == cudaSuccess ? 0 : 4;
  }
  // Items are dealt out one per CTA, which saves the counter and its clearing, up to one round of them, three rounds of items of long sequences
  // (15 sequences of 1..1000 tokens, 4 heads: 28.6 us, fetched 34.4; 37 of them, 1184 items: 59 and 56), and eight rounds where the tokens make
  // about one: under a loose bound most items are empty, and a fetched batch of them costs less only from there on (15 sequences under four
  // times their length, 1800 items: 36.9, fetched 43.2; under eight times, 3600 items: 47.1 and 45.0).
  const bool dealt = items <= slots || (items <= 3 * slots && tiles > 2) || (most <= slots * 4 / 3 && T >= (int64_t)2 * kTile * B && items <= 8 * slots);
  if (dealt) counter = nullptr;
  else if (cudaMemsetAsync(counter, 0, sizeof(unsigned), st) != cudaSuccess) return 4;
  // Items fetched at a time: one where that is about 32 fetches per CTA, more under a loose bound, where most items are empty.
  const int grid = (int)(dealt ? items : std::min<int64_t>(items, slots));
  const int chunk = (int)std::min<int64_t>(32, std::max<int64_t>(1, items / (32 * slots)));
  ragged_attention_fwd_kernel<<<grid, kFwdThreads, kFwdSmem, st>>>(map_qkv, map_rows, offsets, T, B, H, tiles, chunk, scale_log2,
                                                                  reinterpret_cast<__nv_bfloat16*>(out), lse2, counter, status);
  rb::note_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

// Backward of rb_ragged_attention_fwd. out / d_out: bf16 [T, H * 64]; lse2: fp32 [T, H] from the forward; scratch: T * H + 1 floats;
// dq_acc: fp32 [T, H * 64], zero on entry (dQ is accumulated with reductions), needed only when max_len > 128; dqkv: bf16
// [T, 3 * H * 64], written completely. Same return codes as the forward.
extern "C" int rb_ragged_attention_bwd(const void* qkv, const void* out, const void* d_out, const float* lse2, float* scratch,
                                       const int32_t* offsets, int64_t T, int B, int H, int max_len, float scale, float* dq_acc, void* dqkv,
                                       int64_t* status, cudaStream_t st) {
  if (B <= 0 || H <= 0 || max_len <= 0 || T <= 0) return 0;
  const bool single = max_len <= kTile;
  if ((reinterpret_cast<uintptr_t>(qkv) & 15) || (reinterpret_cast<uintptr_t>(d_out) & 15) || (reinterpret_cast<uintptr_t>(dqkv) & 15) ||
      (reinterpret_cast<uintptr_t>(out) & 15) || (!single && (dq_acc == nullptr || (reinterpret_cast<uintptr_t>(dq_acc) & 15))))
    return 1;
  int tiles = (int)(((int64_t)max_len + kTile - 1) / kTile);
  if ((int64_t)tiles * B * H > (int64_t)1 << 30) return 1;
  tiles = (int)std::min<int64_t>(tiles, (T + kTile - 1) / kTile);      // as in the forward
  const int64_t items = (int64_t)tiles * B * H;
  const size_t smem = 1024 + 14 * (size_t)kBlk;
  CUtensorMap map_qkv, map_do, map_dq;
  if (rb_tensor_map_2d(&map_qkv, qkv, T, (int64_t)3 * H * kHead, (int64_t)3 * H * kHead, kHead, kTile, 0) != 0 ||
      rb_tensor_map_2d(&map_do, d_out, T, (int64_t)H * kHead, (int64_t)H * kHead, kHead, kTile, 0) != 0)
    return 1;
  if (single) memset(&map_dq, 0, sizeof(map_dq));
  else if (rb_tensor_map_2d(&map_dq, dq_acc, T, (int64_t)H * kHead, (int64_t)H * kHead, 32, 32, 1) != 0) return 1;
  auto kern = single ? ragged_attention_bwd_kernel<true> : ragged_attention_bwd_kernel<false>;
  static bool attr[2] = {false, false};
  if (!attr[single]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 3;
    attr[single] = true;
  }
  unsigned* counter = reinterpret_cast<unsigned*>(scratch + T * H);
  const int64_t blocks = (T * H + 31) / 32;
  attention_delta_kernel<<<(int)(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, st>>>(
      reinterpret_cast<const __nv_bfloat16*>(out), reinterpret_cast<const __nv_bfloat16*>(d_out), T, H, B, offsets, scratch, counter,
      reinterpret_cast<__nv_bfloat16*>(dqkv));
  rb::note_launch();
  kern<<<(int)(items < 148 ? items : 148), kBwdThreads, smem, st>>>(map_qkv, map_do, lse2, scratch, offsets, B, H, tiles, scale,
                                                                   scale * 1.4426950408889634f, reinterpret_cast<__nv_bfloat16*>(dqkv), map_dq,
                                                                   counter, status);
  rb::note_launch();
  if (!single) {
    const int64_t pieces = T * H * (kHead / 8);
    attention_dq_store_kernel<<<(int)std::min<int64_t>((pieces + 255) / 256, 148 * 16), 256, 0, st>>>(dq_acc, T, H * kHead,
                                                                                                  reinterpret_cast<__nv_bfloat16*>(dqkv));
    rb::note_launch();
  }
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}
