// Epilogue helpers shared by the tcgen05 GEMM kernels: 32 consecutive fp32 values of one output row become bf16 or fp32 and go
// either straight to global memory (row32 / red32) or into a shared-memory slab laid out as boxes of 32 rows x 128 bytes in the
// 128-byte swizzle, which is what a TMA store (or add-reduction) of such a box expects (stage32).
#pragma once
#include "../common/rb_tcgen05.cuh"
#include <cuda_bf16.h>
#include <stdint.h>

namespace rb {
namespace gemm {

template <typename OutT> struct Store;
template <> struct Store<__nv_bfloat16> {
  static __device__ __forceinline__ void row32(__nv_bfloat16* dst, const float (&v)[32], int valid, bool vec_ok) {
    if (vec_ok && valid == 32) {
      uint4* d4 = reinterpret_cast<uint4*>(dst);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        __nv_bfloat162 p0 = __floats2bfloat162_rn(v[q * 8 + 0], v[q * 8 + 1]), p1 = __floats2bfloat162_rn(v[q * 8 + 2], v[q * 8 + 3]);
        __nv_bfloat162 p2 = __floats2bfloat162_rn(v[q * 8 + 4], v[q * 8 + 5]), p3 = __floats2bfloat162_rn(v[q * 8 + 6], v[q * 8 + 7]);
        uint4 u;
        u.x = *reinterpret_cast<uint32_t*>(&p0); u.y = *reinterpret_cast<uint32_t*>(&p1);
        u.z = *reinterpret_cast<uint32_t*>(&p2); u.w = *reinterpret_cast<uint32_t*>(&p3);
        d4[q] = u;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) if (j < valid) dst[j] = __float2bfloat16_rn(v[j]);
    }
  }
  static __device__ __forceinline__ void red32(__nv_bfloat16*, const float (&)[32], int, bool) {}   // split-K needs fp32 output
  // 32 consecutive columns of one row into the swizzled staging slab: box of 64 columns, four 16-byte chunks
  static constexpr int kBoxCols = 64;
  static __device__ __forceinline__ void stage32(uint8_t* slab, int lane, int c0, const float (&v)[32]) {
    uint8_t* row = slab + (c0 >> 6) * 4096 + lane * 128;
    const int jbase = (c0 & 63) >> 3;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      __nv_bfloat162 p0 = __floats2bfloat162_rn(v[q * 8 + 0], v[q * 8 + 1]), p1 = __floats2bfloat162_rn(v[q * 8 + 2], v[q * 8 + 3]);
      __nv_bfloat162 p2 = __floats2bfloat162_rn(v[q * 8 + 4], v[q * 8 + 5]), p3 = __floats2bfloat162_rn(v[q * 8 + 6], v[q * 8 + 7]);
      uint4 u;
      u.x = *reinterpret_cast<uint32_t*>(&p0); u.y = *reinterpret_cast<uint32_t*>(&p1);
      u.z = *reinterpret_cast<uint32_t*>(&p2); u.w = *reinterpret_cast<uint32_t*>(&p3);
      *reinterpret_cast<uint4*>(row + (((jbase + q) ^ (lane & 7)) << 4)) = u;
    }
  }
};
template <> struct Store<float> {
  static __device__ __forceinline__ void row32(float* dst, const float (&v)[32], int valid, bool vec_ok) {
    if (vec_ok && valid == 32) {
      float4* d4 = reinterpret_cast<float4*>(dst);
#pragma unroll
      for (int q = 0; q < 8; ++q) d4[q] = make_float4(v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]);
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) if (j < valid) dst[j] = v[j];
    }
  }
  static __device__ __forceinline__ void red32(float* dst, const float (&v)[32], int valid, bool vec_ok) {
    if (vec_ok && valid == 32) {
#pragma unroll
      for (int q = 0; q < 8; ++q) atomicAdd(reinterpret_cast<float4*>(dst) + q, make_float4(v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]));
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) if (j < valid) atomicAdd(dst + j, v[j]);
    }
  }
  // 32 consecutive columns of one row = one full 128-byte row of a 32-column box: eight 16-byte chunks
  static constexpr int kBoxCols = 32;
  static __device__ __forceinline__ void stage32(uint8_t* slab, int lane, int c0, const float (&v)[32]) {
    uint8_t* row = slab + (c0 >> 5) * 4096 + lane * 128;
#pragma unroll
    for (int q = 0; q < 8; ++q)
      *reinterpret_cast<float4*>(row + ((q ^ (lane & 7)) << 4)) = make_float4(v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]);
  }
};

// v[j] = 0 where the mask row (32 bf16 starting at mrow) is not positive; a row outside the matrix becomes all zeros
__device__ __forceinline__ void apply_mask32(float (&v)[32], const __nv_bfloat16* mrow, int valid, bool row_ok) {
  if (!row_ok) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = 0.f;
    return;
  }
  if (valid == 32 && (reinterpret_cast<uintptr_t>(mrow) & 15) == 0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint4 u = reinterpret_cast<const uint4*>(mrow)[q];
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 y = __bfloat1622float2(h[e]);
        if (!(y.x > 0.f)) v[q * 8 + 2 * e] = 0.f;
        if (!(y.y > 0.f)) v[q * 8 + 2 * e + 1] = 0.f;
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < valid && !(__bfloat162float(mrow[j]) > 0.f)) v[j] = 0.f;
  }
}

// Column sums of a 32 x 32 block held one row per lane: after five exchange steps lane l holds the sum of column l over the warp's
// 32 rows (each step keeps half of the columns and adds the other lane's copy of them), which it adds to dst[l]. Destroys v.
__device__ __forceinline__ void column_sums32(float (&v)[32], int lane, int valid, float* dst) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    const bool up = (lane & off) != 0;
#pragma unroll
    for (int j = 0; j < off; ++j) {
      const float keep = up ? v[j + off] : v[j];
      const float give = up ? v[j] : v[j + off];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, give, off);
    }
  }
  if (lane < valid) atomicAdd(dst + lane, v[0]);
}

// a += b for two neighbouring floats in one instruction
__device__ __forceinline__ void add_f32x2(float& a0, float& a1, float b0, float b1) {
  asm("{\n\t.reg .b64 u, w;\n\tmov.b64 u, {%0, %1};\n\tmov.b64 w, {%2, %3};\n\tadd.rn.f32x2 u, u, w;\n\tmov.b64 {%0, %1}, u;\n\t}"
      : "+f"(a0), "+f"(a1) : "f"(b0), "f"(b1));
}

// What the epilogue does to a finished accumulator. The second input has the layout of the output: the residual that is added (fp32
// output) or the activations whose sign masks the result (bf16 output). Its boxes arrive by TMA in the slots that the output is then
// staged in, in place.
struct EpilogueWork {
  const CUtensorMap* map_o;
  int MM;
  bool relu, reduce, colsum;       // reduce: the output is added to; colsum: column sums are wanted
};

// One box of the accumulator (32 rows of the warp's lane quarter x kCols columns) into registers, in the layout of an MMA accumulator: of every
// 8 columns a lane holds columns 2 (lane & 3) and + 1 of the rows lane / 4 + 8 r, so that v[4 (h kCols / 8 + j) + 2 r + e] is row
// 16 h + 8 r + lane / 4, column 8 j + 2 (lane & 3) + e. A lane then meets a quarter of the columns: the bias costs a quarter of the
// shared-memory and L1 traffic it costs with a row per lane (25 us of 221 at 269000 x 1024 x 256), and a column sum 14 exchanges
// per 64 columns instead of 62. Lanes may arrive one by one (the caller's stores and copies are some lanes' work): they meet here.
template <int kCols> __device__ __forceinline__ void load_box(uint32_t taddr, float (&v)[kCols]) {
  __syncwarp();
  if constexpr (kCols == 64) {
    tc::tmem_ld_16x64(taddr, reinterpret_cast<uint32_t(&)[32]>(v[0]));
    tc::tmem_ld_16x64(taddr + (16u << 16), reinterpret_cast<uint32_t(&)[32]>(v[32]));
  } else {
    tc::tmem_ld_16x32(taddr, reinterpret_cast<uint32_t(&)[16]>(v[0]));
    tc::tmem_ld_16x32(taddr + (16u << 16), reinterpret_cast<uint32_t(&)[16]>(v[16]));
  }
  tc::tmem_ld_wait();
}

// Column sums over the box's 32 rows: this lane's share, columns column_of(lane) .. + kCols / 32 - 1 of the box, is added to `sum`.
template <int kCols> __device__ __forceinline__ void column_sums(const float (&v)[kCols], int lane, float (&sum)[kCols / 32]) {
  constexpr int kBlocks = kCols / 8;
  float s[2 * kBlocks];                          // s[2 j + e]: column 8 j + 2 (lane & 3) + e
#pragma unroll
  for (int j = 0; j < kBlocks; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e)
      s[2 * j + e] = (v[4 * j + e] + v[4 * j + 2 + e]) + (v[kCols / 2 + 4 * j + e] + v[kCols / 2 + 4 * j + 2 + e]);
  // the eight lanes of a column: each step keeps half of the values and adds the other lane's copy of them
#pragma unroll
  for (int step = 0; step < 3; ++step) {
    const int off = 16 >> step, half = kBlocks >> step;
    const bool up = (lane & off) != 0;
#pragma unroll
    for (int k = 0; k < half; ++k) {
      const float keep = up ? s[half + k] : s[k], give = up ? s[k] : s[half + k];
      s[k] = keep + __shfl_xor_sync(0xffffffffu, give, off);
    }
  }
#pragma unroll
  for (int e = 0; e < kCols / 32; ++e) sum[e] += s[e];
}
template <int kCols> __device__ __forceinline__ int column_of(int lane) {
  constexpr int kBlocks = kCols / 8;
  const int at = ((lane & 16) ? kBlocks : 0) + ((lane & 8) ? kBlocks / 2 : 0) + ((lane & 4) ? kBlocks / 4 : 0);
  return 8 * (at >> 1) + 2 * (lane & 3) + (at & 1);
}

// One box of 32 rows x 128 bytes, already in registers (load_box): bias, second input (in `box`, which has landed), ReLU, mask, conversion,
// staging in `box` and the copy out to rows row0 .. and columns col .. of D, as a bulk group of its own. `bias`: null, or the box's first
// column, readable for the whole box and 8-byte aligned. Column sums of the final values are
// added to `sum` (column_sums). Whole-warp call, destroys v.
//
// With two or four warps to a scheduler and a chain of dependent instructions per element the epilogue was bound by its own instruction
// latency, not by memory: 13,000 warp instructions per 128 x 256 tile, 0.32 per cycle and scheduler, and 7 bytes of output per cycle and
// SM whatever the order of the tiles. Hence no per-element conditions here (edges are clipped by the copies), packed additions, the ReLU
// on packed pairs, and second inputs by TMA instead of a row per lane.
template <typename OutT>
__device__ __forceinline__ void finish_box(const EpilogueWork& w, float (&v)[Store<OutT>::kBoxCols], const float* bias, bool has_src, uint8_t* box, int row0,
                                           int col, int lane, float (&sum)[Store<OutT>::kBoxCols / 32]) {
  constexpr int kCols = Store<OutT>::kBoxCols, kBlocks = kCols / 8;
  __syncwarp();                                  // ldmatrix and stmatrix below want the whole warp at once
  if (bias != nullptr) {
#pragma unroll
    for (int j = 0; j < kBlocks; ++j) {
      const float2 b = *reinterpret_cast<const float2*>(bias + 8 * j + 2 * (lane & 3));
#pragma unroll
      for (int r = 0; r < 4; ++r) add_f32x2(v[(r >> 1) * (kCols / 2) + 4 * j + 2 * (r & 1)], v[(r >> 1) * (kCols / 2) + 4 * j + 2 * (r & 1) + 1], b.x, b.y);
    }
  }
  if constexpr (sizeof(OutT) == 4) {
    const uint32_t base = tc::smem_u32(box) + (uint32_t)((lane >> 2) * 128 + ((((lane >> 1) & 1) ^ (lane >> 2)) << 4) + (lane & 1) * 8);
    if (has_src) {
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int j = 0; j < kBlocks; ++j) {
          float x, y;
          asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(x), "=f"(y) : "r"((base ^ (uint32_t)(j << 5)) + (uint32_t)(r * 1024)) : "memory");
          const int at = (r >> 1) * (kCols / 2) + 4 * j + 2 * (r & 1);
          add_f32x2(v[at], v[at + 1], x, y);
        }
    }
    if (w.relu) {
#pragma unroll
      for (int j = 0; j < kCols; ++j) v[j] = fmaxf(v[j], 0.f);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int j = 0; j < kBlocks; ++j) {
        const int at = (r >> 1) * (kCols / 2) + 4 * j + 2 * (r & 1);
        asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"((base ^ (uint32_t)(j << 5)) + (uint32_t)(r * 1024)), "f"(v[at]), "f"(v[at + 1]) : "memory");
      }
  } else {
    // 8 x 8 matrices, four at a time: rows 0 .. 7 and 8 .. 15 of two neighbouring blocks of 8 columns
    const uint32_t base = tc::smem_u32(box) + (uint32_t)((lane & 15) * 128 + (((lane >> 4) ^ (lane & 7)) << 4));
    if (has_src) {
      // 0xffff for every bf16 above zero (a NaN is not), spread to a 32-bit mask per value
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint32_t m[4];
          asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(m[0]), "=r"(m[1]), "=r"(m[2]), "=r"(m[3])
                       : "r"((base ^ (uint32_t)(i << 5)) + (uint32_t)(h * 2048)) : "memory");
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const uint32_t on = __hgt2_mask(*reinterpret_cast<const __nv_bfloat162*>(&m[e]), __float2bfloat162_rn(0.f));
            float& x = v[h * 32 + 8 * i + 2 * e];
            float& y = v[h * 32 + 8 * i + 2 * e + 1];
            x = __uint_as_float(__float_as_uint(x) & __byte_perm(on, 0u, 0x1010));
            y = __uint_as_float(__float_as_uint(y) & __byte_perm(on, 0u, 0x3232));
          }
        }
    }
    if (w.relu && w.colsum) {
#pragma unroll
      for (int j = 0; j < kCols; ++j) v[j] = fmaxf(v[j], 0.f);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint32_t u[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          __nv_bfloat162 p = __floats2bfloat162_rn(v[h * 32 + 8 * i + 2 * e], v[h * 32 + 8 * i + 2 * e + 1]);
          if (w.relu) p = __hmax2(p, __float2bfloat162_rn(0.f));
          u[e] = *reinterpret_cast<uint32_t*>(&p);
        }
        asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};"
                     ::"r"((base ^ (uint32_t)(i << 5)) + (uint32_t)(h * 2048)), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]) : "memory");
      }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  if (lane == 0) {
    if (w.reduce)
      asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.bulk_group [%0, {%2, %3}], [%1];"
                   ::"l"(w.map_o), "r"(tc::smem_u32(box)), "r"(col), "r"(row0) : "memory");
    else
      asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
                   ::"l"(w.map_o), "r"(tc::smem_u32(box)), "r"(col), "r"(row0) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  }
  if (w.colsum) {
    if (row0 + 32 > w.MM) {
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (row0 + 8 * r + (lane >> 2) >= w.MM) {
#pragma unroll
          for (int j = 0; j < kBlocks; ++j) { v[(r >> 1) * (kCols / 2) + 4 * j + 2 * (r & 1)] = 0.f; v[(r >> 1) * (kCols / 2) + 4 * j + 2 * (r & 1) + 1] = 0.f; }
        }
    }
    column_sums<kCols>(v, lane, sum);
  }
}

}  // namespace gemm
}  // namespace rb
