// Target attention over packed (ragged) sequences, sm_100a: one query per sequence, softmax over the sequence's tokens,
// weighted sum of the tokens - forward and backward, each ONE pass over the tokens.
//
//   s_t = scale * <x_t, q_b>,  a = softmax_t(s),  interest_b = sum_t a_t x_t            (t over the tokens of sequence b)
//
// The DIN-style interest extraction of a user-behaviour model. Written with tensor ops it is a chain of gather / multiply /
// segment-max / exp / segment-sum / divide / scatter-add passes, each of which re-reads the [tokens, hidden] activations;
// here one CTA walks a sequence once with an online softmax (running maximum, running sum, rescaled accumulator), so the
// activations cross HBM once in the forward pass and twice (read x, write dx) in the backward pass.
// Layout: a warp owns tokens w, w + W, ... of its sequence; lane l owns columns l*4 + k*128 (float4 per 128 columns), so a
// token row is read with fully coalesced 16-byte loads; hidden must be a multiple of 4 and at most 1024.
// The reference has no such op (its sequence example pools with padded tensor ops, examples/seq2seq/seq2seq_model.py).
#include "../common/rb_common.cuh"
#include "../common/rb_launch.h"
#include "rb_dense.h"
#include <climits>

namespace {

constexpr int kWarps = 8;
constexpr int kMaxQuads = 8;      // float4 slots per lane: hidden <= 8 * 128

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int NQ>
__global__ void __launch_bounds__(kWarps * 32)
target_attention_fwd_kernel(const float* __restrict__ x, const float* __restrict__ q, const int32_t* __restrict__ offsets, int H, float scale,
                            float* __restrict__ interest, float* __restrict__ lse) {
  __shared__ float sm_m[kWarps], sm_l[kWarps];
  __shared__ float sm_acc[kWarps][NQ * 128];
  const int b = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int beg = offsets[b], end = offsets[b + 1];
  float4 qv[NQ], acc[NQ];
#pragma unroll
  for (int k = 0; k < NQ; ++k) {
    const int c = lane * 4 + k * 128;
    qv[k] = c < H ? rb::ld_f4(q + (int64_t)b * H + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float m = -INFINITY, l = 0.f;
  for (int t = beg + warp; t < end; t += kWarps) {
    float4 xv[NQ];
    float dot = 0.f;
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      const int c = lane * 4 + k * 128;
      xv[k] = c < H ? rb::ld_f4(x + (int64_t)t * H + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      dot += xv[k].x * qv[k].x + xv[k].y * qv[k].y + xv[k].z * qv[k].z + xv[k].w * qv[k].w;
    }
    const float s = warp_sum(dot) * scale;
    const float m_new = fmaxf(m, s);
    const float alpha = m == -INFINITY ? 0.f : __expf(m - m_new);
    const float p = __expf(s - m_new);
    l = l * alpha + p;
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      acc[k].x = acc[k].x * alpha + p * xv[k].x; acc[k].y = acc[k].y * alpha + p * xv[k].y;
      acc[k].z = acc[k].z * alpha + p * xv[k].z; acc[k].w = acc[k].w * alpha + p * xv[k].w;
    }
    m = m_new;
  }
  // combine the warps' partial softmaxes
  if (lane == 0) { sm_m[warp] = m; sm_l[warp] = l; }
#pragma unroll
  for (int k = 0; k < NQ; ++k) rb::st_f4(&sm_acc[warp][lane * 4 + k * 128], acc[k]);
  __syncthreads();
  float gm = -INFINITY;
  for (int w = 0; w < kWarps; ++w) gm = fmaxf(gm, sm_m[w]);
  float gl = 0.f;
  for (int w = 0; w < kWarps; ++w) gl += sm_m[w] == -INFINITY ? 0.f : sm_l[w] * __expf(sm_m[w] - gm);
  const float inv = gl > 0.f ? 1.f / gl : 0.f;
  for (int c = threadIdx.x; c < H; c += blockDim.x) {
    float v = 0.f;
    for (int w = 0; w < kWarps; ++w) if (sm_m[w] != -INFINITY) v += sm_acc[w][c] * __expf(sm_m[w] - gm);
    interest[(int64_t)b * H + c] = v * inv;
  }
  if (threadIdx.x == 0) lse[b] = gl > 0.f ? gm + __logf(gl) : 0.f;
}

// d a_t = <dI_b, x_t>;  d s_t = a_t (d a_t - <dI_b, interest_b>);  dx_t = a_t dI_b + scale d s_t q_b;  dq_b = scale sum_t d s_t x_t
template <int NQ>
__global__ void __launch_bounds__(kWarps * 32)
target_attention_bwd_kernel(const float* __restrict__ x, const float* __restrict__ q, const int32_t* __restrict__ offsets,
                            const float* __restrict__ interest, const float* __restrict__ lse, const float* __restrict__ d_interest, int H,
                            float scale, float* __restrict__ dx, float* __restrict__ dq) {
  __shared__ float sm_dq[kWarps][NQ * 128];
  const int b = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int beg = offsets[b], end = offsets[b + 1];
  float4 qv[NQ], gv[NQ], dqa[NQ];
  float delta = 0.f;
#pragma unroll
  for (int k = 0; k < NQ; ++k) {
    const int c = lane * 4 + k * 128;
    const bool on = c < H;
    qv[k] = on ? rb::ld_f4(q + (int64_t)b * H + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    gv[k] = on ? rb::ld_f4(d_interest + (int64_t)b * H + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 iv = on ? rb::ld_f4(interest + (int64_t)b * H + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    delta += gv[k].x * iv.x + gv[k].y * iv.y + gv[k].z * iv.z + gv[k].w * iv.w;
    dqa[k] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  delta = warp_sum(delta);
  const float lse_b = lse[b];
  for (int t = beg + warp; t < end; t += kWarps) {
    float4 xv[NQ];
    float dot_q = 0.f, dot_g = 0.f;
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      const int c = lane * 4 + k * 128;
      xv[k] = c < H ? rb::ld_f4(x + (int64_t)t * H + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      dot_q += xv[k].x * qv[k].x + xv[k].y * qv[k].y + xv[k].z * qv[k].z + xv[k].w * qv[k].w;
      dot_g += xv[k].x * gv[k].x + xv[k].y * gv[k].y + xv[k].z * gv[k].z + xv[k].w * gv[k].w;
    }
    dot_q = warp_sum(dot_q); dot_g = warp_sum(dot_g);
    const float a = __expf(dot_q * scale - lse_b);
    const float ds = a * (dot_g - delta) * scale;
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      const int c = lane * 4 + k * 128;
      if (c < H)
        rb::st_f4(dx + (int64_t)t * H + c, make_float4(a * gv[k].x + ds * qv[k].x, a * gv[k].y + ds * qv[k].y, a * gv[k].z + ds * qv[k].z,
                                                      a * gv[k].w + ds * qv[k].w));
      dqa[k].x += ds * xv[k].x; dqa[k].y += ds * xv[k].y; dqa[k].z += ds * xv[k].z; dqa[k].w += ds * xv[k].w;
    }
  }
#pragma unroll
  for (int k = 0; k < NQ; ++k) rb::st_f4(&sm_dq[warp][lane * 4 + k * 128], dqa[k]);
  __syncthreads();
  for (int c = threadIdx.x; c < H; c += blockDim.x) {
    float v = 0.f;
    for (int w = 0; w < kWarps; ++w) v += sm_dq[w][c];
    dq[(int64_t)b * H + c] = v;
  }
}

// Mean over each sequence's tokens: one block per sequence, a thread owns four columns of every rl-th token (rl = threads / (H / 4)), the
// partial sums meet in shared memory. One read of x; with tensor ops it was an atomic scatter-add over the tokens (467 us for 269k
// tokens x 256) and a gather plus division backward (190 us), now 73 and 60 us. Bound by the memory traffic of x and dx.
// One block reads about 57 GB/s, so sequences of more than kLongTokens are taken in pieces of kPiece tokens (cut at multiples of kPiece of the
// packed matrix) by blocks of their own, and in forward a second launch adds each one's pieces in order. At 256 columns, forward and both
// directions: one sequence of 100000 tokens 3604 -> 46 and 6850 -> 84 us, four of 5000 89 -> 19 and 173 -> 73 us. 512 sequences of 50..1000
// tokens pay 9 us for the second launch when the caller gives no bound, nothing when it does.
constexpr int kLongTokens = 1024, kPiece = 512;

// Sum of the rows x[from], x[from + 1], .. x[to - 1] (of H floats) into the threads with r == 0; all threads of the block call it.
__device__ __forceinline__ float4 block_sum_rows(const float* __restrict__ x, int64_t from, int64_t to, int H, int q, int c, int r, int rl, float4* part) {
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (r < rl) {
#pragma unroll 8
    for (int64_t t = from + r; t < to; t += rl) {
      const float4 v = rb::ld_f4(x + t * H + c * 4);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
  }
  part[threadIdx.x] = s;
  __syncthreads();
  if (r == 0)
    for (int k = 1; k < rl; ++k) { const float4 v = part[k * q + c]; s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w; }
  __syncthreads();
  return s;
}

// The sequence that holds token t, or -1: the last one that starts at or before t (empty ones share their start with it).
__device__ __forceinline__ int sequence_of(const int32_t* __restrict__ offsets, int B, int64_t t) {
  if (t < offsets[0] || t >= offsets[B]) return -1;
  int lo = 0, hi = B;                                   // offsets[lo] <= t < offsets[hi]
  while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (offsets[mid] <= t) lo = mid; else hi = mid; }
  return lo;
}

// The long sequences in piece p: slot 0 is the one that holds its first token, slot 1 the one that starts inside and runs past its end.
// (Two are all there can be: a sequence inside a piece is not long.) Returns the sequence or -1.
__device__ __forceinline__ int long_sequence(const int32_t* __restrict__ offsets, int B, int64_t T, int64_t p, int slot, int long_tokens) {
  const int b = sequence_of(offsets, B, slot == 0 ? p * kPiece : min((p + 1) * (int64_t)kPiece, T) - 1);
  if (b < 0 || offsets[b + 1] - offsets[b] <= long_tokens || (slot == 1 && offsets[b] <= p * kPiece)) return -1;
  return b;
}

// Blocks 0 .. B - 1: a sequence each; further blocks: a piece each (partial [pieces][2][H]). long_tokens: kLongTokens, or INT_MAX without pieces.
__global__ void __launch_bounds__(256)
segment_mean_fwd_kernel(const float* __restrict__ x, const int32_t* __restrict__ offsets, int64_t T, int B, int H, int long_tokens,
                        float* __restrict__ partial, float* __restrict__ out) {
  __shared__ float4 part[256];
  const int q = H >> 2, rl = 256 / q;
  const int c = threadIdx.x % q, r = threadIdx.x / q;
  if (blockIdx.x < (unsigned)B) {
    const int b = blockIdx.x, beg = offsets[b], end = offsets[b + 1];
    if (end - beg > long_tokens) return;
    const float4 s = block_sum_rows(x, beg, end, H, q, c, r, rl, part);
    const float n = (float)max(end - beg, 1);
    if (r == 0) rb::st_f4(out + (int64_t)b * H + c * 4, make_float4(s.x / n, s.y / n, s.z / n, s.w / n));
    return;
  }
  const int64_t p = blockIdx.x - B, p0 = p * kPiece, p1 = p0 + kPiece;
  for (int slot = 0; slot < 2; ++slot) {
    const int b = long_sequence(offsets, B, T, p, slot, long_tokens);
    if (b < 0) continue;                                // uniform for the block
    const float4 s = block_sum_rows(x, max((int64_t)offsets[b], p0), min((int64_t)offsets[b + 1], p1), H, q, c, r, rl, part);
    if (r == 0) rb::st_f4(partial + (2 * p + slot) * H + c * 4, s);
  }
}

// One block per piece: finishes the long sequence that starts in it. Its pieces are slot 0 of every later piece, and slot 0 or 1 of this one.
__global__ void __launch_bounds__(256)
segment_mean_finish_kernel(const float* __restrict__ partial, const int32_t* __restrict__ offsets, int64_t T, int B, int H, int long_tokens,
                           float* __restrict__ out) {
  __shared__ float4 part[256];
  const int q = H >> 2, rl = 256 / q;
  const int c = threadIdx.x % q, r = threadIdx.x / q;
  const int64_t p = blockIdx.x;
  int b = long_sequence(offsets, B, T, p, 1, long_tokens);
  const int slot = b >= 0 ? 1 : 0;
  if (b < 0) {
    b = long_sequence(offsets, B, T, p, 0, long_tokens);
    if (b < 0 || offsets[b] != p * kPiece) return;
  }
  const int64_t last = ((int64_t)offsets[b + 1] - 1) / kPiece;
  float4 s = block_sum_rows(partial, p + 1, last + 1, 2 * H, q, c, r, rl, part);
  if (r == 0) {
    const float4 f = rb::ld_f4(partial + (2 * p + slot) * H + c * 4);
    const float n = (float)(offsets[b + 1] - offsets[b]);
    rb::st_f4(out + (int64_t)b * H + c * 4, make_float4((f.x + s.x) / n, (f.y + s.y) / n, (f.z + s.z) / n, (f.w + s.w) / n));
  }
}

__global__ void __launch_bounds__(256)
segment_mean_bwd_kernel(const float* __restrict__ d_out, const int32_t* __restrict__ offsets, int64_t T, int B, int H, int long_tokens,
                        float* __restrict__ dx) {
  const int q = H >> 2, rl = 256 / q;
  const int c = threadIdx.x % q, r = threadIdx.x / q;
  if (r >= rl) return;
  auto spread = [&](int b, int64_t from, int64_t to) {
    const float n = (float)max(offsets[b + 1] - offsets[b], 1);
    float4 g = rb::ld_f4(d_out + (int64_t)b * H + c * 4);
    g = make_float4(g.x / n, g.y / n, g.z / n, g.w / n);
    for (int64_t t = from + r; t < to; t += rl) rb::st_f4(dx + t * H + c * 4, g);
  };
  if (blockIdx.x >= (unsigned)B) {
    const int64_t p = blockIdx.x - B, p0 = p * kPiece, p1 = p0 + kPiece;
    for (int slot = 0; slot < 2; ++slot) {
      const int b = long_sequence(offsets, B, T, p, slot, long_tokens);
      if (b >= 0) spread(b, max((int64_t)offsets[b], p0), min((int64_t)offsets[b + 1], p1));
    }
    return;
  }
  const int b = blockIdx.x, beg = offsets[b], end = offsets[b + 1];
  if (end - beg <= long_tokens) spread(b, beg, end);
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);                       // tokens of no sequence
  if (b == 0) for (int t = r; t < beg; t += rl) rb::st_f4(dx + (int64_t)t * H + c * 4, zero);
  if (b == B - 1) for (int64_t t = end + r; t < T; t += rl) rb::st_f4(dx + t * H + c * 4, zero);
}

template <typename F>
bool dispatch_quads(int H, F&& f) {
  if (H % 4 != 0 || H > kMaxQuads * 128) return false;
  const int nq = (H + 127) / 128;
  if (nq <= 1) f(std::integral_constant<int, 1>{});
  else if (nq <= 2) f(std::integral_constant<int, 2>{});
  else if (nq <= 4) f(std::integral_constant<int, 4>{});
  else f(std::integral_constant<int, 8>{});
  return true;
}

}  // namespace

// x: fp32 [T, H] packed tokens, q: fp32 [B, H], offsets: int32 [B + 1]; interest: fp32 [B, H], lse: fp32 [B]. Returns 1 when H
// is outside the kernel's range (not a multiple of 4 or above 1024).
extern "C" int rb_target_attention_fwd(const float* x, const float* q, const int32_t* offsets, int B, int H, float scale, float* interest,
                                       float* lse, cudaStream_t st) {
  if (B <= 0) return 0;
  const bool ok = dispatch_quads(H, [&](auto nq) {
    constexpr int NQ = decltype(nq)::value;
    target_attention_fwd_kernel<NQ><<<B, kWarps * 32, 0, st>>>(x, q, offsets, H, scale, interest, lse);
  });
  if (ok) rb::note_launch();
  return ok ? 0 : 1;
}

extern "C" int rb_target_attention_bwd(const float* x, const float* q, const int32_t* offsets, const float* interest, const float* lse,
                                       const float* d_interest, int B, int H, float scale, float* dx, float* dq, cudaStream_t st) {
  if (B <= 0) return 0;
  const bool ok = dispatch_quads(H, [&](auto nq) {
    constexpr int NQ = decltype(nq)::value;
    target_attention_bwd_kernel<NQ><<<B, kWarps * 32, 0, st>>>(x, q, offsets, interest, lse, d_interest, H, scale, dx, dq);
  });
  if (ok) rb::note_launch();
  return ok ? 0 : 1;
}

extern "C" int64_t rb_segment_mean_pieces(int64_t T, int64_t longest) {
  return T > kLongTokens && longest > kLongTokens ? (T + kPiece - 1) / kPiece : 0;
}

extern "C" int rb_segment_mean_fwd(const float* x, const int32_t* offsets, int64_t T, int B, int H, int64_t longest, float* partial, float* out,
                                   cudaStream_t st) {
  if (H % 4 != 0 || H <= 0 || H > 1024) return 1;
  if (B <= 0) return 0;
  const int64_t pieces = rb_segment_mean_pieces(T, longest);
  const int long_tokens = pieces ? kLongTokens : INT_MAX;
  segment_mean_fwd_kernel<<<(unsigned)(B + pieces), 256, 0, st>>>(x, offsets, T, B, H, long_tokens, partial, out);
  if (pieces) segment_mean_finish_kernel<<<(unsigned)pieces, 256, 0, st>>>(partial, offsets, T, B, H, long_tokens, out);
  rb::note_launch(pieces ? 2 : 1);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

extern "C" int rb_segment_mean_bwd(const float* d_out, const int32_t* offsets, int64_t T, int B, int H, int64_t longest, float* dx, cudaStream_t st) {
  if (H % 4 != 0 || H <= 0 || H > 1024) return 1;
  if (B <= 0) return 0;
  const int64_t pieces = rb_segment_mean_pieces(T, longest);
  segment_mean_bwd_kernel<<<(unsigned)(B + pieces), 256, 0, st>>>(d_out, offsets, T, B, H, pieces ? kLongTokens : INT_MAX, dx);
  rb::note_launch();
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}
