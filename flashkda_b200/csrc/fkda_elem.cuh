// Element-wise stage of a 32-token chunk in mma.sync fragment layout, for eight warps that own 16 channels each.
//
// Every tensor is held the way an m16n8 accumulator is: thread (g = lane / 4, t = lane % 4), tile nt of 8 channels, register
// b of a ldmatrix.x4 = token 8 b + g, channels 8 nt + 2 t, + 1.  That layout makes the two expensive parts cheap:
//   * row norms: q q^T on the tensor core from the loaded registers (the A and the B fragment of the product are the same
//     registers), whose diagonal holds the sums of squares of this warp's 16 channels;
//   * running sums of the gate: a product with a triangle of ones.  The summand is tanh in [-1, 1], split into two fp16
//     parts (22 bits, products exact, fp32 accumulation), read by a transposing ldmatrix in the B-fragment layout.
// In the row-per-lane layout these took 19 instructions per element (3 shuffles and 3 predicated adds per element for the
// sums alone); here the whole stage is about 19 instructions per element, counting six decayed operands formed in fp32 with
// packed arithmetic and rounded once.
#pragma once
#include <cuda_fp16.h>

#include "fkda_common.cuh"

namespace fkda {
namespace elem {

// ---- packed fp32 pairs ---------------------------------------------------------------------------------------------
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void upk(f2 x, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x)); }
__device__ __forceinline__ f2 mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 unpack_bf(uint32_t w) { return pk(bf_lo(w), bf_hi(w)); }
__device__ __forceinline__ uint32_t round_bf(f2 x) {
  float a, b;
  upk(x, a, b);
  return pack_bf16(a, b);
}

// x0, x1 = hi + lo, both fp16 pairs (22 bits of a tanh)
__device__ __forceinline__ void split_f16(float x0, float x1, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x0, x1);
  const float2 back = __half22float2(h);
  const __half2 l = __floats2half2_rn(x0 - back.x, x1 - back.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

// D(16x8,f32) += A(16x16,f16,row) * B(16x8,f16,col)
__device__ __forceinline__ void mma_f16_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// What a thread keeps over all chunks: the triangle of ones as A fragments, one sign per sub-block.  Exponents are relative
// to the boundary between the two 16-token sub-blocks: G_i = -sum of the tokens behind i up to the boundary in sub-block
// 0, +sum of the tokens from the boundary up to i in sub-block 1.
struct Const {
  uint32_t tri[2][4];
  float hc[4];              // gate_scale / 2 times the number of summands of token row g + 8 b (signed)
  __device__ __forceinline__ Const(int lane, float hgs) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = g + 8 * (i & 1), k0 = 2 * t + 8 * (i >> 1);
      tri[0][i] = (k0 > row ? 0xbc00u : 0u) | (k0 + 1 > row ? 0xbc000000u : 0u);       // -1
      tri[1][i] = (k0 <= row ? 0x3c00u : 0u) | (k0 + 1 <= row ? 0x3c000000u : 0u);     // +1
    }
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int row = g + 8 * (b & 1);
      hc[b] = hgs * static_cast<float>(b < 2 ? row - 15 : row + 1);
    }
  }
};

// byte offset, inside a [32 tok][128 ch] tile of two 128-byte-swizzled [32 tok][64 ch] boxes, of the row that this lane
// addresses in a ldmatrix.x4 over channel block cb (8 channels) and all 32 tokens
__device__ __forceinline__ uint32_t tile_off(int lane, int cb) {
  return static_cast<uint32_t>((cb >> 3) * 4096 + lane * 128 + (((cb & 7) ^ (lane & 7)) << 4));
}
// the same in a core-matrix [32][128] operand
__device__ __forceinline__ uint32_t core_row(int lane, int cb) { return static_cast<uint32_t>((lane >> 3) * 2048 + cb * 128 + (lane & 7) * 16); }

// Partial sums of squares of the rows over this warp's channels: dst[row * 8], row = g + 8 b, written by one thread per row.
__device__ __forceinline__ void row_squares(const uint32_t (&x)[2][4], float* dst, int lane) {
  const int g = lane >> 2;
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};
    mma_bf16_16816(c0, x[0][2 * m], x[0][2 * m + 1], x[1][2 * m], x[1][2 * m + 1], x[0][2 * m], x[1][2 * m]);
    mma_bf16_16816(c1, x[0][2 * m], x[0][2 * m + 1], x[1][2 * m], x[1][2 * m + 1], x[0][2 * m + 1], x[1][2 * m + 1]);
    if ((lane & 3) == (g >> 1)) {          // this thread holds the diagonal elements of rows g and g + 8
      dst[(16 * m + g) * 8] = (g & 1) ? c0[1] : c0[0];
      dst[(16 * m + 8 + g) * 8] = (g & 1) ? c1[3] : c1[2];
    }
  }
}

// Gate of one channel tile and its running sums: gw = transposed fragments (register b = tokens 8 b + 2 t, + 1 of channel g),
// ha = exp(A_log) / 2, hab = ha * dt_bias of that channel.  G[b] = exponents of token g + 8 b, channels 2 t, + 1;
// tot[m] = log2 decay of the whole sub-block m for those channels.  Tokens from `len` on do not decay.
__device__ __forceinline__ void gate_sums(const uint32_t (&gw)[4], const Const& k, float ha, float hab, float hgs, int len, int lane, f2 (&G)[4],
                                          f2 (&tot)[2]) {
  const int t = lane & 3;
  uint32_t hi[4], lo[4];
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    float x0 = tanh_approx(fmaf(bf_lo(gw[b]), ha, hab)), x1 = tanh_approx(fmaf(bf_hi(gw[b]), ha, hab));
    if (len < kChunk) {
      if (8 * b + 2 * t >= len) x0 = -1.f;
      if (8 * b + 2 * t + 1 >= len) x1 = -1.f;
    }
    split_f16(x0, x1, hi[b], lo[b]);
  }
  const uint32_t ones[4] = {0x3c003c00u, 0x3c003c00u, 0x3c003c00u, 0x3c003c00u};
  const f2 h2 = pk(hgs, hgs);
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    float d[4] = {0.f, 0.f, 0.f, 0.f}, s[4] = {0.f, 0.f, 0.f, 0.f};
    mma_f16_16816(d, k.tri[m], hi[2 * m], hi[2 * m + 1]);
    mma_f16_16816(s, ones, hi[2 * m], hi[2 * m + 1]);
    mma_f16_16816(d, k.tri[m], lo[2 * m], lo[2 * m + 1]);
    mma_f16_16816(s, ones, lo[2 * m], lo[2 * m + 1]);
    G[2 * m] = fma2(pk(d[0], d[1]), h2, pk(k.hc[2 * m], k.hc[2 * m]));
    G[2 * m + 1] = fma2(pk(d[2], d[3]), h2, pk(k.hc[2 * m + 1], k.hc[2 * m + 1]));
    tot[m] = fma2(pk(s[0], s[1]), h2, pk(16.f * hgs, 16.f * hgs));
  }
}
__device__ __forceinline__ f2 exp2_pair(f2 x) {
  float a, b;
  upk(x, a, b);
  return pk(ex2f(a), ex2f(b));
}
__device__ __forceinline__ f2 exp2_neg_pair(f2 x) {
  float a, b;
  upk(x, a, b);
  return pk(ex2f(-a), ex2f(-b));
}

}  // namespace elem
}  // namespace fkda
