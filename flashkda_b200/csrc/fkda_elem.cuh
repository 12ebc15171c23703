// Element-wise stage of a 32-token chunk in mma.sync fragment layout, for eight warps that own 16 channels each.
//
// Every tensor is held the way an m16n8 accumulator is: thread (g = lane / 4, t = lane % 4), tile nt of 8 channels, register
// b of a ldmatrix.x4 = token 8 b + g, channels 8 nt + 2 t, + 1.  That layout makes the two expensive parts cheap:
//   * row norms: q q^T on the tensor core from the loaded registers (the A and the B fragment of the product are the same
//     registers), whose diagonal holds the sums of squares of this warp's 16 channels;
//   * running sums of the gate: a product with a triangle of ones.  The summand is tanh in [-1, 1], split into two fp16
//     parts (22 bits, products exact, fp32 accumulation), read by a transposing ldmatrix in the B-fragment layout.
// In the row-per-lane layout these took 19 instructions per element (3 shuffles and 3 predicated adds per element for the
// sums alone).
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

// The same onto zero (no registers to clear).
__device__ __forceinline__ void mma_f16_16816_zero(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// D(16x8,f32) = A(16x8,f16,row) * B(8x8,f16,col), then D += ...
__device__ __forceinline__ void mma_f16_1688_zero(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
               : "r"(a0), "r"(a1), "r"(b), "f"(0.f));
}
__device__ __forceinline__ void mma_f16_1688(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(b));
}
// The same with bf16 operands.
__device__ __forceinline__ void mma_bf16_1688_zero(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
               : "r"(a0), "r"(a1), "r"(b), "f"(0.f));
}
__device__ __forceinline__ void mma_bf16_1688(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(b));
}

// What a thread keeps over all chunks: the triangle of ones as A fragments, and the gate's constant part of the running sums.
// (Opaque to the compiler, which would otherwise work them out again in every chunk to save the registers.)
struct Const {
  uint32_t tri[4];
  float hc[2];              // gate_scale / 2 times the number of summands of row g + 8 b of a sub-block
  __device__ __forceinline__ Const(int lane, float hgs) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = g + 8 * (i & 1), k0 = 2 * t + 8 * (i >> 1);
      tri[i] = (k0 <= row ? 0x3c00u : 0u) | (k0 + 1 <= row ? 0x3c000000u : 0u);
      asm volatile("" : "+r"(tri[i]));
    }
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      hc[b] = hgs * static_cast<float>(g + 8 * b + 1);
      asm volatile("" : "+f"(hc[b]));
    }
  }
};

// Shared memory by 32-bit address.
__device__ __forceinline__ void sts_f32(uint32_t addr, float x) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(x) : "memory"); }
__device__ __forceinline__ void sts_f2(uint32_t addr, f2 x) { asm volatile("st.shared.b64 [%0], %1;" ::"r"(addr), "l"(x) : "memory"); }
__device__ __forceinline__ float lds_f32(uint32_t addr) {
  float x;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x) : "r"(addr) : "memory");
  return x;
}
__device__ __forceinline__ int lds_s32(uint32_t addr) {
  int x;
  asm volatile("ld.shared.s32 %0, [%1];" : "=r"(x) : "r"(addr) : "memory");
  return x;
}
__device__ __forceinline__ void sts_u4(uint32_t addr, uint32_t x) { asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(addr), "r"(x) : "memory"); }
__device__ __forceinline__ float4 lds_f4(uint32_t addr) {
  float4 x;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "r"(addr) : "memory");
  return x;
}

// byte offset, inside a [32 tok][128 ch] tile of two 128-byte-swizzled [32 tok][64 ch] boxes, of the row that this lane
// addresses in a ldmatrix.x4 over channel block cb (8 channels) and all 32 tokens
__device__ __forceinline__ uint32_t tile_off(int lane, int cb) {
  return static_cast<uint32_t>((cb >> 3) * 4096 + lane * 128 + (((cb & 7) ^ (lane & 7)) << 4));
}
// the same in a core-matrix [32][128] operand
__device__ __forceinline__ uint32_t core_row(int lane, int cb) { return static_cast<uint32_t>((lane >> 3) * 2048 + cb * 128 + (lane & 7) * 16); }

// Partial sums of squares of the rows over this warp's channels, fp32 at dst + 32 row, row = g + 8 b, written by one thread per row.
// (Products of depth 8: their operands are the registers as ldmatrix leaves them.)
__device__ __forceinline__ void row_squares(const uint32_t (&x)[2][4], uint32_t dst, int lane) {
  const int g = lane >> 2;
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    float c0[4], c1[4];
    mma_bf16_1688_zero(c0, x[0][2 * m], x[0][2 * m + 1], x[0][2 * m]);
    mma_bf16_1688_zero(c1, x[0][2 * m], x[0][2 * m + 1], x[0][2 * m + 1]);
    mma_bf16_1688(c0, x[1][2 * m], x[1][2 * m + 1], x[1][2 * m]);
    mma_bf16_1688(c1, x[1][2 * m], x[1][2 * m + 1], x[1][2 * m + 1]);
    if ((lane & 3) == (g >> 1)) {          // this thread holds the diagonal elements of rows g and g + 8
      sts_f32(dst + (16 * m + g) * 32, (g & 1) ? c0[1] : c0[0]);
      sts_f32(dst + (16 * m + 8 + g) * 32, (g & 1) ? c1[3] : c1[2]);
    }
  }
}

// Gate of one channel tile and its running sums: gw = transposed fragments (register b = tokens 8 b + 2 t, + 1 of channel g),
// ha = exp(A_log) / 2, hab = ha * dt_bias of that channel.  G[b] = exponents of token g + 8 b, channels 2 t, + 1, relative to
// the boundary between the two 16-token sub-blocks (minus the sum of the tokens behind in sub-block 0, plus the sum up to it in
// sub-block 1); tot[m] = log2 decay of the whole sub-block m for those channels.
__device__ __forceinline__ void gate_sums(const uint32_t (&gw)[4], const Const& k, float ha, float hab, float hgs, int lane, f2 (&G)[4],
                                          f2 (&tot)[2]) {
  float th[8];
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    th[2 * b] = tanh_approx(fmaf(bf_lo(gw[b]), ha, hab));
    th[2 * b + 1] = tanh_approx(fmaf(bf_hi(gw[b]), ha, hab));
  }
  uint32_t hi[4], lo[4];
#pragma unroll
  for (int b = 0; b < 4; ++b) split_f16(th[2 * b], th[2 * b + 1], hi[b], lo[b]);
  float d[2][4];
#pragma unroll
  for (int m = 0; m < 2; ++m) mma_f16_16816_zero(d[m], k.tri, hi[2 * m], hi[2 * m + 1]);
#pragma unroll
  for (int m = 0; m < 2; ++m) mma_f16_16816(d[m], k.tri, lo[2 * m], lo[2 * m + 1]);
  float x[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) x[e] = fmaf(d[e >> 2][e & 3], hgs, k.hc[(e >> 1) & 1]);
  const int last = lane | 28;              // the thread that holds the sums at token 15 of a sub-block for these channels
  const float t0 = __shfl_sync(0xffffffffu, x[2], last), t1 = __shfl_sync(0xffffffffu, x[3], last);
  tot[1] = pk(__shfl_sync(0xffffffffu, x[6], last), __shfl_sync(0xffffffffu, x[7], last));
  tot[0] = pk(t0, t1);
  G[0] = pk(x[0] - t0, x[1] - t1);
  G[1] = pk(x[2] - t0, x[3] - t1);
  G[2] = pk(x[4], x[5]);
  G[3] = pk(x[6], x[7]);
}
__device__ __forceinline__ f2 exp2_pair(f2 x) {
  float a, b;
  upk(x, a, b);
  return pk(ex2f(a), ex2f(b));
}
// 1 / x for powers of two inside the operands' range: no negated exponent to form
__device__ __forceinline__ f2 rcp_pair(f2 x) {
  float a, b;
  upk(x, a, b);
  asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(a));
  asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(b));
  return pk(a, b);
}

}  // namespace elem
}  // namespace fkda
