// Token-parallel half of the KDA prefill for the compact operand record (fkda_record.cuh).
//
// Replaces the reference's K1 (csrc/smxx/fwd_kernel1.cuh:107-586).  Two CTAs per SM, each a loop over (32-token chunk, head)
// items; inside a CTA
//   warps 0-7    element-wise stage in mma fragment layout, 16 channels each (fkda_elem.cuh)
//   warp  8, 10  T = (I + A)^-1 and TB = T diag(beta) of even / odd items
//   warp  9      loads of the item after next, stores of the record, tril(M)
//   warp  11     first products [A; M] = [k+; q+] k-^T on tcgen05
//
// 770 bytes read and 912 written per token-head: 0.27 ms of HBM time on a million token-heads.  Alone it takes 0.322 ms in a
// burst of calls (5.5 TB/s, 84 % of the measured copy rate) and 0.366 kept up under the power cap.
// What it took to get there from 0.379 / 0.413 ms (4 x 8192 tokens x 32 heads, cycles per item and CTA by clock64):
//   * The row norms went through a warp that also issued the products: an element warp waited 1000 of its 5700 cycles for them.
//     Every element warp now sums the eight partial sums itself (two rows per lane, handed round by shuffles).  That alone made
//     the kernel slower, 0.414 ms: the element warps' code had grown past what a sub-partition's instruction cache holds beside
//     the inverse (stalls for instructions 0.7 -> 1.4 cycles per issue).
//   * So the code shrank: the triangle of ones and the gate's constants are opaque to the compiler, which had been working
//     them out again in every chunk (kept in registers, with one triangle for both sub-blocks and the totals taken from its last
//     row by a shuffle instead of a product with ones); shared memory is addressed by 32-bit registers; the norms' products
//     have a depth of 8, whose operands are the registers as ldmatrix leaves them; rows past a sequence's end are written
//     over in the tile, so that the loop has no masks.  6590 -> 6120 warp instructions per item, and no spills.
//   * A wait without a suspend-time hint: the hint is emulated by sleeping.  0.355 -> 0.349 ms.  (A tight loop of attempts:
//     0.358; explicit sleeps of 20 to 100 ns: 0.350.)
//   * One 4-d copy per tensor instead of two 3-d ones, issued before the next item is decoded (a request costs its issuer 120
//     cycles), and no prefetch to the L2 any more, which the earlier loads do not need: 0.339 / 0.387 -> 0.336 / 0.380 ms.
//   * The first products issued by a whole warp (elect.sync) with operands that the compiler can see to be uniform, 300 cycles instead
//     of 940 between the operands and the element warps' next store: 0.338 / 0.379 -> 0.322 / 0.366 ms.
//
// Decay ranges: with G the running log2 decay inside the chunk and P its value after the first 16 tokens, the first products
// use k+ = khat 2^(G - P) and k- = khat 2^(P - G): both stay inside 2^(+-115.4) for lower_bound >= -5 (16 tokens x 5 x
// log2 e), every needed product k+_i k-_j (j <= i) is <= 1 in magnitude, and one 32 x 32 product covers both sub-blocks.
#include <stddef.h>

#include "fkda_common.cuh"
#include "fkda_elem.cuh"
#include "fkda_record.cuh"
#include "fkda_tma.cuh"

namespace fkda {
namespace operands {

constexpr int kThreads = 384;
constexpr uint32_t kTmemCols = 64;                 // two results of the first products, 32 columns each
// shared memory (bytes from a 1024-byte aligned base)
constexpr int kSlotBytes = 3 * 8192;               // q | k | g tiles, then KP | QP | KR over them
constexpr int kSmSlot = 0;                         // 2 slots
constexpr int kSmScr = kSmSlot + 2 * kSlotBytes;   // operands of the first products, relative to the sub-block boundary:
                                                   //   k- | k+ | q+ (even items) or k- | q+ | k+ (odd items)
constexpr int kSmTB = kSmScr + 3 * 8192;           // 2 x TB
constexpr int kSmMqk = kSmTB + 2 * 2048;           // 2 x MQK
constexpr int kSmInv = kSmMqk + 2 * 2048;          // 2 x fp32 scratch of the inverse
constexpr int kLd = 20;                            // floats per row of its 16 x 16 blocks
constexpr int kInvBytes = (32 + 16 + 32) * kLd * 4;
constexpr int kSmE = kSmInv + 2 * kInvBytes;       // 2 x E
constexpr int kSmBias = kSmE + 2 * 512;            // 2 x dt_bias[h]
constexpr int kSmSsq = kSmBias + 2 * 512;          // 2 x [q|k][32 rows][8 warps] partial sums of squares
constexpr int kSmBeta = kSmSsq + 2 * 2048;         // 4 x [32] sigmoid(beta)
constexpr int kInfos = 8;
constexpr int kSmInfo = kSmBeta + 4 * 128;
constexpr int kSmBars = kSmInfo + kInfos * 32;
constexpr int kSmMisc = kSmBars + 128;
constexpr int kSmemBytes = (kSmMisc + 16 + 1023) / 1024 * 1024;
// (the first products' A operand is 128 rows: those beyond k+ and q+ are read from whatever follows, inside this CTA's memory)
static_assert(kSmScr + 8192 + 32768 <= kSmemBytes, "rows 64-127 of the A operand lie inside the allocation");
static_assert(2 * (kSmemBytes + 1024) <= 227 * 1024, "two CTAs per SM");

enum { B_IN = 0 /*[2]*/, B_NORMP = 2 /*[2]*/, B_OPS = 4 /*[2]*/, B_D1 = 6 /*[2]*/, B_D1_FREE = 8 /*[2]*/, B_COUNT = 10 };
static_assert(B_COUNT * 8 <= 128, "barrier area");

struct Info {
  long long t0;        // first token of the chunk
  int len, h, gc;      // valid tokens, head, chunk (record index of the head)
  float ha;            // exp(A_log[h]) / 2
  int pad[2];
};
static_assert(sizeof(Info) == 32, "info");

// Where an item lies (all but ha, which takes a load from memory).
template <bool kSlice>
__device__ __forceinline__ Info decode(const PrepParams& p, unsigned item) {
  Info r;
  r.h = static_cast<int>(item % static_cast<unsigned>(p.H));        // consecutive items: consecutive heads of a chunk, adjacent in memory
  r.gc = static_cast<int>(item / static_cast<unsigned>(p.H));
  r.pad[0] = r.pad[1] = 0;
  if (p.cu_seqlens != nullptr) {
    int lo = 0, hi = p.N - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (p.chunk_prefix[mid] <= r.gc) lo = mid; else hi = mid - 1;
    }
    long long bos = p.cu_seqlens[lo], eos = p.cu_seqlens[lo + 1];
    bos = bos < 0 ? 0 : (bos > p.T_total ? p.T_total : bos);
    eos = eos < bos ? bos : (eos > p.T_total ? p.T_total : eos);
    r.t0 = bos + static_cast<long long>(r.gc - p.chunk_prefix[lo]) * kChunk;
    const long long rem = eos - r.t0;
    r.len = rem < kChunk ? static_cast<int>(rem) : kChunk;
  } else {
    const unsigned cps = kSlice ? static_cast<unsigned>(p.slice_chunks) : static_cast<unsigned>((p.T + kChunk - 1) / kChunk);
    const unsigned n = static_cast<unsigned>(r.gc) / cps, lc = static_cast<unsigned>(r.gc) - n * cps + (kSlice ? static_cast<unsigned>(p.slice_begin) : 0u);
    if (kSlice) r.gc = static_cast<int>(n * static_cast<unsigned>(p.seq_chunks) + lc);
    r.t0 = static_cast<long long>(n) * p.T + static_cast<long long>(lc) * kChunk;
    const long long rem = p.T - static_cast<long long>(lc) * kChunk;
    r.len = rem < kChunk ? static_cast<int>(rem) : kChunk;
  }
  return r;
}
__device__ __forceinline__ float gate_factor(const PrepParams& p, int h) {
  const float ha = 0.5f * ex2f(__ldg(p.A_log + h) * kLog2e);
  // (off zero and infinity: a gate input of minus infinity stands for a token that is not there)
  return ha < 1e-30f ? 1e-30f : ha > 1e30f ? 1e30f : ha;
}
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xffffffffu, mbar_wait_parked(bar, parity, abort_flag));
}

// A (this lane's row in `a`, 32 columns) -> T = (I + A diag_rows(beta))^-1 -> T diag(beta), bf16 [32][32] in core layout at tb.
// fp32 throughout: forward substitution on the two 16 x 16 diagonal blocks, one column per lane, and two tf32 products for the
// block below them.  Scratch: diagonal blocks of A | block A10 | diagonal blocks of T, kLd floats per row.
__device__ __forceinline__ void inverse(const uint32_t (&a)[32], float* scratch, const float* s_beta, uint8_t* tb, float bi, int lane) {
  float* Ad = scratch;
  float* A10 = scratch + 32 * kLd;
  float* Td = scratch + 48 * kLd;
  const bool low = lane >= 16;
  {
    float* dst = low ? A10 + (lane - 16) * kLd : Ad + lane * kLd;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float x[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) x[e] = 4 * q + e < lane ? __uint_as_float(a[4 * q + e]) * bi : 0.f;
      *reinterpret_cast<float4*>(dst + 4 * q) = make_float4(x[0], x[1], x[2], x[3]);
    }
    if (low) {
#pragma unroll
      for (int q = 4; q < 8; ++q) {
        float x[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = 4 * q + e < lane ? __uint_as_float(a[4 * q + e]) * bi : 0.f;
        *reinterpret_cast<float4*>(Ad + lane * kLd + 4 * q - 16) = make_float4(x[0], x[1], x[2], x[3]);
      }
    }
  }
  __syncwarp();
  {
    const int bb = lane >> 4, c = lane & 15;
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (4 * q < i) {
          const float4 r = *reinterpret_cast<const float4*>(Ad + (bb * 16 + i) * kLd + 4 * q);
          part[q] = fmaf(r.x, x[4 * q], part[q]);
          part[q] = fmaf(r.y, x[4 * q + 1], part[q]);
          part[q] = fmaf(r.z, x[4 * q + 2], part[q]);
          part[q] = fmaf(r.w, x[4 * q + 3], part[q]);
        }
      }
      x[i] = ((i == c) ? 1.f : 0.f) - ((part[0] + part[1]) + (part[2] + part[3]));
      Td[(bb * 16 + i) * kLd + c] = x[i];
    }
  }
  __syncwarp();
  {
    const int g = lane >> 2, t4 = lane & 3;
    auto product = [&](const float* A, const float* B, float* D, float sign) {
      float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
      for (int k0 = 0; k0 < 16; k0 += 8) {
        const uint32_t f0 = to_tf32(A[g * kLd + k0 + t4]), f1 = to_tf32(A[(g + 8) * kLd + k0 + t4]);
        const uint32_t f2 = to_tf32(A[g * kLd + k0 + t4 + 4]), f3 = to_tf32(A[(g + 8) * kLd + k0 + t4 + 4]);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
          mma_tf32_1688(acc[nt], f0, f1, f2, f3, to_tf32(B[(k0 + t4) * kLd + 8 * nt + g]), to_tf32(B[(k0 + t4 + 4) * kLd + 8 * nt + g]));
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        *reinterpret_cast<float2*>(D + g * kLd + 8 * nt + 2 * t4) = make_float2(sign * acc[nt][0], sign * acc[nt][1]);
        *reinterpret_cast<float2*>(D + (g + 8) * kLd + 8 * nt + 2 * t4) = make_float2(sign * acc[nt][2], sign * acc[nt][3]);
      }
    };
    product(A10, Td, Ad, 1.f);                       // X = A10 T00, over the first diagonal block of A
    __syncwarp();
    product(Td + 16 * kLd, Ad, A10, -1.f);           // T10 = -T11 X, over A10
  }
  __syncwarp();
  {
    uint8_t* row = tb + (lane >> 3) * 512 + (lane & 7) * 16;
    const float* left = low ? A10 + (lane - 16) * kLd : Td + lane * kLd;
#pragma unroll
    for (int cb = 0; cb < 4; ++cb) {
      uint32_t w[4] = {0u, 0u, 0u, 0u};
      if (cb < 2 || low) {
        const float* src = cb < 2 ? left + 8 * cb : Td + lane * kLd + 8 * cb - 16;
        const float4 x = *reinterpret_cast<const float4*>(src), y = *reinterpret_cast<const float4*>(src + 4);
        const float4 u = *reinterpret_cast<const float4*>(s_beta + 8 * cb), v = *reinterpret_cast<const float4*>(s_beta + 8 * cb + 4);
        w[0] = pack_bf16(x.x * u.x, x.y * u.y);
        w[1] = pack_bf16(x.z * u.z, x.w * u.w);
        w[2] = pack_bf16(y.x * v.x, y.y * v.y);
        w[3] = pack_bf16(y.z * v.z, y.w * v.w);
      }
      *reinterpret_cast<uint4*>(row + cb * 128) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

// Element-wise stage of all items, warp w of eight.
__device__ __forceinline__ bool element_role(const PrepParams& p, uint32_t sbase, int n_it, int w, int lane, volatile int* abort_flag) {
  using namespace elem;
  const int g = lane >> 2, t = lane & 3;
  const float hgs = 0.5f * p.gate_scale;
  const Const kc(lane, hgs);
  asm volatile("" : "+r"(sbase));      // (kept in a register rather than worked out again wherever it is used)
  auto bar = [&](int i) { return sbase + kSmBars + 8 * i; };
  for (int i = 0; i < n_it; ++i) {
    const int b = i & 1;
    const uint32_t ph = (i >> 1) & 1;
    if (!warp_wait(bar(B_IN + b), ph, abort_flag)) return false;
    const uint32_t info = sbase + kSmInfo + (i & (kInfos - 1)) * static_cast<int>(sizeof(Info));
    const int len = lds_s32(info + offsetof(Info, len));
    const float ha = lds_f32(info + offsetof(Info, ha));
    const uint32_t tile = sbase + kSmSlot + b * kSlotBytes;
    if (lane >= len) {               // rows past the sequence end belong to somebody else: no keys, no queries, no decay
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const uint32_t row = tile + tile_off(lane, 2 * w + nt);
        sts_u4(row, 0u);
        sts_u4(row + 8192, 0u);
        sts_u4(row + 16384, 0xff80ff80u);      // minus infinity, whose tanh is -1 ...
      }
    }
    if (len < kChunk && lane < 16) {           // ... on top of a finite bias
      const uint32_t bias = sbase + kSmBias + b * 512 + (16 * w + lane) * 4;
      const float x = lds_f32(bias), most = 3e38f / fmaxf(ha, 1.f);
      if (fabsf(x) > most) sts_f32(bias, copysignf(most, x));
    }
    __syncwarp();
    uint32_t q[2][4], k[2][4], gw[2][4];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      const uint32_t off = tile_off(lane, 2 * w + nt);
      ldsm_x4(tile + off, q[nt][0], q[nt][1], q[nt][2], q[nt][3]);
      ldsm_x4(tile + 8192 + off, k[nt][0], k[nt][1], k[nt][2], k[nt][3]);
      ldsm_x4_trans(tile + 16384 + off, gw[nt][0], gw[nt][1], gw[nt][2], gw[nt][3]);
    }
    const uint32_t ssq = sbase + kSmSsq + b * 2048;
    const int part = 4 * (w ^ (g & 4));    // (rows 4-7 of eight have the halves exchanged: sixteen-byte reads by row do not conflict)
    row_squares(q, ssq + part, lane);
    row_squares(k, ssq + 1024 + part, lane);
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(B_NORMP + b));       // (also: this warp has read its share of the tiles)

    // The two tiles of eight channels; the waits lie behind the gate of the first.
    float rq[4], rk[4];
    uint32_t off = core_row(lane, 2 * w);
    const uint32_t scr = sbase + kSmScr, scr_k = scr + (b ? 16384 : 8192), scr_q = scr + (b ? 8192 : 16384);
    uint32_t bias = sbase + kSmBias + b * 512 + (16 * w + g) * 4, decay = sbase + kSmE + b * 512 + (16 * w + 2 * t) * 4;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      f2 G[4], tot[2];
      gate_sums(gw[nt], kc, ha, ha * lds_f32(bias), hgs, lane, G, tot);
      if (nt == 0) {
        if (!warp_wait(bar(B_NORMP + b), ph, abort_flag)) return false;     // all eight warps have read the tiles: the slot may be written over
        const uint32_t row = ssq + lane * 32 + (lane & 4) * 4;
        auto sum = [&](uint32_t s) {
          const float4 x = lds_f4(s), y = lds_f4(s ^ 16);
          return rsqrtf(((x.x + x.y) + (x.z + x.w)) + ((y.x + y.y) + (y.z + y.w)) + 1e-6f);
        };
        const float nq = sum(row) * p.scale, nk = sum(row + 1024);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          rq[j] = __shfl_sync(0xffffffffu, nq, g + 8 * j);
          rk[j] = __shfl_sync(0xffffffffu, nk, g + 8 * j);
        }
        if (i >= 1 && !warp_wait(bar(B_D1 + (b ^ 1)), ((i - 1) >> 1) & 1, abort_flag)) return false;   // the first products' operands are read
      }
      const f2 cP = exp2_pair(tot[0]), cQ = exp2_pair(tot[1]), nP = mul(cP, pk(-1.f, -1.f));
      if (g == 0) sts_f2(decay, mul(cP, cQ));
      uint32_t kpm[4], kmm[4], qpm[4], kp[4], qp[4], kr[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const f2 kh = pk(bf_lo(k[nt][r]) * rk[r], bf_hi(k[nt][r]) * rk[r]), qh = pk(bf_lo(q[nt][r]) * rq[r], bf_hi(q[nt][r]) * rq[r]);
        const f2 pw = exp2_pair(G[r]), ip = rcp_pair(pw);
        const f2 a = mul(kh, pw), m = mul(kh, ip), c = mul(qh, pw);
        kpm[r] = round_bf(a);
        kmm[r] = round_bf(m);
        qpm[r] = round_bf(c);
        kp[r] = round_bf(mul(a, nP));
        qp[r] = round_bf(mul(c, cP));
        kr[r] = round_bf(mul(m, cQ));
      }
      stsm_x4(scr + off, kmm[0], kmm[1], kmm[2], kmm[3]);
      stsm_x4(scr_k + off, kpm[0], kpm[1], kpm[2], kpm[3]);
      stsm_x4(scr_q + off, qpm[0], qpm[1], qpm[2], qpm[3]);
      stsm_x4(tile + off, kp[0], kp[1], kp[2], kp[3]);
      stsm_x4(tile + 8192 + off, qp[0], qp[1], qp[2], qp[3]);
      stsm_x4(tile + 16384 + off, kr[0], kr[1], kr[2], kr[3]);
      off += 128;
      bias += 32;
      decay += 32;
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(B_OPS + b));
  }
  return true;
}

// T diag(beta) of the items of one parity.
__device__ __forceinline__ bool inverse_role(const PrepParams& p, uint8_t* smem, uint32_t sbase, uint32_t tmem, int n_it, int b, int lane,
                                             volatile int* abort_flag) {
  auto bar = [&](int i) { return sbase + kSmBars + 8 * i; };
  bool ok = true;
  for (int i = b; i < n_it; i += 2) {
    // (only this barrier: it cannot run a phase ahead of a warp that frees its result)
    if (!warp_wait(bar(B_D1 + b), (i >> 1) & 1, abort_flag)) { ok = false; break; }
    const int h = reinterpret_cast<const Info*>(smem + kSmInfo)[i & (kInfos - 1)].h, gc = reinterpret_cast<const Info*>(smem + kSmInfo)[i & (kInfos - 1)].gc;
    const float* s_beta = reinterpret_cast<const float*>(smem + kSmBeta + (i & 3) * 128);
    tc_fence_after();
    uint32_t a[32];
    tmem_ld32(tmem + (static_cast<uint32_t>(64 * b) << 16) + 32 * b, a);
    tmem_wait_ld();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(B_D1_FREE + b));
    if (lane == 0) bulk_wait_read0();                // the previous TB of this warp has left its staging
    __syncwarp();
    inverse(a, reinterpret_cast<float*>(smem + kSmInv + b * kInvBytes), s_beta, smem + kSmTB + b * 2048, s_beta[lane], lane);
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      bulk_s2g(p.records + (static_cast<size_t>(h) * p.total_chunks + gc) * kCrBytes + kCrTB, sbase + kSmTB + b * 2048, 2048);
      bulk_commit();
    }
  }
  if (lane == 0) bulk_wait_read0();                  // giving up too: the store reads this CTA's shared memory
  return ok;
}

// Loads, stores and tril(M).
template <bool kSlice>
__device__ __forceinline__ bool copy_role(const PrepParams& p, const CUtensorMap* tq, const CUtensorMap* tk, const CUtensorMap* tg, uint8_t* smem,
                                          uint32_t sbase, uint32_t tmem, int n_it, int lane, volatile int* abort_flag) {
  auto bar = [&](int i) { return sbase + kSmBars + 8 * i; };
  Info* infos = reinterpret_cast<Info*>(smem + kSmInfo);
  auto load = [&](int i, const Info& f) {
    const uint32_t full = bar(B_IN + (i & 1)), dst = sbase + kSmSlot + (i & 1) * kSlotBytes;
    const int tc = static_cast<int>(f.t0), h = f.h;
    mbar_arrive_expect_tx(full, kSlotBytes + 512);
    tma_load_4d(dst, tq, 0, tc, 0, h, full);
    tma_load_4d(dst + 8192, tk, 0, tc, 0, h, full);
    tma_load_4d(dst + 16384, tg, 0, tc, 0, h, full);
    bulk_g2s(sbase + kSmBias + (i & 1) * 512, p.dt_bias + static_cast<size_t>(h) * kD, 512, full);
  };
  auto look_ahead = [&](int i, Info f) {
    f.ha = gate_factor(p, f.h);
    infos[i & (kInfos - 1)] = f;
  };
  auto item = [&](int i) { return decode<kSlice>(p, blockIdx.x + static_cast<unsigned>(i) * gridDim.x); };
  int loaded = 0;
  bool ok = true;
  if (lane == 0) {
    // the first items' loads before their gate factor, which has to come from memory; the barrier also waits for what is said about them
    for (int i = 0; i < 2 && i < n_it; ++i) {
      const Info f = item(i);
      const bool first_only = i == 1 && p.first_load_only;       // test aid: a wait that nothing completes
      if (!first_only) {
        load(i, f);
        ++loaded;
      }
      look_ahead(i, f);
      if (first_only) break;
      mbar_arrive(bar(B_IN + i));
    }
    if (n_it > 2) look_ahead(2, item(2));
  }
  __syncwarp();
  for (int i = 0; i < n_it; ++i) {
    const int b = i & 1;
    const uint32_t ph = (i >> 1) & 1;
    if (!warp_wait(bar(B_OPS + b), ph, abort_flag)) { ok = false; break; }
    const int h = infos[i & (kInfos - 1)].h, gc = infos[i & (kInfos - 1)].gc;
    uint8_t* rec = p.records + (static_cast<size_t>(h) * p.total_chunks + gc) * kCrBytes;
    if (lane == 0) {
      bulk_s2g(rec, sbase + kSmSlot + b * kSlotBytes, kSlotBytes);
      bulk_s2g(rec + kCrE, sbase + kSmE + b * 512, 512);
      bulk_commit();
      bulk_wait_read0();             // (also the tril(M) of the item before)
      if (i + 2 < n_it && !p.first_load_only) {
        load(i + 2, infos[(i + 2) & (kInfos - 1)]);
        mbar_arrive(bar(B_IN + b));
        ++loaded;
      }
      if (i + 3 < n_it) look_ahead(i + 3, item(i + 3));
    }
    __syncwarp();
    if (!warp_wait(bar(B_D1 + b), ph, abort_flag)) { ok = false; break; }
    tc_fence_after();
    uint32_t m[32];
    tmem_ld32(tmem + (32u << 16) + 32 * b, m);
    tmem_wait_ld();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(B_D1_FREE + b));
    uint8_t* row = smem + kSmMqk + b * 2048 + (lane >> 3) * 512 + (lane & 7) * 16;
#pragma unroll
    for (int cb = 0; cb < 4; ++cb) {
      uint32_t x[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int c = 8 * cb + 2 * e;
        x[e] = pack_bf16(c <= lane ? __uint_as_float(m[c]) : 0.f, c + 1 <= lane ? __uint_as_float(m[c + 1]) : 0.f);
      }
      *reinterpret_cast<uint4*>(row + cb * 128) = make_uint4(x[0], x[1], x[2], x[3]);
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      bulk_s2g(rec + kCrMQK, sbase + kSmMqk + b * 2048, 2048);
      bulk_commit();
    }
  }
  if (lane == 0) {
    bulk_wait_read0();
    if (!ok || *abort_flag > 0) {
      // (giving up) loads in flight must land before the CTA's shared memory goes away
      for (int k = loaded > 2 ? loaded - 2 : 0; k < loaded; ++k) {
        const uint64_t t0 = globaltimer_ns();
        while (!mbar_try_wait(bar(B_IN + (k & 1)), (k >> 1) & 1))
          if (globaltimer_ns() - t0 > 20000000ull) break;
      }
    }
  }
  return ok;
}

// The first products, and sigmoid(beta) beside them.
__device__ __forceinline__ bool product_role(const PrepParams& p, uint8_t* smem, uint32_t sbase, uint32_t tmem, int n_it, int lane,
                                             volatile int* abort_flag) {
  auto bar = [&](int i) { return sbase + kSmBars + 8 * i; };
  bool ok = true;
  int i = 0;
  tmem = __shfl_sync(0xffffffffu, tmem, 0);
  n_it = __shfl_sync(0xffffffffu, n_it, 0);
  for (; i < n_it; ++i) {
    const int b = i & 1;
    const uint32_t ph = (i >> 1) & 1;
    if (!warp_wait(bar(B_NORMP + b), ph, abort_flag)) { ok = false; break; }
    const Info* f = reinterpret_cast<const Info*>(smem + kSmInfo) + (i & (kInfos - 1));
    float beta = 0.f;
    if (lane < f->len) beta = __bfloat162float(p.beta[static_cast<size_t>(f->t0 + lane) * p.H + f->h]);
    if (!warp_wait(bar(B_OPS + b), ph, abort_flag)) { ok = false; break; }
    if (i >= 2 && !warp_wait(bar(B_D1_FREE + b), ((i >> 1) - 1) & 1, abort_flag)) { ok = false; break; }
    // (the inverse of item i - 4, which used this slot, ended before item i - 2 gave its result back)
    reinterpret_cast<float*>(smem + kSmBeta + (i & 3) * 128)[lane] = lane < f->len ? sigmoid_fast(beta) : 0.f;
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(B_D1 + b));
    if (elect_one()) {       // (operands that are plainly the same in all lanes: from one lane's branch a product costs 100 cycles to issue)
      // rows of the A operand: even items k+ | q+ from row 0 (A in lanes 0-31, M in 32-63); odd items, whose k+ lies behind
      // q+, from row 32 on (M in lanes 32-63, A in 64-95).  What the other rows hold does not matter: nobody reads their lanes.
      constexpr uint32_t idesc = umma_idesc_bf16(128, 32, 0, 0);
      tc_fence_after();
      const uint64_t a = umma_desc(sbase + kSmScr + (b ? 0 : 8192), 128, 2048), k = umma_desc(sbase + kSmScr, 128, 2048);
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) umma_ss(tmem + 32 * b, a + ks * 16, k + ks * 16, idesc, ks > 0);
      umma_commit(bar(B_D1 + b));
    }
    __syncwarp();
  }
  if (lane == 0 && i > 0) {
    // the commit issued last must land before the barrier's memory goes away
    const uint64_t t0 = globaltimer_ns();
    while (!mbar_try_wait(bar(B_D1 + ((i - 1) & 1)), ((i - 1) >> 1) & 1))
      if (globaltimer_ns() - t0 > (ok ? kWaitLimitNs : 20000000ull)) { ok = false; break; }
  }
  return ok;
}

// kSlice: a time slice of equal-length sequences (PrepParams::slice_*); the other form has fewer registers to hold
template <bool kSlice>
__global__ void __launch_bounds__(kThreads, 2)
operands_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_g,
                const PrepParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sbase = smem_u32(smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + kSmMisc + 4);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kSmMisc);
  auto bar = [&](int i) { return sbase + kSmBars + 8 * i; };
  if (tid == 0) {
    // the swizzled tiles need this alignment: report instead of computing garbage (below zero: a wait limit, test aid)
    *abort_flag = (sbase & 1023u) != 0u ? 1 : -p.wait_limit_us;
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(B_IN + i), 2);                     // the copies, and what is said about the item
      mbar_init(bar(B_NORMP + i), 8);
      mbar_init(bar(B_OPS + i), 8);
      mbar_init(bar(B_D1 + i), 2);                     // the commit, and the warp that leaves sigmoid(beta) beside it
      mbar_init(bar(B_D1_FREE + i), 2);
    }
    fence_mbar_init();
  }
  if (warp == 11) {
    tmem_alloc(smem_u32(tmem_slot), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  bool ok = *abort_flag <= 0;
  if (!kSlice || !p.beside) grid_dependency_wait();
  const unsigned items = static_cast<unsigned>(p.cu_seqlens != nullptr ? p.chunk_prefix[p.N] : kSlice ? p.N * p.slice_chunks : p.total_chunks) * static_cast<unsigned>(p.H);
  const int n_it = !ok || blockIdx.x >= items ? 0 : static_cast<int>((items - blockIdx.x + gridDim.x - 1) / gridDim.x);
  if (warp < 8) {
    if (!element_role(p, sbase, n_it, warp, lane, abort_flag)) ok = false;
  } else if (warp == 9) {
    if (!copy_role<kSlice>(p, &tm_q, &tm_k, &tm_g, smem, sbase, tmem, n_it, lane, abort_flag)) ok = false;
  } else if (warp == 11) {
    if (!product_role(p, smem, sbase, tmem, n_it, lane, abort_flag)) ok = false;
  } else {
    if (!inverse_role(p, smem, sbase, tmem, n_it, (warp - 8) >> 1, lane, abort_flag)) ok = false;
  }
  if (!ok || *abort_flag > 0) atomicCAS(p.status, kStatusOk, kStatusWaitTimeout);
  tc_fence_before();
  __syncthreads();
  if (warp == 11) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
  if (kSlice && p.beside && blockIdx.x == gridDim.x - 1) grid_dependency_wait();
}

}  // namespace operands

// one_per_cta: a CTA per item, so that no CTA reuses a buffer, accumulator or barrier phase (slower; the form to compare against)
cudaError_t launch_operands(const PrepParams& p, bool one_per_cta, cudaStream_t stream) {
  if (p.total_chunks == 0 || p.H == 0 || p.T_total == 0) return cudaSuccess;
  CUtensorMap tq, tk, tg;
  if (!make_map_halves(&tq, p.q, p.T_total, p.H) || !make_map_halves(&tk, p.k, p.T_total, p.H) || !make_map_halves(&tg, p.g, p.T_total, p.H)) return cudaErrorInvalidValue;
  const bool slice = p.slice_chunks != p.seq_chunks;
  auto kernel = slice ? operands::operands_kernel<true> : operands::operands_kernel<false>;
  static SmemOptIn opt_in[2];
  cudaError_t e = opt_in[slice].ensure(kernel, operands::kSmemBytes);
  if (e != cudaSuccess) return e;
  const long long items = (slice ? static_cast<long long>(p.N) * p.slice_chunks : static_cast<long long>(p.total_chunks)) * p.H;
  const long long slots = one_per_cta ? items : p.beside ? p.beside : 2ll * device_sm_count();
  return launch_after(kernel, static_cast<unsigned>(items < slots ? items : slots), operands::kThreads, operands::kSmemBytes,
                      stream, tq, tk, tg, p);
}

}  // namespace fkda
