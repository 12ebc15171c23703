// Inter-chunk recurrence of the KDA prefill over compact records: the state of a (sequence, head) chain in registers, the
// products on its copy on tcgen05.
//
// Replaces the reference's K2 (csrc/smxx/fwd_kernel2.cuh:115-839).  The rows v of S^T never meet each other in the
// recurrence, so four warps hold 32 rows each as fp32 mma.sync accumulator fragments:
//     R^T = v^T - S^T k+^T                     on tcgen05, together with S^T q+^T: A = the bf16 copy of the state in tensor
//                                              memory, B = k+ | q+ of the record                  [128 v x 64]
//     U^T = R^T (T diag(beta))^T               mma.sync; R^T is read from tensor memory in fragment layout
//     S^T = S^T diag(e) + U^T kr               mma.sync; A = U^T, the packed accumulators of the line above
//     O^T = S^T q+^T + U^T mqk^T               the second product on top of the first, tcgen05; four other warps write it
// With k+ and q+ in one operand the product on the chain costs the tensor cores no more than the output's alone, and it replaces
// nearly half of a warp's mma.sync.  What made it pay (4 x 8192 tokens x 32 heads, cycles per chunk by clock64):
//   * all of it on mma.sync but the output, which interrupts it: 2700 cycles, 0.342 ms; R^T on tcgen05 at first 2680;
//   * no wait for a store to tensor memory right behind it (200 cycles each): 2530;
//   * the products issued by a whole warp with operands that the compiler can see to be uniform (elect.sync) instead of from one
//     lane's branch, where each costs 75 cycles: 2230;
//   * one accumulator for both halves of k: 2140;
//   * the state's decay while the product on its copy is under way, not between the mma.sync of the update: 2040;
//   * the first half of the copy announced three quarters through the update: 2010.  0.280 ms in a burst of calls, 0.323 -
//     0.335 kept up under the power cap (0.342 and 0.372 - 0.378 before).
// Eight recurrence warps of 16 rows: 2700 (every operand is read twice as often); three groups of k instead of two: 0.325 ms; a
// part of the decay left in the update: 0.297.  What bounds it now is the chain itself, of which a warp works 1900 cycles: update 1090,
// the product's way through tensor memory 470, R and U 360.
//
// Warps 0-3: recurrence; 4-7: output, and one of them each the tcgen05 products and the copies.  The code of a
// recurrence warp and of the output warp on the same SM sub-partition together stay near 8 KB: beyond that a sub-partition's
// instruction cache misses and straight-line code runs at three cycles per instruction and warp at best.
#include "fkda_common.cuh"
#include "fkda_record.cuh"
#include "fkda_tma.cuh"

namespace fkda {
namespace recur {

constexpr int kThreads = 256;                      // two warps per SM sub-partition: 255 registers each
constexpr int kStages = 5;
constexpr int kStageBytes = 37 * 1024;             // v tile (two swizzled [32 tok][64 ch] halves) | record
static_assert(8192 + kCrBytes <= kStageBytes, "stage");
constexpr int kSmStg = kStages * kStageBytes;      // output staging: [32 tok][32 v] per output warp
constexpr int kStgStride = 80;                     // bytes per token: conflict-free stmatrix
constexpr int kInfos = 16;
constexpr int kSmInfo = kSmStg + 4 * 32 * kStgStride;
constexpr int kSmBars = kSmInfo + kInfos * 32;
constexpr int kSmMisc = kSmBars + 256;
constexpr int kWalkInfos = 8;                      // (persistent form) more than stages, and a walk has an item at least
constexpr int kClaimAhead = 6;                     // (persistent form) items left of a walk to copy when the next one is claimed
constexpr int kSmWalks = kSmMisc + 16;
constexpr int kSmem = kSmWalks + kWalkInfos * 48;
static_assert(kSmem <= 227 * 1024, "shared memory plan");
// tensor memory columns.  One copy of S and of U each: when the products of a chunk on S are complete, those of the chunk
// before on U are too (one thread issues both), and the state's copy may be written over.
constexpr uint32_t kTmemCols = 256;
constexpr uint32_t kColSb = 0;                     // 64: bf16 copy of S^T [v][k], two k per column
constexpr uint32_t kColUt = kColSb + 64;           // 16: bf16 U^T [v][tok]
constexpr uint32_t kColD = 128;                    // two chunks x 64: S^T k+^T | S^T q+^T [v][tok], O^T on top of the latter
static_assert(kColUt + 16 <= kColD && kColD + 128 <= kTmemCols, "tensor memory plan");
enum { B_FULL = 0, B_EMPTY = kStages, B_S = 2 * kStages /*[2] halves of k*/, B_R = B_S + 2, B_U = B_R + 1, B_O = B_U + 1 /*[2]*/, B_O_FREE = B_O + 2 /*[2]*/, B_LAST = B_O_FREE + 2, B_COUNT };
static_assert(B_COUNT * 8 <= 256, "barrier area");

__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}
__device__ __forceinline__ void tmem_st_16x128b_x4(uint32_t taddr, const uint32_t (&a)[4], const uint32_t (&b)[4]) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]),
               "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3])
               : "memory");
}

// What the copying thread says about a chunk (written before its stage's barrier is armed).
struct Info {
  long long out_off;   // element offset of the first token's row in `out`
  int len;             // valid tokens
  int flags;
  int walk;            // (persistent form) which WalkInfo
  int pad[3];
};
// What it says about a walk, so that the recurrence warps need not look the chain up again (three dependent loads).
struct WalkInfo {
  const void* init_base;
  void* fin_base;
  long long tokens;
  int nchunks, init_mode, fin_fp32, pad[3];
};
static_assert(sizeof(WalkInfo) == 48, "walk info");
static_assert(sizeof(Info) == 32, "info");
enum { kEnd = 1 };

// The bf16 copy of half of the state's columns into tensor memory.
__device__ __forceinline__ void put_copy(const float (&S)[2][16][4], uint32_t tq, int half, int vt) {
  uint32_t a[16];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    a[2 * j] = pack_bf16(S[vt][8 * half + j][0], S[vt][8 * half + j][1]);
    a[2 * j + 1] = pack_bf16(S[vt][8 * half + j][2], S[vt][8 * half + j][3]);
  }
  tmem_st_16x128b_x8(tq + (static_cast<uint32_t>(16 * vt) << 16) + kColSb + 32 * half, a);
}

// The chunks of one walk on the recurrence warps, from stage s (phase par) on; ready: that stage is known to be full; item: its index in the
// CTA's stream.  S: rows v = row0 + 16 vt + g (+ 8), columns 8 jt + 2 t, + 1.
__device__ __forceinline__ bool walk(float (&S)[2][16][4], uint8_t* smem, uint32_t sbase, uint32_t tq, int nchunks, int64_t tokens, int row0, int lane,
                                     volatile int* abort_flag, int& s, uint32_t& par, bool& ready, uint32_t item) {
  auto bar = [&](int i) { return sbase + kSmBars + 8 * i; };
  const int mi = lane >> 3, r = lane & 7, t = lane & 3;
  const uint32_t kr_lane = 8192 + kCrKR + mi * 2048 + r * 16;
  const uint32_t v_lane = (row0 >> 6) * 4096 + lane * 128;
  const uint32_t tb_lane = 8192 + kCrTB + r * 16;
  auto arrive_after_st = [&](int b) {
    tmem_wait_st();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(b));
  };
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    put_copy(S, tq, half, 0);
    put_copy(S, tq, half, 1);
    arrive_after_st(B_S + half);
  }
  for (int c = 0; c < nchunks; ++c, ++item) {
    if (!__all_sync(0xffffffffu, ready) && !warp_wait(bar(B_FULL + s), par, abort_flag)) return false;
    const uint32_t stage = sbase + s * kStageBytes;

    // R^T = v^T - S^T k+^T; T diag(beta) and the first of kr meanwhile
    float R[2][4][4];
    {
      uint32_t x[4][4];              // v^T: channel blocks of 8 rows; register = token block
#pragma unroll
      for (int i = 0; i < 4; ++i) ldsm_x4_trans(stage + v_lane + ((((row0 >> 3) + i) & 7) ^ r) * 16, x[i][0], x[i][1], x[i][2], x[i][3]);
      const int64_t left = tokens - static_cast<int64_t>(c) * kChunk;
      if (left < kChunk) {           // rows past the sequence end belong to somebody else
        const int len = static_cast<int>(left);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          const uint32_t keep = (8 * nt + 2 * t < len ? 0xffffu : 0u) | (8 * nt + 2 * t + 1 < len ? 0xffff0000u : 0u);
#pragma unroll
          for (int i = 0; i < 4; ++i) x[i][nt] &= keep;
        }
      }
#pragma unroll
      for (int vt = 0; vt < 2; ++vt)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          R[vt][nt][0] = bf_lo(x[2 * vt][nt]);
          R[vt][nt][1] = bf_hi(x[2 * vt][nt]);
          R[vt][nt][2] = bf_lo(x[2 * vt + 1][nt]);
          R[vt][nt][3] = bf_hi(x[2 * vt + 1][nt]);
        }
    }
    uint32_t l[4], m[4], n[4];       // T diag(beta): token tiles 0 and 1 (tokens 0-15 only: lower triangle), 2, 3
    ldsm_x4(stage + tb_lane + (mi >> 1) * 512 + (mi & 1) * 128, l[0], l[1], l[2], l[3]);
    ldsm_x4(stage + tb_lane + 1024 + mi * 128, m[0], m[1], m[2], m[3]);
    ldsm_x4(stage + tb_lane + 1536 + mi * 128, n[0], n[1], n[2], n[3]);
    uint32_t kr[2][4];
    ldsm_x4_trans(stage + kr_lane, kr[0][0], kr[0][1], kr[0][2], kr[0][3]);
    // and the state's decay: its copy has been taken
    const float2* e2 = reinterpret_cast<const float2*>(smem + s * kStageBytes + 8192 + kCrE) + t;
    bool there = false;
#pragma unroll
    for (int jt = 0; jt < 16; ++jt) {
      if (jt == 12) there = mbar_test(bar(B_R), item & 1u);
      const float2 e = e2[4 * jt];
#pragma unroll
      for (int vt = 0; vt < 2; ++vt) {
        uint32_t y[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) y[k] = __float_as_uint(S[vt][jt][k]);
        mul2(y[0], y[1], e);
        mul2(y[2], y[3], e);
#pragma unroll
        for (int k = 0; k < 4; ++k) S[vt][jt][k] = __uint_as_float(y[k]);
      }
    }
    if (!__all_sync(0xffffffffu, there) && !warp_wait(bar(B_R), item & 1u, abort_flag)) return false;
    tc_fence_after();
    uint32_t u[2][2][4];             // A fragments, k-step = 16 tokens: first of R^T, then of U^T
    auto as_operand = [&](uint32_t(&d)[2][4], const float(&x)[4][4]) {
#pragma unroll
      for (int ks = 0; ks < 2; ++ks)
#pragma unroll
        for (int e = 0; e < 4; ++e)  // e & 1: rows + 8, e >> 1: tokens + 8
          d[ks][e] = pack_bf16(x[2 * ks + (e >> 1)][2 * (e & 1)], x[2 * ks + (e >> 1)][2 * (e & 1) + 1]);
    };
    {
      const uint32_t d = tq + kColD + 64 * (item & 1u);
      uint32_t y[2][16];
#pragma unroll
      for (int vt = 0; vt < 2; ++vt) tmem_ld_16x256b_x4(d + (static_cast<uint32_t>(16 * vt) << 16), y[vt]);
      tmem_wait_ld();
#pragma unroll
      for (int vt = 0; vt < 2; ++vt) {
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e) R[vt][nt][e] += __uint_as_float(y[vt][4 * nt + e]);
        as_operand(u[vt], R[vt]);
      }
    }
    // U^T = R^T (T diag(beta))^T
    {
      float U[2][4][4];
#pragma unroll
      for (int vt = 0; vt < 2; ++vt) {
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) U[vt][nt][0] = U[vt][nt][1] = U[vt][nt][2] = U[vt][nt][3] = 0.f;
        mma_bf16_16816(U[vt][0], u[vt][0][0], u[vt][0][1], u[vt][0][2], u[vt][0][3], l[0], l[1]);
        mma_bf16_16816(U[vt][1], u[vt][0][0], u[vt][0][1], u[vt][0][2], u[vt][0][3], l[2], l[3]);
        mma_bf16_16816(U[vt][2], u[vt][0][0], u[vt][0][1], u[vt][0][2], u[vt][0][3], m[0], m[1]);
        mma_bf16_16816(U[vt][3], u[vt][0][0], u[vt][0][1], u[vt][0][2], u[vt][0][3], n[0], n[1]);
        mma_bf16_16816(U[vt][2], u[vt][1][0], u[vt][1][1], u[vt][1][2], u[vt][1][3], m[2], m[3]);
        mma_bf16_16816(U[vt][3], u[vt][1][0], u[vt][1][1], u[vt][1][2], u[vt][1][3], n[2], n[3]);
      }
#pragma unroll
      for (int vt = 0; vt < 2; ++vt) {
        as_operand(u[vt], U[vt]);
        tmem_st_16x128b_x4(tq + (static_cast<uint32_t>(16 * vt) << 16) + kColUt, u[vt][0], u[vt][1]);
      }
    }
    // S^T = S^T diag(e) + U^T kr, and the copy of it for the next chunk as its halves are done; the next stage's barrier is looked at meanwhile
    const int s1 = s + 1 == kStages ? 0 : s + 1;
    const uint32_t par1 = s1 == 0 ? par ^ 1u : par;
    const bool more = c + 1 < nchunks;
    ready = mbar_test(bar(B_FULL + s1), par1);
#pragma unroll
    for (int jt = 0; jt < 16; ++jt) {
      const uint32_t(&B)[4] = kr[jt & 1];
      if (jt < 15) {
        uint32_t(&N)[4] = kr[(jt + 1) & 1];
        ldsm_x4_trans(stage + kr_lane + (jt + 1) * 128, N[0], N[1], N[2], N[3]);
      }
#pragma unroll
      for (int ks = 0; ks < 2; ++ks)
#pragma unroll
        for (int vt = 0; vt < 2; ++vt)
          mma_bf16_16816(S[vt][jt], u[vt][ks][0], u[vt][ks][1], u[vt][ks][2], u[vt][ks][3], B[2 * ks], B[2 * ks + 1]);
      if (jt == 4) arrive_after_st(B_U);
      if (more) {
        if (jt == 8) put_copy(S, tq, 0, 0);
        if (jt == 9) put_copy(S, tq, 0, 1);
        if (jt == 13) arrive_after_st(B_S);
      }
    }
    if (more) {
      put_copy(S, tq, 1, 0);
      put_copy(S, tq, 1, 1);
      arrive_after_st(B_S + 1);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(B_EMPTY + s));
    s = s1;
    par = par1;
  }
  return true;
}

__device__ __forceinline__ void load_state(float (&S)[2][16][4], const ChainView& cv, int row0, int lane) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int vt = 0; vt < 2; ++vt) {
    const int v = row0 + 16 * vt + g;
    if (cv.init_mode == 1) {
      const float* src = static_cast<const float*>(cv.init_base) + v * kD + 2 * t;
#pragma unroll
      for (int jt = 0; jt < 16; ++jt) {
        const float2 lo = __ldg(reinterpret_cast<const float2*>(src + 8 * jt)), hi = __ldg(reinterpret_cast<const float2*>(src + 8 * kD + 8 * jt));
        S[vt][jt][0] = lo.x; S[vt][jt][1] = lo.y; S[vt][jt][2] = hi.x; S[vt][jt][3] = hi.y;
      }
    } else if (cv.init_mode == 2) {
      const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(cv.init_base) + v * kD + 2 * t;
#pragma unroll
      for (int jt = 0; jt < 16; ++jt) {
        const uint32_t lo = __ldg(reinterpret_cast<const uint32_t*>(src + 8 * jt)), hi = __ldg(reinterpret_cast<const uint32_t*>(src + 8 * kD + 8 * jt));
        S[vt][jt][0] = bf_lo(lo); S[vt][jt][1] = bf_hi(lo); S[vt][jt][2] = bf_lo(hi); S[vt][jt][3] = bf_hi(hi);
      }
    } else {
#pragma unroll
      for (int jt = 0; jt < 16; ++jt)
#pragma unroll
        for (int i = 0; i < 4; ++i) S[vt][jt][i] = 0.f;
    }
  }
}
__device__ __forceinline__ void store_state(const float (&S)[2][16][4], const ChainView& cv, int row0, int lane) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int vt = 0; vt < 2; ++vt) {
    const int v = row0 + 16 * vt + g;
    if (cv.fin_fp32) {
      float* dst = static_cast<float*>(cv.fin_base) + v * kD + 2 * t;
#pragma unroll
      for (int jt = 0; jt < 16; ++jt) {
        *reinterpret_cast<float2*>(dst + 8 * jt) = make_float2(S[vt][jt][0], S[vt][jt][1]);
        *reinterpret_cast<float2*>(dst + 8 * kD + 8 * jt) = make_float2(S[vt][jt][2], S[vt][jt][3]);
      }
    } else {
      __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(cv.fin_base) + v * kD + 2 * t;
#pragma unroll
      for (int jt = 0; jt < 16; ++jt) {
        *reinterpret_cast<uint32_t*>(dst + 8 * jt) = pack_bf16(S[vt][jt][0], S[vt][jt][1]);
        *reinterpret_cast<uint32_t*>(dst + 8 * kD + 8 * jt) = pack_bf16(S[vt][jt][2], S[vt][jt][3]);
      }
    }
  }
}

// (runs) The rows of a warp that hold an infinity or not-a-number, a bit each.
__device__ __forceinline__ uint32_t bad_rows(const float (&S)[2][16][4]) {
  uint32_t rows = 0;
#pragma unroll
  for (int vt = 0; vt < 2; ++vt)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      uint32_t most = 0;
#pragma unroll
      for (int jt = 0; jt < 16; ++jt)
#pragma unroll
        for (int k = 0; k < 2; ++k) most = max(most, __float_as_uint(S[vt][jt][2 * i + k]) & 0x7fffffffu);
      const uint32_t lanes = __ballot_sync(0xffffffffu, most >= 0x7f800000u);
#pragma unroll
      for (int g = 0; g < 8; ++g) rows |= (lanes >> (4 * g) & 15u) != 0u ? 1u << (16 * vt + 8 * i + g) : 0u;
    }
  return rows;
}

// (runs, at the end of a CTA) A row of S^T that holds an infinity or not-a-number once holds one to the end of its sequence, and every
// output of that channel is one: R = v - S k+, U and S e + U kr take in the whole row.  A map that was found to be zero says
// otherwise: the runs behind it start from its offset, whatever is in front.  So the last CTA of a chain to come here, where some run
// has left such rows, writes not-a-number over what the runs behind that one have made of them.  Other calls pay
// for an atomic at the end of each CTA: 0.8 to 1.4 us of 48 to 600.
__device__ __forceinline__ void spoil_runs(const ScanParams& p, float* slots, volatile int* last, bool bad) {
  const int tid = threadIdx.x;
  if (tid == 0) {
    int done;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], %2;" : "=r"(done) : "l"(seg_done_word(slots)), "r"(bad ? 1 + kSegBad : 1) : "memory");
    *last = (done & (kSegBad - 1)) == p.n_segs - 1 && (bad || done >= kSegBad);
  }
  __syncthreads();
  if (!*last) return;
  const ChainView cv = chain_view<false>(p, static_cast<int>(blockIdx.x) / p.n_segs);
  const int v = tid & (kD - 1), part = tid / kD, run_len = p.seg_chunks_dev != nullptr ? *p.seg_chunks_dev : p.seg_chunks;
  int run = 0;
  while (run < p.n_segs - 1 && !(__ldcg(seg_bad_rows(slots, run) + (v >> 5)) >> (v & 31) & 1u)) ++run;
  if (run == p.n_segs - 1) return;
  const int64_t chunk = static_cast<int64_t>(run + 1) * run_len, covered = cv.bos + static_cast<int64_t>(cv.nchunks) * kChunk;
  const int64_t end = covered < cv.eos ? covered : cv.eos;
  for (int64_t t = cv.bos + chunk * kChunk + part; t < end; t += kThreads / kD)
    p.out[(t * p.H + cv.h) * kD + v] = __ushort_as_bfloat16(0x7fff);
  if (cv.fin_base != nullptr && part == 0)
    for (int k = 0; k < kD; ++k) {
      if (cv.fin_fp32) static_cast<uint32_t*>(cv.fin_base)[v * kD + k] = 0x7fffffffu;
      else static_cast<uint16_t*>(cv.fin_base)[v * kD + k] = 0x7fffu;
    }
}

// kStream: the CTA is persistent and goes through its walks (whole chains) as
// one stream of chunks, so that records, v and state of the next walk are on their way while the last chunks of this one
// are computed.  Equal lengths: walks in turn, every other round backwards; packed batches take the next longest
// sequence from a device counter.  Otherwise one walk per CTA: a chunk costs 5 to 8 % less (768 chains of 64 chunks 467 against 500
// us), a walk up to 3 us more.
// kSlice: one walk per CTA, a time slice of it (ScanParams::slice_*).
template <bool kSeg, bool kStream, bool kSlice>
__global__ void __launch_bounds__(kThreads, 1) recur_kernel(const __grid_constant__ CUtensorMap tm_v, const ScanParams p, const int walks) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sbase = smem_u32(smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + kSmMisc + 4);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kSmMisc);
  Info* infos = reinterpret_cast<Info*>(smem + kSmInfo);
  auto bar = [&](int i) { return sbase + kSmBars + 8 * i; };
  // (runs) whether some rows are not finite at the end, the chain's slots (unless the recurrence could not begin)
  volatile int* bad = reinterpret_cast<volatile int*>(smem + kSmMisc + 8);
  float** chain_slots = reinterpret_cast<float**>(smem + kSmWalks);
  if (tid == 0) {
    // the swizzled tiles need this alignment: report instead of computing garbage (below zero: a wait limit, test aid)
    *abort_flag = (sbase & 1023u) != 0u ? 1 : -p.wait_limit_us;
    *bad = 0;
    if (kSeg) *chain_slots = nullptr;
    for (int s = 0; s < kStages; ++s) {
      mbar_init(bar(B_FULL + s), 1);
      mbar_init(bar(B_EMPTY + s), 4 + 1);              // recurrence warps + commit of the products on U
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(B_S + i), 4);
      mbar_init(bar(B_O + i), 1);
      mbar_init(bar(B_O_FREE + i), 4);
    }
    mbar_init(bar(B_R), 1);
    mbar_init(bar(B_LAST), 1);
    mbar_init(bar(B_U), 4);
    fence_mbar_init();
  }
  if (warp == 4) {
    tmem_alloc(smem_u32(tmem_slot), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot, utmem = __shfl_sync(0xffffffffu, tmem, 0);
  bool ok = *abort_flag <= 0;
  grid_dependency_wait();
  if (p.release_next) grid_release_next();

  if (warp < 4) {
    // ===== recurrence ================================================================================================
    const int row0 = 32 * warp;
    const uint32_t tq = tmem + (static_cast<uint32_t>(row0) << 16);
    float S[2][16][4];
    int s = 0;
    uint32_t par = 0;
    bool ready = false;
    for (int i = 0; ok;) {
      ChainView cv{};
      if (kStream) {
        if (!__all_sync(0xffffffffu, ready) && !warp_wait(bar(B_FULL + s), par, abort_flag)) { ok = false; break; }
        const volatile Info* f = infos + (i & (kInfos - 1));
        ready = true;
        if (f->flags & kEnd) break;
        const WalkInfo* wi = reinterpret_cast<const WalkInfo*>(smem + kSmWalks) + f->walk;
        cv.init_base = wi->init_base;
        cv.init_mode = wi->init_mode;
        cv.fin_base = wi->fin_base;
        cv.fin_fp32 = wi->fin_fp32;
        cv.bos = 0;
        cv.eos = wi->tokens;
        cv.nchunks = wi->nchunks;
      } else {
        cv = chain_view<kSeg, kSlice>(p, static_cast<int>(blockIdx.x));
      }
      load_state(S, cv, row0, lane);
      // (an empty run hands its state through)
      if (cv.nchunks > 0) ok = walk(S, smem, sbase, tq, cv.nchunks, cv.eos - cv.bos, row0, lane, abort_flag, s, par, ready, static_cast<uint32_t>(i));
      if (ok && cv.fin_base != nullptr) store_state(S, cv, row0, lane);
      if (kSeg) {
        const uint32_t rows = ok ? bad_rows(S) : 0u;
        if (lane == 0) {
          float* slots = p.seg_buf + (static_cast<size_t>(cv.n) * p.H + cv.h) * p.n_segs * 3 * kSegSlotFloats;
          seg_bad_rows(slots, static_cast<int>(blockIdx.x) % p.n_segs)[warp] = rows;
          if (rows != 0u) *bad = 1;
          if (warp == 0) *chain_slots = slots;
        }
      }
      if (!kStream) break;
      i += cv.nchunks;
    }
  } else {
    const int w = warp - 4, mi = lane >> 3, r = lane & 7;
    const uint32_t tq = tmem + (static_cast<uint32_t>(32 * w) << 16) + kColD + 32;
    const uint32_t stg = sbase + kSmStg + w * 32 * kStgStride;
    const uint8_t* src = smem + kSmStg + w * 32 * kStgStride + (lane >> 2) * kStgStride + (lane & 3) * 16;
    __nv_bfloat16* const out0 = p.out + static_cast<size_t>(lane >> 2) * p.H * kD + 32 * w + (lane & 3) * 8;
    const size_t step = static_cast<size_t>(8) * p.H * kD;      // eight tokens on

    // ===== one lane of the second warp: the stream of chunks into the ring ==========================================
    struct { long long bos, eos; const uint8_t* rec; int walk, h, c, n, turn; bool ended; } cur{};
    // The next walk, looked up a step per item (a packed batch: the counter, the order by length, then the sequence's ends and first record
    // are loads that depend on one another; in a row they would keep this warp's output waiting for more than a chunk's time).  Not
    // before the walk's last items: what a CTA holds nobody else can take, and walks are handed out longest first.  With the look-up begun at
    // a walk's second item one SM had a sequence of 6400 tokens behind the one of 16384: 16384 + 4 x 6400 + 60 x 64 tokens on 32
    // heads 1283 us, now 1056; 96 decode tokens among four prompts 236.2 -> 237.3.  Three items ahead, one for each step, 200
    // short sequences need 417 us, as the last step's loads are waited for; six ahead 414.5.
    struct { ChainView cv; int walk, step; } next{};
    auto look = [&]() {
      if (!kStream || next.step >= 3) return;
      if (next.step == 0) {
        const int base = cur.turn * static_cast<int>(gridDim.x);
        next.walk = p.next_walk != nullptr ? atomicAdd(p.next_walk, 1)
                    : base + ((cur.turn & 1) ? static_cast<int>(gridDim.x - 1 - blockIdx.x) : static_cast<int>(blockIdx.x));
        ++cur.turn;
      } else if (next.walk >= walks || next.walk < 0) {
        next.step = 2;
      } else if (next.step == 1) {
        const int slot = next.walk / p.H;
        next.cv.h = next.walk - slot * p.H;
        next.cv.n = p.seq_order != nullptr ? p.seq_order[slot] : slot;
      } else if (p.cu_seqlens != nullptr) {
        next.cv.bos = p.cu_seqlens[next.cv.n];
        next.cv.eos = p.cu_seqlens[next.cv.n + 1];
        next.cv.chunk_base = p.chunk_prefix[next.cv.n];
      } else {
        next.cv.bos = static_cast<int64_t>(next.cv.n) * p.T;
        next.cv.eos = next.cv.bos + p.T;
        next.cv.chunk_base = next.cv.n * static_cast<int>((p.T + kChunk - 1) / kChunk);
      }
      ++next.step;
    };
    int copied = 0;
    int cs = 0;                        // stage of the next item
    auto copy = [&]() {
      const int s = cs;
      if (p.stop_copies_after > 0 && copied >= p.stop_copies_after) return;      // test aid: the next wait for a record runs out
      Info* f = infos + (copied & (kInfos - 1));
      if (cur.c == cur.n) {            // the next walk
        if (!kStream && cur.turn > 0) {
          cur.ended = true;
          return;
        }
        for (;;) {
          ChainView cv{};
          bool past = false;
          if (kStream) {
            while (next.step < 3) look();
            next.step = 0;
            past = next.walk >= walks || next.walk < 0;
            if (!past) {
              cv = next.cv;
              cv.bos = cv.bos < 0 ? 0 : (cv.bos > p.T_total ? p.T_total : cv.bos);
              cv.eos = cv.eos < cv.bos ? cv.bos : (cv.eos > p.T_total ? p.T_total : cv.eos);
              chain_finish<false>(p, cv, 0, 0);
            }
          } else {
            ++cur.turn;
            cv = chain_view<kSeg, kSlice>(p, static_cast<int>(blockIdx.x));
          }
          if (past || (kStream && cv.nchunks == 0 && p.N <= kOrderMax)) {
            // (The last round may be shorter than the grid: a CTA without a walk in it is done, there is no round after it.
            // Skipped sequences come last in the order by length.)
            cur.ended = true;
            f->flags = kEnd;
            mbar_arrive(bar(B_FULL + s));
            if (++cs == kStages) cs = 0;
            ++copied;
            return;
          }
          if (kStream && cv.nchunks == 0) continue;
          cur.walk = (cur.walk + 1) & (kWalkInfos - 1);
          cur.h = cv.h;
          cur.bos = cv.bos;
          cur.eos = cv.eos;
          cur.c = 0;
          cur.n = cv.nchunks;
          cur.rec = p.records + (static_cast<size_t>(cv.h) * p.total_chunks + cv.chunk_base) * kCrBytes;
          if (kStream) {
            WalkInfo* wi = reinterpret_cast<WalkInfo*>(smem + kSmWalks) + cur.walk;
            wi->init_base = cv.init_base;
            wi->init_mode = cv.init_mode;
            wi->fin_base = cv.fin_base;
            wi->fin_fp32 = cv.fin_fp32;
            wi->tokens = cv.eos - cv.bos;
            wi->nchunks = cv.nchunks;
          }
          if (copied > 0 && (cv.init_mode == 1 || cv.init_mode == 2)) bulk_prefetch_l2(cv.init_base, kD * kD * (cv.init_mode == 1 ? 4 : 2));
          break;
        }
      } else if (cur.n - cur.c <= kClaimAhead) {
        look();
      }
      const long long t0 = cur.bos + static_cast<long long>(cur.c) * kChunk;
      f->out_off = (t0 * p.H + cur.h) * kD;
      f->len = cur.eos - t0 < kChunk ? static_cast<int>(cur.eos - t0) : kChunk;
      f->walk = cur.walk;
      f->flags = 0;
      const uint32_t dst = sbase + s * kStageBytes;
      mbar_arrive_expect_tx(bar(B_FULL + s), kCrBytes + 8192);
      bulk_g2s(dst + 8192, cur.rec + static_cast<size_t>(cur.c) * kCrBytes, kCrBytes, bar(B_FULL + s));
      tma_load_3d(dst, &tm_v, 0, cur.h, static_cast<int>(t0), bar(B_FULL + s));
      tma_load_3d(dst + 4096, &tm_v, 64, cur.h, static_cast<int>(t0), bar(B_FULL + s));
      ++cur.c;
      ++copied;
      if (++cs == kStages) cs = 0;
    };
    int n_one = 0;                     // (one walk per CTA) its items
    if (!kStream) n_one = chain_view<kSeg, kSlice>(p, static_cast<int>(blockIdx.x)).nchunks;
    const bool work = kStream || n_one > 0;
    if (w == 1 && lane == 0 && ok && work)
      for (int k = 0; k < kStages && !cur.ended; ++k) copy();

    // ===== the first warp: S^T [k+; q+]^T of an item as soon as the copy of S is there, half of k by half; later O^T = S^T q+^T +
    // U^T mqk^T on top of it.  The output of the item before lies between the two.  (All lanes go through this, with operands
    // that the compiler can see to be the same in all of them: issued from one lane's branch a product costs 75 cycles.) =====
    int ps = 0, items = 0;             // stage of the item, with its phase; items begun
    uint32_t ps_par = 0;
    bool ended = false;
    const uint64_t desc_s = umma_desc(sbase + 8192 + kCrKN, 128, 2048), desc_u = umma_desc(sbase + 8192 + kCrMQK, 128, 512);
    auto products_s = [&](int i) -> bool {
      constexpr uint32_t idesc = umma_idesc_bf16(128, 64, 0, 0);
      if (!warp_wait(bar(B_FULL + ps), ps_par, abort_flag)) return false;
      if (kStream && (static_cast<const volatile Info*>(infos)[i & (kInfos - 1)].flags & kEnd)) {
        if (lane == 0) mbar_arrive(bar(B_O + (i & 1)));
        ended = true;
        return true;
      }
      if (i >= 2 && !warp_wait(bar(B_O_FREE + (i & 1)), ((i >> 1) - 1) & 1, abort_flag)) return false;
      const uint32_t d = utmem + kColD + 64 * (i & 1);
      const uint64_t b = desc_s + static_cast<uint32_t>(ps * (kStageBytes >> 4));
      items = i + 1;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        if (!warp_wait(bar(B_S + half), i & 1, abort_flag)) return false;
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_ts(d, utmem + kColSb + 32 * half + 8 * k, b + (4 * half + k) * 16, idesc, half + k > 0);
          if (half == 1) umma_commit(bar(B_R));
        }
        __syncwarp();
      }
      return true;
    };
    auto products_u = [&](int i) -> bool {
      constexpr uint32_t idesc = umma_idesc_bf16(128, 32, 0, 0);
      if (!warp_wait(bar(B_U), i & 1, abort_flag)) return false;
      tc_fence_after();
      const uint64_t b = desc_u + static_cast<uint32_t>(ps * (kStageBytes >> 4));
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) umma_ts(utmem + kColD + 64 * (i & 1) + 32, utmem + kColUt + 8 * ks, b + ks * 16, idesc, 1);
        umma_commit(bar(B_O + (i & 1)));
        umma_commit(bar(B_EMPTY + ps));
      }
      __syncwarp();
      if (++ps == kStages) { ps = 0; ps_par ^= 1u; }
      return true;
    };

    int o = 0, es = 0;                 // output buffer and stage of the item whose output is written, with their phases
    uint32_t o_par = 0, es_par = 0;
    for (int i = 0; kStream || i <= n_one; ++i) {
      const bool begin = kStream ? !ended : i < n_one;
      if (w == 0 && ok && begin) ok = products_s(i);
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      if (i > 0) {
        if (!__all_sync(0xffffffffu, mbar_wait_parked(bar(B_O + o), o_par, abort_flag))) { ok = false; break; }
        const volatile Info* f = infos + ((i - 1) & (kInfos - 1));
        if (kStream && (f->flags & kEnd)) break;
        const long long off = f->out_off;
        const int len = f->len;
        tc_fence_after();
        uint32_t y[2][16];
        tmem_ld_16x256b_x4(tq + 64 * o, y[0]);
        tmem_ld_16x256b_x4(tq + (16u << 16) + 64 * o, y[1]);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(B_O_FREE + o));
#pragma unroll
        for (int vt = 0; vt < 2; ++vt)
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const uint32_t* x = y[vt] + 8 * k;
            auto pk2 = [&](int e) { return pack_bf16(__uint_as_float(x[e]), __uint_as_float(x[e + 1])); };
            stsm_x4_trans(stg + (8 * (2 * k + (mi >> 1)) + r) * kStgStride + vt * 32 + (mi & 1) * 16, pk2(0), pk2(2), pk2(4), pk2(6));
          }
        __syncwarp();
        __nv_bfloat16* dst = out0 + off;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (8 * k + (lane >> 2) < len) *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(src + 8 * k * kStgStride);
          dst += step;
        }
        __syncwarp();
        if (w == 1 && lane == 0 && !cur.ended) {
          if (!mbar_wait_parked(bar(B_EMPTY + es), es_par, abort_flag)) ok = false;
          else copy();
        }
        if (++o == 2) { o = 0; o_par ^= 1u; }
        if (++es == kStages) { es = 0; es_par ^= 1u; }
      }
      if (w == 0 && ok && begin && !ended) ok = products_u(i);
    }
    if (w == 0 && items > 0 && elect_one()) {
      // what was issued must land before the CTA may exit: a commit behind all of it
      umma_commit(bar(B_LAST));
      const uint64_t t0 = globaltimer_ns();
      while (!mbar_try_wait(bar(B_LAST), 0))
        if (globaltimer_ns() - t0 > (ok ? kWaitLimitNs : 20000000ull)) { ok = false; break; }
    }
    if (w == 1 && lane == 0 && (!ok || *abort_flag > 0)) {
      // (giving up) copies in flight must land before the CTA's shared memory goes away
      for (int c = copied > kStages ? copied - kStages : 0; c < copied; ++c) {
        const uint64_t t0 = globaltimer_ns();
        while (!mbar_try_wait(bar(B_FULL + c % kStages), (c / kStages) & 1))
          if (globaltimer_ns() - t0 > 20000000ull) break;
      }
    }
  }
  if (!ok || *abort_flag > 0) atomicCAS(p.status, kStatusOk, kStatusWaitTimeout);
  tc_fence_before();
  __syncthreads();
  if (warp == 4) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
  if (kSeg && *chain_slots != nullptr) spoil_runs(p, *chain_slots, reinterpret_cast<volatile int*>(smem + kSmMisc + 12), *bad != 0);
}

// ---- maps of runs (fkda_segscan.cu) ---------------------------------------------------------------------------------------
// A CTA per (chain, run but the last): first the run's transition map M, from its last chunk to its first, then its offset N,
// the walk from a zero state.  Walked backwards, Q <- Q Phi^T from the identity, the rows of M^T = Q never meet each other either, and
// after c chunks Q is the map of the run's last c chunks: once it is zero to the last bit (103 nats of decay; a few hundred
// tokens of ordinary gates), so is M, and nothing finite in front of those chunks can be seen behind the run (spoil_runs sees to the rest).  Both walks then end there:
// what they cost is a handful of chunks instead of two runs, and chaining such runs costs nothing at all.  A run
// whose gates hold some channel to the end costs what it always did, a walk each for M and N, plus the test for zero (a hundred
// cycles in the first sixteen chunks and then in every eighth).
// 8 heads of 131072 tokens (lower_bound -2), recurrence with all its passes: 820 -> 340 us, 795 with gates that never decay; 16
// heads of 32768 tokens, the whole call: 619 -> 365 us (610); the walks themselves have become faster since (281 and 733 us).  (Few
// chains where nothing decays: kPair below.)
// One chunk of a walk without outputs, from stage s, every product on mma.sync.  `ready`: whether the next stage is full already.
// kBack: the transposed step, S^T Phi^T with Phi = diag(e) + kn^T TB^T kr the chunk's transition and no v: the same products with k+ and
// kr exchanged and TB transposed.
template <bool kBack>
__device__ __forceinline__ void step(float (&S)[2][16][4], uint8_t* smem, uint32_t sbase, int s, int len, int row0, int lane, uint32_t next_full,
                                     uint32_t next_par, bool& ready) {
  const int mi = lane >> 3, r = lane & 7, t = lane & 3;
  const uint32_t kn_lane = 8192 + (kBack ? kCrKR : kCrKN) + (mi >> 1) * 2048 + (mi & 1) * 128 + r * 16;
  const uint32_t kr_lane = 8192 + (kBack ? kCrKN : kCrKR) + mi * 2048 + r * 16;
  const uint32_t v_lane = (row0 >> 6) * 4096 + lane * 128;
  const uint32_t tb_lane = 8192 + kCrTB + r * 16;
  const uint32_t stage = sbase + s * kStageBytes;

  // R^T = v^T - S^T k+^T: the accumulators start from v^T; operands of a k-step are loaded during the one before
  float R[2][4][4];
  if (kBack) {
#pragma unroll
    for (int vt = 0; vt < 2; ++vt)
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) R[vt][nt][0] = R[vt][nt][1] = R[vt][nt][2] = R[vt][nt][3] = 0.f;
  } else {
    uint32_t x[4][4];              // v^T: channel blocks of 8 rows; register = token block
#pragma unroll
    for (int i = 0; i < 4; ++i) ldsm_x4_trans(stage + v_lane + ((((row0 >> 3) + i) & 7) ^ r) * 16, x[i][0], x[i][1], x[i][2], x[i][3]);
    if (len < kChunk) {            // rows past the sequence end belong to somebody else
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const uint32_t keep = (8 * nt + 2 * t < len ? 0xffffu : 0u) | (8 * nt + 2 * t + 1 < len ? 0xffff0000u : 0u);
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i][nt] &= keep;
      }
    }
#pragma unroll
    for (int vt = 0; vt < 2; ++vt)
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        R[vt][nt][0] = bf_lo(x[2 * vt][nt]);
        R[vt][nt][1] = bf_hi(x[2 * vt][nt]);
        R[vt][nt][2] = bf_lo(x[2 * vt + 1][nt]);
        R[vt][nt][3] = bf_hi(x[2 * vt + 1][nt]);
      }
  }
  uint32_t bb[2][8];
  ldsm_x4(stage + kn_lane, bb[0][0], bb[0][1], bb[0][2], bb[0][3]);
  ldsm_x4(stage + kn_lane + 4096, bb[0][4], bb[0][5], bb[0][6], bb[0][7]);
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    uint32_t a[2][16];               // bf16 copy of the state: A fragments of four k-steps
#pragma unroll
    for (int vt = 0; vt < 2; ++vt)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        a[vt][2 * j] = pack_bf16(S[vt][8 * half + j][0], S[vt][8 * half + j][1]);
        a[vt][2 * j + 1] = pack_bf16(S[vt][8 * half + j][2], S[vt][8 * half + j][3]);
      }
#pragma unroll
    for (int k4 = 0; k4 < 4; ++k4) {
      const int ks = 4 * half + k4;
      const uint32_t(&B)[8] = bb[ks & 1];
      if (ks < 7) {
        uint32_t(&N)[8] = bb[(ks + 1) & 1];
        ldsm_x4(stage + kn_lane + (ks + 1) * 256, N[0], N[1], N[2], N[3]);
        ldsm_x4(stage + kn_lane + 4096 + (ks + 1) * 256, N[4], N[5], N[6], N[7]);
      }
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int vt = 0; vt < 2; ++vt)
          mma_bf16_16816(R[vt][nt], a[vt][4 * k4], a[vt][4 * k4 + 1], a[vt][4 * k4 + 2], a[vt][4 * k4 + 3], B[2 * nt], B[2 * nt + 1]);
    }
  }
  // U^T = R^T (T diag(beta))^T
  uint32_t l[4], m[4], n[4];       // T diag(beta): token tiles 0 and 1 (tokens 0-15 only: lower triangle), 2, 3; transposed: 0, 1, 2 and 3 (16-31 only)
  if (kBack) {
    ldsm_x4_trans(stage + tb_lane + mi * 512, l[0], l[1], l[2], l[3]);
    ldsm_x4_trans(stage + tb_lane + mi * 512 + 128, m[0], m[1], m[2], m[3]);
    ldsm_x4_trans(stage + tb_lane + 1024 + (mi & 1) * 512 + 256 + (mi >> 1) * 128, n[0], n[1], n[2], n[3]);
  } else {
    ldsm_x4(stage + tb_lane + (mi >> 1) * 512 + (mi & 1) * 128, l[0], l[1], l[2], l[3]);
    ldsm_x4(stage + tb_lane + 1024 + mi * 128, m[0], m[1], m[2], m[3]);
    ldsm_x4(stage + tb_lane + 1536 + mi * 128, n[0], n[1], n[2], n[3]);
  }
  uint32_t kr[2][4];
  ldsm_x4_trans(stage + kr_lane, kr[0][0], kr[0][1], kr[0][2], kr[0][3]);
  uint32_t u[2][2][4];             // A fragments, k-step = 16 tokens: first of R^T, then of U^T
  auto as_operand = [&](uint32_t(&d)[2][4], const float(&x)[4][4]) {
#pragma unroll
    for (int ks = 0; ks < 2; ++ks)
#pragma unroll
      for (int e = 0; e < 4; ++e)  // e & 1: rows + 8, e >> 1: tokens + 8
        d[ks][e] = pack_bf16(x[2 * ks + (e >> 1)][2 * (e & 1)], x[2 * ks + (e >> 1)][2 * (e & 1) + 1]);
  };
#pragma unroll
  for (int vt = 0; vt < 2; ++vt) as_operand(u[vt], R[vt]);
  {
    float U[2][4][4];
#pragma unroll
    for (int vt = 0; vt < 2; ++vt) {
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) U[vt][nt][0] = U[vt][nt][1] = U[vt][nt][2] = U[vt][nt][3] = 0.f;
      if (kBack) {
        mma_bf16_16816(U[vt][0], u[vt][0][0], u[vt][0][1], u[vt][0][2], u[vt][0][3], l[0], l[1]);
        mma_bf16_16816(U[vt][1], u[vt][0][0], u[vt][0][1], u[vt][0][2], u[vt][0][3], m[0], m[1]);
        mma_bf16_16816(U[vt][2], u[vt][1][0], u[vt][1][1], u[vt][1][2], u[vt][1][3], n[0], n[1]);
        mma_bf16_16816(U[vt][3], u[vt][1][0], u[vt][1][1], u[vt][1][2], u[vt][1][3], n[2], n[3]);
        mma_bf16_16816(U[vt][0], u[vt][1][0], u[vt][1][1], u[vt][1][2], u[vt][1][3], l[2], l[3]);
        mma_bf16_16816(U[vt][1], u[vt][1][0], u[vt][1][1], u[vt][1][2], u[vt][1][3], m[2], m[3]);
      } else {
        mma_bf16_16816(U[vt][0], u[vt][0][0], u[vt][0][1], u[vt][0][2], u[vt][0][3], l[0], l[1]);
        mma_bf16_16816(U[vt][1], u[vt][0][0], u[vt][0][1], u[vt][0][2], u[vt][0][3], l[2], l[3]);
        mma_bf16_16816(U[vt][2], u[vt][0][0], u[vt][0][1], u[vt][0][2], u[vt][0][3], m[0], m[1]);
        mma_bf16_16816(U[vt][3], u[vt][0][0], u[vt][0][1], u[vt][0][2], u[vt][0][3], n[0], n[1]);
        mma_bf16_16816(U[vt][2], u[vt][1][0], u[vt][1][1], u[vt][1][2], u[vt][1][3], m[2], m[3]);
        mma_bf16_16816(U[vt][3], u[vt][1][0], u[vt][1][1], u[vt][1][2], u[vt][1][3], n[2], n[3]);
      }
    }
#pragma unroll
    for (int vt = 0; vt < 2; ++vt) as_operand(u[vt], U[vt]);
  }
  // S^T = S^T diag(e) + U^T kr; the next stage's barrier is looked at meanwhile
  const float2* e2 = reinterpret_cast<const float2*>(smem + s * kStageBytes + 8192 + kCrE) + t;
  ready = mbar_test(next_full, next_par);
#pragma unroll
  for (int jt = 0; jt < 16; ++jt) {
    const uint32_t(&B)[4] = kr[jt & 1];
    if (jt < 15) {
      uint32_t(&N)[4] = kr[(jt + 1) & 1];
      ldsm_x4_trans(stage + kr_lane + (jt + 1) * 128, N[0], N[1], N[2], N[3]);
    }
    const float2 e = e2[4 * jt];
#pragma unroll
    for (int vt = 0; vt < 2; ++vt) {
      uint32_t y[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) y[k] = __float_as_uint(S[vt][jt][k]);
      mul2(y[0], y[1], e);
      mul2(y[2], y[3], e);
#pragma unroll
      for (int k = 0; k < 4; ++k) S[vt][jt][k] = __uint_as_float(y[k]);
    }
#pragma unroll
    for (int ks = 0; ks < 2; ++ks)
#pragma unroll
      for (int vt = 0; vt < 2; ++vt)
        mma_bf16_16816(S[vt][jt], u[vt][ks][0], u[vt][ks][1], u[vt][ks][2], u[vt][ks][3], B[2 * ks], B[2 * ks + 1]);
  }
}

__device__ __forceinline__ bool is_zero(const float (&S)[2][16][4]) {
  uint32_t any = 0;
#pragma unroll
  for (int vt = 0; vt < 2; ++vt)
#pragma unroll
    for (int jt = 0; jt < 16; ++jt)
#pragma unroll
      for (int k = 0; k < 4; ++k) any |= __float_as_uint(S[vt][jt][k]);
  return !__any_sync(0xffffffffu, (any << 1) != 0u);
}

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Into another CTA's shared memory, at the place that `smem` is here.
__device__ __forceinline__ void cluster_store(uint32_t smem, uint32_t cta, int x) {
  asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, %1;\n\tst.relaxed.cluster.shared::cluster.b32 [a], %2;\n\t}" ::"r"(smem), "r"(cta), "r"(x) : "memory");
}

// kPair: a cluster of two CTAs per run.  The first one does as above but for the offset of a run whose map lasts, which the second
// one walks beside it from the run's first chunk; it leaves off when the first one tells it that the map has vanished.  Taken where all
// clusters are resident at once: there M and N in turn are the longest path of a call whose gates hold.  Whole calls without
// decay, M and N in turn and beside one another, heads x tokens: 1 x 4096 80.0 -> 69.8 us, 1 x 16384 in 32 runs 132.6 -> 117.1, 2 x 22400 in 37
// 161.6 -> 144.5, 4 x 4128 85.1 -> 74.6, 1 x 131072 in 75 359.1 -> 307.4; where maps vanish the cluster costs 0.6 to 2.8 us.  (Runs of
// more CTAs than that gain nothing: the second round is as long as the second walk.)
template <bool kPair>
__global__ void __launch_bounds__(kThreads, 1) maps_kernel(const __grid_constant__ CUtensorMap tm_v, const ScanParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sbase = smem_u32(smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool offset_only = kPair && (blockIdx.x & 1u) != 0u;     // (the cluster's second CTA)
  const int block = static_cast<int>(kPair ? blockIdx.x >> 1 : blockIdx.x);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + kSmMisc + 4);
  int* zeros = reinterpret_cast<int*>(smem + kSmMisc + 8);       // warps whose rows of the map are zero (second CTA: 4 once the first has said so) ...
  int* longest = reinterpret_cast<int*>(smem + kSmMisc + 12);    // ... after so many chunks
  Info* infos = reinterpret_cast<Info*>(smem + kSmInfo);
  constexpr int B_TURN = B_U;                                    // M is done, N may be fetched
  auto bar = [&](int i) { return sbase + kSmBars + 8 * i; };
  if (tid == 0) {
    *abort_flag = (sbase & 1023u) != 0u ? 1 : -p.wait_limit_us;
    *zeros = 0;
    *longest = 0;
    for (int s = 0; s < kStages; ++s) {
      mbar_init(bar(B_FULL + s), 1);
      mbar_init(bar(B_EMPTY + s), 4);
    }
    mbar_init(bar(B_TURN), 4);
    fence_mbar_init();
  }
  if (kPair) cluster_sync();
  else __syncthreads();
  bool ok = *abort_flag <= 0;
  grid_dependency_wait();
  const ChainView cv = chain_view<true>(p, block);
  const int n = ok ? cv.nchunks : 0, run = block % (p.n_segs - 1);
  if (warp < 4) {
    float* slots = p.seg_buf + (static_cast<size_t>(cv.n) * p.H + cv.h) * p.n_segs * 3 * kSegSlotFloats;
    const int row0 = 32 * warp, g = lane >> 2, t = lane & 3;
    float S[2][16][4];
    auto fill = [&](float diagonal) {
#pragma unroll
      for (int vt = 0; vt < 2; ++vt)
#pragma unroll
        for (int jt = 0; jt < 16; ++jt)
#pragma unroll
          for (int i = 0; i < 4; ++i) S[vt][jt][i] = 8 * jt + 2 * t + (i & 1) == row0 + 16 * vt + g + 8 * (i >> 1) ? diagonal : 0.f;
    };
    int s = 0;
    uint32_t par = 0;
    bool ready = false, zero = false;
    auto next = [&](int& s1, uint32_t& par1) {
      s1 = s + 1 == kStages ? 0 : s + 1;
      par1 = s1 == 0 ? par ^ 1u : par;
    };
    auto release = [&](int s1, uint32_t par1) {
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(B_EMPTY + s));
      s = s1;
      par = par1;
    };
    fill(1.f);
    for (int c = 0; ok && !offset_only; ++c) {
      if (!__all_sync(0xffffffffu, ready) && !warp_wait(bar(B_FULL + s), par, abort_flag)) { ok = false; break; }
      int s1;
      uint32_t par1;
      next(s1, par1);
      ready = false;
      const bool end = static_cast<const volatile Info*>(infos)[c & (kInfos - 1)].flags & kEnd;
      if (!end && !zero) {
        step<true>(S, smem, sbase, s, kChunk, row0, lane, bar(B_FULL + s1), par1, ready);
        if ((c < 16 || (c & 7) == 7) && is_zero(S)) {
          zero = true;
          if (lane == 0) {
            atomicMax(longest, c + 1);
            __threadfence_block();
            atomicAdd(zeros, 1);
          }
        }
      }
      release(s1, par1);
      if (end) break;
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");
    const bool all_zero = !offset_only && *static_cast<volatile int*>(zeros) == 4;
    const int first = all_zero ? n - *static_cast<volatile int*>(longest) : 0;
    if (kPair && ok && all_zero && tid == 0) cluster_store(smem_u32(zeros), 1, 4);
    bool left_off = false;
    if (ok) {
      if (!all_zero && !offset_only) {           // M, transposed back
        float* M = slots + (run * 3 + 0) * kSegSlotFloats;
#pragma unroll
        for (int vt = 0; vt < 2; ++vt)
#pragma unroll
          for (int jt = 0; jt < 16; ++jt)
#pragma unroll
            for (int i = 0; i < 4; ++i) M[(8 * jt + 2 * t + (i & 1)) * kSegMapStride + row0 + 16 * vt + g + 8 * (i >> 1)] = S[vt][jt][i];
      }
      if (tid == 0 && !offset_only) *seg_zero_word(slots, run) = all_zero;
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(B_TURN));
      fill(0.f);
      ready = false;
      const bool mine = !kPair || offset_only || all_zero;
      for (int c = first; mine && c < n; ++c) {
        if (!__all_sync(0xffffffffu, ready) && !warp_wait(bar(B_FULL + s), par, abort_flag)) { ok = false; break; }
        if (offset_only && (static_cast<const volatile Info*>(infos)[c & (kInfos - 1)].flags & kEnd)) { left_off = true; break; }
        int s1;
        uint32_t par1;
        next(s1, par1);
        const int64_t left = cv.eos - cv.bos - static_cast<int64_t>(c) * kChunk;
        step<false>(S, smem, sbase, s, left < kChunk ? static_cast<int>(left) : kChunk, row0, lane, bar(B_FULL + s1), par1, ready);
        release(s1, par1);
      }
      if (ok && mine && !left_off) {
        // behind a map of zero the offset is the state at the start of the next run
        float* N = all_zero ? slots + ((run + 1) * 3 + 2) * kSegSlotFloats : slots + (run * 3 + 1) * kSegSlotFloats;
#pragma unroll
        for (int vt = 0; vt < 2; ++vt)
#pragma unroll
          for (int jt = 0; jt < 16; ++jt)
#pragma unroll
            for (int i = 0; i < 2; ++i)
              *reinterpret_cast<float2*>(N + (row0 + 16 * vt + g + 8 * i) * kD + 8 * jt + 2 * t) = make_float2(S[vt][jt][2 * i], S[vt][jt][2 * i + 1]);
      }
    }
  } else if (warp != 5 && ok && !offset_only) {
    // (the warps without a part in the walks) The caller's state goes where the second pass starts run 0 from: by then the CTA of the
    // last run may have written the final state over it, which may be the same tensor.  A share for every CTA of the chain: all
    // of it takes one CTA longer than walks that vanish (8 heads of 131072 tokens 592 -> 599 us).
    const size_t chain = static_cast<size_t>(cv.n) * p.H + cv.h;
    float* slots = p.seg_buf + chain * p.n_segs * 3 * kSegSlotFloats;
    float4* dst = reinterpret_cast<float4*>(slots + 2 * kSegSlotFloats);
    const float4* wide = static_cast<const float4*>(p.initial_state) + chain * (kD * kD / 4);
    const uint2* narrow = static_cast<const uint2*>(p.initial_state) + chain * (kD * kD / 4);
    const int first = (run * 3 + (warp == 4 ? 0 : warp - 5)) * 32 + lane;
    if (first == 0) *seg_done_word(slots) = 0;
#pragma unroll 8
    for (int i = first; i < kD * kD / 4; i += (p.n_segs - 1) * 3 * 32) {
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (p.initial_state != nullptr && p.state_fp32) {
        x = __ldg(wide + i);
      } else if (p.initial_state != nullptr) {
        const uint2 y = __ldg(narrow + i);
        x = make_float4(bf_lo(y.x), bf_hi(y.x), bf_lo(y.y), bf_hi(y.y));
      }
      dst[i] = x;
    }
  } else if (warp == 5 && lane == 0 && ok) {
    const uint8_t* rec = p.records + (static_cast<size_t>(cv.h) * p.total_chunks + cv.chunk_base) * kCrBytes;
    int item = 0;
    // an item of the ring: a chunk of the backward or of the forward walk, or (c < 0) the end of the backward one
    auto put = [&](int c, bool with_v) -> bool {
      const int s = item % kStages;
      if (p.stop_copies_after > 0 && item >= p.stop_copies_after) return false;      // test aid: the next wait for a record runs out
      if (item >= kStages && !mbar_wait_parked(bar(B_EMPTY + s), (item / kStages - 1) & 1, abort_flag)) { ok = false; return false; }
      infos[item & (kInfos - 1)].flags = c < 0 ? kEnd : 0;
      if (c < 0) {
        mbar_arrive(bar(B_FULL + s));
      } else {
        const uint32_t dst = sbase + s * kStageBytes, full = bar(B_FULL + s);
        mbar_arrive_expect_tx(full, kCrBytes + (with_v ? 8192 : 0));
        bulk_g2s(dst + 8192, rec + static_cast<size_t>(c) * kCrBytes, kCrBytes, full);
        if (with_v) {
          const int t0 = static_cast<int>(cv.bos + static_cast<int64_t>(c) * kChunk);
          tma_load_3d(dst, &tm_v, 0, cv.h, t0, full);
          tma_load_3d(dst + 4096, &tm_v, 64, cv.h, t0, full);
        }
      }
      ++item;
      return true;
    };
    bool more = true;
    if (offset_only) {
      int c = 0;
      for (; more && c < n && *static_cast<volatile int*>(zeros) < 4; ++c) more = put(c, true);
      if (more && c < n) more = put(-1, false);
    } else {
      for (int c = n - 1; more && c >= 0 && *static_cast<volatile int*>(zeros) < 4; --c) more = put(c, false);
      more = more && put(-1, false);
      if (more && !mbar_wait_parked(bar(B_TURN), 0, abort_flag)) more = ok = false;
      const bool all_zero = *static_cast<volatile int*>(zeros) == 4;
      if (more && (!kPair || all_zero))
        for (int c = all_zero ? n - *static_cast<volatile int*>(longest) : 0; more && c < n; ++c) more = put(c, true);
    }
    if (!ok || *abort_flag > 0 || !more) {
      // (giving up) copies in flight must land before the CTA's shared memory goes away
      for (int c = item > kStages ? item - kStages : 0; c < item; ++c) {
        const uint64_t t0 = globaltimer_ns();
        while (!mbar_try_wait(bar(B_FULL + c % kStages), (c / kStages) & 1))
          if (globaltimer_ns() - t0 > 20000000ull) break;
      }
    }
  }
  if (!ok || *abort_flag > 0) atomicCAS(p.status, kStatusOk, kStatusWaitTimeout);
  if (kPair) cluster_sync();                                     // (what the first CTA stores into goes away with the second)
  else __syncthreads();
}

}  // namespace recur

// v: the value tensor [T_total][H][128]
cudaError_t launch_recur(const ScanParams& p, const __nv_bfloat16* v, cudaStream_t stream) {
  int64_t walks = static_cast<int64_t>(p.N) * p.H;
  if (p.seg_chunks > 0) walks *= p.seg_pass == kSegMaps ? p.n_segs - 1 : p.n_segs;
  if (walks <= 0) return cudaSuccess;
  CUtensorMap tv;
  if (!make_map(&tv, v, p.T_total, p.H)) return cudaErrorInvalidValue;
  if (p.seg_chunks > 0 && p.seg_pass == kSegMaps) {
    const bool pair = walks * 2 <= device_sm_count();
    const auto maps = pair ? recur::maps_kernel<true> : recur::maps_kernel<false>;
    static SmemOptIn opt_in[2];
    cudaError_t e = opt_in[pair].ensure(maps, recur::kSmem);
    if (e != cudaSuccess) return e;
    return launch_clusters_after(maps, static_cast<unsigned>(pair ? 2 * walks : walks), pair ? 2 : 1, recur::kThreads, recur::kSmem, stream, tv, p);
  }
  // More walks than SMs and short ones on average: one persistent CTA per SM.  Stage alone, a CTA per walk against this form: 2048 equal
  // chains of 8 chunks 222 / 206 us, of 10 256 / 243; 768 of 8 99.3 / 98.9, of 12 123 / 126, of 24 196 / 206; 24 ragged sequences x 32
  // heads of 12 chunks on average 132 / 124, of 20 160 / 156, of 28 214 / 215, of 40 303 / 312.  The line lies where ragged
  // batches, which gain by the order by length, break even; a few rounds of equal chains of 12 to 24 chunks lose up to a twentieth by it.
  const int64_t sms = device_sm_count();
  const bool stream_form = p.seg_chunks == 0 && walks > sms && (p.T_total + static_cast<int64_t>(p.N) * (kChunk / 2)) / kChunk <= 24 * static_cast<int64_t>(p.N);
  // (a time slice is for fewer walks than SMs; its own form, as what it looks up costs the others 0.8 %)
  void (*const kernels[4])(CUtensorMap, ScanParams, int) = {recur::recur_kernel<false, false, false>, recur::recur_kernel<true, false, false>,
                                                            recur::recur_kernel<false, true, false>, recur::recur_kernel<false, false, true>};
  const int form = p.seg_chunks > 0 ? 1 : p.slice_end > 0 ? 3 : stream_form ? 2 : 0;
  const auto kernel = kernels[form];
  static SmemOptIn opt_in[4];
  cudaError_t e = opt_in[form].ensure(kernel, recur::kSmem);
  if (e != cudaSuccess) return e;
  return launch_after(kernel, static_cast<unsigned>(stream_form ? sms : walks), recur::kThreads, recur::kSmem, stream, tv, p, static_cast<int>(walks));
}

}  // namespace fkda
