// Inter-chunk recurrence over compact records for batches with few chains: a chain is split over CTAs by value channels.
//
// Replaces the reference's K2 (csrc/smxx/fwd_kernel2.cuh:115-839) where there are fewer chains than SMs and the time is that
// of one chunk step times the length.  The rows v of S^T never meet each other in the recurrence, so two or four CTAs
// (64 or 32 rows each) share a chain with nothing exchanged.  A warp holds 16 rows of the state as mma.sync accumulator
// fragments (fkda_recur.cu has the algebra and the fragment forms); what is not on the chain, the output products
//     O^T = S^T q+^T + U^T mqk^T,
// is done by a second warp per sixteen rows, which gets the bf16 copies of S^T and U^T through shared memory as the very
// fragments it needs.  With 32 rows the two kinds of warp sit on different SM sub-partitions and the chain's warp has a
// tensor pipe to itself: 70 mma.sync of 8 cycles per chunk and the latencies between them, which bound it.  Hence no wait
// on the chain but the one for the record, looked at ahead (a second one, for a free box, cost 0.08 us per chunk although
// it never had to wait), and the decay of the state under the latency of U^T (32 rows; with 64 the output warp of the same
// sub-partition fills that time, and it gives nothing).  Per chunk, 8 heads of 4096 tokens: 0.73 -> 0.60 us.  Two warps per
// sixteen rows with half of the channels each and an exchange of partial sums: 0.78.
// Warps 0 .. NW-1: recurrence; NW .. 2 NW-1: output; 2 NW: copies.
#include "fkda_common.cuh"
#include "fkda_record.cuh"
#include "fkda_tma.cuh"

namespace fkda {
namespace recur_split {

template <int NW>
struct Plan {
  static constexpr int kRows = 16 * NW;                   // value channels of a CTA
  static constexpr int kSplits = kD / kRows;              // CTAs per chain
  static constexpr int kStages = 4;
  static constexpr int kStageBytes = 33 * 1024;           // v box [32 tok][64 ch], 128-byte swizzle | record
  static constexpr int kBoxBytes = 5 * 1024;              // fragments of S^T (4 KB) and U^T (1 KB) of one warp, one per stage
  static constexpr int kStgStride = 48;                   // output staging, bytes per token: conflict-free stmatrix
  static constexpr int kSmBox = kStages * kStageBytes;    // [kStages][NW]
  static constexpr int kSmStg = kSmBox + kStages * NW * kBoxBytes;
  static constexpr int kSmBars = kSmStg + NW * 32 * kStgStride;
  static constexpr int kSmMisc = kSmBars + 256;
  static constexpr int kSmem = kSmMisc + 16;
  static constexpr int kDecayAhead = NW == 2 ? 16 : 0;  // column tiles of the state that are decayed while U^T is computed
  static constexpr int kThreads = 32 * (2 * NW + 1);
  static constexpr int B_FULL = 0, B_EMPTY = kStages, B_BOX = 2 * kStages, B_COUNT = B_BOX + kStages * NW;
  static_assert(kSmem <= 227 * 1024 && B_COUNT * 8 <= 256 && 4096 + kCrBytes <= kStageBytes, "shared memory plan");
};

__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}

template <int NW>
__global__ void __launch_bounds__(Plan<NW>::kThreads, 1) recur_split_kernel(const __grid_constant__ CUtensorMap tm_v, const ScanParams p) {
  using P = Plan<NW>;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sbase = smem_u32(smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + P::kSmMisc);
  auto bar = [&](int i) { return sbase + P::kSmBars + 8 * i; };
  if (tid == 0) {
    // the swizzled tiles need this alignment: report instead of computing garbage (below zero: a wait limit, test aid)
    *abort_flag = (sbase & 1023u) != 0u ? 1 : -p.wait_limit_us;
    for (int s = 0; s < P::kStages; ++s) {
      mbar_init(bar(P::B_FULL + s), 1);
      mbar_init(bar(P::B_EMPTY + s), 2 * NW);             // (a full stage's boxes are free too: their readers arrive here)
    }
    for (int i = 0; i < P::kStages * NW; ++i) mbar_init(bar(P::B_BOX + i), 1);
    fence_mbar_init();
  }
  __syncthreads();
  bool ok = *abort_flag <= 0;
  grid_dependency_wait();
  if (p.release_next) grid_release_next();
  const ChainView cv = chain_view<false>(p, blockIdx.x / P::kSplits);
  const int cta_row = static_cast<int>(blockIdx.x % P::kSplits) * P::kRows;
  const int nchunks = ok ? cv.nchunks : 0;
  const int mi = lane >> 3, r = lane & 7, g = lane >> 2, t = lane & 3;

  if (warp < NW) {
    // ===== recurrence: rows v = row0 + g (+ 8), columns 8 jt + 2 t, + 1 ================================================
    const int row0 = cta_row + 16 * warp;
    float S[16][4];
    if (cv.init_mode == 1) {
      const float* src = static_cast<const float*>(cv.init_base) + (row0 + g) * kD + 2 * t;
#pragma unroll
      for (int jt = 0; jt < 16; ++jt) {
        const float2 lo = __ldg(reinterpret_cast<const float2*>(src + 8 * jt)), hi = __ldg(reinterpret_cast<const float2*>(src + 8 * kD + 8 * jt));
        S[jt][0] = lo.x; S[jt][1] = lo.y; S[jt][2] = hi.x; S[jt][3] = hi.y;
      }
    } else if (cv.init_mode == 2) {
      const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(cv.init_base) + (row0 + g) * kD + 2 * t;
#pragma unroll
      for (int jt = 0; jt < 16; ++jt) {
        const uint32_t lo = __ldg(reinterpret_cast<const uint32_t*>(src + 8 * jt)), hi = __ldg(reinterpret_cast<const uint32_t*>(src + 8 * kD + 8 * jt));
        S[jt][0] = bf_lo(lo); S[jt][1] = bf_hi(lo); S[jt][2] = bf_lo(hi); S[jt][3] = bf_hi(hi);
      }
    } else {
#pragma unroll
      for (int jt = 0; jt < 16; ++jt) S[jt][0] = S[jt][1] = S[jt][2] = S[jt][3] = 0.f;
    }
    const uint32_t kn_lane = 4096 + kCrKN + (mi >> 1) * 2048 + (mi & 1) * 128 + r * 16;
    const uint32_t kr_lane = 4096 + kCrKR + mi * 2048 + r * 16;
    const uint32_t tb_lane = 4096 + kCrTB + r * 16;
    const uint32_t v_lo = lane * 128 + (((row0 >> 3) & 7) ^ r) * 16, v_hi = lane * 128 + ((((row0 >> 3) + 1) & 7) ^ r) * 16;
    int s = 0;
    uint32_t par = 0;
    bool ready = false;
    for (int c = 0; c < nchunks; ++c) {
      if (!__all_sync(0xffffffffu, ready) && !warp_wait(bar(P::B_FULL + s), par, abort_flag)) { ok = false; break; }
      const int box_i = s * NW + warp;
      const uint32_t stage = sbase + s * P::kStageBytes;
      uint4* box = reinterpret_cast<uint4*>(smem + P::kSmBox + box_i * P::kBoxBytes) + lane;

      // R^T = v^T - S^T k+^T: the accumulators start from v^T
      float R[4][4];
      {
        uint32_t x[2][4];            // v^T: channel blocks of rows 0-7, 8-15; register = token block
        ldsm_x4_trans(stage + v_lo, x[0][0], x[0][1], x[0][2], x[0][3]);
        ldsm_x4_trans(stage + v_hi, x[1][0], x[1][1], x[1][2], x[1][3]);
        const int64_t left = cv.eos - cv.bos - static_cast<int64_t>(c) * kChunk;
        if (left < kChunk) {         // rows past the sequence end belong to somebody else
          const int len = static_cast<int>(left);
#pragma unroll
          for (int nt = 0; nt < 4; ++nt) {
            const uint32_t keep = (8 * nt + 2 * t < len ? 0xffffu : 0u) | (8 * nt + 2 * t + 1 < len ? 0xffff0000u : 0u);
            x[0][nt] &= keep;
            x[1][nt] &= keep;
          }
        }
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          R[nt][0] = bf_lo(x[0][nt]);
          R[nt][1] = bf_hi(x[0][nt]);
          R[nt][2] = bf_lo(x[1][nt]);
          R[nt][3] = bf_hi(x[1][nt]);
        }
      }
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        uint32_t B[8];
        ldsm_x4(stage + kn_lane + ks * 256, B[0], B[1], B[2], B[3]);
        ldsm_x4(stage + kn_lane + 4096 + ks * 256, B[4], B[5], B[6], B[7]);
        const uint32_t a0 = pack_bf16(S[2 * ks][0], S[2 * ks][1]), a1 = pack_bf16(S[2 * ks][2], S[2 * ks][3]);
        const uint32_t a2 = pack_bf16(S[2 * ks + 1][0], S[2 * ks + 1][1]), a3 = pack_bf16(S[2 * ks + 1][2], S[2 * ks + 1][3]);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) mma_bf16_16816(R[nt], a0, a1, a2, a3, B[2 * nt], B[2 * nt + 1]);
        box[32 * ks] = make_uint4(a0, a1, a2, a3);
      }
      // U^T = R^T (T diag(beta))^T
      uint32_t l[4], m[4], n[4];     // T diag(beta): token tiles 0 and 1 (tokens 0-15 only: lower triangle), 2, 3
      ldsm_x4(stage + tb_lane + (mi >> 1) * 512 + (mi & 1) * 128, l[0], l[1], l[2], l[3]);
      ldsm_x4(stage + tb_lane + 1024 + mi * 128, m[0], m[1], m[2], m[3]);
      ldsm_x4(stage + tb_lane + 1536 + mi * 128, n[0], n[1], n[2], n[3]);
      uint32_t u[2][4];              // A fragments, k-step = 16 tokens: first of R^T, then of U^T
      auto as_operand = [&](const float(&x)[4][4]) {
#pragma unroll
        for (int ks = 0; ks < 2; ++ks)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            u[ks][e] = pack_bf16(x[2 * ks + (e >> 1)][2 * (e & 1)], x[2 * ks + (e >> 1)][2 * (e & 1) + 1]);
      };
      as_operand(R);
      const float2* e2 = reinterpret_cast<const float2*>(smem + s * P::kStageBytes + 4096 + kCrE) + t;
      auto decay = [&](int jt) {
        const float2 e = e2[4 * jt];
        uint32_t y[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) y[k] = __float_as_uint(S[jt][k]);
        mul2(y[0], y[1], e);
        mul2(y[2], y[3], e);
#pragma unroll
        for (int k = 0; k < 4; ++k) S[jt][k] = __uint_as_float(y[k]);
      };
      {
        float U[4][4];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) U[nt][0] = U[nt][1] = U[nt][2] = U[nt][3] = 0.f;
        mma_bf16_16816(U[2], u[0][0], u[0][1], u[0][2], u[0][3], m[0], m[1]);
        mma_bf16_16816(U[3], u[0][0], u[0][1], u[0][2], u[0][3], n[0], n[1]);
        mma_bf16_16816(U[0], u[0][0], u[0][1], u[0][2], u[0][3], l[0], l[1]);
        mma_bf16_16816(U[1], u[0][0], u[0][1], u[0][2], u[0][3], l[2], l[3]);
        mma_bf16_16816(U[2], u[1][0], u[1][1], u[1][2], u[1][3], m[2], m[3]);
        mma_bf16_16816(U[3], u[1][0], u[1][1], u[1][2], u[1][3], n[2], n[3]);
#pragma unroll
        for (int jt = 0; jt < P::kDecayAhead; ++jt) decay(jt);   // while they are under way
        as_operand(U);
      }
      box[256] = make_uint4(u[0][0], u[0][1], u[0][2], u[0][3]);
      box[288] = make_uint4(u[1][0], u[1][1], u[1][2], u[1][3]);
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(P::B_BOX + box_i));
      // S^T = S^T diag(e) + U^T kr; the next stage's barrier is looked at meanwhile
      const int s1 = s + 1 == P::kStages ? 0 : s + 1;
      const uint32_t par1 = s1 == 0 ? par ^ 1u : par;
      ready = mbar_test(bar(P::B_FULL + s1), par1);
#pragma unroll
      for (int jt = 0; jt < 16; ++jt) {
        uint32_t B[4];
        ldsm_x4_trans(stage + kr_lane + jt * 128, B[0], B[1], B[2], B[3]);
        if (jt >= P::kDecayAhead) decay(jt);
        mma_bf16_16816(S[jt], u[0][0], u[0][1], u[0][2], u[0][3], B[0], B[1]);
        mma_bf16_16816(S[jt], u[1][0], u[1][1], u[1][2], u[1][3], B[2], B[3]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(P::B_EMPTY + s));
      s = s1;
      par = par1;
    }
    if (ok && cv.fin_base != nullptr) {
      if (cv.fin_fp32) {
        float* dst = static_cast<float*>(cv.fin_base) + (row0 + g) * kD + 2 * t;
#pragma unroll
        for (int jt = 0; jt < 16; ++jt) {
          *reinterpret_cast<float2*>(dst + 8 * jt) = make_float2(S[jt][0], S[jt][1]);
          *reinterpret_cast<float2*>(dst + 8 * kD + 8 * jt) = make_float2(S[jt][2], S[jt][3]);
        }
      } else {
        __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(cv.fin_base) + (row0 + g) * kD + 2 * t;
#pragma unroll
        for (int jt = 0; jt < 16; ++jt) {
          *reinterpret_cast<uint32_t*>(dst + 8 * jt) = pack_bf16(S[jt][0], S[jt][1]);
          *reinterpret_cast<uint32_t*>(dst + 8 * kD + 8 * jt) = pack_bf16(S[jt][2], S[jt][3]);
        }
      }
    }
  } else if (warp < 2 * NW) {
    // ===== output: O^T of the sixteen rows of warp w, [v][tok] -> [tok][v] by stmatrix -> 16-byte pieces of the token rows ===
    const int w = warp - NW;
    const uint32_t stg = sbase + P::kSmStg + w * 32 * P::kStgStride;
    const uint8_t* stg_p = smem + P::kSmStg + w * 32 * P::kStgStride;
    const uint32_t q_lane = 4096 + kCrQP + (mi >> 1) * 2048 + (mi & 1) * 128 + r * 16;
    const uint32_t m_lane = 4096 + kCrMQK + r * 16;
    int s = 0;
    uint32_t par = 0;
    for (int c = 0; c < nchunks; ++c) {
      const int box_i = s * NW + w;
      if (!warp_wait(bar(P::B_BOX + box_i), par, abort_flag)) { ok = false; break; }
      const uint32_t stage = sbase + s * P::kStageBytes;
      const uint4* box = reinterpret_cast<const uint4*>(smem + P::kSmBox + box_i * P::kBoxBytes) + lane;
      float O[4][4];
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) O[nt][0] = O[nt][1] = O[nt][2] = O[nt][3] = 0.f;
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        const uint4 a = box[32 * ks];
        uint32_t B[8];
        ldsm_x4(stage + q_lane + ks * 256, B[0], B[1], B[2], B[3]);
        ldsm_x4(stage + q_lane + 4096 + ks * 256, B[4], B[5], B[6], B[7]);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) mma_bf16_16816(O[nt], a.x, a.y, a.z, a.w, B[2 * nt], B[2 * nt + 1]);
      }
      {
        const uint4 u0 = box[256], u1 = box[288];
        uint32_t l[4], m[4], n[4];
        ldsm_x4(stage + m_lane + (mi >> 1) * 512 + (mi & 1) * 128, l[0], l[1], l[2], l[3]);
        ldsm_x4(stage + m_lane + 1024 + mi * 128, m[0], m[1], m[2], m[3]);
        ldsm_x4(stage + m_lane + 1536 + mi * 128, n[0], n[1], n[2], n[3]);
        mma_bf16_16816(O[0], u0.x, u0.y, u0.z, u0.w, l[0], l[1]);
        mma_bf16_16816(O[1], u0.x, u0.y, u0.z, u0.w, l[2], l[3]);
        mma_bf16_16816(O[2], u0.x, u0.y, u0.z, u0.w, m[0], m[1]);
        mma_bf16_16816(O[3], u0.x, u0.y, u0.z, u0.w, n[0], n[1]);
        mma_bf16_16816(O[2], u1.x, u1.y, u1.z, u1.w, m[2], m[3]);
        mma_bf16_16816(O[3], u1.x, u1.y, u1.z, u1.w, n[2], n[3]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(P::B_EMPTY + s));
#pragma unroll
      for (int k = 0; k < 2; ++k)
        stsm_x4_trans(stg + (8 * (2 * k + (mi >> 1)) + r) * P::kStgStride + (mi & 1) * 16, pack_bf16(O[2 * k][0], O[2 * k][1]),
                      pack_bf16(O[2 * k][2], O[2 * k][3]), pack_bf16(O[2 * k + 1][0], O[2 * k + 1][1]), pack_bf16(O[2 * k + 1][2], O[2 * k + 1][3]));
      __syncwarp();
      const int64_t tok0 = cv.bos + static_cast<int64_t>(c) * kChunk;
      const int len = cv.eos - tok0 < kChunk ? static_cast<int>(cv.eos - tok0) : kChunk;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int tok = 16 * k + (lane >> 1), piece = lane & 1;
        if (tok < len)
          *reinterpret_cast<uint4*>(p.out + (static_cast<size_t>(tok0 + tok) * p.H + cv.h) * kD + cta_row + 16 * w + 8 * piece) =
              *reinterpret_cast<const uint4*>(stg_p + tok * P::kStgStride + piece * 16);
      }
      __syncwarp();
      if (++s == P::kStages) { s = 0; par ^= 1u; }
    }
  } else if (lane == 0) {
    // ===== copies: the record and this CTA's half of the v tile =========================================================
    const uint8_t* rec = p.records + (static_cast<size_t>(cv.h) * p.total_chunks + cv.chunk_base) * kCrBytes;
    int issued = 0;
    for (int c = 0; c < nchunks; ++c) {
      const int s = c % P::kStages;
      if (p.stop_copies_after > 0 && c >= p.stop_copies_after) break;            // test aid: the next wait for a record runs out
      if (c >= P::kStages && !mbar_wait_parked(bar(P::B_EMPTY + s), (c / P::kStages - 1) & 1, abort_flag)) { ok = false; break; }
      const uint32_t dst = sbase + s * P::kStageBytes, full = bar(P::B_FULL + s);
      mbar_arrive_expect_tx(full, kCrBytes + 4096);
      bulk_g2s(dst + 4096, rec + static_cast<size_t>(c) * kCrBytes, kCrBytes, full);
      tma_load_3d(dst, &tm_v, cta_row & 64, cv.h, static_cast<int>(cv.bos + static_cast<int64_t>(c) * kChunk), full);
      issued = c + 1;
    }
    if (!ok || *abort_flag > 0) {
      // (giving up) copies in flight must land before the CTA's shared memory goes away
      for (int c = issued > P::kStages ? issued - P::kStages : 0; c < issued; ++c) {
        const uint64_t t0 = globaltimer_ns();
        while (!mbar_try_wait(bar(P::B_FULL + c % P::kStages), (c / P::kStages) & 1))
          if (globaltimer_ns() - t0 > 20000000ull) break;
      }
    }
  }
  if (!ok || *abort_flag > 0) atomicCAS(p.status, kStatusOk, kStatusWaitTimeout);
}

template <int NW>
cudaError_t launch(const ScanParams& p, const CUtensorMap& tv, cudaStream_t stream) {
  using P = Plan<NW>;
  static SmemOptIn opt_in;
  cudaError_t e = opt_in.ensure(recur_split_kernel<NW>, P::kSmem);
  if (e != cudaSuccess) return e;
  return launch_after(recur_split_kernel<NW>, static_cast<unsigned>(static_cast<int64_t>(p.N) * p.H * P::kSplits), P::kThreads, P::kSmem, stream, tv, p);
}

}  // namespace recur_split

// rows: value channels per CTA (32 or 64)
cudaError_t launch_recur_split(const ScanParams& p, const __nv_bfloat16* v, int rows, cudaStream_t stream) {
  if (static_cast<int64_t>(p.N) * p.H <= 0) return cudaSuccess;
  CUtensorMap tv;
  if (!make_map(&tv, v, p.T_total, p.H)) return cudaErrorInvalidValue;
  return rows == 32 ? recur_split::launch<2>(p, tv, stream) : recur_split::launch<4>(p, tv, stream);
}

}  // namespace fkda
