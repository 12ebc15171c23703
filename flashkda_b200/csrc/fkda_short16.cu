// Fused forward pass for batches of short fixed-length sequences: one CTA per (sequence, head) chain walks the
// sequence in blocks of 16 tokens,
// reads q, k, v, g, beta and the chain's state, and writes out and the new state - no operand record goes through
// global memory, and between blocks the state stays in shared memory in fp32.  This is the shape of a continuation step
// after a prefill: per chain 16 KB of inputs against 128 KB of fp32 state in and out, so the kernel is a stream over the states.
//
// Replaces, for these shapes, both of the reference's kernels (csrc/smxx/fwd_kernel1.cuh:107-586 and
// fwd_kernel2.cuh:115-839), whose K2 spends most of its time loading and converting states here.  The algebra is
// the single sub-block case of the chunked form used by the other kernels:
//     k+ = khat 2^G, q+ = scale qhat 2^G, k- = khat 2^-G, kr = k- 2^Gtot, e = 2^Gtot        (G: running log2 decay)
//     A = tril(k+ k-^T, -1) diag_rows(beta),  M = tril(q+ k-^T),  TB = (I + A)^-1 diag(beta)
//     R = v - k+ S,   U = TB R,   O = q+ S + M U,   S' = diag(e) S + kr^T U                   (S: [k][v], stored [v][k])
// Eight warps own 16 rows v of the state and 16 channels of the element-wise stage each (mma fragment layout, fkda_elem.cuh);
// the state is the A operand of R^T = v^T - S^T k+^T and S^T q+^T and, scaled by e, the accumulator of the update, read
// from shared memory both times so that few registers are held.  Neither product needs T, so a ninth warp works out A, T
// and M meanwhile: three rendezvous per block.  fp32 state rows travel as whole-row bulk copies (fully coalesced)
// through a padded staging buffer, bf16 ones of a single block as tensor copies: the copy in is issued right behind the inputs, the copy out per warp as soon as
// its rows are done.
//
// What bounds it: HBM, as far as the CTAs of an SM cover each other's phases - two of them with fp32 state; four with bf16 and
// one block, for which the operands lie over the staged inputs (three beside them: 302 us below).
// 512 x 32 chains of 16 tokens, twenty calls in a row: 440 us with fp32 states (5.6 TB/s), 259 us with bf16 (5.5 TB/s); kept
// up under the power cap 445 and 274.  bf16 states travel as two swizzled boxes and are read by ldmatrix: with a bulk copy per
// row, each of which costs a dozen instructions, and fragments read word by word 270 / 287 (11.7 thousand warp instructions per CTA,
// 8.7 now); padded fp32 rows have no such form.  Earlier: 506 and 350 with the states asked
// for ahead of the inputs, whose 16 KB then queue behind them; 460 and 402 with w' = TB k+, u' = TB v formed before the state
// was touched (a rendezvous more, and two CTAs per SM for either type).  Asking the L2 for the next chain's state: slower.
#include "fkda_common.cuh"
#include "fkda_elem.cuh"
#include "fkda_tma.cuh"

namespace fkda {
namespace short16 {

constexpr int kRows = 16;
constexpr int kThreads = 288;
constexpr int kLdS = 20;                         // row stride (floats) of the 16x16 fp32 matrices
// shared memory (byte offsets)
constexpr int kStQ = 0;                          // staged q, k, g, v: [16 tok][256 B], 16-byte chunks XOR-swizzled by the row
constexpr int kStK = kStQ + 4096;
constexpr int kStG = kStK + 4096;
constexpr int kStV = kStG + 4096;
constexpr int kStgStride = 48;                   // output staging (over the dead -k+ and k-): [16 tok][16 v] per warp
static_assert(8 * kRows * kStgStride <= 8192, "output staging");

// The rest.  A call of one block has no inputs of a next one to receive, so the operands lie over the staged inputs.
// State rows are fp32 unless a bf16 state needs one block only.
template <bool kWide, bool kOneBlock>
struct Lay {
  static constexpr int kKN = kOneBlock ? 0 : kStV + 4096;          // bf16 [16][128] tiles in the 8x8 core-matrix layout: -k+, k-, q+, kr
  static constexpr int kKM = kKN + 4096;
  static constexpr int kQP = kKM + 4096;
  static constexpr int kKR = kQP + 4096;
  static constexpr int kTB = kKR + 4096;                           // bf16 [16][16] T diag(beta), core layout
  static constexpr int kMQK = kTB + 512;                           // bf16 [16][16]
  static constexpr int kA = kMQK + 512;                            // fp32 [16][20]
  static constexpr int kT = kA + kRows * kLdS * 4;                 // fp32 [16][20]
  static constexpr int kE = kT + kRows * kLdS * 4;                 // fp32 [128] decay of the whole block
  static constexpr int kSsq = kE + 512;                            // fp32 [q|k][16 rows][8 warps] partial sums of squares
  static constexpr int kBeta = kSsq + 1024;                        // fp32 [16]
  static constexpr int kBar = kBeta + 64;                          // mbarrier of the state copy, abort flag
  // State: [128 v] fp32 rows, padded by eight words (8-byte fragment reads hit 32 distinct banks); or two halves of 64 columns of
  // bf16 rows with the 128-byte swizzle, as the tensor copies bring them and ldmatrix wants them.
  static constexpr int kAlign = kWide ? 128 : 1024;
  static constexpr int kState = (kBar + 16 + kAlign - 1) / kAlign * kAlign;
  static constexpr int kStride = 512 + 32;
  static constexpr int kSmemBytes = kState + (kWide ? kD * kStride : kD * 256);
  static constexpr int kCtas = kWide ? 2 : 4;
  static_assert(kCtas * (kSmemBytes + 1024) <= 227 * 1024, "CTAs per SM");
};
constexpr int kBf16Row = 256 + 16;               // where a bf16 row arrives inside a wide slot (its second half)

struct Params {
  const __nv_bfloat16* q;
  const __nv_bfloat16* k;
  const __nv_bfloat16* v;
  const __nv_bfloat16* g;
  const __nv_bfloat16* beta;
  const float* A_log;
  const float* dt_bias;
  const void* initial_state;
  void* final_state;
  __nv_bfloat16* out;
  int T;                 // tokens per sequence
  int H;
  float scale;
  float gate_scale;      // lower_bound * log2(e)
  int* status;           // device status word (a bounded wait that gives up is recorded there)
};

// kFp32: type of the state tensors; kOneBlock: T <= 16, compiled without the block loop's bookkeeping
template <bool kFp32, bool kOneBlock>
__global__ void __launch_bounds__(kThreads, Lay<kFp32 || !kOneBlock, kOneBlock>::kCtas)
short16_kernel(const __grid_constant__ CUtensorMap tm_in, const __grid_constant__ CUtensorMap tm_out, const Params p) {
  using namespace elem;
  constexpr bool kWide = kFp32 || !kOneBlock;
  using L = Lay<kWide, kOneBlock>;
  constexpr int kKN = L::kKN, kKM = L::kKM, kQP = L::kQP, kKR = L::kKR, kTB = L::kTB, kMQK = L::kMQK, kState = L::kState, kStride = L::kStride;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sbase = smem_u32(smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int chain = blockIdx.x;
  const int n = chain / p.H, h = chain - n * p.H;       // consecutive CTAs: consecutive heads of the same tokens
  const int64_t t_seq0 = static_cast<int64_t>(n) * p.T;
  const int nblk = kOneBlock ? 1 : (p.T + kRows - 1) / kRows;
  float* s_e = reinterpret_cast<float*>(smem + L::kE);
  float* s_ssq = reinterpret_cast<float*>(smem + L::kSsq);
  float* s_beta = reinterpret_cast<float*>(smem + L::kBeta);

  const uint32_t bar = sbase + L::kBar;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::kBar + 8);
  constexpr int row_bytes = kFp32 ? 512 : 256;
  constexpr int in_off = kFp32 ? 0 : kBf16Row;
  if (tid == 0) {
    // (the swizzled state needs this alignment: report instead of computing garbage)
    *abort_flag = !kWide && (sbase & 1023u) != 0u ? 1 : 0;
    mbar_init(bar, kWide ? kD : 1);
    fence_mbar_init();
  }
  __syncthreads();
  grid_dependency_wait();
  // ---- inputs: coalesced asynchronous loads, 16 lanes per 256-byte token row; those of the next block are requested as
  // soon as the staging of the current block has been consumed
  auto load_rows = [&](int blk, int dst, const __nv_bfloat16* src) {
    const int lrow = tid >> 4, chunk = tid & 15;
    const bool valid = kRows * blk + lrow < p.T;
    const size_t off = (static_cast<size_t>(t_seq0 + (valid ? kRows * blk + lrow : 0)) * p.H + h) * kD + 8 * chunk;
    cp_async16(sbase + dst + stage_off(lrow, chunk), src + off, valid ? 16u : 0u);
  };
  if (warp < 8) {
    load_rows(0, kStQ, p.q);
    load_rows(0, kStK, p.k);
    load_rows(0, kStG, p.g);
    load_rows(0, kStV, p.v);
  }
  // ---- the state, behind the inputs, which are needed first: one bulk copy per row into the padded staging buffer, or two
  // tensor copies (a copy per row costs a dozen instructions, as the threads of a warp issue theirs one by one) ----
  if (!kWide) {
    if (p.initial_state != nullptr && tid == 0 && *abort_flag == 0) {
      mbar_arrive_expect_tx(bar, kD * 256);
      tma_load_3d(sbase + kState, &tm_in, 0, 0, chain, bar);
      tma_load_3d(sbase + kState + 16384, &tm_in, 64, 0, chain, bar);
    }
  } else if (p.initial_state != nullptr && tid < kD) {
    mbar_arrive_expect_tx(bar, row_bytes);
    bulk_g2s(sbase + kState + tid * kStride + in_off,
             static_cast<const uint8_t*>(p.initial_state) + (static_cast<size_t>(chain) * kD + tid) * row_bytes, row_bytes, bar);
  }
  const int g = lane >> 2, t4 = lane & 3, mi = lane >> 3, r = lane & 7;
  const float ha = 0.5f * ex2f(__ldg(p.A_log + h) * kLog2e), hgs = 0.5f * p.gate_scale;
  float hab[2] = {0.f, 0.f};               // channels 16 warp + 8 nt + g
  if (warp < 8) {
    hab[0] = ha * __ldg(p.dt_bias + h * kD + 16 * warp + g);
    hab[1] = ha * __ldg(p.dt_bias + h * kD + 16 * warp + 8 + g);
  }
  uint8_t* const srow = smem + kState + (16 * (warp & 7) + g) * kStride;
  // (bf16 halves) the row this lane addresses in a ldmatrix.x4 over a 16 x 16 tile of this warp's rows, and its column tile's position
  const uint32_t hrow = sbase + kState + (16 * (warp & 7) + 8 * (mi & 1) + r) * 128, hcol = static_cast<uint32_t>(((mi >> 1) ^ r) << 4);
  auto half_tile = [&](int ks) { return hrow + (ks >> 2) * 16384 + (hcol ^ (32u * (ks & 3))); };
  bool failed = false;

  for (int blk = 0; blk < nblk; ++blk) {
    const int64_t t0 = t_seq0 + kRows * blk;
    const int len = p.T - kRows * blk < kRows ? p.T - kRows * blk : kRows;
    float beta = 0.f;
    if (warp == 8 && lane < len) beta = sigmoid_fast(__bfloat162float(p.beta[static_cast<size_t>(t0 + lane) * p.H + h]));
    cp_async_wait_all();
    __syncthreads();
    if (*abort_flag) { failed = true; break; }

    float R[2][4], O[2][4];                // [token tile]: rows v = 16 warp + g (+ 8), tokens 8 nt + 2 t4, + 1
    uint32_t x[4];                         // v^T of this warp's rows
    if (warp < 8) {
      // ---- element-wise stage: 16 channels of 16 tokens --------------------------------------------------------------
      const uint32_t src = sbase + stage_off(8 * (mi & 1) + r, 2 * warp + (mi >> 1));
      uint32_t q[4], k[4], gw[4];          // registers 2 nt + half: tokens g + 8 half, channels 8 nt + 2 t4, + 1
      ldsm_x4(src + kStQ, q[0], q[1], q[2], q[3]);
      ldsm_x4(src + kStK, k[0], k[1], k[2], k[3]);
      ldsm_x4_trans(src + kStG, gw[0], gw[1], gw[2], gw[3]);
      if (kOneBlock) ldsm_x4_trans(src + kStV, x[0], x[1], x[2], x[3]);
      const int part = 4 * (warp ^ (g & 4));   // (rows 4-7 of eight have the halves exchanged: sixteen-byte reads by row do not conflict)
      auto squares = [&](const uint32_t(&x)[4], uint32_t dst) {
        float c0[4], c1[4];
        mma_bf16_1688_zero(c0, x[0], x[1], x[0]);
        mma_bf16_1688_zero(c1, x[0], x[1], x[1]);
        mma_bf16_1688(c0, x[2], x[3], x[2]);
        mma_bf16_1688(c1, x[2], x[3], x[3]);
        if (t4 == (g >> 1)) {
          sts_f32(dst + g * 32, (g & 1) ? c0[1] : c0[0]);
          sts_f32(dst + (8 + g) * 32, (g & 1) ? c1[3] : c1[2]);
        }
      };
      squares(q, sbase + L::kSsq + part);
      squares(k, sbase + L::kSsq + 512 + part);
      const Const kc(lane, hgs);            // a 16 x 16 triangle of ones as A fragments, and the gate's constant part
      f2 G[2][2], tot[2];
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        uint32_t hi[2], lo[2];
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          float x0 = tanh_approx(fmaf(bf_lo(gw[2 * nt + b]), ha, hab[nt])), x1 = tanh_approx(fmaf(bf_hi(gw[2 * nt + b]), ha, hab[nt]));
          if (len < kRows) {               // tokens that are not there do not decay
            if (8 * b + 2 * t4 >= len) x0 = -1.f;
            if (8 * b + 2 * t4 + 1 >= len) x1 = -1.f;
          }
          split_f16(x0, x1, hi[b], lo[b]);
        }
        float d[4];
        mma_f16_16816_zero(d, kc.tri, hi[0], hi[1]);
        mma_f16_16816(d, kc.tri, lo[0], lo[1]);
#pragma unroll
        for (int e = 0; e < 4; ++e) d[e] = fmaf(d[e], hgs, kc.hc[e >> 1]);
        G[nt][0] = pk(d[0], d[1]);
        G[nt][1] = pk(d[2], d[3]);
        tot[nt] = pk(__shfl_sync(0xffffffffu, d[2], lane | 28), __shfl_sync(0xffffffffu, d[3], lane | 28));     // token 15
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");      // the partial sums of squares are complete, the staged inputs read
      float rq[2], rk[2];
      {
        // lanes 0-15: rows of q, 16-31: rows of k
        const uint32_t at = sbase + L::kSsq + lane * 32 + (lane & 4) * 4;
        const float4 x = lds_f4(at), y = lds_f4(at ^ 16);
        const float n = rsqrtf(((x.x + x.y) + (x.z + x.w)) + ((y.x + y.y) + (y.z + y.w)) + 1e-6f) * (lane < 16 ? p.scale : 1.f);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          rq[b] = __shfl_sync(0xffffffffu, n, g + 8 * b);
          rk[b] = __shfl_sync(0xffffffffu, n, 16 + g + 8 * b);
        }
      }
      uint32_t kn[4], qp[4], km[4], kr[4];
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const f2 e = exp2_pair(tot[nt]);
        if (g == 0) *reinterpret_cast<f2*>(s_e + 16 * warp + 8 * nt + 2 * t4) = e;
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          const uint32_t kw = k[2 * nt + b], qw = q[2 * nt + b];
          const f2 kh = pk(bf_lo(kw) * rk[b], bf_hi(kw) * rk[b]), qh = pk(bf_lo(qw) * rq[b], bf_hi(qw) * rq[b]);
          const f2 pw = exp2_pair(G[nt][b]), m = mul(kh, rcp_pair(pw));
          kn[2 * nt + b] = round_bf(mul(kh, pw)) ^ 0x80008000u;
          qp[2 * nt + b] = round_bf(mul(qh, pw));
          km[2 * nt + b] = round_bf(m);
          kr[2 * nt + b] = round_bf(mul(m, e));
        }
      }
      const uint32_t dst = sbase + (mi & 1) * 2048 + (2 * warp + (mi >> 1)) * 128 + r * 16;
      stsm_x4(dst + kKN, kn[0], kn[1], kn[2], kn[3]);
      stsm_x4(dst + kQP, qp[0], qp[1], qp[2], qp[3]);
      stsm_x4(dst + kKM, km[0], km[1], km[2], km[3]);
      stsm_x4(dst + kKR, kr[0], kr[1], kr[2], kr[3]);
    } else if (lane < kRows) {
      s_beta[lane] = beta;
    }
    __syncthreads();
    if (!kOneBlock && blk + 1 < nblk && warp < 8) {
      load_rows(blk + 1, kStQ, p.q);
      load_rows(blk + 1, kStK, p.k);
      load_rows(blk + 1, kStG, p.g);
    }

    const bool zero_state = blk == 0 && p.initial_state == nullptr;
    if (warp < 8) {
      // ---- R^T = v^T - S^T k+^T, O^T = S^T q+^T ---------------------------------------------------------------------------
      {
        if (!kOneBlock) ldsm_x4_trans(sbase + kStV + stage_off(8 * (mi & 1) + r, 2 * warp + (mi >> 1)), x[0], x[1], x[2], x[3]);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          R[nt][0] = bf_lo(x[nt]);
          R[nt][1] = bf_hi(x[nt]);
          R[nt][2] = bf_lo(x[2 + nt]);
          R[nt][3] = bf_hi(x[2 + nt]);
          O[nt][0] = O[nt][1] = O[nt][2] = O[nt][3] = 0.f;
        }
      }
      if (!zero_state) {
        if (blk == 0) mbar_wait(bar, 0, abort_flag);     // gives up after 2 s and raises the abort flag, seen at the next block top / the exit
        const uint32_t b_lane = sbase + (mi >> 1) * 2048 + (mi & 1) * 128 + r * 16;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          uint32_t a[4], b0, b1, b2, b3;
          if (kWide && (kFp32 || blk > 0)) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {    // e & 1: rows + 8, e >> 1: columns + 8
              const float2 s = *reinterpret_cast<const float2*>(srow + (e & 1) * 8 * kStride + (16 * ks + 8 * (e >> 1) + 2 * t4) * 4);
              a[e] = pack_bf16(s.x, s.y);
            }
          } else if (kWide) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              a[e] = *reinterpret_cast<const uint32_t*>(srow + in_off + (e & 1) * 8 * kStride + (16 * ks + 8 * (e >> 1) + 2 * t4) * 2);
          } else {
            ldsm_x4(half_tile(ks), a[0], a[1], a[2], a[3]);
          }
          ldsm_x4(b_lane + kKN + ks * 256, b0, b1, b2, b3);
          mma_bf16_16816(R[0], a[0], a[1], a[2], a[3], b0, b1);
          mma_bf16_16816(R[1], a[0], a[1], a[2], a[3], b2, b3);
          ldsm_x4(b_lane + kQP + ks * 256, b0, b1, b2, b3);
          mma_bf16_16816(O[0], a[0], a[1], a[2], a[3], b0, b1);
          mma_bf16_16816(O[1], a[0], a[1], a[2], a[3], b2, b3);
        }
      }
    } else {
      // ---- ninth warp: A, T = (I + A)^-1, T diag(beta); tril(M) -----------------------------------------------------------
      float* s_A = reinterpret_cast<float*>(smem + L::kA);
      float* s_T = reinterpret_cast<float*>(smem + L::kT);
      const uint32_t a_lane = sbase + (mi & 1) * 2048 + (mi >> 1) * 128 + r * 16;
      const uint32_t b_lane = sbase + kKM + (mi >> 1) * 2048 + (mi & 1) * 128 + r * 16;
      float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}}, mq[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        uint32_t a0, a1, a2, a3, b0, b1, b2, b3;
        ldsm_x4(b_lane + ks * 256, b0, b1, b2, b3);
        ldsm_x4(a_lane + kKN + ks * 256, a0, a1, a2, a3);
        mma_bf16_16816(acc[0], a0, a1, a2, a3, b0, b1);
        mma_bf16_16816(acc[1], a0, a1, a2, a3, b2, b3);
        ldsm_x4(a_lane + kQP + ks * 256, a0, a1, a2, a3);
        mma_bf16_16816(mq[0], a0, a1, a2, a3, b0, b1);
        mma_bf16_16816(mq[1], a0, a1, a2, a3, b2, b3);
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const int lr = g + 8 * hh, lc = nt * 8 + 2 * t4;
          const float br = -s_beta[lr];      // (the operand is -k+)
          *reinterpret_cast<float2*>(s_A + lr * kLdS + lc) =
              make_float2(lc < lr ? acc[nt][2 * hh] * br : 0.f, lc + 1 < lr ? acc[nt][2 * hh + 1] * br : 0.f);
          *reinterpret_cast<uint32_t*>(smem + kMQK + core_off(lr, lc, kRows)) =
              pack_bf16(lc <= lr ? mq[nt][2 * hh] : 0.f, lc + 1 <= lr ? mq[nt][2 * hh + 1] : 0.f);
        }
      __syncwarp();
      if (lane < kRows) {
        // forward substitution, one column per lane: x_i = [i == c] - sum_{j<i} A_ij x_j
        const int c = lane;
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float a = (i == c) ? 1.f : 0.f;
#pragma unroll
          for (int q4 = 0; 4 * q4 < i; ++q4) {
            const float4 a4 = *reinterpret_cast<const float4*>(s_A + i * kLdS + 4 * q4);
            a = fmaf(-a4.x, x[4 * q4], a);
            a = fmaf(-a4.y, x[4 * q4 + 1], a);
            a = fmaf(-a4.z, x[4 * q4 + 2], a);
            a = fmaf(-a4.w, x[4 * q4 + 3], a);
          }
          x[i] = a;
          s_T[i * kLdS + c] = a;
        }
      }
      __syncwarp();
      if (lane < kRows) {
        // T diag(beta) as a bf16 core-layout operand; lane = row
        const int rr = lane;
        uint8_t* dst = smem + kTB + (rr >> 3) * 256 + (rr & 7) * 16;
#pragma unroll
        for (int q8 = 0; q8 < 2; ++q8) {
          const float4 ta = *reinterpret_cast<const float4*>(s_T + rr * kLdS + 8 * q8);
          const float4 tb = *reinterpret_cast<const float4*>(s_T + rr * kLdS + 8 * q8 + 4);
          const float4 ba = *reinterpret_cast<const float4*>(s_beta + 8 * q8);
          const float4 bb = *reinterpret_cast<const float4*>(s_beta + 8 * q8 + 4);
          *reinterpret_cast<uint4*>(dst + q8 * 128) = make_uint4(pack_bf16(ta.x * ba.x, ta.y * ba.y), pack_bf16(ta.z * ba.z, ta.w * ba.w),
                                                                 pack_bf16(tb.x * bb.x, tb.y * bb.y), pack_bf16(tb.z * bb.z, tb.w * bb.w));
        }
      }
    }
    __syncthreads();
    if (!kOneBlock && blk + 1 < nblk && warp < 8) load_rows(blk + 1, kStV, p.v);

    if (warp < 8) {
      // ---- U^T = R^T TB^T, O^T += U^T mqk^T --------------------------------------------------------------------------------
      uint32_t u[4], b0, b1, b2, b3;         // A fragments: e & 1 rows + 8, e >> 1 tokens + 8
#pragma unroll
      for (int e = 0; e < 4; ++e) u[e] = pack_bf16(R[e >> 1][2 * (e & 1)], R[e >> 1][2 * (e & 1) + 1]);
      ldsm_x4(sbase + kTB + (mi >> 1) * 256 + (mi & 1) * 128 + r * 16, b0, b1, b2, b3);
      float U[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
      mma_bf16_16816(U[0], u[0], u[1], u[2], u[3], b0, b1);
      mma_bf16_16816(U[1], u[0], u[1], u[2], u[3], b2, b3);
#pragma unroll
      for (int e = 0; e < 4; ++e) u[e] = pack_bf16(U[e >> 1][2 * (e & 1)], U[e >> 1][2 * (e & 1) + 1]);
      ldsm_x4(sbase + kMQK + (mi >> 1) * 256 + (mi & 1) * 128 + r * 16, b0, b1, b2, b3);
      mma_bf16_16816(O[0], u[0], u[1], u[2], u[3], b0, b1);
      mma_bf16_16816(O[1], u[0], u[1], u[2], u[3], b2, b3);

      // ---- S^T = S^T diag(e) + U^T kr in place: fp32 between blocks, the caller's type at the end ------------------------
      const bool last = kOneBlock || blk + 1 == nblk;
      if (!last || p.final_state != nullptr) {
#pragma unroll
        for (int jp = 0; jp < 8; ++jp) {     // two column tiles per transposed load
          ldsm_x4_trans(sbase + kKR + (mi & 1) * 2048 + (2 * jp + (mi >> 1)) * 128 + r * 16, b0, b1, b2, b3);
          uint32_t half[4] = {0u, 0u, 0u, 0u};       // (bf16 halves) the tile: c = 0 rows g, rows g + 8, c = 1 the same
          if (!kWide && !zero_state) ldsm_x4(half_tile(jp), half[0], half[1], half[2], half[3]);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int col = 8 * (2 * jp + c) + 2 * t4;
            uint32_t S[4] = {0u, 0u, 0u, 0u};
            if (!zero_state) {
              if (kWide && (kFp32 || blk > 0)) {
                const uint2 lo = *reinterpret_cast<const uint2*>(srow + col * 4), hi = *reinterpret_cast<const uint2*>(srow + 8 * kStride + col * 4);
                S[0] = lo.x; S[1] = lo.y; S[2] = hi.x; S[3] = hi.y;
              } else {
                const uint32_t lo = kWide ? *reinterpret_cast<const uint32_t*>(srow + in_off + col * 2) : half[2 * c];
                const uint32_t hi = kWide ? *reinterpret_cast<const uint32_t*>(srow + in_off + 8 * kStride + col * 2) : half[2 * c + 1];
                S[0] = lo << 16; S[1] = lo & 0xffff0000u; S[2] = hi << 16; S[3] = hi & 0xffff0000u;
              }
              const float2 e2 = *reinterpret_cast<const float2*>(s_e + col);
              mul2(S[0], S[1], e2);
              mul2(S[2], S[3], e2);
            }
            float Z[4] = {__uint_as_float(S[0]), __uint_as_float(S[1]), __uint_as_float(S[2]), __uint_as_float(S[3])};
            mma_bf16_16816(Z, u[0], u[1], u[2], u[3], c ? b2 : b0, c ? b3 : b1);
            if (kFp32 || !last) {
              *reinterpret_cast<float2*>(srow + col * 4) = make_float2(Z[0], Z[1]);
              *reinterpret_cast<float2*>(srow + 8 * kStride + col * 4) = make_float2(Z[2], Z[3]);
            } else if (kWide) {
              *reinterpret_cast<uint32_t*>(srow + col * 2) = pack_bf16(Z[0], Z[1]);
              *reinterpret_cast<uint32_t*>(srow + 8 * kStride + col * 2) = pack_bf16(Z[2], Z[3]);
            } else {
              half[2 * c] = pack_bf16(Z[0], Z[1]);
              half[2 * c + 1] = pack_bf16(Z[2], Z[3]);
            }
          }
          if (!kWide) stsm_x4(half_tile(jp), half[0], half[1], half[2], half[3]);
        }
      }
      // ---- out: [v][tok] -> [tok][v] by stmatrix, one 16-byte piece per lane -------------------------------------------------
      const uint32_t stg = kKN + warp * kRows * kStgStride;
      stsm_x4_trans(sbase + stg + (8 * (mi >> 1) + r) * kStgStride + (mi & 1) * 16, pack_bf16(O[0][0], O[0][1]), pack_bf16(O[0][2], O[0][3]),
                    pack_bf16(O[1][0], O[1][1]), pack_bf16(O[1][2], O[1][3]));
      __syncwarp();
      if ((lane >> 1) < len)
        *reinterpret_cast<uint4*>(p.out + (static_cast<size_t>(t0 + (lane >> 1)) * p.H + h) * kD + 16 * warp + 8 * (lane & 1)) =
            *reinterpret_cast<const uint4*>(smem + stg + (lane >> 1) * kStgStride + (lane & 1) * 16);
    }
  }  // blocks

  if (failed || *abort_flag > 0) {
    // the state copy may still be landing: give it a moment before this CTA's shared memory goes away
    const uint64_t t_begin = globaltimer_ns();
    while (p.initial_state != nullptr && !mbar_try_wait(bar, 0) && globaltimer_ns() - t_begin < 20000000ull) {}
    if (tid == 0) atomicCAS(p.status, kStatusOk, kStatusWaitTimeout);
    return;
  }
  if (p.final_state != nullptr && warp < 8) {      // one bulk copy per row, per warp as soon as its rows are done
    fence_proxy_async_smem();
    __syncwarp();
    if (!kWide) {
      if (lane == 0) {
        tma_store_3d(&tm_out, sbase + kState + warp * 2048, 0, 16 * warp, chain);
        tma_store_3d(&tm_out, sbase + kState + 16384 + warp * 2048, 64, 16 * warp, chain);
        bulk_commit();
        bulk_wait_read0();
      }
    } else if (lane < 16) {
      const int vr = 16 * warp + lane;
      bulk_s2g(static_cast<uint8_t*>(p.final_state) + (static_cast<size_t>(chain) * kD + vr) * row_bytes,
               sbase + kState + vr * kStride, row_bytes);
      bulk_commit();
      bulk_wait_read0();               // shared memory must outlive the copy's reads
    }
  }
}

// ---- at most eight tokens --------------------------------------------------------------------------------------------------
// The same for one block of eight tokens (a speculative step): tiles of eight tokens take half the products, operand loads
// and element-wise work of a block that is half padding, and the two products of the ninth warp are one, [k+; q+] k-^T.
// 64 x 32 chains of 5 tokens: 39.1 -> 31.3 us with bf16 states, 61.4 -> 59.6 with fp32; 512 x 32 bf16 249 -> 206.  Four CTAs per SM: with five
// (40 registers, spills) 33.2.
constexpr int kRows8 = 8;
constexpr int kTile8 = kRows8 * 256;
template <bool kFp32>
struct Lay8 {
  static constexpr int kQ = 0, kK = kTile8, kG = 2 * kTile8, kV = 3 * kTile8;      // staged inputs, and over them, once all are read:
  static constexpr int kKN = 0, kKM = kTile8, kQP = 2 * kTile8, kKR = 3 * kTile8;  // bf16 [8][128] core-matrix tiles
  static constexpr int kTB = 4 * kTile8;                           // bf16 [8][8] T diag(beta)
  static constexpr int kMQK = kTB + 128;                           // bf16 [8][8]
  static constexpr int kA = kMQK + 128;                            // fp32 [8][8]
  static constexpr int kE = kA + 256;                              // fp32 [128]
  static constexpr int kSsq = kE + 512;                            // fp32 [q|k][8 rows][8 warps]
  static constexpr int kBeta = kSsq + 512;                         // fp32 [8]
  static constexpr int kBar = kBeta + 32;
  static constexpr int kAlign = kFp32 ? 128 : 1024;
  static constexpr int kState = (kBar + 16 + kAlign - 1) / kAlign * kAlign;
  static constexpr int kStride = 512 + 32;                         // (fp32 rows)
  static constexpr int kSmemBytes = kState + (kFp32 ? kD * kStride : kD * 256);
  static constexpr int kCtas = kFp32 ? 2 : 4;
  static_assert(kCtas * (kSmemBytes + 1024) <= 227 * 1024 && 8 * kRows8 * kStgStride <= 2 * kTile8, "shared memory plan");
};

template <bool kFp32>
__global__ void __launch_bounds__(kThreads, Lay8<kFp32>::kCtas)
short8_kernel(const __grid_constant__ CUtensorMap tm_in, const __grid_constant__ CUtensorMap tm_out, const Params p) {
  using namespace elem;
  using L = Lay8<kFp32>;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sbase = smem_u32(smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int chain = blockIdx.x;
  const int n = chain / p.H, h = chain - n * p.H;
  const int64_t t0 = static_cast<int64_t>(n) * p.T;
  const uint32_t bar = sbase + L::kBar;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::kBar + 8);
  float* s_beta = reinterpret_cast<float*>(smem + L::kBeta);
  if (tid == 0) {
    // (the swizzled state needs this alignment: report instead of computing garbage)
    *abort_flag = !kFp32 && (sbase & 1023u) != 0u ? 1 : 0;
    mbar_init(bar, kFp32 ? kD : 1);
    fence_mbar_init();
  }
  __syncthreads();
  grid_dependency_wait();
  if (warp < 8) {                        // inputs: q, k by the first four warps, g, v by the others
    const int row = (tid & 127) >> 4, chunk = tid & 15;
    const bool valid = row < p.T;
    const size_t off = (static_cast<size_t>(t0 + (valid ? row : 0)) * p.H + h) * kD + 8 * chunk;
    const uint32_t dst = sbase + stage_off(row, chunk);
    const bool first = warp < 4;
    cp_async16(dst + (first ? L::kQ : L::kG), (first ? p.q : p.g) + off, valid ? 16u : 0u);
    cp_async16(dst + (first ? L::kK : L::kV), (first ? p.k : p.v) + off, valid ? 16u : 0u);
  }
  if (kFp32) {
    if (p.initial_state != nullptr && tid < kD) {
      mbar_arrive_expect_tx(bar, 512);
      bulk_g2s(sbase + L::kState + tid * L::kStride, static_cast<const float*>(p.initial_state) + (static_cast<size_t>(chain) * kD + tid) * kD, 512, bar);
    }
  } else if (p.initial_state != nullptr && tid == 0 && *abort_flag == 0) {
    mbar_arrive_expect_tx(bar, kD * 256);
    tma_load_3d(sbase + L::kState, &tm_in, 0, 0, chain, bar);
    tma_load_3d(sbase + L::kState + 16384, &tm_in, 64, 0, chain, bar);
  }
  const int g = lane >> 2, t = lane & 3, mi = lane >> 3, r = lane & 7;
  const float ha = 0.5f * ex2f(__ldg(p.A_log + h) * kLog2e), hgs = 0.5f * p.gate_scale;
  float bias[2] = {0.f, 0.f}, beta = 0.f;
  if (warp < 8) {
    bias[0] = __ldg(p.dt_bias + h * kD + 16 * warp + g);
    bias[1] = __ldg(p.dt_bias + h * kD + 16 * warp + 8 + g);
  } else if (lane < p.T) {
    beta = sigmoid_fast(__bfloat162float(p.beta[static_cast<size_t>(t0 + lane) * p.H + h]));
  }
  cp_async_wait_all();
  __syncthreads();
  const bool failed = *abort_flag > 0;

  float R[4], O[4] = {0.f, 0.f, 0.f, 0.f};   // rows v = 16 warp + g (+ 8), tokens 2 t, + 1
  const bool zero_state = p.initial_state == nullptr;
  if (!failed && warp < 8) {
    // ---- element-wise stage: 16 channels of 8 tokens --------------------------------------------------------------------
    const uint32_t at = stage_off(r, 2 * warp + (mi & 1)) + (mi >> 1) * kTile8;
    uint32_t q[2], k[2], gw[2], x[2];        // (channels 8 nt + 2 t, + 1 of token g); g and v transposed: tokens 2 t, + 1 of channel 8 nt + g
    ldsm_x4(sbase + L::kQ + at, q[0], q[1], k[0], k[1]);
    ldsm_x4_trans(sbase + L::kG + at, gw[0], gw[1], x[0], x[1]);
    R[0] = bf_lo(x[0]);
    R[1] = bf_hi(x[0]);
    R[2] = bf_lo(x[1]);
    R[3] = bf_hi(x[1]);
    {
      float cq[4], ck[4];                    // [q; k] times q^T and k^T: the diagonals of their first and second half
      mma_bf16_1688_zero(cq, q[0], k[0], q[0]);
      mma_bf16_1688_zero(ck, q[0], k[0], k[0]);
      mma_bf16_1688(cq, q[1], k[1], q[1]);
      mma_bf16_1688(ck, q[1], k[1], k[1]);
      if (t == (g >> 1)) {
        const uint32_t dst = sbase + L::kSsq + g * 32 + 4 * (warp ^ (g & 4));
        sts_f32(dst, (g & 1) ? cq[1] : cq[0]);
        sts_f32(dst + 256, (g & 1) ? ck[3] : ck[2]);
      }
    }
    f2 G[2], tot[2];
    const uint32_t tri = (2 * t <= g ? 0x3c00u : 0u) | (2 * t + 1 <= g ? 0x3c000000u : 0u), ones = 0x3c003c00u;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      const float hab = ha * bias[nt];
      float x0 = tanh_approx(fmaf(bf_lo(gw[nt]), ha, hab)), x1 = tanh_approx(fmaf(bf_hi(gw[nt]), ha, hab));
      if (2 * t >= p.T) x0 = -1.f;           // tokens that are not there do not decay
      if (2 * t + 1 >= p.T) x1 = -1.f;
      uint32_t hi, lo;
      split_f16(x0, x1, hi, lo);
      float d[4];                            // sums up to token g, and over all eight
      mma_f16_1688_zero(d, tri, ones, hi);
      mma_f16_1688(d, tri, ones, lo);
      const float c = hgs * static_cast<float>(g + 1);
      G[nt] = pk(fmaf(d[0], hgs, c), fmaf(d[1], hgs, c));
      tot[nt] = pk(fmaf(d[2], hgs, 8.f * hgs), fmaf(d[3], hgs, 8.f * hgs));
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");      // the partial sums of squares are complete, the staged inputs read
    float rq, rk;
    {
      // lanes 0-7: rows of q, 8-15: rows of k
      const uint32_t s = sbase + L::kSsq + (lane & 15) * 32 + (lane & 4) * 4;
      const float4 y = lds_f4(s), z = lds_f4(s ^ 16);
      const float nrm = rsqrtf(((y.x + y.y) + (y.z + y.w)) + ((z.x + z.y) + (z.z + z.w)) + 1e-6f) * ((lane & 8) ? 1.f : p.scale);
      rq = __shfl_sync(0xffffffffu, nrm, g);
      rk = __shfl_sync(0xffffffffu, nrm, 8 + g);
    }
    uint32_t kn[2], qp[2], km[2], kr[2];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      const f2 e = exp2_pair(tot[nt]);
      if (g == 0) sts_f2(sbase + L::kE + (16 * warp + 8 * nt + 2 * t) * 4, e);
      const f2 kh = pk(bf_lo(k[nt]) * rk, bf_hi(k[nt]) * rk), qh = pk(bf_lo(q[nt]) * rq, bf_hi(q[nt]) * rq);
      const f2 pw = exp2_pair(G[nt]), m = mul(kh, rcp_pair(pw));
      kn[nt] = round_bf(mul(kh, pw)) ^ 0x80008000u;
      qp[nt] = round_bf(mul(qh, pw));
      km[nt] = round_bf(m);
      kr[nt] = round_bf(mul(m, e));
    }
    const uint32_t dst = sbase + (2 * warp + (mi & 1)) * 128 + r * 16;
    stsm_x4(dst + (mi < 2 ? L::kKN : L::kQP), kn[0], kn[1], qp[0], qp[1]);
    stsm_x4(dst + (mi < 2 ? L::kKM : L::kKR), km[0], km[1], kr[0], kr[1]);
  } else if (lane < kRows8) {
    s_beta[lane] = beta;
  }
  __syncthreads();

  // the row this lane addresses in a ldmatrix.x4 over a 16 x 16 tile of this warp's rows of the swizzled state, and its column tile's position
  const uint32_t hrow = sbase + L::kState + (16 * (warp & 7) + 8 * (mi & 1) + r) * 128, hcol = static_cast<uint32_t>(((mi >> 1) ^ r) << 4);
  auto half_tile = [&](int ks) { return hrow + (ks >> 2) * 16384 + (hcol ^ (32u * (ks & 3))); };
  uint8_t* const srow = smem + L::kState + (16 * (warp & 7) + g) * L::kStride;
  if (failed) {
  } else if (warp < 8) {
    // ---- R^T = v^T - S^T k+^T, O^T = S^T q+^T ---------------------------------------------------------------------------
    if (!zero_state) {
      mbar_wait(bar, 0, abort_flag);         // gives up after 2 s and raises the abort flag, seen at the exit
      const uint32_t b_lane = sbase + (mi < 2 ? L::kKN : L::kQP) + (mi & 1) * 128 + r * 16;
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        uint32_t a[4], b0, b1, b2, b3;
        if (kFp32) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {      // e & 1: rows + 8, e >> 1: columns + 8
            const float2 s = *reinterpret_cast<const float2*>(srow + (e & 1) * 8 * L::kStride + (16 * ks + 8 * (e >> 1) + 2 * t) * 4);
            a[e] = pack_bf16(s.x, s.y);
          }
        } else {
          ldsm_x4(half_tile(ks), a[0], a[1], a[2], a[3]);
        }
        ldsm_x4(b_lane + ks * 256, b0, b1, b2, b3);
        mma_bf16_16816(R, a[0], a[1], a[2], a[3], b0, b1);
        mma_bf16_16816(O, a[0], a[1], a[2], a[3], b2, b3);
      }
    }
  } else {
    // ---- ninth warp: [A; M] = [k+; q+] k-^T, T = (I + A)^-1, T diag(beta); tril(M) ------------------------------------------
    float* s_A = reinterpret_cast<float*>(smem + L::kA);
    const uint32_t a_lane = sbase + ((mi & 1) ? L::kQP : L::kKN) + (mi >> 1) * 128 + r * 16, b_lane = sbase + L::kKM + mi * 128 + r * 16;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) {
      uint32_t b[4];
      ldsm_x4(b_lane + k2 * 512, b[0], b[1], b[2], b[3]);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        uint32_t a0, a1, a2, a3;
        ldsm_x4(a_lane + (2 * k2 + i) * 256, a0, a1, a2, a3);
        mma_bf16_16816(acc, a0, a1, a2, a3, b[2 * i], b[2 * i + 1]);
      }
    }
    const float br = -s_beta[g];             // (the operand is -k+)
    *reinterpret_cast<float2*>(s_A + g * 8 + 2 * t) = make_float2(2 * t < g ? acc[0] * br : 0.f, 2 * t + 1 < g ? acc[1] * br : 0.f);
    *reinterpret_cast<uint32_t*>(smem + L::kMQK + g * 16 + t * 4) = pack_bf16(2 * t <= g ? acc[2] : 0.f, 2 * t + 1 <= g ? acc[3] : 0.f);
    __syncwarp();
    if (lane < kRows8) {
      // forward substitution, one column per lane: x_i = [i == c] - sum_{j<i} A_ij x_j
      const int c = lane;
      const float bc = s_beta[c];
      float x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float a = (i == c) ? 1.f : 0.f;
#pragma unroll
        for (int q4 = 0; 4 * q4 < i; ++q4) {
          const float4 y = *reinterpret_cast<const float4*>(s_A + i * 8 + 4 * q4);
          a = fmaf(-y.x, x[4 * q4], a);
          a = fmaf(-y.y, x[4 * q4 + 1], a);
          a = fmaf(-y.z, x[4 * q4 + 2], a);
          a = fmaf(-y.w, x[4 * q4 + 3], a);
        }
        x[i] = a;
        *reinterpret_cast<__nv_bfloat16*>(smem + L::kTB + i * 16 + c * 2) = __float2bfloat16_rn(a * bc);
      }
    }
  }
  __syncthreads();

  if (!failed && warp < 8) {
    // ---- U^T = R^T TB^T, O^T += U^T mqk^T --------------------------------------------------------------------------------
    float U[4];
    mma_bf16_1688_zero(U, pack_bf16(R[0], R[1]), pack_bf16(R[2], R[3]), *reinterpret_cast<const uint32_t*>(smem + L::kTB + g * 16 + t * 4));
    const uint32_t u0 = pack_bf16(U[0], U[1]), u1 = pack_bf16(U[2], U[3]);
    mma_bf16_1688(O, u0, u1, *reinterpret_cast<const uint32_t*>(smem + L::kMQK + g * 16 + t * 4));

    // ---- S^T = S^T diag(e) + U^T kr in place ---------------------------------------------------------------------------------
    if (p.final_state != nullptr) {
      const uint32_t e_lane = sbase + L::kE + 8 * t;
#pragma unroll
      for (int j4 = 0; j4 < 4; ++j4) {
        uint32_t b[4];                       // four column tiles
        ldsm_x4_trans(sbase + L::kKR + (4 * j4 + mi) * 128 + r * 16, b[0], b[1], b[2], b[3]);
#pragma unroll
        for (int jp = 0; jp < 2; ++jp) {
          uint32_t half[4] = {0u, 0u, 0u, 0u};       // (bf16) the tile: c = 0 rows g, rows g + 8, c = 1 the same
          if (!kFp32 && !zero_state) ldsm_x4(half_tile(2 * j4 + jp), half[0], half[1], half[2], half[3]);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int tile = 4 * j4 + 2 * jp + c;
            float2* const lo = reinterpret_cast<float2*>(srow + (8 * tile + 2 * t) * 4);
            float2* const hi = reinterpret_cast<float2*>(srow + 8 * L::kStride + (8 * tile + 2 * t) * 4);
            uint32_t S[4] = {0u, 0u, 0u, 0u};
            if (!zero_state) {
              if (kFp32) {
                S[0] = __float_as_uint(lo->x);
                S[1] = __float_as_uint(lo->y);
                S[2] = __float_as_uint(hi->x);
                S[3] = __float_as_uint(hi->y);
              } else {
                S[0] = half[2 * c] << 16;
                S[1] = half[2 * c] & 0xffff0000u;
                S[2] = half[2 * c + 1] << 16;
                S[3] = half[2 * c + 1] & 0xffff0000u;
              }
              float2 e2;
              asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(e2.x), "=f"(e2.y) : "r"(e_lane + 32 * tile));
              mul2(S[0], S[1], e2);
              mul2(S[2], S[3], e2);
            }
            float Z[4] = {__uint_as_float(S[0]), __uint_as_float(S[1]), __uint_as_float(S[2]), __uint_as_float(S[3])};
            mma_bf16_1688(Z, u0, u1, b[2 * jp + c]);
            if (kFp32) {
              *lo = make_float2(Z[0], Z[1]);
              *hi = make_float2(Z[2], Z[3]);
            } else {
              half[2 * c] = pack_bf16(Z[0], Z[1]);
              half[2 * c + 1] = pack_bf16(Z[2], Z[3]);
            }
          }
          if (!kFp32) stsm_x4(half_tile(2 * j4 + jp), half[0], half[1], half[2], half[3]);
        }
      }
    }
    // ---- out: [v][tok] -> [tok][v] by stmatrix (over -k+ and k-, which are done with) ------------------------------------------
    const uint32_t stg = L::kKN + warp * kRows8 * kStgStride;
    stsm_x2_trans(sbase + stg + r * kStgStride + (mi & 1) * 16, pack_bf16(O[0], O[1]), pack_bf16(O[2], O[3]));
    __syncwarp();
    if ((lane >> 1) < p.T)
      *reinterpret_cast<uint4*>(p.out + (static_cast<size_t>(t0 + (lane >> 1)) * p.H + h) * kD + 16 * warp + 8 * (lane & 1)) =
          *reinterpret_cast<const uint4*>(smem + stg + (lane >> 1) * kStgStride + (lane & 1) * 16);
  }

  if (failed || *abort_flag > 0) {
    // the state copy may still be landing: give it a moment before this CTA's shared memory goes away
    const uint64_t t_begin = globaltimer_ns();
    while (p.initial_state != nullptr && !mbar_try_wait(bar, 0) && globaltimer_ns() - t_begin < 20000000ull) {}
    if (tid == 0) atomicCAS(p.status, kStatusOk, kStatusWaitTimeout);
    return;
  }
  if (p.final_state != nullptr && warp < 8) {
    fence_proxy_async_smem();
    __syncwarp();
    if (kFp32) {
      if (lane < 16) {
        const int vr = 16 * warp + lane;
        bulk_s2g(static_cast<float*>(p.final_state) + (static_cast<size_t>(chain) * kD + vr) * kD, sbase + L::kState + vr * L::kStride, 512);
        bulk_commit();
        bulk_wait_read0();               // shared memory must outlive the copy's reads
      }
    } else if (lane == 0) {
      tma_store_3d(&tm_out, sbase + L::kState + warp * 2048, 0, 16 * warp, chain);
      tma_store_3d(&tm_out, sbase + L::kState + 16384 + warp * 2048, 64, 16 * warp, chain);
      bulk_commit();
      bulk_wait_read0();
    }
  }
}

}  // namespace short16

cudaError_t launch_short16(const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* v, const __nv_bfloat16* g,
                           const __nv_bfloat16* beta, const float* A_log, const float* dt_bias, const void* initial_state,
                           void* final_state, __nv_bfloat16* out, int64_t N, int T, int H, int state_fp32, float scale,
                           float gate_scale, int* status, cudaStream_t stream) {
  if (N * H == 0) return cudaSuccess;
  using namespace short16;
  const Params p{q, k, v, g, beta, A_log, dt_bias, initial_state, final_state, out, T, H, scale, gate_scale, status};
  const int form = 3 * (state_fp32 ? 1 : 0) + (T <= kRows8 ? 2 : T <= kRows ? 1 : 0);
  void (*const kernels[6])(CUtensorMap, CUtensorMap, Params) = {short16_kernel<false, false>, short16_kernel<false, true>, short8_kernel<false>,
                                                                short16_kernel<true, false>, short16_kernel<true, true>, short8_kernel<true>};
  constexpr int sizes[6] = {Lay<true, false>::kSmemBytes, Lay<false, true>::kSmemBytes, Lay8<false>::kSmemBytes,
                            Lay<true, false>::kSmemBytes, Lay<true, true>::kSmemBytes, Lay8<true>::kSmemBytes};
  const int smem = sizes[form];
  static SmemOptIn opt_in[6];
  cudaError_t e = opt_in[form].ensure(kernels[form], smem);
  if (e != cudaSuccess) return e;
  CUtensorMap in{}, fin{};
  if ((form == 1 || form == 2) && ((initial_state != nullptr && !make_state_map(&in, initial_state, N * H, kD)) ||
                    (final_state != nullptr && !make_state_map(&fin, final_state, N * H, 16))))
    return cudaErrorInvalidValue;
  return launch_after(kernels[form], static_cast<unsigned>(N * H), kThreads, smem, stream, in, fin, p);
}

}  // namespace fkda
