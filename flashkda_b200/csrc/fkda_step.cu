// The forward pass of a few tokens per sequence (decode and speculative steps): the per-token recurrence in fp32.
//
// Replaces, for these shapes, both of the reference's kernels (csrc/smxx/fwd_kernel1.cuh:107-586, fwd_kernel2.cuh:115-839),
// which pad every sequence to a 16-token tile.  Per token, with e = 2^gate and S [k][v] (stored [v][k]):
//     u = beta (v - (e k)^T S),   o = (e q)^T S + (k.q) u,   S = diag(e) S + k u^T
// A CTA of four warps owns the 128 rows v of one chain, 32 at a time with the next 32 on their way; where there are too few
// chains to fill the chip, 32 of them only, so that a single sequence already spreads over four SMs per head.
// Sixteen lanes share four rows, each with eight of their channels in registers: a vector element read from shared memory then
// serves four rows (with four lanes to a row the reads alone took 2100 cycles per token, chain and SM), and the eight dot
// products of a token fold into one value per lane on the way through the reduction.  Every CTA works out the tokens'
// vectors for itself (a few hundred elements) while its rows of the state arrive.
//
// In a packed batch it runs beside the recurrence over the longer sequences, on the SMs that this leaves free: it reads none of
// the call's intermediate results, and when the recurrence starts, all that came before the call is complete.  One CTA waits for
// the recurrence at its end, so that a kernel that waits for this one waits for both.
//
// What bounds it: the stream over the states at one token (512 x 32 chains: 173 us with bf16 states, 324 with fp32:
// 6.3 and 6.7 TB/s, the measured copy rate; the tile kernel, whose time hardly depends on the tokens, 273 and 425), then the shared-memory pipe: 840 cycles per token,
// chain and SM, 512 of them the reads of the vectors, 230 the shuffles.  Above kStepMaxT the tile form
// (fkda_short16.cu) takes over.
#include "fkda_common.cuh"
#include "fkda_elem.cuh"

namespace fkda {
namespace step {

constexpr int kThreads = 128;
constexpr int kRows = 32;
constexpr int kTokenBytes = 4 * kD * 4 + kD * 4 + kD * 2 + 8;
static_assert(kTokenBytes * kStepMaxT <= 48 * 1024, "shared memory without an opt-in");

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
  const int64_t* cu_seqlens;   // packed batch: only sequences of at most kStepMaxT tokens are done here; or nullptr
  int64_t T_total;
  int T;                 // tokens per sequence (packed: kStepMaxT)
  int H;
  float scale;
  float gate_scale;      // lower_bound * log2(e)
};

using elem::f2;
using elem::fma2;
using elem::mul;
using elem::pk;
__device__ __forceinline__ float sum2(f2 x) {
  float a, b;
  elem::upk(x, a, b);
  return a + b;
}
__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) x += __shfl_xor_sync(0xffffffffu, x, d);
  return x;
}

// kFp32: type of the state tensors; kWhole: a CTA does the whole chain, else a quarter of its rows
template <bool kFp32, bool kWhole, bool kPacked>
__global__ void __launch_bounds__(kThreads, kWhole ? 5 : 6) step_kernel(const Params p) {
  // per token, sized by T so that short steps leave room for more CTAs: e k | e q | e | k; v; the outputs; beta, k.q
  extern __shared__ __align__(16) uint8_t smem[];
  constexpr int kOwn = kWhole ? kD : kRows;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int chain = static_cast<int>(kWhole ? blockIdx.x : blockIdx.x >> 2), row0 = kWhole ? 0 : static_cast<int>(blockIdx.x & 3) * kRows;
  const int n = chain / p.H, h = chain - n * p.H;
  if (!kPacked) grid_dependency_wait();
  int T = p.T;
  int64_t bos = static_cast<int64_t>(n) * p.T;
  if constexpr (kPacked) {
    int64_t eos = p.cu_seqlens[n + 1];
    bos = p.cu_seqlens[n];
    bos = bos < 0 ? 0 : (bos > p.T_total ? p.T_total : bos);
    eos = eos < bos ? bos : (eos > p.T_total ? p.T_total : eos);
    if (eos - bos > kStepMaxT) {
      if (blockIdx.x == 0) grid_dependency_wait();
      return;
    }
    T = static_cast<int>(eos - bos);
  }
  float4(*const s_vec)[4][kD / 4] = reinterpret_cast<float4(*)[4][kD / 4]>(smem);
  float(*const s_v)[kOwn] = reinterpret_cast<float(*)[kOwn]>(smem + static_cast<size_t>(p.T) * 4 * kD * 4);
  __nv_bfloat16(*const s_out)[kOwn] = reinterpret_cast<__nv_bfloat16(*)[kOwn]>(s_v + p.T);
  float* const s_beta = reinterpret_cast<float*>(s_out + p.T);
  float* const s_kq = s_beta + p.T;
  // this thread: rows rows4 .. + 3 of the 32 at hand, channels 4 j .. + 3 and 64 + 4 j .. + 3
  const int j = lane & 15, rows4 = 8 * warp + 4 * (lane >> 4);
  const size_t state_off = (static_cast<size_t>(chain) * kD + row0 + rows4) * kD + 4 * j;

  using Raw = typename std::conditional<kFp32, float4, uint2>::type;
  Raw raw[8];
  auto load = [&](int part) {
    if (p.initial_state == nullptr) {
#pragma unroll
      for (int i = 0; i < 8; ++i) raw[i] = Raw{};
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const size_t off = state_off + static_cast<size_t>(part) * kRows * kD + (i >> 1) * kD + 64 * (i & 1);
        if constexpr (kFp32) raw[i] = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(p.initial_state) + off));
        else raw[i] = __ldg(reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(p.initial_state) + off));
      }
    }
  };
  load(0);

  // ---- the tokens' vectors, a warp per token, four channels per lane -----------------------------------------------
  const float ha = 0.5f * ex2f(__ldg(p.A_log + h) * kLog2e), hgs = 0.5f * p.gate_scale;
  const float4 bias = __ldg(reinterpret_cast<const float4*>(p.dt_bias + h * kD) + lane);
  for (int t = warp; t < T; t += 4) {
    const size_t tok = static_cast<size_t>(bos + t) * p.H + h;
    const uint2 qw = __ldg(reinterpret_cast<const uint2*>(p.q + tok * kD) + lane);
    const uint2 kw = __ldg(reinterpret_cast<const uint2*>(p.k + tok * kD) + lane);
    const uint2 gw = __ldg(reinterpret_cast<const uint2*>(p.g + tok * kD) + lane);
    uint2 vw = make_uint2(0u, 0u);
    if constexpr (kWhole) vw = __ldg(reinterpret_cast<const uint2*>(p.v + tok * kD) + lane);
    else vw.x = *reinterpret_cast<const uint16_t*>(p.v + tok * kD + row0 + lane);
    const float bb = __bfloat162float(p.beta[tok]);
    float4 q = make_float4(bf_lo(qw.x), bf_hi(qw.x), bf_lo(qw.y), bf_hi(qw.y));
    float4 k = make_float4(bf_lo(kw.x), bf_hi(kw.x), bf_lo(kw.y), bf_hi(kw.y));
    float4 e;
    e.x = ex2f(fmaf(tanh_approx(fmaf(bf_lo(gw.x), ha, ha * bias.x)), hgs, hgs));
    e.y = ex2f(fmaf(tanh_approx(fmaf(bf_hi(gw.x), ha, ha * bias.y)), hgs, hgs));
    e.z = ex2f(fmaf(tanh_approx(fmaf(bf_lo(gw.y), ha, ha * bias.z)), hgs, hgs));
    e.w = ex2f(fmaf(tanh_approx(fmaf(bf_hi(gw.y), ha, ha * bias.w)), hgs, hgs));
    const float rq = rsqrtf(warp_sum(fmaf(q.x, q.x, fmaf(q.y, q.y, fmaf(q.z, q.z, q.w * q.w)))) + 1e-6f) * p.scale;
    const float rk = rsqrtf(warp_sum(fmaf(k.x, k.x, fmaf(k.y, k.y, fmaf(k.z, k.z, k.w * k.w)))) + 1e-6f);
    q = make_float4(q.x * rq, q.y * rq, q.z * rq, q.w * rq);
    k = make_float4(k.x * rk, k.y * rk, k.z * rk, k.w * rk);
    const float kq = warp_sum(fmaf(q.x, k.x, fmaf(q.y, k.y, fmaf(q.z, k.z, q.w * k.w))));
    s_vec[t][0][lane] = make_float4(e.x * k.x, e.y * k.y, e.z * k.z, e.w * k.w);
    s_vec[t][1][lane] = make_float4(e.x * q.x, e.y * q.y, e.z * q.z, e.w * q.w);
    s_vec[t][2][lane] = e;
    s_vec[t][3][lane] = k;
    if constexpr (kWhole) *reinterpret_cast<float4*>(&s_v[t][4 * lane]) = make_float4(bf_lo(vw.x), bf_hi(vw.x), bf_lo(vw.y), bf_hi(vw.y));
    else s_v[t][lane] = bf_lo(vw.x);
    if (lane == 0) {
      s_beta[t] = sigmoid_fast(bb);
      s_kq[t] = kq;
    }
  }
  __syncthreads();

  // ---- token by token ---------------------------------------------------------------------------------------------
  // which of the eight sums a lane ends up with: bit 3 = the dot with q, bits 2, 1 = the row
  const bool is_o = (lane & 8) != 0, hi2 = (lane & 4) != 0, hi1 = (lane & 2) != 0;
  for (int part = 0; part < (kWhole ? kD / kRows : 1); ++part) {
    f2 S[4][4];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if constexpr (kFp32) {
        S[i >> 1][2 * (i & 1)] = pk(raw[i].x, raw[i].y);
        S[i >> 1][2 * (i & 1) + 1] = pk(raw[i].z, raw[i].w);
      } else {
        S[i >> 1][2 * (i & 1)] = pk(bf_lo(raw[i].x), bf_hi(raw[i].x));
        S[i >> 1][2 * (i & 1) + 1] = pk(bf_lo(raw[i].y), bf_hi(raw[i].y));
      }
    }
    if (kWhole && part + 1 < kD / kRows) load(part + 1);
    const int my_row = kRows * part + rows4 + ((lane >> 1) & 3);
    for (int t = 0; t < T; ++t) {
      const ulonglong2* vec = reinterpret_cast<const ulonglong2*>(s_vec[t]) + j;       // e k | e q | e | k, 32 groups of four each
      float sum[8];
      {
        const ulonglong2 a0 = vec[0], a1 = vec[16], b0 = vec[32], b1 = vec[48];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          sum[r] = sum2(fma2(S[r][0], a0.x, fma2(S[r][1], a0.y, fma2(S[r][2], a1.x, mul(S[r][3], a1.y)))));
          sum[4 + r] = sum2(fma2(S[r][0], b0.x, fma2(S[r][1], b0.y, fma2(S[r][2], b1.x, mul(S[r][3], b1.y)))));
        }
      }
      float x[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) x[r] = (is_o ? sum[4 + r] : sum[r]) + __shfl_xor_sync(0xffffffffu, is_o ? sum[r] : sum[4 + r], 8);
      const float y0 = (hi2 ? x[2] : x[0]) + __shfl_xor_sync(0xffffffffu, hi2 ? x[0] : x[2], 4);
      const float y1 = (hi2 ? x[3] : x[1]) + __shfl_xor_sync(0xffffffffu, hi2 ? x[1] : x[3], 4);
      float z = (hi1 ? y1 : y0) + __shfl_xor_sync(0xffffffffu, hi1 ? y0 : y1, 2);
      z += __shfl_xor_sync(0xffffffffu, z, 1);
      const float u = s_beta[t] * (s_v[t][my_row] - z);                               // (lanes with bit 3 clear)
      const float u_of_row = __shfl_sync(0xffffffffu, u, lane & ~8);
      if ((lane & 9) == 8) s_out[t][my_row] = __float2bfloat16_rn(fmaf(s_kq[t], u_of_row, z));
      const ulonglong2 e0 = vec[64], e1 = vec[80], k0 = vec[96], k1 = vec[112];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float ur = __shfl_sync(0xffffffffu, u, (lane & 16) | (2 * r));
        const f2 u2 = pk(ur, ur);
        S[r][0] = fma2(S[r][0], e0.x, mul(k0.x, u2));
        S[r][1] = fma2(S[r][1], e0.y, mul(k0.y, u2));
        S[r][2] = fma2(S[r][2], e1.x, mul(k1.x, u2));
        S[r][3] = fma2(S[r][3], e1.y, mul(k1.y, u2));
      }
    }
    if (p.final_state != nullptr) {
      const size_t off = state_off + static_cast<size_t>(part) * kRows * kD;
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if constexpr (kFp32) {
            *reinterpret_cast<ulonglong2*>(static_cast<float*>(p.final_state) + off + r * kD + 64 * i) = make_ulonglong2(S[r][2 * i], S[r][2 * i + 1]);
          } else {
            float a, b, c, d;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(S[r][2 * i]));
            asm("mov.b64 {%0, %1}, %2;" : "=f"(c), "=f"(d) : "l"(S[r][2 * i + 1]));
            *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.final_state) + off + r * kD + 64 * i) = make_uint2(pack_bf16(a, b), pack_bf16(c, d));
          }
        }
    }
  }
  __syncthreads();
  // the outputs in 16-byte pieces
  constexpr int kPieces = kOwn / 8;
  for (int i = tid; i < kPieces * T; i += kThreads) {
    const int t = i / kPieces, c = (i % kPieces) * 8;
    *reinterpret_cast<uint4*>(p.out + (static_cast<size_t>(bos + t) * p.H + h) * kD + row0 + c) = *reinterpret_cast<const uint4*>(&s_out[t][c]);
  }
  if (kPacked && blockIdx.x == 0) grid_dependency_wait();
}

}  // namespace step

// cu_seqlens == nullptr: N sequences of T tokens; else the sequences of at most kStepMaxT tokens of a packed batch
cudaError_t launch_step(const PrepParams& p, const ScanParams& s, cudaStream_t stream) {
  const int64_t chains = static_cast<int64_t>(s.N) * s.H;
  if (chains == 0) return cudaSuccess;
  const bool packed = s.cu_seqlens != nullptr;
  const int T = packed ? static_cast<int>(kStepMaxT) : static_cast<int>(s.T);
  const step::Params q{p.q, p.k, p.v, p.g, p.beta, p.A_log, p.dt_bias, s.initial_state, s.final_state, s.out, s.cu_seqlens, s.T_total,
                       T, s.H, p.scale, p.gate_scale};
  // whole chains once they give every SM a full set of CTAs
  const bool whole = packed || chains >= 5ll * device_sm_count();
  auto kernel = packed ? (s.state_fp32 ? step::step_kernel<true, true, true> : step::step_kernel<false, true, true>)
                : s.state_fp32 ? (whole ? step::step_kernel<true, true, false> : step::step_kernel<true, false, false>)
                               : (whole ? step::step_kernel<false, true, false> : step::step_kernel<false, false, false>);
  return launch_after(kernel, static_cast<unsigned>(whole ? chains : 4 * chains), step::kThreads, static_cast<size_t>(step::kTokenBytes) * T, stream, q);
}

}  // namespace fkda
