// Segment-parallel form of the inter-chunk recurrence for batches with few, long chains.
//
// The reference walks every (sequence, head) chain with one CTA from the first chunk to the last
// (csrc/smxx/fwd_kernel2.cuh:434-742), so a call with fewer chains than SMs leaves most of the GPU idle.  A run
// of chunks acts on the state Z = S^T ([v][k]) as an affine map, Z_end = Z_start M + N, because every chunk does
//     Z' = Z (diag(e) - w'^T kr) + u'^T kr ,          w' = T diag(beta) k+,  u' = T diag(beta) v .
// Here each sequence is cut into runs, whose maps are worked out in parallel, this file chains them into the state at the start of
// every run, and a second pass walks all runs in parallel from those states.  Over compact records maps_kernel gives M and N of every
// run but the last, and finds the maps that are zero, which need no chaining (fkda_recur.cu); recur_kernel walks the runs.  In the
// two-stage form the look-ahead or the compact kernel, whichever gets the pass's CTAs through faster, gives M (walk from the
// identity with v = 0) and N (walk from zero) of the inner runs while run 0 is walked from the caller's state, and then walks the
// others.
#include "fkda_common.cuh"

namespace fkda {

cudaError_t launch_scan2(const ScanParams& p, cudaStream_t stream);
cudaError_t launch_recur(const ScanParams& p, const __nv_bfloat16* v, cudaStream_t stream);
cudaError_t launch_scan(const ScanParams& p, cudaStream_t stream);

namespace {

// Two-stage form: whether a pass of `ctas` CTAs takes less time on the compact kernel (two CTAs per SM at 1.58 times the
// chunk step, measured) than on the look-ahead kernel (one).
bool compact_is_faster(int64_t ctas, int64_t sms) {
  return (ctas + 2 * sms - 1) / (2 * sms) * 158 < (ctas + sms - 1) / sms * 100;
}

constexpr int kCmbRows = 8;                               // state rows per CTA: the n of an mma, whose m are columns of the map
constexpr int kMapStride = kSegMapStride;                 // floats per map row, in its slot and here (fragments: bank 8 t + g)
constexpr int kMapStg = kD * kMapStride * 4;
constexpr int kMapBufs = 3;                               // maps in flight
constexpr int kCmbM = 0;                                  // kMapBufs x [128][136] fp32: transition maps
constexpr int kCmbZ = kCmbM + kMapBufs * kMapStg;         // [16 k-steps][32 lanes]: this CTA's rows of the state as B fragments, leading and trailing parts
constexpr int kCmbPart = kCmbZ + 16 * 512;                // [8 warps][32 lanes][4] fp32: partial sums of the upper half of k
constexpr int kCmbBars = kCmbPart + 8 * 512;
constexpr int kCmbList = kCmbBars + 64;                   // the runs, a byte each
constexpr int kCmbThreads = 512;
constexpr int kCmbSmemBytes = kCmbList + 256 + 128;
static_assert(kCmbSmemBytes <= 227 * 1024, "map buffers fit one SM");

// x = hi + lo, both tf32, hi rounded to nearest (away from zero on ties, as cvt.rna does) by integer arithmetic: the
// conversion instruction issues at a fraction of that rate.  lo <= 2^-11 |x| is cut off 2^-21 below x.
__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
  hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
  lo = __float_as_uint(x - __uint_as_float(hi)) & 0xffffe000u;
}

// Z_start[run + 1] = Z_start[run] M[run] + N[run] for run = first .. n_segs-2, Z_start[first] in its slot; rows of Z are independent, so each CTA
// carries eight of them through all runs, as Z^T[run + 1] = M^T Z^T + N^T.  The maps arrive by bulk copies (one per map: its
// slot holds it with padded rows) three runs ahead.  The products run on the tensor cores in tf32 with both operands split into a leading and a
// trailing part (three mma per tile: the error of the split, about 2^-21 relative, is that of an fp32 product), fp32
// accumulation on top of N.
// What bounds it: the serial chain of runs.  So a run's map waits in registers, split, before the state that it is applied to
// is there: each k-step's fragments are replaced by the next run's as soon as its products are issued, in the issue slots
// that these leave.  What remains on the chain is 48 mma per warp and one exchange of the state through shared memory, split
// once by its producer.  Per run: 3.2 us with sixteen rows per CTA and both operands read and split on the chain, 1.4 us now
// (2 heads of 65536 tokens: 331 -> 274 us).  Sixteen warps, two per sixteen columns with half of k each: with eight the loop is 8 KB of code,
// which the instruction caches no longer hold (1.7 us).
// Runs whose map is zero (`flagged`: their words are looked at) are left out: the state behind such a run is in its slot already.
__global__ void __launch_bounds__(kCmbThreads, 1)
seg_combine_kernel(float* seg_buf, int n_segs, int first, int flagged, int* status, int wait_limit_us, int stop_maps_after) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~static_cast<uintptr_t>(127));
  const uint32_t sbase = smem_u32(smem);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + kCmbBars + 32);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  float* slots = seg_buf + static_cast<size_t>(blockIdx.x) * n_segs * 3 * kSegSlotFloats;
  const int r_base = blockIdx.y * kCmbRows;
  // the runs whose maps are applied, in order
  uint8_t* list = smem + kCmbList;
  auto load_map = [&](int pos, int count) {      // one thread: the whole slot, rows padded as the recurrence kernel left them
    if (pos >= count || (stop_maps_after > 0 && pos >= stop_maps_after)) return;         // (test aid: the next wait for a map runs out)
    const int b = pos % kMapBufs, run = list[pos];
    mbar_arrive_expect_tx(sbase + kCmbBars + 8 * b, kMapStg);
    bulk_g2s(sbase + kCmbM + b * kMapStg, slots + (run * 3 + 0) * kSegSlotFloats, kMapStg, sbase + kCmbBars + 8 * b);
  };
  auto wait_map = [&](int pos) { return mbar_wait(sbase + kCmbBars + 8 * (pos % kMapBufs), (pos / kMapBufs) & 1, abort_flag); };
  // rows g, g + 8 of an m-tile stand for the columns n0 + 2 g, + 1, so that two fragment registers are one 8-byte load;
  // accumulators: rows 2 t, + 1 of the state (i & 1), those columns (i >> 1)
  auto put_z = [&](int n0, const float(&x)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int col = n0 + 2 * g + (i >> 1), row = 2 * t + (i & 1);
      uint32_t hi, lo;
      split_tf32(x[i], hi, lo);
      uint32_t* dst = reinterpret_cast<uint32_t*>(smem + kCmbZ) + (col >> 3) * 128 + (4 * row + (col & 3)) * 4 + ((col >> 2) & 1);
      dst[0] = hi;
      dst[2] = lo;
    }
  };
  if (tid == 0) {
    *abort_flag = -wait_limit_us;       // (below zero: a wait limit, test aid)
    for (int i = 0; i < kMapBufs; ++i) mbar_init(sbase + kCmbBars + 8 * i, 1);
    fence_mbar_init();
  }
  __syncthreads();
  grid_dependency_wait();
  if (warp == 0) {
    int n = 0;
    for (int base = first; base + 1 < n_segs; base += 32) {
      const int run = base + lane;
      const bool use = run + 1 < n_segs && (!flagged || *seg_zero_word(slots, run) == 0);
      const unsigned mask = __ballot_sync(0xffffffffu, use);
      if (use) list[n + __popc(mask & ((1u << lane) - 1u))] = static_cast<uint8_t>(run);
      n += __popc(mask);
    }
    if (lane == 0) *reinterpret_cast<volatile int*>(smem + kCmbBars + 40) = n;
  }
  __syncthreads();
  const int count = *reinterpret_cast<volatile int*>(smem + kCmbBars + 40);
  if (count == 0) return;
  if (tid == 0)
    for (int pos = 0; pos < kMapBufs; ++pos) load_map(pos, count);
  const int n0 = (warp & 7) * 16, half = warp >> 3;        // this warp's sixteen output columns, its half of k
  // a CTA's rows of a slot in the accumulators' layout
  auto load_rows = [&](const float* slot, float (&d)[4]) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float2 y = *reinterpret_cast<const float2*>(slot + static_cast<size_t>(r_base + 2 * t + i) * kD + n0 + 2 * g);
      d[i] = y.x;
      d[2 + i] = y.y;
    }
  };
  float x[4], next_n[4];                 // N of a run is fetched one run ahead
  load_rows(slots + (list[0] * 3 + 2) * kSegSlotFloats, x);      // the state at the start of that run
  if (half == 0) put_z(n0, x);
  load_rows(slots + (list[0] * 3 + 1) * kSegSlotFloats, next_n);
  // this warp's columns of a map, split: [k-step][leading, trailing part][A fragment]
  uint32_t m[8][2][4];
  auto load_m = [&](int pos, int ks) {
    const float* M = reinterpret_cast<const float*>(smem + kCmbM + (pos % kMapBufs) * kMapStg) + (64 * half + 8 * ks + t) * kMapStride + n0 + 2 * g;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float2 y = *reinterpret_cast<const float2*>(M + 4 * e * kMapStride);
      split_tf32(y.x, m[ks][0][2 * e], m[ks][1][2 * e]);
      split_tf32(y.y, m[ks][0][2 * e + 1], m[ks][1][2 * e + 1]);
    }
  };
  bool ok = wait_map(0);
#pragma unroll
  for (int ks = 0; ks < 8; ++ks) load_m(0, ks);
  for (int pos = 0;; ++pos) {
    if (!__syncthreads_and(ok)) {
      if (tid == 0) {
        atomicCAS(status, kStatusOk, kStatusWaitTimeout);
        // do not leave while a copy may still be landing in this CTA's shared memory
        for (int q = pos; q < pos + kMapBufs && q < count; ++q) {     // the maps that have been asked for
          const uint64_t t0 = globaltimer_ns();
          while (!mbar_try_wait(sbase + kCmbBars + 8 * (q % kMapBufs), (q / kMapBufs) & 1))
            if (globaltimer_ns() - t0 > 20000000ull) break;
        }
      }
      break;
    }
    // here: z holds the state at the start of the run, m its map, whose buffer is free
    if (pos >= count) break;
    const int run = list[pos];
    if (tid == 0) load_map(pos + kMapBufs, count);
    float acc[3][4];                  // hi hi on top of N, lo hi, hi lo
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      acc[0][i] = half == 0 ? next_n[i] : 0.f;
      acc[1][i] = acc[2][i] = 0.f;
    }
    float jump[4] = {0.f, 0.f, 0.f, 0.f};       // the next map is not the next run's: the state in front of it, from its slot
    bool jumps = false;
    if (pos + 1 < count) {
      const int to = list[pos + 1];
      jumps = to != run + 1;
      if (half == 0) {
        load_rows(slots + (to * 3 + 1) * kSegSlotFloats, next_n);
        if (jumps) load_rows(slots + (to * 3 + 2) * kSegSlotFloats, jump);
      }
      ok = wait_map(pos + 1);
    }
    if (tid < 32 && pos + 4 < count)     // and the lines of a later N into the L2: eight rows of 512 bytes
      asm volatile("prefetch.global.L2 [%0];" ::"l"(slots + (list[pos + 4] * 3 + 1) * kSegSlotFloats +
                                                     static_cast<size_t>(r_base + (tid >> 2)) * kD + (tid & 3) * 32));
    const uint4* z = reinterpret_cast<const uint4*>(smem + kCmbZ) + 256 * half + lane;
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      const uint4 b = z[32 * ks];     // two registers of the leading part, two of the trailing one
      mma_tf32_1688(acc[1], m[ks][1][0], m[ks][1][1], m[ks][1][2], m[ks][1][3], b.x, b.y);
      mma_tf32_1688(acc[2], m[ks][0][0], m[ks][0][1], m[ks][0][2], m[ks][0][3], b.z, b.w);
      mma_tf32_1688(acc[0], m[ks][0][0], m[ks][0][1], m[ks][0][2], m[ks][0][3], b.x, b.y);
      load_m(pos + 1, ks);            // (behind the last one: whatever the buffer holds, not used)
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = acc[0][i] + (acc[1][i] + acc[2][i]);
    float4* part = reinterpret_cast<float4*>(smem + kCmbPart) + (warp & 7) * 32 + lane;
    if (half == 1) *part = make_float4(x[0], x[1], x[2], x[3]);
    __syncthreads();                  // every thread is done with z; the partial sums are there
    if (half == 0) {
      const float4 y = *part;
      x[0] += y.x;
      x[1] += y.y;
      x[2] += y.z;
      x[3] += y.w;
      float* zs = slots + ((run + 1) * 3 + 2) * kSegSlotFloats;
#pragma unroll
      for (int i = 0; i < 2; ++i)
        *reinterpret_cast<float2*>(zs + static_cast<size_t>(r_base + 2 * t + i) * kD + n0 + 2 * g) = make_float2(x[i], x[2 + i]);
      if (jumps) {
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = jump[i];
      }
      put_z(n0, x);
    }
  }
}

}  // namespace

// v: the value tensor where the records are the compact ones (both passes then run on the register-resident kernel), else nullptr
cudaError_t launch_scan_segmented(const ScanParams& base, int n_segs, int seg_chunks, float* seg_buf, int kernel_choice, const __nv_bfloat16* v,
                                  cudaStream_t stream) {
  ScanParams p = base;
  p.seg_chunks = seg_chunks;
  p.n_segs = n_segs;
  p.seg_buf = seg_buf;
  const int64_t chains = static_cast<int64_t>(p.N) * p.H;
  const int sms = device_sm_count();
  bool compact1 = compact_is_faster(chains * (2 * n_segs - 3), sms), compact2 = compact_is_faster(chains * (n_segs - 1), sms);
  if (kernel_choice) compact1 = compact2 = kernel_choice == 1;   // forced: 1 compact, 2 look-ahead
  p.seg_pass = v != nullptr ? kSegMaps : 1;
  cudaError_t e = v != nullptr ? launch_recur(p, v, stream) : compact1 ? launch_scan(p, stream) : launch_scan2(p, stream);
  if (e != cudaSuccess) return e;
  if (n_segs > 2 || v != nullptr) {
    static SmemOptIn opt_in;
    e = opt_in.ensure(seg_combine_kernel, kCmbSmemBytes);
    if (e != cudaSuccess) return e;
    const dim3 grid(static_cast<unsigned>(chains), kD / kCmbRows);
    e = launch_after(seg_combine_kernel, grid, kCmbThreads, kCmbSmemBytes, stream, seg_buf, n_segs, v != nullptr ? 0 : 1,
                     v != nullptr && p.stop_maps_after == 0 ? 1 : 0, p.status, p.map_wait_limit_us, p.stop_maps_after);
    if (e != cudaSuccess) return e;
  }
  p.seg_pass = v != nullptr ? kSegWalks : 2;
  return v != nullptr ? launch_recur(p, v, stream) : compact2 ? launch_scan(p, stream) : launch_scan2(p, stream);
}

}  // namespace fkda
