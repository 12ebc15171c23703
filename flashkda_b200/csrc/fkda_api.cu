// C ABI of the library (include/fkda.h): argument validation, workspace carving and launches.
// Host-side counterpart of the reference's csrc/flash_kda.cpp (validation, dispatch) and
// csrc/smxx/fwd_launch.cu (workspace carving, launches), without torch types.
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>

#include "../../include/fkda.h"
#include "../../include/fkda_testing.h"
#include "fkda_common.cuh"

namespace fkda {
cudaError_t launch_chunk_prefix(const int64_t* cu, int N, int64_t T_total, int H, int n_segs, bool skip_short, int* prefix, int* status,
                                cudaStream_t stream);
cudaError_t launch_prepare(const PrepParams& p, cudaStream_t stream);
cudaError_t launch_prepare_tc4(const PrepParams& p, cudaStream_t stream);
cudaError_t launch_prepare_pipe(const PrepParams& p, cudaStream_t stream);
cudaError_t launch_scan(const ScanParams& p, cudaStream_t stream);
cudaError_t launch_scan_simt(const ScanParams& p, cudaStream_t stream);
cudaError_t launch_scan2(const ScanParams& p, cudaStream_t stream);
cudaError_t launch_recur_split(const ScanParams& p, const __nv_bfloat16* v, int rows, cudaStream_t stream);
cudaError_t launch_operands(const PrepParams& p, bool one_per_cta, cudaStream_t stream);
cudaError_t launch_recur(const ScanParams& p, const __nv_bfloat16* v, cudaStream_t stream);
cudaError_t launch_scan_short(const ScanParams& p, int sm_count, cudaStream_t stream);
cudaError_t launch_short16(const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* v, const __nv_bfloat16* g,
                           const __nv_bfloat16* beta, const float* A_log, const float* dt_bias, const void* initial_state,
                           void* final_state, __nv_bfloat16* out, int64_t N, int T, int H, int state_fp32, float scale,
                           float gate_scale, int* status, cudaStream_t stream);
cudaError_t launch_step(const PrepParams& p, const ScanParams& s, cudaStream_t stream);
cudaError_t launch_refmode(const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* v, const __nv_bfloat16* g,
                           const __nv_bfloat16* beta, const float* A_log, const float* dt_bias, const void* initial_state,
                           void* final_state, __nv_bfloat16* out, const int64_t* cu_seqlens, int64_t N, int64_t T, int64_t T_total,
                           int H, int state_fp32, float scale, float gate_scale, cudaStream_t stream);
cudaError_t launch_scan_segmented(const ScanParams& base, int n_segs, int seg_chunks, float* seg_buf, int kernel_choice, const __nv_bfloat16* v,
                                  cudaStream_t stream);
#ifdef FKDA_TUNING
void set_prepare_trace(long long* buf);
void set_scan_trace(unsigned long long* buf);
cudaError_t launch_tmem_bench(int nwarps, int reps, long long* out, cudaStream_t stream);
cudaError_t launch_umma_bench(int nissuers, int reps, int ksteps, int n, int ts, long long* out, int* status, cudaStream_t stream);
#endif
cudaError_t launch_tmem_layout_probe(uint32_t* out, cudaStream_t stream);
cudaError_t launch_prologue(const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* g, const __nv_bfloat16* beta,
                            const float* A_log, const float* dt_bias, float gate_scale, int64_t rows, int H, __nv_bfloat16* qn,
                            __nv_bfloat16* kn, float* gact, float* beta_act, cudaStream_t stream);
cudaError_t launch_umma_selftest(const __nv_bfloat16* A, const __nv_bfloat16* B, float* D, int mode, int reps, int* status,
                                 cudaStream_t stream);
}  // namespace fkda

namespace {

thread_local char g_err[512] = "";

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

int cuda_fail(cudaError_t e, const char* what) {
  return fail(FKDA_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

struct Layout {
  int64_t prefix_off;      // int32 [N+1]
  int64_t records_off;
  int64_t chunks_per_head; // records per head
  int64_t seg_off;         // fp32 slots of the segment-parallel scan (seg_bytes may be 0)
  int64_t seg_bytes;
  int n_segs;              // runs per sequence (1: whole sequences), of seg_chunks chunks each
  int seg_chunks;
  int64_t total_bytes;
};

// How many runs to cut each sequence of a batch into (1 = walk whole sequences), at most `most` of them, and their length in
// chunks.  The first pass has a CTA for every run but the last, which works out the run's map M and offset N; the second one a CTA
// per run.  Where the gates' decay makes M vanish, which the first pass finds out (fkda_recur.cu), its two walks are a few chunks
// long; where it does not, they are as long as the run, beside one another if a CTA for each is resident, and the maps are chained.  The plan
// is made for the former, among those that cost in the latter at most a tenth more than whole sequences and no more than `before`: the
// best plan of the form that walked M and N forwards in a CTA each whatever the gates (its own fitted costs), which a call that never forgets
// must not fall behind.  Microseconds without decay / with, chains x chunks, that form, a twelfth above the best plan instead, now:
// 1 x 4096 346, 372 / 122, 305 / 145; 2 x 700 154, 166 / 74, 143 / 81; 3 x 700 169, 172 / 84, 152 / 96; 1 x 1500 207, 225 / 82, 203 / 86.
// Where that form was not worth it, a twelfth above the best plan: 24 x 256 265 / 162 against 239 in whole sequences.
// Of plans within 5 % and 3 us, which is what the costs are off by, the one with the fewest runs.  The one planner: the workspace size, the launch and fkda_plan_segments ask here.
// Its costs are those of the default path's kernels, in hundredths of a microsecond, fitted to 150 timed calls of 1 to 48
// heads and 64 to 4096 chunks, half of them without decay: a chunk step of a chain split over four or two CTAs (fkda_recur_split.cu) or
// in one CTA (fkda_recur.cu), the latter with and without outputs; the chunks that a map takes to vanish; what the passes cost
// beside their steps, and every round of CTAs after the first; the chaining of the maps per run and round of its CTAs.  (The
// two-stage form walks its runs by the same plan.)
int plan_runs(int64_t chains, int64_t chunks, int64_t most, int sms, int* len) {
  constexpr int64_t kQuad = 59, kHalf = 87, kOne = 108, kQuiet = 95, kVanish = 9, kPasses = 1300, kRound = 640, kChaining = 160, kMostRuns = 160, kLeast = 10;
  *len = 0;
  if (chains <= 0 || chains * 3 > sms || chunks < 48) return 1;
  const int64_t whole = (chains * 4 <= sms ? kQuad : kHalf) * chunks;
  auto rounds = [&](int64_t ctas) { return (ctas + sms - 1) / sms; };
  struct Cost { int64_t vanishing, lasting, before; };
  auto cost = [&](int64_t n, int64_t l) {
    const int64_t r1 = rounds(chains * (n - 1)), r2 = rounds(chains * n), common = r2 * kOne * l + kPasses + (r1 + r2 - 2) * kRound;
    const int64_t walks = chains * (n - 1) * 2 <= sms ? 1 : r1 * 2;
    const int64_t b1 = rounds(chains * (2 * n - 3)), b2 = rounds(chains * (n - 1));
    const bool slow_end = (chains - 1) * (2 * n - 3) >= (b1 - 1) * sms;      // run 0, with outputs, was in its first pass
    return Cost{common + r1 * 2 * kQuiet * (l < kVanish ? l : kVanish), common + walks * kQuiet * l + kChaining * (n - 1) * rounds(chains * 16),
                (slow_end ? (b1 - 1) * 88 + 132 : b1 * 88) * l + b2 * 132 * l + 1100 + (b1 + b2 - 2) * kRound + 165 * (n - 2) * rounds(chains * 16)};
  };
  int64_t least_lasting = INT64_MAX, before = whole, best = INT64_MAX;
  int best_n = 1;
  for (int pass = 0; pass < 3; ++pass) {
    for (int64_t n = 3; n <= (most < kMostRuns ? most : kMostRuns); ++n) {
      const int64_t l = (chunks + n - 1) / n;
      if (l < kLeast) break;
      if ((n - 1) * l >= chunks) continue;     // the last run would be empty
      const Cost c = cost(n, l);
      if (pass == 0) {
        if (c.lasting < least_lasting) least_lasting = c.lasting;
        if (c.before < before) before = c.before;
        continue;
      }
      if (c.lasting > (before == whole ? least_lasting * 13 / 12 : before > least_lasting ? before : least_lasting) || c.lasting * 100 > whole * 110 || c.vanishing * 100 > whole * 97) continue;
      if (pass == 1) {
        if (c.vanishing < best) best = c.vanishing;
      } else if (c.vanishing * 100 <= best * 105 && c.vanishing <= best + 300) {
        best_n = static_cast<int>(n);
        break;
      }
    }
  }
  if (best_n > 1) *len = static_cast<int>((chunks + best_n - 1) / best_n);
  return best_n;
}

// Runs per sequence under `flags`: forced by FKDA_FLAG_SEGMENTS(n), switched off by the
// kernel-selection flags, else planned from the sizes.
int segments_for(int64_t chains, int64_t chunks_per_seq, int64_t planned_chunks, int64_t most, int64_t flags, int* seg_chunks) {
  *seg_chunks = 0;
  if (flags & (FKDA_FLAG_SCAN_SIMT | FKDA_FLAG_SCAN_NO_SEGMENTS)) return 1;
  const int64_t forced = (flags >> 8) & 0xff;
  if ((flags & FKDA_FLAG_SCAN_PLAIN) && forced < 2) return 1;
  if (forced >= 2) {
    if (chunks_per_seq < forced || forced > most) return 1;
    *seg_chunks = static_cast<int>((chunks_per_seq + forced - 1) / forced);
    return static_cast<int>(forced);
  }
  if (flags & FKDA_FLAG_SCAN_LOOKAHEAD) return 1;
  // The planner tries up to 158 run counts with a dozen 64-bit divisions each (several microseconds), and a call asks
  // twice, a packed one for two lengths; it is a pure function of these four numbers, so each thread keeps its last two answers.
  struct Answer { int64_t chains = -1, chunks = -1, most = -1; int sms = -1, n = 1, len = 0; };
  thread_local Answer kept[2];
  thread_local int newest = 0;
  const int sms = fkda::device_sm_count();
  for (const Answer& a : kept)
    if (a.chains == chains && a.chunks == planned_chunks && a.most == most && a.sms == sms) {
      *seg_chunks = a.len;
      return a.n;
    }
  newest ^= 1;
  Answer& a = kept[newest];
  a.n = plan_runs(chains, planned_chunks, most, sms, &a.len);
  a.chains = chains;
  a.chunks = planned_chunks;
  a.most = most;
  a.sms = sms;
  *seg_chunks = a.len;
  return a.n;
}

constexpr int64_t kAnyRoom = INT64_MAX;

// `varlen` < 0: size for whichever mode needs more (the upper bound T_total/32 + N covers both).  `room`: no more runs are
// planned than fit a workspace of so many bytes.
bool make_layout(int64_t T_total, int64_t H, int64_t N, int varlen, int64_t T_per_seq, int64_t flags, Layout* L, int64_t room = kAnyRoom) {
  if (T_total < 0 || H <= 0 || N <= 0) return false;
  int64_t chunks;
  if (varlen == 0) chunks = N * ((T_per_seq + fkda::kChunk - 1) / fkda::kChunk);
  else chunks = T_total / fkda::kChunk + N;
  bool fixed = varlen == 0;
  if (varlen < 0) {
    int64_t fixed_ub = (T_total + fkda::kChunk - 1) / fkda::kChunk + N;
    chunks = fixed_ub > chunks ? fixed_ub : chunks;
    fixed = T_total % N == 0;                                         // a fixed-length call has T_total = N T
    if (fixed) T_per_seq = T_total / N;
  }
  L->prefix_off = fkda::kWsHeaderBytes;
  int64_t prefix_bytes = ((2 * N + 1) * 4 + 255) / 256 * 256;   // chunk prefix [N+1] followed by the chain order [N]
  L->records_off = L->prefix_off + prefix_bytes;
  L->chunks_per_head = chunks;
  L->seg_off = L->records_off + chunks * H * static_cast<int64_t>(fkda::kRecBytes);
  L->n_segs = 1;
  L->seg_chunks = 0;
  if (N * H <= 0x7fffffffLL) {
    const int64_t run_bytes = N * H * 3 * fkda::kSegSlotFloats * 4;
    const int64_t most = room == kAnyRoom ? room : room > L->seg_off ? (room - L->seg_off) / run_bytes : 0;
    auto chunks_of = [](int64_t tokens) { return (tokens + fkda::kChunk - 1) / fkda::kChunk; };
    // Fixed-length: planned from the sequence length.  Packed batches: the lengths are on the device.  The longest sequence sets
    // the time, one a third above the average is planned for, and the run length follows the longest one on the device; no more
    // runs than sequences of the average length would have, so that a size query, which does not know the mode, needs one plan.
    if (fixed) {
      L->n_segs = segments_for(N * H, chunks_of(T_per_seq), chunks_of(T_per_seq), most, flags, &L->seg_chunks);
    } else if (varlen != 0) {
      const int64_t average = chunks_of(T_total / N);
      L->n_segs = segments_for(N * H, average, chunks_of(N > 1 ? T_total * 4 / (N * 3) : T_total), most, flags, &L->seg_chunks);
      int len = 0;
      const int n = N > 1 ? segments_for(N * H, average, average, most, flags, &len) : L->n_segs;
      if (n < L->n_segs) {
        L->n_segs = n;
        L->seg_chunks = len;
      }
    }
  }
  L->seg_bytes = L->n_segs > 1 ? N * H * L->n_segs * 3 * fkda::kSegSlotFloats * 4 : 0;
  L->total_bytes = L->seg_off + L->seg_bytes;
  return true;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// whether the call takes the fused short-sequence kernel, which needs the workspace for its status word only
bool fused_short(const fkda_fwd_params* p) {
  const bool any_t = (p->flags & 0xff57u) == FKDA_FLAG_FUSED_ANY_T;
  return p->cu_seqlens == nullptr && p->T > 0 && (any_t || (p->T <= fkda::kFusedMaxT && (p->flags & 0xff57u) == 0));
}

// whether the call is one of the per-token kernel, and with it needs no scratch memory: that kernel has no wait whose end a
// status word could tell (FKDA_FLAG_REFERENCE_ROUNDING, not among the flags that fused_short looks at, comes first and clears the header)
bool takes_step_kernel(const fkda_fwd_params* p) {
  return fused_short(p) && p->T <= fkda::kStepMaxT && !(p->flags & (FKDA_FLAG_FUSED_ANY_T | FKDA_FLAG_REFERENCE_ROUNDING));
}
int64_t scratch_bytes(const fkda_fwd_params* p, const Layout& L) {
  if (!(p->flags & FKDA_FLAG_STATUS_UNREAD) || !fused_short(p)) return L.total_bytes;
  return takes_step_kernel(p) ? 0 : static_cast<int64_t>(fkda::kWsHeaderBytes);
}

// `whole_call`: the operator (fkda_fwd) rather than one of its stages; `fit`: its plan keeps to the given workspace
int validate(const fkda_fwd_params* p, Layout* L, bool whole_call = false, bool fit = false) {
  if (!p) return fail(FKDA_ERR_INVALID_ARGUMENT, "params is NULL");
  if (!p->q || !p->k || !p->v || !p->g || !p->beta || !p->out) return fail(FKDA_ERR_INVALID_ARGUMENT, "q, k, v, g, beta and out must be non-NULL");
  if (!p->A_log || !p->dt_bias) return fail(FKDA_ERR_INVALID_ARGUMENT, "A_log and dt_bias must be non-NULL");
  if (p->B <= 0 || p->H <= 0 || p->T < 0) return fail(FKDA_ERR_INVALID_ARGUMENT, "B and H must be positive and T non-negative");
  if (p->cu_seqlens) {
    if (p->B != 1) return fail(FKDA_ERR_INVALID_ARGUMENT, "B must be 1 when cu_seqlens is provided");
    if (p->N <= 0) return fail(FKDA_ERR_INVALID_ARGUMENT, "cu_seqlens must have at least 2 elements");
  } else if (p->N != p->B) {
    return fail(FKDA_ERR_INVALID_ARGUMENT, "N must equal B when cu_seqlens is not provided");
  }
  if ((p->initial_state || p->final_state) && p->state_dtype != FKDA_STATE_BF16 && p->state_dtype != FKDA_STATE_FP32)
    return fail(FKDA_ERR_INVALID_ARGUMENT, "state_dtype must be bf16 or fp32 when a state tensor is given");
  if (!std::isfinite(p->scale) || !std::isfinite(p->lower_bound)) return fail(FKDA_ERR_INVALID_ARGUMENT, "scale and lower_bound must be finite");
  if (p->lower_bound > 0.f || p->lower_bound < -5.2f)
    return fail(FKDA_ERR_INVALID_ARGUMENT, "lower_bound must lie in [-5.2, 0]: a 16-token sub-block may decay by at most 2^120");
  const void* ptrs[] = {p->q, p->k, p->v, p->g, p->out, p->dt_bias, p->initial_state, p->final_state};
  for (const void* x : ptrs)
    if (x && !aligned16(x)) return fail(FKDA_ERR_INVALID_ARGUMENT, "tensor base addresses must be 16-byte aligned");
  const int64_t T_total = p->B * p->T;
  if (p->H > 65535) return fail(FKDA_ERR_INVALID_ARGUMENT, "H must be at most 65535");
  if (p->N * p->H > 0x7fffffffLL) return fail(FKDA_ERR_INVALID_ARGUMENT, "N*H exceeds 2^31-1 chains");
  if (!make_layout(T_total, p->H, p->N, p->cu_seqlens ? 1 : 0, p->T, p->flags, L, fit ? p->workspace_bytes : kAnyRoom)) return fail(FKDA_ERR_INVALID_ARGUMENT, "bad sizes");
  if (L->chunks_per_head * p->H > 0x7fffffffLL) return fail(FKDA_ERR_INVALID_ARGUMENT, "too many (chunk, head) pairs for one call");
  // (a caller who can read the status word sized the workspace by fkda_get_workspace_size, which is held to)
  const int64_t needed = whole_call ? scratch_bytes(p, *L) : L->total_bytes;
  if (needed == 0) return FKDA_OK;
  if (!p->workspace) return fail(FKDA_ERR_INVALID_ARGUMENT, "workspace is NULL");
  if (reinterpret_cast<uintptr_t>(p->workspace) & 255u) return fail(FKDA_ERR_INVALID_ARGUMENT, "workspace must be 256-byte aligned");
  if (p->workspace_bytes < needed)
    return fail(FKDA_ERR_WORKSPACE_TOO_SMALL, "workspace has %lld bytes, %lld needed", (long long)p->workspace_bytes, (long long)needed);
  return FKDA_OK;
}

// The status word starts at zero.  (Varlen calls: the chunk-prefix kernel, which runs first and alone, clears it.)
cudaError_t clear_status(const fkda_fwd_params* p, cudaStream_t stream) {
  if (p->flags & FKDA_FLAG_STATUS_UNREAD) return cudaSuccess;
  return cudaMemsetAsync(p->workspace, 0, fkda::kWsHeaderBytes, stream);
}

fkda::PrepParams prep_params(const fkda_fwd_params* p, const Layout& L) {
  uint8_t* ws = static_cast<uint8_t*>(p->workspace);
  fkda::PrepParams q{};
  q.q = static_cast<const __nv_bfloat16*>(p->q);
  q.k = static_cast<const __nv_bfloat16*>(p->k);
  q.v = static_cast<const __nv_bfloat16*>(p->v);
  q.g = static_cast<const __nv_bfloat16*>(p->g);
  q.beta = static_cast<const __nv_bfloat16*>(p->beta);
  q.A_log = p->A_log;
  q.dt_bias = p->dt_bias;
  q.cu_seqlens = p->cu_seqlens;
  q.chunk_prefix = reinterpret_cast<const int*>(ws + L.prefix_off);
  q.records = ws + L.records_off;
  q.status = reinterpret_cast<int*>(ws);
  q.T = p->T;
  q.T_total = p->B * p->T;
  q.H = static_cast<int>(p->H);
  q.N = static_cast<int>(p->N);
  q.total_chunks = static_cast<int>(L.chunks_per_head);
  q.seq_chunks = q.slice_chunks = static_cast<int>((p->T + fkda::kChunk - 1) / fkda::kChunk);
  q.scale = p->scale;
  q.gate_scale = static_cast<float>(static_cast<double>(p->lower_bound) * 1.4426950408889634);
  return q;
}

int do_prepare(const fkda_fwd_params* p, const Layout& L, cudaStream_t stream, int wait_limit_us = 0, int first_load_only = 0) {
  uint8_t* ws = static_cast<uint8_t*>(p->workspace);
  int* status = reinterpret_cast<int*>(ws);
  int* prefix = reinterpret_cast<int*>(ws + L.prefix_off);
  cudaError_t e = p->cu_seqlens ? cudaSuccess : clear_status(p, stream);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync(status)");
  if (p->cu_seqlens) {
    e = fkda::launch_chunk_prefix(p->cu_seqlens, static_cast<int>(p->N), p->B * p->T, static_cast<int>(p->H), L.n_segs, false, prefix, status, stream);
    if (e != cudaSuccess) return cuda_fail(e, "chunk_prefix launch");
  }
  fkda::PrepParams q = prep_params(p, L);
  q.wait_limit_us = wait_limit_us;
  q.first_load_only = first_load_only;
#ifdef FKDA_TUNING
  {
    static const char* dbg_env = getenv("FKDA_PREPARE_SKIP");   // phase-skip timing of the prepare kernel (results are wrong when set)
    q.dbg = dbg_env ? atoi(dbg_env) : 0;
  }
#endif
  if (p->flags & FKDA_FLAG_PREPARE_MMA_SYNC) e = fkda::launch_prepare(q, stream);
  else if (p->flags & FKDA_FLAG_PREPARE_TCGEN05) e = fkda::launch_prepare_tc4(q, stream);
  else e = fkda::launch_prepare_pipe(q, stream);
  if (e != cudaSuccess) return cuda_fail(e, "prepare launch");
  return FKDA_OK;
}

fkda::ScanParams scan_params(const fkda_fwd_params* p, const Layout& L) {
  uint8_t* ws = static_cast<uint8_t*>(p->workspace);
  fkda::ScanParams s{};
  s.records = ws + L.records_off;
  s.cu_seqlens = p->cu_seqlens;
  s.chunk_prefix = reinterpret_cast<const int*>(ws + L.prefix_off);
  s.seq_order = p->cu_seqlens ? s.chunk_prefix + (p->N + 1) : nullptr;
  s.initial_state = p->initial_state;
  s.final_state = p->final_state;
  s.out = static_cast<__nv_bfloat16*>(p->out);
  s.status = reinterpret_cast<int*>(ws);
  s.T = p->T;
  s.T_total = p->B * p->T;
  s.H = static_cast<int>(p->H);
  s.N = static_cast<int>(p->N);
  s.total_chunks = static_cast<int>(L.chunks_per_head);
  s.state_fp32 = p->state_dtype == FKDA_STATE_FP32 ? 1 : 0;
  if (p->cu_seqlens && L.n_segs > 1) s.seg_chunks_dev = s.status + 2;     // set by the chunk-prefix kernel
  return s;
}

int do_scan(const fkda_fwd_params* p, const Layout& L, cudaStream_t stream) {
  uint8_t* ws = static_cast<uint8_t*>(p->workspace);
  fkda::ScanParams s = scan_params(p, L);
  const int sms = fkda::device_sm_count();
  cudaError_t e;
  if (p->flags & FKDA_FLAG_SCAN_SIMT) e = fkda::launch_scan_simt(s, stream);
  else if ((p->flags & (FKDA_FLAG_SCAN_PLAIN | FKDA_FLAG_SCAN_LOOKAHEAD)) && L.n_segs > 1) {
    // a forced run count together with a forced kernel: both passes on that kernel
    e = fkda::launch_scan_segmented(s, L.n_segs, L.seg_chunks, reinterpret_cast<float*>(ws + L.seg_off),
                                    (p->flags & FKDA_FLAG_SCAN_PLAIN) ? 1 : 2, nullptr, stream);
  } else if (p->flags & FKDA_FLAG_SCAN_PLAIN) e = fkda::launch_scan(s, stream);
  else if (!(p->flags & FKDA_FLAG_SCAN_LOOKAHEAD) && p->cu_seqlens == nullptr && p->T > 0 &&
             (p->T <= 2 * fkda::kChunk || (p->T <= 5 * fkda::kChunk && p->N * p->H > sms))) {
    // short chains: the state-I/O-oriented persistent kernel (up to two chunks always; up to five when there are more
    // chains than SMs, where it still beats the compact kernel: 0.122 against 0.150 ms at 2048 chains of three chunks,
    // 0.190 against 0.194 at six)
    e = fkda::launch_scan_short(s, sms, stream);
  } else if (!(p->flags & FKDA_FLAG_SCAN_LOOKAHEAD) && p->N * p->H > sms) {
    // More chains than SMs: the compact kernel, two CTAs per SM.  Equal-length chains: always.  Varlen: the
    // chunk-prefix kernel has decided on the device (status word 1); both kernels are launched and the CTAs of the
    // one that was not chosen leave at once.
    if (p->cu_seqlens == nullptr || p->N * p->H > 1024) {
      // (beyond about a thousand chains the empty launch would cost more than a wrong choice, and one long sequence
      // among so many chains rarely sets the duration)
      e = fkda::launch_scan(s, stream);
    } else {
      s.select = s.status + 1;
      s.select_want = 1;
      e = fkda::launch_scan(s, stream);
      s.select_want = 0;
      if (e == cudaSuccess) e = fkda::launch_scan2(s, stream);
    }
  } else if (L.n_segs > 1) {
    // few long chains: cut them into runs that are walked in parallel
    e = fkda::launch_scan_segmented(s, L.n_segs, L.seg_chunks, reinterpret_cast<float*>(ws + L.seg_off), 0, nullptr, stream);
  } else e = fkda::launch_scan2(s, stream);
  if (e != cudaSuccess) return cuda_fail(e, "scan launch");
  return FKDA_OK;
}

// Where fewer chains than SMs have a CTA each, the SMs beyond them can work out operands meanwhile.  The call is then cut in two
// time slices, and the second one's operands are computed beside the first one's recurrence, by kSliceWaves waves of two
// CTAs on each free SM that end with it.  The costs are those of the kernels at the time of the fit - 1.32 us for a chunk of the
// recurrence, 3.7 us per item and CTA of the token-parallel stage and 5 us to fill and drain its pipeline; both have become a fifth
// faster since, and the cut lies where it did: the best of seven was the planned one, or next to it, for 96, 110 and 120 chains of 256
// chunks, 75 x 512, 80 x 128 and 124 x 1024.  Returns the chunks of the first slice, or 0 where what the stage is shortened by is
// not worth it: the second pair of launches costs about 20 us, and the stage takes its share of the recurrence's bandwidth.
// Gains measured against one piece, chains x chunks: 75 x 512 14 %, 80 x 128 10 %, 96 x 256 10 %, 110 x 256 7 %, 120 x 256 5 to 9 %, 126 x
// 256 5 %, 124 x 1024 2 to 6 %, 128 x 512 -2 to 3 %; beyond the line 130 x 2048, 134 x 2048 and 140 x 2048 1 %, 144 x 1024 and 147 x 2048
// -1 to -5 %.  Equal lengths only: a packed batch's lengths, which the slices would have to follow, are on the
// device.  Chains split over CTAs leave too few SMs free beside them (20 at 32 chains, none at 37 or 74).
constexpr int kSliceWaves = 2;
int plan_slice(int64_t chains, int64_t chunks, int sms) {
  if (chains >= sms || chunks < 16) return 0;
  const double c = static_cast<double>(chunks), n = static_cast<double>(chains), per_us = 2.0 * kSliceWaves * (sms - n) / (3.7 * n);
  const double second = per_us * (1.32 / kSliceWaves * c - 5.0) / (1.0 + 1.32 / kSliceWaves * per_us);
  const double saved = second * 0.0118 * n, call = c * (0.0118 * n + 1.32);
  if (saved < 40.0 || saved < 0.05 * call) return 0;
  return static_cast<int>(c - second);
}

// What the test entry points ask of do_compact: one of its stages alone, and a wait that nothing completes.
struct TestAid {
  bool operands, recurrence;
  int wait_limit_us;       // 0: nothing is held back
  int stop_copies_after;   // records per CTA of the recurrence, or (negative) maps of the chaining of runs
};

// The forward pass over compact records (fkda_record.cuh): token-parallel stage, then the recurrence in the form that suits
// the number of chains.
int do_compact(const fkda_fwd_params* p, const Layout& L, cudaStream_t stream, const TestAid* aid = nullptr) {
  uint8_t* ws = static_cast<uint8_t*>(p->workspace);
  int* status = reinterpret_cast<int*>(ws);
  const int64_t chains = p->N * p->H, T_total = p->B * p->T;
  const int sms = fkda::device_sm_count();
  const int runs = L.n_segs, run_len = L.seg_chunks;
  cudaError_t e = cudaSuccess;
  if (p->cu_seqlens)
    e = fkda::launch_chunk_prefix(p->cu_seqlens, static_cast<int>(p->N), T_total, static_cast<int>(p->H), runs, true,
                                  reinterpret_cast<int*>(ws + L.prefix_off), status, stream);
  else e = clear_status(p, stream);
  if (e != cudaSuccess) return cuda_fail(e, "scheduling launch");
  // Fewer chains than a quarter or half of the SMs: a chain's time is what counts, it is split over four or two CTAs.
  // (FKDA_FLAG_SCAN_NO_SEGMENTS: one CTA walks the whole chain.)
  const bool whole = (p->flags & FKDA_FLAG_SCAN_NO_SEGMENTS) != 0, one_item = (p->flags & FKDA_FLAG_OPERANDS_PER_ITEM) != 0;
  const int rows = runs > 1 || whole ? 0 : chains * 4 <= sms ? 32 : chains * 2 <= sms ? 64 : 0;
  fkda::PrepParams q = prep_params(p, L);
  const bool one_stage = aid != nullptr && !(aid->operands && aid->recurrence);
  const int slice = p->cu_seqlens || runs > 1 || rows || whole || one_item || one_stage ? 0 : plan_slice(chains, q.seq_chunks, sms);
  if (slice) q.slice_chunks = slice;
  if (aid != nullptr && !aid->recurrence) {
    q.wait_limit_us = aid->wait_limit_us;
    q.first_load_only = aid->wait_limit_us > 0;
  }
  if (aid == nullptr || aid->operands) e = fkda::launch_operands(q, one_item, stream);
  if (e != cudaSuccess) return cuda_fail(e, "token-parallel launch");
  if (aid != nullptr && !aid->recurrence) return FKDA_OK;
  fkda::ScanParams s = scan_params(p, L);
  const __nv_bfloat16* v = static_cast<const __nv_bfloat16*>(p->v);
  if (aid != nullptr) {
    (aid->stop_copies_after < 0 ? s.map_wait_limit_us : s.wait_limit_us) = aid->wait_limit_us;
    s.stop_copies_after = aid->stop_copies_after > 0 ? aid->stop_copies_after : 0;
    s.stop_maps_after = aid->stop_copies_after < 0 ? -aid->stop_copies_after : 0;
  }
  s.skip_short = p->cu_seqlens != nullptr;
  s.release_next = p->cu_seqlens != nullptr && runs == 1;      // (to the step kernel below)
  if (runs > 1) {
    e = fkda::launch_scan_segmented(s, runs, run_len, reinterpret_cast<float*>(ws + L.seg_off), 0, v, stream);
  } else {
    s.seg_chunks_dev = nullptr;
    s.next_walk = p->cu_seqlens ? status + 3 : nullptr;
    if (rows) {
      e = fkda::launch_recur_split(s, v, rows, stream);
    } else if (slice) {
      s.slice_end = slice;
      s.release_next = 1;
      e = fkda::launch_recur(s, v, stream);
      if (e != cudaSuccess) return cuda_fail(e, "recurrence launch");
      q.slice_begin = slice;
      q.slice_chunks = q.seq_chunks - slice;
      q.beside = 2 * kSliceWaves * (sms - static_cast<int>(chains));
      e = fkda::launch_operands(q, false, stream);
      if (e != cudaSuccess) return cuda_fail(e, "token-parallel launch");
      s.slice_begin = slice;
      s.slice_end = q.seq_chunks;
      s.release_next = 0;
      e = fkda::launch_recur(s, v, stream);
    } else {
      e = fkda::launch_recur(s, v, stream);
    }
  }
  if (e != cudaSuccess) return cuda_fail(e, "recurrence launch");
  // The sequences of a few tokens, decode steps among the prompts: a padded chunk each would cost several times their own work.
  if (p->cu_seqlens) e = fkda::launch_step(prep_params(p, L), s, stream);
  if (e != cudaSuccess) return cuda_fail(e, "step kernel launch");
  return FKDA_OK;
}

int do_fwd(const fkda_fwd_params* p, void* cuda_stream, bool fit) {
  Layout L;
  int rc = validate(p, &L, true, fit);
  if (rc != FKDA_OK) return rc;
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  if (p->flags & FKDA_FLAG_REFERENCE_ROUNDING) {
    // debugging aid: the reference's tile size, state type and rounding points (one kernel, any shape)
    cudaError_t e = cudaMemsetAsync(p->workspace, 0, fkda::kWsHeaderBytes, stream);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync(status)");
    e = fkda::launch_refmode(static_cast<const __nv_bfloat16*>(p->q), static_cast<const __nv_bfloat16*>(p->k),
                             static_cast<const __nv_bfloat16*>(p->v), static_cast<const __nv_bfloat16*>(p->g),
                             static_cast<const __nv_bfloat16*>(p->beta), p->A_log, p->dt_bias, p->initial_state, p->final_state,
                             static_cast<__nv_bfloat16*>(p->out), p->cu_seqlens, p->N, p->T, p->B * p->T, static_cast<int>(p->H),
                             p->state_dtype == FKDA_STATE_FP32 ? 1 : 0, p->scale,
                             static_cast<float>(static_cast<double>(p->lower_bound) * 1.4426950408889634), stream);
    if (e != cudaSuccess) return cuda_fail(e, "reference-rounding kernel launch");
    return FKDA_OK;
  }
  if (fused_short(p)) {
    // short fixed-length sequences (a continuation step): one fused kernel, no operand records
    cudaError_t e = clear_status(p, stream);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync(status)");
    if (takes_step_kernel(p)) {
      e = fkda::launch_step(prep_params(p, L), scan_params(p, L), stream);
      if (e != cudaSuccess) return cuda_fail(e, "step kernel launch");
      return FKDA_OK;
    }
    e = fkda::launch_short16(static_cast<const __nv_bfloat16*>(p->q), static_cast<const __nv_bfloat16*>(p->k),
                             static_cast<const __nv_bfloat16*>(p->v), static_cast<const __nv_bfloat16*>(p->g),
                             static_cast<const __nv_bfloat16*>(p->beta), p->A_log, p->dt_bias, p->initial_state, p->final_state,
                             static_cast<__nv_bfloat16*>(p->out), p->N, static_cast<int>(p->T), static_cast<int>(p->H),
                             p->state_dtype == FKDA_STATE_FP32 ? 1 : 0, p->scale,
                             static_cast<float>(static_cast<double>(p->lower_bound) * 1.4426950408889634),
                             static_cast<int*>(p->workspace), stream);
    if (e != cudaSuccess) return cuda_fail(e, "short-sequence kernel launch");
    return FKDA_OK;
  }
  // No kernel of the two-stage form is asked for: compact records.  (Packed batches with FKDA_FLAG_SCAN_NO_SEGMENTS take the
  // two-stage form: the whole walk on kernels that share nothing with the runs it is compared against.)
  const bool cross_check = p->cu_seqlens != nullptr && (p->flags & FKDA_FLAG_SCAN_NO_SEGMENTS);
  if (p->B * p->T > 0 && !cross_check && (p->flags & ~static_cast<uint32_t>(FKDA_FLAG_STATUS_UNREAD | FKDA_FLAG_SCAN_NO_SEGMENTS | FKDA_FLAG_NO_FUSED_SHORT |
                                                            FKDA_FLAG_OPERANDS_PER_ITEM)) == 0)
    return do_compact(p, L, stream);
  rc = do_prepare(p, L, stream);
  if (rc != FKDA_OK) return rc;
  return do_scan(p, L, stream);
}

}  // namespace

namespace fkda {
int fwd_within(const fkda_fwd_params* p, void* cuda_stream) { return do_fwd(p, cuda_stream, true); }
}  // namespace fkda

extern "C" {

int fkda_get_workspace_size_flags(int64_t T_total, int64_t H, int64_t N, int64_t flags, int64_t* bytes) {
  Layout L;
  if (!bytes) return fail(FKDA_ERR_INVALID_ARGUMENT, "bytes is NULL");
  if (!make_layout(T_total, H, N, -1, 0, flags, &L)) return fail(FKDA_ERR_INVALID_ARGUMENT, "T_total >= 0, H > 0 and N > 0 required");
  *bytes = L.total_bytes;
  return FKDA_OK;
}

int fkda_get_workspace_size(int64_t T_total, int64_t H, int64_t N, int64_t* bytes) {
  return fkda_get_workspace_size_flags(T_total, H, N, 0, bytes);
}

int fkda_plan_segments(int64_t chains, int64_t chunks_per_sequence, int* segments, int* chunks_per_segment) {
  if (!segments || !chunks_per_segment) return fail(FKDA_ERR_INVALID_ARGUMENT, "NULL pointer");
  *segments = plan_runs(chains, chunks_per_sequence, kAnyRoom, fkda::device_sm_count(), chunks_per_segment);
  return FKDA_OK;
}

int fkda_workspace_layout(int64_t T_total, int64_t H, int64_t N, int varlen, int64_t T_per_seq, int64_t* records_offset,
                          int64_t* record_bytes, int64_t* chunks_per_head) {
  Layout L;
  if (!make_layout(T_total, H, N, varlen ? 1 : 0, T_per_seq, 0, &L)) return fail(FKDA_ERR_INVALID_ARGUMENT, "bad sizes");
  if (records_offset) *records_offset = L.records_off;
  if (record_bytes) *record_bytes = fkda::kRecBytes;
  if (chunks_per_head) *chunks_per_head = L.chunks_per_head;
  return FKDA_OK;
}

int fkda_workspace_bytes_exact(int64_t T_total, int64_t H, int64_t N, int varlen, int64_t T_per_seq, int64_t flags, int64_t* bytes) {
  Layout L;
  if (!bytes) return fail(FKDA_ERR_INVALID_ARGUMENT, "bytes is NULL");
  if (!make_layout(T_total, H, N, varlen ? 1 : 0, T_per_seq, flags, &L)) return fail(FKDA_ERR_INVALID_ARGUMENT, "bad sizes");
  *bytes = L.total_bytes;
  return FKDA_OK;
}

int fkda_fwd_scratch_bytes(const fkda_fwd_params* p, int64_t* bytes) {
  Layout L;
  if (!p || !bytes) return fail(FKDA_ERR_INVALID_ARGUMENT, "NULL pointer");
  if (!make_layout(p->B * p->T, p->H, p->N, p->cu_seqlens ? 1 : 0, p->T, p->flags, &L)) return fail(FKDA_ERR_INVALID_ARGUMENT, "bad sizes");
  *bytes = scratch_bytes(p, L);
  return FKDA_OK;
}

int fkda_prepare(const fkda_fwd_params* p, void* cuda_stream) {
  Layout L;
  int rc = validate(p, &L);
  if (rc != FKDA_OK) return rc;
  return do_prepare(p, L, static_cast<cudaStream_t>(cuda_stream));
}

int fkda_scan(const fkda_fwd_params* p, void* cuda_stream) {
  Layout L;
  int rc = validate(p, &L);
  if (rc != FKDA_OK) return rc;
  return do_scan(p, L, static_cast<cudaStream_t>(cuda_stream));
}

int fkda_fwd(const fkda_fwd_params* p, void* cuda_stream) { return do_fwd(p, cuda_stream, false); }

int fkda_prologue(const void* q, const void* k, const void* g, const void* beta, const float* A_log, const float* dt_bias,
                  float lower_bound, int64_t T_total, int64_t H, void* qn, void* kn, float* gate, float* beta_act,
                  void* cuda_stream) {
  if (!q || !k || !g || !beta || !A_log || !dt_bias || !qn || !kn || !gate || !beta_act)
    return fail(FKDA_ERR_INVALID_ARGUMENT, "NULL pointer");
  if (T_total < 0 || H <= 0 || H > 0x7fffffffLL) return fail(FKDA_ERR_INVALID_ARGUMENT, "bad sizes");
  cudaError_t e = fkda::launch_prologue(
      static_cast<const __nv_bfloat16*>(q), static_cast<const __nv_bfloat16*>(k), static_cast<const __nv_bfloat16*>(g),
      static_cast<const __nv_bfloat16*>(beta), A_log, dt_bias, static_cast<float>(static_cast<double>(lower_bound) * 1.4426950408889634),
      T_total * H, static_cast<int>(H), static_cast<__nv_bfloat16*>(qn), static_cast<__nv_bfloat16*>(kn), gate, beta_act,
      static_cast<cudaStream_t>(cuda_stream));
  if (e != cudaSuccess) return cuda_fail(e, "prologue launch");
  return FKDA_OK;
}

int fkda_read_status(const void* workspace, void* cuda_stream, int* status) {
  if (!workspace || !status) return fail(FKDA_ERR_INVALID_ARGUMENT, "NULL pointer");
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  cudaError_t e = cudaMemcpyAsync(status, workspace, sizeof(int), cudaMemcpyDeviceToHost, stream);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyAsync(status)");
  e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return cuda_fail(e, "cudaStreamSynchronize");
  if (*status != 0) return fail(FKDA_ERR_DEVICE_STATUS, "device status %d (%s)", *status,
                                *status == 1 ? "cu_seqlens not monotone inside [0, T_total]" : "a bounded wait inside a kernel gave up");
  return FKDA_OK;
}

int fkda_selftest_umma(const void* A, const void* B, float* D, int mode, int reps, int* status, void* cuda_stream) {
  if (!A || !B || !D || !status || mode < 0 || mode > 4 || reps < 1) return fail(FKDA_ERR_INVALID_ARGUMENT, "bad arguments");
  cudaError_t e = fkda::launch_umma_selftest(static_cast<const __nv_bfloat16*>(A), static_cast<const __nv_bfloat16*>(B), D, mode,
                                             reps, status, static_cast<cudaStream_t>(cuda_stream));
  if (e != cudaSuccess) return cuda_fail(e, "selftest launch");
  return FKDA_OK;
}

int fkda_debug_plan_slice(int64_t chains, int64_t chunks_per_sequence) {
  return chains > 0 ? plan_slice(chains, chunks_per_sequence, fkda::device_sm_count()) : 0;
}

int fkda_debug_scan_giveup(const fkda_fwd_params* p, int stop_copies_after, int wait_limit_us, void* cuda_stream) {
  Layout L;
  int rc = validate(p, &L);
  if (rc != FKDA_OK) return rc;
  if (stop_copies_after < 1 || wait_limit_us < 1 || wait_limit_us > 1000000)
    return fail(FKDA_ERR_INVALID_ARGUMENT, "stop_copies_after >= 1 and 1 <= wait_limit_us <= 1000000 required");
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  rc = do_prepare(p, L, stream);
  if (rc != FKDA_OK) return rc;
  fkda::ScanParams s = scan_params(p, L);
  s.seg_chunks_dev = nullptr;          // whole sequences on the look-ahead kernel
  s.wait_limit_us = wait_limit_us;
  s.stop_copies_after = stop_copies_after;
  cudaError_t e = fkda::launch_scan2(s, stream);
  if (e != cudaSuccess) return cuda_fail(e, "scan launch");
  return FKDA_OK;
}

int fkda_debug_prepare_giveup(const fkda_fwd_params* p, int wait_limit_us, void* cuda_stream) {
  Layout L;
  int rc = validate(p, &L);
  if (rc != FKDA_OK) return rc;
  if (wait_limit_us < 1 || wait_limit_us > 1000000) return fail(FKDA_ERR_INVALID_ARGUMENT, "1 <= wait_limit_us <= 1000000 required");
  if (p->flags & (FKDA_FLAG_PREPARE_TCGEN05 | FKDA_FLAG_PREPARE_MMA_SYNC))
    return fail(FKDA_ERR_INVALID_ARGUMENT, "the give-up aid drives the pipelined kernel: no kernel-selection flag");
  return do_prepare(p, L, static_cast<cudaStream_t>(cuda_stream), wait_limit_us, 1);
}

int fkda_debug_operands(const fkda_fwd_params* p, int wait_limit_us, void* cuda_stream) {
  Layout L;
  int rc = validate(p, &L);
  if (rc != FKDA_OK) return rc;
  if (wait_limit_us < 0 || wait_limit_us > 1000000) return fail(FKDA_ERR_INVALID_ARGUMENT, "0 <= wait_limit_us <= 1000000 required");
  const TestAid aid{true, false, wait_limit_us, 0};
  return do_compact(p, L, static_cast<cudaStream_t>(cuda_stream), &aid);
}

int fkda_debug_recurrence(const fkda_fwd_params* p, void* cuda_stream) {
  Layout L;
  int rc = validate(p, &L);
  if (rc != FKDA_OK) return rc;
  const TestAid aid{false, true, 0, 0};
  return do_compact(p, L, static_cast<cudaStream_t>(cuda_stream), &aid);
}

int fkda_debug_recurrence_giveup(const fkda_fwd_params* p, int stop_copies_after, int wait_limit_us, void* cuda_stream) {
  Layout L;
  int rc = validate(p, &L);
  if (rc != FKDA_OK) return rc;
  if (stop_copies_after == 0 || wait_limit_us < 1 || wait_limit_us > 1000000)
    return fail(FKDA_ERR_INVALID_ARGUMENT, "stop_copies_after != 0 and 1 <= wait_limit_us <= 1000000 required");
  const TestAid aid{true, true, wait_limit_us, stop_copies_after};
  return do_compact(p, L, static_cast<cudaStream_t>(cuda_stream), &aid);
}

#ifdef FKDA_TUNING
int fkda_debug_tmem_bench(int nwarps, int reps, void* out, void* cuda_stream) {
  if (nwarps < 1 || nwarps > 16 || reps < 1 || !out) return fail(FKDA_ERR_INVALID_ARGUMENT, "bad arguments");
  cudaError_t e = fkda::launch_tmem_bench(nwarps, reps, static_cast<long long*>(out), static_cast<cudaStream_t>(cuda_stream));
  if (e != cudaSuccess) return cuda_fail(e, "tmem bench launch");
  return FKDA_OK;
}

int fkda_debug_umma_bench(int issuers, int reps, int ksteps, int n, int a_in_tmem, void* out, int* status, void* cuda_stream) {
  if (issuers < 1 || issuers > 4 || reps < 1 || reps > 4096 || ksteps < 1 || ksteps > 8 || (n != 32 && n != 64 && n != 128) || !out || !status)
    return fail(FKDA_ERR_INVALID_ARGUMENT, "bad arguments");
  cudaError_t e = fkda::launch_umma_bench(issuers, reps, ksteps, n, a_in_tmem ? 1 : 0, static_cast<long long*>(out), status,
                                          static_cast<cudaStream_t>(cuda_stream));
  if (e != cudaSuccess) return cuda_fail(e, "umma bench launch");
  return FKDA_OK;
}

#endif  // FKDA_TUNING

int fkda_debug_tmem_layout_probe(void* out, void* cuda_stream) {
  if (!out) return fail(FKDA_ERR_INVALID_ARGUMENT, "out is NULL");
  cudaError_t e = fkda::launch_tmem_layout_probe(static_cast<uint32_t*>(out), static_cast<cudaStream_t>(cuda_stream));
  if (e != cudaSuccess) return cuda_fail(e, "tmem layout probe launch");
  return FKDA_OK;
}

#ifdef FKDA_TUNING
int fkda_debug_set_prepare_trace(void* device_buffer) {
  fkda::set_prepare_trace(static_cast<long long*>(device_buffer));
  return FKDA_OK;
}

int fkda_debug_set_scan_trace(void* device_buffer) {
  fkda::set_scan_trace(static_cast<unsigned long long*>(device_buffer));
  return FKDA_OK;
}
#endif

const char* fkda_last_error(void) { return g_err; }

const char* fkda_version(void) { return "fkda 0.1 (sm_100a)"; }

}  // extern "C"
