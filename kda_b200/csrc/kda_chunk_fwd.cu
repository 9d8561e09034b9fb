// Chunked KDA forward for sm_100a: chunk tables, per-chunk preparation, and the state scan.
//
//  kda_chunk_tables_kernel   cu_seqlens -> (first chunk of each sequence, sequence of each chunk); device only,
//                            so that variable-length calls need no device->host copy.
//  kda_chunk_prepare_kernel  (kda_chunk_prepare.cu) one CTA per (chunk, head): everything that does not depend on the state:
//                            G = cumsum(g), Aqk, Akk, Tm = (I+Akk)^-1, w, u, qg, kg  -> tiles in the workspace.
//  kda_chunk_scan_kernel     (kda_chunk_scan.cu; many units: kda_chunk_scan_tc.cu) walks the chunks of a (sequence, head) in order with
//                            the fp32 state in registers or tensor memory.
//                            v_new = u - w h;  o = qg h + Aqk v_new;  h = Diag(Gam_last) h + kg^T v_new.
#include <mutex>

#include "kda_chunk.cuh"
#include "kda_device.cuh"
#include "kda_prepare.cuh"
#include "kda_scan.cuh"

namespace kda {

// =================================================================================================
// chunk tables
// =================================================================================================
// A cu_seqlens that does not describe `tokens` tokens (a negative first entry, a negative length, more tokens than the
// tensors hold, or more chunks than the workspace was sized for) would send every later kernel past the end of the
// workspace.  The tables kernel checks it on the device: it then sets KDA_STATUS_BAD_CU_SEQLENS in the status word
// and writes empty tables (zero chunks for every sequence), so that prepare, the scans and the backward kernels do
// nothing; no device->host synchronisation is needed for the check.
__global__ void __launch_bounds__(1024) kda_chunk_tables_kernel(const int* __restrict__ cu, int N, long long tokens, int max_chunks,
                                                                int* __restrict__ seq_chunk_off, int* __restrict__ chunk_seq,
                                                                int* __restrict__ seq_order, unsigned* __restrict__ status) {
  chain_point();
  __shared__ int warp_sum_[32];
  __shared__ int offs[1025];      // chunk offsets of the first 1,024 sequences (all of them in ordinary calls)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int per = (N + 1023) / 1024;
  const int n0 = min(N, tid * per), n1 = min(N, n0 + per);
  // a partial sum that would overflow is certainly beyond max_chunks: sums saturate there instead of wrapping
  const int cap = max_chunks + 1;
  int sum = 0;
  bool bad = (tid == 0) && (cu[0] < 0 || static_cast<long long>(cu[N]) > tokens);
  for (int n = n0; n < n1; ++n) {
    const int len = cu[n + 1] - cu[n];
    bad |= len < 0;
    const int nc = (len > 0) ? (len + C - 1) / C : 0;
    sum = min(cap, sum + min(cap, nc));
  }
  int incl = sum;                 // inclusive scan over the block: within the warp, then over the warps' totals
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl = min(cap, incl + x);
  }
  if (lane == 31) warp_sum_[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int x = warp_sum_[lane];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, off);
      if (lane >= off) x = min(cap, x + y);
    }
    warp_sum_[lane] = x;
  }
  __syncthreads();
  if (warp > 0) incl = min(cap, incl + warp_sum_[warp - 1]);
  const int total = warp_sum_[31];
  bad |= total > max_chunks;
  bad = __syncthreads_or(bad) != 0;
  if (tid < 4) status[tid] = (tid == 0 && bad) ? KDA_STATUS_BAD_CU_SEQLENS : 0u;
  if (bad) {
    for (int n = n0; n < n1; ++n) {
      seq_chunk_off[n] = 0;
      seq_order[n] = n;
    }
    if (tid == 1023) seq_chunk_off[N] = 0;
    return;
  }
  int run = incl - sum;           // exclusive prefix
  for (int n = n0; n < n1; ++n) {
    const int len = cu[n + 1] - cu[n];
    seq_chunk_off[n] = run;
    if (n < 1024) offs[n] = run;
    run += (len > 0) ? (len + C - 1) / C : 0;
  }
  if (tid == 1023) seq_chunk_off[N] = total;
  if (tid == 0 && N <= 1024) offs[N] = total;
  __syncthreads();
  // sequence of every chunk: a thread per chunk, binary search over the offsets (a thread per SEQUENCE would write a long
  // prompt's whole range alone: 512 chunks took 5.8 us)
  const int* table = N <= 1024 ? offs : seq_chunk_off;
  for (int c = tid; c < total; c += 1024) {
    int lo = 0, hi = N;           // the last n with offset <= c
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (table[mid] <= c) lo = mid; else hi = mid;
    }
    chunk_seq[c] = lo;
  }
  // Longest first for the state scans, whose CTAs each walk one sequence: with more (sequence, head) units than SMs a long
  // sequence that starts last would run on alone.  Rank by counting; beyond 1,024 sequences the tail is short anyway.
  if (N > 1024) {
    for (int n = n0; n < n1; ++n) seq_order[n] = n;
  } else if (tid < N) {
    const int mine = offs[tid + 1] - offs[tid];
    int rank = 0;
    for (int n = 0; n < N; ++n) {
      const int other = offs[n + 1] - offs[n];
      rank += (other > mine || (other == mine && n < tid)) ? 1 : 0;
    }
    seq_order[rank] = tid;
  }
}

int validate_chunk_args(const kda_chunk_args& a, bool backward);
int validate_chunk_args(const kda_chunk_args& a, bool backward) {
  if (a.tokens < 0 || a.N < 0 || a.H <= 0) return KDA_E_SHAPE;
  if (a.HQ < 0 || (a.HQ > 0 && (a.HQ > a.H || a.H % a.HQ != 0))) return KDA_E_SHAPE;
  if (a.K != KD || a.V != VD) return KDA_E_SHAPE;
  if (a.k_cols < 0 || a.k_cols > KD || a.k_cols % 8 || a.v_cols < 0 || a.v_cols > VD || a.v_cols % 8) return KDA_E_SHAPE;
  if (a.scan_slices != 0 && a.scan_slices != 1 && a.scan_slices != 4) return KDA_E_SHAPE;
  if (a.io_dtype != KDA_BF16) return KDA_E_DTYPE;      // float32: the token-recurrent entry points
  if (a.tokens / C + a.N > 0x3fffffffLL) return KDA_E_SHAPE;
  if (a.tokens == 0 || a.N == 0) return KDA_OK;
  const bool raw_g = !backward && a.g_raw, raw_b = !backward && a.beta_raw;
  if (!a.q || !a.k || !a.v || (!a.g && !raw_g) || (!a.beta && !raw_b) || !a.workspace) return KDA_E_NULL;
  if (raw_g && !a.A_log) return KDA_E_NULL;
  if ((raw_g && a.g_raw_dtype != KDA_BF16 && a.g_raw_dtype != KDA_FP32) || (raw_b && a.beta_raw_dtype != KDA_BF16 && a.beta_raw_dtype != KDA_FP32))
    return KDA_E_DTYPE;
  if (!a.cu_seqlens && a.tokens % a.N != 0) return KDA_E_SHAPE;
  if (!backward && !a.o) return KDA_E_NULL;
  uintptr_t bits = reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k) | reinterpret_cast<uintptr_t>(a.v) |
                   reinterpret_cast<uintptr_t>(a.g) | reinterpret_cast<uintptr_t>(a.o) | reinterpret_cast<uintptr_t>(a.h0) |
                   reinterpret_cast<uintptr_t>(a.ht) | reinterpret_cast<uintptr_t>(a.g_raw) | reinterpret_cast<uintptr_t>(a.dt_bias);
  if (backward) {
    if (!a.d_o || !a.dq || !a.dk || !a.dv || !a.dg || !a.dbeta || !a.bwd_workspace) return KDA_E_NULL;
    bits |= reinterpret_cast<uintptr_t>(a.d_o) | reinterpret_cast<uintptr_t>(a.dq) | reinterpret_cast<uintptr_t>(a.dk) |
            reinterpret_cast<uintptr_t>(a.dv) | reinterpret_cast<uintptr_t>(a.dg) | reinterpret_cast<uintptr_t>(a.d_ht) |
            reinterpret_cast<uintptr_t>(a.dh0) | (reinterpret_cast<uintptr_t>(a.bwd_workspace) & 255u);
  }
  if (bits & 15u) return KDA_E_ALIGN;
  if (reinterpret_cast<uintptr_t>(a.workspace) & 255u) return KDA_E_ALIGN;
  return KDA_OK;
}

static void launch_tables(const kda_chunk_args& a, int max_chunks, int* off, int* seq, int* order, unsigned* status, cudaStream_t st) {
  kda_chunk_tables_kernel<<<1, 1024, 0, st>>>(a.cu_seqlens, a.N, a.tokens, max_chunks, off, seq, order, status);
}

}  // namespace kda

extern "C" int64_t kda_chunk_max_chunks(int64_t tokens, int32_t N) { return tokens / kda::C + N; }

extern "C" size_t kda_chunk_workspace_bytes(int64_t tokens, int32_t N, int32_t H, int32_t K, int32_t V, int32_t save) {
  (void)K; (void)V;
  return kda::carve_ws(nullptr, nullptr, tokens, N, H, (save & 1) != 0, true, false, (save & 2) != 0).fwd_bytes;
}

extern "C" int kda_chunk_fwd(const kda_chunk_args* args, void* stream) {
  using namespace kda;
  if (!args) return KDA_E_NULL;
  const kda_chunk_args& a = *args;
  int rc = validate_chunk_args(a, false);
  if (rc != KDA_OK) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (a.N == 0) return KDA_OK;
  const int kc = a.k_cols > 0 ? a.k_cols : KD, vc = a.v_cols > 0 ? a.v_cols : VD;
  if (a.tokens == 0) {
    if (a.ht && a.ht != a.h0) {
      const size_t bytes = static_cast<size_t>(a.N) * a.H * kc * vc * sizeof(float);
      return static_cast<int>(a.h0 ? cudaMemcpyAsync(a.ht, a.h0, bytes, cudaMemcpyDeviceToDevice, st)
                                   : cudaMemsetAsync(a.ht, 0, bytes, st));
    }
    return KDA_OK;
  }
  const bool save = (a.save_for_backward & 1) != 0;
  const bool keep_qn = save && (a.save_for_backward & 2) != 0 && a.use_qk_l2norm != 0;
  ChunkWs w = carve_ws(static_cast<unsigned char*>(a.workspace), nullptr, a.tokens, a.N, a.H, save, true, false,
                       (a.save_for_backward & 2) != 0);
  if (a.workspace_bytes < w.fwd_bytes) return KDA_E_WORKSPACE;
  cudaError_t e = cudaSuccess;
  const int NTmax = static_cast<int>(a.tokens / C + a.N);

  ProfCall* prof = prof_begin(st);
  const ChunkMap map = chunk_map(w, a.cu_seqlens, a.tokens, a.N);
  if (a.cu_seqlens) {
    launch_tables(a, NTmax, w.seq_chunk_off, w.chunk_seq, w.seq_order, w.status, st);
    if ((e = cudaGetLastError()) != cudaSuccess) return static_cast<int>(e);
  }
  prof_mark(prof, KDA_STAGE_TABLES, st);

  PrepParams pp{};
  pp.q = static_cast<const __nv_bfloat16*>(a.q);
  pp.k = static_cast<const __nv_bfloat16*>(a.k);
  pp.v = static_cast<const __nv_bfloat16*>(a.v);
  pp.g = a.g; pp.beta = a.beta; pp.map = map;
  pp.g_raw = a.g_raw; pp.beta_raw = a.beta_raw; pp.A_log = a.A_log; pp.dt_bias = a.dt_bias;
  pp.g_out = a.g_raw ? const_cast<float*>(a.g) : nullptr; pp.beta_out = a.beta_raw ? const_cast<float*>(a.beta) : nullptr;
  pp.g_fp32 = a.g_raw_dtype == KDA_FP32; pp.beta_fp32 = a.beta_raw_dtype == KDA_FP32; pp.use_lb = a.use_lower_bound; pp.lb = a.lower_bound;
  pp.status = w.status; pp.clear_status = a.cu_seqlens == nullptr;
  pp.W = w.W; pp.UT = w.UT; pp.KG = w.KG; pp.QG = w.QG; pp.AQK = w.AQK; pp.GL = w.GL; pp.TI = save ? w.TI : nullptr; pp.RKK = save ? w.RKK : nullptr;
  pp.dbg = g_dbg_clocks; pp.H = a.H; pp.kc = kc; pp.vc = vc; pp.use_l2norm = a.use_qk_l2norm; pp.scale = a.scale;
  pp.HQ = a.HQ > 0 ? a.HQ : a.H; pp.grp = a.H / pp.HQ;
  pp.QN = keep_qn ? w.QN : nullptr; pp.KN = keep_qn ? w.KN : nullptr; pp.RSTD = keep_qn ? w.RSTD : nullptr;
  pp.qrows = static_cast<long long>(a.tokens) * pp.HQ;
  const long long chunks = map.T > 0 ? static_cast<long long>(a.N) * map.per_seq : NTmax;
  if ((rc = launch_prepare(pp, chunks * a.H, a.tokens, keep_qn, a.safe_gate != 0, st)) != KDA_OK) return rc;
  prof_mark(prof, KDA_STAGE_PREPARE, st);

  ScanParams sp{};
  sp.map = map;
  sp.W = w.W; sp.UT = w.UT; sp.KG = w.KG; sp.QG = w.QG; sp.AQK = w.AQK; sp.GL = w.GL;
  sp.HS = save ? w.HS : nullptr; sp.VNEWT = save ? w.VNEWT : nullptr;
  sp.h0 = a.h0; sp.ht = a.ht; sp.o = static_cast<__nv_bfloat16*>(a.o); sp.status = w.status; sp.dbg = g_dbg_clocks;
  sp.H = a.H; sp.kc = kc; sp.vc = vc;
  if ((rc = launch_scan(sp, a.N * a.H, a.scan_slices, st)) != KDA_OK) return rc;
  prof_mark(prof, KDA_STAGE_SCAN, st);
  return KDA_OK;
}

// =================================================================================================
// forward without any allocation: the workspace is a fixed array inside the library's device image
// =================================================================================================
// The name below is a device symbol.  In host code it is only a handle: its device address has to be
// asked for with cudaGetSymbolAddress, once per device, with that device current.
static __device__ __align__(256) unsigned char g_noalloc_scratch[KDA_NOALLOC_SCRATCH_BYTES];

namespace {
constexpr int kMaxDevices = kda::kMaxDeviceOrdinals;
std::mutex g_noalloc_mu;
unsigned char* g_noalloc_addr[kMaxDevices] = {};   // device address of g_noalloc_scratch, per device ordinal
}  // namespace

// Forward-only variant of kda_chunk_fwd for callers that cannot allocate device memory (a server whose
// memory pool is frozen after start-up, a thread inside a no-allocation region, a C caller without an
// allocator).  Inputs and outputs are the caller's; the per-chunk tiles live in g_noalloc_scratch.
// The first call on a device resolves the array's address (do it at start-up, before stream capture).
// Calls that overlap on one GPU share the array and race; the array keeps the previous call's bytes,
// which is harmless because every call rewrites all it reads.
extern "C" int kda_chunk_fwd_noalloc(const kda_chunk_args* args, void* stream) {
  if (!args) return KDA_E_NULL;
  if (args->save_for_backward != 0) return KDA_E_SHAPE;
  if (args->tokens < 0 || args->N < 0 || args->H <= 0) return KDA_E_SHAPE;
  const size_t need = kda::carve_ws(nullptr, nullptr, args->tokens, args->N, args->H, false).fwd_bytes;
  if (need > static_cast<size_t>(KDA_NOALLOC_SCRATCH_BYTES)) return KDA_E_LIMIT;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (dev < 0 || dev >= kMaxDevices) return KDA_E_LIMIT;
  unsigned char* scratch = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_addr[dev]) {
      void* p = nullptr;
      e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
      if (e != cudaSuccess) return static_cast<int>(e);
      g_noalloc_addr[dev] = static_cast<unsigned char*>(p);
    }
    scratch = g_noalloc_addr[dev];
  }
  kda_chunk_args a = *args;
  a.workspace = scratch;
  a.workspace_bytes = KDA_NOALLOC_SCRATCH_BYTES;
  a.bwd_workspace = nullptr;
  a.bwd_workspace_bytes = 0;
  return kda_chunk_fwd(&a, stream);
}

// Status word of the chunked kernels (see the header): copies it to the host, which waits for the device.
extern "C" int kda_chunk_status(const void* workspace, uint32_t* host_out) {
  if (!host_out) return KDA_E_NULL;
  *host_out = 0;
  const unsigned char* base = static_cast<const unsigned char*>(workspace);
  if (!base) {      // the array kda_chunk_fwd_noalloc uses on the current device; never used there: nothing to report
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev < 0 || dev >= kMaxDevices) return KDA_E_LIMIT;
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    base = g_noalloc_addr[dev];
    if (!base) return KDA_OK;
  }
  const kda::ChunkWs w = kda::carve_ws(const_cast<unsigned char*>(base), nullptr, 0, 0, 1, false);
  unsigned v = 0;
  const cudaError_t e = cudaMemcpy(&v, w.status, sizeof(v), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return static_cast<int>(e);
  *host_out = v;
  return KDA_OK;
}
