// Decode step of KDA for large batches, one or (with a state slot per token) several tokens per sequence: the [K x V] fp32 state of
// one (sequence, head) is 64 KiB that has to be read once and written once per token -- nothing else matters for speed.
// A unit is HV value columns of a state (the recurrence is independent per value column), moved by the bulk-copy engine through three
// shared-memory buffers per CTA.  HV / 16 warps keep the unit's state in registers and update it; one more issues every copy and
// waits for slot numbers, so that the loads of the next unit and the stores of the last tokens are in flight beside the arithmetic.
// HV = 64, two persistent CTAs per SM, for several tokens per sequence: the two CTAs of an SM fill each other's waits and the last round of
// units is shorter (24 sequences x 4 tokens x 32 heads: 47.7 us, whole states 59.9).  HV = 128, one CTA per SM, for one token: contiguous
// 64 KiB copies, which DRAM likes better (1,024 sequences x 32 heads: 657 to 662 us = the measured copy rate, half states 692).
// Whatever a warp does between a unit's arrival and its store adds to every unit: o leaves behind the hand-over (in front of it 4 us more).
// Per token (order as in fla/ops/kda/fused_recurrent.py:146-192): S *= exp(g); v' = beta (v - S^T k);
// S += k v'^T; o = scale S^T q.
#include <algorithm>

#include "kda_common.cuh"
#include "kda_device.cuh"
#include "kda_tma.cuh"

namespace kda {

namespace {

constexpr int DK = 128, DV = 128;
constexpr int DEC_BUFS = 3;
#ifndef KDA_DECODE_BULK_MIN_UNITS_PER_SM
#define KDA_DECODE_BULK_MIN_UNITS_PER_SM 32      // one token per sequence, fewer (sequence, head) states per SM: the per-warp kernel is used
#endif

template <int HV>
struct DecSmem {
  static constexpr int NW = HV / 16;      // compute warps
  float S[DEC_BUFS][DK * HV];
  float red[2][NW][HV];       // per-warp partial sums of S^T k, by step parity
  float red2[2][NW][HV];      // the same of S^T q
  float kv[3][DK], qv[3][DK], eg[3][DK], vv[3][HV];   // a step's vectors: written one step ahead, so three sets are in use
  float nrm[3][8];            // partial sums of squares: q (warps 0..3), k (warps 0..3)
  float beta[3];
  int dead;                   // a wait gave up
  uint64_t full[DEC_BUFS], ready[DEC_BUFS], gone[DEC_BUFS];      // loaded; written by the compute warps; read by the store
};
static_assert(2 * (sizeof(DecSmem<64>) + 128 + 1024) <= 227 * 1024 && sizeof(DecSmem<128>) + 128 <= 227 * 1024, "DecSmem too large");

struct DecParams {
  kda_recurrent_args a;
  int total, step, dn, dh;    // units; grid; what a step of the grid adds to (sequence, head)
  alignas(64) CUtensorMap tm_in, tm_out;      // states as [rows][128] fp32 in boxes of 128 rows x HV columns
};

// Bit 0: a bounded wait on a state tile gave up (the step's results are incomplete).
__device__ unsigned g_decode_status = 0;

template <typename IO> __device__ __forceinline__ void st1o(IO* p, float x);
template <> __device__ __forceinline__ void st1o<float>(float* p, float x) { *p = x; }
template <> __device__ __forceinline__ void st1o<__nv_bfloat16>(__nv_bfloat16* p, float x) { *p = __float2bfloat16_rn(x); }
template <typename IO> __device__ __forceinline__ void st4o(IO* p, float4 x);
template <> __device__ __forceinline__ void st4o<float>(float* p, float4 x) { *reinterpret_cast<float4*>(p) = x; }
template <> __device__ __forceinline__ void st4o<__nv_bfloat16>(__nv_bfloat16* p, float4 x) {
  *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(x.x, x.y), pack_bf16(x.z, x.w));
}

// Sum over the 32 lanes of 16 per-lane values at once: lane L returns the total of v[L & 15].
__device__ __forceinline__ float butterfly_sum16(float (&v)[16], int lane) {
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], 16);
#pragma unroll
  for (int o = 8; o >= 1; o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float mine = up ? v[i + o] : v[i];
      const float other = up ? v[i] : v[i + o];
      v[i] = mine + __shfl_xor_sync(0xffffffffu, other, o);
    }
  }
  return v[0];
}
__device__ __forceinline__ float4 lds4f(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float part4(const float4& x, int i) { return i == 0 ? x.x : (i == 1 ? x.y : (i == 2 ? x.z : x.w)); }

// where a CTA stands: unit -> (sequence, head, half), token of the sequence
struct Pos {
  int u, n, h, t;
  __device__ __forceinline__ void next_unit(const DecParams& p) {
    u += p.step;
    n += p.dn;
    h += p.dh;
    if (h >= p.a.H) { h -= p.a.H; ++n; }
    t = 0;
  }
  __device__ __forceinline__ void next(const DecParams& p) {
    if (++t >= p.a.T) next_unit(p);
  }
};

}  // namespace

// TR: the states are [slots, H, V, K] (fla's transpose_state_layout): a unit is HV contiguous value rows, a warp owns 16 of them and a
// lane four key columns, so both sums over K stay inside the warp (two butterflies).
// GATE: g and / or beta are the raw layer outputs and are activated here (see kda_recurrent_args::A_log, beta_sigmoid).
template <typename IO, bool TR, bool GATE, int HV>
__global__ void __launch_bounds__(HV * 2 + 32, 128 / HV) kda_decode_bulk_kernel(const __grid_constant__ DecParams p) {
  chain_point();
  extern __shared__ unsigned char smem_raw[];
  constexpr int NW = HV / 16, PARTS = DV / HV;
  constexpr unsigned DEC_TILE = DK * HV * 4;       // bytes of one unit's state
  DecSmem<HV>& s = *reinterpret_cast<DecSmem<HV>*>(smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u));
  const kda_recurrent_args& a = p.a;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int HQ = a.HQ > 0 ? a.HQ : a.H, grp = a.H / HQ;
  if (tid == 0) {
    for (int i = 0; i < DEC_BUFS; ++i) {
      mbar_init(&s.full[i], 1);
      mbar_init(&s.ready[i], NW);
      mbar_init(&s.gone[i], 1);
    }
    s.dead = 0;
    fence_mbar_init();
  }
  __syncthreads();
  Pos first;
  first.u = blockIdx.x;
  first.n = first.u / PARTS / a.H;
  first.h = first.u / PARTS - first.n * a.H;
  first.t = 0;
  const int half = first.u % PARTS;      // the halves of a state stay with neighbouring CTAs: the grid is a multiple of PARTS
  const bool slotted = a.state_indices != nullptr;
  auto wait = [&](uint64_t* bar, unsigned phases, int b) {
    if (*reinterpret_cast<volatile int*>(&s.dead)) return;
    if (!mbar_wait_unrolled(bar + b, (phases >> b) & 1u)) {
      s.dead = 1;
      atomicOr(&g_decode_status, 1u);
    }
  };

  if (warp == NW) {
    // ================= copies =================
    if (lane == 0) {
      auto start_slot = [&](const Pos& q) -> long long {
        if (!slotted) return q.n;
        const int32_t* row = a.state_indices + static_cast<size_t>(q.n) * a.state_indices_stride;
        return row[a.num_accepted_tokens ? a.num_accepted_tokens[q.n] - 1 : 0];
      };
      auto load = [&](long long slot, int h, int b) {
        mbar_expect_tx(&s.full[b], DEC_TILE);
        const long long st = slot * a.H + h;
        if constexpr (TR || HV == DV) bulk_g2s(s.S[b], a.h0 + static_cast<size_t>(st) * (DK * DV) + half * (HV * DK), DEC_TILE, &s.full[b]);
        else tma_load_2d(s.S[b], &p.tm_in, HV * half, static_cast<int>(st * DK), &s.full[b]);
      };
      unsigned ready = 0;
      Pos cur = first, ahead = first;
      load(start_slot(ahead), ahead.h, 0);
      ahead.next_unit(p);
      if (ahead.u < p.total) load(start_slot(ahead), ahead.h, 1);
      ahead.next_unit(p);
      int x = 0, z = 1, y = 2, last = -1;      // this unit's buffer, the next unit's, the spare one; buffer of the last store
      for (; cur.u < p.total; cur.next_unit(p)) {
        const bool more = ahead.u < p.total;
        const long long lslot = more ? start_slot(ahead) : 0;
        const int nst = slotted ? a.T : 1;
        // Two tokens of a sequence may name the same slot, whose last state counts.  Stores of the copy engine are not ordered among each
        // other: at most four are in flight, and one to a slot among theirs waits until those have been written.
        long long recent[4] = {-1, -1, -1, -1};
        for (int c = 0; c < nst; ++c) {
          const int b = (c & 1) ? y : x;
          const long long st = (slotted ? static_cast<long long>(a.state_indices[static_cast<size_t>(cur.n) * a.state_indices_stride + c]) : cur.n) * a.H + cur.h;
          if (HV != DV && (st == recent[0] || st == recent[1] || st == recent[2] || st == recent[3])) bulk_wait<0>();
          wait(s.ready, ready, b);
          ready ^= 1u << b;
          if (s.dead) break;
          if constexpr (TR || HV == DV) bulk_s2g(a.ht + static_cast<size_t>(st) * (DK * DV) + half * (HV * DK), s.S[b], DEC_TILE);
          else tma_store_2d(&p.tm_out, HV * half, static_cast<int>(st * DK), s.S[b]);
          bulk_commit();
          bulk_wait_read<1>();
          if constexpr (HV != DV) {
            bulk_wait<4>();
            recent[3] = recent[2]; recent[2] = recent[1]; recent[1] = recent[0]; recent[0] = st;
          }
          if (last >= 0) mbar_arrive(&s.gone[last]);
          last = b;
        }
        if (s.dead) break;
        const int other = last == x ? y : x;      // its store, if any, has been read: every store but the last one has
        if (more) {
          // whole states: the load waits until the store has left shared memory.  Loads issued earlier mix with the stores in DRAM
          // (1,024 sequences x 32 heads, the variant without gates: 692 us issued in front of the store, 663..668 right behind it or so)
          if constexpr (HV == DV) bulk_wait_read<0>();
          load(lslot, ahead.h, other);
        }
        ahead.next_unit(p);
        x = z;
        z = other;
        y = last;
      }
      if (s.dead) {      // give the loads that may still be in flight into this CTA's memory a bounded time
        for (int i = 0; i < DEC_BUFS; ++i) mbar_drain(&s.full[i]);
      }
      bulk_wait<0>();      // the stores read shared memory and write the states: both complete before the CTA leaves
    }
    __syncwarp();
    return;
  }

  // ================= the compute warps =================
  // A thread fetches its elements of a step's vectors (HV = 64: one of each; 128: of q and k, or of g and v) two steps ahead of its use and keeps the untouched bits in registers until
  // stash(): an instruction that depends on a load makes the thread wait for it right there, and a small load takes longer than
  // a unit's update when the memory system is saturated.  Plain loads, no read-only ones (__ldg): see kda_recurrent.cu.
  // Four registers a step, not seven: with gates the rest made the compiler touch loads still in flight (1,000 x 32, the layer's call: 682 -> 649 us)
  // (HV = 128: the threads of q, k and those of g, v use the same registers; beta waits in thread 0's slot for A_log, which it has no use for)
  constexpr int RQ = 0, RK = 1, RG = HV == 64 ? 2 : 0, RV = HV == 64 ? 3 : 1, RA = HV == 64 ? 4 : 2, RBIAS = HV == 64 ? 5 : 3, RB = HV == 64 ? 6 : 2;
  struct Raw { uint32_t x[HV == 64 ? 7 : 4]; };
  constexpr bool IO16 = sizeof(IO) == 2;
  auto ld_bits = [&](const void* ptr, size_t i, bool bf16) -> uint32_t {
    if (bf16) return static_cast<const unsigned short*>(ptr)[i];
    return static_cast<const uint32_t*>(ptr)[i];
  };
  auto to_float = [&](uint32_t bits, bool bf16) -> float { return __uint_as_float(bf16 ? bits << 16 : bits); };
  const int e = tid & 127;
  const bool has_qk = HV == 64 || warp < 4, has_gv = HV == 64 || warp >= 4;
  auto fetch = [&](const Pos& q, Raw& r) {
    const size_t tok = static_cast<size_t>(q.n) * a.T + q.t, row = tok * a.H + q.h;
    const size_t rowq = (tok * HQ + q.h / grp) * DK + e;
    if (has_qk) {
      r.x[RQ] = ld_bits(a.q, rowq, IO16);
      r.x[RK] = ld_bits(a.k, rowq, IO16);
    }
    if (has_gv) {
      if constexpr (GATE) {
        r.x[RG] = ld_bits(a.g, row * DK + e, a.A_log && a.g_raw_dtype == KDA_BF16);
        if (a.A_log) {
          r.x[RA] = __float_as_uint(a.A_log[q.h]);
          r.x[RBIAS] = a.dt_bias ? __float_as_uint(a.dt_bias[static_cast<size_t>(q.h) * DK + e]) : 0u;
        }
      } else {
        r.x[RG] = __float_as_uint(a.g[row * DK + e]);
      }
      if (e < HV) r.x[RV] = ld_bits(a.v, row * DV + half * HV + e, IO16);
    }
    if (tid == 0) {
      if constexpr (GATE) r.x[RB] = ld_bits(a.beta, row, a.beta_sigmoid && a.beta_raw_dtype == KDA_BF16);
      else r.x[RB] = __float_as_uint(a.beta[row]);
    }
  };
  auto stash = [&](int buf, const Raw& r) {
    if (has_qk) {
      const float q = to_float(r.x[RQ], IO16), k = to_float(r.x[RK], IO16);
      s.qv[buf][e] = q;
      s.kv[buf][e] = k;
      if (a.use_qk_l2norm) {
        const float sq = warp_sum(q * q), sk = warp_sum(k * k);
        if (lane == 0) {
          s.nrm[buf][warp] = sq;
          s.nrm[buf][4 + warp] = sk;
        }
      }
    }
    if (has_gv) {
      float g = __uint_as_float(r.x[RG]);
      if constexpr (GATE) {
        if (a.A_log) {
          const float x = to_float(r.x[RG], a.g_raw_dtype == KDA_BF16) + __uint_as_float(r.x[RBIAS]);
          const float al = __expf(__uint_as_float(r.x[RA]));
          g = a.use_lower_bound ? a.lower_bound * sigmoid_fast(al * x) : -al * softplus_fast(x);
        }
      }
      s.eg[buf][e] = __expf(g);
      if (e < HV) s.vv[buf][e] = to_float(r.x[RV], IO16);
    }
    if (tid == 0) {
      float b = __uint_as_float(r.x[RB]);
      if constexpr (GATE) {
        if (a.beta_sigmoid) b = sigmoid_fast(to_float(r.x[RB], a.beta_raw_dtype == KDA_BF16));
      }
      s.beta[buf] = b;
    }
  };
  auto meet = [] { asm volatile("bar.sync 1, %0;" ::"n"(NW * 32) : "memory"); };      // the compute warps
  IO* const op = static_cast<IO*>(a.o);
  // !TR: this thread's four value columns and sixteen key rows
  const int col = HV == 64 ? 4 * (lane & 15) : 4 * lane, row0 = HV == 64 ? 32 * warp + 16 * (lane >> 4) : 16 * warp;
  const bool lead = HV == 128 || lane < 16;      // HV = 64: the two halves of a warp share columns
  auto write_o = [&](size_t row, int par) {                               // !TR: o of a finished step (one warp)
    if (lead) {
      float4 o = lds4f(&s.red2[par][0][col]);
#pragma unroll
      for (int w = 1; w < NW; ++w) {
        const float4 x = lds4f(&s.red2[par][w][col]);
        o.x += x.x; o.y += x.y; o.z += x.z; o.w += x.w;
      }
      st4o(op + row * DV + half * HV + col, o);
    }
  };

  Pos cur = first, nxt = first, ahead = first;
  size_t prev = 0;
  Raw rx = {}, ry;
  {
    Raw r0 = {};
    fetch(cur, r0);
    nxt.next(p);
    if (nxt.u < p.total) fetch(nxt, rx);
    stash(0, r0);
    ahead = nxt;
    ahead.next(p);
  }
  meet();
  unsigned full = 0, sp = 0, any = 0;      // parities of the next load of each buffer; of its stores so far; has it been stored from
  int x = 0, z = 1, y = 2, buf = 0, c = 0;
  float4 Sr[16];
  for (int step = 0; cur.u < p.total; ++step) {
    const int par = step & 1;
    ry = Raw{};
    if (ahead.u < p.total) fetch(ahead, ry);
    const bool fresh = cur.t == 0, keep = slotted || cur.t == a.T - 1;
    if (fresh) {
      wait(s.full, full, x);
      full ^= 1u << x;
      c = 0;
    }
    const int dst = (c & 1) ? y : x;
    float rq = a.scale, rk = 1.f;
    if (a.use_qk_l2norm) {
      const float4 nq = lds4f(&s.nrm[buf][0]), nk = lds4f(&s.nrm[buf][4]);
      rq *= rsqrtf(nq.x + nq.y + nq.z + nq.w + L2NORM_EPS);
      rk = rsqrtf(nk.x + nk.y + nk.z + nk.w + L2NORM_EPS);
    }
    const int buf1 = buf == 2 ? 0 : buf + 1;
    float4 hk = make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (TR) {
      if (fresh) {
#pragma unroll
        for (int i = 0; i < 16; ++i) Sr[i] = lds4f(&s.S[x][(16 * warp + i) * DK + 4 * lane]);
      }
    } else {
      if (fresh) {
#pragma unroll
        for (int i = 0; i < 16; ++i) Sr[i] = lds4f(&s.S[x][(row0 + i) * HV + col]);
      }
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const float4 e4 = lds4f(&s.eg[buf][row0 + 4 * g]), k4 = lds4f(&s.kv[buf][row0 + 4 * g]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float4& S = Sr[4 * g + j];
          const float e = part4(e4, j), kk = part4(k4, j) * rk;
          S.x *= e; S.y *= e; S.z *= e; S.w *= e;
          hk.x = fmaf(kk, S.x, hk.x); hk.y = fmaf(kk, S.y, hk.y); hk.z = fmaf(kk, S.z, hk.z); hk.w = fmaf(kk, S.w, hk.w);
        }
      }
      if constexpr (HV == 64) {
        hk.x += __shfl_xor_sync(0xffffffffu, hk.x, 16);
        hk.y += __shfl_xor_sync(0xffffffffu, hk.y, 16);
        hk.z += __shfl_xor_sync(0xffffffffu, hk.z, 16);
        hk.w += __shfl_xor_sync(0xffffffffu, hk.w, 16);
      }
      if (lead) *reinterpret_cast<float4*>(&s.red[par][warp][col]) = hk;
    }
    if (nxt.u < p.total) stash(buf1, rx);
    rx = ry;
    meet();
    if (keep && c > 0 && ((any >> dst) & 1u)) wait(s.gone, ~sp, dst);      // the copy engine has read the buffer's last store
    if constexpr (TR) {
      const float4 e4 = lds4f(&s.eg[buf][4 * lane]);
      float4 k4 = lds4f(&s.kv[buf][4 * lane]), q4 = lds4f(&s.qv[buf][4 * lane]);
      k4.x *= rk; k4.y *= rk; k4.z *= rk; k4.w *= rk;
      q4.x *= rq; q4.y *= rq; q4.z *= rq; q4.w *= rq;
      float part[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        Sr[i].x *= e4.x; Sr[i].y *= e4.y; Sr[i].z *= e4.z; Sr[i].w *= e4.w;
        part[i] = fmaf(k4.x, Sr[i].x, fmaf(k4.y, Sr[i].y, fmaf(k4.z, Sr[i].z, k4.w * Sr[i].w)));
      }
      const float h = butterfly_sum16(part, lane);                     // value row 16 warp + (lane & 15)
      const float dvl = s.beta[buf] * (s.vv[buf][16 * warp + (lane & 15)] - h);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float dvi = __shfl_sync(0xffffffffu, dvl, i);
        Sr[i].x = fmaf(k4.x, dvi, Sr[i].x); Sr[i].y = fmaf(k4.y, dvi, Sr[i].y); Sr[i].z = fmaf(k4.z, dvi, Sr[i].z); Sr[i].w = fmaf(k4.w, dvi, Sr[i].w);
        part[i] = fmaf(q4.x, Sr[i].x, fmaf(q4.y, Sr[i].y, fmaf(q4.z, Sr[i].z, q4.w * Sr[i].w)));
        if (keep) *reinterpret_cast<float4*>(&s.S[dst][(16 * warp + i) * DK + 4 * lane]) = Sr[i];
      }
      const float o = butterfly_sum16(part, lane);
      if (lane < 16) st1o(op + ((static_cast<size_t>(cur.n) * a.T + cur.t) * a.H + cur.h) * DV + half * HV + 16 * warp + lane, o);
    } else {
      hk = lds4f(&s.red[par][0][col]);
#pragma unroll
      for (int w = 1; w < NW; ++w) {
        const float4 v = lds4f(&s.red[par][w][col]);
        hk.x += v.x; hk.y += v.y; hk.z += v.z; hk.w += v.w;
      }
      const float4 vt = lds4f(&s.vv[buf][col]);
      const float beta = s.beta[buf];
      const float4 dv = make_float4(beta * (vt.x - hk.x), beta * (vt.y - hk.y), beta * (vt.z - hk.z), beta * (vt.w - hk.w));
      float4 oa = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const float4 k4 = lds4f(&s.kv[buf][row0 + 4 * g]), q4 = lds4f(&s.qv[buf][row0 + 4 * g]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float4& S = Sr[4 * g + j];
          const float kk = part4(k4, j) * rk, qq = part4(q4, j) * rq;
          S.x = fmaf(kk, dv.x, S.x); S.y = fmaf(kk, dv.y, S.y); S.z = fmaf(kk, dv.z, S.z); S.w = fmaf(kk, dv.w, S.w);
          oa.x = fmaf(qq, S.x, oa.x); oa.y = fmaf(qq, S.y, oa.y); oa.z = fmaf(qq, S.z, oa.z); oa.w = fmaf(qq, S.w, oa.w);
          if (keep) *reinterpret_cast<float4*>(&s.S[dst][(row0 + 4 * g + j) * HV + col]) = S;
        }
      }
      if constexpr (HV == 64) {
        oa.x += __shfl_xor_sync(0xffffffffu, oa.x, 16);
        oa.y += __shfl_xor_sync(0xffffffffu, oa.y, 16);
        oa.z += __shfl_xor_sync(0xffffffffu, oa.z, 16);
        oa.w += __shfl_xor_sync(0xffffffffu, oa.w, 16);
      }
      if (lead) *reinterpret_cast<float4*>(&s.red2[par][warp][col]) = oa;
    }
    if (keep) {
      fence_proxy_async();          // the updated state becomes visible to the copy engine
      __syncwarp();
      if (lane == 0) mbar_arrive(&s.ready[dst]);
      sp ^= 1u << dst;
      any |= 1u << dst;
      ++c;
    }
    if (!TR && step > 0 && warp == (step % NW)) write_o(prev, par ^ 1);      // behind the hand-over: in front of it this warp held up the unit's store
    if (!TR) prev = (static_cast<size_t>(cur.n) * a.T + cur.t) * a.H + cur.h;
    if (cur.t == a.T - 1) {         // the buffers take the roles the copying warp gives them
      const int last = (c & 1) ? x : y, other = last == x ? y : x;
      x = z;
      z = other;
      y = last;
    }
    cur = nxt;
    nxt = ahead;
    ahead.next(p);
    buf = buf1;
    if (!TR && cur.u >= p.total) {
      meet();
      if (warp == 0) write_o(prev, par);
    }
  }
}

namespace {

template <typename IO, bool TR, bool GATE, int HV>
int launch_hv(const kda_recurrent_args& a, cudaStream_t st) {
  const int smem = static_cast<int>(sizeof(DecSmem<HV>)) + 128;
  static DeviceOnce once;      // per template variant, per device
  const int rc = once.run([&] {
    return cudaFuncSetAttribute(kda_decode_bulk_kernel<IO, TR, GATE, HV>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  });
  if (rc != KDA_OK) return rc;
  constexpr int PARTS = DV / HV;
  DecParams p{};
  p.a = a;
  p.total = PARTS * a.N * a.H;
  p.step = std::min(p.total, PARTS * sm_count());
  p.dn = p.step / PARTS / a.H;
  p.dh = p.step / PARTS % a.H;
  if (!TR && HV != DV && (make_states_tmap(&p.tm_in, a.h0, DV, HV, DK) || make_states_tmap(&p.tm_out, a.ht, DV, HV, DK))) return KDA_E_TMAP;
  return static_cast<int>(launch_chained(kda_decode_bulk_kernel<IO, TR, GATE, HV>, static_cast<unsigned>(p.step), HV * 2 + 32, smem, st, p));
}

template <typename IO, bool TR, bool GATE>
int launch(const kda_recurrent_args& a, cudaStream_t st) {
  if constexpr (TR || GATE) {
    if (a.T == 1) return launch_hv<IO, TR, GATE, 128>(a, st);
  }
  return launch_hv<IO, TR, GATE, 64>(a, st);
}

}  // namespace

// Whether the bulk-copy decode kernel takes this call (K = V = 128, states carried from h0 to ht, either layout).
// Several tokens per sequence, each with its slot: on half states, from half a state per SM on (us, this kernel | the per-warp one; 32
// heads: 2 x 4 tokens 7.2 | 7.9, 4 x 4 10.7 | 11.4, 8 x 4 18.6 | 18.1, 24 x 4 47.7 | 48.3, 128 x 3 180 | 192).
// One token: whole states, from 32 states per SM on.  Below, the per-warp kernel spreads the work more finely (48 sequences x 32 heads:
// 38.3 | 34.8; 128: 88.8 | 87.7; 160: 109.7 | 109.5; 256: 171 | 181; 1,024: 672 | 703).
bool decode_bulk_covers(const kda_recurrent_args& a) {
  if (a.K != DK || a.V != DV || !a.h0 || !a.ht || a.cu_seqlens || a.T < 1 || (a.T > 1 && !a.state_indices)) return false;
  if (a.io_dtype != KDA_BF16 && a.io_dtype != KDA_FP32) return false;
  const long long states = static_cast<long long>(a.N) * a.H;
  if (a.T > 1) return 2 * states > sm_count() && states <= 0x3fffffff;
  return states >= KDA_DECODE_BULK_MIN_UNITS_PER_SM * static_cast<long long>(sm_count()) && states <= 0x3fffffff;
}

int decode_bulk_launch(const kda_recurrent_args& a, cudaStream_t st) {
  // One token, states [K, V]: the variant with gates also serves the calls without.  At the copy rate it is when the loads and stores of the SMs
  // meet in DRAM that decides, and that variant's steps fall better (without gates, us, its own variant | this one: 148 sequences x 32 heads
  // 102.0 | 100.5, 512: 340 | 334, 1,024: 666 | 657, 1,500: 978 | 962).  States [V, K]: its own is better (1,024: 655 | 680).
  const bool gate = a.A_log != nullptr || a.beta_sigmoid != 0 || (a.T == 1 && !a.transpose_state);
  const int which = (a.io_dtype == KDA_BF16 ? 0 : 4) + (a.transpose_state ? 2 : 0) + (gate ? 1 : 0);
  switch (which) {
    case 0: return launch<__nv_bfloat16, false, false>(a, st);
    case 1: return launch<__nv_bfloat16, false, true>(a, st);
    case 2: return launch<__nv_bfloat16, true, false>(a, st);
    case 3: return launch<__nv_bfloat16, true, true>(a, st);
    case 4: return launch<float, false, false>(a, st);
    case 5: return launch<float, false, true>(a, st);
    case 6: return launch<float, true, false>(a, st);
    default: return launch<float, true, true>(a, st);
  }
}

}  // namespace kda

extern "C" int kda_recurrent_status(uint32_t* host_out) {
  if (!host_out) return KDA_E_NULL;
  unsigned v = 0, zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, kda::g_decode_status, sizeof(v));
  if (e == cudaSuccess && v) e = cudaMemcpyToSymbol(kda::g_decode_status, &zero, sizeof(zero));
  *host_out = v;
  return static_cast<int>(e);
}
