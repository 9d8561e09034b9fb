// Token-recurrent KDA training in fp32 (K, V in {32, 64, 128}): forward that keeps what the backward needs, and its exact reverse mode.
// The recurrence of fla/ops/kda/naive.py:12-66,
//
//   S' = Diag(exp g_t) S_{t-1};   r = v - S'^T k;   w = beta_t r;   S_t = S' + k w^T;   o_t = scale S_t^T q_t,
//
// differentiated step by step, with no chunk formula in between (those lose dg to cancellation: 3e-6 against 1.4e-7):
//
//   dS += scale q do^T;  dq^ = scale S_t do;  dw = dS^T k;  dk^ = dS w - S' (beta dw);  dbeta = <dw, r>;
//   dv = beta dw;  dS' = dS - k (beta dw)^T;  dg = rowsum(dS' . S');  dS <- Diag(exp g) dS'.
//
// Only two chains run through a whole sequence, and both fall apart into the state's columns: S forward (its sums run over k) and dS
// backward (needs q, k, g, beta, do, but no S).  So three kernels:
//   walk forward    S alone.  Leaves the state at every border of a sequence's 32-token pieces and r of every token.
//   walk backward   dS alone.  Leaves dS at the same borders, dv, and dbeta summed over 16 columns.
//   middle          every piece (32 tokens or the rest of the sequence, 32 rows of the state) on its own.  With r and beta dw known a step needs no sum over
//                   k: S and dS of a row follow from that row's q, k, g, and its dq^, dk^, dg are sums along the row.
// What the forward walk leaves (2.5 KB per token and head of 128) is kept until the backward where the caller has the memory; otherwise the backward
// replays the walk.  Heads may be worked on in groups, one after another, in a part of the scratch.  Neither changes a bit.
// Walks: a warp holds 16 or 32 columns of all K rows (a lane 16 rows x 4 or 8 columns, packed two rows to a register pair), and nothing is
// shared between warps but the staged q, k, exp g.
// Middle: a thread holds 8 columns of 4 rows of S and dS.  S' of four tokens lives in registers; the states between are replayed once and kept as they
// are, every fourth token, in tensor memory (256 columns a CTA, which nothing else here uses): 10.5 multiply-adds per element and token, and no
// per-token state through memory (128 KB per token: what a CTA per sequence waited for).  The tile's shape is set by shared-memory bandwidth, which is
// 128 bytes per cycle delivered to registers, broadcast or not: with 16 columns of one row a thread reads 90 floats per 16 elements and token (92 % of
// the LSU's rate, 7.5 ms), with 4 x 8 it reads 36.  With every eighth token's state in shared memory, replayed further from there: 5.0 ms; every fourth
// in tensor memory 4.7; loops that end with the piece's tokens instead of unrolled to 32 4.5.
// What bounds them: the FP32 pipe (61 % busy in the middle, 50 % in the walks; one CTA's load of its rows and states under the other's arithmetic) and,
// in the walks, the 256 units' uneven share of 148 SMs.  8 x 2048 tokens x 32 heads of 128: forward walk 2.11, backward walk 2.11, middle 4.5 ms; the
// whole step 25.7 ms as a CTA per sequence, 8.77 with what the forward kept, 10.6 with the replay.  One sequence x 32 heads: 12.8 -> 2.4 (3.1) ms;
// 2 x 200 tokens x 8 heads: 1.25 -> 0.27 (0.33); 2,000 sequences of five tokens x 8: 3.5 -> 2.3 (2.6).
// (Walks of two tokens a step, seven multiply-adds instead of eight and one reduction: 1 % less at 256 units, 5 % more at 32.)
// dq^, dk^ (gradients w.r.t. the possibly L2-normalised rows, per VALUE head) go to the workspace; a last kernel sums grouped value
// heads, applies the normalisation's backward (fla/modules/l2norm.py:190-240) and writes dq, dk; with neither they are dq, dk.  Every sum has a
// fixed order.
#include <algorithm>

#include "kda_common.cuh"
#include "kda_device.cuh"
#include "kda_f32x2.cuh"
#include "kda_umma.cuh"

namespace kda {

namespace {

constexpr int TC = 32;      // tokens between two kept states
constexpr int TS = 8;       // tokens staged at a time in the walks (TC is a multiple)

struct TrainParams {
  const float *q, *k, *v, *g, *beta, *h0, *d_o, *d_ht;
  const int32_t* cu;
  float *o, *ht;
  float *dqh, *dkh;            // [tokens, H, K] per value head, w.r.t. the normalised rows
  float *dv, *dg, *dbeta, *dh0;
  float *ckpt;                 // [tokens / 32][H][K][V] states at the borders of a sequence's 32-token pieces (its ends are h0 and ht)
  float *resid;                // [tokens, H, V] r
  float *norms;                // [tokens, H, 2] reciprocal norms of q, k (only with use_l2)
  float *dckpt;                // like ckpt: dS at the same borders
  float *dbp;                  // [tokens, H, V / 16] dbeta over 16 columns
  long long T, slots;
  int N, H, HQ, V;             // H, HQ: heads of the tensors
  int HL;                      // value heads of this launch: every pointer starts at the first of them
  int HS, HD, HW;              // heads per token or border in ckpt, resid, norms; in dqh, dkh; in dckpt, dbp
  int use_l2, wide;            // wide: q, k, g start on 16-byte boundaries
  float scale, dq_scale;       // dq_scale: what dqh still gets (without grouped heads and norms dqh, dkh are dq, dk themselves)
};

// first token and length of sequence n.  Its 32-token pieces are numbered from bos / 32 + n (disjoint for any lengths), the borders between them from
// bos / 32: ceil(len / 32) - 1 of them, at most floor((bos + len - 1) / 32) - floor(bos / 32).
struct Seq { long long bos, len; };
__device__ __forceinline__ long long seq_start(const TrainParams& p, long long n) { return p.cu ? p.cu[n] : n * p.T; }
__device__ __forceinline__ Seq sequence(const TrainParams& p, int n) {
  const long long b = seq_start(p, n);
  return {b, seq_start(p, n + 1) - b};
}

__device__ __forceinline__ void cp_async16(void* dst_smem, const void* src_gmem, bool valid) {
  const unsigned sz = valid ? 16u : 0u;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst_smem)), "l"(src_gmem), "r"(sz) : "memory");
}
// 16 bytes of q, k or g, which a caller of the backward may hand over at any 4-byte boundary
__device__ __forceinline__ void cp_row16(float* dst_smem, const float* src_gmem, int wide) {
  if (wide) {
    cp_async16(dst_smem, src_gmem, true);
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) cp_async4(dst_smem + e, src_gmem + e, true);
  }
}
// E consecutive floats of a row in shared memory
template <int E>
__device__ __forceinline__ void row_get(float (&x)[E], const float* p) {
  if constexpr (E == 4) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
  } else if constexpr (E == 2) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    x[0] = v.x; x[1] = v.y;
  } else {
    x[0] = *p;
  }
}
template <int E>
__device__ __forceinline__ void row_put(float* p, const float (&x)[E]) {
  if constexpr (E == 4) *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
  else if constexpr (E == 2) *reinterpret_cast<float2*>(p) = make_float2(x[0], x[1]);
  else *p = x[0];
}
__device__ __forceinline__ float dot4(const float4 a, const float4 b) { return a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w; }

// ---------------------------------------------------------------------------------------------------------------------
// the walks
// ---------------------------------------------------------------------------------------------------------------------
template <int K, int CPL>
struct WalkSmem {
  static constexpr int COLS = CPL * 16;      // a CTA's columns, at most
  float q[2][TS][K];          // scale * q^
  float k[2][TS][K];          // k^
  float a[2][TS][K];          // exp g
  float x[2][TS][COLS];       // this CTA's columns of v (forward), do (backward)
  float y[2][TS][COLS];       // of r (backward)
  float beta[2][TS];
};

// A warp's share of a [K, V] state, 4 CPL columns: a lane has columns col + 16 m + (0..3), m < CPL / 4, of rows 32 i + 4 rg + (0..3);
// pairs are two neighbouring rows.
template <int K, int CPL>
struct Slice {
  f32x2 v[K / 32][2][CPL];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < K / 32; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int c = 0; c < CPL; ++c) v[i][e][c] = 0ull;
  }
  __device__ __forceinline__ void load(const float* base, int rg, int V) {      // base: row 0, column col
#pragma unroll
    for (int i = 0; i < K / 32; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int m = 0; m < CPL / 4; ++m) {
          const float4 x = *reinterpret_cast<const float4*>(base + static_cast<size_t>(32 * i + 4 * rg + 2 * e) * V + 16 * m);
          const float4 y = *reinterpret_cast<const float4*>(base + static_cast<size_t>(32 * i + 4 * rg + 2 * e + 1) * V + 16 * m);
          v[i][e][4 * m] = pair(x.x, y.x); v[i][e][4 * m + 1] = pair(x.y, y.y);
          v[i][e][4 * m + 2] = pair(x.z, y.z); v[i][e][4 * m + 3] = pair(x.w, y.w);
        }
  }
  __device__ __forceinline__ void store(float* base, int rg, int V) const {
#pragma unroll
    for (int i = 0; i < K / 32; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int m = 0; m < CPL / 4; ++m) {
          const float2 c0 = halves(v[i][e][4 * m]), c1 = halves(v[i][e][4 * m + 1]), c2 = halves(v[i][e][4 * m + 2]), c3 = halves(v[i][e][4 * m + 3]);
          *reinterpret_cast<float4*>(base + static_cast<size_t>(32 * i + 4 * rg + 2 * e) * V + 16 * m) = make_float4(c0.x, c1.x, c2.x, c3.x);
          *reinterpret_cast<float4*>(base + static_cast<size_t>(32 * i + 4 * rg + 2 * e + 1) * V + 16 * m) = make_float4(c0.y, c1.y, c2.y, c3.y);
        }
  }
};
// sums over the rows of a lane's columns: the pairs' halves, then the eight row groups of the warp (lane bits 2..4); every lane gets all
template <int CPL>
__device__ __forceinline__ void column_sums(const f32x2 (&h)[CPL], float (&s)[CPL]) {
#pragma unroll
  for (int c = 0; c < CPL; ++c) s[c] = halves(h[c]).x + halves(h[c]).y;
#pragma unroll
  for (int o = 4; o < 32; o <<= 1)
#pragma unroll
    for (int c = 0; c < CPL; ++c) s[c] += __shfl_xor_sync(0xffffffffu, s[c], o);
}
// one of two values with the other lane's share of it added: the lane whose bit `o` is set keeps `hi`
__device__ __forceinline__ float fold(float lo, float hi, int o, int lane) {
  const bool up = (lane & o) != 0;
  return (up ? hi : lo) + __shfl_xor_sync(0xffffffffu, up ? lo : hi, o);
}

// FWD: v comes in, o (when wanted), r and the states leave; otherwise do and r come in, dv, dbeta's parts and the dS leave.
template <int K, int CPL, bool FWD>
__global__ void __launch_bounds__(128, CPL == 8 ? 2 : 4) kda_recurrent_walk_kernel(const TrainParams p) {
  chain_point();
  constexpr int I = K / 32, E = K / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  WalkSmem<K, CPL>& s = *reinterpret_cast<WalkSmem<K, CPL>*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5, nt = blockDim.x;
  const int ncols = 4 * CPL * nw, parts = p.V / ncols;
  const int unit = blockIdx.x / parts, part = blockIdx.x % parts;
  const int n = unit / p.HL, h = unit % p.HL, hq = h / (p.H / p.HQ);
  const int V = p.V, cg = lane & 3, rg = lane >> 2, lcol = 4 * CPL * warp + 4 * cg, col = part * ncols + lcol;
  const Seq sq = sequence(p, n);
  const int stages = static_cast<int>((sq.len + TS - 1) / TS);
  const bool keeps = !FWD || p.ckpt;      // (a forward that leaves nothing: no states, no r, no norms)
  const int HK = FWD ? p.HS : p.HW;
  float* const kept = (FWD ? p.ckpt : p.dckpt) + ((sq.bos / TC) * HK + h) * static_cast<size_t>(K) * V + col;
  const size_t sbase = (static_cast<size_t>(n) * p.H + h) * K * V + col;

  const long long out_step = FWD ? 1LL * p.HS * V : -1LL * p.H * V, aux_step = FWD ? 1LL * p.H * V : -1LL * p.HW * (V / 16);
  const int oc = CPL == 8 ? rg : rg >> 1, ocol = col + 16 * (oc >> 2) + (oc & 3);      // the column whose o this lane ends with

  auto tokens_of = [&](int st) { return static_cast<int>(min(static_cast<long long>(TS), sq.len - static_cast<long long>(st) * TS)); };
  auto issue = [&](int st) {      // raw rows of stage st on their way
    const int b = st & 1, cnt = tokens_of(st);
    const size_t tok0 = static_cast<size_t>(sq.bos + static_cast<long long>(st) * TS);
    for (int i = tid; i < cnt * (K / 4); i += nt) {
      const int j = i / (K / 4), c = 4 * (i % (K / 4));
      const size_t rowq = ((tok0 + j) * p.HQ + hq) * K + c;
      cp_row16(&s.k[b][j][c], p.k + rowq, p.wide);
      if (!FWD || p.o) cp_row16(&s.q[b][j][c], p.q + rowq, p.wide);
      cp_row16(&s.a[b][j][c], p.g + ((tok0 + j) * p.H + h) * K + c, p.wide);
    }
    for (int i = tid; i < cnt * (ncols / 4); i += nt) {
      const int j = i / (ncols / 4), c = 4 * (i % (ncols / 4));
      const size_t row = ((tok0 + j) * p.H + h) * V + part * ncols + c;
      cp_async16(&s.x[b][j][c], (FWD ? p.v : p.d_o) + row, true);
      if (!FWD) cp_async16(&s.y[b][j][c], p.resid + ((tok0 + j) * p.HS + h) * V + part * ncols + c, true);
    }
    if (tid < cnt) cp_async4(&s.beta[b][tid], p.beta + (tok0 + tid) * p.H + h, true);
    cp_async_commit();
  };
  auto activate = [&](int st) {      // in place: exp g, normalised rows, scale; a warp per token
    const int b = st & 1, cnt = tokens_of(st);
    for (int j = warp; j < cnt; j += nw) {
      float kf[E], qf[E], gf[E];
      row_get<E>(kf, &s.k[b][j][lane * E]);
      row_get<E>(gf, &s.a[b][j][lane * E]);
      const bool with_q = !FWD || p.o || p.use_l2;
      if (!FWD || p.o) row_get<E>(qf, &s.q[b][j][lane * E]);
      float qs = p.scale, ks = 1.f;
      if (p.use_l2) {
        const size_t tok = static_cast<size_t>(sq.bos + static_cast<long long>(st) * TS + j), row = tok * p.HS + h;
        if (FWD) {
          if (!p.o) {      // (replay in front of a backward: q is only here for its norm)
#pragma unroll
            for (int e = 0; e < E; ++e) qf[e] = p.q[(tok * p.HQ + hq) * K + lane * E + e];
          }
          float ssq = 0.f, ssk = 0.f;
#pragma unroll
          for (int e = 0; e < E; ++e) {
            ssq += qf[e] * qf[e];
            ssk += kf[e] * kf[e];
          }
          const float rq = rsqrtf(warp_sum(ssq) + L2NORM_EPS), rk = rsqrtf(warp_sum(ssk) + L2NORM_EPS);
          if (lane == 0 && part == 0 && p.norms) *reinterpret_cast<float2*>(p.norms + 2 * row) = make_float2(rq, rk);
          qs *= rq;
          ks = rk;
        } else {
          const float2 r = *reinterpret_cast<const float2*>(p.norms + 2 * row);
          qs *= r.x;
          ks = r.y;
        }
      }
#pragma unroll
      for (int e = 0; e < E; ++e) {
        if (with_q) qf[e] *= qs;
        kf[e] *= ks;
        gf[e] = expf(gf[e]);
      }
      row_put<E>(&s.k[b][j][lane * E], kf);
      row_put<E>(&s.a[b][j][lane * E], gf);
      if (!FWD || p.o) row_put<E>(&s.q[b][j][lane * E], qf);
    }
  };

  Slice<K, CPL> S;
  const float* const start = FWD ? p.h0 : p.d_ht;
  if (start) S.load(start + sbase, rg, V);
  else S.zero();
  if (stages > 0) issue(FWD ? 0 : stages - 1);
  for (int it = 0; it < stages; ++it) {
    const int st = FWD ? it : stages - 1 - it, b = st & 1, cnt = tokens_of(st);
    cp_async_wait<0>();
    __syncthreads();      // stage st has arrived; everybody is done with the other buffer
    if (it + 1 < stages) issue(FWD ? st + 1 : st - 1);
    activate(st);
    if (keeps && it > 0 && st % (TC / TS) == (FWD ? 0 : TC / TS - 1))      // behind piece st / 4 - 1 (forward), st / 4
      S.store(kept + static_cast<size_t>(st / (TC / TS) - (FWD ? 1 : 0)) * HK * K * V, rg, V);
    __syncthreads();
    // (running pointers: the products of 64-bit indices cost more than a tenth of a token's instructions)
    const size_t tok1 = static_cast<size_t>(sq.bos + static_cast<long long>(st) * TS + (FWD ? 0 : cnt - 1));
    float* out = (FWD ? p.resid + (tok1 * p.HS + h) * V : p.dv + (tok1 * p.H + h) * V) + col + 16 * rg;                // r, dv: row groups 0 (and 1) store
    float* aux = FWD ? p.o + (tok1 * p.H + h) * V + ocol : p.dbp + (tok1 * p.HW + h) * (V / 16) + col / 16;      // o, dbeta's parts
    for (int jj = 0; jj < cnt; ++jj, out += out_step, aux += aux_step) {
      const int j = FWD ? jj : cnt - 1 - jj;
      const float* const kr = &s.k[b][j][4 * rg];
      const float* const ar = &s.a[b][j][4 * rg];
      const float* const qr = &s.q[b][j][4 * rg];
      float x[CPL];
#pragma unroll
      for (int m = 0; m < CPL / 4; ++m) {
        const float4 y = *reinterpret_cast<const float4*>(&s.x[b][j][lcol + 16 * m]);
        x[4 * m] = y.x; x[4 * m + 1] = y.y; x[4 * m + 2] = y.z; x[4 * m + 3] = y.w;
      }
      const float beta = s.beta[b][j];
      // (one sum a column, whatever the lane's number of columns: every sequence gets the same bits alone and in a large batch)
      f32x2 acc[CPL];
      F4 k[I];
#pragma unroll
      for (int i = 0; i < I; ++i) k[i] = lds4(kr + 32 * i);
#pragma unroll
      for (int c = 0; c < CPL; ++c) acc[c] = 0ull;
      if constexpr (FWD) {
#pragma unroll
        for (int i = 0; i < I; ++i) {
          const F4 a = lds4(ar + 32 * i);
#pragma unroll
          for (int c = 0; c < CPL; ++c) {
            S.v[i][0][c] = mul2(S.v[i][0][c], a.a);
            S.v[i][1][c] = mul2(S.v[i][1][c], a.b);
            acc[c] = fma2(S.v[i][0][c], k[i].a, acc[c]);
            acc[c] = fma2(S.v[i][1][c], k[i].b, acc[c]);
          }
        }
        float hk[CPL];
        column_sums(acc, hk);
        f32x2 w2[CPL];
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
          x[c] -= hk[c];      // r
          w2[c] = pair(beta * x[c], beta * x[c]);
          acc[c] = 0ull;
        }
        if (keeps && rg < CPL / 4)
          *reinterpret_cast<float4*>(out) =
              CPL == 8 && rg ? make_float4(x[CPL - 4], x[CPL - 3], x[CPL - 2], x[CPL - 1]) : make_float4(x[0], x[1], x[2], x[3]);
#pragma unroll
        for (int i = 0; i < I; ++i) {
          const F4 q = lds4(qr + 32 * i);
#pragma unroll
          for (int c = 0; c < CPL; ++c) {
            S.v[i][0][c] = fma2(k[i].a, w2[c], S.v[i][0][c]);
            S.v[i][1][c] = fma2(k[i].b, w2[c], S.v[i][1][c]);
            acc[c] = fma2(S.v[i][0][c], q.a, acc[c]);
            acc[c] = fma2(S.v[i][1][c], q.b, acc[c]);
          }
        }
        if (p.o) {      // summed off the chain: a lane ends with one column
          float y[CPL];
#pragma unroll
          for (int c = 0; c < CPL; ++c) y[c] = halves(acc[c]).x + halves(acc[c]).y;
          int o = 16;
#pragma unroll
          for (int half = CPL / 2; half >= 1; half >>= 1, o >>= 1)
#pragma unroll
            for (int c = 0; c < half; ++c) y[c] = fold(y[c], y[c + half], o, lane);
          if (CPL == 4) y[0] += __shfl_xor_sync(0xffffffffu, y[0], 4);
          if (CPL == 8 || !(lane & 4)) *aux = y[0];
        }
      } else {
        f32x2 d2[CPL];
#pragma unroll
        for (int c = 0; c < CPL; ++c) d2[c] = pair(x[c], x[c]);
#pragma unroll
        for (int i = 0; i < I; ++i) {
          const F4 q = lds4(qr + 32 * i);
#pragma unroll
          for (int c = 0; c < CPL; ++c) {
            S.v[i][0][c] = fma2(q.a, d2[c], S.v[i][0][c]);
            S.v[i][1][c] = fma2(q.b, d2[c], S.v[i][1][c]);
            acc[c] = fma2(S.v[i][0][c], k[i].a, acc[c]);
            acc[c] = fma2(S.v[i][1][c], k[i].b, acc[c]);
          }
        }
        float dw[CPL], dr[CPL];
        column_sums(acc, dw);
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
          dr[c] = beta * dw[c];
          d2[c] = pair(-dr[c], -dr[c]);
        }
        if (rg < CPL / 4)
          *reinterpret_cast<float4*>(out) =
              CPL == 8 && rg ? make_float4(dr[CPL - 4], dr[CPL - 3], dr[CPL - 2], dr[CPL - 1]) : make_float4(dr[0], dr[1], dr[2], dr[3]);
#pragma unroll
        for (int i = 0; i < I; ++i) {
          const F4 a = lds4(ar + 32 * i);
#pragma unroll
          for (int c = 0; c < CPL; ++c) {
            S.v[i][0][c] = mul2(fma2(k[i].a, d2[c], S.v[i][0][c]), a.a);
            S.v[i][1][c] = mul2(fma2(k[i].b, d2[c], S.v[i][1][c]), a.b);
          }
        }
        // dbeta over 16 columns: four lanes, and with eight columns a lane two groups of them
#pragma unroll
        for (int m = 0; m < CPL / 4; ++m) {
          float pb = dot4(make_float4(dw[4 * m], dw[4 * m + 1], dw[4 * m + 2], dw[4 * m + 3]), *reinterpret_cast<const float4*>(&s.y[b][j][lcol + 16 * m]));
          pb += __shfl_xor_sync(0xffffffffu, pb, 1);
          pb += __shfl_xor_sync(0xffffffffu, pb, 2);
          if (lane == 0) aux[m] = pb;
        }
      }
    }
  }
  float* const end = FWD ? p.ht : p.dh0;
  if (end) S.store(end + sbase, rg, V);
}

// ---------------------------------------------------------------------------------------------------------------------
// the middle: 32 tokens of ROWS rows of a state
// ---------------------------------------------------------------------------------------------------------------------
template <int K, int V>
struct Mid {
  static constexpr int LPR = V / 8;                          // lanes along a row, 8 columns each: 4 l + 4 LPR m + (0..3), m < 2
  static constexpr int RPW = 4 * (32 / LPR);                 // rows per warp, four per lane
  static constexpr int NW = K / RPW < 4 ? K / RPW : 4;       // warps
  static constexpr int ROWS = NW * RPW, SLICES = K / ROWS, NT = 32 * NW;
  static constexpr int RP = ROWS + 8;                        // padded row of a token's values: the sums of four tokens go to different banks
  struct Smem {
    float w[TC][V];              // r, then beta r
    float d_o[TC][V];
    float dr[TC][V];             // beta dw, then -beta dw
    float q[TC][RP];             // scale q^, then dq^
    float k[TC][RP];             // k^, then dk^
    float a[TC][RP];             // exp g, then dg
    float wdo[TC];               // <w, do>
    float beta[TC];
    uint32_t tmem_slot;
    int n;
  };
};

template <int K, int V>
__global__ void __launch_bounds__(Mid<K, V>::NT, 2) kda_recurrent_mid_kernel(const TrainParams p) {
  chain_point();
  using M = Mid<K, V>;
  constexpr int NT = M::NT, ROWS = M::ROWS, LPR = M::LPR;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  typename M::Smem& s = *reinterpret_cast<typename M::Smem*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int slice = blockIdx.x % M::SLICES, h = blockIdx.x / M::SLICES % p.HL, hq = h / (p.H / p.HQ);
  const long long slot = blockIdx.x / M::SLICES / p.HL;
  if (tid == 0) {      // the last sequence whose first slot is not behind this one
    int lo = 0, hi = p.N - 1;
    while (lo < hi) {
      const int m = (lo + hi + 1) >> 1;
      if (seq_start(p, m) / TC + m <= slot) lo = m;
      else hi = m - 1;
    }
    s.n = lo;
  }
  __syncthreads();
  const int n = s.n;
  const Seq sq = sequence(p, n);
  const long long c = slot - (sq.bos / TC + n);
  if (c < 0 || c * TC >= sq.len) return;
  const int cnt = static_cast<int>(min(static_cast<long long>(TC), sq.len - c * TC));
  const size_t tok0 = static_cast<size_t>(sq.bos + c * TC);
  // the last four tokens that hold any: a short piece is not walked to its 32nd token (64 sequences of one token x 32 heads: 557 -> 148 us)
  const int last = (cnt - 1) >> 2, rows = 4 * last + 4;

  // Tensor memory holds the states between: this thread's part of the state in front of tokens 0, 4, .. 24, 32 words each (the fp32 values themselves)
  if (warp == 0) umma::tmem_alloc(&s.tmem_slot, 256);
  // ---- this thread's eight columns of four rows of S and dS; the tokens' rows -------------------------------------------------------
  const int l = lane % LPR, lrow = warp * M::RPW + 4 * (lane / LPR);
  using Tile = f32x2[4][4];      // [row][pair of columns]
  auto load_state = [&](Tile& x, const float* base, size_t index, int heads) {      // of [..][heads][K][V]; no base: zeros
    const float* const from = base + ((index * heads + h) * K + slice * ROWS + lrow) * V + 4 * l;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const F4 y = base ? lds4(from + i * V + 4 * LPR * m) : F4{0ull, 0ull};
        x[i][2 * m] = y.a;
        x[i][2 * m + 1] = y.b;
      }
  };
  for (int i = tid; i < rows * (V / 4); i += NT) {
    const int t = i / (V / 4), cc = 4 * (i % (V / 4));
    const bool ok = t < cnt;
    const size_t tok = tok0 + (ok ? t : 0), row = (tok * p.H + h) * V + cc;
    cp_async16(&s.w[t][cc], p.resid + (tok * p.HS + h) * V + cc, ok);
    cp_async16(&s.d_o[t][cc], p.d_o + row, ok);
    cp_async16(&s.dr[t][cc], p.dv + row, ok);
  }
  cp_async_commit();
  if (tid < TC) s.beta[tid] = tid < cnt ? p.beta[(tok0 + tid) * p.H + h] : 0.f;
  Tile dS, S;
  // a sequence's own ends are where the caller has them: short sequences move no other states
  const bool head = c == 0, tail = (c + 1) * TC >= sq.len;
  load_state(S, head ? p.h0 : p.ckpt, head ? static_cast<size_t>(n) : static_cast<size_t>(sq.bos / TC + c - 1), head ? p.H : p.HS);
  load_state(dS, tail ? p.d_ht : p.dckpt, tail ? static_cast<size_t>(n) : static_cast<size_t>(sq.bos / TC + c), tail ? p.H : p.HW);
  for (int i = tid; i < rows * ROWS; i += NT) {      // tokens beyond the sequence leave S and dS as they are
    const int t = i / ROWS, row = i % ROWS;
    const bool ok = t < cnt;
    const size_t tok = tok0 + (ok ? t : 0), rq = (tok * p.HQ + hq) * K + slice * ROWS + row, rv = tok * p.H + h;
    float2 r = make_float2(1.f, 1.f);
    if (p.use_l2) r = *reinterpret_cast<const float2*>(p.norms + 2 * (tok * p.HS + h));
    s.q[t][row] = ok ? p.q[rq] * (p.scale * r.x) : 0.f;
    s.k[t][row] = ok ? p.k[rq] * r.y : 0.f;
    s.a[t][row] = ok ? expf(p.g[rv * K + slice * ROWS + row]) : 1.f;
  }
  if (slice == 0 && tid < cnt) {
    const float* const part = p.dbp + ((tok0 + tid) * p.HW + h) * (V / 16);
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < V / 16; ++i) sum += part[i];
    p.dbeta[(tok0 + tid) * p.H + h] = sum;
  }
  cp_async_wait<0>();
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tq = __shfl_sync(0xffffffffu, s.tmem_slot, 0) + (static_cast<uint32_t>(32 * warp) << 16);      // this warp's lanes
  for (int t = warp; t < rows; t += M::NW) {
    constexpr int E = V / 32;
    float w[E], d[E], dot = 0.f;
    row_get<E>(w, &s.w[t][lane * E]);
    row_get<E>(d, &s.d_o[t][lane * E]);
#pragma unroll
    for (int e = 0; e < E; ++e) {
      w[e] *= s.beta[t];
      dot += w[e] * d[e];
    }
    row_put<E>(&s.w[t][lane * E], w);
    row_get<E>(w, &s.dr[t][lane * E]);
#pragma unroll
    for (int e = 0; e < E; ++e) w[e] = -w[e];
    row_put<E>(&s.dr[t][lane * E], w);
    dot = warp_sum(dot);
    if (lane == 0) s.wdo[t] = dot;
  }
  __syncthreads();

  auto rows4 = [&](const float (&x)[TC][M::RP], int t, float (&y)[4]) {      // a token's values of this thread's rows
    const float4 z = *reinterpret_cast<const float4*>(&x[t][lrow]);
    y[0] = z.x; y[1] = z.y; y[2] = z.z; y[3] = z.w;
  };
  auto step = [&](Tile& to, const Tile& from, int t) {      // `from` is S' of token t: S' + k w^T
    float k[4];
    rows4(s.k, t, k);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const F4 w = lds4(&s.w[t][4 * l + 4 * LPR * m]);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const f32x2 k2 = pair(k[i], k[i]);
        to[i][2 * m] = fma2(k2, w.a, from[i][2 * m]);
        to[i][2 * m + 1] = fma2(k2, w.b, from[i][2 * m + 1]);
      }
    }
  };
  auto decay = [&](Tile& to, const Tile& from, int t) {
    float a[4];
    rows4(s.a, t, a);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const f32x2 a2 = pair(a[i], a[i]);
#pragma unroll
      for (int m = 0; m < 4; ++m) to[i][m] = mul2(from[i][m], a2);
    }
  };
  auto step4 = [&](int t) {      // S over four tokens
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      decay(S, S, t + j);
      step(S, S, t + j);
    }
  };
  auto keep = [&](int slot) {
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      float x[16];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float2 y = halves(S[2 * m + (i >> 2)][i & 3]);
        x[2 * i] = y.x;
        x[2 * i + 1] = y.y;
      }
      umma::tmem_st16(tq + 32 * slot + 16 * m, x);
    }
  };
  auto fetch = [&](int slot) {
    float x[2][16];
    umma::tmem_ld16(tq + 32 * slot, x[0]);
    umma::tmem_ld16(tq + 32 * slot + 16, x[1]);
    umma::tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 16; ++i) S[i >> 2][i & 3] = pair(x[i >> 3][2 * (i & 7)], x[i >> 3][2 * (i & 7) + 1]);
  };
#pragma unroll 1
  for (int i = 0; i < last; ++i) {
    keep(i);
    step4(4 * i);
  }
  umma::tmem_st_wait();
#pragma unroll 1
  for (int half = last; half >= 0; --half) {      // four tokens each, the last first
    const int t0 = 4 * half;
    if (half < last) fetch(half);
    Tile Sp[4];      // S' of the four tokens
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      decay(Sp[j], S, t0 + j);
      if (j < 3) step(S, Sp[j], t0 + j);
    }
    // sums of the lane's 8 columns, folded over the lanes of a row: first the four rows (one per lane pair), then the tokens
    float part[4][3];
    constexpr int R1 = LPR / 2, R2 = LPR / 4;      // lane bits that pick the row
#pragma unroll
    for (int j = 3; j >= 0; --j) {
      const int t = t0 + j;
      float q[4], k[4], a[4];
      rows4(s.q, t, q);
      rows4(s.k, t, k);
      rows4(s.a, t, a);
      f32x2 pq[4], pk[4], pg[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) pq[i] = pk[i] = pg[i] = 0ull;
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int cc = 4 * l + 4 * LPR * m;
        const F4 d = lds4(&s.d_o[t][cc]), w = lds4(&s.w[t][cc]), r = lds4(&s.dr[t][cc]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const f32x2 q2 = pair(q[i], q[i]), k2 = pair(k[i], k[i]), a2 = pair(a[i], a[i]);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const f32x2 x = Sp[j][i][2 * m + e], dd = e ? d.b : d.a, ww = e ? w.b : w.a, rr = e ? r.b : r.a;
            f32x2 y = fma2(q2, dd, dS[i][2 * m + e]);      // dS_t
            pq[i] = fma2(x, dd, pq[i]);
            pk[i] = fma2(y, ww, pk[i]);
            pk[i] = fma2(x, rr, pk[i]);
            y = fma2(k2, rr, y);                            // dS'
            pg[i] = fma2(x, y, pg[i]);
            dS[i][2 * m + e] = mul2(y, a2);
          }
        }
      }
      float sum[4][3];
      const float wdo = s.wdo[t];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 hq2 = halves(pq[i]), hk2 = halves(pk[i]), hg2 = halves(pg[i]);
        sum[i][0] = hq2.x + hq2.y;
        sum[i][1] = hk2.x + hk2.y;
        sum[i][2] = hg2.x + hg2.y;
        if (l == 0) sum[i][0] = fmaf(k[i], wdo, sum[i][0]);      // S_t do = S' do + k <w, do>
      }
#pragma unroll
      for (int i = 0; i < 3; ++i)
        part[j][i] = fold(fold(sum[0][i], sum[2][i], R1, lane), fold(sum[1][i], sum[3][i], R1, lane), R2, lane);
    }
    const int row = lrow + 2 * ((lane & R1) != 0) + ((lane & R2) != 0);
    auto put = [&](int t, float x, float y, float z) {      // over the tokens' q, k, exp g of these rows, which the whole warp is done with
      s.q[t][row] = x;
      s.k[t][row] = y;
      s.a[t][row] = z;
    };
    if constexpr (LPR == 16) {
      float x[3];
#pragma unroll
      for (int i = 0; i < 3; ++i)
        x[i] = fold(fold(part[0][i], part[2][i], 2, lane), fold(part[1][i], part[3][i], 2, lane), 1, lane);
      put(t0 + (lane & 3), x[0], x[1], x[2]);
    } else if constexpr (LPR == 8) {
      float x[2][3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        x[0][i] = fold(part[0][i], part[2][i], 1, lane);
        x[1][i] = fold(part[1][i], part[3][i], 1, lane);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) put(t0 + 2 * (lane & 1) + j, x[j][0], x[j][1], x[j][2]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) put(t0 + j, part[j][0], part[j][1], part[j][2]);
    }
    __syncwarp();
  }
  umma::fence_before_sync();
  __syncthreads();
  for (int i = tid; i < cnt * ROWS; i += NT) {
    const int t = i / ROWS, row = i % ROWS;
    const int at = slice * ROWS + row;
    const size_t o = ((tok0 + t) * p.HD + h) * K + at;
    p.dqh[o] = s.q[t][row] * p.dq_scale;
    p.dkh[o] = s.k[t][row];
    p.dg[((tok0 + t) * p.H + h) * K + at] = s.a[t][row];
  }
  if (warp == 0) umma::tmem_dealloc(s.tmem_slot, 256);
}

// dq, dk from the per-value-head gradients w.r.t. the rows the recurrence saw: sum over the value heads of a group,
// scale (q only), then the backward of x^ = x rsqrt(sum x^2 + eps) when the rows were normalised.  One warp per row.
template <int K>
__global__ void __launch_bounds__(256) kda_recurrent_bwd_finish_kernel(const TrainParams p, float* __restrict__ dq, float* __restrict__ dk,
                                                                       long long rows) {
  chain_point();
  constexpr int E = K / 32;
  const long long item = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);      // token, q head of this launch
  const int lane = threadIdx.x & 31;
  if (item >= rows) return;
  const int grp = p.H / p.HQ, heads = p.HL / grp;
  const long long tok = item / heads;
  const int hq = static_cast<int>(item % heads);
  const long long row = tok * p.HQ + hq;
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    const float* x = (which ? p.k : p.q) + row * K + lane * E;
    const float* src = (which ? p.dkh : p.dqh) + (tok * p.HD + static_cast<long long>(hq) * grp) * K + lane * E;
    float d[E], xf[E];
    float ss = 0.f;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      float acc = 0.f;
      for (int j = 0; j < grp; ++j) acc += src[static_cast<size_t>(j) * K + e];
      d[e] = which ? acc : acc * p.scale;
      xf[e] = x[e];
      ss += xf[e] * xf[e];
    }
    if (p.use_l2) {
      const float rs = rsqrtf(warp_sum(ss) + L2NORM_EPS);
      float dot = 0.f;
#pragma unroll
      for (int e = 0; e < E; ++e) dot += xf[e] * rs * d[e];
      dot = warp_sum(dot);
#pragma unroll
      for (int e = 0; e < E; ++e) d[e] = rs * (d[e] - xf[e] * rs * dot);
    }
    float* out = (which ? dk : dq) + row * K + lane * E;
#pragma unroll
    for (int e = 0; e < E; ++e) out[e] = d[e];
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// buffers and launches
// ---------------------------------------------------------------------------------------------------------------------
size_t up256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }
size_t kept_states(int64_t tokens) { return static_cast<size_t>(tokens) / TC; }

struct SavedLayout {      // what the forward leaves for the backward
  size_t ckpt, resid, norms, total;
};
SavedLayout saved_layout(int64_t tokens, int H, int K, int V, bool l2) {
  SavedLayout l{};
  size_t off = 0;
  l.ckpt = off; off = up256(off + kept_states(tokens) * H * K * V * 4);
  l.resid = off; off = up256(off + static_cast<size_t>(tokens) * H * V * 4);
  l.norms = off; off = up256(off + (l2 ? static_cast<size_t>(tokens) * H * 2 * 4 : 0));
  l.total = off;
  return l;
}
struct WorkLayout {      // the backward's scratch; a replaying backward's continues with a SavedLayout
  size_t dqh, dkh, dckpt, dbp, h0, d_ht, total;
};
// What a call does without: dq^, dk^ when they are dq, dk; copies of h0 and d_ht, which the last kernel still reads, unless dh0 overwrites them
struct Skip { bool dqk, h0, d_ht; };
WorkLayout work_layout(int64_t tokens, int N, int H, int all_heads, int K, int V, const Skip& skip) {
  WorkLayout l{};
  size_t off = 0;
  const size_t rows = skip.dqk ? 0 : static_cast<size_t>(tokens) * H * K * 4, states = static_cast<size_t>(N) * all_heads * K * V * 4;
  l.dqh = off; off = up256(off + rows);
  l.dkh = off; off = up256(off + rows);
  l.dckpt = off; off = up256(off + kept_states(tokens) * H * K * V * 4);
  l.dbp = off; off = up256(off + static_cast<size_t>(tokens) * H * (V / 16) * 4);
  l.h0 = off; off = up256(off + (skip.h0 ? 0 : states));
  l.d_ht = off; off = up256(off + (skip.d_ht ? 0 : states));
  l.total = off;
  return l;
}
bool overlap(const void* a, const void* b, size_t bytes) {
  const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
  return a && b && (x < y ? y - x : x - y) < bytes;
}
size_t state_bytes(const kda_recurrent_bwd_args& a) { return static_cast<size_t>(a.N) * a.H * a.K * a.V * 4; }
Skip skips(const kda_recurrent_bwd_args& a) {
  const int HQ = a.HQ > 0 ? a.HQ : a.H;
  return {HQ == a.H && !a.use_qk_l2norm, !overlap(a.dh0, a.h0, state_bytes(a)), !overlap(a.dh0, a.d_ht, state_bytes(a))};
}
constexpr Skip NOTHING{false, false, false};

// The heads may be worked on in groups, one after another, in the scratch of one group.
int heads_of(const kda_recurrent_bwd_args& a, int passes) {      // value heads a pass, evened out; whole groups of value heads
  const int HQ = a.HQ > 0 ? a.HQ : a.H;
  return (HQ + passes - 1) / passes * (a.H / HQ);
}
size_t scratch_bytes(const kda_recurrent_bwd_args& a, int heads, bool with_saved) {
  return work_layout(a.tokens, a.N, heads, a.H, a.K, a.V, skips(a)).total + (with_saved ? 0 : saved_layout(a.tokens, heads, a.K, a.V, a.use_qk_l2norm != 0).total);
}
// the fewest passes whose scratch `bytes` holds; 0: not even one group fits
int heads_per_pass(const kda_recurrent_bwd_args& a, bool with_saved, size_t bytes) {
  for (int passes = 1; passes <= (a.HQ > 0 ? a.HQ : a.H); ++passes)
    if (scratch_bytes(a, heads_of(a, passes), with_saved) <= bytes) return heads_of(a, passes);
  return 0;
}
bool head_size_ok(int d) { return d == 32 || d == 64 || d == 128; }
void use_saved(TrainParams& p, void* saved, const SavedLayout& l) {
  unsigned char* const b = static_cast<unsigned char*>(saved);
  p.ckpt = reinterpret_cast<float*>(b + l.ckpt);
  p.resid = reinterpret_cast<float*>(b + l.resid);
  p.norms = reinterpret_cast<float*>(b + l.norms);
}
int wide(const void* q, const void* k, const void* g) {
  return ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(g)) & 15) == 0;
}

template <int K, int CPL, bool FWD>
int launch_walk(const TrainParams& p, bool first, cudaStream_t st) {
  static DeviceOnce once;
  const auto kernel = kda_recurrent_walk_kernel<K, CPL, FWD>;
  const int smem = static_cast<int>(sizeof(WalkSmem<K, CPL>));
  const int rc = once.run([&] { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); });
  if (rc != KDA_OK) return rc;
  const int cols = std::min(p.V, WalkSmem<K, CPL>::COLS);
  const long long grid = static_cast<long long>(p.N) * p.HL * (p.V / cols);
  if (grid > 0x7fffffffLL) return KDA_E_SHAPE;
  const unsigned threads = static_cast<unsigned>(cols / (4 * CPL) * 32);
  if (!first) return static_cast<int>(launch_chained(kernel, static_cast<unsigned>(grid), threads, smem, st, p));
  kernel<<<static_cast<unsigned>(grid), threads, smem, st>>>(p);
  return static_cast<int>(cudaGetLastError());
}
// 32 columns a warp read a row of q, k, exp g for 128 state values instead of 64, and two warps a scheduler are enough to keep the FP32
// pipe fed; while there are fewer than that, more and narrower warps shorten the chain.  Both add up in the same order
bool wide_slices(const TrainParams& p) { return static_cast<long long>(p.N) * p.HL * p.V > 32LL * 4 * sm_count(); }
template <bool FWD>
int launch_walk(const TrainParams& p, int K, bool first, cudaStream_t st) {
  const bool w = wide_slices(p);
  switch (K) {
    case 32: return w ? launch_walk<32, 8, FWD>(p, first, st) : launch_walk<32, 4, FWD>(p, first, st);
    case 64: return w ? launch_walk<64, 8, FWD>(p, first, st) : launch_walk<64, 4, FWD>(p, first, st);
    default: return w ? launch_walk<128, 8, FWD>(p, first, st) : launch_walk<128, 4, FWD>(p, first, st);
  }
}
template <int K, int V>
int launch_mid(const TrainParams& p, cudaStream_t st) {
  static DeviceOnce once;
  const auto kernel = kda_recurrent_mid_kernel<K, V>;
  const int smem = static_cast<int>(sizeof(typename Mid<K, V>::Smem));
  const int rc = once.run([&] { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); });
  if (rc != KDA_OK) return rc;
  const long long grid = p.slots * p.HL * Mid<K, V>::SLICES;
  if (grid > 0x7fffffffLL) return KDA_E_SHAPE;
  return static_cast<int>(launch_chained(kernel, static_cast<unsigned>(grid), Mid<K, V>::NT, smem, st, p));
}
template <int K>
int launch_mid(const TrainParams& p, cudaStream_t st) {
  switch (p.V) {
    case 32: return launch_mid<K, 32>(p, st);
    case 64: return launch_mid<K, 64>(p, st);
    default: return launch_mid<K, 128>(p, st);
  }
}
template <int K>
int launch_finish(const TrainParams& p, float* dq, float* dk, long long rows, cudaStream_t st) {
  return static_cast<int>(launch_chained(kda_recurrent_bwd_finish_kernel<K>, static_cast<unsigned>((rows + 7) / 8), 256, 0, st, p, dq, dk, rows));
}

int check_backward(const kda_recurrent_bwd_args* a) {
  if (!a) return KDA_E_NULL;
  if (!a->q || !a->k || !a->v || !a->g || !a->beta || !a->d_o || !a->dq || !a->dk || !a->dv || !a->dg || !a->dbeta || !a->workspace)
    return KDA_E_NULL;
  if (a->io_dtype != KDA_FP32) return KDA_E_DTYPE;
  if (a->N < 0 || a->H <= 0 || a->tokens < 0 || (!a->cu_seqlens && a->T < 0)) return KDA_E_SHAPE;
  if (!head_size_ok(a->K) || !head_size_ok(a->V)) return KDA_E_SHAPE;
  if (a->H % (a->HQ > 0 ? a->HQ : a->H)) return KDA_E_SHAPE;
  return KDA_OK;
}

// saved == NULL: the forward walk runs here first, into the end of the workspace
int backward(const kda_recurrent_bwd_args* a, const void* saved, size_t saved_bytes, void* stream) {
  const bool with_saved = saved != nullptr;
  const int HQ = a->HQ > 0 ? a->HQ : a->H, grp = a->H / HQ, K = a->K, V = a->V;
  const Skip skip = skips(*a);
  const int most = heads_per_pass(*a, with_saved, a->workspace_bytes);
  if (!most) return KDA_E_WORKSPACE;
  if (with_saved && saved_bytes < saved_layout(a->tokens, a->H, K, V, true).total) return KDA_E_WORKSPACE;
  if ((reinterpret_cast<uintptr_t>(a->workspace) | reinterpret_cast<uintptr_t>(saved)) & 255) return KDA_E_ALIGN;
  const void* sixteen[] = {a->v, a->h0, a->d_o, a->d_ht, a->dv, a->dh0};      // 16-byte loads and stores
  for (const void* p : sixteen)
    if (reinterpret_cast<uintptr_t>(p) & 15) return KDA_E_ALIGN;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (a->N == 0) return KDA_OK;
  if (a->tokens == 0) {      // empty sequences: the initial state is the final state
    if (!a->dh0) return KDA_OK;
    return static_cast<int>(a->d_ht ? cudaMemcpyAsync(a->dh0, a->d_ht, state_bytes(*a), cudaMemcpyDeviceToDevice, st)
                                    : cudaMemsetAsync(a->dh0, 0, state_bytes(*a), st));
  }
  if (!a->cu_seqlens && static_cast<int64_t>(a->N) * a->T != a->tokens) return KDA_E_SHAPE;
  unsigned char* const ws = static_cast<unsigned char*>(a->workspace);
  const WorkLayout l = work_layout(a->tokens, a->N, most, a->H, K, V, skip);
  const float *h0 = a->h0, *d_ht = a->d_ht;
  int rc = KDA_OK;
  auto keep = [&](bool not_needed, const float*& x, size_t at) {
    if (not_needed || rc != KDA_OK) return;
    rc = static_cast<int>(cudaMemcpyAsync(ws + at, x, state_bytes(*a), cudaMemcpyDeviceToDevice, st));
    x = reinterpret_cast<const float*>(ws + at);
  };
  keep(skip.h0, h0, l.h0);
  keep(skip.d_ht, d_ht, l.d_ht);
  for (int h = 0; h < a->H && rc == KDA_OK; h += most) {
    TrainParams p{};
    p.N = a->N; p.H = a->H; p.HQ = HQ; p.V = V; p.T = a->T; p.slots = a->tokens / TC + a->N; p.cu = a->cu_seqlens;
    p.HL = std::min(most, a->H - h); p.HS = with_saved ? a->H : p.HL; p.HW = p.HL;
    p.use_l2 = a->use_qk_l2norm; p.scale = a->scale; p.wide = wide(a->q, a->k, a->g);
    auto from = [&](auto* x, int per_head) { return x ? x + static_cast<size_t>(h) * per_head : x; };
    const size_t qk = static_cast<size_t>(h / grp) * K;
    p.q = static_cast<const float*>(a->q) + qk; p.k = static_cast<const float*>(a->k) + qk;
    p.v = from(static_cast<const float*>(a->v), V); p.d_o = from(static_cast<const float*>(a->d_o), V); p.dv = from(static_cast<float*>(a->dv), V);
    p.g = from(a->g, K); p.dg = from(a->dg, K); p.beta = from(a->beta, 1); p.dbeta = from(a->dbeta, 1);
    p.h0 = from(h0, K * V); p.d_ht = from(d_ht, K * V); p.dh0 = from(a->dh0, K * V);
    p.dckpt = reinterpret_cast<float*>(ws + l.dckpt); p.dbp = reinterpret_cast<float*>(ws + l.dbp);
    float *const dq = static_cast<float*>(a->dq) + qk, *const dk = static_cast<float*>(a->dk) + qk;
    const bool direct = skip.dqk;      // nothing to sum or to take back: no pass of its own (0.27 ms at 8 x 2048 x 32)
    p.dqh = direct ? dq : reinterpret_cast<float*>(ws + l.dqh); p.dkh = direct ? dk : reinterpret_cast<float*>(ws + l.dkh);
    p.HD = direct ? a->H : p.HL;
    p.dq_scale = direct ? p.scale : 1.f;
    if (with_saved) {
      use_saved(p, const_cast<void*>(saved), saved_layout(a->tokens, a->H, K, V, true));
      p.ckpt = from(p.ckpt, K * V); p.resid = from(p.resid, V); p.norms = from(p.norms, 2);
    } else {
      use_saved(p, ws + l.total, saved_layout(a->tokens, most, K, V, p.use_l2 != 0));
      rc = launch_walk<true>(p, K, h == 0, st);
    }
    if (rc == KDA_OK) rc = launch_walk<false>(p, K, with_saved && h == 0, st);
    if (rc == KDA_OK) rc = K == 32 ? launch_mid<32>(p, st) : (K == 64 ? launch_mid<64>(p, st) : launch_mid<128>(p, st));
    const long long rows = a->tokens * (p.HL / grp);
    if (rc == KDA_OK && !direct)
      rc = K == 32 ? launch_finish<32>(p, dq, dk, rows, st) : (K == 64 ? launch_finish<64>(p, dq, dk, rows, st) : launch_finish<128>(p, dq, dk, rows, st));
  }
  return rc;
}

}  // namespace

}  // namespace kda

using namespace kda;

extern "C" size_t kda_recurrent_saved_bytes(int64_t tokens, int32_t N, int32_t H, int32_t K, int32_t V) {
  if (tokens < 0 || N < 0 || H <= 0 || K <= 0 || V <= 0) return 0;
  return saved_layout(tokens, H, K, V, true).total;
}

// (an upper bound over all options; kda_recurrent_bwd_scratch_bytes knows them)
extern "C" size_t kda_recurrent_bwd_workspace_bytes(int64_t tokens, int32_t N, int32_t H, int32_t K, int32_t V) {
  if (tokens < 0 || N < 0 || H <= 0 || K <= 0 || V <= 0) return 0;
  return work_layout(tokens, N, H, H, K, V, NOTHING).total + saved_layout(tokens, H, K, V, true).total;
}

extern "C" size_t kda_recurrent_bwd_scratch_bytes(const kda_recurrent_bwd_args* a, int32_t with_saved, int32_t passes) {
  if (!a || a->tokens < 0 || a->N < 0 || a->H <= 0 || !head_size_ok(a->K) || !head_size_ok(a->V)) return 0;
  const int HQ = a->HQ > 0 ? a->HQ : a->H;
  if (a->H % HQ) return 0;
  return scratch_bytes(*a, heads_of(*a, std::max(1, std::min(passes, HQ))), with_saved != 0);
}

// the forward walk; with_saved: leaves what a backward then need not compute again
static int forward(const kda_recurrent_args* a, void* saved, size_t saved_bytes, bool with_saved, void* stream) {
  if (!a) return KDA_E_NULL;
  if (a->N < 0 || a->H <= 0 || a->tokens < 0 || (!a->cu_seqlens && a->T < 0)) return KDA_E_SHAPE;
  if (!head_size_ok(a->K) || !head_size_ok(a->V)) return KDA_E_SHAPE;
  const int HQ = a->HQ > 0 ? a->HQ : a->H;
  if (a->HQ < 0 || a->H % HQ) return KDA_E_SHAPE;
  // whole sequences, activated gates, [K, V] states
  if (a->state_indices || a->num_accepted_tokens || a->transpose_state || a->A_log || a->beta_sigmoid || (a->ht && a->ht == a->h0)) return KDA_E_SHAPE;
  if (a->N == 0 || a->tokens == 0) return kda_recurrent_fwd(a, stream);      // nothing to walk: the final state is the initial one
  if (!a->q || !a->k || !a->v || !a->g || !a->beta || !a->o || (with_saved && !saved)) return KDA_E_NULL;
  if (a->io_dtype != KDA_FP32) return KDA_E_DTYPE;
  if (!a->cu_seqlens && static_cast<int64_t>(a->N) * a->T != a->tokens) return KDA_E_SHAPE;
  const SavedLayout sl = saved_layout(a->tokens, a->H, a->K, a->V, true);
  if (with_saved && saved_bytes < sl.total) return KDA_E_WORKSPACE;
  if (reinterpret_cast<uintptr_t>(saved) & 255) return KDA_E_ALIGN;
  const void* sixteen[] = {a->q, a->k, a->v, a->g, a->o, a->h0, a->ht};      // as kda_recurrent_fwd
  for (const void* p : sixteen)
    if (reinterpret_cast<uintptr_t>(p) & 15) return KDA_E_ALIGN;
  TrainParams p{};
  p.q = static_cast<const float*>(a->q); p.k = static_cast<const float*>(a->k); p.v = static_cast<const float*>(a->v);
  p.g = a->g; p.beta = a->beta; p.h0 = a->h0; p.ht = a->ht; p.o = static_cast<float*>(a->o);
  p.cu = a->cu_seqlens;
  p.T = a->T;
  p.N = a->N; p.H = p.HL = p.HS = a->H; p.HQ = HQ; p.V = a->V; p.use_l2 = a->use_qk_l2norm; p.scale = a->scale;
  p.wide = wide(a->q, a->k, a->g);
  if (with_saved) use_saved(p, saved, sl);
  return launch_walk<true>(p, a->K, true, static_cast<cudaStream_t>(stream));
}

extern "C" int kda_recurrent_train_fwd(const kda_recurrent_args* args, void* saved, size_t saved_bytes, void* stream) {
  return forward(args, saved, saved_bytes, true, stream);
}

extern "C" int kda_recurrent_walk_fwd(const kda_recurrent_args* args, void* stream) { return forward(args, nullptr, 0, false, stream); }

extern "C" int kda_recurrent_bwd_scratch(const kda_recurrent_bwd_args* args, const void* saved, size_t saved_bytes, void* stream) {
  const int rc = check_backward(args);
  return rc != KDA_OK ? rc : backward(args, saved, saved_bytes, stream);
}

extern "C" int kda_recurrent_bwd(const kda_recurrent_bwd_args* args, void* stream) {
  const int rc = check_backward(args);
  if (rc != KDA_OK) return rc;
  if (args->workspace_bytes < kda_recurrent_bwd_workspace_bytes(args->tokens, args->N, args->H, args->K, args->V)) return KDA_E_WORKSPACE;
  return backward(args, nullptr, 0, stream);
}

extern "C" int kda_recurrent_train_bwd(const kda_recurrent_bwd_args* args, const void* saved, size_t saved_bytes, void* stream) {
  const int rc = check_backward(args);
  if (rc != KDA_OK) return rc;
  if (!saved) return KDA_E_NULL;
  if (args->workspace_bytes < work_layout(args->tokens, args->N, args->H, args->H, args->K, args->V, NOTHING).total) return KDA_E_WORKSPACE;
  return backward(args, saved, saved_bytes, stream);
}
