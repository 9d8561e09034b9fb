// float32 chunked forward: per-chunk preparation and state scan, every product in float32 accuracy on the tensor cores (kda_fp32.cuh).
//
// Replaces the token-recurrent pair of kernels for calls with gradients and for long forward-only calls: those walk a (sequence,
// head) token by token on CUDA cores (1.8 us a token forward, 11 us backward), this one 64 tokens at a time.  8 x 2048 tokens x 32
// heads: preparation 1.24 ms, scan 0.7; forward and backward 26.0 -> 5.2.  What bounds it is the operands' way into shared
// memory (split in two TF32 parts, swizzled stores), one CTA per SM with its phases in a row.
#include "kda_device.cuh"
#include "kda_fp32.cuh"

namespace kda {

using namespace f32;

namespace {

// =================================================================================================
// preparation
// =================================================================================================
// One CTA per (chunk, head); a thread owns four key columns of four rows (a warp whole rows) and keeps their q, k and lam = e^g in
// registers.  Decays are running products of lam (all factors <= 1) and the intra-chunk products come in levels 16, 8, 4 and
// pairwise 4 x 4 blocks exactly as in kda_chunk_prepare.cu; here levels 8 and 4 form one product (128 x 64), level 16 another one
// (96 x 96: the q and k rows of blocks 1..3 against the columns as each of those blocks sees them), of which the matching blocks
// are read.
constexpr int AS = 68, DS = 20;
constexpr uint32_t S96 = 96 * 128;

struct PrepSmem32 {
  unsigned char R[196608];        // operand tiles, see the phases
  float A[C * AS];                // raw Akk, then beta Akk, then Tm
  union {
    float T[16][KD];              // decay over every four rows
    float X[32 * 33];             // scratch of the block merges
  };
  float TB[4][KD];                // decay over every 16-row block
  float beta[C];
  uint64_t bar;
  uint32_t tmem;
};
constexpr int PREP32_SMEM = static_cast<int>(sizeof(PrepSmem32)) + 1024;
static_assert(PREP32_SMEM <= 227 * 1024, "PrepSmem32 too large");

__device__ __forceinline__ float4 mulv(const float4 a, const float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float dotv(const float4 a, const float4 b) { return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, a.x * b.x))); }
__device__ __forceinline__ float4 lds4v(const float* p) { return *reinterpret_cast<const float4*>(p); }

}  // namespace

__global__ void __launch_bounds__(NT, 1) kda_f32_prepare_kernel(const F32Params p) {
  chain_point();
  extern __shared__ unsigned char smem_raw[];
  PrepSmem32& s = *reinterpret_cast<PrepSmem32*>(smem_raw + pad_to_1024(smem_raw));
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int c = blockIdx.x / p.H, h = blockIdx.x % p.H;
  if (p.clear_status && blockIdx.x == 0 && tid < 4) p.w.status[tid] = 0u;
  if (c >= p.map.total()) return;
  const ChunkInfo ci = p.map.info(c);
  const int len = ci.len;
  const size_t tile = blockIdx.x;
  const int blk = warp >> 2, quad = warp & 3, kk = 4 * lane, t0 = 4 * warp;
  float* const gAQK = p.w.AQK + tile * C * C;

  if (tid == 0) {
    mbar_init(&s.bar, 1);
    fence_mbar_init();
  }
  __syncwarp();
  if (warp == 0) umma::tmem_alloc(&s.tmem, 256);
  float4 q[4], k[4], lam[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const bool ok = t0 + i < len && kk < p.kc;
    const size_t tok = static_cast<size_t>(ci.tok0 + t0 + i);
    lam[i] = ld4(p.g + (tok * p.H + h) * p.kc + kk, ok);
    q[i] = ld4(p.q + (tok * p.HQ + h / p.grp) * p.kc + kk, ok);
    k[i] = ld4(p.k + (tok * p.HQ + h / p.grp) * p.kc + kk, ok);
  }
  if (tid < C) s.beta[tid] = tid < len ? __ldg(p.beta + static_cast<size_t>(ci.tok0 + tid) * p.H + h) : 0.f;
  for (int i = tid; i < C * AS / 4; i += NT) reinterpret_cast<float4*>(s.A)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int i = tid; i < C * C / 4; i += NT) reinterpret_cast<float4*>(gAQK)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int i = 0; i < 4; ++i) lam[i] = make_float4(expf(lam[i].x), expf(lam[i].y), expf(lam[i].z), expf(lam[i].w));
  *reinterpret_cast<float4*>(&s.T[warp][kk]) = mulv(mulv(lam[0], lam[1]), mulv(lam[2], lam[3]));
  if (p.use_l2) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      q[i] = mul4(rsqrtf(warp_sum(dotv(q[i], q[i])) + L2NORM_EPS), q[i]);
      k[i] = mul4(rsqrtf(warp_sum(dotv(k[i], k[i])) + L2NORM_EPS), k[i]);
      if (p.save) {
        *reinterpret_cast<float4*>(p.w.QN + tile * C * KD + static_cast<size_t>(t0 + i) * KD + kk) = q[i];
        *reinterpret_cast<float4*>(p.w.KN + tile * C * KD + static_cast<size_t>(t0 + i) * KD + kk) = k[i];
      }
    }
  }
  umma::fence_before_sync();
  __syncthreads();      // T; A, AQK are cleared; tensor memory is there
  umma::fence_after_sync();
  const uint32_t tb = s.tmem;
  uint32_t phase = 0;

  // ---- the 4 x 4 diagonal block of these rows pairwise
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float4 E = k[j];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      if (t < j) continue;
      if (t > j) E = mulv(E, lam[t]);
      const float aq = warp_sum(dotv(q[t], E));
      if (lane == 0) gAQK[(t0 + t) * C + t0 + j] = p.scale * aq;
      if (t > j) {
        const float ak = warp_sum(dotv(k[t], E));
        if (lane == 0) s.A[(t0 + t) * AS + t0 + j] = ak;
      }
    }
  }
  // ---- operands of levels 8 and 4: A rows 0..63 = per block q 8..15, k 8..15; 64..127 = per block q 4..7, k 4..7, q 12..15, k 12..15;
  // B rows 0..31 = per block k 0..7, 32..63 = per block k 0..3, k 8..11
  {
    unsigned char* const A = s.R + (lane >> 3) * 2 * S128;
    unsigned char* const B = s.R + 131072 + (lane >> 3) * 2 * S64;
    const int pc = lane & 7, u = quad >> 1;
    if (quad >= 2) {
      float4 f = quad == 3 ? mulv(lds4v(&s.T[warp - 1][kk]), lam[0]) : lam[0];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (i > 0) f = mulv(f, lam[i]);
        put4(A, S128, 16 * blk + 4 * (quad - 2) + i, pc, mulv(q[i], f));
        put4(A, S128, 16 * blk + 8 + 4 * (quad - 2) + i, pc, mulv(k[i], f));
      }
    } else {
      float4 f = quad == 0 ? lds4v(&s.T[warp + 1][kk]) : make_float4(1.f, 1.f, 1.f, 1.f);
#pragma unroll
      for (int j = 3; j >= 0; --j) {
        if (j < 3) f = mulv(f, lam[j + 1]);
        put4(B, S64, 8 * blk + 4 * quad + j, pc, mulv(k[j], f));
      }
    }
    if (quad & 1) {
      float4 f = lam[0];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (i > 0) f = mulv(f, lam[i]);
        put4(A, S128, 64 + 16 * blk + 8 * u + i, pc, mulv(q[i], f));
        put4(A, S128, 64 + 16 * blk + 8 * u + 4 + i, pc, mulv(k[i], f));
      }
    } else {
      float4 f = make_float4(1.f, 1.f, 1.f, 1.f);
#pragma unroll
      for (int j = 3; j >= 0; --j) {
        if (j < 3) f = mulv(f, lam[j + 1]);
        put4(B, S64, 32 + 8 * blk + 4 * u + j, pc, mulv(k[j], f));
      }
    }
  }
  if (quad == 3)
    *reinterpret_cast<float4*>(&s.TB[blk][kk]) =
        mulv(mulv(lds4v(&s.T[warp - 3][kk]), lds4v(&s.T[warp - 2][kk])), mulv(lds4v(&s.T[warp - 1][kk]), lds4v(&s.T[warp][kk])));
  staged();
  const uint32_t aR = smem_u32(s.R);
  if (tid == 0) {
#pragma unroll 1
    for (int sl = 0; sl < 4; ++sl) mma_slice(tb, aR + sl * 2 * S128, S128, aR + 131072 + sl * 2 * S64, S64, idesc(128, 64), sl > 0);
    umma::commit(&s.bar);
  }
  // ---- meanwhile: QG, KG, GL; the products of lam for the next operands
  float4 F[4], R[4], pre = make_float4(1.f, 1.f, 1.f, 1.f), post = pre;      // F = prod(block start .. i), R = prod(i+1 .. block end)
  {
    F[0] = lam[0];
    if (quad > 0) F[0] = mulv(F[0], lds4v(&s.T[4 * blk][kk]));
    if (quad > 1) F[0] = mulv(F[0], lds4v(&s.T[4 * blk + 1][kk]));
    if (quad > 2) F[0] = mulv(F[0], lds4v(&s.T[4 * blk + 2][kk]));
    R[3] = make_float4(1.f, 1.f, 1.f, 1.f);
    if (quad < 3) R[3] = lds4v(&s.T[4 * blk + 3][kk]);
    if (quad < 2) R[3] = mulv(R[3], lds4v(&s.T[4 * blk + 2][kk]));
    if (quad < 1) R[3] = mulv(R[3], lds4v(&s.T[4 * blk + 1][kk]));
#pragma unroll
    for (int i = 1; i < 4; ++i) F[i] = mulv(F[i - 1], lam[i]);
#pragma unroll
    for (int i = 2; i >= 0; --i) R[i] = mulv(R[i + 1], lam[i + 1]);
    for (int b = 0; b < blk; ++b) pre = mulv(pre, lds4v(&s.TB[b][kk]));
    for (int b = blk + 1; b < 4; ++b) post = mulv(post, lds4v(&s.TB[b][kk]));
    if (warp == 15) *reinterpret_cast<float4*>(p.w.GL + tile * KD + kk) = mulv(pre, lds4v(&s.TB[3][kk]));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const size_t o = tile * C * KD + static_cast<size_t>(t0 + i) * KD + kk;
      *reinterpret_cast<float4*>(p.w.QG + o) = mulv(mul4(p.scale, q[i]), mulv(pre, F[i]));
      *reinterpret_cast<float4*>(p.w.KG + o) = mulv(k[i], mulv(post, R[i]));
    }
  }
  wait_mma(&s.bar, phase, p.w.status, KDA_STATUS_PREP_LOAD_WAIT);
  if (warp < 4) {
    float x[32];
    const uint32_t ta = tb + (static_cast<uint32_t>(32 * warp) << 16) + (warp < 2 ? 0u : 32u);
    {
      float a[16], b[16];
      umma::tmem_ld16(ta, a);
      umma::tmem_ld16(ta + 16, b);
      umma::tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 16; ++i) { x[i] = a[i]; x[16 + i] = b[i]; }
    }
    const int L = (32 * warp + lane) & 63, b = L >> 4, r = L & 15;
    float y[8];
#pragma unroll
    for (int bb = 0; bb < 4; ++bb)
      if (bb == b) {
#pragma unroll
        for (int i = 0; i < 8; ++i) y[i] = x[8 * bb + i];
      }
    const int u = r >> 3;
    const bool wide = warp < 2, is_k = wide ? u != 0 : (r & 4) != 0;
    const int row = 16 * b + (wide ? 8 + (r & 7) : 8 * u + 4 + (r & 3)), col = 16 * b + (wide ? 0 : 8 * u), n = wide ? 8 : 4;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (i < n) {
        const float val = wide ? y[i] : (u ? y[(i + 4) & 7] : y[i]);
        if (is_k) s.A[row * AS + col + i] = val;
        else gAQK[row * C + col + i] = p.scale * val;
      }
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  // ---- operands of level 16: A rows 32 (I - 1) = q of block I, + 16 = k of block I; B rows (0, 16, 48)[I - 1] + j = columns j < 16 I
  {
    unsigned char* const A = s.R + (lane >> 3) * 2 * S96;
    unsigned char* const B = s.R + 4 * 2 * S96 + (lane >> 3) * 2 * S96;
    const int pc = lane & 7;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (blk > 0) {
        put4(A, S96, 32 * (blk - 1) + 4 * quad + i, pc, mulv(q[i], F[i]));
        put4(A, S96, 32 * (blk - 1) + 16 + 4 * quad + i, pc, mulv(k[i], F[i]));
      }
      float4 kr = mulv(k[i], R[i]);
      for (int I = blk + 1; I < 4; ++I) {
        if (I > blk + 1) kr = mulv(kr, lds4v(&s.TB[I - 1][kk]));
        put4(B, S96, (I == 1 ? 0 : (I == 2 ? 16 : 48)) + 16 * blk + 4 * quad + i, pc, kr);
      }
    }
  }
  staged();
  if (tid == 0) {
#pragma unroll 1
    for (int sl = 0; sl < 4; ++sl) mma_slice(tb + 64, aR + sl * 2 * S96, S96, aR + 4 * 2 * S96 + sl * 2 * S96, S96, idesc(128, 96), sl > 0);
    umma::commit(&s.bar);
  }
  // v of these rows, beta v
  float4 v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    v[i] = mul4(s.beta[t0 + i], ld4(p.v + (static_cast<size_t>(ci.tok0 + t0 + i) * p.H + h) * p.vc + kk, t0 + i < len && kk < p.vc));
  wait_mma(&s.bar, phase, p.w.status, KDA_STATUS_PREP_LOAD_WAIT);
  if (warp < 3) {
    const int I = warp + 1, row = 16 * I + (lane & 15);
    for (int n = 0; n < I; ++n) {
      float x[16];
      umma::tmem_ld16(tb + (static_cast<uint32_t>(32 * warp) << 16) + 64 + (I == 1 ? 0 : (I == 2 ? 16 : 48)) + 16 * n, x);
      umma::tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 16; i += 4) {
        if (lane < 16) *reinterpret_cast<float4*>(&gAQK[row * C + 16 * n + i]) = mul4(p.scale, make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]));
        else *reinterpret_cast<float4*>(&s.A[row * AS + 16 * n + i]) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
      }
    }
  }
  umma::fence_before_sync();
  __syncthreads();      // raw Akk complete; the operand region is free
  umma::fence_after_sync();
  // ---- operands of the last products (they need Tm only as B): A1 = (beta v)^T, A2 = (beta k Gam)^T, two slices over the tokens each
  {
    unsigned char* const A1 = s.R + (t0 >> 5) * 2 * S128;
    unsigned char* const A2 = s.R + 65536 + (t0 >> 5) * 2 * S128;
    const int pc = (t0 & 31) >> 2;
    float4 kg[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      kg[i] = mulv(k[i], mulv(pre, F[i]));
      if (p.save) *reinterpret_cast<float4*>(p.w.KB + tile * C * KD + static_cast<size_t>(t0 + i) * KD + kk) = kg[i];
      kg[i] = mul4(s.beta[t0 + i], kg[i]);
    }
    put4(A1, S128, kk, pc, make_float4(v[0].x, v[1].x, v[2].x, v[3].x));
    put4(A1, S128, kk + 1, pc, make_float4(v[0].y, v[1].y, v[2].y, v[3].y));
    put4(A1, S128, kk + 2, pc, make_float4(v[0].z, v[1].z, v[2].z, v[3].z));
    put4(A1, S128, kk + 3, pc, make_float4(v[0].w, v[1].w, v[2].w, v[3].w));
    put4(A2, S128, kk, pc, make_float4(kg[0].x, kg[1].x, kg[2].x, kg[3].x));
    put4(A2, S128, kk + 1, pc, make_float4(kg[0].y, kg[1].y, kg[2].y, kg[3].y));
    put4(A2, S128, kk + 2, pc, make_float4(kg[0].z, kg[1].z, kg[2].z, kg[3].z));
    put4(A2, S128, kk + 3, pc, make_float4(kg[0].w, kg[1].w, kg[2].w, kg[3].w));
  }
  // ---- raw Akk for dbeta, then Tm = (I + diag(beta) Akk)^-1 in fp32: 16 x 16 blocks by forward substitution, two levels of merges
  for (int i = tid; i < C * C / 4; i += NT) {
    const int r = i >> 4, cc = (i & 15) * 4;
    float4* a = reinterpret_cast<float4*>(&s.A[r * AS + cc]);
    if (p.save) *reinterpret_cast<float4*>(p.w.RKK + tile * C * C + r * C + cc) = *a;
    *a = mul4(s.beta[r], *a);
  }
  __syncthreads();
  {
    float x[16];
    const int b = 16 * warp, cc = lane & 15;
    if (warp < 4) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float acc = i == cc ? 1.f : 0.f;
#pragma unroll
        for (int m = 0; m < i; ++m) acc = fmaf(-s.A[(b + i) * AS + b + m], x[m], acc);
        x[i] = acc;
      }
      __syncwarp();
      if (lane < 16) {
#pragma unroll
        for (int i = 0; i < 16; ++i) s.A[(b + i) * AS + b + cc] = x[i];
      }
    }
  }
  __syncthreads();
  {      // level 1: T21 = -T22 A21 T11 for the pairs (1, 0) and (3, 2)
    const int b = 32 * (tid >> 8), i = (tid >> 4) & 15, j = tid & 15;
    float acc = 0.f;
#pragma unroll
    for (int m = 0; m < 16; ++m) acc = fmaf(s.A[(b + 16 + i) * AS + b + m], s.A[(b + m) * AS + b + j], acc);
    float* X = s.X + (tid >> 8) * 272;
    X[i * 17 + j] = acc;
    __syncthreads();
    acc = 0.f;
#pragma unroll
    for (int m = 0; m < 16; ++m) acc = fmaf(s.A[(b + 16 + i) * AS + b + 16 + m], X[m * 17 + j], acc);
    s.A[(b + 16 + i) * AS + b + j] = -acc;
    __syncthreads();
  }
  {      // level 2: rows 32..63, columns 0..31
    const int i = tid >> 5, j = tid & 31;
    float a0 = 0.f, a1 = 0.f;
#pragma unroll 8
    for (int m = 0; m < 32; ++m) {
      const float t = s.A[m * AS + j];
      a0 = fmaf(s.A[(32 + i) * AS + m], t, a0);
      a1 = fmaf(s.A[(48 + i) * AS + m], t, a1);
    }
    s.X[i * 33 + j] = a0;
    s.X[(16 + i) * 33 + j] = a1;
    __syncthreads();
    a0 = a1 = 0.f;
#pragma unroll 8
    for (int m = 0; m < 32; ++m) {
      const float t = s.X[m * 33 + j];
      a0 = fmaf(s.A[(32 + i) * AS + 32 + m], t, a0);
      a1 = fmaf(s.A[(48 + i) * AS + 32 + m], t, a1);
    }
    s.A[(32 + i) * AS + j] = -a0;
    s.A[(48 + i) * AS + j] = -a1;
    __syncthreads();
  }
  for (int i = tid; i < C * C / 4; i += NT) {
    const int r = i >> 4, c4 = i & 15;
    const float4 a = *reinterpret_cast<const float4*>(&s.A[r * AS + c4 * 4]);
    if (p.save) *reinterpret_cast<float4*>(p.w.TM + tile * C * C + r * C + c4 * 4) = a;
    put4(s.R + 131072 + (c4 >> 3) * 2 * S64, S64, r, c4 & 7, a);
  }
  staged();
  if (tid == 0) {
#pragma unroll 1
    for (int sl = 0; sl < 2; ++sl) {
      mma_slice(tb, aR + sl * 2 * S128, S128, aR + 131072 + sl * 2 * S64, S64, idesc(128, 64), sl > 0);                   // u^T
      mma_slice(tb + 64, aR + 65536 + sl * 2 * S128, S128, aR + 131072 + sl * 2 * S64, S64, idesc(128, 64), sl > 0);      // w^T
    }
    umma::commit(&s.bar);
  }
  wait_mma(&s.bar, phase, p.w.status, KDA_STATUS_PREP_LOAD_WAIT);
  {
    const int q4 = warp & 3, part = warp >> 2, col = 32 * q4 + lane;
    float x[16], y[16];
    umma::tmem_ld16(tb + (static_cast<uint32_t>(32 * q4) << 16) + 16 * part, x);
    umma::tmem_ld16(tb + (static_cast<uint32_t>(32 * q4) << 16) + 64 + 16 * part, y);
    umma::tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      p.w.U[tile * C * VD + (16 * part + i) * VD + col] = x[i];
      p.w.W[tile * C * KD + (16 * part + i) * KD + col] = y[i];
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tb, 256);
}

// =================================================================================================
// forward state scan
// =================================================================================================
// One CTA per (sequence, head) walks its chunks; tensor memory holds the state hT[v][k] (lane = value column).  Per chunk
//   v_part^T = hT w^T,  o^T = hT qg^T,  v_new^T = u^T - v_part^T,  hT = Gam_last hT + v_new^T kg,  o^T += v_new^T Aqk^T.
// Shared memory: the state as an operand (four slices, 128 KB; afterwards v_new^T and kg^T, 64 KB each) and 96 KB for w, qg, Aqk.
// The tiles of the next products are loaded into registers while the current ones execute.
namespace {

struct ScanSmem32 {
  unsigned char H[131072];       // hT: slices over k.  Later v_new^T (two slices over t) | kg^T (two slices over t)
  unsigned char B[98304];        // w (64 KB) | qg slices 0, 1 (32 KB); then qg slices 2, 3 where w was; then Aqk
  uint64_t bar[2];
  uint32_t tmem;
};
constexpr int SCAN32_SMEM = static_cast<int>(sizeof(ScanSmem32)) + 1024;
static_assert(SCAN32_SMEM <= 227 * 1024, "ScanSmem32 too large");
constexpr int TC_H = 0, TC_VN = 128, TC_O = 192;

}  // namespace

__global__ void __launch_bounds__(NT, 1) kda_f32_scan_kernel(const F32Params p) {
  chain_point();
  extern __shared__ unsigned char smem_raw[];
  ScanSmem32& s = *reinterpret_cast<ScanSmem32*>(smem_raw + pad_to_1024(smem_raw));
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0), q4 = warp & 3, part = warp >> 2;
  const int seq = p.map.started(blockIdx.x / p.H), h = blockIdx.x % p.H;
  const int c_begin = p.map.first_chunk(seq), nchunks = p.map.first_chunk(seq + 1) - c_begin;
  const long long tok_begin = p.map.first_token(seq), tok_end = p.map.first_token(seq + 1);
  const int v = 32 * q4 + lane;
  if (tid == 0) {
    mbar_init(&s.bar[0], 1);
    mbar_init(&s.bar[1], 1);
    fence_mbar_init();
  }
  __syncwarp();
  if (warp == 0) umma::tmem_alloc(&s.tmem, 256);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tb = s.tmem, tq = tb + (static_cast<uint32_t>(32 * q4) << 16);
  const size_t sb = (static_cast<size_t>(seq) * p.H + h) * p.kc * p.vc;
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int kk = 32 * part + 16 * g + i;
      x[i] = p.h0 && kk < p.kc && v < p.vc ? __ldg(p.h0 + sb + static_cast<size_t>(kk) * p.vc + v) : 0.f;
    }
    umma::tmem_st16(tq + TC_H + 32 * part + 16 * g, x);
  }
  umma::tmem_st_wait();
  const uint32_t aH = smem_u32(s.H), aB = smem_u32(s.B);
  uint32_t ph0 = 0, ph1 = 0;
  for (int i = 0; i < nchunks; ++i) {
    const size_t tile = static_cast<size_t>(c_begin + i) * p.H + h;
    const long long tok0 = tok_begin + static_cast<long long>(i) * C;
    const int len = static_cast<int>(tok_end - tok0 < C ? tok_end - tok0 : C);
    float4 w[4], qg[4];
    load64(w, p.w.W + tile * C * KD);
    load64(qg, p.w.QG + tile * C * KD);
    // ---- state: operand image, HS, hT * Gam_last
    umma::fence_after_sync();
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      float x[16];
      umma::tmem_ld16(tq + TC_H + 32 * part + 16 * g, x);
      umma::tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 4; ++e) put4(s.H + part * 2 * S128, S128, v, 4 * g + e, make_float4(x[4 * e], x[4 * e + 1], x[4 * e + 2], x[4 * e + 3]));
      const float* gl = p.w.GL + tile * KD + 32 * part + 16 * g;
      if (p.save) {
#pragma unroll
        for (int e = 0; e < 16; ++e) p.w.HS[tile * KD * VD + static_cast<size_t>(32 * part + 16 * g + e) * VD + v] = x[e];
      }
#pragma unroll
      for (int e = 0; e < 16; ++e) x[e] *= __ldg(gl + e);
      umma::tmem_st16(tq + TC_H + 32 * part + 16 * g, x);
    }
    umma::tmem_st_wait();
    put64(s.B, w);
    // qg slices 0, 1 behind w: the threads that hold their columns (float4 0..15 of a row)
    const int c4 = lane;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (c4 < 16) put4(s.B + 65536 + (c4 >> 3) * 2 * S64, S64, (tid >> 5) + 16 * j, c4 & 7, qg[j]);
    staged();
    if (tid == 0) {
#pragma unroll 1
      for (int sl = 0; sl < 4; ++sl) mma_slice(tb + TC_VN, aH + sl * 2 * S128, S128, aB + sl * 2 * S64, S64, idesc(128, 64), sl > 0);
      umma::commit(&s.bar[0]);
#pragma unroll 1
      for (int sl = 0; sl < 2; ++sl) mma_slice(tb + TC_O, aH + sl * 2 * S128, S128, aB + 65536 + sl * 2 * S64, S64, idesc(128, 64), sl > 0);
    }
    float4 kt[4], aq[2];
    load64t(kt, p.w.KG + tile * C * KD);
    load_tt(aq, p.w.AQK + tile * C * C);
    float u[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) u[e] = __ldg(p.w.U + tile * C * VD + (16 * part + e) * VD + v);
    wait_mma(&s.bar[0], ph0, p.w.status, KDA_STATUS_SCAN_MMA_WAIT);      // v_part is there, w has been read
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (c4 >= 16) put4(s.B + ((c4 >> 3) - 2) * 2 * S64, S64, (tid >> 5) + 16 * j, c4 & 7, qg[j]);
    staged();
    if (tid == 0) {
#pragma unroll 1
      for (int sl = 2; sl < 4; ++sl) mma_slice(tb + TC_O, aH + sl * 2 * S128, S128, aB + (sl - 2) * 2 * S64, S64, idesc(128, 64), true);
      umma::commit(&s.bar[1]);
    }
    {      // v_new^T = u^T - v_part^T
      float x[16];
      umma::tmem_ld16(tq + TC_VN + 16 * part, x);
      umma::tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        u[e] -= x[e];
        if (p.save) p.w.VN[tile * C * VD + (16 * part + e) * VD + v] = u[e];
      }
    }
    wait_mma(&s.bar[1], ph1, p.w.status, KDA_STATUS_SCAN_MMA_WAIT);      // the state image and qg have been read
#pragma unroll
    for (int e = 0; e < 4; ++e)
      put4(s.H + (part >> 1) * 2 * S128, S128, v, 4 * (part & 1) + e, make_float4(u[4 * e], u[4 * e + 1], u[4 * e + 2], u[4 * e + 3]));
    put64t(s.H + 65536, kt);
    put_tt(s.B + 65536, aq);
    staged();
    if (tid == 0) {
#pragma unroll 1
      for (int sl = 0; sl < 2; ++sl) mma_slice(tb + TC_H, aH + sl * 2 * S128, S128, aH + 65536 + sl * 2 * S128, S128, idesc(128, 128), true);
#pragma unroll 1
      for (int sl = 0; sl < 2; ++sl) mma_slice(tb + TC_O, aH + sl * 2 * S128, S128, aB + 65536 + sl * 2 * S64, S64, idesc(128, 64), true);
      umma::commit(&s.bar[0]);
    }
    wait_mma(&s.bar[0], ph0, p.w.status, KDA_STATUS_SCAN_MMA_WAIT);
    {
      float x[16];
      umma::tmem_ld16(tq + TC_O + 16 * part, x);
      umma::tmem_ld_wait();
      float* o = p.o + (static_cast<size_t>(tok0 + 16 * part) * p.H + h) * p.vc + v;
      if (v < p.vc) {
#pragma unroll
        for (int e = 0; e < 16; ++e)
          if (16 * part + e < len) o[static_cast<size_t>(e) * p.H * p.vc] = x[e];
      }
    }
    umma::fence_before_sync();
    __syncthreads();      // o has been read; the tiles may be rewritten
    umma::fence_after_sync();
  }
  if (p.ht) {
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      float x[16];
      umma::tmem_ld16(tq + TC_H + 32 * part + 16 * g, x);
      umma::tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int kk = 32 * part + 16 * g + i;
        if (kk < p.kc && v < p.vc) p.ht[sb + static_cast<size_t>(kk) * p.vc + v] = x[i];
      }
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tb, 256);
}

int launch_f32_fwd(const F32Params& p, long long tiles, cudaStream_t st) {
  static DeviceOnce once;
  const int rc = once.run([] {
    cudaError_t e = cudaFuncSetAttribute(kda_f32_prepare_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PREP32_SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kda_f32_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SCAN32_SMEM);
    return e;
  });
  if (rc != KDA_OK) return rc;
  if (tiles > 0x7fffffffLL) return KDA_E_SHAPE;
  kda_f32_prepare_kernel<<<static_cast<unsigned>(tiles), NT, PREP32_SMEM, st>>>(p);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return static_cast<int>(e);
  return static_cast<int>(launch_chained(kda_f32_scan_kernel, static_cast<unsigned>(p.map.N * p.H), NT, SCAN32_SMEM, st, p));
}

}  // namespace kda
