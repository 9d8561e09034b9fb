// float32 chunked backward: reverse state scan and per-chunk backward, every product in float32 accuracy on the tensor cores
// (kda_fp32.cuh).  The formulas are those of the bf16 kernels (kda_chunk_bwd_scan_tc.cu, kda_chunk_bwd_tc.cu).
// 8 x 2048 tokens x 32 heads: scan 0.7 ms, main 2.5 (bound like the forward by building the split operands in shared memory).
#include "kda_device.cuh"
#include "kda_fp32.cuh"

namespace kda {

using namespace f32;

// =================================================================================================
// reverse state scan
// =================================================================================================
// dhT[v][k] in tensor memory; per chunk, last one first:
//   dv_new^T = dhT kg^T + dO^T Aqk,   dhT = Gam_last dhT + dO^T qg - dv_new^T w.
namespace {

struct RScanSmem32 {
  unsigned char H[131072];       // dhT: slices over k.  Later dO^T | dv_new^T (two slices over t each)
  unsigned char B[65536];        // kg; then qg^T; then -w^T
  unsigned char A[32768];        // Aqk^T
  uint64_t bar, barQ;
  uint32_t tmem;
};
constexpr int RSCAN32_SMEM = static_cast<int>(sizeof(RScanSmem32)) + 1024;
static_assert(RSCAN32_SMEM <= 227 * 1024, "RScanSmem32 too large");
constexpr int TC_H = 0, TC_DV = 128;

// the transpose of 64 rows of a [tokens, H, vc] tensor (rows >= len and columns >= vc zero), see load64t
__device__ __forceinline__ void load_rows_t(float4 (&x)[4], const float* base, size_t stride, int cols, int len) {
  const int r = threadIdx.x & 127, t4 = threadIdx.x >> 7;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = 4 * (t4 + 4 * i);
    float y[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) y[e] = r < cols && t + e < len ? __ldg(base + static_cast<size_t>(t + e) * stride + r) : 0.f;
    x[i] = make_float4(y[0], y[1], y[2], y[3]);
  }
}

}  // namespace

__global__ void __launch_bounds__(NT, 1) kda_f32_bwd_scan_kernel(const F32Params p) {
  chain_point();
  extern __shared__ unsigned char smem_raw[];
  RScanSmem32& s = *reinterpret_cast<RScanSmem32*>(smem_raw + pad_to_1024(smem_raw));
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0), q4 = warp & 3, part = warp >> 2;
  const int seq = p.map.started(blockIdx.x / p.H), h = blockIdx.x % p.H;
  const int c_begin = p.map.first_chunk(seq), nchunks = p.map.first_chunk(seq + 1) - c_begin;
  const long long tok_begin = p.map.first_token(seq), tok_end = p.map.first_token(seq + 1);
  const int v = 32 * q4 + lane;
  if (tid == 0) {
    mbar_init(&s.bar, 1);
    mbar_init(&s.barQ, 1);
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
      x[i] = p.d_ht && kk < p.kc && v < p.vc ? __ldg(p.d_ht + sb + static_cast<size_t>(kk) * p.vc + v) : 0.f;
    }
    umma::tmem_st16(tq + TC_H + 32 * part + 16 * g, x);
  }
  umma::tmem_st_wait();
  const uint32_t aH = smem_u32(s.H), aB = smem_u32(s.B), aA = smem_u32(s.A);
  uint32_t ph = 0, phq = 0;
  for (int i = nchunks - 1; i >= 0; --i) {
    const size_t tile = static_cast<size_t>(c_begin + i) * p.H + h;
    const long long tok0 = tok_begin + static_cast<long long>(i) * C;
    const int len = static_cast<int>(tok_end - tok0 < C ? tok_end - tok0 : C);
    float4 kg[4], dot_[4];
    float4 aq[2];
    load64(kg, p.w.KG + tile * C * KD);
    load_ttt(aq, p.w.AQK + tile * C * C);
    load_rows_t(dot_, p.d_o + (static_cast<size_t>(tok0) * p.H + h) * p.vc, static_cast<size_t>(p.H) * p.vc, p.vc, len);
    umma::fence_after_sync();
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      float x[16];
      umma::tmem_ld16(tq + TC_H + 32 * part + 16 * g, x);
      umma::tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 4; ++e) put4(s.H + part * 2 * S128, S128, v, 4 * g + e, make_float4(x[4 * e], x[4 * e + 1], x[4 * e + 2], x[4 * e + 3]));
      const float* gl = p.w.GL + tile * KD + 32 * part + 16 * g;
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        p.w.DH[tile * KD * VD + static_cast<size_t>(32 * part + 16 * g + e) * VD + v] = x[e];
        x[e] *= __ldg(gl + e);
      }
      umma::tmem_st16(tq + TC_H + 32 * part + 16 * g, x);
    }
    umma::tmem_st_wait();
    put64(s.B, kg);
    put_ttt(s.A, aq);
    staged();
    if (tid == 0) {
#pragma unroll 1
      for (int sl = 0; sl < 4; ++sl) mma_slice(tb + TC_DV, aH + sl * 2 * S128, S128, aB + sl * 2 * S64, S64, idesc(128, 64), sl > 0);
      umma::commit(&s.bar);
    }
    float4 qt[4], wt[4];
    load64t(qt, p.w.QG + tile * C * KD);
    load64t(wt, p.w.W + tile * C * KD);
    wait_mma(&s.bar, ph, p.w.status, KDA_STATUS_BWD_SCAN_MMA_WAIT);
    put64t(s.H, dot_);
    put64t(s.B, qt);
    staged();
    if (tid == 0) {
#pragma unroll 1
      for (int sl = 0; sl < 2; ++sl) mma_slice(tb + TC_DV, aH + sl * 2 * S128, S128, aA + sl * 2 * S64, S64, idesc(128, 64), true);
      umma::commit(&s.bar);
#pragma unroll 1
      for (int sl = 0; sl < 2; ++sl) mma_slice(tb + TC_H, aH + sl * 2 * S128, S128, aB + sl * 2 * S128, S128, idesc(128, 128), true);
      umma::commit(&s.barQ);      // its own barrier: nothing but this wait separates the two, and no thread may miss a phase
    }
    wait_mma(&s.bar, ph, p.w.status, KDA_STATUS_BWD_SCAN_MMA_WAIT);      // dv_new is there; dO^T qg still runs
    float x[16];
    umma::tmem_ld16(tq + TC_DV + 16 * part, x);
    umma::tmem_ld_wait();
#pragma unroll
    for (int e = 0; e < 16; ++e) p.w.DVN[tile * C * VD + (16 * part + e) * VD + v] = x[e];
#pragma unroll
    for (int e = 0; e < 4; ++e)
      put4(s.H + 65536 + (part >> 1) * 2 * S128, S128, v, 4 * (part & 1) + e, make_float4(x[4 * e], x[4 * e + 1], x[4 * e + 2], x[4 * e + 3]));
    wait_mma(&s.barQ, phq, p.w.status, KDA_STATUS_BWD_SCAN_MMA_WAIT);      // qg^T has been read
#pragma unroll
    for (int j = 0; j < 4; ++j) wt[j] = mul4(-1.f, wt[j]);
    put64t(s.B, wt);
    staged();
    if (tid == 0) {
#pragma unroll 1
      for (int sl = 0; sl < 2; ++sl) mma_slice(tb + TC_H, aH + 65536 + sl * 2 * S128, S128, aB + sl * 2 * S128, S128, idesc(128, 128), true);
      umma::commit(&s.bar);
    }
    wait_mma(&s.bar, ph, p.w.status, KDA_STATUS_BWD_SCAN_MMA_WAIT);
  }
  if (p.dh0) {
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      float x[16];
      umma::tmem_ld16(tq + TC_H + 32 * part + 16 * g, x);
      umma::tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int kk = 32 * part + 16 * g + i;
        if (kk < p.kc && v < p.vc) p.dh0[sb + static_cast<size_t>(kk) * p.vc + v] = x[i];
      }
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tb, 256);
}

// =================================================================================================
// per-chunk backward
// =================================================================================================
// One CTA per (chunk, head).  Accumulators with the key (or value) column as tensor-memory lane, as in the bf16 kernel:
//   A   over four slices of 32 value columns, each staged once for all its products while the next one loads into registers:
//       dqg^T = h dO^T,  dw^T = -h dv_new^T,  dkg^T = dh v_new^T,  dAqk = dO v_new^T,  dTm = dv_new v^T
//   B   dTm += dw (k Gam)^T (columns times beta_j from here on),  dbv^T = dv_new^T Tm,  dbk^T = dw^T Tm,  X = dTm Tm^T,  Y = Tm^T X,  dAkk = -tril(Y, -1)
//   D   on CUDA cores, a thread per key column and 16-row block: off-diagonal blocks with the decay cut at block borders, diagonal
//       blocks pairwise with running products, then dq, dk, dg.
namespace {

constexpr int DA = 66;            // float2 per padded row of (scale dAqk, beta dAkk)
struct MainSmem32 {
  union {
    unsigned char R[163840];      // operand tiles: A h | dh | dO | dv_new | v_new | v (hi, lo of one slice each); B see there
    struct {
      float kR[C][KD], qL[C][KD], kL[C][KD];     // D: k prod(j+1 .. block end), q and k prod(block start .. t)
      float2 dA[C * DA];
      float T[4][KD], dgl[4][KD], carry[4][KD];  // per block: decay, sum of k dk_end, total of dG
    };
  };
  float beta[C];
  float hdh[KD];                  // sum over v of h dh
  float dbp[8][C];                // dbeta partial sums
  uint64_t bar;
  uint32_t tmem;
};
constexpr int MAIN32_SMEM = static_cast<int>(sizeof(MainSmem32)) + 1024;
static_assert(MAIN32_SMEM <= 227 * 1024, "MainSmem32 too large");
// tensor-memory columns
constexpr int M_DQG = 0, M_DW = 64, M_DKG = 128, M_DAQ = 192, M_DTM = 256, M_DBV = 320, M_DBK = 384, M_XY = 448;

}  // namespace

__global__ void __launch_bounds__(NT, 1) kda_f32_bwd_main_kernel(const F32Params p) {
  chain_point();
  extern __shared__ unsigned char smem_raw[];
  MainSmem32& s = *reinterpret_cast<MainSmem32*>(smem_raw + pad_to_1024(smem_raw));
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0), q4 = warp & 3, part = warp >> 2;
  const int c = blockIdx.x / p.H, h = blockIdx.x % p.H;
  if (c >= p.map.total()) return;
  const ChunkInfo ci = p.map.info(c);
  const int len = ci.len;
  const size_t tile = blockIdx.x, tTK = tile * C * KD, tTT = tile * C * C, tKV = tile * KD * VD;
  const size_t vrow = (static_cast<size_t>(ci.tok0) * p.H + h) * p.vc, vstr = static_cast<size_t>(p.H) * p.vc;
  if (tid == 0) {
    mbar_init(&s.bar, 1);
    fence_mbar_init();
  }
  __syncwarp();
  if (warp == 0) umma::tmem_alloc(&s.tmem, 512);
  if (tid < C) s.beta[tid] = tid < len ? __ldg(p.beta + static_cast<size_t>(ci.tok0 + tid) * p.H + h) : 0.f;
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tb = s.tmem, tq = tb + (static_cast<uint32_t>(32 * q4) << 16), aR = smem_u32(s.R);
  uint32_t ph = 0;
  constexpr unsigned BIT = KDA_STATUS_BWD_MAIN_MMA_WAIT;

  // ---- A: four slices of 32 value columns
  {
    const int r = tid >> 3, pc = tid & 7;
    float4 x[8];
    auto load = [&](int sl) {
      const int col = 32 * sl + 4 * pc;
      const bool ok = r < len && col < p.vc;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        x[i] = __ldg(reinterpret_cast<const float4*>(p.w.HS + tKV + static_cast<size_t>(r + 64 * i) * VD + col));
        x[2 + i] = __ldg(reinterpret_cast<const float4*>(p.w.DH + tKV + static_cast<size_t>(r + 64 * i) * VD + col));
      }
      x[4] = ld4(p.d_o + vrow + r * vstr + col, ok);
      x[5] = __ldg(reinterpret_cast<const float4*>(p.w.DVN + tTK + r * VD + col));
      x[6] = __ldg(reinterpret_cast<const float4*>(p.w.VN + tTK + r * VD + col));
      x[7] = ld4(p.v + vrow + r * vstr + col, ok);
    };
    load(0);
    float hd[2] = {0.f, 0.f};
#pragma unroll 1
    for (int sl = 0; sl < 4; ++sl) {
      if (sl > 0) wait_mma(&s.bar, ph, p.w.status, BIT);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        put4(s.R, S128, r + 64 * i, pc, x[i]);
        put4(s.R + 32768, S128, r + 64 * i, pc, x[2 + i]);
        hd[i] += x[i].x * x[2 + i].x + x[i].y * x[2 + i].y + x[i].z * x[2 + i].z + x[i].w * x[2 + i].w;
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) put4(s.R + 65536 + i * S64, 2 * S64, r, pc, x[4 + i]);
#pragma unroll
      for (int i = 2; i < 4; ++i) put4(s.R + 65536 + 16384 * i, S64, r, pc, x[4 + i]);
      staged();
      if (tid == 0) {
        // dO and dv_new stand one behind the other as one B operand of 128 rows: dqg^T and dw^T are one product, h is read once
        mma_slice(tb + M_DQG, aR, S128, aR + 65536, 2 * S64, idesc(128, 128), sl > 0);
        mma_slice(tb + M_DKG, aR + 32768, S128, aR + 98304, S64, idesc(128, 64), sl > 0);
        mma_slice(tb + M_DAQ, aR + 65536, 2 * S64, aR + 98304, S64, idesc(64, 64), sl > 0);
        mma_slice(tb + M_DTM, aR + 65536 + S64, 2 * S64, aR + 114688, S64, idesc(64, 64), sl > 0);
        umma::commit(&s.bar);
      }
      if (sl < 3) load(sl + 1);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) hd[i] += __shfl_xor_sync(0xffffffffu, hd[i], o);
      if (pc == 0) s.hdh[r + 64 * i] = hd[i];
    }
  }
  float4 kb[4], tt[2];
  load64(kb, p.w.KB + tTK);
  load_ttt(tt, p.w.TM + tTT);
  wait_mma(&s.bar, ph, p.w.status, BIT);
  // ---- B1: dTm += dw (k Gam)^T.  dw [64 t][k] at 0, k Gam at 64 K, Tm^T at 128 K
  float dw[16];
  {
    umma::tmem_ld16(tq + M_DW + 16 * part, dw);
    umma::tmem_ld_wait();
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      dw[e] = -dw[e];
      put1(s.R + q4 * 2 * S64, S64, 16 * part + e, lane, dw[e]);
    }
    put64(s.R + 65536, kb);
    put_ttt(s.R + 131072, tt);
    staged();
    if (tid == 0) {
#pragma unroll 1
      for (int sl = 0; sl < 4; ++sl) mma_slice(tb + M_DTM, aR + sl * 2 * S64, S64, aR + 65536 + sl * 2 * S64, S64, idesc(64, 64), true);
      umma::commit(&s.bar);
    }
    load64t(kb, p.w.DVN + tTK);
    wait_mma(&s.bar, ph, p.w.status, BIT);
  }
  // ---- B2: dbv^T = dv_new^T Tm, dbk^T = dw^T Tm.  dv_new^T at 0, dw^T at 64 K (two slices over the tokens each)
  put64t(s.R, kb);
#pragma unroll
  for (int e = 0; e < 4; ++e)
    put4(s.R + 65536 + (part >> 1) * 2 * S128, S128, 32 * q4 + lane, 4 * (part & 1) + e, make_float4(dw[4 * e], dw[4 * e + 1], dw[4 * e + 2], dw[4 * e + 3]));
  staged();
  if (tid == 0) {
#pragma unroll 1
    for (int sl = 0; sl < 2; ++sl) {
      mma_slice(tb + M_DBV, aR + sl * 2 * S128, S128, aR + 131072 + sl * 2 * S64, S64, idesc(128, 64), sl > 0);
      mma_slice(tb + M_DBK, aR + 65536 + sl * 2 * S128, S128, aR + 131072 + sl * 2 * S64, S64, idesc(128, 64), sl > 0);
    }
    umma::commit(&s.bar);
  }
  const int row = 16 * q4 + (lane & 15);      // M = 64 accumulators: rows 16 q4 .. in lanes 0..15 of the quadrant
  const bool low = lane < 16;
  float d[16];
  umma::tmem_ld16(tq + M_DTM + 16 * part, d);
  umma::tmem_ld_wait();
  {      // dbeta_j += sum_t Tm[t][j] dTm[t][j]: sixteen columns, summed over the lanes at once
    float y[16];
#pragma unroll
    for (int e = 0; e < 16; e += 4) {
      const float4 t = ld4(p.w.TM + tTT + row * C + 16 * part + e, low);
      y[e] = t.x * d[e]; y[e + 1] = t.y * d[e + 1]; y[e + 2] = t.z * d[e + 2]; y[e + 3] = t.w * d[e + 3];
    }
    if (!low) {
#pragma unroll
      for (int e = 0; e < 16; ++e) y[e] = 0.f;
    }
#pragma unroll
    for (int o = 8; o >= 1; o >>= 1) {
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int e = 0; e < o; ++e) {
        const float mine = up ? y[e + o] : y[e], other = up ? y[e] : y[e + o];
        y[e] = mine + __shfl_xor_sync(0xffffffffu, other, o);
      }
    }
    y[0] += __shfl_xor_sync(0xffffffffu, y[0], 16);
    if (low) s.dbp[q4][16 * part + lane] = y[0];
  }
  load_tt(tt, p.w.TM + tTT);
  wait_mma(&s.bar, ph, p.w.status, BIT);
  // ---- B3: X = dTm diag(beta) Tm^T.  dTm diag(beta) at 0, Tm at 32 K
  if (low) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float4 b = *reinterpret_cast<const float4*>(&s.beta[16 * part + 4 * e]);
      put4(s.R + (part >> 1) * 2 * S64, S64, row, 4 * (part & 1) + e, make_float4(b.x * d[4 * e], b.y * d[4 * e + 1], b.z * d[4 * e + 2], b.w * d[4 * e + 3]));
    }
  }
  put_tt(s.R + 32768, tt);
  staged();
  if (tid == 0) {
#pragma unroll 1
    for (int sl = 0; sl < 2; ++sl) mma_slice(tb + M_XY, aR + sl * 2 * S64, S64, aR + 32768 + sl * 2 * S64, S64, idesc(64, 64), sl > 0);
    umma::commit(&s.bar);
  }
  {      // dv = beta dbv
    float x[16];
    const int v = 32 * q4 + lane;
    umma::tmem_ld16(tq + M_DBV + 16 * part, x);
    umma::tmem_ld_wait();
    if (v < p.vc) {
#pragma unroll
      for (int e = 0; e < 16; ++e)
        if (16 * part + e < len) p.dv[vrow + (16 * part + e) * vstr + v] = s.beta[16 * part + e] * x[e];
    }
  }
  wait_mma(&s.bar, ph, p.w.status, BIT);
  // ---- B4: Y = Tm^T X.  X^T at 64 K, Tm^T still at 128 K
  umma::tmem_ld16(tq + M_XY + 16 * part, d);
  umma::tmem_ld_wait();
  if (low) {
#pragma unroll
    for (int e = 0; e < 16; ++e) put1(s.R + 65536 + (row >> 5) * 2 * S64, S64, 16 * part + e, row & 31, d[e]);
  }
  staged();
  if (tid == 0) {
#pragma unroll 1
    for (int sl = 0; sl < 2; ++sl) mma_slice(tb + M_XY, aR + 131072 + sl * 2 * S64, S64, aR + 65536 + sl * 2 * S64, S64, idesc(64, 64), sl > 0);
    umma::commit(&s.bar);
  }
  // ---- this thread's key column and rows for the last phase
  const int kk = tid & 127, blk = tid >> 7, t0 = 16 * blk;
  float qv[16], kv[16], lam[16];
  {
    const bool okk = kk < p.kc;
    const size_t grow = (static_cast<size_t>(ci.tok0 + t0) * p.H + h) * p.kc + kk, qrow = (static_cast<size_t>(ci.tok0 + t0) * p.HQ + h / p.grp) * p.kc + kk;
    const size_t gs = static_cast<size_t>(p.H) * p.kc, qs = static_cast<size_t>(p.HQ) * p.kc;
    // all 48 loads first: anything that waits for one of them in between would expose a latency per row
    const float* qs_ = p.use_l2 ? p.w.QN + tTK + t0 * KD + kk : p.q + qrow;
    const float* ks_ = p.use_l2 ? p.w.KN + tTK + t0 * KD + kk : p.k + qrow;
    const size_t st = p.use_l2 ? static_cast<size_t>(KD) : qs;
#pragma unroll
    for (int i = 0; i < 16; ++i) lam[i] = okk && t0 + i < len ? __ldg(p.g + grow + i * gs) : 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) qv[i] = okk && t0 + i < len ? __ldg(qs_ + i * st) : 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) kv[i] = okk && t0 + i < len ? __ldg(ks_ + i * st) : 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) lam[i] = expf(lam[i]);
  }
  float rk[16];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float4 x = ld4(p.w.RKK + tTT + row * C + 16 * part + 4 * e, low);
    rk[4 * e] = x.x; rk[4 * e + 1] = x.y; rk[4 * e + 2] = x.z; rk[4 * e + 3] = x.w;
  }
  wait_mma(&s.bar, ph, p.w.status, BIT);
  __syncthreads();      // every product is complete: the operand region becomes the last phase's arrays
  {
    float y[16], a[16];
    umma::tmem_ld16(tq + M_XY + 16 * part, y);
    umma::tmem_ld16(tq + M_DAQ + 16 * part, a);
    umma::tmem_ld_wait();
    if (low) {
      float pb = 0.f;
      const float b = s.beta[row];
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const int j = 16 * part + e;
        const float x = j < row ? -y[e] : 0.f;
        pb = fmaf(x, rk[e], pb);
        s.dA[row * DA + j] = make_float2(j <= row ? p.scale * a[e] : 0.f, b * x);
      }
      s.dbp[4 + part][row] = pb;
    }
  }
  // ---- D: decays of this block as running products; the arrays the other blocks read
  {
    float f = 1.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      f *= lam[i];
      s.qL[t0 + i][kk] = qv[i] * f;
      s.kL[t0 + i][kk] = kv[i] * f;
    }
    s.T[blk][kk] = f;
    f = 1.f;
#pragma unroll
    for (int i = 15; i >= 0; --i) {
      s.kR[t0 + i][kk] = kv[i] * f;
      f *= lam[i];
    }
  }
  __syncthreads();
  float cq[16], cp[16], cn[16];
  float gam_last;
  {
    float pre = 1.f, post = 1.f;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      if (b < blk) pre *= s.T[b][kk];
      if (b > blk) post *= s.T[b][kk];
    }
    gam_last = pre * post * s.T[blk][kk];
    umma::tmem_ld16(tq + M_DQG + t0, cq);
    umma::tmem_ld16(tq + M_DBK + t0, cp);
    umma::tmem_ld16(tq + M_DKG + t0, cn);
    umma::tmem_ld_wait();
    float dgl = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      cq[i] *= p.scale * pre;
      cp[i] *= s.beta[t0 + i] * pre;
      cn[i] *= post;
      dgl = fmaf(s.kR[t0 + i][kk], cn[i], dgl);
    }
    s.dgl[blk][kk] = dgl;
  }
  // off-diagonal blocks: rows of this block against the columns of earlier ones (cq, cp), columns against the rows of later ones (cn)
  {
    float m = 1.f;
    for (int J = blk - 1; J >= 0; --J) {
#pragma unroll 1
      for (int j = 0; j < 16; j += 2) {
        const float k0 = s.kR[16 * J + j][kk] * m, k1 = s.kR[16 * J + j + 1][kk] * m;
#pragma unroll
        for (int t = 0; t < 16; ++t) {
          const float4 a = *reinterpret_cast<const float4*>(&s.dA[(t0 + t) * DA + 16 * J + j]);
          cq[t] = fmaf(a.x, k0, fmaf(a.z, k1, cq[t]));
          cp[t] = fmaf(a.y, k0, fmaf(a.w, k1, cp[t]));
        }
      }
      m *= s.T[J][kk];
    }
    m = 1.f;
    for (int I = blk + 1; I < 4; ++I) {
#pragma unroll 1
      for (int t = 0; t < 16; ++t) {
        const float ql = s.qL[16 * I + t][kk] * m, kl = s.kL[16 * I + t][kk] * m;
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          const float4 a = *reinterpret_cast<const float4*>(&s.dA[(16 * I + t) * DA + t0 + j]);
          cn[j] = fmaf(a.x, ql, fmaf(a.y, kl, cn[j]));
          cn[j + 1] = fmaf(a.z, ql, fmaf(a.w, kl, cn[j + 1]));
        }
      }
      m *= s.T[I][kk];
    }
    float f = 1.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      f *= lam[i];
      cq[i] *= f;
      cp[i] *= f;
    }
    f = 1.f;
#pragma unroll
    for (int i = 15; i >= 0; --i) {
      cn[i] *= f;
      f *= lam[i];
    }
  }
  // the diagonal block pairwise
#pragma unroll
  for (int t = 0; t < 16; ++t) {
    float D = 1.f;
#pragma unroll
    for (int j = t; j >= 0; --j) {
      const float2 a = s.dA[(t0 + t) * DA + t0 + j];
      const float kd = kv[j] * D;
      cq[t] = fmaf(a.x, kd, cq[t]);
      cp[t] = fmaf(a.y, kd, cp[t]);
      cn[j] = fmaf(D, fmaf(a.y, kv[t], a.x * qv[t]), cn[j]);
      D *= lam[j];
    }
  }
  const bool direct = p.grp == 1 && !p.use_l2;
  float* const dqo = direct ? p.dq : p.w.DQ;
  float* const dko = direct ? p.dk : p.w.DK;
  const size_t orow = (static_cast<size_t>(ci.tok0 + t0) * p.H + h) * p.kc + kk, ostr = static_cast<size_t>(p.H) * p.kc;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    if (kk < p.kc && t0 + i < len) {
      dqo[orow + i * ostr] = cq[i];
      dko[orow + i * ostr] = cp[i] + cn[i];
    }
    cq[i] = qv[i] * cq[i] + kv[i] * (cp[i] - cn[i]);      // dG
  }
  if (blk == 3) cq[15] += s.dgl[0][kk] + s.dgl[1][kk] + s.dgl[2][kk] + s.dgl[3][kk] + gam_last * s.hdh[kk];
#pragma unroll
  for (int i = 14; i >= 0; --i) cq[i] += cq[i + 1];
  s.carry[blk][kk] = cq[0];
  umma::fence_before_sync();
  __syncthreads();
  float add = 0.f;
#pragma unroll
  for (int b = 1; b < 4; ++b)
    if (b > blk) add += s.carry[b][kk];
#pragma unroll
  for (int i = 0; i < 16; ++i)
    if (kk < p.kc && t0 + i < len) p.dg[orow + i * ostr] = cq[i] + add;
  if (tid < len) {
    float b = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) b += s.dbp[i][tid];
    p.dbeta[static_cast<size_t>(ci.tok0 + tid) * p.H + h] = b;
  }
  if (warp == 0) umma::tmem_dealloc(tb, 512);
}

// dq, dk from the gradients w.r.t. the rows the chunk kernels saw, per value head: sum over the heads of a group, then the backward of
// x^ = x rsqrt(sum x^2 + eps).  One warp per row of q and k.
__global__ void __launch_bounds__(256) kda_f32_bwd_finish_kernel(const F32Params p, long long rows) {
  chain_point();
  const long long row = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31, kk = 4 * lane;
  if (row >= rows) return;
  const long long tok = row / p.HQ, src = (tok * p.H + (row % p.HQ) * p.grp) * p.kc + kk, out = row * p.kc + kk;
  const bool ok = kk < p.kc;
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    const float* g = which ? p.w.DK : p.w.DQ;
    float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int j = 0; j < p.grp; ++j) {
      const float4 x = ld4(g + src + static_cast<long long>(j) * p.kc, ok);
      d = make_float4(d.x + x.x, d.y + x.y, d.z + x.z, d.w + x.w);
    }
    if (p.use_l2) {
      const float4 x = ld4((which ? p.k : p.q) + out, ok);
      const float rs = rsqrtf(warp_sum(x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w) + L2NORM_EPS);
      const float dot = warp_sum(x.x * d.x + x.y * d.y + x.z * d.z + x.w * d.w) * rs * rs;
      d = make_float4(rs * (d.x - x.x * dot), rs * (d.y - x.y * dot), rs * (d.z - x.z * dot), rs * (d.w - x.w * dot));
    }
    if (ok) *reinterpret_cast<float4*>((which ? p.dk : p.dq) + out) = d;
  }
}

int launch_f32_bwd(const F32Params& p, long long tiles, cudaStream_t st) {
  static DeviceOnce once;
  const int rc = once.run([] {
    cudaError_t e = cudaFuncSetAttribute(kda_f32_bwd_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RSCAN32_SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kda_f32_bwd_main_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MAIN32_SMEM);
    return e;
  });
  if (rc != KDA_OK) return rc;
  if (tiles > 0x7fffffffLL) return KDA_E_SHAPE;
  kda_f32_bwd_scan_kernel<<<static_cast<unsigned>(p.map.N * p.H), NT, RSCAN32_SMEM, st>>>(p);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return static_cast<int>(e);
  return static_cast<int>(launch_chained(kda_f32_bwd_main_kernel, static_cast<unsigned>(tiles), NT, MAIN32_SMEM, st, p));
}
int launch_f32_finish(const F32Params& p, long long rows, cudaStream_t st) {
  return static_cast<int>(launch_chained(kda_f32_bwd_finish_kernel, static_cast<unsigned>((rows + 7) / 8), 256, 0, st, p, rows));
}

}  // namespace kda
