// Forward state scan of chunked KDA with the fp32 state in registers (sm_100a).
//
//   v_new = u - w h;   o = qg h + Aqk v_new;   h <- Diag(Gam_last) h + kg^T v_new          per chunk of 64 tokens, in order
//
// The recurrence is independent per value column.  Two STATE WARPS own a group of 16 of them: each holds hT[16 v][64 k] as mma.sync
// accumulators (32 fp32 registers a thread) for the whole sequence and computes 32 of the chunk's tokens.  Per chunk they leave the bf16
// image of hT in shared memory, v_part^T = hT w^T, leave v_new^T = u^T - v_part^T there, and update hT += v_new^T kg: two hand-overs between
// two warps.  OUTPUT WARPS form o^T = hT qg^T + v_new^T Aqk^T beside them from the same images, up to two chunks behind; in training these are
// the chunk's HS and VNEWT tiles and leave from there.  Operand tiles arrive through a ring of bulk copies.
// A CTA has 2 or 4 groups (32 or 64 value columns of one (sequence, head) unit): as few as keep the grid within one CTA per SM.  With 4
// an output warp takes two groups, so that it reads its qg and Aqk rows once for both.
//
// What bounds it: the fragments' reads of shared memory (1.2 k of 2.3 k cycles a chunk with 2 groups, besides 0.5 k for the
// copies' writes) and the latency of the two hand-overs; loads alone (QG and Aqk left out, or two stages for three) change nothing.  One warp for
// all 128 k of a group: 174 us for 128 chunks on 32 units, this split: 165, with the state in tensor memory and tcgen05 products, whose
// hand-overs between the issuing thread and the warps take 290 cycles each: 192.  4 groups: 300 (tensor memory, whole units) -> 244.
// One unit of 128 value columns per CTA stays on tensor memory (kda_chunk_scan_tc.cu): eight groups on one SM wait for its shared
// memory, 260 against 160 us at 64 chunks.  Every layout forms the same sums: the bits do not depend on it.
#include "kda_chunk.cuh"
#include "kda_device.cuh"
#include "kda_scan.cuh"

namespace kda {

namespace {

template <int NP>
struct ScanCfg {
  static constexpr int VS = 16 * NP;                         // value columns of the CTA
  static constexpr int STAGES = NP == 2 ? 3 : 2;
  static constexpr int GW = NP / 2;                          // groups of an output warp
  static constexpr int THREADS = 32 * (2 * NP + 4 + 1);      // state warps, output warps, one warp that issues the copies
};

template <int NP>
struct ScanStage {
  unsigned char W[TILE_TK], QG[TILE_TK], KG[TILE_TK], AQK[TILE_TT], UT[16 * NP * 128];
  float GL[KD];
  unsigned char pad[512];
};
template <int NP>
struct ScanSmem {
  ScanStage<NP> st[ScanCfg<NP>::STAGES];
  unsigned char H[2][2][16 * NP * 128];   // bf16 hT of even and odd chunks: two spans [VS v][64 k] (= the CTA's rows of the HS tile)
  unsigned char VN[2][16 * NP * 128];     // bf16 v_new^T [VS v][64 t] (= its rows of the VNEWT tile)
  unsigned char oS[4][NP * 512];          // o of an output warp: [32 t][16 GW v]
  uint64_t full[ScanCfg<NP>::STAGES], empty[ScanCfg<NP>::STAGES];
  uint64_t hReady[2][NP], vReady[2][NP], hFree[2][NP], vFree[2][NP];      // of even and odd chunks: one side may be two chunks ahead
};
template <int NP>
constexpr unsigned SCAN_TX = 3 * TILE_TK + TILE_TT + 16 * NP * 128 + TILE_GL;
static_assert(sizeof(ScanStage<2>) % 1024 == 0 && sizeof(ScanStage<4>) % 1024 == 0, "stage alignment");
static_assert(sizeof(ScanSmem<2>) + 1024 <= 227 * 1024 && sizeof(ScanSmem<4>) + 1024 <= 227 * 1024, "ScanSmem too large");

__device__ __forceinline__ void stsm_x4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void stsm_x4_t(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

}  // namespace

template <int NP>
__global__ void __launch_bounds__(ScanCfg<NP>::THREADS, 1) kda_chunk_scan_kernel(const ScanParams p) {
  chain_point();
  using Cfg = ScanCfg<NP>;
  constexpr int VS = Cfg::VS, ST = Cfg::STAGES, GW = Cfg::GW;
  extern __shared__ unsigned char smem_raw[];
  ScanSmem<NP>& s = *reinterpret_cast<ScanSmem<NP>*>(smem_raw + pad_to_1024(smem_raw));
  const int tid = threadIdx.x, lane = tid & 31, gid = lane >> 2, tig = lane & 3;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  constexpr int PARTS = VD / VS;
  const int unit = blockIdx.x / PARTS, v0 = VS * (blockIdx.x % PARTS);
  const int seq = p.map.started(unit / p.H), h = unit % p.H;
  const int c_begin = p.map.first_chunk(seq), nchunks = p.map.first_chunk(seq + 1) - c_begin;
  const long long tok_begin = p.map.first_token(seq), tok_end = p.map.first_token(seq + 1);
  if (tid == 0) {
    for (int i = 0; i < ST; ++i) {
      mbar_init(&s.full[i], 1);
      mbar_init(&s.empty[i], 2 * NP + 4);
    }
    for (int i = 0; i < 2 * NP; ++i) {
      mbar_init(&s.hReady[0][0] + i, 2);
      mbar_init(&s.vReady[0][0] + i, 2);
      mbar_init(&s.hFree[0][0] + i, 2);
      mbar_init(&s.vFree[0][0] + i, 2);
    }
    fence_mbar_init();
  }
  __syncthreads();
  auto gave_up = [&](unsigned bit) {
    if (lane == 0) atomicOr(p.status, bit);
  };

  if (warp == 2 * NP + 4) {
    // ================= copies =================
    if (lane == 0) {
      int i = 0;
      for (; i < nchunks; ++i) {
        if (i >= ST && !mbar_wait(&s.empty[i % ST], (i / ST + 1) & 1)) {
          atomicOr(p.status, KDA_STATUS_SCAN_LOAD_WAIT);
          break;
        }
        ScanStage<NP>& d = s.st[i % ST];
        uint64_t* const bar = &s.full[i % ST];
        const size_t tile = static_cast<size_t>(c_begin + i) * p.H + h;
        mbar_expect_tx(bar, SCAN_TX<NP>);
        bulk_g2s(d.W, p.W + tile * TILE_TK, TILE_TK, bar);
        bulk_g2s(d.UT, p.UT + tile * TILE_VT + static_cast<size_t>(v0) * 128, VS * 128, bar);
        bulk_g2s(d.GL, p.GL + tile * TILE_GL, TILE_GL, bar);
        bulk_g2s(d.KG, p.KG + tile * TILE_TK, TILE_TK, bar);
        bulk_g2s(d.QG, p.QG + tile * TILE_TK, TILE_TK, bar);
        bulk_g2s(d.AQK, p.AQK + tile * TILE_TT, TILE_TT, bar);
      }
      for (int j = i > ST ? i - ST : 0; j < i; ++j) mbar_wait(&s.full[j % ST], (j / ST) & 1);      // no copy in flight outlives the CTA, also where others gave up
    }
    return;      // (nothing waits for this warp; the CTA's memory lives until the others leave)
  }
  const size_t sb = (static_cast<size_t>(seq) * p.H + h) * p.kc * p.vc;
  const int lr = lane & 7, l8 = (lane >> 3) & 1, l16 = lane >> 4;
  // ldmatrix addresses inside a swizzled tile: row * 128 + ((piece ^ row) & 7) * 16; the row part is fixed per lane
  const int arow = lr + 8 * l8, brow = lr + 8 * l16;      // A: rows v, pieces l16; B: rows of two 8-row tiles, pieces l8

  if (warp < 2 * NP) {
    // ================= state warps: 16 value columns, half of the key columns =================
    const int grp = warp >> 1, half = warp & 1;
    const uint32_t rowb = static_cast<uint32_t>(16 * grp) * 128u;                 // the group's 16 rows in [VS][64] tiles
    const int va = v0 + 16 * grp + gid, vb = va + 8;
    float hs[8][4];      // hT[v][64 half + k]: [8-column tile of k][fragment]
#pragma unroll
    for (int n = 0; n < 8; ++n) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int k = 64 * half + 8 * n + 2 * tig + (e & 1), v = e < 2 ? va : vb;
        hs[n][e] = p.h0 && k < p.kc && v < p.vc ? __ldg(p.h0 + sb + static_cast<size_t>(k) * p.vc + v) : 0.f;
      }
    }
    const bool keep = p.HS != nullptr;      // the images also leave by bulk stores
    bool ok = true;
    for (int i = 0; i < nchunks; ++i) {
      ScanStage<NP>& d = s.st[i % ST];
      const uint32_t aH = smem_u32(s.H[i & 1][0]) + rowb + arow * 128, aV = smem_u32(s.VN[i & 1]) + rowb + arow * 128;
      if (i > 1 && !mbar_wait(&s.hFree[i & 1][grp], ((i >> 1) + 1) & 1)) { ok = false; break; }
      // the bf16 image of this half of the state
#pragma unroll
      for (int n = 0; n < 4; ++n)
        stsm_x4(aH + half * (VS * 128) + (((2 * n + l16) ^ lr) << 4), pack_bf16(hs[2 * n][0], hs[2 * n][1]), pack_bf16(hs[2 * n][2], hs[2 * n][3]),
                pack_bf16(hs[2 * n + 1][0], hs[2 * n + 1][1]), pack_bf16(hs[2 * n + 1][2], hs[2 * n + 1][3]));
      if (keep) fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s.hReady[i & 1][grp]);
      if (!mbar_wait(&s.full[i % ST], (i / ST) & 1)) { ok = false; break; }
      const uint32_t aW = smem_u32(d.W) + (32 * half + brow) * 128;
      uint32_t a[2][4], b[2][2][4];
      auto load_b = [&](int ks, uint32_t (&f)[2][4]) {      // w[t][k] of this half's four 8-token tiles
#pragma unroll
        for (int n = 0; n < 2; ++n) ldsm_x4(f[n], aW + (ks >> 2) * 8192 + n * 2048 + (((2 * (ks & 3) + l8) ^ lr) << 4));
      };
      auto load_h = [&](int ks, uint32_t (&f)[4]) { ldsm_x4(f, aH + (ks >> 2) * (VS * 128) + (((2 * (ks & 3) + l16) ^ lr) << 4)); };
      load_b(0, b[0]);
      uint32_t ut[4][2];      // u^T, needed behind product 1
      {
        const unsigned char* const uA = d.UT + rowb + gid * 128 + tig * 4;
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          ut[n][0] = *reinterpret_cast<const uint32_t*>(uA + (((4 * half + n) ^ gid) << 4));
          ut[n][1] = *reinterpret_cast<const uint32_t*>(uA + (((4 * half + n) ^ gid) << 4) + 1024);
        }
      }
#pragma unroll
      for (int n = 0; n < 8; ++n) {      // hT *= Gam_last
        const float2 g = *reinterpret_cast<const float2*>(&d.GL[64 * half + 8 * n + 2 * tig]);
        hs[n][0] *= g.x; hs[n][1] *= g.y; hs[n][2] *= g.x; hs[n][3] *= g.y;
      }
      float acc[4][4];      // v_part^T: [8-token tile][fragment]
#pragma unroll
      for (int n = 0; n < 4; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
      if (!mbar_wait(&s.hReady[i & 1][grp], (i >> 1) & 1)) { ok = false; break; }
      // fragments are loaded one step ahead of their products: nobody else hides their latency
      load_h(0, a[0]);
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        if (ks < 7) {
          load_h(ks + 1, a[(ks + 1) & 1]);
          load_b(ks + 1, b[(ks + 1) & 1]);
        }
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          mma16816(acc[2 * n], a[ks & 1], b[ks & 1][n][0], b[ks & 1][n][1]);
          mma16816(acc[2 * n + 1], a[ks & 1], b[ks & 1][n][2], b[ks & 1][n][3]);
        }
      }
      if (i > 1 && !mbar_wait(&s.vFree[i & 1][grp], ((i >> 1) + 1) & 1)) { ok = false; break; }
      // v_new^T = u^T - v_part^T, as bf16
#pragma unroll
      for (int n = 0; n < 4; n += 2) {
        const float2 ua = unpack_bf16(ut[n][0]), ub = unpack_bf16(ut[n][1]), uc = unpack_bf16(ut[n + 1][0]), ud = unpack_bf16(ut[n + 1][1]);
        stsm_x4(aV + (((4 * half + n + l16) ^ lr) << 4), pack_bf16(ua.x - acc[n][0], ua.y - acc[n][1]), pack_bf16(ub.x - acc[n][2], ub.y - acc[n][3]),
                pack_bf16(uc.x - acc[n + 1][0], uc.y - acc[n + 1][1]), pack_bf16(ud.x - acc[n + 1][2], ud.y - acc[n + 1][3]));
      }
      if (keep) fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s.vReady[i & 1][grp]);
      // hT += v_new^T kg: kg fragments of 16 tokens and this half's 64 key columns
      const uint32_t aK = smem_u32(d.KG) + half * 8192 + arow * 128;
      uint32_t f[2][4][4];
      auto load_k = [&](int t, uint32_t (&x)[4][4]) {
#pragma unroll
        for (int n = 0; n < 4; ++n) ldsm_x4_t(x[n], aK + t * 2048 + (((2 * n + l16) ^ lr) << 4));
      };
      auto load_v = [&](int t, uint32_t (&x)[4]) { ldsm_x4(x, aV + (((2 * t + l16) ^ lr) << 4)); };
      load_k(0, f[0]);
      if (!mbar_wait(&s.vReady[i & 1][grp], (i >> 1) & 1)) { ok = false; break; }
      load_v(0, a[0]);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        if (t < 3) {
          load_v(t + 1, a[(t + 1) & 1]);
          load_k(t + 1, f[(t + 1) & 1]);
        }
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          mma16816(hs[2 * n], a[t & 1], f[t & 1][n][0], f[t & 1][n][1]);
          mma16816(hs[2 * n + 1], a[t & 1], f[t & 1][n][2], f[t & 1][n][3]);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&s.empty[i % ST]);
    }
    if (!ok) gave_up(KDA_STATUS_SCAN_LOAD_WAIT);
    else if (p.ht) {
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int k = 64 * half + 8 * n + 2 * tig + (e & 1), v = e < 2 ? va : vb;
          if (k < p.kc && v < p.vc) p.ht[sb + static_cast<size_t>(k) * p.vc + v] = hs[n][e];
        }
    }
    return;
  }

  // ================= output warps: o of 16 GW value columns, 32 tokens =================
  {
    const int g0 = ((warp - 2 * NP) >> 1) * GW, part = warp & 1;
    const uint32_t rowb = static_cast<uint32_t>(16 * g0) * 128u;
    const bool stores = part == 0 && lane == 0 && p.HS != nullptr;
    bool ok = true;
    for (int i = 0; i < nchunks; ++i) {
      ScanStage<NP>& d = s.st[i % ST];
      const size_t tile = static_cast<size_t>(c_begin + i) * p.H + h;
      const unsigned ph = (i >> 1) & 1;
      unsigned char *const H0 = s.H[i & 1][0] + rowb, *const H1 = s.H[i & 1][1] + rowb, *const VN = s.VN[i & 1] + rowb;
      if (!mbar_wait(&s.full[i % ST], (i / ST) & 1) || !mbar_wait(&s.hReady[i & 1][g0], ph) || (GW > 1 && !mbar_wait(&s.hReady[i & 1][g0 + GW - 1], ph))) { ok = false; break; }
      if (stores) {
        bulk_s2g(p.HS + tile * TILE_VK + static_cast<size_t>(v0) * 128 + rowb, H0, GW * 2048);
        bulk_s2g(p.HS + tile * TILE_VK + 16384 + static_cast<size_t>(v0) * 128 + rowb, H1, GW * 2048);
        bulk_commit();
      }
      float acc[GW][4][4];      // o^T: [group][8-token tile][fragment]
#pragma unroll
      for (int g = 0; g < GW; ++g)
#pragma unroll
        for (int n = 0; n < 4; ++n) acc[g][n][0] = acc[g][n][1] = acc[g][n][2] = acc[g][n][3] = 0.f;
      const uint32_t aH = smem_u32(H0) + arow * 128, aQ = smem_u32(d.QG) + (32 * part + brow) * 128;
      uint32_t a[2][GW][4], b[2][2][4];
      auto load_q = [&](int ks, uint32_t (&fa)[GW][4], uint32_t (&f)[2][4]) {
#pragma unroll
        for (int g = 0; g < GW; ++g) ldsm_x4(fa[g], aH + g * 2048 + (ks >> 2) * (VS * 128) + (((2 * (ks & 3) + l16) ^ lr) << 4));
#pragma unroll
        for (int n = 0; n < 2; ++n) ldsm_x4(f[n], aQ + (ks >> 2) * 8192 + n * 2048 + (((2 * (ks & 3) + l8) ^ lr) << 4));
      };
      load_q(0, a[0], b[0]);
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        if (ks < 7) load_q(ks + 1, a[(ks + 1) & 1], b[(ks + 1) & 1]);
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int g = 0; g < GW; ++g) {
            mma16816(acc[g][2 * n], a[ks & 1][g], b[ks & 1][n][0], b[ks & 1][n][1]);
            mma16816(acc[g][2 * n + 1], a[ks & 1][g], b[ks & 1][n][2], b[ks & 1][n][3]);
          }
      }
      if (stores) bulk_wait_read<0>();
      __syncwarp();
      if (lane < GW) mbar_arrive(&s.hFree[i & 1][g0 + lane]);
      if (!mbar_wait(&s.vReady[i & 1][g0], ph) || (GW > 1 && !mbar_wait(&s.vReady[i & 1][g0 + GW - 1], ph))) { ok = false; break; }
      if (stores) {
        bulk_s2g(p.VNEWT + tile * TILE_VT + static_cast<size_t>(v0) * 128 + rowb, VN, GW * 2048);
        bulk_commit();
      }
      const uint32_t aV = smem_u32(VN) + arow * 128, aA = smem_u32(d.AQK) + (32 * part + brow) * 128;
      // Aqk is lower triangular: 16-token tile 2 part + n needs the k-steps up to its own
      auto load_a = [&](int t, uint32_t (&fa)[GW][4], uint32_t (&f)[2][4]) {
#pragma unroll
        for (int g = 0; g < GW; ++g) ldsm_x4(fa[g], aV + g * 2048 + (((2 * t + l16) ^ lr) << 4));
#pragma unroll
        for (int n = 0; n < 2; ++n)
          if (2 * part + n >= t) ldsm_x4(f[n], aA + n * 2048 + (((2 * t + l8) ^ lr) << 4));
      };
      load_a(0, a[0], b[0]);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        if (t >= 2 && part == 0) break;      // (the warp's number: uniform)
        if (t == 0 || (t < 3 && part)) load_a(t + 1, a[(t + 1) & 1], b[(t + 1) & 1]);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          if (2 * part + n < t) continue;
#pragma unroll
          for (int g = 0; g < GW; ++g) {
            mma16816(acc[g][2 * n], a[t & 1][g], b[t & 1][n][0], b[t & 1][n][1]);
            mma16816(acc[g][2 * n + 1], a[t & 1][g], b[t & 1][n][2], b[t & 1][n][3]);
          }
        }
      }
      if (stores) bulk_wait_read<0>();
      __syncwarp();
      if (lane < GW) mbar_arrive(&s.vFree[i & 1][g0 + lane]);
      if (lane == 0) mbar_arrive(&s.empty[i % ST]);
      // o^T -> o[t][16 GW v] through shared memory (transposed stores; with 64-byte rows the pieces are swizzled), then whole rows
      constexpr int PR = 2 * GW;      // 16-byte pieces of a row
      unsigned char* const oS = s.oS[warp - 2 * NP];
      auto piece = [](int r, int pc) { return (r * PR + (GW == 2 ? pc ^ ((r >> 1) & 3) : pc)) << 4; };
#pragma unroll
      for (int g = 0; g < GW; ++g)
#pragma unroll
        for (int n = 0; n < 4; n += 2)
          stsm_x4_t(smem_u32(oS) + piece(8 * (n + l16) + lr, 2 * g + l8), pack_bf16(acc[g][n][0], acc[g][n][1]),
                    pack_bf16(acc[g][n][2], acc[g][n][3]), pack_bf16(acc[g][n + 1][0], acc[g][n + 1][1]), pack_bf16(acc[g][n + 1][2], acc[g][n + 1][3]));
      __syncwarp();
      const long long tok0 = tok_begin + static_cast<long long>(i) * C;
      const int len = static_cast<int>(tok_end - tok0 < C ? tok_end - tok0 : C);
      const int vcol = v0 + 16 * g0 + 8 * (lane & (PR - 1));
#pragma unroll
      for (int j = 0; j < PR; ++j) {
        const int r = (32 / PR) * j + lane / PR, t = 32 * part + r;
        const uint4 x = *reinterpret_cast<const uint4*>(oS + piece(r, lane & (PR - 1)));
        if (t < len && vcol < p.vc) *reinterpret_cast<uint4*>(p.o + (static_cast<size_t>(tok0 + t) * p.H + h) * p.vc + vcol) = x;
      }
      __syncwarp();      // the staging rows are rewritten by the next chunk
    }
    if (!ok) gave_up(KDA_STATUS_SCAN_MMA_WAIT);
    if (lane == 0) bulk_wait<0>();      // the stores read shared memory that dies with the CTA
  }
}

namespace {
template <int NP>
int launch_np(const ScanParams& p, int units, cudaStream_t st) {
  static DeviceOnce once;
  const int smem = static_cast<int>(sizeof(ScanSmem<NP>)) + 1024;
  const int rc = once.run([&] { return cudaFuncSetAttribute(kda_chunk_scan_kernel<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); });
  if (rc != KDA_OK) return rc;
  return static_cast<int>(launch_chained(kda_chunk_scan_kernel<NP>, units * (8 / NP), ScanCfg<NP>::THREADS, smem, st, p));
}
}  // namespace

// `requested` CTAs per unit (1, 4; 0: four, then two, while the grid stays within one CTA per SM: a chunk costs 1.3, 1.9 and 2.3 us
// with four, two and one CTA per unit, and two CTAs on one SM would share it)
int launch_scan(const ScanParams& p, int units, int requested, cudaStream_t st) {
  const int sms = sm_count();
  if (requested == 4 || (requested == 0 && 4 * units <= sms)) return launch_np<2>(p, units, st);
  if (requested == 0 && 2 * units <= sms) return launch_np<4>(p, units, st);
  return launch_scan_tc(p, units, st);
}

}  // namespace kda
