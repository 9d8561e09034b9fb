// Forward state scan of chunked KDA with the fp32 state in registers (sm_100a).
//
//   v_new = u - w h;   o = qg h + Aqk v_new;   h <- Diag(Gam_last) h + kg^T v_new          per chunk of 64 tokens, in order
//
// The recurrence is independent per value column.  A STATE WARP owns 16 of them and holds hT[16 v][128 k] as mma.sync accumulators (64
// fp32 registers a thread) for the whole sequence: an accumulator fragment is, rounded to bf16, the A fragment of the next
// product, so the chunk-to-chunk chain  hT -> v_part^T = hT w^T -> v_new^T = u^T - v_part^T -> hT += v_new^T kg  runs inside one warp,
// without a barrier or a trip through memory.  Its OUTPUT WARP forms o^T = hT qg^T + v_new^T Aqk^T beside it from the bf16 images of hT and
// v_new^T that the state warp leaves in shared memory; in training these are the chunk's HS and VNEWT tiles and leave from there.
// A CTA has 2 or 4 such pairs (32 or 64 value columns of one (sequence, head) unit): as few as keep the grid within one CTA per
// SM.  Operand tiles arrive through a ring of bulk copies.
//
// What bounds it: the chain of one warp, 128 m16n8k16 products a chunk with their operand loads.  The same scan with the
// state in tensor memory and tcgen05 products spends its time on hand-overs between the issuing thread and the warps (290 cycles a
// round besides 56 per product).  32 units, 512 chunks: 766 -> 652 us; one unit of 128 value columns per CTA stays on tensor memory
// (kda_chunk_scan_tc.cu): eight pairs on one SM wait for its shared memory, 260 against 160 us at 64 chunks.  Every layout
// forms the same sums: the bits do not depend on it.
#include "kda_chunk.cuh"
#include "kda_device.cuh"
#include "kda_scan.cuh"

namespace kda {

namespace {

template <int NP>
struct ScanCfg {
  static constexpr int VS = 16 * NP;                         // value columns of the CTA
  static constexpr int STAGES = NP == 2 ? 3 : 2;
  static constexpr int THREADS = 64 * NP + 32;               // one more warp issues the copies
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
  unsigned char H[2][16 * NP * 128];      // bf16 hT: two spans [VS v][64 k] (= the CTA's rows of the HS tile)
  unsigned char VN[16 * NP * 128];        // bf16 v_new^T [VS v][64 t] (= its rows of the VNEWT tile)
  unsigned char oS[NP][C * 32];           // o of a pair: [64 t][16 v]
  uint64_t full[ScanCfg<NP>::STAGES], empty[ScanCfg<NP>::STAGES];
  uint64_t hReady[NP], vReady[NP], hFree[NP], vFree[NP];
};
template <int NP>
constexpr unsigned SCAN_TX = 3 * TILE_TK + TILE_TT + 16 * NP * 128 + TILE_GL;
static_assert(sizeof(ScanStage<2>) % 1024 == 0 && sizeof(ScanStage<4>) % 1024 == 0, "stage alignment");
static_assert(sizeof(ScanSmem<2>) + 1024 <= 227 * 1024 && sizeof(ScanSmem<4>) + 1024 <= 227 * 1024, "ScanSmem too large");

__device__ __forceinline__ void stsm_x4_t(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

}  // namespace

template <int NP>
__global__ void __launch_bounds__(ScanCfg<NP>::THREADS, 1) kda_chunk_scan_kernel(const ScanParams p) {
  chain_point();
  using Cfg = ScanCfg<NP>;
  constexpr int VS = Cfg::VS, ST = Cfg::STAGES;
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
      mbar_init(&s.empty[i], 2 * NP);
    }
    for (int i = 0; i < NP; ++i) {
      mbar_init(&s.hReady[i], 1);
      mbar_init(&s.vReady[i], 1);
      mbar_init(&s.hFree[i], 1);
      mbar_init(&s.vFree[i], 1);
    }
    fence_mbar_init();
  }
  __syncthreads();
  auto gave_up = [&](unsigned bit) {
    if (lane == 0) atomicOr(p.status, bit);
  };

  if (warp == 2 * NP) {
    // ================= copies =================
    if (lane == 0) {
      for (int i = 0; i < nchunks; ++i) {
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
    }
    return;      // (nothing waits for this warp; the CTA's memory lives until the others leave)
  }
  const int pair_ = warp < NP ? warp : warp - NP;
  const uint32_t rowb = static_cast<uint32_t>(16 * pair_) * 128u;                 // the pair's 16 rows in [VS][64] tiles
  const size_t sb = (static_cast<size_t>(seq) * p.H + h) * p.kc * p.vc;
  const int va = v0 + 16 * pair_ + gid, vb = va + 8;                              // state warp: its accumulator rows

  if (warp < NP) {
    // ================= state warp =================
    float hs[16][4];      // [8-column tile of k][fragment]
#pragma unroll
    for (int n = 0; n < 16; ++n) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int k = 8 * n + 2 * tig + (e & 1), v = e < 2 ? va : vb;
        hs[n][e] = p.h0 && k < p.kc && v < p.vc ? __ldg(p.h0 + sb + static_cast<size_t>(k) * p.vc + v) : 0.f;
      }
    }
    // ldmatrix addresses inside a swizzled tile: row * 128 + ((piece ^ row) & 7) * 16; the row part is fixed per lane
    const int wrow = (lane & 7) + ((lane >> 4) << 3), wpc = (lane >> 3) & 1;      // W: rows t of two 8-row tiles, pieces k
    const int krow = (lane & 7) + (((lane >> 3) & 1) << 3), kpc = lane >> 4;      // KG (transposed read): rows t, pieces k
    bool ok = true;
    for (int i = 0; i < nchunks; ++i) {
      ScanStage<NP>& d = s.st[i % ST];
      if (!mbar_wait(&s.full[i % ST], (i / ST) & 1) || (i > 0 && !mbar_wait(&s.hFree[pair_], (i - 1) & 1))) { ok = false; break; }
      float acc[8][4];      // v_part^T: [8-token tile][fragment]
#pragma unroll
      for (int n = 0; n < 8; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
      const uint32_t aW = smem_u32(d.W) + wrow * 128;
      unsigned char* const hA = s.H[0] + rowb + gid * 128 + tig * 4;
      // B fragments are loaded one step ahead of their products: one warp per scheduler, nobody else hides their latency
      uint32_t b[2][4][4];
      auto load_w = [&](int ks, uint32_t (&f)[4][4]) {      // w[t][k] of eight 8-token tiles
#pragma unroll
        for (int n = 0; n < 4; ++n) ldsm_x4(f[n], aW + (ks >> 2) * 8192 + n * 2048 + (((2 * (ks & 3) + wpc) ^ (lane & 7)) << 4));
      };
      load_w(0, b[0]);
      uint32_t ut[8][2];      // u^T, needed behind product 1
      {
        const unsigned char* const uA = d.UT + rowb + gid * 128 + tig * 4;
#pragma unroll
        for (int n = 0; n < 8; ++n) {
          ut[n][0] = *reinterpret_cast<const uint32_t*>(uA + ((n ^ gid) << 4));
          ut[n][1] = *reinterpret_cast<const uint32_t*>(uA + ((n ^ gid) << 4) + 1024);
        }
      }
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        if (ks < 7) load_w(ks + 1, b[(ks + 1) & 1]);
        const float2 g0 = *reinterpret_cast<const float2*>(&d.GL[16 * ks + 2 * tig]), g1 = *reinterpret_cast<const float2*>(&d.GL[16 * ks + 8 + 2 * tig]);
        uint32_t a[4];
        a[0] = pack_bf16(hs[2 * ks][0], hs[2 * ks][1]);
        a[1] = pack_bf16(hs[2 * ks][2], hs[2 * ks][3]);
        a[2] = pack_bf16(hs[2 * ks + 1][0], hs[2 * ks + 1][1]);
        a[3] = pack_bf16(hs[2 * ks + 1][2], hs[2 * ks + 1][3]);
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          mma16816(acc[2 * n], a, b[ks & 1][n][0], b[ks & 1][n][1]);
          mma16816(acc[2 * n + 1], a, b[ks & 1][n][2], b[ks & 1][n][3]);
        }
        // the bf16 image of the state; both rows have row & 7 == gid
        const uint32_t pc0 = ((2 * (ks & 3)) ^ gid) << 4, pc1 = ((2 * (ks & 3) + 1) ^ gid) << 4, span = (ks >> 2) * (VS * 128);
        *reinterpret_cast<uint32_t*>(hA + span + pc0) = a[0];
        *reinterpret_cast<uint32_t*>(hA + span + pc0 + 1024) = a[1];
        *reinterpret_cast<uint32_t*>(hA + span + pc1) = a[2];
        *reinterpret_cast<uint32_t*>(hA + span + pc1 + 1024) = a[3];
        // hT *= Gam_last
        hs[2 * ks][0] *= g0.x; hs[2 * ks][1] *= g0.y; hs[2 * ks][2] *= g0.x; hs[2 * ks][3] *= g0.y;
        hs[2 * ks + 1][0] *= g1.x; hs[2 * ks + 1][1] *= g1.y; hs[2 * ks + 1][2] *= g1.x; hs[2 * ks + 1][3] *= g1.y;
      }
      fence_proxy_async();      // (the image also leaves by a bulk store in training)
      __syncwarp();
      if (lane == 0) mbar_arrive(&s.hReady[pair_]);
      if (i > 0 && !mbar_wait(&s.vFree[pair_], (i - 1) & 1)) { ok = false; break; }
      // kg fragments of the update: step 2 t + half covers 16 tokens and 64 key columns
      const uint32_t aK = smem_u32(d.KG) + krow * 128;
      auto load_k = [&](int st, uint32_t (&f)[4][4]) {
#pragma unroll
        for (int n = 0; n < 4; ++n) ldsm_x4_t(f[n], aK + (st & 1) * 8192 + (st >> 1) * 2048 + (((2 * n + kpc) ^ (lane & 7)) << 4));
      };
      load_k(0, b[0]);
      // v_new^T = u^T - v_part^T, as bf16: the A fragments of the update and the image for the output warp
      uint32_t vn[4][4];
      unsigned char* const nA = s.VN + rowb + gid * 128 + tig * 4;
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        const float2 ua = unpack_bf16(ut[n][0]), ub = unpack_bf16(ut[n][1]);
        vn[n >> 1][(n & 1) * 2] = pack_bf16(ua.x - acc[n][0], ua.y - acc[n][1]);
        vn[n >> 1][(n & 1) * 2 + 1] = pack_bf16(ub.x - acc[n][2], ub.y - acc[n][3]);
      }
      // hT += v_new^T kg
#pragma unroll
      for (int st = 0; st < 8; ++st) {
        if (st < 7) load_k(st + 1, b[(st + 1) & 1]);
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          mma16816(hs[8 * (st & 1) + 2 * n], vn[st >> 1], b[st & 1][n][0], b[st & 1][n][1]);
          mma16816(hs[8 * (st & 1) + 2 * n + 1], vn[st >> 1], b[st & 1][n][2], b[st & 1][n][3]);
        }
        if (st == 0) {      // beside the products
#pragma unroll
          for (int n = 0; n < 8; ++n) {
            *reinterpret_cast<uint32_t*>(nA + ((n ^ gid) << 4)) = vn[n >> 1][(n & 1) * 2];
            *reinterpret_cast<uint32_t*>(nA + ((n ^ gid) << 4) + 1024) = vn[n >> 1][(n & 1) * 2 + 1];
          }
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) mbar_arrive(&s.vReady[pair_]);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&s.empty[i % ST]);
    }
    if (!ok) gave_up(KDA_STATUS_SCAN_LOAD_WAIT);
    else if (p.ht) {
#pragma unroll
      for (int n = 0; n < 16; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int k = 8 * n + 2 * tig + (e & 1), v = e < 2 ? va : vb;
          if (k < p.kc && v < p.vc) p.ht[sb + static_cast<size_t>(k) * p.vc + v] = hs[n][e];
        }
    }
    return;
  }

  // ================= output warp =================
  {
    const int arow = (lane & 7) + (((lane >> 3) & 1) << 3), apc = lane >> 4;      // A: rows v, pieces k
    const int brow = (lane & 7) + ((lane >> 4) << 3), bpc = (lane >> 3) & 1;      // B: rows t of two 8-row tiles
    bool ok = true;
    for (int i = 0; i < nchunks; ++i) {
      ScanStage<NP>& d = s.st[i % ST];
      const size_t tile = static_cast<size_t>(c_begin + i) * p.H + h;
      if (!mbar_wait(&s.full[i % ST], (i / ST) & 1) || !mbar_wait(&s.hReady[pair_], i & 1)) { ok = false; break; }
      if (p.HS && lane == 0) {
        bulk_s2g(p.HS + tile * TILE_VK + static_cast<size_t>(v0) * 128 + rowb, s.H[0] + rowb, 2048);
        bulk_s2g(p.HS + tile * TILE_VK + 16384 + static_cast<size_t>(v0) * 128 + rowb, s.H[1] + rowb, 2048);
        bulk_commit();
      }
      float acc[8][4];
#pragma unroll
      for (int n = 0; n < 8; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
      const uint32_t aH = smem_u32(s.H[0]) + rowb + arow * 128, aQ = smem_u32(d.QG) + brow * 128;
      uint32_t a[2][4], b[2][4][4];
      auto load_q = [&](int ks, uint32_t (&fa)[4], uint32_t (&f)[4][4]) {
        ldsm_x4(fa, aH + (ks >> 2) * (VS * 128) + (((2 * (ks & 3) + apc) ^ (lane & 7)) << 4));
#pragma unroll
        for (int n = 0; n < 4; ++n) ldsm_x4(f[n], aQ + (ks >> 2) * 8192 + n * 2048 + (((2 * (ks & 3) + bpc) ^ (lane & 7)) << 4));
      };
      load_q(0, a[0], b[0]);
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        if (ks < 7) load_q(ks + 1, a[(ks + 1) & 1], b[(ks + 1) & 1]);
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          mma16816(acc[2 * n], a[ks & 1], b[ks & 1][n][0], b[ks & 1][n][1]);
          mma16816(acc[2 * n + 1], a[ks & 1], b[ks & 1][n][2], b[ks & 1][n][3]);
        }
      }
      if (p.HS && lane == 0) bulk_wait_read<0>();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s.hFree[pair_]);
      if (!mbar_wait(&s.vReady[pair_], i & 1)) { ok = false; break; }
      if (p.VNEWT && lane == 0) {
        bulk_s2g(p.VNEWT + tile * TILE_VT + static_cast<size_t>(v0) * 128 + rowb, s.VN + rowb, 2048);
        bulk_commit();
      }
      const uint32_t aV = smem_u32(s.VN) + rowb + arow * 128, aA = smem_u32(d.AQK) + brow * 128;
      auto load_a = [&](int t, uint32_t (&fa)[4], uint32_t (&f)[4][4]) {      // Aqk is lower triangular: token tiles before a k-step see nothing of it
        ldsm_x4(fa, aV + (((2 * t + apc) ^ (lane & 7)) << 4));
#pragma unroll
        for (int n = t; n < 4; ++n) ldsm_x4(f[n], aA + n * 2048 + (((2 * t + bpc) ^ (lane & 7)) << 4));
      };
      load_a(0, a[0], b[0]);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        if (t < 3) load_a(t + 1, a[(t + 1) & 1], b[(t + 1) & 1]);
#pragma unroll
        for (int n = t; n < 4; ++n) {
          mma16816(acc[2 * n], a[t & 1], b[t & 1][n][0], b[t & 1][n][1]);
          mma16816(acc[2 * n + 1], a[t & 1], b[t & 1][n][2], b[t & 1][n][3]);
        }
      }
      if (p.VNEWT && lane == 0) bulk_wait_read<0>();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&s.vFree[pair_]);
        mbar_arrive(&s.empty[i % ST]);
      }
      // o^T -> o[t][16 v] through shared memory (transposed stores), then 32 contiguous bytes per row
      unsigned char* const oS = s.oS[pair_];
      const uint32_t aO = smem_u32(oS) + (lane & 7) * 32 + (((lane >> 3) & 1) << 4) + ((lane >> 4) << 8);
#pragma unroll
      for (int n = 0; n < 8; n += 2)
        stsm_x4_t(aO + n * 256, pack_bf16(acc[n][0], acc[n][1]), pack_bf16(acc[n][2], acc[n][3]), pack_bf16(acc[n + 1][0], acc[n + 1][1]),
                  pack_bf16(acc[n + 1][2], acc[n + 1][3]));
      __syncwarp();
      const long long tok0 = tok_begin + static_cast<long long>(i) * C;
      const int len = static_cast<int>(tok_end - tok0 < C ? tok_end - tok0 : C);
      const int vcol = v0 + 16 * pair_ + 8 * (lane & 1);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int t = 16 * j + (lane >> 1);
        const uint4 x = *reinterpret_cast<const uint4*>(oS + t * 32 + 16 * (lane & 1));
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

// `requested` CTAs per unit (1, 4; 0: as many as keep the grid within one CTA per SM)
int launch_scan(const ScanParams& p, int units, int requested, cudaStream_t st) {
  const int sms = sm_count();
  if (requested == 4 || (requested == 0 && 4 * units <= sms)) return launch_np<2>(p, units, st);
  if (requested == 0 && 2 * units <= sms) return launch_np<4>(p, units, st);
  return launch_scan_tc(p, units, st);
}

}  // namespace kda
