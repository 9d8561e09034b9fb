// Per-chunk KDA backward on the 5th-generation tensor cores (tcgen05 + TMEM), sm_100a.
//
// One persistent CTA per SM walks (chunk, head) tiles.  Every matrix product of the chunk's backward is a
// tcgen05.mma issued by one thread, with bf16 operands in 128-byte-swizzled shared-memory tiles and fp32
// accumulators in tensor memory.  The products are arranged so that the accumulators that end up in dq / dk
// have the KEY COLUMN as their TMEM lane ("transposed": D^T[kk][t]); a thread then owns one key column, which
// is exactly what the last phase needs (pairwise decay inside the diagonal 16x16 blocks, reverse cumsum for
// dg) -- no shared-memory transposition of fp32 matrices is needed.  The 64 x 64 products of the backward
// through Tm = (I + Akk)^-1 use M = 64 (token row = TMEM lane).
//
// Phases per tile (G = in-chunk cumsum of g in the log2 domain, Gam = 2^G, D[t,j] = 2^(G_t - G_j)):
//   A   dqg^T = h dO^T,  dw^T = -h dv_new^T,  dkg^T = dh' v_new^T      (M=128 kk, N=64 t, K=128 v)
//       dAqk  = dO v_new^T                                             (M=64 t,  N=64 j)
//   B1  dTm = du (beta v)^T + dw (beta k Gam)^T                        (M=64)
//       dbv^T = du^T Tm,  dbk^T = dw^T Tm                              (M=128, N=64 t, K=64 t')
//   B2  X = dTm Tm^T      B3  Y = Tm^T X,  dAkk = -tril(Y, -1)
//   C   off-diagonal 16x16 blocks of the intra-chunk terms, decay factored around a row that lies between
//       j and t (both factors <= 1):  Cq^T, Cp^T (reference = first row of t's block),
//       Cn^T (reference = last row of j's block)                       (M=128 kk, N=32 (q and p) or 16, K=16..48)
//   D   per key column: diagonal blocks pairwise with running products of 2^(g), dG = q dq + k (dk+ - dk-),
//       dg = reverse cumsum, final dq, dk, dg;  dbeta from  <Tm, dTm_raw> + <dAkk, raw kk>.
//
// What bounds it: the work around the products, about 52 k warp instructions a tile (22 to 25 k cycles), of which the last phase has a third; the
// waits for products are filled with it: the operands of phase C are built under B1 and B2, the last phase's parts that need only the
// accumulators of A and B1 run under B2, B3 and C, and between those a warp hands its share of an operand over instead of meeting everybody.
// q and k are interleaved into one word per element once they have arrived, and the last phase adds up dq and dk+ as register pairs, one
// instruction for both sides.  Row numbers are left to the uniform registers.
// 8 x 8192 tokens x 32 heads, whole step: 6.05 ms with 61 k instructions -> 5.91; operands handed over 5.81; dg from registers and the next q, k early
// 5.73.  Packed documents with the L2 norm 7.13 -> 6.78 ms (its epilogue reads q and k where they are instead of from global memory); 2 x 1000 x 8
// heads of 64: 108 -> 98 us, of which 9 are the code's size: 135 KB with every issue loop and wait unrolled, 85 now, and a short step fetches
// all of it anew.  (One scaled copy of each operand row instead of one per reference row halves the builds, 5 %.  It rounds to bf16 at other points:
// nearer to fp32, but dA_log moves by 4 % of itself, and a gradient of the layer's call may move by 2 % from one build to the next.)
#include "kda_chunk_bwd.cuh"
#include "kda_device.cuh"
#include "kda_f32x2.cuh"
#include "kda_umma.cuh"

#include <type_traits>

namespace kda {

namespace {

constexpr uint32_t SPAN = 16384;    // bytes of one [128 rows][64] tile
constexpr int NT = 512;             // threads per CTA: 16 warps = 4 TMEM lane quadrants x 4 column parts

struct TcSmem {
  // ---- SW128 operand tiles; every offset is a multiple of 1024 -------------------------------------------------
  unsigned char HS[TILE_VK];    // A.  later: KG = k Gam [64 j][128 kk] (16K) | DWT = dw^T [128 kk][64 t] (16K);  from B1's end: DT (8K) | X (8K) | qL, J > 0 (12K)
  unsigned char DH[TILE_VK];    // A.  later: DAK, DAQ (16K, eight rows of one behind eight of the other) |
  unsigned char VN[TILE_VT];    // A.                                                  | with the rest of DH and dO 48K: kR (24K), qL, kL of J = 0 (12K each)
  unsigned char dO[TILE_TK];    // A (two [64 t][64 v] sub-tiles).  later: see VN
  unsigned char DVN[TILE_VT];   // A, B1.  later: dv staging, four parts [64 t][32 v]
  unsigned char V[TILE_TK];     // B1 (two [64 j][64 v] sub-tiles).  B2, C: kL, J > 0.  D: dq staging [64][128]
  unsigned char TI[TILE_TT];    // B1..B3.  D (with RKK): dk staging [64][128]
  unsigned char RKK[TILE_TT];   // post-B3
  // ---- plain arrays -----------------------------------------------------------------------------------------------
  union {
    struct {
      __nv_bfloat16 q[C * KD];      // [64][128], as they arrive
      __nv_bfloat16 k[C * KD];
    };
    uint32_t qk[C * KD];            // from phase B1 on: (q, k) of an element in one word, q in the low half
  };
  float G[C * KD];              // log2-domain cumsum of g (g of the NEXT tile arrives here during phase D)
  float2 Ad[4][16][18];         // diagonal blocks: (a1, a2) = (scale dAqk, beta dAkk); rows 16-byte aligned
  float beta[C];
  float hdh[KD];                // sum over v of h dh'
  union {
    float hdh_part[8][KD];      // its partial sums (phase A only)
    struct {
      float dbp[8][C];          // dbeta partial sums (from phase B1 on)
      float dglp[4][KD];        // partial sums over rows of k dk_end (phase D)
    };
  };
  float carry[4][KD];           // block totals of the reverse cumsum
  uint64_t barS, barG, barQ, barB, barM;      // (in this order: drained together)
  uint64_t barT;                // every warp's share of an operand tile of B2, B3 or C is written
  long long ci_tok0[2];         // first token and length of the chunk of the current / next tile (written by thread 0)
  int ci_len[2];
  uint32_t tmem_slot;
};
static_assert(sizeof(TcSmem) + 1024 <= 227 * 1024, "TcSmem too large");

// TMEM columns (512 allocated): 64 each; in phase C 32 per row block I = 1..3 for Cq, Cp (eight columns of one behind eight of the other), 48 for Cn
constexpr int C_DQG = 0, C_DKG = 64, C_DW = 128 /* later dbk^T */, C_DAQ = 192 /* later dTm */, C_XY = 320, C_DBV = 384;
constexpr int C_CQP = 192, C_CN = 288, C_DBK = C_DW;

// eight floats -> one 16-byte piece of bf16
__device__ __forceinline__ uint4 pack8(const float* v) {
  return make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
}
// address of the 16-byte piece `chunk` (0..7) of row `row` in an SW128 tile
__device__ __forceinline__ unsigned char* sw_piece(unsigned char* tile, int row, int chunk) {
  return tile + row * 128 + (((chunk ^ row) & 7) << 4);
}
// a word of the interleaved tile
__device__ __forceinline__ float q_of(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float k_of(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

}  // namespace

// L2: q, k are L2-normalised rows and dq, dk leave through the normalisation's backward (fla/modules/l2norm.py:190-240).
template <bool L2>
__global__ void __launch_bounds__(512, 1) kda_chunk_bwd_main_tc_kernel(const __grid_constant__ MainParams p) {
  chain_point();
  extern __shared__ unsigned char smem_raw[];
  TcSmem& s = *reinterpret_cast<TcSmem*>(smem_raw + pad_to_1024(smem_raw));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int total_tiles = p.map.total() * p.H;      // the launch checks that it fits

  // aliases inside the tile regions
  unsigned char* const sKG = s.HS;
  unsigned char* const sDWT = s.HS + SPAN;
  unsigned char* const sDT = s.HS;
  unsigned char* const sX = s.HS + 8192;
  unsigned char* const sDA = s.DH;      // rows t of dAqk at da_row(t), of dAkk eight rows behind: one product takes the same rows of both
  auto da_row = [](int t) { return 2 * (t & 56) + (t & 7); };
  unsigned char* const sKR = s.DH + 16384;
  constexpr uint32_t KR_SPAN = 12288, L_SPAN = 6144;      // between the two 64-column spans of kR; of qL, kL
  unsigned char* const sQL0 = sKR + 2 * KR_SPAN;           // J = 0
  unsigned char* const sKL0 = sQL0 + 2 * L_SPAN;
  unsigned char* const sQL1 = s.HS + 16384;                // J > 0
  unsigned char* const sKL1 = s.V;
  __nv_bfloat16* const stq = reinterpret_cast<__nv_bfloat16*>(s.V);      // phase D: dq, dk before their coalesced stores
  __nv_bfloat16* const stk = reinterpret_cast<__nv_bfloat16*>(s.TI);

  // thread 0: the phase-A operands of tile idx -- state tiles by bulk copy, dO by two tiled loads (64 value columns each)
  // thread 0: first token and length of tile idx's chunk into slot (two dependent global loads: done early, off the
  // critical path, while phase B2 executes and the other warps build operands)
  auto stash_chunk = [&](int idx, int slot) {
    const ChunkInfo cn = p.map.info(idx / p.H);
    s.ci_tok0[slot] = cn.tok0;
    s.ci_len[slot] = cn.len;
  };
  // copy `which` of the seven that bring tile idx's state tiles and dO (barS) and g (barG); after stash_chunk(idx, slot).  One warp issues
  // one each: a copy costs its thread 200 cycles.
  auto fetch = [&](int idx, int slot, int which) {
    const size_t tl = static_cast<size_t>(idx);
    const int hh = idx % p.H, tk = static_cast<int>(s.ci_tok0[slot]);
    mbar_expect_tx(which < 6 ? &s.barS : &s.barG, which < 2 ? TILE_VK : (which < 4 ? TILE_VT : (which < 6 ? TILE_TK / 2 : C * KD * 4)));
    switch (which) {
      case 0: bulk_g2s(s.HS, p.HS + tl * TILE_VK, TILE_VK, &s.barS); break;
      case 1: bulk_g2s(s.DH, p.DH + tl * TILE_VK, TILE_VK, &s.barS); break;
      case 2: bulk_g2s(s.VN, p.VNEWT + tl * TILE_VT, TILE_VT, &s.barS); break;
      case 3: bulk_g2s(s.DVN, p.DVNEWT + tl * TILE_VT, TILE_VT, &s.barS); break;
      case 4: tma_load_rows(s.dO, &p.tm_do, 0, hh, tk, &s.barS); break;
      case 5: tma_load_rows(s.dO + 8192, &p.tm_do, 64, hh, tk, &s.barS); break;
      default: tma_load_rows(s.G, &p.tm_g, 0, hh, tk, &s.barG); break;
    }
  };
  // copy `which` of the six whose memory the previous tile used to its end: q, k (barQ, needed behind phase A; asked for when it ends), Tm, raw
  // kk, v (barB, from phase B1 on; they land where it staged dq and dk, and warps 2 and 3, which stored those, bring them)
  auto fetch_late = [&](int idx, int h, int tk, int which) {
    const size_t tl = static_cast<size_t>(idx);
    mbar_expect_tx(which < 2 ? &s.barQ : &s.barB, which < 2 ? TILE_TK : TILE_TT);
    switch (which) {
      case 0: tma_load_rows(s.k, &p.tm_k, 0, h / p.grp, tk, &s.barQ); break;
      case 1: tma_load_rows(s.q, &p.tm_q, 0, h / p.grp, tk, &s.barQ); break;
      case 2: bulk_g2s(s.TI, p.TI + tl * TILE_TT, TILE_TT, &s.barB); break;
      case 3: bulk_g2s(s.RKK, p.RKK + tl * TILE_TT, TILE_TT, &s.barB); break;
      case 4: tma_load_rows(s.V, &p.tm_v, 0, h, tk, &s.barB); break;
      default: tma_load_rows(s.V + 8192, &p.tm_v, 64, h, tk, &s.barB); break;
    }
  };
  auto dv_stage = [&](int i) { return s.DVN + 4096 * i; };      // [64 t][32 v] of dv
  // rows of a partial chunk beyond its length hold the next sequence's tokens after a tiled load: clear them
  auto zero_rows_sw = [&](unsigned char* tile, int len) {          // [64][64] bf16 sub-tile, 128-byte rows
#pragma unroll 1
    for (int i = len * 8 + tid; i < C * 8; i += NT) *reinterpret_cast<uint4*>(tile + i * 16) = make_uint4(0u, 0u, 0u, 0u);
  };
  if (tid == 0) {
    mbar_init(&s.barS, 6);      // one arrival per copy
    mbar_init(&s.barG, 1);
    mbar_init(&s.barQ, 2);
    mbar_init(&s.barB, 4);
    mbar_init(&s.barM, 1);
    mbar_init(&s.barT, NT / 32);
    fence_mbar_init();
    if (static_cast<int>(blockIdx.x) < total_tiles) {
      stash_chunk(blockIdx.x, 0);
      for (int i = 0; i < 7; ++i) fetch(blockIdx.x, 0, i);
      fetch_late(blockIdx.x, blockIdx.x % p.H, static_cast<int>(s.ci_tok0[0]), 0);
      fetch_late(blockIdx.x, blockIdx.x % p.H, static_cast<int>(s.ci_tok0[0]), 1);
    }
  }
  __syncwarp();
  if (warp == 0) umma::tmem_alloc(&s.tmem_slot, 512);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tb = __shfl_sync(0xffffffffu, s.tmem_slot, 0);          // warp-uniform for the compiler
  const int warp_u = __shfl_sync(0xffffffffu, warp, 0);
  const uint32_t lead = lane == 0;                                      // the lane of warp 0 that issues the MMAs
  // TMEM lane quadrant of a warp: warp & 3; which 16 of the 64 columns: warp >> 2
  const uint32_t tq = tb + (static_cast<uint32_t>(32 * (warp_u & 3)) << 16);     // this warp's lanes

  // Operands of phase C, built while the phase-B products run (rows R of the stacked tiles):
  // kR_I[j][kk] = k_j 2^(G_r - G_j),  r = 16 I,  j < 16 I            rows stacked: I=1 -> 0..15, I=2 -> 16..47, I=3 -> 48..95
  // qL_J[t][kk] = scale q_t 2^(G_t - G_e), kL_J = k_t 2^(G_t - G_e), e = 16 J + 15, t >= 16 (J+1)
  //                                                                   rows: J=0 -> 0..47 of one tile, J=1 -> 0..31, J=2 -> 32..47 of another
  // A warp takes whole rows, a lane four key columns.  The row number is the same for the whole warp, so that it and the addresses that come of it are
  // left to the uniform registers: with items counted through per thread, a third of a row's instructions were its indices.
  auto four = [&](const void* rows, int row, int lane) { return reinterpret_cast<const unsigned char*>(rows) + row * (KD * 4) + lane * 16; };
  auto minus2 = [](const F4& x, const F4& y) {      // 2^(x - y)
    const f32x2 m1 = pair(-1.f, -1.f);
    const float2 a = halves(fma2(y.a, m1, x.a)), b = halves(fma2(y.b, m1, x.b));
    return F4{pair(ex2(a.x), ex2(a.y)), pair(ex2(b.x), ex2(b.y))};
  };
  auto put4 = [](unsigned char* dst, f32x2 a, f32x2 b) {
    const float2 x = halves(a), y = halves(b);
    *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16(x.x, x.y), pack_bf16(y.x, y.y));
  };
  auto betas = [&](int t, float (&b)[16]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 x = *reinterpret_cast<const float4*>(&s.beta[t + 4 * i]);
      b[4 * i] = x.x; b[4 * i + 1] = x.y; b[4 * i + 2] = x.z; b[4 * i + 3] = x.w;
    }
  };
  auto build_kR = [&](int first, int stride, int lane) {
    unsigned char* const dst = sKR + (lane >> 4) * KR_SPAN + (lane & 1) * 8;
#pragma unroll 1
    for (int R = first; R < 96; R += stride) {
      const int I = (R < 16) ? 1 : (R < 48 ? 2 : 3);
      const int j = R - (I == 1 ? 0 : (I == 2 ? 16 : 48));
      const uint4 w = *reinterpret_cast<const uint4*>(four(s.qk, j, lane));
      const F4 f = minus2(lds4(reinterpret_cast<const float*>(four(s.G, 16 * I, lane))), lds4(reinterpret_cast<const float*>(four(s.G, j, lane))));
      put4(dst + R * 128 + ((((lane >> 1) ^ R) & 7) << 4), mul2(pair(k_of(w.x), k_of(w.y)), f.a), mul2(pair(k_of(w.z), k_of(w.w)), f.b));
    }
  };
  auto build_qkL = [&](unsigned char* const tq_, unsigned char* const tk_, const bool first_J, int first, int stride, int lane) {
    const uint32_t off = (lane >> 4) * L_SPAN + (lane & 1) * 8;
    const f32x2 sc = pair(p.scale, p.scale);
#pragma unroll 1
    for (int R = first; R < 48; R += stride) {
      const int t = first_J || R >= 32 ? 16 + R : 32 + R;
      const int e = first_J ? 15 : (R < 32 ? 31 : 47);
      const uint4 w = *reinterpret_cast<const uint4*>(four(s.qk, t, lane));
      const F4 f = minus2(lds4(reinterpret_cast<const float*>(four(s.G, t, lane))), lds4(reinterpret_cast<const float*>(four(s.G, e, lane))));
      const uint32_t at = off + R * 128 + ((((lane >> 1) ^ R) & 7) << 4);
      put4(tq_ + at, mul2(mul2(pair(q_of(w.x), q_of(w.y)), sc), f.a), mul2(mul2(pair(q_of(w.z), q_of(w.w)), sc), f.b));
      put4(tk_ + at, mul2(pair(k_of(w.x), k_of(w.y)), f.a), mul2(pair(k_of(w.z), k_of(w.w)), f.b));
    }
  };

  // heads narrower than the tiles (zeros beyond kc, vc): products stop at the last 16 columns that hold something
  const int v_steps = (p.vc + 15) >> 4, k_steps = (p.kc + 15) >> 4;
  // Operands of B2, B3 and C go to the issuing warp through barT: a warp hands its share over and goes on with what does not depend on the product,
  // instead of meeting everybody at a barrier first (the products then start while dv, dbeta and the rest are still being written)
  uint32_t tph = 0;      // phase counter of barT
  auto hand_over = [&](int lane) {
    fence_proxy_async();
    umma::fence_before_sync();
    __syncwarp();
    if (lane == 0) mbar_arrive(&s.barT);
    ++tph;
  };
  auto handed_over = [&] {
    const bool ok = mbar_wait(&s.barT, (tph - 1) & 1);
    umma::fence_after_sync();
    return ok;
  };
  uint32_t mph = 0;      // phase counter of barM
  bool alive = true;
  int it = 0;
  // An opaque copy of the thread number, taken afresh in the phases: what is derived from it (shared-memory addresses above all) then
  // lives for that phase alone.  Kept across a tile it all together left the last phase 40 registers short, and its spills miss
  // the little L1 that is left beside 224 KB of shared memory.
  auto fresh_tid = [&] {
    int t = threadIdx.x;
    asm volatile("" : "+r"(t));
    return t;
  };
  for (int idx = blockIdx.x; idx < total_tiles && alive; idx += gridDim.x, ++it) {
    const int tid = fresh_tid(), lane = tid & 31, q4 = warp_u & 3, part = warp_u >> 2;
    const int h = idx % p.H;
    struct { int tok0; int len; } ci;
    ci.tok0 = static_cast<int>(s.ci_tok0[it & 1]);
    ci.len = s.ci_len[it & 1];
    const int len = ci.len;
    const int next_idx = idx + gridDim.x;
    long long* const dbg = (it == 2) ? p.dbg : nullptr;   // development aid: clocks of a steady-state tile

    KDA_DBG_CLOCK(dbg, 0);
    if (tid < C) cp_async4(&s.beta[tid], p.beta + static_cast<size_t>(ci.tok0 + (tid < len ? tid : 0)) * p.H + h, tid < len);
    cp_async_commit();
    if (!mbar_wait(&s.barS, it & 1)) {
      if (tid == 0) atomicOr(p.status, 32u);
      alive = false;
    }
    if (len < C) {                 // uniform over the CTA
      zero_rows_sw(s.dO, len);
      zero_rows_sw(s.dO + 8192, len);
      fence_proxy_async();
      __syncthreads();
    }
    umma::fence_after_sync();

    KDA_DBG_CLOCK(dbg, 1);
    // ---- sum_v h dh' (all warps, before warp 0 starts issuing) -------------------------------------------------------
    {
      const int kp = tid & 63, vq = tid >> 6;
      f32x2 acc = 0ull;
      const uint32_t lo = vk_off(16 * vq, 2 * kp);      // row 16 vq + i: + 128 i, and i & 7 in the swizzled piece
      auto wide = [](uint32_t u) { return pair(q_of(u), k_of(u)); };
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const uint32_t at = (lo ^ ((i & 7) << 4)) + 128 * i;
        acc = fma2(wide(*reinterpret_cast<const uint32_t*>(s.HS + at)), wide(*reinterpret_cast<const uint32_t*>(s.DH + at)), acc);
      }
      const float ax = halves(acc).x, ay = halves(acc).y;
      s.hdh_part[vq][2 * kp] = ax;
      s.hdh_part[vq][2 * kp + 1] = ay;
    }
    // ---- second load group: Tm, raw kk, v (not earlier: the stores of the previous tile's results have to have read this memory)
    if (lane == 0 && warp_u >= 2 && warp_u < 4) {
      fence_proxy_async();
      bulk_wait_read<0>();
      fetch_late(idx, h, ci.tok0, 2 * (warp_u - 1));
      fetch_late(idx, h, ci.tok0, 2 * (warp_u - 1) + 1);
    }
    // =========================== phase A: state-dependent products ==================================================
    if (warp_u == 0 && alive) {
      const uint32_t aHS = smem_u32(s.HS), aDH = smem_u32(s.DH), aVN = smem_u32(s.VN), aDVN = smem_u32(s.DVN), aDO = smem_u32(s.dO);
      constexpr uint32_t i1 = umma::instr_desc(128, 64, true, false);
      constexpr uint32_t i2 = umma::instr_desc(128, 64, true, true, false, true);
      constexpr uint32_t i3 = umma::instr_desc(128, 64, true, true);
      constexpr uint32_t i4 = umma::instr_desc(64, 64, false, true);
      // base descriptors once; a k-step advances an MN-major operand by two atoms (2048 B) and a K-major one by 32 B
      const uint64_t dHS = umma::desc_mnmajor(aHS, 0, SPAN), dDHm = umma::desc_mnmajor(aDH, 0, SPAN);
      const uint64_t dVNm = umma::desc_mnmajor(aVN, 0, SPAN), dDVNm = umma::desc_mnmajor(aDVN, 0, SPAN);
      const uint64_t dDO0 = umma::desc_kmajor(aDO, 0), dDO1 = umma::desc_kmajor(aDO + 8192, 0);
#pragma unroll 1
      for (int sK = 0; sK < v_steps; ++sK) {
        const uint64_t mn = static_cast<uint64_t>(sK) * 128u, dDOk = ((sK >> 2) ? dDO1 : dDO0) + static_cast<uint64_t>(sK & 3) * 2u;
        umma::mma_ss_lead(tb + C_DQG, dHS + mn, dDOk, i1, sK > 0, lead);                 // dqg^T = h dO^T
        umma::mma_ss_lead(tb + C_DW, dHS + mn, dDVNm + mn, i2, sK > 0, lead);            // dw^T = -h dv_new^T
        umma::mma_ss_lead(tb + C_DKG, dDHm + mn, dVNm + mn, i3, sK > 0, lead);           // dkg^T = dh' v_new^T
        umma::mma_ss_lead(tb + C_DAQ, dDOk, dVNm + mn, i4, sK > 0, lead);                // dAqk = dO v_new^T
      }
      if (lead) umma::commit(&s.barM);
    }
    KDA_DBG_CLOCK(dbg, 2);
    // ---- meanwhile, on warps 1..15 (warp 0 is held up by the issue loop; a barrier that includes it would make
    // everybody wait for the loop's end, so these warps meet at named barrier 1 and warp 1 takes warp 0's columns):
    // G = cumsum(g) log2(e)  (g arrived during the previous tile's phase D) ------------------------------------
    if (warp_u != 0) {
      if (alive && !mbar_wait(&s.barG, it & 1)) alive = false;
      if (len < C) {
#pragma unroll 1
        for (int i = len * 16 + tid - 32; i < C * 16; i += NT - 32) {
          reinterpret_cast<uint4*>(s.G)[2 * i] = make_uint4(0u, 0u, 0u, 0u);
          reinterpret_cast<uint4*>(s.G)[2 * i + 1] = make_uint4(0u, 0u, 0u, 0u);
        }
      }
      asm volatile("bar.sync 1, 480;" ::: "memory");
      // item = (column, quarter of 16 rows): a thread's own, and for warp 1 also the one warp 0 would have had
      float gv[2][16];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        if (r == 1 && warp_u != 1) break;
        const int item = r ? tid - 32 : tid;
        const int col = item & 127, qr = item >> 7;
#pragma unroll
        for (int i = 0; i < 16; ++i) gv[r][i] = s.G[(qr * 16 + i) * KD + col];
        float run = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          run += gv[r][i];
          gv[r][i] = run;
        }
        s.carry[qr][col] = run;
      }
      asm volatile("bar.sync 1, 480;" ::: "memory");
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        if (r == 1 && warp_u != 1) break;
        const int item = r ? tid - 32 : tid;
        const int col = item & 127, qr = item >> 7;
        float pre = 0.f;
#pragma unroll
        for (int b = 0; b < 3; ++b) pre += (b < qr) ? s.carry[b][col] : 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) s.G[(qr * 16 + i) * KD + col] = (pre + gv[r][i]) * LOG2E;
      }
    }
    if (alive && !mbar_wait(&s.barM, mph & 1)) {
      if (tid == 0) atomicOr(p.status, 64u);
      alive = false;
    }
    ++mph;
    alive = __syncthreads_and(alive);      // also: G complete, hdh partials complete, phase A products complete for everybody
    if (!alive) {
      if (tid == 0) atomicOr(p.status, 32u);
      break;
    }
    umma::fence_after_sync();
    if (tid < KD)
      s.hdh[tid] = s.hdh_part[0][tid] + s.hdh_part[1][tid] + s.hdh_part[2][tid] + s.hdh_part[3][tid] + s.hdh_part[4][tid] +
                   s.hdh_part[5][tid] + s.hdh_part[6][tid] + s.hdh_part[7][tid];      // consumed long before dbp is written

    KDA_DBG_CLOCK(dbg, 3);
    // ---- post-A: dw^T -> bf16 tile; dAqk -> masked bf16 tile + diagonal blocks; k Gam tile -------------------------
    {
      float v[16], w16[16];                            // both loads in flight together
      umma::tmem_ld16(tq + C_DW + 16 * part, w16);
      umma::tmem_ld16(tq + C_DAQ + 16 * part, v);      // M = 64: rows 16 q4 .. +15 live in lanes 0..15 of this quadrant
      umma::tmem_ld_wait();
      const int kk = 32 * q4 + lane;
      *reinterpret_cast<uint4*>(sw_piece(sDWT, kk, 2 * part)) = pack8(&w16[0]);
      *reinterpret_cast<uint4*>(sw_piece(sDWT, kk, 2 * part + 1)) = pack8(&w16[8]);
      if (lane < 16) {
        const int t = 16 * q4 + lane;
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = (16 * part + i <= t) ? v[i] : 0.f;
        *reinterpret_cast<uint4*>(sw_piece(sDA, da_row(t), 2 * part)) = pack8(&v[0]);
        *reinterpret_cast<uint4*>(sw_piece(sDA, da_row(t), 2 * part + 1)) = pack8(&v[8]);
        if (part == q4) {                              // these 16 columns are the diagonal block of row block q4
#pragma unroll
          for (int cc = 0; cc < 16; ++cc) s.Ad[q4][lane][cc].x = p.scale * v[cc];
        }
      }
    }
    if (!mbar_wait(&s.barQ, it & 1)) alive = false;
    if (len < C) {                 // uniform over the CTA
#pragma unroll 1
      for (int i = len * 16 + tid; i < C * 16; i += NT) {
        reinterpret_cast<uint4*>(s.q)[i] = make_uint4(0u, 0u, 0u, 0u);
        reinterpret_cast<uint4*>(s.k)[i] = make_uint4(0u, 0u, 0u, 0u);
      }
      __syncthreads();
    }
    {      // k Gam as two K-major sub-tiles [64 j][64 kk]; q and k interleaved over themselves
      static_assert(C * 32 == 4 * NT, "four pieces per thread");
      uint2 qr[4], kr[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        qr[u] = *reinterpret_cast<const uint2*>(&s.q[4 * (tid + u * NT)]);
        kr[u] = *reinterpret_cast<const uint2*>(&s.k[4 * (tid + u * NT)]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = warp_u + u * (NT / 32);
        const F4 Ga = lds4(reinterpret_cast<const float*>(four(s.G, j, lane)));
        const float2 a = halves(Ga.a), b = halves(Ga.b), k0 = unpack_bf16(kr[u].x), k1 = unpack_bf16(kr[u].y);
        put4(sKG + (lane >> 4) * 8192 + (lane & 1) * 8 + j * 128 + ((((lane >> 1) ^ j) & 7) << 4), mul2(pair(k0.x, k0.y), pair(ex2(a.x), ex2(a.y))),
             mul2(pair(k1.x, k1.y), pair(ex2(b.x), ex2(b.y))));
      }
      __syncthreads();      // everybody has read q and k
#pragma unroll
      for (int u = 0; u < 4; ++u)
        *reinterpret_cast<uint4*>(&s.qk[4 * (tid + u * NT)]) =
            make_uint4(__byte_perm(qr[u].x, kr[u].x, 0x5410), __byte_perm(qr[u].x, kr[u].x, 0x7632), __byte_perm(qr[u].y, kr[u].y, 0x5410),
                       __byte_perm(qr[u].y, kr[u].y, 0x7632));
    }
    cp_async_wait<0>();
    if (!mbar_wait(&s.barB, it & 1)) alive = false;       // Tm, raw kk, v
    if (len < C) {
      zero_rows_sw(s.V, len);
      zero_rows_sw(s.V + 8192, len);
    }
    fence_proxy_async();
    umma::fence_before_sync();
    alive = __syncthreads_and(alive);
    if (!alive) {
      if (tid == 0) atomicOr(p.status, 32u);
      break;
    }
    umma::fence_after_sync();

    KDA_DBG_CLOCK(dbg, 4);
    // =========================== phase B1 ===========================================================================
    if (warp_u == 0) {
      const uint32_t aDVN = smem_u32(s.DVN), aV = smem_u32(s.V), aDWT = smem_u32(sDWT), aKG = smem_u32(sKG), aTI = smem_u32(s.TI);
      constexpr uint32_t iT = umma::instr_desc(64, 64, true, false);
      constexpr uint32_t iB = umma::instr_desc(128, 64, false, true);
      const uint64_t dDuM = umma::desc_mnmajor(aDVN, 0, SPAN), dDwM = umma::desc_mnmajor(aDWT, 0, SPAN), dTiM = umma::desc_mnmajor(aTI, 0, SPAN);
      const uint64_t dV0 = umma::desc_kmajor(aV, 0), dV1 = umma::desc_kmajor(aV + 8192, 0);
      const uint64_t dKg0 = umma::desc_kmajor(aKG, 0), dKg1 = umma::desc_kmajor(aKG + 8192, 0);
      const uint64_t dDuK = umma::desc_kmajor(aDVN, 0), dDwK = umma::desc_kmajor(aDWT, 0);
#pragma unroll 1
      for (int sK = 0; sK < v_steps; ++sK) {
        const uint64_t mn = static_cast<uint64_t>(sK) * 128u, dVk = ((sK >> 2) ? dV1 : dV0) + static_cast<uint64_t>(sK & 3) * 2u;
        umma::mma_ss_lead(tb + C_DAQ, dDuM + mn, dVk, iT, sK > 0, lead);       // dTm[t][j]   += sum_v du[t][v] v[j][v]
      }
#pragma unroll 1
      for (int sK = 0; sK < k_steps; ++sK) {
        const uint64_t mn = static_cast<uint64_t>(sK) * 128u, dKg = ((sK >> 2) ? dKg1 : dKg0) + static_cast<uint64_t>(sK & 3) * 2u;
        umma::mma_ss_lead(tb + C_DAQ, dDwM + mn, dKg, iT, 1, lead);            // += sum_kk dw[t][kk] kGam[j][kk]
      }
#pragma unroll 1
      for (int sK = 0; sK < 4; ++sK) {
        const uint64_t dTi = dTiM + static_cast<uint64_t>(sK) * 128u;
        umma::mma_ss_lead(tb + C_DBV, dDuK + static_cast<uint64_t>(sK) * 2u, dTi, iB, sK > 0, lead);     // dbv^T[v][t] = sum_t' du[t'][v] Tm[t'][t]
        umma::mma_ss_lead(tb + C_DBK, dDwK + static_cast<uint64_t>(sK) * 2u, dTi, iB, sK > 0, lead);     // dbk^T[kk][t] = sum_t' dw[t'][kk] Tm[t'][t]
      }
      if (lead) umma::commit(&s.barM);
    }
    // meanwhile two thirds of phase C's operands (warp 0 is busy issuing), into the v_new, dO and dh tiles, which only phase A read; the next tile's
    // chunk is looked up by a warp that waits here anyway
    if (warp_u != 0) {
      if (warp_u == NT / 32 - 1 && lane == 0 && next_idx < total_tiles) stash_chunk(next_idx, (it + 1) & 1);
      __syncwarp();
      build_kR(warp_u - 1, NT / 32 - 1, lane);
      build_qkL(sQL0, sKL0, true, warp_u - 1, NT / 32 - 1, lane);
    }
    if (!mbar_wait(&s.barM, mph & 1)) alive = false;
    ++mph;
    umma::fence_after_sync();
    KDA_DBG_CLOCK(dbg, 5);
    {
      float v[16], bt[16];
      umma::tmem_ld16(tq + C_DAQ + 16 * part, v);      // dTm rows (M = 64 layout): scale the columns by beta_j
      betas(16 * part, bt);
      umma::tmem_ld_wait();
      if (lane < 16) {
        const int t = 16 * q4 + lane;
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = v[i] * bt[i];
        *reinterpret_cast<uint4*>(sw_piece(sDT, t, 2 * part)) = pack8(&x[0]);
        *reinterpret_cast<uint4*>(sw_piece(sDT, t, 2 * part + 1)) = pack8(&x[8]);
      }
      hand_over(lane);
      // =========================== phase B2: X = dTm Tm^T ============================================================
      if (warp_u == 0) {
        if (!handed_over()) alive = false;
        const uint32_t aDT = smem_u32(sDT), aTI = smem_u32(s.TI);
        constexpr uint32_t iX = umma::instr_desc(64, 64, false, false);
        const uint64_t dDt = umma::desc_kmajor(aDT, 0), dTiK = umma::desc_kmajor(aTI, 0);
        if (alive) {
#pragma unroll
          for (int sK = 0; sK < 4; ++sK) umma::mma_ss_lead(tb + C_XY, dDt + static_cast<uint64_t>(sK) * 2u, dTiK + static_cast<uint64_t>(sK) * 2u, iX, sK > 0, lead);
          if (lead) umma::commit(&s.barM);
        }
      }
      {      // dbeta_j += sum_t Tm[t][j] dTm_raw[t][j]: rows t are lanes 0..15 (what the others compute is not used); afterwards lane j holds column j
#pragma unroll
        for (int cix = 0; cix < 2; ++cix) {
          const uint4 tm = *reinterpret_cast<const uint4*>(sw_piece(s.TI, 16 * q4 + (lane & 15), 2 * part + cix));
          const uint32_t w[4] = {tm.x, tm.y, tm.z, tm.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 y = unpack_bf16(w[e]);
            v[8 * cix + 2 * e] *= y.x;
            v[8 * cix + 2 * e + 1] *= y.y;
          }
        }
#pragma unroll
        for (int o = 8; o >= 1; o >>= 1) {
          const bool up = (lane & o) != 0;
#pragma unroll
          for (int i = 0; i < o; ++i) v[i] = (up ? v[i + o] : v[i]) + __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + o], o);
        }
        if (lane < 16) s.dbp[q4][16 * part + lane] = v[0];
      }
      umma::tmem_ld16(tq + C_DBV + 16 * part, v);      // dbv^T rows v: dv[t][v] = beta_t dbv[t][v]
      umma::tmem_ld_wait();
      if (len == C) {      // staged in the dv_new tile, which the products have read, and stored by the copy engine
        __nv_bfloat16* const st = reinterpret_cast<__nv_bfloat16*>(dv_stage(q4)) + 16 * part * 32 + lane;
#pragma unroll
        for (int i = 0; i < 16; ++i) st[32 * i] = __float2bfloat16_rn(bt[i] * v[i]);
      } else {
        const int vcol = 32 * q4 + lane;
        __nv_bfloat16* const dvp = p.dv + (static_cast<size_t>(ci.tok0 + 16 * part) * p.H + h) * p.vc + vcol;
        const size_t tstride = static_cast<size_t>(p.H) * p.vc;
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (16 * part + i < len && vcol < p.vc) dvp[i * tstride] = __float2bfloat16_rn(bt[i] * v[i]);
      }
    }
    KDA_DBG_CLOCK(dbg, 6);
    // =========================== phase D: one thread per key column and 16-row block ================================
    // Its first part needs only accumulators of phases A and B1 and runs in three pieces while the products of B2, B3 and C execute.
    build_qkL(sQL1, sKL1, false, warp_u, NT / 32, lane);      // the rest of phase C's operands: into the dw^T and v tiles, which phase B1 read last
    // Decay inside the block as running products of lam_i = 2^(G_i - G_{i-1}) (every factor <= 1):
    //   2^(G_i - G_first) = lam_1 .. lam_i,  2^(G_i) = g_first lam_1 .. lam_i,  2^(G_e - G_i) = lam_{i+1} .. lam_15,  2^(G_last - G_e) = e_last
    const int kk = fresh_tid() & 127, blk = warp_u >> 2, t0 = 16 * blk;
    float cq[16], cp[16], lam[16];
    float g_first, e_last;
    {
      float prev = s.G[t0 * KD + kk];
      g_first = ex2(prev);
      lam[0] = 1.f;
#pragma unroll
      for (int i = 1; i < 16; ++i) {
        const float cur = s.G[(t0 + i) * KD + kk];
        lam[i] = ex2(cur - prev);
        prev = cur;
      }
      const float Gl = s.G[(C - 1) * KD + kk];
      if (blk == 3) s.hdh[kk] *= ex2(Gl);      // the state's own share of dG at the chunk's last row
      e_last = ex2(Gl - prev);
    }
    {      // sum of k dk_end feeds dG at the chunk's last row (dk_end = dkg 2^(G_last - G))
      float a[16];
      umma::tmem_ld16(tq + C_DKG + t0, a);
      umma::tmem_ld_wait();
      float dglp = 0.f, fr = e_last;
#pragma unroll
      for (int i = 15; i >= 0; --i) {
        dglp = fmaf(k_of(s.qk[(t0 + i) * KD + kk]), a[i] * fr, dglp);
        fr *= lam[i];
      }
      s.dglp[blk][kk] = dglp;
    }
    if (!mbar_wait(&s.barM, mph & 1)) alive = false;
    ++mph;
    umma::fence_after_sync();
    {
      float v[16];
      umma::tmem_ld16(tq + C_XY + 16 * part, v);
      umma::tmem_ld_wait();
      if (lane < 16) {
        const int m = 16 * q4 + lane;
        *reinterpret_cast<uint4*>(sw_piece(sX, m, 2 * part)) = pack8(&v[0]);
        *reinterpret_cast<uint4*>(sw_piece(sX, m, 2 * part + 1)) = pack8(&v[8]);
      }
    }
    hand_over(lane);      // (dv is staged, too)

    KDA_DBG_CLOCK(dbg, 7);
    // =========================== phase B3: Y = Tm^T X,  dAkk = -tril(Y, -1) ==========================================
    if (warp_u == 0) {
      if (!handed_over()) alive = false;
      const uint32_t aX = smem_u32(sX), aTI = smem_u32(s.TI);
      constexpr uint32_t iY = umma::instr_desc(64, 64, true, true);
      const uint64_t dTiM = umma::desc_mnmajor(aTI, 0, SPAN), dXm = umma::desc_mnmajor(aX, 0, SPAN);
      if (alive) {
#pragma unroll
        for (int sK = 0; sK < 4; ++sK)
          umma::mma_ss_lead(tb + C_XY, dTiM + static_cast<uint64_t>(sK) * 128u, dXm + static_cast<uint64_t>(sK) * 128u, iY, sK > 0, lead);
        if (lead) umma::commit(&s.barM);
      }
    }
    if (warp_u == 4 && len == C) {
      if (!handed_over()) alive = false;
      if (lane == 0 && alive) {
#pragma unroll 1
        for (int i = 0; i < 4 && 32 * i < p.vc; ++i) tma_store_rows(&p.tm_dv, 32 * i, h, ci.tok0, dv_stage(i));
        bulk_commit();
      }
      __syncwarp();
    }
    {      // dq: scale Gam dqg
      float a[16];
      umma::tmem_ld16(tq + C_DQG + t0, a);
      umma::tmem_ld_wait();
      float fl = p.scale * g_first;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        fl *= lam[i];
        cq[i] = fl * a[i];
      }
    }
    if (!mbar_wait(&s.barM, mph & 1)) alive = false;
    ++mph;
    umma::fence_after_sync();
    {
      float v[16];
      umma::tmem_ld16(tq + C_XY + 16 * part, v);
      umma::tmem_ld_wait();
      if (lane < 16) {
        const int i0 = 16 * q4 + lane;                 // row i of dAkk
        const float br = s.beta[i0];
        float pb = 0.f;
#pragma unroll
        for (int cix = 0; cix < 2; ++cix) {
          const uint4 rw = *reinterpret_cast<const uint4*>(sw_piece(s.RKK, i0, 2 * part + cix));
          const uint32_t rws[4] = {rw.x, rw.y, rw.z, rw.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 raw = unpack_bf16(rws[e]);
            const int j = 16 * part + 8 * cix + 2 * e;
            const float x0 = (j < i0) ? -v[8 * cix + 2 * e] : 0.f;
            const float x1 = (j + 1 < i0) ? -v[8 * cix + 2 * e + 1] : 0.f;
            pb += x0 * raw.x + x1 * raw.y;
            v[8 * cix + 2 * e] = br * x0;
            v[8 * cix + 2 * e + 1] = br * x1;
          }
        }
        *reinterpret_cast<uint4*>(sw_piece(sDA, da_row(i0) + 8, 2 * part)) = pack8(&v[0]);
        *reinterpret_cast<uint4*>(sw_piece(sDA, da_row(i0) + 8, 2 * part + 1)) = pack8(&v[8]);
        s.dbp[4 + part][i0] = pb;
        if (part == q4) {
#pragma unroll
          for (int cc = 0; cc < 16; ++cc) s.Ad[q4][lane][cc].y = v[cc];
        }
      }
    }
    hand_over(lane);
    KDA_DBG_CLOCK(dbg, 8);

    KDA_DBG_CLOCK(dbg, 9);
    // =========================== phase C: off-diagonal blocks of the intra-chunk terms ==============================
    if (warp_u == 0) {
      if (!handed_over()) alive = false;
      constexpr uint32_t iC1 = umma::instr_desc(128, 32, true, false);
      constexpr uint32_t iC2 = umma::instr_desc(128, 16, true, true);
      const uint64_t dKr = umma::smem_desc(smem_u32(sKR), KR_SPAN, umma::ATOM_BYTES), dDa = umma::smem_desc(smem_u32(sDA), 16, umma::ATOM_BYTES);
      const uint64_t dAq = umma::smem_desc(smem_u32(sDA), 16, 2 * umma::ATOM_BYTES), dAk = dAq + umma::ATOM_BYTES / 16;      // every other atom
#pragma unroll
      for (int I = 1; I < 4; ++I) {
        const int rb = (I == 1) ? 0 : (I == 2 ? 16 : 48);
#pragma unroll
        for (int sK = 0; sK < I; ++sK)      // A[kk][j] = kR_I[j][kk]: row offset in 16-byte units;  B[t][j]: rows 16 I.. of both, k-step sK
          umma::mma_ss_lead(tb + C_CQP + 32 * (I - 1), dKr + static_cast<uint64_t>((rb + 16 * sK) * 8), dDa + static_cast<uint64_t>(32 * I * 8 + sK * 2), iC1, sK > 0, lead);
      }
      const uint64_t dQl0 = umma::smem_desc(smem_u32(sQL0), L_SPAN, umma::ATOM_BYTES), dKl0 = umma::smem_desc(smem_u32(sKL0), L_SPAN, umma::ATOM_BYTES);
      const uint64_t dQl1 = umma::smem_desc(smem_u32(sQL1), L_SPAN, umma::ATOM_BYTES), dKl1 = umma::smem_desc(smem_u32(sKL1), L_SPAN, umma::ATOM_BYTES);
#pragma unroll
      for (int J = 0; J < 3; ++J) {
        const int rb = J == 2 ? 32 : 0;
#pragma unroll
        for (int sK = 0; sK < 3 - J; ++sK) {
          const uint64_t ao = static_cast<uint64_t>((rb + 16 * sK) * 8);
          const uint64_t bo = static_cast<uint64_t>(32 * (J + 1 + sK) * 8 + 2 * J);            // B[j][t] = dA[t][j]: rows t, columns 16 J..
          umma::mma_ss_lead(tb + C_CN + 16 * J, (J ? dQl1 : dQl0) + ao, dAq + bo, iC2, sK > 0, lead);
          umma::mma_ss_lead(tb + C_CN + 16 * J, (J ? dKl1 : dKl0) + ao, dAk + bo, iC2, 1, lead);
        }
      }
      if (lead) umma::commit(&s.barM);
    }
    {      // dk+: Gam beta dbk
      float a[16];
      umma::tmem_ld16(tq + C_DBK + t0, a);
      float bt[16];
      betas(t0, bt);
      umma::tmem_ld_wait();
      float fl = g_first;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        fl *= lam[i];
        cp[i] = fl * bt[i] * a[i];
      }
    }
    // Diagonal block.  Rows 8..15 against columns 0..7, then 4..7 against 0..3 and 12..15 against 8..11, with the decay cut at the
    // border between them: L_t = prod(border .. t) on the row side, R_j = prod(j+1 .. border-1) on the column side, both running products
    // of lam (range-safe).  Factored this way an entry costs four multiply-adds instead of the eight operations of a pair with its
    // own decay; only the 4 x 4 blocks on the diagonal stay pairwise.
    // Four columns at a time, in rising order: behind its own columns a row is final (it only sees earlier ones), so dk- lives for four
    // rows only (its other terms wait in tensor memory) and dq, dk leave for their staging tiles at once.  With dk- of all sixteen
    // rows in registers the phase spilled, and spills miss the little L1 that is left: it took 6.4 k of a tile's 30 k cycles.
    // dq and dk+ of a row, and the q- and k-side of everything they are made from, travel as a register pair: one instruction for both.
    auto word = [&](int i) { return s.qk[(t0 + i) * KD + kk]; };
    auto both = [&](int i) {      // (q, k) of a row
      const uint32_t w = word(i);
      return pair(q_of(w), k_of(w));
    };
    f32x2 cc[16];      // (dq, dk+)
#pragma unroll
    for (int i = 0; i < 16; ++i) cc[i] = pair(cq[i], cp[i]);
    // keeps the compiler from carrying q, k (read from shared memory where they are used) or products of lam, and (a warp barrier orders memory accesses) from starting later
    // loads early: sixteen loads of four registers in front of a part would not fit
    auto step = [&] {
#pragma unroll
      for (int i = 0; i < 16; ++i) asm volatile("" : "+f"(lam[i])::"memory");
      __syncwarp();
    };
    float cn[4];
    // rows r0 .. r0 + W - 1 against the four columns c0 .. c0 + 3, the border in front of row r0
    auto part4 = [&](auto width, const int r0, const int c0) {
      constexpr int W = decltype(width)::value;
      f32x2 kR[4], sn[4];
      float Rc = 1.f;
#pragma unroll
      for (int j = c0 + 4; j < r0; ++j) Rc *= lam[j];
      {
        float R = Rc;
#pragma unroll
        for (int j = 3; j >= 0; --j) {
          const float x = k_of(word(c0 + j)) * R;
          kR[j] = pair(x, x);
          sn[j] = 0ull;
          R *= lam[c0 + j];
        }
      }
      float L = 1.f;
#pragma unroll
      for (int t = 0; t < W; ++t) {
        if (t && t % 4 == 0) __syncwarp();
        L *= lam[r0 + t];
        const f32x2 LL = pair(L, L), ql = mul2(both(r0 + t), LL);
        f32x2 sum = 0ull;
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
          const F4 a = lds4(reinterpret_cast<const float*>(&s.Ad[blk][r0 + t][c0 + j]));
          sum = fma2(a.a, kR[j], sum);
          sn[j] = fma2(a.a, ql, sn[j]);
          sum = fma2(a.b, kR[j + 1], sum);
          sn[j + 1] = fma2(a.b, ql, sn[j + 1]);
        }
        cc[r0 + t] = fma2(LL, sum, cc[r0 + t]);
      }
#pragma unroll
      for (int j = 3; j >= 0; --j) {
        const float2 x = halves(sn[j]);
        cn[j] = fmaf(Rc, x.x + x.y, cn[j]);
        Rc *= lam[c0 + j];
      }
    };
    // the first four columns' share of the rows behind them, while the products of phase C execute
    if (!handed_over()) alive = false;      // the diagonal blocks of dAkk are there
#pragma unroll
    for (int j = 0; j < 4; ++j) cn[j] = 0.f;
    step();
    part4(std::integral_constant<int, 8>{}, 8, 0);
    step();
    part4(std::integral_constant<int, 4>{}, 4, 0);
    step();
    if (warp_u == 4 && lane == 0) bulk_wait_read<0>();      // dv has left before the next tile's state tiles arrive there (phase D)
    if (!mbar_wait(&s.barM, mph & 1)) alive = false;
    ++mph;
    alive = __syncthreads_and(alive);      // phase C complete; G has been read by everybody; dglp is complete
    if (!alive) {
      if (tid == 0) atomicOr(p.status, 64u);
      break;
    }
    umma::fence_after_sync();
    KDA_DBG_CLOCK(dbg, 10);
    // every shared-memory operand tile is dead now and g is in registers (lam): fetch the next tile behind the rest
    if (next_idx < total_tiles && warp_u < 7 && lane == 0) fetch(next_idx, (it + 1) & 1, warp_u);
    if (tid < len)
      p.dbeta[static_cast<size_t>(ci.tok0 + tid) * p.H + h] = s.dbp[0][tid] + s.dbp[1][tid] + s.dbp[2][tid] + s.dbp[3][tid] +
                                                             s.dbp[4][tid] + s.dbp[5][tid] + s.dbp[6][tid] + s.dbp[7][tid];

    KDA_DBG_CLOCK(dbg, 11);
    {
      {
        // the off-diagonal blocks of phase C, scaled back from their reference rows
        if (blk > 0) {                          // dq: + scale L Cq;  dk+: + L Cp
          float fl = 1.f;
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            float b[16];                        // eight rows of Cq, of Cp
            umma::tmem_ld16(tq + C_CQP + 32 * (blk - 1) + 16 * hf, b);
            umma::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              fl *= lam[8 * hf + i];
              const float2 c = halves(cc[8 * hf + i]);
              cc[8 * hf + i] = pair(fmaf(p.scale * fl, b[i], c.x), fmaf(fl, b[8 + i], c.y));
            }
          }
        }
      }
      KDA_DBG_CLOCK(dbg, 12);
      auto columns = [&](auto first) {
        constexpr int c0 = decltype(first)::value;
        {      // dk-: 2^(G_e - G) (2^(G_last - G_e) dkg + Cn)
          float d4[4], b4[4];
          umma::tmem_ld4(tq + C_DKG + t0 + c0, d4);
          if (blk < 3) umma::tmem_ld4(tq + C_CN + t0 + c0, b4);
          umma::tmem_ld_wait();
          float fr = 1.f;
#pragma unroll
          for (int j = c0 + 4; j < 16; ++j) fr *= lam[j];
#pragma unroll
          for (int j = 3; j >= 0; --j) {
            const float x = fr * (blk < 3 ? fmaf(e_last, d4[j], b4[j]) : e_last * d4[j]);
            cn[j] = c0 ? x : cn[j] + x;
            fr *= lam[c0 + j];
          }
        }
        step();
        if constexpr (c0 == 4) {
          part4(std::integral_constant<int, 8>{}, 8, c0);
          step();
        }
        if constexpr (c0 == 8) {
          part4(std::integral_constant<int, 4>{}, c0 + 4, c0);
          step();
        }
        uint32_t w[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) w[t] = word(c0 + t);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const float qt = q_of(w[t]), kt = k_of(w[t]);
          float2 c = halves(cc[c0 + t]);
          {
            const float ax = s.Ad[blk][c0 + t][c0 + t].x;      // dAkk has no diagonal
            c.x = fmaf(ax, kt, c.x);
            cn[t] = fmaf(ax, qt, cn[t]);
          }
          float D = 1.f;
#pragma unroll
          for (int j = t - 1; j >= 0; --j) {
            D *= lam[c0 + j + 1];
            const float2 a = s.Ad[blk][c0 + t][c0 + j];
            const float kd = k_of(w[j]) * D;
            c.x = fmaf(a.x, kd, c.x);
            c.y = fmaf(a.y, kd, c.y);
            cn[j] = fmaf(D, fmaf(a.y, kt, a.x * qt), cn[j]);
          }
          cc[c0 + t] = pair(c.x, c.y);
        }
        // dq, dk into their staging tiles; cq becomes dG
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int i = c0 + t;
          const float2 c = halves(cc[i]);
          stq[(t0 + i) * KD + kk] = __float2bfloat16_rn(c.x);
          stk[(t0 + i) * KD + kk] = __float2bfloat16_rn(c.y + cn[t]);
          cq[i] = q_of(w[t]) * c.x + k_of(w[t]) * (c.y - cn[t]);
        }
        step();
      };
      columns(std::integral_constant<int, 0>{});
      columns(std::integral_constant<int, 4>{});
      columns(std::integral_constant<int, 8>{});
      columns(std::integral_constant<int, 12>{});
      KDA_DBG_CLOCK(dbg, 13);
      if (blk == 3)          // the chunk's last row carries the chunk-end terms
        cq[15] += s.dglp[0][kk] + s.dglp[1][kk] + s.dglp[2][kk] + s.dglp[3][kk] + s.hdh[kk];
      {
        float run = 0.f;
#pragma unroll
        for (int i = 15; i >= 0; --i) {
          run += cq[i];
          cq[i] = run;
        }
        s.carry[blk][kk] = run;
      }
      // L2: the reciprocal norms of this thread's two copy-out pieces, asked for before the barrier so that they arrive behind it
      float rq2[2], rk2[2];
      if constexpr (L2) {
        static_assert(C * 16 == 2 * NT, "two copy-out pieces per thread");
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int r = (tid + u * NT) >> 4;
          const size_t grow = static_cast<size_t>(ci.tok0 + (r < len ? r : 0)) * p.H + h;
          rq2[u] = __ldg(p.rstd + grow);
          rk2[u] = __ldg(p.rstd + p.qrows + grow);
        }
      }
      __syncthreads();       // block totals and the staged dq, dk are complete
      if (L2 || len < C)
#pragma unroll
      for (int u = 0; u < C * 16 / NT; ++u) {
        const int i = tid + u * NT, r = i >> 4, pc = i & 15;
        const size_t row = (static_cast<size_t>(ci.tok0 + (r < len ? r : 0)) * p.H + h) * p.dqc + pc * 8;
        uint4 oq = *reinterpret_cast<const uint4*>(&stq[r * KD + pc * 8]);
        uint4 ok = *reinterpret_cast<const uint4*>(&stk[r * KD + pc * 8]);
        if constexpr (L2) {
          // dx = rstd (dy - y <y, dy>) per row; sixteen consecutive lanes hold one row (y: the normalised q, k; dy: the staged bf16 values, as
          // the separate pass would read them)
          uint32_t y[8];
          *reinterpret_cast<uint4*>(&y[0]) = *reinterpret_cast<const uint4*>(&s.qk[r * KD + pc * 8]);
          *reinterpret_cast<uint4*>(&y[4]) = *reinterpret_cast<const uint4*>(&s.qk[r * KD + pc * 8 + 4]);
          const uint32_t dqw[4] = {oq.x, oq.y, oq.z, oq.w}, dkw[4] = {ok.x, ok.y, ok.z, ok.w};
          float2 dqf[4], dkf[4], yqf[4], ykf[4];
          float sq = 0.f, sk = 0.f;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            dqf[e] = unpack_bf16(dqw[e]); dkf[e] = unpack_bf16(dkw[e]);
            yqf[e] = make_float2(q_of(y[2 * e]), q_of(y[2 * e + 1])); ykf[e] = make_float2(k_of(y[2 * e]), k_of(y[2 * e + 1]));
            sq = fmaf(yqf[e].x, dqf[e].x, fmaf(yqf[e].y, dqf[e].y, sq));
            sk = fmaf(ykf[e].x, dkf[e].x, fmaf(ykf[e].y, dkf[e].y, sk));
          }
#pragma unroll
          for (int o = 8; o >= 1; o >>= 1) {
            sq += __shfl_xor_sync(0xffffffffu, sq, o);
            sk += __shfl_xor_sync(0xffffffffu, sk, o);
          }
          const float rq = rq2[u], rk = rk2[u];
          uint32_t wq[4], wk[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            wq[e] = pack_bf16(rq * (dqf[e].x - yqf[e].x * sq), rq * (dqf[e].y - yqf[e].y * sq));
            wk[e] = pack_bf16(rk * (dkf[e].x - ykf[e].x * sk), rk * (dkf[e].y - ykf[e].y * sk));
          }
          oq = make_uint4(wq[0], wq[1], wq[2], wq[3]);
          ok = make_uint4(wk[0], wk[1], wk[2], wk[3]);
        }
        if (r < len && pc * 8 < p.dqc) {
          *reinterpret_cast<uint4*>(p.dq + row) = oq;
          *reinterpret_cast<uint4*>(p.dk + row) = ok;
        }
      }
      if constexpr (L2) __syncthreads();      // q and k have been read
      {
        float add = 0.f;             // totals of the later blocks
#pragma unroll
        for (int bb = 1; bb < 4; ++bb) add += (bb > blk) ? s.carry[bb][kk] : 0.f;
        // (straight from registers, not staged over q and k: the next tile's q and k are on their way as soon as everybody has read these, 8 x 8192 x 32
        // 5.81 -> 5.73 ms)
        float* dgp = p.dg + (static_cast<size_t>(ci.tok0 + t0) * p.H + h) * p.kc + kk;      // a warp stores 128 contiguous bytes
        const size_t gstep = static_cast<size_t>(p.H) * p.kc;
#pragma unroll
        for (int i = 0; i < 16; ++i, dgp += gstep)
          if (t0 + i < len && kk < p.kc) *dgp = cq[i] + add;
      }
    }
    KDA_DBG_CLOCK(dbg, 14);
    fence_proxy_async();
    umma::fence_before_sync();
    __syncthreads();   // beta, Ad, the staging tiles, TMEM ... may be overwritten by the next tile
    if (lane == 0 && len == C) {      // full chunks leave by the copy engine (partial ones: the rows behind them are another sequence's)
      if (!L2 && warp_u == 2) tma_store_rows(&p.tm_dk, 0, h, ci.tok0, stk);
      if (!L2 && warp_u == 3) tma_store_rows(&p.tm_dq, 0, h, ci.tok0, stq);
      if (warp_u >= 2 && warp_u <= 3) bulk_commit();
    }
    if (warp_u == 1 && lane == 0 && next_idx < total_tiles) {      // q, k of the next tile
      fence_proxy_async();
      const int tk = static_cast<int>(s.ci_tok0[(it + 1) & 1]);
      fetch_late(next_idx, next_idx % p.H, tk, 0);
      fetch_late(next_idx, next_idx % p.H, tk, 1);
    }
  }

  // drain: a copy that is still in flight must not outlive the CTA's shared memory
  if (!alive && lane == 0 && warp_u < 5) mbar_drain(&s.barS + warp_u);      // a wait gave up: loads and products may be under way on any of the five barriers
  bulk_wait<0>();      // stores
  cp_async_wait<0>();
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tb, 512);
}

int launch_bwd_main_tc(const MainParams& p, int grid, cudaStream_t st) {
  static DeviceOnce once;
  const int smem = static_cast<int>(sizeof(TcSmem)) + 1024;
  const int rc = once.run([&] {
    cudaError_t e = cudaFuncSetAttribute(kda_chunk_bwd_main_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kda_chunk_bwd_main_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    return e;
  });
  if (rc != KDA_OK) return rc;
  const auto kernel = p.rstd != nullptr && p.grp == 1 ? kda_chunk_bwd_main_tc_kernel<true> : kda_chunk_bwd_main_tc_kernel<false>;
  return static_cast<int>(launch_chained(kernel, grid, NT, smem, st, p));
}

}  // namespace kda
