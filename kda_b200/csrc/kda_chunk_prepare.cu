// Per-chunk preparation of chunked KDA for sm_100a: one CTA (512 threads) per (chunk, head) turns q, k, v, g, beta of 64 tokens into
// everything that does not depend on the state: Aqk, Akk, Tm = (I + diag(beta) Akk)^-1, w, u, qg, kg -> tiles in the workspace.
//
// A thread owns FOUR key columns of FOUR rows and keeps their q, k and lam_t = 2^(g_t log2 e) in registers from the load to the last
// operand: every decay the chunk needs is a running product of lam (all factors <= 1: range-safe for any gate, and no cumulative
// sum of g whose rounding grows with its magnitude).  A warp holds four whole rows, so row norms and the pairwise dot products
// are sums inside one warp.
//
// The intra-chunk products A[t][j] = sum_k x_t 2^(G_t - G_j) k_j (x = q, k) come in levels; at each level the decay is cut at a
// row that lies between j and t, so that both factors are products of lam:
//   16   blocks I > J of 16 x 16:   rows x_t prod(16 I .. t),   columns k_j prod(j+1 .. 16 J + 15) times the blocks in between
//    8   rows 8..15 against 0..7 of a 16-row block, cut at row 8
//    4   rows 4..7 against 0..3 and 12..15 against 8..11, cut at rows 4 and 12
//   the 4 x 4 diagonal blocks pairwise.
// Levels 16 and 8 are products of bf16 rows on tensor cores; level 4 and the diagonal blocks, which hold the largest entries, stay float32
// sums over the lanes (level 4 as a bf16 product, as it was: o 1.7 % further from 64 bits with slowly decaying gates).
// With the caller's promise of bounded gates (SAFE) the 16 x 16 diagonal blocks go whole, cut at their row 8 from both sides.
// Product operands are written to shared memory once as bf16 and read by ldmatrix; the level 8 product stacks q and k rows into one m16
// tile.  The same pass writes QG = scale q Gam, KG = k Gam_last / Gam and k Gam.
//
// What bounds it: instruction issue and shared-memory wavefronts, about 23 k cycles per CTA with two CTAs per SM; its bytes take 0.81 ms
// at 8 x 8192 tokens x 32 heads, where it takes 1.55 ms (with level 4 as a bf16 product 1.50; a thread per key column and row, decays as exp2
// of cumulative sums and row references, 256 threads: 1.98).  Bounded gates at 1 x 32768 x 32: 0.74 ms with the gate's activation.  Without the
// L2 prefetch of the next wave's rows 1.65, two waves ahead 1.59.
#include "kda_device.cuh"
#include "kda_f32x2.cuh"
#include "kda_gate.cuh"
#include "kda_prepare.cuh"

namespace kda {

namespace {

constexpr int PREP_THREADS = 512;
constexpr int QS = 136;   // bf16 elements per padded row of an operand tile (272 B: ldmatrix rows hit distinct banks)
constexpr int AS = 68;    // floats per padded row of the fp32 64x64 matrix
constexpr int TS = 72;    // bf16 elements per padded row of a bf16 64x64 matrix (144 B)
constexpr int DS = 20;    // floats per row of a 16 x 16 fp32 block

// Operand rows of the region `op`: every 16-row block has its own part, written and (levels 8, 4) read by its four warps alone, so that
// they meet at a barrier of 128 threads instead of the whole CTA.  Inside a part:
//   levels 8 and 4:  A8 16 rows (q 8..15, k 8..15) | B8 8 | C4: columns 0..3 and 8..11 of level 4 in fp32 (eight rows of 512 bytes)
//   SAFE diagonal:   q 16 | k 16 (row side) | k 16 (column side)
//   level 16:        blocks 1..3: q 16 | k 16; then columns for the blocks at distance 1, 2, 3 (16 rows each)
// Afterwards the region holds v (two 64-column tiles in the 128-byte swizzle), the staged UT tile and Tm as bf16 (times beta: TB;
// plain: TI, in its tile image).
constexpr int OP_ROWS = 208;
constexpr int OP_B8 = 16, OP_C4 = 24;
static_assert(8 * KD * 4 <= (48 - OP_C4) * QS * 2, "the columns of level 4 must fit behind the level 8 operands");
__device__ __forceinline__ int op_base(int blk) { return blk == 0 ? 0 : 48 * blk + (blk > 1 ? 16 : 0); }      // 48, 64, 48, 48 rows
__device__ __forceinline__ int op_cols(int blk, int dist) { return op_base(blk) + (blk > 0 ? 32 : 0) + 16 * (dist - 1); }

struct PrepSmem {
  __nv_bfloat16 op[OP_ROWS * QS];
  __nv_bfloat16 kG[C * QS];    // k, then k * Gam
  float Akk[C * AS];           // raw <k_t D, k_j> below the diagonal (nothing else is written); at the end the staged W tile
  unsigned char Aqk[TILE_TT];  // scale <q_t D, k_j>, lower triangle incl. diagonal: the tile image that leaves by a bulk store
  union {
    float T[16][KD];             // decay over every four rows (P2, P3)
    struct {
      float TD[4][16 * DS];      // inverses of the diagonal 16 x 16 blocks of I + diag(beta) Akk (P4)
      float TM[2][16 * DS];      // blocks (1, 0) and (3, 2) of the inverse
    };
  };
  float TB[4][KD];               // decay over every 16-row block
  float beta[C];
  uint64_t barV;
};
constexpr int UT_OFF = static_cast<int>(TILE_TK), TI_OFF = UT_OFF + static_cast<int>(TILE_VT), TB_OFF = TI_OFF + static_cast<int>(TILE_TT);      // bytes, behind v
static_assert(TB_OFF + C * TS * 2 <= OP_ROWS * QS * 2, "the last phase's tiles must fit the operand region");
static_assert(TILE_TK <= C * AS * 4, "the staged W tile must fit Akk");
constexpr int PREP_SMEM = static_cast<int>(sizeof(PrepSmem)) + 1024;      // 1024-byte alignment for the swizzled v tiles
static_assert(2 * (PREP_SMEM + 1024) <= 227 * 1024, "two CTAs per SM");

// Sum over the 32 lanes of N per-lane values at once (N = 4, 8): afterwards lane L holds the total of slot L % N.
template <int N>
__device__ __forceinline__ float butterfly(float (&v)[N], int lane) {
#pragma unroll
  for (int o = N / 2; o >= 1; o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float mine = up ? v[i + o] : v[i];
      const float other = up ? v[i] : v[i + o];
      v[i] = mine + __shfl_xor_sync(0xffffffffu, other, o);
    }
  }
#pragma unroll
  for (int o = N; o < 32; o <<= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  return v[0];
}

// A thread's four adjacent key columns of a row are an F4.
__device__ __forceinline__ F4 mul4c(const F4& x, const F4& y) { return {mul2(x.a, y.a), mul2(x.b, y.b)}; }
__device__ __forceinline__ f32x2 widen2(uint32_t u) {      // two bf16 -> two fp32
  f32x2 d;
  asm("{\n .reg .b32 lo, hi;\n shl.b32 lo, %1, 16;\n and.b32 hi, %1, 0xffff0000;\n mov.b64 %0, {lo, hi};\n}\n" : "=l"(d) : "r"(u));
  return d;
}
__device__ __forceinline__ uint32_t narrow2(f32x2 v) {
  const float2 f = halves(v);
  return pack_bf16(f.x, f.y);
}
__device__ __forceinline__ F4 widen(const uint2 u) { return {widen2(u.x), widen2(u.y)}; }
__device__ __forceinline__ uint2 narrow(const F4& x) { return make_uint2(narrow2(x.a), narrow2(x.b)); }
__device__ __forceinline__ F4 splat(float x) { return {pair(x, x), pair(x, x)}; }
__device__ __forceinline__ float dot(const F4& x, const F4& y) {
  const float2 v = halves(fma2(x.b, y.b, mul2(x.a, y.a)));
  return v.x + v.y;
}
// read-once global loads: no L1 allocation
__device__ __forceinline__ uint2 ldg_u2(const void* p) {
  uint2 r;
  asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(r.x), "=r"(r.y) : "l"(p));
  return r;
}
__device__ __forceinline__ unsigned long long ldg_u64(const void* p) {
  unsigned long long r;
  asm volatile("ld.global.nc.L1::no_allocate.u64 %0, [%1];" : "=l"(r) : "l"(p));
  return r;
}
__device__ __forceinline__ float4 ldg_f4(const float* p) {
  float4 r;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "l"(p));
  return r;
}

// acc[n] (16 x 8) = A (16 rows) * B_n^T (8 rows each, B_1 behind B_0) over the 128 key columns
template <int NB>
__device__ __forceinline__ void prep_mma(float (&acc)[NB][4], const __nv_bfloat16* A, const __nv_bfloat16* B, const int lane) {
  const uint32_t aa = smem_u32(A + (lane & 15) * QS + ((lane >> 4) << 3));
  const uint32_t ba = smem_u32(B + (lane & 7) * QS + ((lane >> 3) << 3));
  float c1[NB][4];
#pragma unroll
  for (int n = 0; n < NB; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[n][e] = c1[n][e] = 0.f;
#pragma unroll
  for (int ks = 0; ks < 8; ks += 2) {
    uint32_t a0[4], a1[4], b[NB][4];
#pragma unroll
    for (int n = 0; n < NB; ++n) ldsm_x4(b[n], ba + n * 8 * QS * 2 + ks * 32);
    ldsm_x4(a0, aa + ks * 32);
    ldsm_x4(a1, aa + ks * 32 + 32);
#pragma unroll
    for (int n = 0; n < NB; ++n) {
      mma16816(acc[n], a0, b[n][0], b[n][1]);
      mma16816(c1[n], a1, b[n][2], b[n][3]);
    }
  }
#pragma unroll
  for (int n = 0; n < NB; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[n][e] += c1[n][e];
}

}  // namespace

// KEEP_QN: also leave the L2-normalised q, k and their reciprocal norms in the workspace (training with use_l2norm).
// SAFE: the caller promises bounded gates (safe_gate: at least -5 per token), see above.
template <bool KEEP_QN, bool SAFE>
__global__ void __launch_bounds__(PREP_THREADS, 2) kda_chunk_prepare_kernel(const __grid_constant__ PrepParams p) {
  chain_point();
  extern __shared__ unsigned char smem_raw[];
  PrepSmem& s = *reinterpret_cast<PrepSmem*>(smem_raw + pad_to_1024(smem_raw));
  const int tid = threadIdx.x, lane = tid & 31, gid = lane >> 2, tig = lane & 3;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);      // warp-uniform for the compiler: role branches need no reconvergence code
  const int c = blockIdx.x / p.H, h = blockIdx.x % p.H;        // neighbouring CTAs take neighbouring heads: contiguous rows and tiles
  if (p.clear_status && blockIdx.x == 0 && tid < 5) {      // no tables kernel has run: its share of the workspace that others read
    if (tid < 4) p.status[tid] = 0u;
    else const_cast<int*>(p.map.seq_chunk_off)[p.map.N] = p.map.total();      // kda_chunk_export_states
  }
  if (c >= p.map.total()) return;
  const ChunkInfo ci = p.map.info(c);
  const int len = ci.len;
  const size_t tile = blockIdx.x;
  const int blk = warp >> 2, quad = warp & 3;      // 16-row block and which four of its rows
  const int kk = 4 * lane, t0 = 4 * warp, b0 = 16 * blk;
  KDA_DBG_CLOCK(p.dbg, 16);

  // ---- P1: q, k, g of this thread's columns and rows; rows >= len and columns >= kc: q = k = 0, no decay ---------------------------------
  F4 lam[4];
  uint2 q[4], k[4];
  uint32_t beta_bits = 0u;
  {
    const size_t goff = (static_cast<size_t>(ci.tok0 + t0) * p.H + h) * p.kc + kk;
    const size_t qoff = (static_cast<size_t>(ci.tok0 + t0) * p.HQ + h / p.grp) * p.kc + kk;
    const __nv_bfloat16 *qp = p.q + qoff, *kp = p.k + qoff;
    const size_t gs = static_cast<size_t>(p.H) * p.kc, qs = static_cast<size_t>(p.HQ) * p.kc;
    // every load is issued before anything waits for one
    const bool bf16_gate = p.g_raw && !p.g_fp32;
    if (bf16_gate) {
      const __nv_bfloat16* gp = static_cast<const __nv_bfloat16*>(p.g_raw) + goff;
#pragma unroll
      for (int i = 0; i < 4; ++i) lam[i].a = t0 + i < len && kk < p.kc ? ldg_u64(gp + i * gs) : 0ull;      // four bf16 for now
    } else {
      const float* gp = p.g_raw ? static_cast<const float*>(p.g_raw) + goff : p.g + goff;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 g4 = t0 + i < len && kk < p.kc ? ldg_f4(gp + i * gs) : make_float4(0.f, 0.f, 0.f, 0.f);
        lam[i] = {pair(g4.x, g4.y), pair(g4.z, g4.w)};
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bool ok = t0 + i < len && kk < p.kc;
      q[i] = ok ? ldg_u2(qp + i * qs) : make_uint2(0u, 0u);
      k[i] = ok ? ldg_u2(kp + i * qs) : make_uint2(0u, 0u);
    }
    if (tid < len) {      // (only threads below C keep a value)
      const size_t i = static_cast<size_t>(ci.tok0 + tid) * p.H + h;
      if (!p.beta_raw) beta_bits = __float_as_uint(__ldg(p.beta + i));
      else if (p.beta_fp32) beta_bits = __ldg(static_cast<const uint32_t*>(p.beta_raw) + i);
      else beta_bits = static_cast<uint32_t>(__ldg(static_cast<const unsigned short*>(p.beta_raw) + i)) << 16;
    }
    // the gate's parameters with the rest: asked for where they are used, behind the wait for g, they cost a round trip of their own
    float al = 0.f;
    float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p.g_raw) {
      al = __ldg(p.A_log + h);
      if (p.dt_bias && kk < p.kc) bias = __ldg(reinterpret_cast<const float4*>(p.dt_bias + static_cast<size_t>(h) * p.kc + kk));
    }
    if (tid == 0) {
      mbar_init(&s.barV, 1);
      fence_mbar_init();
    }
    // the inputs of the tile that will take this CTA's place into L2, one tiled prefetch by each of five warps (500 cycles a piece: by one
    // thread, as it was, the whole CTA waited for them at the next barrier)
    if (lane == 0 && warp >= 8 && warp < 13) {
      const long long nt = static_cast<long long>(blockIdx.x) + p.ahead;
      if (nt < static_cast<long long>(p.map.total()) * p.H) {
        const int tok = static_cast<int>(p.map.info(static_cast<int>(nt / p.H)).tok0), hn = static_cast<int>(nt % p.H);
        switch (warp) {
          case 8: tma_prefetch_rows(&p.tm_g, 0, hn, tok); break;
          case 9: tma_prefetch_rows(&p.tm_q, 0, hn / p.grp, tok); break;
          case 10: tma_prefetch_rows(&p.tm_k, 0, hn / p.grp, tok); break;
          case 11: tma_prefetch_rows(&p.tm_v, 0, hn, tok); break;
          default: tma_prefetch_rows(&p.tm_v, 64, hn, tok); break;
        }
      }
    }
    static_assert(TILE_TT == 16 * PREP_THREADS, "one piece per thread");
    reinterpret_cast<uint4*>(s.Aqk)[tid] = make_uint4(0u, 0u, 0u, 0u);
    if (bf16_gate) {
#pragma unroll
      for (int i = 0; i < 4; ++i) lam[i] = widen(make_uint2(static_cast<uint32_t>(lam[i].a), static_cast<uint32_t>(lam[i].a >> 32)));
    }
    // the gate's activation here instead of in a kernel of its own: one launch less, and the fp32 g is never read back (forward only: never written)
    if (p.g_raw) {
      al = __expf(al);
      // every element first, then the choice: a branch per row would keep the rows' exponentials apart
      auto activate = [&](const int use_lb) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 x = halves(lam[i].a), y = halves(lam[i].b);
          lam[i] = {pair(gate_value(x.x + bias.x, al, use_lb, p.lb), gate_value(x.y + bias.y, al, use_lb, p.lb)),
                    pair(gate_value(y.x + bias.z, al, use_lb, p.lb), gate_value(y.y + bias.w, al, use_lb, p.lb))};
        }
      };
      if (p.use_lb) activate(1);
      else activate(0);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const bool ok = t0 + i < len && kk < p.kc;
        if (ok && p.g_out) *reinterpret_cast<ulonglong2*>(p.g_out + goff + i * gs) = make_ulonglong2(lam[i].a, lam[i].b);
        if (!ok) lam[i] = {0ull, 0ull};
      }
    }
  }
  KDA_DBG_CLOCK(p.dbg, 17);
  // ---- P2: lam, the decay over these four rows -------------------------------------------------------------------------
  {
    const f32x2 le = pair(LOG2E, LOG2E);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = halves(mul2(lam[i].a, le)), y = halves(mul2(lam[i].b, le));
      lam[i] = {pair(ex2(x.x), ex2(x.y)), pair(ex2(y.x), ex2(y.y))};
    }
    sts4(&s.T[warp][kk], mul4c(mul4c(lam[0], lam[1]), mul4c(lam[2], lam[3])));
  }
  // ---- P1b: optional L2 normalisation of q and k rows (result rounded to bf16, as the unfused op does)
  if (p.use_l2norm) {
    float ss[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const F4 x = widen(q[i]), y = widen(k[i]);
      ss[i] = dot(x, x);
      ss[4 + i] = dot(y, y);
    }
    const float r = rsqrtf(butterfly<8>(ss, lane) + L2NORM_EPS);      // slots 0..3: q rows, 4..7: k rows
    const bool keep = KEEP_QN && p.QN != nullptr && h % p.grp == 0;      // once per q/k head
    const long long row0 = static_cast<long long>(ci.tok0 + t0) * p.HQ + h / p.grp;
    if (keep && lane < 8 && t0 + (lane & 3) < len) p.RSTD[(lane >> 2) * p.qrows + row0 + static_cast<long long>(lane & 3) * p.HQ] = r;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      q[i] = narrow(mul4c(widen(q[i]), splat(__shfl_sync(0xffffffffu, r, i))));
      k[i] = narrow(mul4c(widen(k[i]), splat(__shfl_sync(0xffffffffu, r, 4 + i))));
      if (keep && t0 + i < len) {
        *reinterpret_cast<uint2*>(p.QN + (row0 + static_cast<long long>(i) * p.HQ) * KD + kk) = q[i];
        *reinterpret_cast<uint2*>(p.KN + (row0 + static_cast<long long>(i) * p.HQ) * KD + kk) = k[i];
      }
    }
  }
  // k waits in this thread's own part of the k Gam tile (its final value replaces it there): eight registers less
#pragma unroll
  for (int i = 0; i < 4; ++i) *reinterpret_cast<uint2*>(&s.kG[(t0 + i) * QS + kk]) = k[i];
  auto key = [&](int i) { return widen(*reinterpret_cast<const uint2*>(&s.kG[(t0 + i) * QS + kk])); };
  __nv_bfloat16* const mine = s.op + op_base(blk) * QS + kk;      // this block's operand rows, this thread's columns
  auto put = [&](int row, const F4& x) { *reinterpret_cast<uint2*>(mine + row * QS) = narrow(x); };
  // keeps the compiler from carrying widened (fp32) q, k or products of lam from one use to the next: they would not fit the registers
  auto forget = [&] {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      asm volatile("" : "+r"(q[i].x), "+r"(q[i].y), "+l"(lam[i].a), "+l"(lam[i].b));
  };
  if (tid < C) {
    float b = __uint_as_float(beta_bits);
    if (p.beta_raw && tid < len) {
      b = sigmoid_fast(b);
      if (p.beta_out) p.beta_out[static_cast<size_t>(ci.tok0 + tid) * p.H + h] = b;
    }
    s.beta[tid] = b;
  }
  __syncthreads();      // T; beta; Aqk is cleared
  KDA_DBG_CLOCK(p.dbg, 18);

  if constexpr (!SAFE) {
    // ---- P3a: the 4 x 4 diagonal block of these rows pairwise: E = k_j prod(j+1 .. t) is carried upwards per column j and dotted with
    // q_t and k_t.  The 16 values are summed over the lanes four at a time (all at once they do not fit the registers beside lam, q,
    // k, and spills miss the small L1: 2 k cycles of the tile).
    {
      float val[4];
      F4 E = key(0), F;
      val[0] = dot(widen(q[0]), E);
      E = mul4c(E, lam[1]);
      F = key(1);
      val[2] = dot(F, E);
      {
        const F4 qt = widen(q[1]);
        val[1] = dot(qt, E);
        val[3] = dot(qt, F);
      }
      float x = butterfly<4>(val, lane);
      auto two_rows = [&] {            // rows 2 and 3 against the column carried in E
        E = mul4c(E, lam[2]);
        val[0] = dot(widen(q[2]), E);
        val[1] = dot(key(2), E);
        E = mul4c(E, lam[3]);
        val[2] = dot(widen(q[3]), E);
        val[3] = dot(key(3), E);
        return butterfly<4>(val, lane);
      };
      float y = two_rows();
      x = (lane & 4) ? y : x;
      forget();
      E = key(1);
      y = two_rows();
      x = (lane & 12) == 8 ? y : x;
      forget();
      E = key(2);
      val[0] = dot(widen(q[2]), E);
      E = mul4c(E, lam[3]);
      F = key(3);
      val[3] = dot(F, E);
      {
        const F4 qt = widen(q[3]);
        val[1] = dot(qt, F);
        val[2] = dot(qt, E);
      }
      y = butterfly<4>(val, lane);
      x = (lane & 12) == 12 ? y : x;
      if (lane < 16) {      // row, column (two bits per lane) and matrix of the lane's value
        const int r = t0 + ((0xfefafa54u >> (2 * lane)) & 3), cl = t0 + ((0xae550040u >> (2 * lane)) & 3);
        if ((0x8aa4u >> lane) & 1) s.Akk[r * AS + cl] = x;                            // raw; beta_t is applied later
        else *reinterpret_cast<__nv_bfloat16*>(s.Aqk + swz<128>(r, cl)) = __float2bfloat16_rn(p.scale * x);
      }
    }
    forget();
    // ---- P3b: operands of levels 8 and 4
    if (quad >= 2) {                                    // rows 8..15: prod(8 .. i)
      F4 f = quad == 3 ? mul4c(lds4(&s.T[warp - 1][kk]), lam[0]) : lam[0];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (i > 0) f = mul4c(f, lam[i]);
        put(4 * (quad - 2) + i, mul4c(widen(q[i]), f));
        put(8 + 4 * (quad - 2) + i, mul4c(key(i), f));
      }
    } else {                                            // columns 0..7: prod(j+1 .. 7)
      F4 f = quad == 0 ? lds4(&s.T[warp + 1][kk]) : splat(1.f);
#pragma unroll
      for (int j = 3; j >= 0; --j) {
        if (j < 3) f = mul4c(f, lam[j + 1]);
        put(OP_B8 + 4 * quad + j, mul4c(key(j), f));
      }
    }
    forget();
    if (!(quad & 1)) {                                  // level 4, columns 0..3, 8..11: prod up to row 3, 11
      float* const c4 = reinterpret_cast<float*>(s.op + (op_base(blk) + OP_C4) * QS) + 2 * quad * KD + kk;
      sts4(c4 + 3 * KD, key(3));
      F4 f = lam[3];
#pragma unroll
      for (int j = 2; j >= 0; --j) {
        if (j < 2) f = mul4c(f, lam[j + 1]);
        sts4(c4 + j * KD, mul4c(key(j), f));
      }
    }
  } else {
    // ---- P3b, bounded gates: the diagonal 16 x 16 blocks whole, cut between rows 7 and 8: row side prod(8 .. t) above the cut and
    // 1 / prod(t+1 .. 7) below it, column side the reciprocals (every factor within 2^58 under the bound)
    auto inv = [](const F4& f) {
      const float2 a = halves(f.a), b = halves(f.b);
      return F4{pair(__fdividef(1.f, a.x), __fdividef(1.f, a.y)), pair(__fdividef(1.f, b.x), __fdividef(1.f, b.y))};
    };
    if (quad >= 2) {
      F4 f = quad == 3 ? mul4c(lds4(&s.T[warp - 1][kk]), lam[0]) : lam[0];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (i > 0) f = mul4c(f, lam[i]);
        put(4 * quad + i, mul4c(widen(q[i]), f));
        put(16 + 4 * quad + i, mul4c(key(i), f));
        put(32 + 4 * quad + i, mul4c(key(i), inv(f)));
      }
    } else {
      F4 f = quad == 0 ? lds4(&s.T[warp + 1][kk]) : splat(1.f);
#pragma unroll
      for (int i = 3; i >= 0; --i) {
        if (i < 3) f = mul4c(f, lam[i + 1]);
        const F4 r = inv(f);
        put(4 * quad + i, mul4c(widen(q[i]), r));
        put(16 + 4 * quad + i, mul4c(key(i), r));
        put(32 + 4 * quad + i, mul4c(key(i), f));
      }
    }
  }
  asm volatile("bar.sync %0, 128;" ::"r"(1 + blk) : "memory");      // the four warps of this 16-row block
  KDA_DBG_CLOCK(p.dbg, 19);
  forget();
  const __nv_bfloat16* const part = s.op + op_base(blk) * QS;
  if constexpr (!SAFE) {
    float a[1][4];
    if (quad == 0) {             // level 8: accumulator rows 0..7: q rows 8.., rows 8..15: k rows 8..
      prep_mma<1>(a, part, part + OP_B8 * QS, lane);
      const int row = b0 + 8 + gid, col = b0 + 2 * tig;
      *reinterpret_cast<uint32_t*>(s.Aqk + swz<128>(row, col)) = pack_bf16(p.scale * a[0][0], p.scale * a[0][1]);
      *reinterpret_cast<float2*>(&s.Akk[row * AS + col]) = make_float2(a[0][2], a[0][3]);
    } else if (quad & 1) {
      // level 4: these rows, prod from row 4 or 12, against the four columns in front, float32 sums over the lanes.  A lane takes the columns in
      // an order of its own, j = i ^ (lane & 3): the first two steps of the sums then pass values on without choosing any.
      const float* const c4 = reinterpret_cast<const float*>(part + OP_C4 * QS) + 2 * (quad - 1) * KD + kk;
      float w[8];      // q and k of the four rows, column lane & 3, summed over four lanes
      F4 f = lam[0];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        if (t > 0) f = mul4c(f, lam[t]);
        const F4 qt = mul4c(widen(q[t]), f), kt = mul4c(key(t), f);
        float vq[4], vk[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const F4 c = lds4(c4 + (i ^ (lane & 3)) * KD);
          vq[i] = dot(qt, c);
          vk[i] = dot(kt, c);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          vq[i] += __shfl_xor_sync(0xffffffffu, vq[i + 2], 2);
          vk[i] += __shfl_xor_sync(0xffffffffu, vk[i + 2], 2);
        }
        w[2 * t] = vq[0] + __shfl_xor_sync(0xffffffffu, vq[1], 1);
        w[2 * t + 1] = vk[0] + __shfl_xor_sync(0xffffffffu, vk[1], 1);
        forget();
      }
#pragma unroll
      for (int o = 4; o >= 1; o >>= 1) {      // lanes 4, 8, 16 apart
        const bool up = (lane & (16 / o)) != 0;
#pragma unroll
        for (int i = 0; i < o; ++i) {
          const float mine = up ? w[i + o] : w[i];
          const float other = up ? w[i] : w[i + o];
          w[i] = mine + __shfl_xor_sync(0xffffffffu, other, 16 / o);
        }
      }
      const int row = t0 + ((lane >> 1) & 2) + ((lane >> 3) & 1), col = t0 - 4 + (lane & 3);
      if (lane & 16) s.Akk[row * AS + col] = w[0];
      else *reinterpret_cast<__nv_bfloat16*>(s.Aqk + swz<128>(row, col)) = __float2bfloat16_rn(p.scale * w[0]);
    }
  } else {
    // one product per warp: q or k rows of the block against one half of its columns; Aqk keeps j <= t, Akk j < t
    const int is_k = quad >> 1, nh = quad & 1;
    float a[1][4];
    prep_mma<1>(a, part + 16 * is_k * QS, part + (32 + 8 * nh) * QS, lane);
    const int ra = gid, rb = gid + 8, col = 8 * nh + 2 * tig, lim = is_k ? 0 : 1;
    const float v0 = (col < ra + lim) ? a[0][0] : 0.f, v1 = (col + 1 < ra + lim) ? a[0][1] : 0.f;
    const float v2 = (col < rb + lim) ? a[0][2] : 0.f, v3 = (col + 1 < rb + lim) ? a[0][3] : 0.f;
    if (is_k) {
      *reinterpret_cast<float2*>(&s.Akk[(b0 + ra) * AS + b0 + col]) = make_float2(v0, v1);
      *reinterpret_cast<float2*>(&s.Akk[(b0 + rb) * AS + b0 + col]) = make_float2(v2, v3);
    } else {
      *reinterpret_cast<uint32_t*>(s.Aqk + swz<128>((b0 + ra), b0 + col)) = pack_bf16(p.scale * v0, p.scale * v1);
      *reinterpret_cast<uint32_t*>(s.Aqk + swz<128>((b0 + rb), b0 + col)) = pack_bf16(p.scale * v2, p.scale * v3);
    }
  }
  if (quad == 2) {               // the decay over the whole block, for the next phase
    sts4(&s.TB[blk][kk], mul4c(mul4c(lds4(&s.T[warp - 2][kk]), lds4(&s.T[warp - 1][kk])), mul4c(lds4(&s.T[warp][kk]), lds4(&s.T[warp + 1][kk]))));
  }
  __syncthreads();      // the level 8 / 4 operands have been read; TB is there
  KDA_DBG_CLOCK(p.dbg, 20);

  // ---- P3c: operands of level 16, and the tiles QG, KG, k Gam, GL ---------------------------------------------------------
  {
    const uint32_t toff = (static_cast<uint32_t>(lane >> 4) << 13) + static_cast<uint32_t>(t0) * 128u + static_cast<uint32_t>(lane & 1) * 8u;
    unsigned char* const gQG = p.QG + tile * TILE_TK + toff;
    unsigned char* const gKG = p.KG + tile * TILE_TK + toff;
    const uint32_t piece = (lane & 15) >> 1;
    // columns seen from the blocks behind: distance 1 needs only this block's rest, 2 and 3 the blocks in between
    F4 f = splat(1.f);
    if (quad < 3) f = lds4(&s.T[4 * blk + 3][kk]);
    if (quad < 2) f = mul4c(f, lds4(&s.T[4 * blk + 2][kk]));
    if (quad < 1) f = mul4c(f, lds4(&s.T[4 * blk + 1][kk]));
    {
      F4 post = splat(1.f);
      if (blk < 3) post = lds4(&s.TB[blk + 1][kk]);
      if (blk < 2) post = mul4c(post, lds4(&s.TB[blk + 2][kk]));
      if (blk < 1) post = mul4c(post, lds4(&s.TB[3][kk]));
      const int cb = (blk > 0 ? 32 : 0) + 4 * quad;
      // (the block decays between are read again for every row: kept in registers they spilled; bounded gates 1,370 -> 1,336 us at 1 x 32768)
#pragma unroll
      for (int i = 3; i >= 0; --i) {                    // f = prod(i+1 .. last row of the block)
        if (i < 3) f = mul4c(f, lam[i + 1]);
        F4 kf = mul4c(key(i), f);
        *reinterpret_cast<uint2*>(gKG + i * 128 + ((piece ^ ((t0 + i) & 7)) << 4)) = narrow(mul4c(kf, post));
        if (blk < 3) put(cb + i, kf);
        if (blk < 2) {
          kf = mul4c(kf, lds4(&s.TB[blk + 1][kk]));
          put(cb + 16 + i, kf);
        }
        if (blk < 1) put(cb + 32 + i, mul4c(kf, lds4(&s.TB[blk + 2][kk])));
      }
    }
    // decay over the rows of the block in front of these; over the blocks in front
    f = lam[0];
    if (quad > 0) f = mul4c(f, lds4(&s.T[4 * blk][kk]));
    if (quad > 1) f = mul4c(f, lds4(&s.T[4 * blk + 1][kk]));
    if (quad > 2) f = mul4c(f, lds4(&s.T[4 * blk + 2][kk]));
    F4 pre = splat(1.f);
    if (blk > 0) pre = lds4(&s.TB[0][kk]);
    if (blk > 1) pre = mul4c(pre, lds4(&s.TB[1][kk]));
    if (blk > 2) pre = mul4c(pre, lds4(&s.TB[2][kk]));
    if (warp == 15) {
      sts4(reinterpret_cast<float*>(p.GL + tile * TILE_GL) + kk, mul4c(pre, lds4(&s.TB[3][kk])));
    }
    const F4 preq = mul4c(pre, splat(p.scale));
#pragma unroll
    for (int i = 0; i < 4; ++i) {                       // f = prod(first row of the block .. i)
      if (i > 0) f = mul4c(f, lam[i]);
      const F4 qf = mul4c(widen(q[i]), f), kf = mul4c(key(i), f);
      if (blk > 0) {
        put(4 * quad + i, qf);
        put(16 + 4 * quad + i, kf);
      }
      *reinterpret_cast<uint2*>(gQG + i * 128 + ((piece ^ ((t0 + i) & 7)) << 4)) = narrow(mul4c(qf, preq));
      *reinterpret_cast<uint2*>(&s.kG[(t0 + i) * QS + kk]) = narrow(mul4c(kf, pre));
    }
  }
  __syncthreads();
  KDA_DBG_CLOCK(p.dbg, 21);
  // ---- P4a: one warp per block: inverse of the diagonal 16 x 16 block of I + diag(beta) Akk by fp32 forward substitution, a
  // column per lane.  The other twelve warps meanwhile: the level-16 products, six blocks (I, J) x (q, k).
  if (quad == 0) {
    const int cc = lane & 15;
    float x[16];
    const float* A = &s.Akk[b0 * AS + b0];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float s0 = 0.f, s1 = 0.f;
#pragma unroll
      for (int m = 0; m < i; m += 4) {
        const float4 a = *reinterpret_cast<const float4*>(&A[i * AS + m]);      // entries at and above the diagonal are undefined (nothing writes them) and not used
        s0 = fmaf(a.x, x[m], s0);
        if (m + 1 < i) s1 = fmaf(a.y, x[m + 1], s1);
        if (m + 2 < i) s0 = fmaf(a.z, x[m + 2], s0);
        if (m + 3 < i) s1 = fmaf(a.w, x[m + 3], s1);
      }
      x[i] = fmaf(-s.beta[b0 + i], s0 + s1, i == cc ? 1.f : 0.f);
    }
    if (lane < 16) {
#pragma unroll
      for (int i = 0; i < 16; ++i) s.TD[blk][i * DS + cc] = x[i];
    }
  } else {
    const int m = blk * 3 + quad - 1, unit = m >> 1;
    const bool is_k = (m & 1) != 0;
    const int I = (unit < 1) ? 1 : (unit < 3 ? 2 : 3), J = (unit < 1) ? 0 : (unit < 3 ? unit - 1 : unit - 3);
    float a[2][4];
    prep_mma<2>(a, s.op + (op_base(I) + (is_k ? 16 : 0)) * QS, s.op + op_cols(J, I - J) * QS, lane);
    const int ra = 16 * I + gid, rb = ra + 8;
#pragma unroll
    for (int nh = 0; nh < 2; ++nh) {
      const int col = 16 * J + 8 * nh + 2 * tig;
      if (is_k) {
        *reinterpret_cast<float2*>(&s.Akk[ra * AS + col]) = make_float2(a[nh][0], a[nh][1]);
        *reinterpret_cast<float2*>(&s.Akk[rb * AS + col]) = make_float2(a[nh][2], a[nh][3]);
      } else {
        *reinterpret_cast<uint32_t*>(s.Aqk + swz<128>(ra, col)) = pack_bf16(p.scale * a[nh][0], p.scale * a[nh][1]);
        *reinterpret_cast<uint32_t*>(s.Aqk + swz<128>(rb, col)) = pack_bf16(p.scale * a[nh][2], p.scale * a[nh][3]);
      }
    }
  }
  fence_proxy_async();  // Aqk leaves by a bulk store, v arrives in the operand region
  __syncthreads();      // Aqk, Akk, TD complete; the operand region is free
  KDA_DBG_CLOCK(p.dbg, 22);

  if (tid == 128) {      // v, needed by the last phase; AQK
    mbar_expect_tx(&s.barV, TILE_TK);
    tma_load_rows(s.op, &p.tm_v, 0, h, static_cast<int>(ci.tok0), &s.barV);
    tma_load_rows(reinterpret_cast<unsigned char*>(s.op) + 8192, &p.tm_v, 64, h, static_cast<int>(ci.tok0), &s.barV);
    bulk_s2g(p.AQK + tile * TILE_TT, s.Aqk, TILE_TT);
    bulk_commit();
  }
  __nv_bfloat16* const sTB = reinterpret_cast<__nv_bfloat16*>(reinterpret_cast<unsigned char*>(s.op) + TB_OFF);      // Tm diag(beta)
  unsigned char* const sTI = reinterpret_cast<unsigned char*>(s.op) + TI_OFF;                                            // Tm
  auto put_tm = [&](int row, int col, float x, float y) {      // two adjacent entries of Tm = (I + diag(beta) Akk)^-1
    *reinterpret_cast<uint32_t*>(&sTB[row * TS + col]) = pack_bf16(x * s.beta[col], y * s.beta[col + 1]);
    if (p.TI) *reinterpret_cast<uint32_t*>(sTI + swz<128>(row, col)) = pack_bf16(x, y);
  };
  if (warp < 4) {
    // ---- P4b: the two levels of block merges  T21 = -T22 A21 T11  on tensor cores, every fp32 operand split into bf16 hi + lo
    // (three MMAs per product: about 16 bits of mantissa, better than TF32).  A warp owns eight columns from the first product to
    // the last: the accumulators of A21 T11 become the B operand of the second product through movmatrix, without shared memory.
    struct Frag { uint32_t h[4], l[4]; };
    auto split = [](float x, float y, uint32_t& hi, uint32_t& lo) {
      hi = pack_bf16(x, y);
      const float2 f = unpack_bf16(hi);
      lo = pack_bf16(x - f.x, y - f.y);
    };
    auto load_a = [&](Frag& f, const float* A) {                  // 16 x 16, row stride DS
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 v = *reinterpret_cast<const float2*>(&A[(gid + (e & 1) * 8) * DS + tig * 2 + (e >> 1) * 8]);
        split(v.x, v.y, f.h[e], f.l[e]);
      }
    };
    auto load_akk = [&](Frag& f, int r0, int c0) {                // 16 x 16 of diag(beta) Akk
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int r = r0 + gid + (e & 1) * 8;
        const float2 v = *reinterpret_cast<const float2*>(&s.Akk[r * AS + c0 + tig * 2 + (e >> 1) * 8]);
        split(v.x * s.beta[r], v.y * s.beta[r], f.h[e], f.l[e]);
      }
    };
    auto load_b = [&](Frag& f, const float* B, int bc) {          // 16 x 8 (entries 0, 1), row stride DS
#pragma unroll
      for (int e = 0; e < 2; ++e)
        split(B[(tig * 2 + e * 8) * DS + bc + gid], B[(tig * 2 + 1 + e * 8) * DS + bc + gid], f.h[e], f.l[e]);
    };
    auto turn = [&](Frag& f, const float (&c)[4]) {               // accumulators (16 x 8) -> B operand
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        uint32_t hi, lo;
        split(c[2 * e], c[2 * e + 1], hi, lo);
        asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(f.h[e]) : "r"(hi));
        asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(f.l[e]) : "r"(lo));
      }
    };
    auto mma3 = [](float (&c)[4], const Frag& a, const Frag& b) {
      mma16816(c, a.h, b.h[0], b.h[1]);
      mma16816(c, a.h, b.l[0], b.l[1]);
      mma16816(c, a.l, b.h[0], b.h[1]);
    };
    {      // level 1: blocks (1, 0) and (3, 2); warp = (pair, 8 columns)
      const int pr = warp >> 1, bc = 8 * (warp & 1), base = 32 * pr;
      Frag a, b;
      float c1[4] = {0.f, 0.f, 0.f, 0.f}, c2[4] = {0.f, 0.f, 0.f, 0.f};
      load_akk(a, base + 16, base);
      load_b(b, s.TD[2 * pr], bc);
      mma3(c1, a, b);
      turn(b, c1);
      load_a(a, s.TD[2 * pr + 1]);
      mma3(c2, a, b);
      *reinterpret_cast<float2*>(&s.TM[pr][gid * DS + bc + 2 * tig]) = make_float2(-c2[0], -c2[1]);
      *reinterpret_cast<float2*>(&s.TM[pr][(gid + 8) * DS + bc + 2 * tig]) = make_float2(-c2[2], -c2[3]);
      put_tm(base + 16 + gid, base + bc + 2 * tig, -c2[0], -c2[1]);
      put_tm(base + 24 + gid, base + bc + 2 * tig, -c2[2], -c2[3]);
    }
    asm volatile("bar.sync 5, 128;" ::: "memory");
    {      // level 2: rows 32..63, columns 0..31; warp = 8 columns (of block column warp / 2)
      const int bc = 8 * (warp & 1);
      Frag a, b0, b1;
      float x0[4] = {0.f, 0.f, 0.f, 0.f}, x1[4] = {0.f, 0.f, 0.f, 0.f};
      if (warp < 2) {      // T11 = [TD0 0; TM0 TD1]: block column 0 has two blocks, block column 1 only the lower one
        load_b(b0, s.TD[0], bc);
        load_akk(a, 32, 0);
        mma3(x0, a, b0);
        load_akk(a, 48, 0);
        mma3(x1, a, b0);
      }
      load_b(b1, warp < 2 ? s.TM[0] : s.TD[1], bc);
      load_akk(a, 32, 16);
      mma3(x0, a, b1);
      load_akk(a, 48, 16);
      mma3(x1, a, b1);
      turn(b0, x0);
      turn(b1, x1);
      float y0[4] = {0.f, 0.f, 0.f, 0.f}, y1[4] = {0.f, 0.f, 0.f, 0.f};
      load_a(a, s.TD[2]);
      mma3(y0, a, b0);
      load_a(a, s.TM[1]);
      mma3(y1, a, b0);
      load_a(a, s.TD[3]);
      mma3(y1, a, b1);
      const int col = 8 * warp + 2 * tig;
      put_tm(32 + gid, col, -y0[0], -y0[1]);
      put_tm(40 + gid, col, -y0[2], -y0[3]);
      put_tm(48 + gid, col, -y1[0], -y1[1]);
      put_tm(56 + gid, col, -y1[2], -y1[3]);
    }
  } else {
    // ---- the other twelve warps: Tm's diagonal blocks; for the backward the raw k-k products (dbeta) and the zeros of Tm
    const int u = tid - 128;
    for (int i = u; i < C * 8; i += PREP_THREADS - 128) {      // 64 rows x 8 column pairs of the diagonal blocks
      const int r = i >> 3, cp = (i & 7) * 2;
      const float2 x = *reinterpret_cast<const float2*>(&s.TD[r >> 4][(r & 15) * DS + cp]);
      put_tm(r, (r & 48) + cp, x.x, x.y);
    }
    if (p.RKK) {
      unsigned char* const gR = p.RKK + tile * TILE_TT;
      for (int i = u; i < C * 8; i += PREP_THREADS - 128) {
        const int r = i >> 3, pc = i & 7, below = r - pc * 8;      // entries of the piece left of the diagonal
        const uint32_t off = swz<128>(r, pc * 8);
        uint4 o = make_uint4(0u, 0u, 0u, 0u);
        if (below > 0) {
          const float4 a0 = *reinterpret_cast<const float4*>(&s.Akk[r * AS + pc * 8]);
          const float4 a1 = *reinterpret_cast<const float4*>(&s.Akk[r * AS + pc * 8 + 4]);
          o = make_uint4(pack_bf16(a0.x, below > 1 ? a0.y : 0.f), pack_bf16(below > 2 ? a0.z : 0.f, below > 3 ? a0.w : 0.f),
                         pack_bf16(below > 4 ? a1.x : 0.f, below > 5 ? a1.y : 0.f), pack_bf16(below > 6 ? a1.z : 0.f, below > 7 ? a1.w : 0.f));
        }
        *reinterpret_cast<uint4*>(gR + off) = o;
        if ((pc >> 1) > (r >> 4)) *reinterpret_cast<uint4*>(sTI + off) = make_uint4(0u, 0u, 0u, 0u);      // block above the diagonal
      }
    }
  }
  if (!mbar_wait(&s.barV, 0) && tid == 0) atomicOr(p.status, KDA_STATUS_PREP_LOAD_WAIT);
  if (len < C) {      // rows beyond the sequence hold the next one's tokens: clear them
    for (int i = len * 8 + tid; i < C * 8; i += PREP_THREADS) {
      reinterpret_cast<uint4*>(s.op)[i] = make_uint4(0u, 0u, 0u, 0u);
      reinterpret_cast<uint4*>(s.op)[C * 8 + i] = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  __syncthreads();
  KDA_DBG_CLOCK(p.dbg, 23);

  // ---- P5: u^T = v^T (Tm beta)^T,  w = (Tm beta) kGam on tensor cores.  Tm is lower triangular: row tile mt needs the tokens of
  // tiles 0..mt only.  A warp takes the row tiles pr and 3 - pr (five k-steps together, the same for every warp) and 16 columns; the
  // fragments of Tm beta serve both products (A operand of w, B operand of u^T, whose accumulators then hold adjacent
  // tokens of one value row and are stored as pairs).  The tiles leave through shared memory with two bulk stores.
  {
    unsigned char* stUT = reinterpret_cast<unsigned char*>(s.op) + UT_OFF;
    unsigned char* stW = reinterpret_cast<unsigned char*>(s.Akk);
    const int pr = warp & 1, n0 = 16 * (warp >> 1);
    uint32_t a[2][4][4];      // [row tile 3 - pr, pr][k-step][fragment]
    const uint32_t ta0 = smem_u32(&sTB[(16 * (3 - pr) + (lane & 15)) * TS + ((lane >> 4) << 3)]);
    const uint32_t ta1 = smem_u32(&sTB[(16 * pr + (lane & 15)) * TS + ((lane >> 4) << 3)]);
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      if (ks <= 3 - pr) ldsm_x4(a[0][ks], ta0 + ks * 32);
      if (ks < 2 && ks <= pr) ldsm_x4(a[1][ks], ta1 + ks * 32);
    }
    {      // u^T: rows = value columns n0 .. n0 + 15, columns = tokens
      const uint32_t av = smem_u32(s.op) + (static_cast<uint32_t>(n0 >> 6) << 13) + swz<128>((lane & 7) + ((lane >> 4) << 3), (n0 & 63) + (((lane >> 3) & 1) << 3));
      float acc[2][2][4];      // [row tile][8 tokens][fragment]
#pragma unroll
      for (int i = 0; i < 16; ++i) (&acc[0][0][0])[i] = 0.f;
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        if (ks <= 3 - pr) {
          uint32_t x[4];
          ldsm_x4_t(x, av + ks * 2048);
          mma16816(acc[0][0], x, a[0][ks][0], a[0][ks][2]);
          mma16816(acc[0][1], x, a[0][ks][1], a[0][ks][3]);
          if (ks < 2 && ks <= pr) {
            mma16816(acc[1][0], x, a[1][ks & 1][0], a[1][ks & 1][2]);
            mma16816(acc[1][1], x, a[1][ks & 1][1], a[1][ks & 1][3]);
          }
        }
      }
#pragma unroll
      for (int w = 0; w < 2; ++w)
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const int t = (w ? pr : 3 - pr) * 16 + 8 * n + 2 * tig, va = n0 + gid;
          *reinterpret_cast<uint32_t*>(stUT + swz<128>(va, t)) = pack_bf16(acc[w][n][0], acc[w][n][1]);
          *reinterpret_cast<uint32_t*>(stUT + swz<128>(va + 8, t)) = pack_bf16(acc[w][n][2], acc[w][n][3]);
        }
    }
    {      // w: rows = tokens, columns n0 .. n0 + 15
      float acc[2][2][4];
#pragma unroll
      for (int i = 0; i < 16; ++i) (&acc[0][0][0])[i] = 0.f;
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        if (ks <= 3 - pr) {
          uint32_t b[4];
          ldsm_x4_t(b, smem_u32(&s.kG[(ks * 16 + (lane & 7) + (((lane >> 3) & 1) << 3)) * QS + n0 + ((lane >> 4) << 3)]));
          mma16816(acc[0][0], a[0][ks], b[0], b[1]);
          mma16816(acc[0][1], a[0][ks], b[2], b[3]);
          if (ks < 2 && ks <= pr) {
            mma16816(acc[1][0], a[1][ks & 1], b[0], b[1]);
            mma16816(acc[1][1], a[1][ks & 1], b[2], b[3]);
          }
        }
      }
#pragma unroll
      for (int w = 0; w < 2; ++w)
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const int ta = (w ? pr : 3 - pr) * 16 + gid, col = n0 + n * 8 + tig * 2;
          *reinterpret_cast<uint32_t*>(stW + tk_off(ta, col)) = pack_bf16(acc[w][n][0], acc[w][n][1]);
          *reinterpret_cast<uint32_t*>(stW + tk_off(ta + 8, col)) = pack_bf16(acc[w][n][2], acc[w][n][3]);
        }
    }
    fence_proxy_async();   // the staged tiles (generic-proxy writes) are read next by the bulk-copy engine
    __syncthreads();
    if (tid == 0) {
      bulk_s2g(p.UT + tile * TILE_VT, stUT, TILE_VT);
      bulk_s2g(p.W + tile * TILE_TK, stW, TILE_TK);
      if (p.TI) bulk_s2g(p.TI + tile * TILE_TT, sTI, TILE_TT);
      bulk_commit();
      bulk_wait_read<0>();   // shared memory must stay valid until the engine has read it
    }
    if (tid == 128) bulk_wait_read<0>();
    KDA_DBG_CLOCK(p.dbg, 24);
  }
}

int launch_prepare(PrepParams& p, long long tiles, long long tokens, bool keep_qn, bool safe_gate, cudaStream_t st) {
  static DeviceOnce once;
  const int smem = PREP_SMEM;
  const int rc = once.run([&] {
    cudaError_t e = cudaSuccess;
    for (auto fn : {kda_chunk_prepare_kernel<false, false>, kda_chunk_prepare_kernel<true, false>, kda_chunk_prepare_kernel<false, true>,
                    kda_chunk_prepare_kernel<true, true>}) {
      if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    }
    return e;
  });
  if (rc != KDA_OK) return rc;
  if (tiles > 0x7fffffffLL) return KDA_E_SHAPE;
  p.ahead = 2 * sm_count();
  if (make_rows_tmap(&p.tm_v, p.v, false, tokens, p.H, p.vc, 64, C, true)) return KDA_E_TMAP;
  if (tiles > p.ahead &&
      (make_rows_tmap(&p.tm_q, p.q, false, tokens, p.HQ, p.kc, KD, C, false) || make_rows_tmap(&p.tm_k, p.k, false, tokens, p.HQ, p.kc, KD, C, false) ||
       make_rows_tmap(&p.tm_g, p.g_raw ? p.g_raw : p.g, !p.g_raw || p.g_fp32, tokens, p.H, p.kc, KD, C, false)))
    return KDA_E_TMAP;
  const unsigned grid = static_cast<unsigned>(tiles);
  const auto kernel = safe_gate ? (keep_qn ? kda_chunk_prepare_kernel<true, true> : kda_chunk_prepare_kernel<false, true>)
                                : (keep_qn ? kda_chunk_prepare_kernel<true, false> : kda_chunk_prepare_kernel<false, false>);
  if (!p.clear_status) return static_cast<int>(launch_chained(kernel, grid, PREP_THREADS, smem, st, p));      // behind the tables kernel
  kernel<<<grid, PREP_THREADS, smem, st>>>(p);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace kda
