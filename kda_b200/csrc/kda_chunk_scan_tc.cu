// Forward state scan of chunked KDA on tcgen05 with the fp32 state resident in tensor memory (sm_100a).
//
// One CTA per (sequence, head) walks the sequence's chunks in order.  TMEM lane = value column v, so the state
// is held transposed, hT[v][k] (128 lanes x 128 fp32 columns), for the whole sequence.  Per chunk:
//   state pass   every thread reads its slice of hT and leaves the bf16 copy that the next products use as their A operand: forward only in
//                tensor memory, in training as a K-major tile in shared memory, which is also stored as the chunk's HS tile;
//                hT * Gam_last goes back to TMEM (forward only: while products 1 execute, which do not need it)
//   products 1   v_part^T = hT_bf16 w^T,   o^T = hT_bf16 qg^T                          (M=128 v, N=64 t, K=128 k)
//   epilogue 1   v_new^T = u^T - v_part^T  -> bf16, A operand of products 2 (in training the chunk's VNEWT tile)
//   products 2   hT += v_new^T kg,   o^T += v_new^T Aqk^T                              (K = 64 tokens)
//   epilogue 2   o^T -> bf16 -> staged in shared memory -> coalesced stores of o[t][v]; forward only a chunk later, under products 2.
// What bounds it: HBM from about 150 units on (0.73 ms, 0.95 of the copy rate at 8 x 8192 x 32 in training), below that the chain of a chunk's
// phases, in which the products wait for shared memory.  With A there a product reads 6 KB, with A in tensor memory 2: 4 x 4096 x 32 heads (128
// units), whole call: 535 -> 523 us; with o read out under the next products 520, with the decay behind the hand-over 515.  In training the same costs
// nothing and gains nothing (604 and 610 us at 6 x 2000 x 16): the tiles have to be written to shared memory in any case.
// Operand tiles (W, QG, KG, AQK, UT, GL of the chunk) arrive through a 2-stage TMA bulk-copy / mbarrier ring.
#include "kda_chunk.cuh"
#include "kda_device.cuh"
#include "kda_scan.cuh"
#include "kda_umma.cuh"

namespace kda {

namespace {

constexpr int SCT = 256;     // 8 compute warps: TMEM lane quadrant = warp & 3, column half = warp >> 2
constexpr int SNT = SCT + 32;  // + one warp whose first lane issues every MMA, bulk copy and bulk store: the time it spends issuing
                             // (about 75 cycles per product, 760 cycles for a stage refill) stays off the compute warps' path

struct TcScanStage {
  unsigned char W[TILE_TK], QG[TILE_TK], KG[TILE_TK], AQK[TILE_TT], UT[TILE_VT];
  float GL[KD];
  unsigned char pad[512];
};
static_assert(sizeof(TcScanStage) % 1024 == 0, "stage must keep 1024-byte alignment");
constexpr unsigned TC_STAGE_TX = 3 * TILE_TK + TILE_TT + TILE_VT + TILE_GL;

struct TcScanSmem {
  TcScanStage st[2];
  unsigned char Hb[TILE_VK];     // bf16 copy of hT: two [128 v][64 k] spans (K-major A operand; = the HS tile image)
  unsigned char VNT[TILE_VT];    // bf16 v_new^T [128 v][64 t] (K-major A operand; = the VNEWT tile image)
  __nv_bfloat16 oS[C * VD];      // o staged as [64 t][128 v]
  uint64_t full[2], barM;
  uint32_t tmem_slot;
};
static_assert(sizeof(TcScanSmem) + 1024 <= 227 * 1024, "TcScanSmem too large");

// TMEM columns; o is double buffered: C_O + 64 * (chunk & 1); forward only: the bf16 copies of hT and v_new^T, two to a column
constexpr int C_H = 0, C_VN = 128, C_O = 192, C_HB = 320, C_VB = 384;

__device__ __forceinline__ uint4 pack8f(const float* v) {
  return make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
}
__device__ __forceinline__ unsigned char* swp(unsigned char* tile, int row, int chunk) {
  return tile + row * 128 + (((chunk ^ row) & 7) << 4);
}

}  // namespace

// TRAIN: the bf16 copies of hT and v_new^T go through shared memory, from where they also leave as the chunk's HS and VNEWT tiles.  Otherwise they
// stay in tensor memory: the products read their A operand there, and shared memory feeds B alone.
template <bool TRAIN>
__global__ void __launch_bounds__(SNT, 1) kda_chunk_scan_tc_kernel(const ScanParams p) {
  chain_point();
  extern __shared__ unsigned char smem_raw[];
  TcScanSmem& s = *reinterpret_cast<TcScanSmem*>(smem_raw + pad_to_1024(smem_raw));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int q4 = warp & 3, half = warp >> 2;
  const int seq = p.map.started(blockIdx.x / p.H), h = blockIdx.x % p.H;
  const int c_begin = p.map.first_chunk(seq), c_end = p.map.first_chunk(seq + 1);
  const int nchunks = c_end - c_begin;
  const long long seq_tok0 = p.map.first_token(seq), seq_tok1 = p.map.first_token(seq + 1);
  const int v = 32 * q4 + lane;                       // this thread's value column = TMEM lane

  if (tid == 0) {
    mbar_init(&s.full[0], 1);
    mbar_init(&s.full[1], 1);
    mbar_init(&s.barM, 1);
    fence_mbar_init();
  }
  if (warp == 0) umma::tmem_alloc(&s.tmem_slot, 512);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tb = s.tmem_slot;
  const uint32_t tq = tb + (static_cast<uint32_t>(32 * q4) << 16);

  auto issue_load = [&](int i) {                      // issuing thread: operand tiles of the sequence's chunk i
    TcScanStage& d = s.st[i & 1];
    const size_t tile = static_cast<size_t>(c_begin + i) * p.H + h;
    mbar_expect_tx(&s.full[i & 1], TC_STAGE_TX);
    bulk_g2s(d.W, p.W + tile * TILE_TK, TILE_TK, &s.full[i & 1]);
    bulk_g2s(d.QG, p.QG + tile * TILE_TK, TILE_TK, &s.full[i & 1]);
    bulk_g2s(d.KG, p.KG + tile * TILE_TK, TILE_TK, &s.full[i & 1]);
    bulk_g2s(d.AQK, p.AQK + tile * TILE_TT, TILE_TT, &s.full[i & 1]);
    bulk_g2s(d.UT, p.UT + tile * TILE_VT, TILE_VT, &s.full[i & 1]);
    bulk_g2s(d.GL, p.GL + tile * TILE_GL, TILE_GL, &s.full[i & 1]);
  };
  const bool issuer = warp == 8, lead = issuer && lane == 0;
  if (lead) {
    if (nchunks > 0) issue_load(0);
    if (nchunks > 1) issue_load(1);
  }

  // initial state -> TMEM: lane v, columns k = 64 half .. +63
  if (!issuer) {
    const size_t sb = (static_cast<size_t>(seq) * p.H + h) * p.kc * p.vc;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      float x[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int kk = 64 * half + 16 * g + i;
        x[i] = p.h0 && kk < p.kc && v < p.vc ? __ldg(p.h0 + sb + static_cast<size_t>(kk) * p.vc + v) : 0.f;
      }
      umma::tmem_st16(tq + C_H + 64 * half + 16 * g, x);
    }
    umma::tmem_st_wait();
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();

  // o of chunk i: out of tensor memory into the staging tile; from there in coalesced rows (compute warps)
  auto stage_o = [&](int i) {
    const uint32_t to = C_O + 64 * (i & 1);
    float x[16], y[16];
    umma::tmem_ld16(tq + to + 32 * half, x);
    umma::tmem_ld16(tq + to + 32 * half + 16, y);
    umma::tmem_ld_wait();
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      s.oS[(32 * half + e) * VD + v] = __float2bfloat16_rn(x[e]);
      s.oS[(32 * half + 16 + e) * VD + v] = __float2bfloat16_rn(y[e]);
    }
  };
  auto store_o = [&](long long tok0, int len) {
    asm volatile("bar.sync 1, 256;" ::: "memory");      // the eight compute warps only
    for (int e = tid; e < C * 16; e += SCT) {
      const int r = e >> 4, pc = e & 15;
      if (r < len && pc * 8 < p.vc)
        *reinterpret_cast<uint4*>(p.o + (static_cast<size_t>(tok0 + r) * p.H + h) * p.vc + pc * 8) = *reinterpret_cast<const uint4*>(&s.oS[r * VD + pc * 8]);
    }
  };

  auto decay = [](float (&x)[16], const float* gl) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float4 y = *reinterpret_cast<const float4*>(gl + 4 * e);
      x[4 * e] *= y.x; x[4 * e + 1] *= y.y; x[4 * e + 2] *= y.z; x[4 * e + 3] *= y.w;
    }
  };

  uint32_t mph = 0;
  bool alive = true;
  for (int i = 0; i < nchunks; ++i) {       // a failed wait leaves through the uniform vote at the top of the next iteration
    TcScanStage& d = s.st[i & 1];
    const int c = c_begin + i;
    // every chunk of this CTA belongs to its one sequence: first token and length by arithmetic (a table look-up would
    // be three dependent loads on the chunk-to-chunk chain)
    struct { long long tok0; int len; } ci;
    ci.tok0 = seq_tok0 + static_cast<long long>(i) * C;
    ci.len = static_cast<int>(seq_tok1 - ci.tok0 < C ? seq_tok1 - ci.tok0 : C);
    const size_t tile = static_cast<size_t>(c) * p.H + h;
    const uint32_t to = C_O + 64 * (i & 1);
    long long* const dbg = (i == 8) ? p.dbg : nullptr;      // development aid: clocks of a steady-state chunk
    KDA_DBG_CLOCK(dbg, 32);

    if (!mbar_wait(&s.full[i & 1], (i >> 1) & 1)) alive = false;
    // the previous chunk's bulk stores must have read Hb / VNT before they are rewritten
    if (lead) bulk_wait_read<0>();
    alive = __syncthreads_and(alive);
    if (!alive) {
      if (tid == 0) atomicOr(p.status, 1u);
      break;
    }
    KDA_DBG_CLOCK(dbg, 33);

    // ---- state pass: bf16 copy of hT for the products, hT *= Gam_last in TMEM (forward only: behind the barrier, the products do not need it) ----
    float hx[TRAIN ? 1 : 4][16];
    if (!issuer) {
      if constexpr (TRAIN) {
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          float x[16];
          umma::tmem_ld16(tq + C_H + 64 * half + 16 * g, x);
          umma::tmem_ld_wait();
          *reinterpret_cast<uint4*>(swp(s.Hb + half * 16384, v, 2 * g)) = pack8f(&x[0]);
          *reinterpret_cast<uint4*>(swp(s.Hb + half * 16384, v, 2 * g + 1)) = pack8f(&x[8]);
          decay(x, &d.GL[64 * half + 16 * g]);
          umma::tmem_st16(tq + C_H + 64 * half + 16 * g, x);
        }
        umma::tmem_st_wait();
        fence_proxy_async();
      } else {
#pragma unroll
        for (int g = 0; g < 4; ++g) umma::tmem_ld16(tq + C_H + 64 * half + 16 * g, hx[g]);
        umma::tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < 4; ++g) umma::tmem_st8(tq + C_HB + 32 * half + 8 * g, pack8f(&hx[g][0]), pack8f(&hx[g][8]));
        umma::tmem_st_wait();
      }
    }
    KDA_DBG_CLOCK(dbg, 34);
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    KDA_DBG_CLOCK(dbg, 35);

    // ---- products 1: the chain from chunk to chunk runs through v_part only; it goes first with its own commit, the
    // products for o execute behind it while the compute warps already turn v_part into v_new
    if (lead) {
      const uint32_t aHb = smem_u32(s.Hb), aW = smem_u32(d.W), aQG = smem_u32(d.QG);
      constexpr uint32_t id1 = umma::instr_desc(128, 64, false, false);
      const uint64_t dH0 = umma::desc_kmajor(aHb, 0), dH1 = umma::desc_kmajor(aHb + 16384, 0);
      const uint64_t dW0 = umma::desc_kmajor(aW, 0), dW1 = umma::desc_kmajor(aW + 8192, 0);
      const uint64_t dQ0 = umma::desc_kmajor(aQG, 0), dQ1 = umma::desc_kmajor(aQG + 8192, 0);
#pragma unroll
      for (int sK = 0; sK < 8; ++sK) {
        const uint64_t o2 = static_cast<uint64_t>(sK & 3) * 2u;
        if constexpr (TRAIN) umma::mma_ss(tb + C_VN, ((sK >> 2) ? dH1 : dH0) + o2, ((sK >> 2) ? dW1 : dW0) + o2, id1, sK > 0);      // v_part^T = hT w^T
        else umma::mma_ts(tb + C_VN, tb + C_HB + 8 * sK, ((sK >> 2) ? dW1 : dW0) + o2, id1, sK > 0);
      }
      umma::commit(&s.barM);
#pragma unroll
      for (int sK = 0; sK < 8; ++sK) {
        const uint64_t o2 = static_cast<uint64_t>(sK & 3) * 2u;
        if constexpr (TRAIN) umma::mma_ss(tb + to, ((sK >> 2) ? dH1 : dH0) + o2, ((sK >> 2) ? dQ1 : dQ0) + o2, id1, sK > 0);        // o^T = hT qg^T
        else umma::mma_ts(tb + to, tb + C_HB + 8 * sK, ((sK >> 2) ? dQ1 : dQ0) + o2, id1, sK > 0);
      }
      if constexpr (TRAIN) {                            // the bf16 state image is the chunk's HS tile
        bulk_s2g(p.HS + tile * TILE_VK, s.Hb, TILE_VK);
        bulk_commit();
      }
    }
    __syncwarp();

    // ---- epilogue 1: v_new^T = u^T - v_part^T -> bf16 tile --------------------------------------------------------------
    if (!issuer) {
      if constexpr (!TRAIN) {
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          decay(hx[g], &d.GL[64 * half + 16 * g]);
          umma::tmem_st16(tq + C_H + 64 * half + 16 * g, hx[g]);
        }
        umma::tmem_st_wait();
      }
      if (!mbar_wait(&s.barM, mph & 1)) alive = false;
      umma::fence_after_sync();
      KDA_DBG_CLOCK(dbg, 36);
      if (alive) {
        float x[16], y[16];
        umma::tmem_ld16(tq + C_VN + 32 * half, x);
        umma::tmem_ld16(tq + C_VN + 32 * half + 16, y);
        umma::tmem_ld_wait();
        uint4 w[4];
#pragma unroll
        for (int cix = 0; cix < 4; ++cix) {
          const uint4 u4 = *reinterpret_cast<const uint4*>(swp(d.UT, v, 4 * half + cix));
          const uint32_t uw[4] = {u4.x, u4.y, u4.z, u4.w};
          float* src = (cix < 2) ? &x[8 * cix] : &y[8 * (cix - 2)];
          float r[8];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 uu = unpack_bf16(uw[e]);
            r[2 * e] = uu.x - src[2 * e];
            r[2 * e + 1] = uu.y - src[2 * e + 1];
          }
          w[cix] = pack8f(r);
          if constexpr (TRAIN) *reinterpret_cast<uint4*>(swp(s.VNT, v, 4 * half + cix)) = w[cix];
        }
        if constexpr (!TRAIN) {
          umma::tmem_st8(tq + C_VB + 16 * half, w[0], w[1]);
          umma::tmem_st8(tq + C_VB + 16 * half + 8, w[2], w[3]);
          umma::tmem_st_wait();
        }
      }
      if constexpr (TRAIN) fence_proxy_async();
    }
    ++mph;
    umma::fence_before_sync();
    alive = __syncthreads_and(alive);
    if (!alive) {
      if (tid == 0) atomicOr(p.status, 2u);
      break;
    }
    umma::fence_after_sync();
    KDA_DBG_CLOCK(dbg, 37);

    // ---- products 2 ---------------------------------------------------------------------------------------------------
    if (lead) {
      const uint32_t aVN = smem_u32(s.VNT), aKG = smem_u32(d.KG), aAQ = smem_u32(d.AQK);
      constexpr uint32_t idH = umma::instr_desc(128, 128, false, true);      // B = kg as MN-major: rows t, two spans of 64 k
      constexpr uint32_t idO = umma::instr_desc(128, 64, false, false);
      const uint64_t dV = umma::desc_kmajor(aVN, 0), dK = umma::smem_desc(aKG, 8192, umma::ATOM_BYTES), dA = umma::desc_kmajor(aAQ, 0);
#pragma unroll
      for (int sK = 0; sK < 4; ++sK) {
        if constexpr (TRAIN) {
          umma::mma_ss(tb + C_H, dV + static_cast<uint64_t>(sK) * 2u, dK + static_cast<uint64_t>(sK) * 128u, idH, 1);      // hT += v_new^T kg
          umma::mma_ss(tb + to, dV + static_cast<uint64_t>(sK) * 2u, dA + static_cast<uint64_t>(sK) * 2u, idO, 1);         // o^T += v_new^T Aqk^T
        } else {
          umma::mma_ts(tb + C_H, tb + C_VB + 8 * sK, dK + static_cast<uint64_t>(sK) * 128u, idH, 1);
          umma::mma_ts(tb + to, tb + C_VB + 8 * sK, dA + static_cast<uint64_t>(sK) * 2u, idO, 1);
        }
      }
      umma::commit(&s.barM);
      if constexpr (TRAIN) {
        bulk_s2g(p.VNEWT + tile * TILE_VT, s.VNT, TILE_VT);
        bulk_commit();
      }
    }
    __syncwarp();
    if constexpr (!TRAIN)
      if (!issuer && i > 0) {      // the previous chunk's o
        stage_o(i - 1);
        store_o(ci.tok0 - C, C);
      }
    if (!mbar_wait(&s.barM, mph & 1)) alive = false;
    ++mph;
    umma::fence_after_sync();
    KDA_DBG_CLOCK(dbg, 38);
    if (issuer) {
      // this stage's operand tiles are free: fetch chunk i + 2 into it (the compute warps do not wait for this)
      if (lead && alive && i + 2 < nchunks) issue_load(i + 2);
      __syncwarp();
      continue;
    }

    // ---- epilogue 2 (compute warps): o^T -> bf16 -> staged [t][v] -> coalesced rows; forward only: of the last chunk, for the others see above
    if (TRAIN || i == nchunks - 1) {
      if constexpr (!TRAIN) asm volatile("bar.sync 1, 256;" ::: "memory");      // the chunk before has left the staging tile
      if (alive) stage_o(i);
      umma::fence_before_sync();
      store_o(ci.tok0, ci.len);
    }
    // (the next iteration's first barrier orders these reads of oS before it is rewritten)
    KDA_DBG_CLOCK(dbg, 39);
  }
  alive = __syncthreads_and(alive);

  // final state
  if (alive && p.ht && !issuer) {
    umma::fence_after_sync();
    const size_t sb = (static_cast<size_t>(seq) * p.H + h) * p.kc * p.vc;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      float x[16];
      umma::tmem_ld16(tq + C_H + 64 * half + 16 * g, x);
      umma::tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const int kk = 64 * half + 16 * g + e;
        if (kk < p.kc && v < p.vc) p.ht[sb + static_cast<size_t>(kk) * p.vc + v] = x[e];
      }
    }
  }
  if (!alive && tid == 0) {              // a wait gave up: loads and products may still be under way
    mbar_drain(&s.full[0]);
    mbar_drain(&s.full[1]);
    mbar_drain(&s.barM);
  }
  if (lead) bulk_wait<0>();              // outstanding bulk stores read shared memory that dies with the CTA
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tb, 512);
}

int launch_scan_tc(const ScanParams& p, int blocks, cudaStream_t st) {
  static DeviceOnce once;
  const int smem = static_cast<int>(sizeof(TcScanSmem)) + 1024;
  const int rc = once.run([&] {
    cudaError_t e = cudaFuncSetAttribute(kda_chunk_scan_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kda_chunk_scan_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    return e;
  });
  if (rc != KDA_OK) return rc;
  return static_cast<int>(launch_chained(p.HS ? kda_chunk_scan_tc_kernel<true> : kda_chunk_scan_tc_kernel<false>, blocks, SNT, smem, st, p));
}

}  // namespace kda
