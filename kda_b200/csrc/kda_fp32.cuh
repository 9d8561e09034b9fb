// float32 chunked path: tile formats, parameters, and the matrix products on tcgen05 kind::tf32 with every fp32 operand split in two.
//
// x = hi + lo, hi = x rounded to TF32, lo = the rest (exact in fp32, rounded to TF32 by the tensor core): a product is
// A_hi B_hi + A_hi B_lo + A_lo B_hi with fp32 accumulation, relative error about 2^-22 -- float32 results from the tensor cores.
// Operands are staged by the threads from fp32 rows in global memory (or from tensor memory) into pairs of SW128 tiles of
// 32 fp32 columns (128-byte rows, K-major: the only order TF32 operands have here; the other orientation is turned while staging).
#pragma once

#include "kda_chunk.cuh"
#include "kda_umma.cuh"

namespace kda {

// Workspace tiles per (chunk, head), plain row-major fp32, 128 columns wide whatever the tensors' widths (zero beyond):
//   W, QG, KG [64 t][128 k]   U [64 t][128 v]   AQK [64 t][64 j]   GL [128]
//   training: TM = (I + diag(beta) Akk)^-1 and RKK = raw <k_t D, k_j> [64][64], KB = k Gam [64 t][128 k], HS [128 k][128 v] state
//   at chunk start, VN [64 t][128 v]; QN, KN [64 t][128 k] the normalised rows (use_qk_l2norm)
//   backward: DH [128 k][128 v] its gradient at chunk end, DVN [64 t][128 v]; DQ, DK [tokens][H][kc] w.r.t. the (normalised) rows
constexpr size_t F_TK = size_t(C) * KD * 4, F_TT = size_t(C) * C * 4, F_KV = size_t(KD) * VD * 4;

struct F32Ws {
  unsigned* status;
  int *seq_chunk_off, *chunk_seq, *seq_order;
  float *W, *QG, *KG, *U, *AQK, *GL, *TM, *RKK, *KB, *HS, *VN, *QN, *KN, *DH, *DVN, *DQ, *DK;
  size_t fwd_bytes, bwd_bytes;
};
inline F32Ws carve_f32(unsigned char* base, unsigned char* bwd_base, int64_t tokens, int N, int H, bool save, bool keep_qn) {
  F32Ws w{};
  const size_t NTmax = static_cast<size_t>(tokens / C + N), tiles = NTmax * static_cast<size_t>(H);
  size_t off = 0;
  unsigned char* b = base;
  auto take = [&](size_t bytes) { unsigned char* p = b ? b + off : nullptr; off += align_up(bytes); return p; };
  auto takef = [&](size_t bytes) { return reinterpret_cast<float*>(take(bytes)); };
  w.status = reinterpret_cast<unsigned*>(take(16));
  w.seq_chunk_off = reinterpret_cast<int*>(take(sizeof(int) * (static_cast<size_t>(N) + 1)));
  w.chunk_seq = reinterpret_cast<int*>(take(sizeof(int) * (NTmax + 1)));
  w.seq_order = reinterpret_cast<int*>(take(sizeof(int) * (static_cast<size_t>(N) + 1)));
  w.W = takef(tiles * F_TK); w.QG = takef(tiles * F_TK); w.KG = takef(tiles * F_TK); w.U = takef(tiles * F_TK);
  w.AQK = takef(tiles * F_TT); w.GL = takef(tiles * KD * 4);
  if (save) {
    w.TM = takef(tiles * F_TT); w.RKK = takef(tiles * F_TT); w.KB = takef(tiles * F_TK); w.HS = takef(tiles * F_KV); w.VN = takef(tiles * F_TK);
    if (keep_qn) { w.QN = takef(tiles * F_TK); w.KN = takef(tiles * F_TK); }
  }
  w.fwd_bytes = off;
  off = 0;
  b = bwd_base;
  w.DH = takef(tiles * F_KV); w.DVN = takef(tiles * F_TK);
  w.DQ = takef(static_cast<size_t>(tokens) * H * KD * 4); w.DK = takef(static_cast<size_t>(tokens) * H * KD * 4);
  w.bwd_bytes = off;
  return w;
}

struct F32Params {
  const float *q, *k, *v, *g, *beta, *h0, *d_o, *d_ht;
  float *o, *ht, *dq, *dk, *dv, *dg, *dbeta, *dh0;
  F32Ws w;
  ChunkMap map;
  bool clear_status, save;
  int H, HQ, grp, kc, vc, use_l2;
  float scale;
};

int launch_f32_fwd(const F32Params& p, long long tiles, cudaStream_t st);      // prepare, forward scan
int launch_f32_bwd(const F32Params& p, long long tiles, cudaStream_t st);      // reverse scan, per-chunk backward
int launch_f32_finish(const F32Params& p, long long rows, cudaStream_t st);    // dq, dk through group sums and the normalisation
inline ChunkMap chunk_map(const F32Ws& w, const int32_t* cu, int64_t tokens, int N) {
  ChunkWs c{};
  c.seq_chunk_off = w.seq_chunk_off; c.chunk_seq = w.chunk_seq; c.seq_order = w.seq_order;
  return chunk_map(c, cu, tokens, N);
}

#ifdef __CUDACC__
namespace f32 {

constexpr int NT = 512;                       // 16 warps: tensor-memory lane quadrant = warp & 3, column part = warp >> 2
constexpr uint32_t S64 = 64 * 128, S128 = 128 * 128;      // bytes of one 32-column slice of a 64- / 128-row operand (hi or lo)

__host__ __device__ constexpr uint32_t idesc(int M, int N) {      // kind::tf32, fp32 accumulation, both operands K-major
  return (1u << 4) | (2u << 7) | (2u << 10) | (static_cast<uint32_t>(N >> 3) << 17) | (static_cast<uint32_t>(M >> 4) << 24);
}
// D (+)= A B^T over one 32-column slice: a, b = shared-memory addresses of the hi tiles, alo, blo = bytes from there to the lo tiles.
// One asm block for the twelve products (hi hi + hi lo + lo hi of four k-steps): consecutive products then issue about 60 cycles apart,
// as separate statements 88.
__device__ __forceinline__ void mma_slice(uint32_t d, uint32_t a, uint32_t alo, uint32_t b, uint32_t blo, uint32_t id, bool acc) {
  asm volatile(
      "{\n\t"
      ".reg .pred p0, p1;\n\t"
      ".reg .b64 ah, al, bh, bl;\n\t"
      "setp.ne.b32 p0, %6, 0;\n\t"
      "setp.eq.b32 p1, %6, %6;\n\t"
      "mov.b64 ah, %1;\n\t"
      "mov.b64 al, %2;\n\t"
      "mov.b64 bh, %3;\n\t"
      "mov.b64 bl, %4;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], ah, bh, %5, p0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], ah, bl, %5, p1;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], al, bh, %5, p1;\n\t"
      "add.u64 ah, ah, 2;\n\t"
      "add.u64 al, al, 2;\n\t"
      "add.u64 bh, bh, 2;\n\t"
      "add.u64 bl, bl, 2;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], ah, bh, %5, p1;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], ah, bl, %5, p1;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], al, bh, %5, p1;\n\t"
      "add.u64 ah, ah, 2;\n\t"
      "add.u64 al, al, 2;\n\t"
      "add.u64 bh, bh, 2;\n\t"
      "add.u64 bl, bl, 2;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], ah, bh, %5, p1;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], ah, bl, %5, p1;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], al, bh, %5, p1;\n\t"
      "add.u64 ah, ah, 2;\n\t"
      "add.u64 al, al, 2;\n\t"
      "add.u64 bh, bh, 2;\n\t"
      "add.u64 bl, bl, 2;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], ah, bh, %5, p1;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], ah, bl, %5, p1;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], al, bh, %5, p1;\n\t"
      "}\n" ::"r"(d),
      "l"(umma::desc_kmajor(a, 0)), "l"(umma::desc_kmajor(a + alo, 0)), "l"(umma::desc_kmajor(b, 0)), "l"(umma::desc_kmajor(b + blo, 0)), "r"(id),
      "r"(static_cast<uint32_t>(acc))
      : "memory");
}
__device__ __forceinline__ float tf32_hi(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}
// four adjacent columns (16-byte piece `piece` of row `row`) of an operand slice: hi at tile, lo at tile + lo
__device__ __forceinline__ void put4(unsigned char* tile, uint32_t lo, int row, int piece, const float4 x) {
  unsigned char* const p = tile + row * 128 + (((piece ^ row) & 7) << 4);
  const float4 h = make_float4(tf32_hi(x.x), tf32_hi(x.y), tf32_hi(x.z), tf32_hi(x.w));
  *reinterpret_cast<float4*>(p) = h;
  *reinterpret_cast<float4*>(p + lo) = make_float4(x.x - h.x, x.y - h.y, x.z - h.z, x.w - h.w);
}
__device__ __forceinline__ void put1(unsigned char* tile, uint32_t lo, int row, int col, float x) {      // col 0..31
  unsigned char* const p = tile + row * 128 + ((((col >> 2) ^ row) & 7) << 4) + (col & 3) * 4;
  const float h = tf32_hi(x);
  *reinterpret_cast<float*>(p) = h;
  *reinterpret_cast<float*>(p + lo) = x - h;
}
__device__ __forceinline__ float4 ld4(const float* p, bool ok) { return ok ? __ldg(reinterpret_cast<const float4*>(p)) : make_float4(0.f, 0.f, 0.f, 0.f); }
__device__ __forceinline__ float4 mul4(float s, const float4 x) { return make_float4(s * x.x, s * x.y, s * x.z, s * x.w); }
// waits for a commit (bounded); a wait that gives up leaves its mark in the status word and the results are incomplete
__device__ __forceinline__ void wait_mma(uint64_t* bar, uint32_t& phase, unsigned* status, unsigned bit) {
  if (!mbar_wait(bar, phase & 1) && (threadIdx.x & 31) == 0) atomicOr(status, bit);
  ++phase;
  umma::fence_after_sync();
}
// makes staged operands visible to the tensor core, for the whole CTA
__device__ __forceinline__ void staged() {
  fence_proxy_async();
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
}

// Operand [64 rows][128 columns] (four slices) from rows of 128 floats: piece loads of this thread's four items, then the tiles.
// Item i of thread tid: row (tid + 512 i) / 32, float4 (tid + 512 i) % 32 -- a warp covers one row.
__device__ __forceinline__ void load64(float4 (&x)[4], const float* tile) {
#pragma unroll
  for (int i = 0; i < 4; ++i) x[i] = __ldg(reinterpret_cast<const float4*>(tile) + threadIdx.x + NT * i);
}
__device__ __forceinline__ void put64(unsigned char* dst, const float4 (&x)[4]) {      // slices 2 S64 apart, lo S64 behind hi
  const int c4 = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < 4; ++i) put4(dst + (c4 >> 3) * 2 * S64, S64, static_cast<int>(threadIdx.x >> 5) + 16 * i, c4 & 7, x[i]);
}
// The transpose of a [64 t][128] tile as an operand of 128 rows and two 32-column slices over t: item = (row, four tokens), lanes
// along the rows: coalesced scalar loads, conflict-free 16-byte stores.
__device__ __forceinline__ void load64t(float4 (&x)[4], const float* tile) {
  const int r = threadIdx.x & 127, t4 = threadIdx.x >> 7;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float* p = tile + (4 * (t4 + 4 * i)) * 128 + r;
    x[i] = make_float4(__ldg(p), __ldg(p + 128), __ldg(p + 256), __ldg(p + 384));
  }
}
__device__ __forceinline__ void put64t(unsigned char* dst, const float4 (&x)[4]) {      // slices 2 S128 apart, lo S128 behind hi
  const int r = threadIdx.x & 127, t4 = threadIdx.x >> 7;
#pragma unroll
  for (int i = 0; i < 4; ++i) put4(dst + (i >> 1) * 2 * S128, S128, r, (t4 + 4 * i) & 7, x[i]);
}
// [64][64] tile as it is / transposed: two slices of 64 rows, 2 S64 apart
__device__ __forceinline__ void load_tt(float4 (&x)[2], const float* tile) {
#pragma unroll
  for (int i = 0; i < 2; ++i) x[i] = __ldg(reinterpret_cast<const float4*>(tile) + threadIdx.x + NT * i);
}
__device__ __forceinline__ void put_tt(unsigned char* dst, const float4 (&x)[2]) {
  const int c4 = threadIdx.x & 15;
#pragma unroll
  for (int i = 0; i < 2; ++i) put4(dst + (c4 >> 3) * 2 * S64, S64, static_cast<int>(threadIdx.x >> 4) + 32 * i, c4 & 7, x[i]);
}
__device__ __forceinline__ void load_ttt(float4 (&x)[2], const float* tile) {
  const int r = threadIdx.x & 63, t4 = threadIdx.x >> 6;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float* p = tile + (4 * (t4 + 8 * i)) * 64 + r;
    x[i] = make_float4(__ldg(p), __ldg(p + 64), __ldg(p + 128), __ldg(p + 192));
  }
}
__device__ __forceinline__ void put_ttt(unsigned char* dst, const float4 (&x)[2]) {
  const int r = threadIdx.x & 63, t4 = threadIdx.x >> 6;
#pragma unroll
  for (int i = 0; i < 2; ++i) put4(dst + i * 2 * S64, S64, r, t4, x[i]);
}

}  // namespace f32
#endif

}  // namespace kda
