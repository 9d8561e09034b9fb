// Parameters of the per-chunk preparation kernel (kda_chunk_prepare.cu).
#pragma once

#include "kda_chunk.cuh"
#include "kda_tma.cuh"

namespace kda {

struct PrepParams {
  const __nv_bfloat16 *q, *k, *v;
  const float *g, *beta;
  // gate front end (g_raw / beta_raw not NULL): g, beta are computed here, and written to g_out / beta_out unless those are NULL
  const void *g_raw, *beta_raw;
  const float *A_log, *dt_bias;
  float *g_out, *beta_out;
  int g_fp32, beta_fp32, use_lb;      // dtype of the raw tensors: float32 or bf16
  float lb;
  ChunkMap map;
  unsigned* status;
  bool clear_status;  // there is no tables kernel in front (equal lengths): prepare clears the status word
  unsigned char *W, *UT, *KG, *QG, *AQK, *GL, *TI, *RKK;   // TI, RKK may be NULL
  long long* dbg;
  int H;
  int kc, vc;         // key and value columns of the tensors (<= 128, multiples of 8; tiles are 128 wide, zero beyond)
  int use_l2norm;
  float scale;
  int HQ, grp;      // q/k heads and value heads per q/k head (grouped value heads); H counts value heads
  __nv_bfloat16 *QN, *KN;   // [tokens][HQ][128]: the normalised q, k kept for the backward (use_l2norm, training), or NULL
  float* RSTD;              // [2][tokens * HQ] reciprocal norms of q, k
  long long qrows;          // tokens * HQ
  int ahead;                // tiles between a CTA and the one that will take its place: its inputs are fetched into L2 now
  alignas(64) CUtensorMap tm_q, tm_k, tm_g;      // [tokens, heads, 128] in boxes of 64 tokens of one head, for that prefetch
  alignas(64) CUtensorMap tm_v;                  // 64-column boxes in the 128-byte swizzle
};

// `tiles` = chunks x heads (an upper bound is fine); returns KDA_OK, a negative KDA_E_* or a positive cudaError_t
int launch_prepare(PrepParams& p, long long tiles, long long tokens, bool keep_qn, bool safe_gate, cudaStream_t st);

}  // namespace kda
