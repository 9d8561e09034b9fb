// Parameters of the forward state-scan kernels.
#pragma once

#include "kda_chunk.cuh"
#include "kda_device.cuh"

namespace kda {

struct ScanParams {
  ChunkMap map;
  const unsigned char *W, *UT, *KG, *QG, *AQK, *GL;
  unsigned char *HS, *VNEWT;    // NULL unless saving for backward
  const float* h0;
  float* ht;
  __nv_bfloat16* o;
  unsigned* status;
  long long* dbg;       // development aid: phase clocks (NULL unless built with the clock marks and a buffer is registered)
  int H;
  int kc, vc;           // key and value columns of the tensors (<= 128; tiles and state are 128 wide, zero beyond)
};

// kda_chunk_scan.cu; `requested` CTAs per (sequence, head) unit (1 or 4), 0: chosen from the number of units and of SMs.  Returns KDA_OK, a
// negative KDA_E_* or a positive cudaError_t.
int launch_scan(const ScanParams& p, int units, int requested, cudaStream_t st);
int launch_scan_tc(const ScanParams& p, int blocks, cudaStream_t st);

// How many CTAs per unit the reverse scan uses: `requested` (1 or 4) if the caller chose, otherwise four while the
// grid stays within one CTA per SM of the current device.  (Two slices of 64 columns were built and measured: slower
// than one CTA per unit at every size, because the chain's cost is latency, not the width of its products.)
inline int scan_slices_for(int units, int requested) {
  if (requested == 1 || requested == 4) return requested;
  return units * 4 <= sm_count() ? 4 : 1;
}

}  // namespace kda
