// Attention of one query token per sequence over compressed keys and values, read from memory
// straight into registers: what the launcher hands over (kernel: decode_direct_kernel.cuh).
#pragma once

#include "fq_common.cuh"

namespace fq {

struct DirectArgs {
  const void* q;          // (seqs, hq, 128)
  const float* rotation;  // of the keys: q_rot = round(q Pi^T)
  const float* cent_k;
  int nck;
  const float* cent_v;
  int ncv;
  int seqs, hq, hkv;
  int n_splits;           // slices of a sequence's 16-token tiles = gridDim.x
  float scale_log2;
  float* part;            // [(slice * seqs * hq + row) * 132]: o (128) | m | l | - | -
  uint32_t* status;       // workspace head: status word, scale record behind it
  // (seqs, hkv, kv_stride, 64) codes and (seqs, hkv, kv_stride) norms, nkv tokens each
  const uint8_t* k_codes;
  const float* k_norms;
  const uint8_t* v_codes;
  const float* v_norms;
  int nkv;
  int64_t kv_stride;
};

// Streams the tiles and leaves partial rows; rotate_back_merged takes them from there.
int launch_decode_direct(const DirectArgs& a, int dtype, cudaStream_t stream);

}  // namespace fq
