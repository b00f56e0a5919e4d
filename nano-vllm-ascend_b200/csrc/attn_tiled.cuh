// attn_tiled.cuh -- the 64-row form of attn_generic (attn_tiled.cu), chosen by b200_attn_generic for prompt portions.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

struct AttnTiledParams {
  void* out;                        // [tokens, H * vdim]
  const void *q, *k, *v;            // v == nullptr: the values are the first vdim columns of the key rows
  int64_t q_stride, k_stride, v_stride;
  const int* block_tables;          // nullptr: packed keys
  int bt_stride, block_size;
  const int *cu_q, *cu_k;
  int H, G, dim, vdim;
  int chunks, num_seqs;             // set by the launcher: 16-byte chunks of fp32 per staged row, spans
  float scale;
  int window, keep_first, chunk;
  float softcap;
  const float* sink;
  const void* gate;
  int64_t gate_stride;
};

// The form on the tensor cores (attn_split.cu). total_q: the step's tokens, 0 if the caller has not said
bool attn_split_fits(const AttnTiledParams& P, int num_seqs, int max_q, int64_t total_q, int dtype);
int attn_split_launch(AttnTiledParams P, int num_seqs, int max_q, int64_t total_q, int64_t wait_ns, cudaStream_t stream);
bool attn_tiled_fits(int max_q, int rep, int G, int num_seqs, int dim, int vdim);
int attn_tiled_launch(AttnTiledParams P, int num_seqs, int max_q, int dtype, cudaStream_t stream);

}  // namespace b200
