// delta_rule.cuh -- what the forms of the gated delta rule (delta_rule.cu, delta_chunks.cu) share.
#pragma once
#include "seq_common.cuh"

namespace b200 {

enum { kDecayPerChannel = 0, kDecayPerHead = 1, kWkv = 2 };

struct DeltaParams {
  const float *q, *k;               // [tokens, groups * kdim]
  const float* g;                   // [tokens, H * kdim]; one decay per head: [tokens, H]
  const float* beta;                // [tokens, H]; wkv: the current token's coefficient
  const void* v;                    // [tokens, H * vdim], element type
  int64_t q_stride, k_stride, v_stride;
  float* out;                       // [tokens, H * vdim] fp32
  float* state;                     // [slots, H, kdim, vdim] fp32 or nullptr
  const int *state_slots, *cu_q, *cu_k, *ctx_lens;
  int H, groups, kdim, vdim;
};

// ---- chunks of 64 tokens (delta_chunks.cu). The chunks of a step are numbered through, sequence after sequence, and taken in passes of
// `count`; a (chunk, head) of the pass in hand has a record in the workspace.
constexpr int kDcL = 64;                               // tokens per chunk
struct DeltaChunks {
  uint8_t* records;                                    // [count][H] of `bytes` each, then the two below
  // Where the caller keeps no state, [H, kdim, vdim] fp32 of the sequence that came into this pass from the one before, and of the one that goes
  // on into the next. Two places, for these may be two sequences whose CTAs (and launches, where a head is left aside) run in any order;
  // one where a pass is a chunk, and so of one sequence
  const float* carry_in;
  float* carry_out;
  int64_t bytes;
  int first, count;                                    // the pass
  int flag_at;                                         // where a record says that its head's tokens are to be taken one at a time
};
__host__ __device__ __forceinline__ int chunks_of(int q_len) { return (q_len + kDcL - 1) / kDcL; }

// number of chunks before sequence s; all threads of a warp
__device__ __forceinline__ int chunks_before(const int* cu_q, int s) {
  int n = 0;
  for (int i = threadIdx.x & 31; i < s; i += 32) n += chunks_of(cu_q[i + 1] - cu_q[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  return n;
}
// the state between spans of a pass and the next: the sequence's slot, or what is carried from pass to pass
__device__ __forceinline__ const float* chunk_state_in(const DeltaParams& P, const DeltaChunks& C, int s, int h) {
  const int64_t size = (int64_t)P.kdim * P.vdim;
  return P.state != nullptr ? P.state + ((int64_t)P.state_slots[s] * P.H + h) * size : C.carry_in + (int64_t)h * size;
}
__device__ __forceinline__ float* chunk_state_out(const DeltaParams& P, const DeltaChunks& C, int s, int h) {
  const int64_t size = (int64_t)P.kdim * P.vdim;
  return P.state != nullptr ? P.state + ((int64_t)P.state_slots[s] * P.H + h) * size : C.carry_out + (int64_t)h * size;
}

// Bytes of workspace that the chunks would like for a step (0: such a step is not for them), and what they do with them: as many passes
// as it takes. true: the step is one for chunks, and `bytes` are enough for one chunk at least
int64_t delta_chunks_workspace(int mode, int dtype, int num_seqs, int max_q, int64_t total_q, int H, int groups, int kdim, int vdim);
bool delta_chunks_ok(const DeltaParams& P, int mode, int dtype, int num_seqs, int max_q, int64_t total_q, const void* workspace, int64_t bytes);
int delta_chunks_launch(const DeltaParams& P, int mode, int num_seqs, int64_t total_q, void* workspace, int64_t bytes, int64_t wait_ns,
                        cudaStream_t stream);
// delta_rule.cu: the tokens of the heads that the pass leaves aside, one at a time
int delta_rest_launch(const DeltaParams& P, const DeltaChunks& C, int mode, int num_seqs, bool only_pass, cudaStream_t stream);

}  // namespace b200
