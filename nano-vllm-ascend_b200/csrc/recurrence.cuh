// recurrence.cuh -- what the forms of linear_recurrence (seq_mixers.cu, recurrence_umma.cu) share.
#pragma once
#include "seq_common.cuh"

namespace b200 {

struct RecParams {
  const void *q, *k, *v;            // q, k: [tokens, groups * kdim] of type T; v: [tokens, H * vdim] of type TV
  int64_t q_stride, k_stride, v_stride;
  float* out;                       // [tokens, H * vdim] fp32
  float* state;                     // [slots, H, kdim, vdim] fp32 or nullptr (start from zero, keep nothing)
  const int *state_slots, *cu_q, *cu_k, *ctx_lens;
  int H, groups, kdim, vdim;
  int mode;                         // 0: constant decay per head; 1: selective (dt); 2: `k` holds a forget gate f per
                                    //    key channel (fp32): S <- diag(f) S + (1 - f) v^T
  int act_silu;                     // silu on q, k, v as they are read (mode 0)
  const float* decay;               // mode 0: [H]
  const void* dt;                   // mode 1: [tokens, H] element type T, before bias and softplus
  int64_t dt_stride;
  const float *dt_bias, *a_log, *d_skip;   // mode 1: [H] each
};

// silu for 16-bit activations: its result is rounded to 8 or 11 bits, the fast exponential is good to ~21
__device__ __forceinline__ float silu_fast(float x) { return __fdividef(x, 1.0f + __expf(-x)); }

// two fp32 -> three packed bf16 pairs hi, mid, lo (first value in the low half), each term the rounding of what the ones
// before it leave. The packed conversion runs at half of the fp32 rate, the scalar one on the special-function unit at
// an eighth (which is 3 % busy now).
__device__ __forceinline__ void split3x2(float x, float y, uint32_t (&w)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w[i]) : "f"(y), "f"(x));
    if (i < 2) x -= __uint_as_float(w[i] << 16), y -= __uint_as_float(w[i] & 0xffff0000u);
  }
}
// the same by cutting off: 24 bits in three terms of 8, exact. 9 instructions a pair (the subtractions packed, the packing a byte
// permutation) for 11, three of which run at half rate
__device__ __forceinline__ void split3cut(float x, float y, uint32_t (&w)[3]) {
  float2 r = make_float2(x, y);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    w[i] = __byte_perm(__float_as_uint(r.x), __float_as_uint(r.y), 0x7632);
    if (i < 2) {
      const float2 cut = make_float2(__uint_as_float(__float_as_uint(r.x) & 0xffff0000u), __uint_as_float(__float_as_uint(r.y) & 0xffff0000u));
      const float2 less = make_float2(-1.f, -1.f);
      asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(reinterpret_cast<uint64_t&>(r)) : "l"(reinterpret_cast<const uint64_t&>(cut)), "l"(reinterpret_cast<const uint64_t&>(less)));
    }
  }
}
__device__ __forceinline__ uint32_t bf16_bits(float x) { return __bfloat16_as_ushort(__float2bfloat16_rn(x)); }
__device__ __forceinline__ float bits_f32(uint32_t b16) { return __uint_as_float(b16 << 16); }

// The form on the 5th-generation tensor cores (recurrence_umma.cu), for chunks of 64 tokens. total_q: the step's tokens, 0 if the
// caller has not said
bool recurrence_umma_ok(const RecParams& P, int dtype, int num_seqs, int max_q, int64_t total_q);
int recurrence_umma_launch(const RecParams& P, int num_seqs, int64_t wait_ns, cudaStream_t stream);

}  // namespace b200
