// delta_chunks.cu -- the gated delta rule over prompts on the 5th-generation tensor cores, 64 tokens at a time.
//
// With P_i the decay from a chunk's start to and with token i (a vector per key channel, or a number), S0 the state before the chunk and
// w_i what token i writes,
//   w_i = beta_i (v_i - (P_i k_i) S0 - sum_(j<i) A_ij w_j)       A_ij = sum_d k_id (P_i / P_j)_d k_jd
//   o_i = (P_i q_i) S0 + sum_(j<=i) B_ij w_j                     B_ij = sum_d q_id (P_i / P_j)_d k_jd
//   S   = P_end S0 + sum_j (P_end / P_j) k_j w_j^T
// so that with X = [I; B] (I + diag(beta) A)^-1 diag(beta), 128 x 64,
//   [U; O0] = X V        [W; Y] = X (P k)        w = U - W S0        o = O0 + (P q - Y) S0.
// All of X, U, O0, W and P q - Y is independent of S0: delta_chunk_kernel computes it for all chunks at once, and delta_scan_kernel walks
// the chunks of a head with two products each.
//
// delta_chunk_kernel, one CTA of 8 warps per (chunk, head), two CTAs per SM:
//   scores [K~; Q~] K^^T   M128 N64 K = D, 32 channels to an accumulator (the tensor core cuts sums off: the small products of later
//                          channels on top of a full sum would cost 6e-7). Decays per channel are split at the chunk's middle,
//                          K~ = k P_i / P_mid, K^ = k P_mid / P_j, each a product of decays or its reciprocal. One decay per head:
//                          K~ = K^ = k, and the decay goes on the scores.
//   X                      a thread per row: back substitution over columns, 64 x 64 / 2 packed multiply-adds, rows of A as broadcasts
//   [W; Y], [U; O0]        M128 N = D K64, X from tensor memory
// delta_scan_kernel, one CTA per (sequence, 128 value channels = one head of 128 or two of 64), S^T in fp32 registers:
//   E^T = S0^T [W; P q - Y]^T    M128 (channels) N128 K = D, S0 in three terms from tensor memory, in two halves of its rows
//   w -> three terms; o out;  dS^T = w^T (P_end / P_j k_j)    M128 N = D K64;   S = P_end S + dS in registers.
// Every fp32 operand is three bf16 terms (24 bits, exact), six products, small ones first; values are bf16 as they are. One operand of every
// product is split by rounding: where both are by cutting off, the three products left out have one sign and lack 6e-8 on average.
// Outputs are 0.45 to 0.98 times as far from 64 bits as the token form's, states 0.34 to 1.15 times, where the last token is nearly all of a
// state 1.3 to 1.5 (test_no_precision_is_lost: operands of random signs; where all have one sign, outputs 0.72 to 1.4).
//
// What bounds them, 16 prompts of 500-1250 tokens, 8 heads of 128 (delta_rule_kernel 700 us): delta_chunk_kernel 213, a CTA's phases behind
// one another (loads, scores, substitution, products, 48000 cycles, of which 11000 are issue, and code that has to be fetched); delta_scan_kernel
// 104, the chain E -> w -> dS -> S -> E of 8500 cycles a chunk, 6000 of them for 72 MMAs. The records that pass between them (216 KB per chunk and head
// of 128, written and read once) would take 2 x 63 at HBM's rate.
//
// Decays per channel that come to less than 2^-83 over half a chunk (0.17 a token) would take the reciprocals, or low terms, out of the range: a CTA
// that meets them computes its scores in blocks of 16 tokens (dc_block_scores), for which no decay is too small.
//
// Not for chunks, and left to delta_rule_kernel, which runs behind them over the heads that a record flags: values that are not finite
// (0 x inf would reach tokens before them) or beyond 2^60, decays of 2 and more, keys, queries or values all below 2^-60 (the low terms
// would be lost), and, where scores go by reciprocals, keys or queries from 2^30 on or all below 2^-20.
//
// Waits are bounded (mbar_warp_wait): one that runs out makes its role leave, those that wait for it run out as well, the products under
// way are waited for, the CTA sets the host's word and the library reports it.
#include <limits.h>

#include <algorithm>
#include <type_traits>

#include "delta_rule.cuh"
#include "recurrence.cuh"
#include "umma.cuh"

namespace b200 {

// ---- a record: bytes of its parts
template <int D>
struct DcRecord {
  static constexpr int kWq = 3 * 2 * D * 128;            // [W; P q - Y]: [3 terms][2 panels of 64 rows r][D rows n][128 bytes]
  static constexpr int kKe = 3 * (D / 64) * 8192;        // P_end / P_j k_j: [3 terms][D / 64 panels][64 rows j][128 bytes]
  static constexpr int kUoRow = 132;                     // floats of a row of [U; O0]: 16-byte groups of eight rows in different banks
  static constexpr int kUo = D * kUoRow * 4;             // [U; O0]: [D rows c][128 r] fp32
  static constexpr int kPe = 1024;                       // P_end [D] fp32, the flag
  static constexpr int kKeAt = kWq, kUoAt = kWq + kKe, kPeAt = kUoAt + kUo, kFlagAt = kPeAt + D * 4, kBytes = kPeAt + kPe;
};
// terms of A and B in the i-th of six products, small ones first: 0 2, 1 1, 2 0, 0 1, 1 0, 0 0
__device__ __forceinline__ uint32_t term_a(int i) { return i == 2 ? 2 : (i == 1 || i == 4); }
__device__ __forceinline__ uint32_t term_b(int i) { return i == 0 ? 2 : (i == 1 || i == 3); }

struct DcParams {
  DeltaParams d;
  DeltaChunks c;
  int num_seqs, wait_tries;
  int* wait_status;
};

__device__ __forceinline__ void mma_ts_half_low(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_low, uint32_t idesc, uint32_t accumulate, int half) {
  const uint32_t off0 = half == 0 ? 0u : 0xffffffffu, off1 = ~off0;        // lanes whose bit is set are left alone
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 b;\n\t"
      "mov.b64 b, {%2, %7};\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %3, {%5, %5, %6, %6}, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "r"(b_low), "r"(idesc), "r"(accumulate), "r"(off0), "r"(off1), "n"(umma::kDescHigh)
      : "memory");
}
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(smem_dst)), "l"(src),
               "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// The tensor core cuts a sum off where fp32 arithmetic rounds it: half a unit of the last place is lost on average, ln 2 / 2 x 2^-23 of a number. It is
// given back where the sum meets another number or is split in terms (alone, 24 bits could not hold it).
constexpr float kCut = 4.13e-8f;
__device__ __forceinline__ uint32_t magnitude(float x) { return __float_as_uint(x) & 0x7fffffffu; }
__device__ __forceinline__ float largest(float most, float2 x) {             // of |x|; NaN stays
  asm("max.NaN.f32 %0, %0, %1, %2;" : "+f"(most) : "f"(fabsf(x.x)), "f"(fabsf(x.y)));
  return most;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<uint64_t&>(r)) : "l"(reinterpret_cast<const uint64_t&>(a)), "l"(reinterpret_cast<const uint64_t&>(b)));
  return r;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<uint64_t&>(r)) : "l"(reinterpret_cast<const uint64_t&>(a)), "l"(reinterpret_cast<const uint64_t&>(b)));
  return r;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(reinterpret_cast<uint64_t&>(c)) : "l"(reinterpret_cast<const uint64_t&>(a)), "l"(reinterpret_cast<const uint64_t&>(b)));
  return c;
}
__device__ __forceinline__ float2 both(uint32_t x, uint32_t y) { return make_float2(__uint_as_float(x), __uint_as_float(y)); }
// split3x2 (each term the rounding of what those before leave) of x (1 + part)
__device__ __forceinline__ void split3more(float2 x, float2 part, uint32_t (&w)[3]) {
  float2 r = x;
  const float2 less = make_float2(-1.f, -1.f);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    if (i == 2) r = fma2(x, part, r);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w[i]) : "f"(r.y), "f"(r.x));
    if (i < 2) r = fma2(both(w[i] << 16, w[i] & 0xffff0000u), less, r);
  }
}
// 1 / x to within a unit: an approximation, and Newton's step from it
__device__ __forceinline__ float rcp_newton(float x) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return fmaf(fmaf(-x, r, 1.f), r, r);
}
constexpr uint32_t kBig = (127u + 60u) << 23, kSmall = (127u - 60u) << 23, kTwo = 128u << 23;
constexpr float kNear = 0x1p-83f;                        // between eight tokens and the middle: with each of those, 2^-90 and more
constexpr uint32_t kBigUp = (127u + 30u) << 23, kSmallDn = (127u - 20u) << 23;       // of what meets 2^90 and, in its third term, 2^-90: within 2^+-126

constexpr int kDcThreads = 256;
constexpr int kDcARow = 68;                              // floats of a row of A: 16-byte groups of eight rows in different banks
template <int D>
struct DcSmem {
  static constexpr int kScores = 3 * 16384 + 3 * 8192;   // [K~; Q~] [3 terms][128 rows], K^ [3 terms][64 rows], 64 channels at a time
  static constexpr int kKb = 3 * (D / 64) * 8192;        // behind it: P k [3 terms][D / 64 panels][64 rows j]
  static constexpr int kA = kDcL * kDcARow * 4;          // A (then V)
  static constexpr int kQRow = D + 4;
  static constexpr int kQs = kDcL * kQRow * 4;           // P q
  static constexpr int kAAt = kKb, kQsAt = kKb + kA;
  // strong decays: scores inside blocks of 16 tokens, [4 parts][16 i][4 groups of j][k, q][4 blocks][4 j], and, where A will be, their sum in rows of kBlockRow and
  // [k, q][tokens 16-31, 48-63] those of the block before
  static constexpr int kParts = 4 * 2 * kDcL * 16 * 4, kPartsAt = kScores, kBlockRow = 20, kBlocks = 2 * kDcL * kBlockRow * 4, kNear = kBlocks / 2;
  static constexpr int kEnd = kQsAt + kQs > kPartsAt + kParts ? kQsAt + kQs : kPartsAt + kParts;
  static_assert(kBlocks + kNear <= kA, "room for the blocks");
  static constexpr int kTau = (D / 64) * 8 * 64 * 4;     // decays of 8 tokens
  static constexpr int kBytes = 1024 + kEnd + kTau + 4 * 64 * 4 + 256;
};

// a CTA's shared memory
template <int D>
struct DcLocal {
  using M = DcSmem<D>;
  uint8_t* at;
  __device__ __forceinline__ DcLocal() {
    extern __shared__ __align__(1024) uint8_t dc_smem_raw[];
    at = dc_smem_raw + (-smem_u32(dc_smem_raw) & 1023u);               // (not through an integer: the compiler has to know that it is shared memory)
  }
  __device__ __forceinline__ float* A() const { return reinterpret_cast<float*>(at + M::kAAt); }
  __device__ __forceinline__ float* Qs() const { return reinterpret_cast<float*>(at + M::kQsAt); }
  __device__ __forceinline__ float* parts() const { return reinterpret_cast<float*>(at + M::kPartsAt); }
  __device__ __forceinline__ float* tau() const { return reinterpret_cast<float*>(at + M::kEnd); }             // [D / 64][8][64]
  __device__ __forceinline__ float* beta() const { return tau() + (D / 64) * 8 * 64; }
  __device__ __forceinline__ float* g() const { return beta() + 64; }  // one decay per head: of a token, P, P_end / P
  __device__ __forceinline__ float* p() const { return beta() + 128; }
  __device__ __forceinline__ float* e() const { return beta() + 192; }
  __device__ __forceinline__ uint64_t* scored() const { return reinterpret_cast<uint64_t*>(beta() + 256); }
  __device__ __forceinline__ uint64_t* made() const { return scored() + 1; }
  __device__ __forceinline__ uint64_t* drained() const { return scored() + 2; }
  __device__ __forceinline__ uint32_t* max() const { return reinterpret_cast<uint32_t*>(scored() + 3); }       // largest magnitudes: k, q, v, and what must stay below two
  __device__ __forceinline__ uint32_t* tmem_slot() const { return max() + 4; }
  __device__ __forceinline__ int* where() const { return reinterpret_cast<int*>(max() + 5); }                  // two
  __device__ __forceinline__ int* next() const { return where() + 2; }
  __device__ __forceinline__ volatile int* gave_up() const { return where() + 3; }
};
constexpr uint32_t kTmSC = 0, kTmX = 128;                // scores of 64 channels each, then [W; Y] and [U; O0], 128 columns; X 3 x 32

// ---- scores
struct DcTokens {                                        // a chunk's rows of a head: found by 32-bit offsets from the first
  const float *k, *q, *g;
  uint32_t k_step, q_step, g_step;
  int nt;
};
struct DcChunk {                                         // and what a CTA knows once its scores are on their way
  DcTokens t;
  const __nv_bfloat16* v;
  int64_t v_stride;
  uint8_t* record;
  uint32_t tb;                                           // its columns
  int issued, wait_tries;                                // commits to `scored`
  bool alive;
  int* wait_status;
  __device__ __forceinline__ bool wait(uint64_t* bar, int parity, volatile int* gave_up) const { return mbar_warp_wait(bar, parity & 1, wait_tries, gave_up); }
};
// 8 tokens of two channels. (Full chunks without the questions, in code of their own, were slower: 316 us for 314, strong decays 415 for 401)
template <bool PER_HEAD>
__device__ __forceinline__ void dc_fetch(const DcTokens& C, int t0, int ch, float2 (&kk)[8], float2 (&qq)[8], float2 (&gg)[8]) {
  uint32_t ka = t0 * C.k_step + ch * 4, qa = t0 * C.q_step + ch * 4, ga = t0 * C.g_step + ch * 4;
#pragma unroll
  for (int x = 0; x < 8; ++x) {
    const bool ok = t0 + x < C.nt;
    kk[x] = ok ? *reinterpret_cast<const float2*>(reinterpret_cast<const uint8_t*>(C.k) + ka) : make_float2(0.f, 0.f);
    qq[x] = ok ? *reinterpret_cast<const float2*>(reinterpret_cast<const uint8_t*>(C.q) + qa) : make_float2(0.f, 0.f);
    if (!PER_HEAD) gg[x] = ok ? *reinterpret_cast<const float2*>(reinterpret_cast<const uint8_t*>(C.g) + ga) : make_float2(1.f, 1.f);
    ka += C.k_step, qa += C.q_step, ga += C.g_step;
  }
}
// two channels of a token into row x of a group of eight rows of the operands: of K~ and Q~, of K^
__device__ __forceinline__ void dc_put_up(uint8_t* group, int lane, int x, float2 kk, float2 qq, float2 up) {
  uint32_t a[3], b[3];
  const float2 kx = mul2(kk, up), qx = mul2(qq, up);
  split3cut(kx.x, kx.y, a);
  split3cut(qx.x, qx.y, b);
  const uint32_t at = x * 128 + (((lane >> 2) ^ x) << 4);
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    *reinterpret_cast<uint32_t*>(group + p * 16384 + at) = a[p];
    *reinterpret_cast<uint32_t*>(group + p * 16384 + 8192 + at) = b[p];
  }
}
__device__ __forceinline__ void dc_put_dn(uint8_t* group, int lane, int x, float2 kk, float2 dn) {
  uint32_t c[3];
  const float2 kx = mul2(kk, dn);
  split3x2(kx.x, kx.y, c);
  const uint32_t at = x * 128 + (((lane >> 2) ^ x) << 4);
#pragma unroll
  for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t*>(group + 49152 + p * 8192 + at) = c[p];
}
template <int D>
__device__ __forceinline__ void dc_issue_scores(uint8_t* smem, uint32_t to, uint64_t* scored) {
  const uint32_t id = umma::make_idesc<__nv_bfloat16>(128, 64, 0, 0);
  const uint32_t a0 = umma::desc_low(smem_u32(smem), 16), b0 = umma::desc_low(smem_u32(smem + 49152), 16);
#pragma unroll
  for (int i = 0; i < 6; ++i)
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
      umma::mma_ss_low(to + (ks >> 1) * 64, a0 + ((term_a(i) * 16384 + ks * 32) >> 4), b0 + ((term_b(i) * 8192 + ks * 32) >> 4), id, i > 0 || (ks & 1) > 0);
  umma::commit(scored);
}

// Scores of decays per channel of any size (delta_chunk_kernel's own go by a reciprocal, which has to stay within 2^90). Between tokens of one
// block of 16 in fp32; between blocks on the tensor core, split at token 32 and inside either half at its middle: products of decays alone.
// Accumulators as delta_chunk_kernel's, of which columns 0-31 are what rows of tokens 32 to 63 have of tokens 0 to 31, and columns 32-63 of tokens
// 0 to 15 and 32 to 47, for tokens 16 to 31 in their rows, 48 to 63 in rows 0 to 15. What bounds a CTA here: phases behind one another, of 8 warps
// (an instruction every 3.2 cycles; code that does not fit the instruction cache is the first of its stalls: with the four channels of a lane behind one
// another instead of in a loop, the first figure is 461). us, token form / so / decays that need it not: 16 prompts of 500-1250, 8 heads of 128 700 / 401 /
// 314, 1 x 1024 360 / 108 / 99, 4 x 256 93 / 59 / 49; 32 heads of 64 1 x 1024 299 / 144 / 121
template <int D>
__device__ __forceinline__ void dc_block_scores(DcChunk& W) {
  const DcLocal<D> L;
  uint8_t* const smem = L.at;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float2 one = make_float2(1.f, 1.f);
  float most_k = 0.f, most_q = 0.f, most_g = 0.f;
  uint8_t* to = smem + (lane & 3) * 4;
  float2* raw_kq = reinterpret_cast<float2*>(smem);      // k, q and g as they are, 64 channels at a time: [64][64] pairs of k and q, [64][64] of g
  float* raw_g = reinterpret_cast<float*>(smem + (kDcL * 64 + 16) * 8);        // (rows of a block of 16 are 4 elements on: blocks in other banks)
#pragma unroll 1
  for (int half = 0; half < D / 64; ++half) {
    float2* tau = reinterpret_cast<float2*>(L.tau() + half * 512) + lane;
    if (W.issued > 0) {                                  // the products under way have read their operands
      W.alive = W.alive && W.wait(L.scored(), W.issued - 1, L.gave_up());
      umma::fence_after_sync();
    }
    {
      float2 kk[8], qq[8], gg[8], all = one;
      dc_fetch<false>(W.t, 8 * warp, half * 64 + 2 * lane, kk, qq, gg);
      __syncthreads();
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        most_k = largest(most_k, kk[x]), most_q = largest(most_q, qq[x]), most_g = largest(most_g, gg[x]);
        all = mul2(all, gg[x]);
        const int at = (8 * warp + x) * 64 + 2 * lane + (warp >> 1) * 4;
        *reinterpret_cast<float4*>(raw_kq + at) = make_float4(kk[x].x, qq[x].x, kk[x].y, qq[x].y);
        *reinterpret_cast<float2*>(raw_g + at) = gg[x];
      }
      tau[warp * 32] = all;
    }
    __syncthreads();
    // ---- blocks of 16 tokens: a warp has a quarter of the channels, a lane two tokens j of a block (in turn of two groups of four, 0 and 3 or 1 and 2) and
    // a quarter of those, and walks the tokens i behind them
    auto walk = [&](auto group) {
      constexpr int J = 4 * decltype(group)::value, N = 16 - J;
      const int slice = lane & 3, own = (lane >> 2) & 1, block = lane >> 3;
      int at = (16 * block + J) * 64 + block * 4 + (warp >> 1) * 16 + slice;
      float a[2][N], b[2][N], p[2];
#pragma unroll
      for (int i = 0; i < N; ++i) a[0][i] = a[1][i] = b[0][i] = b[1][i] = 0.f;
#pragma unroll 1
      for (int e = 0; e < 4; ++e, at += 4) {             // (a loop, not unrolled: less code to fetch)
#pragma unroll
        for (int x = 0; x < 2; ++x) p[x] = raw_kq[at + (2 * own + x) * 64].x;
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const float2 y = raw_kq[at + i * 64];
          const float g = raw_g[at + i * 64];
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            if (i >= 4 || i > 2 * own + x) p[x] *= g;
            a[x][i] = fmaf(y.x, p[x], a[x][i]);
            b[x][i] = fmaf(y.y, p[x], b[x][i]);
          }
        }
      }
      // the four slices: a lane keeps k or q of one of the two tokens j
      float* part = L.parts() + (((warp >> 1) * 16 + J) * 4 + J / 4) * 32 + (lane & 1) * 16 + block * 4 + 2 * own + ((lane >> 1) & 1);
#pragma unroll
      for (int i = 0; i < N; ++i) {
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const float keep = lane & 1 ? b[x][i] : a[x][i], give = lane & 1 ? a[x][i] : b[x][i];
          a[x][i] = keep + __shfl_xor_sync(0xffffffffu, give, 1);
        }
        const float keep = lane & 2 ? a[1][i] : a[0][i], give = lane & 2 ? a[0][i] : a[1][i];
        const float sum = keep + __shfl_xor_sync(0xffffffffu, give, 2);
        part[i * 128] = half > 0 ? part[i * 128] + sum : sum;
      }
    };
    if (warp & 1) walk(std::integral_constant<int, 1>{}), walk(std::integral_constant<int, 2>{});
    else walk(std::integral_constant<int, 0>{}), walk(std::integral_constant<int, 3>{});
    // ---- across blocks: relative to token 32 (rows i of 32 and later, columns j before it) and inside either half to its middle (rows 0-15: tokens 48 to 63,
    // rows 16-31: those; columns 32-63: tokens 0 to 15 and 32 to 47): products of decays alone
    float2 kk[8], qq[8], gg[8], f = one, near = one;
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      const int at = (8 * warp + x) * 64 + 2 * lane + (warp >> 1) * 4;
      const float4 y = *reinterpret_cast<const float4*>(raw_kq + at);
      kk[x] = make_float2(y.x, y.z), qq[x] = make_float2(y.y, y.w), gg[x] = *reinterpret_cast<const float2*>(raw_g + at);
    }
    if (warp < 4) {
      for (int w = warp + 1; w < 4; ++w) f = mul2(f, tau[w * 32]);
    } else {
      for (int w = 4; w < warp; ++w) f = mul2(f, tau[w * 32]);
    }
    const bool upper = (warp & 2) != 0;                  // half of its half
    if (upper && (warp & 1)) near = tau[(warp - 1) * 32];
    if (!upper && !(warp & 1)) near = tau[(warp + 1) * 32];
    __syncthreads();                                     // k, q and g have been read
    if (warp < 4) {
#pragma unroll
      for (int x = 7; x >= 0; --x) dc_put_dn(to + warp * 1024, lane, x, kk[x], f), f = mul2(f, gg[x]);
    } else {
#pragma unroll
      for (int x = 0; x < 8; ++x) f = mul2(f, gg[x]), dc_put_up(to + warp * 1024, lane, x, kk[x], qq[x], f);
    }
    if (upper) {
#pragma unroll
      for (int x = 0; x < 8; ++x) near = mul2(near, gg[x]), dc_put_up(to + (warp < 4 ? warp : warp - 6) * 1024, lane, x, kk[x], qq[x], near);
    } else {
#pragma unroll
      for (int x = 7; x >= 0; --x) dc_put_dn(to + (warp < 4 ? warp + 4 : warp + 2) * 1024, lane, x, kk[x], near), near = mul2(near, gg[x]);
    }
    fence_proxy_async_smem();
    __syncthreads();
    if (warp == 0 && W.alive && umma::elect_one()) dc_issue_scores<D>(smem, W.tb + kTmSC + half * 128, L.scored());
    __syncwarp();
    ++W.issued;
  }
  const uint32_t mk = __reduce_max_sync(0xffffffffu, magnitude(most_k)), mq = __reduce_max_sync(0xffffffffu, magnitude(most_q)),
                 mg = __reduce_max_sync(0xffffffffu, magnitude(most_g));
  if (lane == 0) atomicMax(&L.max()[0], mk), atomicMax(&L.max()[1], mq), atomicMax(&L.max()[3], mg);
}

// ---- behind the scores: X, [W; Y], [U; O0], the record. BLOCKS: from dc_block_scores
template <int D, bool PER_HEAD, bool BLOCKS>
__device__ __forceinline__ void dc_chunk_rest(const DcChunk& W) {
  using T = __nv_bfloat16;
  using R = DcRecord<D>;
  using M = DcSmem<D>;
  const DcLocal<D> L;
  uint8_t* const smem = L.at;
  float *const sA = L.A(), *const sQs = L.Qs(), *const s_tau = L.tau(), *const s_beta = L.beta(), *const s_g = L.g(), *const s_p = L.p(), *const s_e = L.e();
  uint64_t *const scored = L.scored(), *const made = L.made(), *const drained = L.drained();
  uint32_t* const s_max = L.max();
  int* const s_next = L.next();
  volatile int* const gave_up = L.gave_up();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nt = W.t.nt;
  const uint32_t tb = W.tb;
  const T* const v = W.v;
  uint8_t* const record = W.record;
  const bool issuer = warp == 0 && umma::elect_one();
  const float2 one = make_float2(1.f, 1.f);
  bool alive = W.alive;
  auto wait = [&](uint64_t* bar, int parity) { return W.wait(bar, parity, gave_up); };
  alive = alive && wait(scored, W.issued - 1);
  umma::fence_after_sync();
  __syncthreads();                                       // all that the scores were made of is free
  if (BLOCKS) {                                          // the blocks' four parts, to where A will be (P q will be where they are)
    static_assert(2 * kDcL * 16 == 8 * kDcThreads, "eight sums a thread");
    const int of = threadIdx.x >> 1;                     // [k, q][block][i]
    const float4* part = reinterpret_cast<const float4*>(L.parts()) + (of & 15) * 32 + (threadIdx.x & 1) * 16 + (of >> 6) * 4 + ((of >> 4) & 3);
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      float4 sum = part[y * 8];
#pragma unroll
      for (int z = 1; z < 4; ++z) {
        const float4 more = part[z * 512 + y * 8];
        sum.x += more.x, sum.y += more.y, sum.z += more.z, sum.w += more.w;
      }
      *reinterpret_cast<float4*>(sA + (threadIdx.x >> 1) * M::kBlockRow + (threadIdx.x & 1) * 8 + 4 * y) = sum;
    }
    __syncthreads();
  }

  uint4 held[D / 16];                                    // values on their way to where A is
  float2 X[32];                                          // warps 0-3: a row of X
  if (warp < 4) {
    const int i = threadIdx.x & 63;                      // token; rows 0-63: of T = (I + beta A)^-1, 64-127: of B T
    const bool of_k = warp < 2;
    const uint32_t base = tb + ((uint32_t)(warp * 32) << 16);
#pragma unroll
    for (int part = 0; part < 2; ++part) {
      uint32_t w[32];
#pragma unroll
      for (int c0 = 0; c0 < 32; c0 += 16) {
        uint32_t y[D / 32][16];
#pragma unroll
        for (int z = 0; z < D / 32; ++z) umma::ld16(base + kTmSC + 64 * z + 32 * part + c0, y[z]);
        umma::wait_ld();
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          float a = __uint_as_float(y[0][c]), b = __uint_as_float(y[1][c]);
          if (D == 128) a += b, b = __uint_as_float(y[D / 32 - 2][c]) + __uint_as_float(y[D / 32 - 1][c]);
          w[c0 + c] = __float_as_uint(a + fmaf(a + b, kCut, b));
        }
      }
#pragma unroll
      for (int c = 0; c < 16; ++c) X[16 * part + c] = make_float2(__uint_as_float(w[2 * c]), __uint_as_float(w[2 * c + 1]));
    }
    if (BLOCKS) {
      // (see dc_block_scores) the columns of a row's own half: of its block, and of the block before, which rows 48 to 63 have had in rows 0 to 15
      float* s_near = sA + M::kBlocks / 4 + (of_k ? 0 : 32 * M::kBlockRow);        // [k, q][tokens 16-31, 48-63][kBlockRow]
      if (!(warp & 1)) {
#pragma unroll
        for (int c = 0; c < 8; ++c) *reinterpret_cast<float2*>(s_near + (lane ^ 16) * M::kBlockRow + 2 * c) = lane < 16 ? X[24 + c] : X[16 + c];
      }
      named_bar_sync(1, 128);
      const float* own = sA + ((of_k ? 0 : kDcL) + i) * M::kBlockRow;
      const float* other = lane < 16 ? own : s_near + (warp & 1 ? lane : lane - 16) * M::kBlockRow;
      if (warp & 1) {
#pragma unroll
        for (int c = 0; c < 8; ++c) X[16 + c] = *reinterpret_cast<const float2*>(other + 2 * c), X[24 + c] = *reinterpret_cast<const float2*>(own + 2 * c);
      } else {
#pragma unroll
        for (int c = 0; c < 8; ++c) X[c] = *reinterpret_cast<const float2*>(other + 2 * c), X[8 + c] = *reinterpret_cast<const float2*>(own + 2 * c);
      }
      named_bar_sync(1, 128);                            // A takes their place
    }
    if (PER_HEAD) {                                      // the decay from j to i
      float d = 1.f;
#pragma unroll
      for (int j = 63; j >= 0; --j) {
        if (j < i) d *= s_g[j + 1];
        (j & 1 ? X[j / 2].y : X[j / 2].x) *= d;
      }
    }
    const float beta = of_k ? s_beta[i] : 1.f;
#pragma unroll
    for (int c = 0; c < 32; ++c) {
      X[c].x = 2 * c < i + (of_k ? 0 : 1) ? X[c].x * beta : 0.f;
      X[c].y = 2 * c + 1 < i + (of_k ? 0 : 1) ? X[c].y * beta : 0.f;
    }
    if (of_k) {
#pragma unroll
      for (int c = 0; c < 16; ++c)
        *reinterpret_cast<float4*>(sA + i * kDcARow + 4 * c) = make_float4(X[2 * c].x, X[2 * c].y, X[2 * c + 1].x, X[2 * c + 1].y);
#pragma unroll
      for (int c = 0; c < 32; ++c) X[c] = make_float2(2 * c == i ? 1.f : 0.f, 2 * c + 1 == i ? 1.f : 0.f);
    }
    named_bar_sync(1, 128);
    // X (I + beta A) = [I; B]: column l is final once those behind it are, and leaves the columns before it
    auto column = [&](int l) {
      const float xl = -(l & 1 ? X[l / 2].y : X[l / 2].x);
      const float2 x2 = make_float2(xl, xl);
      const float* row = sA + l * kDcARow;
#pragma unroll
      for (int c = 0; c < (l + 3) / 4; ++c) {
        const float4 a = *reinterpret_cast<const float4*>(row + 4 * c);
        const float2 a0 = make_float2(a.x, a.y), a1 = make_float2(a.z, a.w);
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(reinterpret_cast<uint64_t&>(X[2 * c])) : "l"(reinterpret_cast<const uint64_t&>(x2)), "l"(reinterpret_cast<const uint64_t&>(a0)));
        if (4 * c + 2 < l) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(reinterpret_cast<uint64_t&>(X[2 * c + 1])) : "l"(reinterpret_cast<const uint64_t&>(x2)), "l"(reinterpret_cast<const uint64_t&>(a1)));
      }
    };
    if (warp & 1) {                                      // tokens 32 and later
#pragma unroll
      for (int l = 63; l >= 32; --l) column(l);
    }
#pragma unroll
    for (int l = 31; l >= 1; --l) column(l);
    // times beta, as the A operand: packed pairs along j
#pragma unroll
    for (int part = 0; part < 4; ++part) {
      uint32_t w[3][8];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float2 b = *reinterpret_cast<const float2*>(s_beta + 16 * part + 2 * c);
        uint32_t y[3];
        split3cut(X[8 * part + c].x * b.x, X[8 * part + c].y * b.y, y);
        w[0][c] = y[0], w[1][c] = y[1], w[2][c] = y[2];
      }
#pragma unroll
      for (int p = 0; p < 3; ++p) umma::st8(base + kTmX + p * 32 + 8 * part, w[p]);
    }
    umma::wait_st();
  } else {
#pragma unroll
    for (int i = 0; i < D / 16; ++i) {
      const int e = i * 128 + threadIdx.x - 128, row = e / (D / 8), c16 = e % (D / 8);
      held[i] = row < nt ? ld_nc_v4(v + row * W.v_stride + c16 * 8) : make_uint4(0, 0, 0, 0);
    }
    uint32_t most_v = 0;
#pragma unroll
    for (int i = 0; i < D / 16; ++i) {
      most_v = __vimax3_u16x2(most_v, held[i].x & 0x7fff7fffu, held[i].y & 0x7fff7fffu);
      most_v = __vimax3_u16x2(most_v, held[i].z & 0x7fff7fffu, held[i].w & 0x7fff7fffu);
    }
    most_v = max(most_v & 0xffffu, most_v >> 16) << 16;
    most_v = __reduce_max_sync(0xffffffffu, most_v);
    if (lane == 0) atomicMax(&s_max[2], most_v);
  }
  // ------------------------------------------------ P k for [W; Y], P q, P_end / P k for the scan: 8 tokens of 64 channels to a warp that is free
  uint8_t* kb = smem + (lane & 3) * 4;
  while (true) {
    int u = lane == 0 ? atomicAdd(s_next, 1) : 0;
    u = __shfl_sync(0xffffffffu, u, 0);
    if (u >= 8 * (D / 64)) break;
    const int half = u >> 3, e = u & 7, ch = half * 64 + 2 * lane;
    float2 kk[8], qq[8], gg[8], to_end[8], p = one, post = one;
    dc_fetch<PER_HEAD>(W.t, 8 * e, ch, kk, qq, gg);
    if (!PER_HEAD) {
      const float2* tau = reinterpret_cast<const float2*>(s_tau + half * 512) + lane;
      for (int w = 0; w < e; ++w) p = mul2(p, tau[w * 32]);
      for (int w = 7; w > e; --w) post = mul2(post, tau[w * 32]);
#pragma unroll
      for (int x = 7; x >= 0; --x) to_end[x] = post, post = mul2(post, gg[x]);
      if (e == 0) *reinterpret_cast<float2*>(record + R::kPeAt + ch * 4) = post;
    } else if (e == 0) {
      *reinterpret_cast<float2*>(record + R::kPeAt + ch * 4) = make_float2(s_p[63], s_p[63]);
    }
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      const int t = 8 * e + x;
      if (!PER_HEAD) p = mul2(p, gg[x]);
      else p = make_float2(s_p[t], s_p[t]), to_end[x] = make_float2(s_e[t], s_e[t]);
      uint32_t a[3], b[3];
      const float2 kp = mul2(kk[x], p), kend = mul2(kk[x], to_end[x]);
      split3x2(kp.x, kp.y, a);
      split3x2(kend.x, kend.y, b);
      const uint32_t at = half * 8192 + e * 1024 + x * 128 + (((lane >> 2) ^ x) << 4);
#pragma unroll
      for (int y = 0; y < 3; ++y) {
        *reinterpret_cast<uint32_t*>(kb + y * (D / 64) * 8192 + at) = a[y];
        *reinterpret_cast<uint32_t*>(record + (R::kKeAt + (lane & 3) * 4 + y * (D / 64) * 8192 + at)) = b[y];
      }
      *reinterpret_cast<float2*>(sQs + t * M::kQRow + ch) = mul2(qq[x], p);
    }
  }
  umma::fence_before_sync();
  __syncthreads();                                       // A has been read
  umma::fence_after_sync();
  uint8_t* sV = smem + M::kAAt;                          // [D / 64 panels][64 rows j]
  static_assert(M::kAAt % 1024 == 0 && M::kA >= (D / 64) * 8192, "values");
  if (warp >= 4) {
#pragma unroll
    for (int i = 0; i < D / 16; ++i) {
      const int e = i * 128 + threadIdx.x - 128, row = e / (D / 8), c16 = e % (D / 8);
      *reinterpret_cast<uint4*>(sV + (c16 >> 3) * 8192 + umma::sw128(row, c16 & 7)) = held[i];
    }
  }
  fence_proxy_async_smem();
  __syncthreads();
  if (threadIdx.x == 0) {
    constexpr uint32_t big = PER_HEAD || BLOCKS ? kBig : kBigUp, small = PER_HEAD || BLOCKS ? kSmall : kSmallDn;
    const bool odd = s_max[0] >= big || s_max[1] >= big || s_max[2] >= kBig || s_max[3] >= kTwo || (s_max[0] > 0 && s_max[0] < small) ||
                     (s_max[1] > 0 && s_max[1] < small) || (s_max[2] > 0 && s_max[2] < kSmall);
    *reinterpret_cast<int*>(record + R::kFlagAt) = odd ? 1 : 0;
  }
  const uint32_t id_w = umma::make_idesc<T>(128, D, 0, 1);
  if (issuer && alive) {
    const uint32_t b0 = umma::desc_low(smem_u32(smem), 8192);
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)
        umma::mma_ts_low(tb + kTmSC, tb + kTmX + term_a(i) * 32 + ks * 8, b0 + ((term_b(i) * (D / 64) * 8192 + ks * 2048) >> 4), id_w,
                         i > 0 || ks > 0);
    umma::commit(made);
  }
  __syncwarp();
  // ------------------------------------------------ out: lane = row r, a warp half of the columns
  const int quarter = warp & 3, side = warp >> 2, r = quarter * 32 + lane, i = r & 63, odd = lane & 1;
  const uint32_t group = ((i >> 3) ^ odd) << 4;          // sw128 of row n + odd, n even, but for n & 6
  const uint32_t base = tb + ((uint32_t)(quarter * 32) << 16) + kTmSC + side * (D / 2);
  alive = alive && wait(made, 0);
  umma::fence_after_sync();
#pragma unroll 1
  for (int c0 = 0; c0 < D / 2; c0 += 16) {
    uint32_t w[16];
    umma::ld16(base + c0, w);
    umma::wait_ld();
    const int n0 = side * (D / 2) + c0;
    float x[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) x[c] = __uint_as_float(w[c]);
    const float part = quarter >= 2 ? 0.f : kCut;
    if (quarter >= 2) {
#pragma unroll
      for (int c = 0; c < 16; c += 4) {
        const float4 qs = *reinterpret_cast<const float4*>(sQs + i * M::kQRow + n0 + c);
        x[c] = fmaf(x[c], -kCut, qs.x) - x[c], x[c + 1] = fmaf(x[c + 1], -kCut, qs.y) - x[c + 1];
        x[c + 2] = fmaf(x[c + 2], -kCut, qs.z) - x[c + 2], x[c + 3] = fmaf(x[c + 3], -kCut, qs.w) - x[c + 3];
      }
    }
    // rows of the record run along r: a lane gets its neighbour's value of one of two channels and writes the pair, in row n0 + c + odd
    const uint32_t at = (quarter >> 1) * (D * 128) + (n0 + odd) * 128 + (i & 6) * 2;
#pragma unroll
    for (int c = 0; c < 16; c += 2) {
      const float other = __shfl_xor_sync(0xffffffffu, odd ? x[c] : x[c + 1], 1);
      uint32_t y[3];
      split3more(make_float2(odd ? other : x[c], odd ? x[c + 1] : other), make_float2(part, part), y);
      uint8_t* to = record + (at + c * 128 + (group ^ ((c & 6) << 4)));
#pragma unroll
      for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t*>(to + p * (2 * D * 128)) = y[p];
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  if (issuer && alive) {
    const uint32_t b0 = umma::desc_low(smem_u32(sV), 8192);
#pragma unroll
    for (int p = 2; p >= 0; --p)
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)
        umma::mma_ts_low(tb + kTmSC, tb + kTmX + p * 32 + ks * 8, b0 + ((ks * 2048) >> 4), id_w, p < 2 || ks > 0);
    umma::commit(made);
  }
  __syncwarp();
  alive = alive && wait(made, 1);
  umma::fence_after_sync();
  const uint32_t uo = R::kUoAt + (side * (D / 2) * R::kUoRow + r) * 4;
#pragma unroll 1
  for (int c0 = 0; c0 < D / 2; c0 += 16) {
    uint32_t w[16];
    umma::ld16(base + c0, w);
    umma::wait_ld();
    float* to = reinterpret_cast<float*>(record + (uo + c0 * R::kUoRow * 4));
#pragma unroll
    for (int c = 0; c < 16; ++c) to[c * R::kUoRow] = __uint_as_float(w[c]);
  }
  umma::fence_before_sync();
  if (*gave_up) {                                        // products under way finish before the columns and the operands go
    if (issuer) umma::commit(drained);
    if (warp == 0) __syncwarp(), mbar_wait_bounded(drained, 0, nullptr, kDrainNs);
  }
  __syncthreads();
  if (warp == 1) umma::tmem_dealloc(tb, 256);
  if (threadIdx.x == 0 && *gave_up) {
    *reinterpret_cast<volatile int*>(W.wait_status) = 1;
    __threadfence_system();
  }
}

// A chunk whose decays are too strong for the scores of delta_chunk_kernel, from there on. A call, as the last thing that CTA does: nothing
// of the kernel's own way lives across it
template <int D>
__device__ __noinline__ void dc_block_chunk(DcChunk W) {
  dc_block_scores<D>(W);
  dc_chunk_rest<D, false, true>(W);
}

template <int D, bool PER_HEAD>
__global__ void __launch_bounds__(kDcThreads, 2)
delta_chunk_kernel(const __grid_constant__ DcParams DP) {
  using T = __nv_bfloat16;
  const DeltaParams& P = DP.d;
  const DcLocal<D> L;
  uint8_t* const smem = L.at;
  float *const s_tau = L.tau(), *const s_beta = L.beta(), *const s_g = L.g(), *const s_p = L.p(), *const s_e = L.e();
  uint64_t *const scored = L.scored(), *const made = L.made(), *const drained = L.drained();
  uint32_t *const s_max = L.max(), *const tmem_slot = L.tmem_slot();
  int *const s_where = L.where(), *const s_next = L.next();
  volatile int* const gave_up = L.gave_up();

  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.x % P.H, lin = DP.c.first + blockIdx.x / P.H;
  if (warp == 0) {                                       // the sequence of chunk `lin`
    int base = 0, found = -1, at = 0;
    for (int s0 = 0; s0 < DP.num_seqs && found < 0; s0 += 32) {
      const int n = s0 + lane < DP.num_seqs ? chunks_of(P.cu_q[s0 + lane + 1] - P.cu_q[s0 + lane]) : 0;
      int to = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, to, o);
        if (lane >= o) to += up;
      }
      const uint32_t hit = __ballot_sync(0xffffffffu, lin < base + to);
      if (hit != 0) {
        const int l = __ffs(hit) - 1;
        found = s0 + l, at = lin - base - __shfl_sync(0xffffffffu, to - n, l);
      }
      base += __shfl_sync(0xffffffffu, to, 31);
    }
    if (lane == 0) s_where[0] = found, s_where[1] = at;
  }
  if (threadIdx.x == 32) {
    mbar_init(scored, 1), mbar_init(made, 1), mbar_init(drained, 1);
    mbar_fence_init();
    for (int i = 0; i < 4; ++i) s_max[i] = 0;
    *s_next = 0, *gave_up = 0;
  }
  __syncthreads();
  const int s = s_where[0], chunk = s_where[1];
  if (s < 0) return;                                     // the grid has room for sequences that all end in a chunk of their own
  if (warp == 1) umma::tmem_alloc(tmem_slot, 256);
  const int64_t tok0 = P.cu_q[s] + chunk * kDcL;
  const int nt = min(kDcL, P.cu_q[s + 1] - (int)tok0);
  const int grp = h / (P.H / P.groups);
  const float* q = P.q + tok0 * P.q_stride + (int64_t)grp * D;
  const float* k = P.k + tok0 * P.k_stride + (int64_t)grp * D;
  const float* g = P.g + tok0 * ((int64_t)P.H * (PER_HEAD ? 1 : D)) + (int64_t)h * (PER_HEAD ? 1 : D);
  const int64_t g_stride = (int64_t)P.H * (PER_HEAD ? 1 : D);
  const T* v = (const T*)P.v + tok0 * P.v_stride + (int64_t)h * D;
  uint8_t* record = DP.c.records + ((int64_t)(lin - DP.c.first) * P.H + h) * DP.c.bytes;
  const bool issuer = warp == 0 && umma::elect_one();
  auto wait = [&](uint64_t* bar, int parity) { return mbar_warp_wait(bar, parity & 1, DP.wait_tries, gave_up); };

  if (threadIdx.x < kDcL) {
    const int t = threadIdx.x;
    const float b = t < nt ? P.beta[(tok0 + t) * P.H + h] : 0.f;
    s_beta[t] = b;
    uint32_t most = magnitude(b);
    if (PER_HEAD) {
      const float d = t < nt ? g[t * g_stride] : 1.f;
      s_g[t] = d;
      most = max(most, magnitude(d));
    }
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0) atomicMax(&s_max[3], most);
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tb = *tmem_slot;
  if (PER_HEAD && threadIdx.x < kDcL) {
    float p = 1.f, e = 1.f;
    for (int i = 0; i <= (int)threadIdx.x; ++i) p *= s_g[i];
    for (int i = kDcL - 1; i > (int)threadIdx.x; --i) e *= s_g[i];
    s_p[threadIdx.x] = p, s_e[threadIdx.x] = e;
  }

  const DcTokens C{k, q, g, (uint32_t)P.k_stride * 4, (uint32_t)P.q_stride * 4, (uint32_t)g_stride * 4, nt};
  bool alive = true;
  // ------------------------------------------------ scores, 64 channels at a time; a thread has two channels and 8 tokens
  float most_k = 0.f, most_q = 0.f, most_g = 0.f;
  const float2 one = make_float2(1.f, 1.f);
#pragma unroll 1
  for (int half = 0; half < D / 64; ++half) {
    const int ch = half * 64 + 2 * lane;
    float2 kk[8], qq[8], gg[8];
    dc_fetch<PER_HEAD>(C, 8 * warp, ch, kk, qq, gg);
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      most_k = largest(most_k, kk[x]), most_q = largest(most_q, qq[x]);
      if (!PER_HEAD) most_g = largest(most_g, gg[x]);
    }
    // the decay between a token and the chunk's middle, between tokens 31 and 32: of this warp's nearest tokens `f`. All warps have the same channels and
    // look at all decays between eight tokens and the middle: one way or the other, they go it together
    float2 f = one;
    if (!PER_HEAD) {
      float2 all = gg[0];
#pragma unroll
      for (int x = 1; x < 8; ++x) all = mul2(all, gg[x]);
      float2* tau = reinterpret_cast<float2*>(s_tau + half * 512) + lane;      // [8][32] pairs
      tau[warp * 32] = all;
      __syncthreads();
      float least = 1.f;
#pragma unroll
      for (int side = 0; side < 2; ++side) {
        float2 r = one;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          if ((side ? 4 + w : 3 - w) == warp) f = r;
          r = mul2(r, tau[(side ? 4 + w : 3 - w) * 32]);
          least = fminf(least, fminf(fabsf(r.x), fabsf(r.y)));
        }
      }
      if (__any_sync(0xffffffffu, !(least >= kNear))) {
        dc_block_chunk<D>(DcChunk{C, v, P.v_stride, record, tb, half, DP.wait_tries, alive, DP.wait_status});
        return;
      }
    }
    if (half > 0) {                                      // the products of the channels before have read their operands
      alive = alive && wait(scored, half - 1);
      umma::fence_after_sync();
    }
    uint8_t* to = smem + (lane & 3) * 4 + warp * 1024;
    auto put_up = [&](int x, float2 up) { dc_put_up(to, lane, x, kk[x], qq[x], up); };
    auto put_dn = [&](int x, float2 dn) { dc_put_dn(to, lane, x, kk[x], dn); };
    if (PER_HEAD) {
#pragma unroll
      for (int x = 0; x < 8; ++x) put_up(x, one), put_dn(x, one);
    } else {
      // (a token's two factors are one and its reciprocal: between tokens that are near each other, no rounding but those of the decays in between)
      auto inverse = [](float2 x) { return make_float2(rcp_newton(x.x), rcp_newton(x.y)); };
      if (warp < 4) {
#pragma unroll
        for (int x = 7; x >= 0; --x) {
          put_dn(x, f);
          put_up(x, inverse(f));
          f = mul2(f, gg[x]);
        }
      } else {
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          f = mul2(f, gg[x]);
          put_up(x, f);
          put_dn(x, inverse(f));
        }
      }
    }
    fence_proxy_async_smem();
    __syncthreads();
    if (issuer && alive) dc_issue_scores<D>(smem, tb + kTmSC + half * 128, scored);
    __syncwarp();
  }
  const uint32_t mk = __reduce_max_sync(0xffffffffu, magnitude(most_k)), mq = __reduce_max_sync(0xffffffffu, magnitude(most_q)),
                 mg = __reduce_max_sync(0xffffffffu, magnitude(most_g));
  if (lane == 0) atomicMax(&s_max[0], mk), atomicMax(&s_max[1], mq), atomicMax(&s_max[3], mg);
  dc_chunk_rest<D, PER_HEAD, false>(DcChunk{C, v, P.v_stride, record, tb, D / 64, DP.wait_tries, alive, DP.wait_status});
}


constexpr int kDsThreads = 288;
template <int D, int NH>
constexpr int ds_smem() {
  return 1024 + NH * (DcRecord<D>::kWq + DcRecord<D>::kKe + DcRecord<D>::kUo) + 2 * NH * D * 4 + 256;
}

template <int D, int NH>
__global__ void __launch_bounds__(kDsThreads, 1)
delta_scan_kernel(const __grid_constant__ DcParams DP) {
  using T = __nv_bfloat16;
  using R = DcRecord<D>;
  static_assert(D * NH == 128, "128 value channels");
  const DeltaParams& P = DP.d;
  extern __shared__ __align__(1024) uint8_t ds_smem_raw[];
  uint8_t* smem = ds_smem_raw + (-smem_u32(ds_smem_raw) & 1023u);       // (not through an integer: the compiler has to know that it is shared memory)
  uint8_t *sWq = smem, *sKe = sWq + NH * R::kWq, *sUo = sKe + NH * R::kKe;
  float* sPe = reinterpret_cast<float*>(sUo + NH * R::kUo);            // [2][NH * D]
  uint64_t *wq_full = reinterpret_cast<uint64_t*>(sPe + 2 * NH * D), *ke_full = wq_full + 1, *uo_full = wq_full + 2, *s_ready = wq_full + 9,
           *e_done = wq_full + 4, *w_ready = wq_full + 5, *d_done = wq_full + 6, *uo_read = wq_full + 7, *drained = wq_full + 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(wq_full + 11);                     // (s_ready: two)
  volatile int* gave_up = reinterpret_cast<volatile int*>(tmem_slot + 1);
  // S 3 x D / 2 (w 3 x 32 in its place), E in two accumulators of 128, dS in place of the second. E starts with the half of every warp's rows of S
  // that is ready first: its accumulator has the products of those rows, largest last, and the other half has one of its own
  constexpr uint32_t kTmS = 0, kTmW = 0, kTmE = 192, kTmD = 320;

  pdl_wait();
  const int s = blockIdx.y, h0 = blockIdx.x * NH, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const SeqSpan sp = seq_span(P.cu_q, P.cu_k, nullptr, s);
  const int before = chunks_before(P.cu_q, s);
  const int lo = max(0, DP.c.first - before), hi = min(chunks_of(sp.q_len), DP.c.first + DP.c.count - before), chunks = hi - lo;
  if (chunks <= 0) return;
  uint8_t* records = DP.c.records + ((int64_t)(before + lo - DP.c.first) * P.H + h0) * DP.c.bytes;       // of chunk lo; a chunk on: P.H records
  const int64_t step = (int64_t)P.H * DP.c.bytes;
  const bool first_pass = lo == 0, last_pass = hi == chunks_of(sp.q_len);

  const int c = (warp & 3) * 32 + lane, half = warp >> 2, hh = NH == 2 ? (c >> 6) : 0;
  float S[D / 2];                                        // S[n][c], n = half * D / 2 + i
  const int64_t own = (int64_t)half * (D / 2) * D + (c & (D - 1));     // of a state [D, D]
  bool odd = false;
  if (warp < 8) {
#pragma unroll
    for (int i = 0; i < D / 2; ++i) S[i] = 0.f;
    if (first_pass ? P.state != nullptr && sp.first_pos() > 0 : true) {
      const float* from = chunk_state_in(P, DP.c, s, h0 + hh) + own;
#pragma unroll
      for (int i = 0; i < D / 2; ++i) S[i] = from[i * D];
#pragma unroll
      for (int i = 0; i < D / 2; ++i) odd = odd || magnitude(S[i]) >= kBig;
    }
  }
  for (int j = threadIdx.x; j < chunks * NH; j += kDsThreads)
    odd = odd || *reinterpret_cast<const int*>(records + (int64_t)(j / NH) * step + (j % NH) * DP.c.bytes + R::kFlagAt) != 0;
  if (threadIdx.x == 0) {
    mbar_init(wq_full, 1), mbar_init(ke_full, 1), mbar_init(uo_full, 1), mbar_init(s_ready, 256), mbar_init(s_ready + 1, 256), mbar_init(e_done, 1), mbar_init(w_ready, 256);
    mbar_init(d_done, 1), mbar_init(uo_read, 256), mbar_init(drained, 1);
    mbar_fence_init();
    *gave_up = 0;
  }
  if (__syncthreads_or(odd)) {                           // one token at a time, behind this kernel
    if (threadIdx.x < NH) *reinterpret_cast<int*>(records + threadIdx.x * DP.c.bytes + R::kFlagAt) = 1;
    return;
  }
  if (warp == 8) umma::tmem_alloc(tmem_slot, 512);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  constexpr uint32_t tb = 0;                             // all 512 columns: they start at 0
  auto wait = [&](uint64_t* bar, int parity) { return mbar_warp_wait(bar, parity & 1, DP.wait_tries, gave_up); };

  if (warp < 8) {
    const uint32_t base = tb + ((uint32_t)((warp & 3) * 32) << 16);
    const int64_t out_stride = (int64_t)P.H * D;
    float* out = P.out + (int64_t)h0 * D + c;
    const float4* uo = reinterpret_cast<const float4*>(sUo + c * (R::kUoRow * 4));
    const float2 part = make_float2(kCut, kCut);
    auto update = [&](int j, int piece) {                // a half of this thread's rows of S after chunk j - 1
      const float* pe = sPe + ((j - 1) & 1) * (NH * D) + hh * D + half * (D / 2);
#pragma unroll
      for (int i0 = piece * (D / 4); i0 < (piece + 1) * (D / 4); i0 += 16) {
        uint32_t w[16];
        umma::ld16(base + kTmD + half * (D / 2) + i0, w);
        umma::wait_ld();
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
          const float4 p = *reinterpret_cast<const float4*>(pe + i0 + i);
#pragma unroll
          for (int y = 0; y < 4; y += 2) {
            const float2 d = both(w[i + y], w[i + y + 1]);
            const float2 r = add2(fma2(y ? make_float2(p.z, p.w) : make_float2(p.x, p.y), make_float2(S[i0 + i + y], S[i0 + i + y + 1]), mul2(d, part)), d);
            S[i0 + i + y] = r.x, S[i0 + i + y + 1] = r.y;
          }
        }
      }
    };
    for (int j = 0;; ++j) {
      if (j > 0) {
        if (!wait(d_done, j - 1)) break;
        umma::fence_after_sync();
      }
      if (j == chunks) {                                 // the last update
        update(j, 0), update(j, 1);
        break;
      }
#pragma unroll
      for (int piece = 0; piece < 2; ++piece) {          // as the A operand: packed pairs along n
        if (j > 0) update(j, piece);
#pragma unroll
        for (int i0 = piece * (D / 4); i0 < (piece + 1) * (D / 4); i0 += 16) {
          uint32_t w[3][8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            uint32_t x[3];
            split3cut(S[i0 + 2 * i], S[i0 + 2 * i + 1], x);
            w[0][i] = x[0], w[1][i] = x[1], w[2][i] = x[2];
          }
#pragma unroll
          for (int p = 0; p < 3; ++p) umma::st8(base + kTmS + p * (D / 2) + half * (D / 4) + i0 / 2, w[p]);
        }
        umma::wait_st();
        umma::fence_before_sync();
        mbar_arrive(s_ready + piece);
      }
      if (!wait(uo_full, j) || !wait(e_done, j)) break;
      umma::fence_after_sync();
#pragma unroll
      for (int u = 0; u < 2; ++u) {                      // what is written: this thread's 32 tokens
        uint32_t e[16], more[16], w[3][8];
        umma::ld16(base + kTmE + half * 32 + 16 * u, e);
        umma::ld16(base + kTmE + 128 + half * 32 + 16 * u, more);
        float4 x[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = uo[half * 8 + 4 * u + i];
        umma::wait_ld();
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int z = 0; z < 4; z += 2) {
            const float2 read_ = add2(both(e[4 * i + z], e[4 * i + z + 1]), both(more[4 * i + z], more[4 * i + z + 1]));
            uint32_t y[3];
            split3more(fma2(read_, make_float2(-1.f, -1.f), z ? make_float2(x[i].z, x[i].w) : make_float2(x[i].x, x[i].y)), part, y);
            w[0][2 * i + z / 2] = y[0], w[1][2 * i + z / 2] = y[1], w[2][2 * i + z / 2] = y[2];
          }
#pragma unroll
        for (int p = 0; p < 3; ++p) umma::st8(base + kTmW + p * 32 + half * 16 + 8 * u, w[p]);
      }
      float read[32];                                    // (P q - Y) S0 for the outputs: dS takes the place of its second half
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        uint32_t e[16], more[16];
        umma::ld16(base + kTmE + 64 + half * 32 + 16 * u, e);
        umma::ld16(base + kTmE + 128 + 64 + half * 32 + 16 * u, more);
        umma::wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) read[16 * u + i] = __uint_as_float(e[i]) + __uint_as_float(more[i]);
      }
      umma::wait_st();
      umma::fence_before_sync();
      mbar_arrive(w_ready);
      const int t0 = (lo + j) * kDcL + half * 32, left = sp.q_len - t0;
      float* to = out + (sp.q_start + (int64_t)t0) * out_stride;
#pragma unroll
      for (int i = 0; i < 32; i += 4) {
        const float4 x = uo[16 + half * 8 + i / 4];
        const float o[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int y = 0; y < 4; ++y) read[i + y] = o[y] + fmaf(o[y] + read[i + y], kCut, read[i + y]);
      }
      if (left >= 32) {
#pragma unroll
        for (int i = 0; i < 32; ++i, to += out_stride) *to = read[i];
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i, to += out_stride)
          if (i < left) *to = read[i];
      }
      umma::fence_before_sync();
      mbar_arrive(uo_read);
    }
    if (P.state != nullptr || !last_pass) {
      float* to = chunk_state_out(P, DP.c, s, h0 + hh) + own;
#pragma unroll
      for (int i = 0; i < D / 2; ++i) to[i * D] = S[i];
    }
  } else {
    const uint32_t id_e = umma::make_idesc<T>(128, 128, 0, 1), id_d = umma::make_idesc<T>(128, D, 0, 1);
    const uint32_t dwq = umma::desc_low(smem_u32(sWq), D * 128), dke = umma::desc_low(smem_u32(sKe), 8192);
    const bool leader = umma::elect_one();
    auto load = [&](int j, int at, int bytes, uint8_t* to, uint64_t* bar, bool ends) {       // (ends: with P_end)
      if (leader) {
        mbar_expect_tx(bar, NH * (bytes + (ends ? D * 4 : 0)));
        for (int n = 0; n < NH; ++n) {
          const uint8_t* from = records + j * step + n * DP.c.bytes;
          bulk_load(to + n * bytes, from + at, bytes, bar);
          if (ends) bulk_load(sPe + (j & 1) * (NH * D) + n * D, from + R::kPeAt, D * 4, bar);
        }
      }
      __syncwarp();
    };
    auto load_wq = [&](int j) { load(j, 0, R::kWq, sWq, wq_full, false); };
    auto load_ke = [&](int j) { load(j, R::kKeAt, R::kKe, sKe, ke_full, false); };
    auto load_uo = [&](int j) { load(j, R::kUoAt, R::kUo, sUo, uo_full, true); };
    int wq = 0, ke = 0, uo = 0;                          // copies begun
    if (DP.wait_tries > 0) load_wq(wq++), load_uo(uo++), load_ke(ke++);      // (a limit of 0 tests the way out: nothing comes)
    for (int j = 0; j < chunks; ++j) {
      const bool more = j + 1 < chunks;
      if (!wait(wq_full, j)) break;
      bool ready = true;
#pragma unroll 1
      for (int piece = 0; ready && piece < 2; ++piece) {
        ready = wait(s_ready + piece, j);
        if (!ready) break;
        umma::fence_after_sync();
        if (leader) {
          const uint32_t to = tb + kTmE + 128 * piece;
#pragma unroll 1
          for (int i = 0; i < 6; ++i) {
            const uint32_t pa = term_a(i), pb = term_b(i);
#pragma unroll
            for (int n = 0; n < NH; ++n)
#pragma unroll
              for (int x = 0; x < D / 32; ++x) {         // 16 rows each: those of the first four warps, then of the others
                const int in = x % (D / 64), ks = (x / (D / 64)) * (D / 32) + piece * (D / 64) + in;
                const uint32_t a = tb + kTmS + pa * (D / 2) + ks * 8, b = dwq + ((n * R::kWq + pb * (2 * D * 128) + ks * 2048) >> 4);
                if (NH == 2) mma_ts_half_low(to, a, b, id_e, i > 0 || x > 0, n);
                else umma::mma_ts_low(to, a, b, id_e, i > 0 || x > 0);
              }
          }
          if (piece == 1) umma::commit(e_done);
        }
        __syncwarp();
      }
      if (!ready) break;
      if (!wait(e_done, j)) break;
      if (more) load_wq(wq++);
      if (!wait(ke_full, j) || !wait(w_ready, j)) break;
      umma::fence_after_sync();
      if (leader) {
#pragma unroll 1
        for (int i = 0; i < 6; ++i) {
          const uint32_t pa = term_a(i), pb = term_b(i);
#pragma unroll
          for (int n = 0; n < NH; ++n)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
              const uint32_t a = tb + kTmW + pa * 32 + ks * 8, b = dke + ((n * R::kKe + pb * (D / 64) * 8192 + ks * 2048) >> 4);
              if (NH == 2) mma_ts_half_low(tb + kTmD, a, b, id_d, i > 0 || ks > 0, n);
              else umma::mma_ts_low(tb + kTmD, a, b, id_d, i > 0 || ks > 0);
            }
        }
        umma::commit(d_done);
      }
      __syncwarp();
      if (!wait(uo_read, j)) break;
      if (more) load_uo(uo++);
      if (!wait(d_done, j)) break;
      if (more) load_ke(ke++);
    }
    // copies and products under way finish before the columns and the operands go
    if (*gave_up) {
      if (wq > 0) mbar_wait_bounded(wq_full, (wq - 1) & 1, nullptr, kDrainNs);
      if (ke > 0) mbar_wait_bounded(ke_full, (ke - 1) & 1, nullptr, kDrainNs);
      if (uo > 0) mbar_wait_bounded(uo_full, (uo - 1) & 1, nullptr, kDrainNs);
      __syncwarp();
    }
    if (leader) umma::commit(drained);
    __syncwarp();
    mbar_wait_bounded(drained, 0, nullptr, kDrainNs);
    __syncwarp();
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 8) umma::tmem_dealloc(tb, 512);
  if (threadIdx.x == 0 && *gave_up) {
    *reinterpret_cast<volatile int*>(DP.wait_status) = 1;
    __threadfence_system();
  }
}

constexpr int64_t kDcWorkspace = 512ll << 20;           // more than this and a step takes several passes

static int64_t dc_chunks(int num_seqs, int64_t total_q) { return total_q / kDcL + num_seqs; }      // no step has more
static int64_t dc_record(int D) { return D == 128 ? DcRecord<128>::kBytes : DcRecord<64>::kBytes; }

// Steps with a span of 96 tokens at least whose chunks are the faster way. Both ways' times in ns, fitted to the times of prompts of 96 to 1024 tokens,
// 1 to 64 at a time: chunks by the waves of delta_chunk_kernel (one that leaves no SM a second CTA takes 0.6 of a full one) and the length that a
// scan's CTA walks; 70 of 75 points are met within 11 %. Strong decays are not the host's to see: the line is for decays that need no blocks. us,
// tokens / chunks (with strong decays), a decay per channel:
//   8 heads of 128:  1 x 128 48 / 37 (46), x 256 93 / 45 (55), x 1024 361 / 99 (108);  4 x 256 93 / 50 (59);  8 x 400 144 / 111 (143);  16 x 96 61 / 57 (72),
//                    x 192 116 / 96 (126), x 256 153 / 106 (144), x 400 236 / 174 (232), x 1024 594 / 325 (416);  64 x 96 231 / 200 (260), x 128 305 / 198 (261);
//                    16 of 500-1250 699 / 314 (401);  1024 beside 32 x 1 364 / 140 (171), beside 64 x 16 430 / 176 (222);  [1 x 96 37 / 37 (47), 8 x 96 38 / 41 (52): tokens]
//   32 heads of 64:  1 x 128 40 / 32 (39), x 256 77 / 43 (50), x 1024 299 / 121 (144);  2 x 400 119 / 79 (92);  4 x 256 77 / 70 (89), x 512 151 / 131 (174),
//                    x 1024 301 / 227 (286);  4 of 300-600 177 / 142 (181);  [4 x 400 119 / 128, 8 x 256 78 / 116, 16 x 1024 510 / 755: tokens]
// A decay per head: tokens 0.86 to 0.93 of that, chunks the same.
static bool dc_shape(int mode, int dtype, int num_seqs, int max_q, int64_t total_q, int H, int kdim, int vdim) {
  if (mode == kWkv || dtype != B200_DTYPE_BF16 || num_seqs <= 0 || num_seqs > 65535 || kdim != vdim || max_q < 96) return false;
  if (!(kdim == 128 || (kdim == 64 && H % 2 == 0)) || H > 65535 || (total_q / kDcL + num_seqs) * H > INT_MAX / 2) return false;
  const bool wide = kdim == 128, even = total_q == (int64_t)num_seqs * max_q;
  const int64_t sms = sm_count(), wave = 2 * sms;        // CTAs at a time
  // waves in tenths: known where all spans are of one length, otherwise as many as half a chunk more per span comes to
  const int64_t chunks = (even ? (int64_t)num_seqs * ((max_q + kDcL - 1) / kDcL) : total_q / kDcL + num_seqs / 2) * H, rest = chunks % wave;
  const int64_t waves = even ? chunks / wave * 10 + (rest > sms ? 10 : rest > 0 ? 6 : 0) : chunks * 10 / wave + 5;
  const int64_t scan = std::max<int64_t>(max_q, total_q * H * kdim / 128 / sms);
  const int64_t chunks_ns = (wide ? 8000 : 11000) + 63 * scan + (wide ? 4050 : 2340) * waves;
  const bool head = mode == kDecayPerHead;
  const int64_t tokens_ns = wide ? 4000 + std::max<int64_t>((head ? 328ll : 350ll) * max_q, total_q * H * (head ? 390 : 445) / 100)
                                 : 2500 + std::max<int64_t>((head ? 284ll : 290ll) * max_q, total_q * H * (head ? 92 : 97) / 100);
  return chunks_ns < tokens_ns * 99 / 100;
}

int64_t delta_chunks_workspace(int mode, int dtype, int num_seqs, int max_q, int64_t total_q, int H, int groups, int kdim, int vdim) {
  if (H <= 0 || groups <= 0 || H % groups != 0 || !dc_shape(mode, dtype, num_seqs, max_q, total_q, H, kdim, vdim)) return 0;
  const int64_t chunk = dc_record(kdim) * H, carry = (int64_t)H * kdim * vdim * 4, all = dc_chunks(num_seqs, total_q) * chunk;
  return carry + std::min(all, std::max(chunk, kDcWorkspace / chunk * chunk));
}

bool delta_chunks_ok(const DeltaParams& P, int mode, int dtype, int num_seqs, int max_q, int64_t total_q, const void* workspace, int64_t bytes) {
  if (P.cu_q == nullptr || workspace == nullptr || !aligned16(workspace)) return false;
  if (!dc_shape(mode, dtype, num_seqs, max_q, total_q, P.H, P.kdim, P.vdim)) return false;
  if (bytes < (int64_t)P.H * (dc_record(P.kdim) + (int64_t)P.kdim * P.vdim * 4)) return false;
  if (std::max(P.q_stride, P.k_stride) >= 1 << 22 || (int64_t)P.H * P.kdim >= 1 << 22) return false;       // (32-bit offsets inside a chunk)
  if (P.q_stride % 4 != 0 || P.k_stride % 4 != 0 || !aligned16(P.q) || !aligned16(P.k) || (mode == kDecayPerChannel && !aligned16(P.g))) return false;
  return P.v_stride % 8 == 0 && aligned16(P.v);
}

template <int D, bool PER_HEAD>
static int delta_chunks_launch_as(DcParams DP, int mode, int64_t total_q, int64_t bytes, cudaStream_t stream) {
  constexpr int NH = 128 / D;
  auto chunk = delta_chunk_kernel<D, PER_HEAD>;
  auto scan = delta_scan_kernel<D, NH>;
  constexpr int chunk_smem = DcSmem<D>::kBytes, scan_smem = ds_smem<D, NH>();
  static_assert(2 * (chunk_smem + 1024) <= 228 * 1024 && scan_smem <= 227 * 1024, "two CTAs' shared memory, one's");
  static std::atomic<uint64_t> chunk_devices{0}, scan_devices{0};
  cudaError_t allowed = allow_smem(chunk, chunk_smem, chunk_devices);
  if (allowed == cudaSuccess) allowed = allow_smem(scan, scan_smem, scan_devices);
  if (allowed != cudaSuccess) return (int)allowed;
  const DeltaParams& P = DP.d;
  const int64_t chunks = dc_chunks(DP.num_seqs, total_q), record = DcRecord<D>::kBytes, carry = (int64_t)P.H * D * D * 4;
  int64_t room = (bytes - carry) / (record * P.H);
  const bool two = P.state == nullptr && room > 1 && room < chunks;      // two carried states, the second in the place of a part of a chunk
  if (two) room = (bytes - 2 * carry) / (record * P.H);
  const int64_t passes = (chunks + room - 1) / room, count = (chunks + passes - 1) / passes;
  static_assert(D * D * 4 < DcRecord<D>::kBytes, "a second carried state leaves one chunk of two");
  DP.c.bytes = record, DP.c.flag_at = DcRecord<D>::kFlagAt, DP.c.count = (int)count;
  float* const carried = reinterpret_cast<float*>(DP.c.records + count * record * P.H);
  const int64_t other = two ? carry / 4 : 0;
  for (int64_t at = 0, pass = 0; at < chunks; at += count, ++pass) {
    DP.c.first = (int)at;
    DP.c.carry_in = carried + (pass & 1 ? 0 : other), DP.c.carry_out = carried + (pass & 1 ? other : 0);
    launch_pdl(chunk, dim3((unsigned)(count * P.H)), dim3(kDcThreads), (size_t)chunk_smem, stream, DP);
    launch_pdl(scan, dim3((unsigned)(P.H / NH), (unsigned)DP.num_seqs), dim3(kDsThreads), (size_t)scan_smem, stream, DP);
    const int code = delta_rest_launch(P, DP.c, mode, DP.num_seqs, count >= chunks, stream);
    if (code != B200_OK) return code;
  }
  return finish_launch((int)(2 * ((chunks + count - 1) / count)));
}

int delta_chunks_launch(const DeltaParams& P, int mode, int num_seqs, int64_t total_q, void* workspace, int64_t bytes, int64_t wait_ns,
                        cudaStream_t stream) {
  B200_RETURN_IF(take_wait_status(), B200_ERR_WAIT);     // of an earlier call
  DcParams DP{};
  DP.d = P, DP.num_seqs = num_seqs, DP.wait_tries = wait_tries(wait_ns), DP.wait_status = wait_status();
  DP.c.records = reinterpret_cast<uint8_t*>(workspace);
  B200_RETURN_IF(DP.wait_status == nullptr, B200_ERR_DRIVER);
  if (mode == kDecayPerHead)
    return P.kdim == 128 ? delta_chunks_launch_as<128, true>(DP, mode, total_q, bytes, stream) : delta_chunks_launch_as<64, true>(DP, mode, total_q, bytes, stream);
  return P.kdim == 128 ? delta_chunks_launch_as<128, false>(DP, mode, total_q, bytes, stream) : delta_chunks_launch_as<64, false>(DP, mode, total_q, bytes, stream);
}

}  // namespace b200
