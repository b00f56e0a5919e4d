// seq_mixers.cu -- the two sequence mixers that the tcgen05 attention kernels do not cover:
//
//   attn_generic       causal softmax attention for ANY head sizes (key size != value size, sizes that are
//                      not 64 or 128), any element type including fp32, packed or paged keys, and any mix of
//                      prompt portions and single tokens in one launch. fp32 scores, softmax and accumulation.
//                      Optional: a sliding window (with first tokens that stay visible) or chunks (a token sees its
//                      own chunk only), scores capped by cap * tanh(s / cap), a sink logit per head that joins the
//                      softmax denominator without a value, an output gate sigmoid(logit) per (token, head).
//   linear_recurrence  S_t = a_t S_(t-1) + k_t (b_t v_t)^T, o_t = S_t^T q_t (+ d v_t) per head with the state S
//                      [key size x value size] held in fp32 registers and carried between steps in a slot.
//                      Three forms: a constant decay per head (lightning attention), a decay and a step size
//                      computed per token from a projected dt (the selective state-space form of Mamba-2), or a
//                      forget gate per key channel that also decides what is written (k = 1 - f: the tied form
//                      of HGRN2), S_t = diag(f_t) S_(t-1) + (1 - f_t) v_t^T.
#include "attn_tiled.cuh"
#include "recurrence.cuh"
#include "seq_common.cuh"

namespace b200 {

// ------------------------------------------------------------------ generic attention
// One CTA = 8 warps = 8 "rows" of one (sequence, kv head): row r is query token r / rep, query head
// g * rep + r % rep (rep = H / G), so that the CTA's rows share every key tile. Keys are staged 32 at a
// time in shared memory as fp32; lane j scores key j, then each lane owns value channels lane, lane+32, ...
constexpr int kAttnRows = 8;
constexpr int kAttnKeys = 32;
constexpr int kAttnMaxVChunks = 16;    // value size <= 512

template <typename T>
__global__ void __launch_bounds__(kAttnRows * 32)
attn_generic_kernel(T* __restrict__ out, const T* __restrict__ q, int64_t q_stride, const T* __restrict__ k,
                    int64_t k_stride, const T* __restrict__ v, int64_t v_stride,
                    const int* __restrict__ block_tables, int bt_stride, int block_size,
                    const int* __restrict__ cu_q, const int* __restrict__ cu_k, const int* __restrict__ ctx_lens,
                    int H, int G, int dim, int vdim, float scale, int window, int keep_first, int chunk, float softcap,
                    const float* __restrict__ sink, const T* __restrict__ gate, int64_t gate_stride) {
  extern __shared__ float smem[];
  pdl_wait();
  const int s = blockIdx.z, g = blockIdx.y;
  const SeqSpan sp = seq_span(cu_q, cu_k, ctx_lens, s);
  const int rep = H / G;
  const int rows = sp.q_len * rep;
  const int r0 = blockIdx.x * kAttnRows;
  if (r0 >= rows) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kpad = dim + 1;
  float* sq = smem;                                   // [8][dim]
  float* sk = sq + kAttnRows * dim;                   // [32][dim + 1]
  // v == nullptr: the values are the first vdim columns of the key rows (one latent row serves as key and value)
  const bool v_in_k = v == nullptr;
  float* sv = v_in_k ? sk : sk + kAttnKeys * kpad;    // [32][vdim]
  const int vpad = v_in_k ? kpad : vdim;

  const int r = r0 + warp;
  const bool live = r < rows;
  const int tok = live ? r / rep : 0, head = g * rep + (live ? r % rep : 0);
  const int pos = sp.first_pos() + tok;               // this row sees keys lo .. pos, and those below keep_first
  auto seen_from = [&](int p) { return window > 0 ? max(0, p - window + 1) : chunk > 0 ? p / chunk * chunk : 0; };
  const int lo = seen_from(pos);
  if (live) {
    const T* qr = q + (int64_t)(sp.q_start + tok) * q_stride + (int64_t)head * dim;
    for (int i = lane; i < dim; i += 32) sq[warp * dim + i] = to_f32<T>(qr[i]);
  }
  const int last_row = min(r0 + kAttnRows, rows) - 1;
  const int max_pos = sp.first_pos() + last_row / rep;
  const int64_t k_base = cu_k != nullptr && block_tables == nullptr ? cu_k[s] : 0;

  // a sink is one more entry of the softmax that has a logit and no value: the running state starts from it
  float m = sink != nullptr ? sink[head] : -INFINITY, l = sink != nullptr ? 1.f : 0.f, acc[kAttnMaxVChunks];
#pragma unroll
  for (int c = 0; c < kAttnMaxVChunks; ++c) acc[c] = 0.f;

  const int min_pos = sp.first_pos() + r0 / rep;
  const int first_key = seen_from(min_pos);
  // tiles of the kept keys first, then from the first key of the earliest row's window on
  const int kept = min(keep_first, first_key);
  for (int j0 = kept > 0 ? 0 : first_key; j0 <= max_pos;
       j0 = (j0 < kept && j0 + kAttnKeys >= kept) ? first_key : j0 + kAttnKeys) {
    __syncthreads();                                  // previous tile fully consumed (and sq written)
    const int nk = min(kAttnKeys, (j0 < kept ? kept : max_pos + 1) - j0);
    for (int e = threadIdx.x; e < nk * dim; e += blockDim.x) {
      const int j = e / dim, i = e - j * dim;
      const int key = j0 + j;
      const int64_t row = block_tables != nullptr
                              ? (int64_t)block_tables[(int64_t)s * bt_stride + key / block_size] * block_size + key % block_size
                              : k_base + key;
      sk[j * kpad + i] = to_f32<T>(k[row * k_stride + (int64_t)g * dim + i]);
    }
    for (int e = threadIdx.x; e < (v_in_k ? 0 : nk * vdim); e += blockDim.x) {
      const int j = e / vdim, i = e - j * vdim;
      const int key = j0 + j;
      const int64_t row = block_tables != nullptr
                              ? (int64_t)block_tables[(int64_t)s * bt_stride + key / block_size] * block_size + key % block_size
                              : k_base + key;
      sv[j * vdim + i] = to_f32<T>(v[row * v_stride + (int64_t)g * vdim + i]);
    }
    __syncthreads();
    if (!live || j0 > pos || (j0 + nk <= lo && j0 >= keep_first)) continue;
    float sc = -INFINITY;
    if (lane < nk && j0 + lane <= pos && (j0 + lane >= lo || j0 + lane < keep_first)) {
      float d = 0.f;
      const float* kr = sk + lane * kpad;
      const float* qr = sq + warp * dim;
      for (int i = 0; i < dim; ++i) d += qr[i] * kr[i];
      sc = d * scale;
      if (softcap > 0.f) sc = softcap * tanhf(sc / softcap);
    }
    const float m_new = fmaxf(m, warp_max(sc));
    if (m_new == -INFINITY) continue;                 // nothing visible so far (a tile between kept keys and the window)
    const float corr = expf(m - m_new);               // m = -inf on the first tile: exp(-inf) = 0
    const float p = sc == -INFINITY ? 0.f : expf(sc - m_new);
    l = l * corr + warp_sum(p);
    m = m_new;
#pragma unroll
    for (int c = 0; c < kAttnMaxVChunks; ++c) acc[c] *= corr;
    for (int j = 0; j < nk; ++j) {
      const float pj = __shfl_sync(0xffffffffu, p, j);
#pragma unroll
      for (int c = 0; c < kAttnMaxVChunks; ++c) {
        const int i = lane + 32 * c;
        if (i < vdim) acc[c] += pj * sv[j * vpad + i];
      }
    }
  }
  if (!live) return;
  T* o = out + (int64_t)(sp.q_start + tok) * ((int64_t)H * vdim) + (int64_t)head * vdim;
  float inv = 1.0f / l;
  if (gate != nullptr) inv *= sigmoid_f(to_f32<T>(gate[(int64_t)(sp.q_start + tok) * gate_stride + head]));
#pragma unroll
  for (int c = 0; c < kAttnMaxVChunks; ++c) {
    const int i = lane + 32 * c;
    if (i < vdim) o[i] = from_f32<T>(acc[c] * inv);
  }
}

// ------------------------------------------------------------------ linear recurrence with an fp32 state
// One CTA = 128 threads works on one (sequence, head) and a band of value columns. A thread owns ONE value column
// and KPT <= 64 key rows of the state in registers (all rows when kdim <= 64; 2 or 4 adjacent lanes share a column
// above that, one or two shuffles per token). Per token it reads k and q as float4 broadcasts from shared memory -- every lane of a warp reads the same
// address -- and its own value, and does KPT updates S <- a S + k v and KPT output terms: the loop is fp32-issue
// bound, and state rows are read and written as full 128-byte
// lines (lanes = consecutive columns). Key rows past kdim and columns past vdim are zero-padded in shared memory,
// so the inner loop has no bounds tests. Tokens are staged kRecTok at a time; the next batch is fetched into
// registers while the current one is consumed.
constexpr int kRecTok = 8;


template <typename T, typename TV, int KPT, int NS>
__global__ void __launch_bounds__(128)
linear_recurrence_kernel(const RecParams P) {
  extern __shared__ __align__(16) float smem[];
  pdl_wait();
  constexpr int KS = KPT;                            // slice stride (padding it against the 2-way bank conflict of
                                                     // the NS broadcasts cost more in index arithmetic than it saved)
  constexpr int KP = NS * KS;                        // row of padded keys
  constexpr int CC = 128 / NS;                       // value columns per CTA
  const int s = blockIdx.z, h = blockIdx.y;
  const SeqSpan sp = seq_span(P.cu_q, P.cu_k, P.ctx_lens, s);
  if (sp.q_len == 0) return;
  const int kdim = P.kdim, vdim = P.vdim;
  const int ksl = threadIdx.x % NS;                  // key slice: rows ksl*KPT .. ksl*KPT + KPT - 1
  const int cl = threadIdx.x / NS;                   // column within the CTA's band
  const int c0 = blockIdx.x * CC;                    // first column of the band
  const int col = c0 + cl;
  const bool col_ok = col < vdim;
  // a warp none of whose columns exist only helps with the staging (warp-uniform, so shuffles stay legal)
  const bool warp_live = c0 + (int)((threadIdx.x & ~31u) / NS) < vdim;
  const int grp = h / (P.H / P.groups);
  float* sq = smem;                                  // [kRecTok][KP]
  float* skk = sq + kRecTok * KP;                    // [kRecTok][KP]
  float* sx = skk + kRecTok * KP;                    // [kRecTok][CC]
  float* sa = sx + kRecTok * CC;                     // [kRecTok] decay of the step
  float* sdt = sa + kRecTok;                         // [kRecTok] step size (1 for a constant decay)

  float S[KPT];
  float* slot = P.state != nullptr
                    ? P.state + (((int64_t)P.state_slots[s] * P.H + h) * kdim) * (int64_t)vdim
                    : nullptr;
  const bool carried = slot != nullptr && sp.first_pos() > 0;
#pragma unroll
  for (int r = 0; r < KPT; ++r) {
    const int i = ksl * KPT + r;
    S[r] = (carried && col_ok && i < kdim) ? slot[(int64_t)i * vdim + col] : 0.f;
  }
  const T* q = (const T*)P.q + (int64_t)grp * kdim;
  const T* k = (const T*)P.k + (int64_t)grp * kdim;
  const TV* v = (const TV*)P.v + (int64_t)h * vdim + c0;
  const T* dt = (const T*)P.dt;
  const float a_const = P.mode == 0 ? P.decay[h] : 0.f;
  const float rate = P.mode == 1 ? expf(P.a_log[h]) : 0.f;
  const float dt_b = P.mode == 1 ? P.dt_bias[h] : 0.f;
  const float d_skip = P.mode == 1 ? P.d_skip[h] : 0.f;
  const int vcols = min(CC, vdim - c0);

  constexpr int NQ = (kRecTok * KP + 127) / 128;     // q (and k) elements per thread per batch
  constexpr int NV = kRecTok * CC / 128;
  T pq[NQ], pk[NQ], pdt = from_f32<T>(0.f);
  TV pv[NV];
  auto fetch = [&](int t0) {
    const int nt = min(kRecTok, sp.q_len - t0);
    const int64_t tok0 = sp.q_start + t0;
#pragma unroll
    for (int n = 0; n < NQ; ++n) {
      const int e = threadIdx.x + n * 128;
      const int tt = e / KP, w = e % KP;
      const int i = (w / KS) * KPT + w % KS;              // key row of this shared-memory word (padding: none)
      const bool ok = tt < nt && w % KS < KPT && i < kdim;
      pq[n] = ok ? q[(tok0 + tt) * P.q_stride + i] : from_f32<T>(0.f);
      pk[n] = ok ? k[(tok0 + tt) * P.k_stride + i] : from_f32<T>(0.f);
    }
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      const int e = threadIdx.x + n * 128;
      const int tt = e / CC, c = e % CC;
      pv[n] = (tt < nt && c < vcols) ? v[(tok0 + tt) * P.v_stride + c] : from_f32<TV>(0.f);
    }
    if (P.mode == 1 && threadIdx.x < nt) pdt = dt[(tok0 + threadIdx.x) * P.dt_stride + h];
  };
  auto stage = [&](int t0) {                         // registers -> shared memory, activations applied once
    const int nt = min(kRecTok, sp.q_len - t0);
#pragma unroll
    for (int n = 0; n < NQ; ++n) {
      const int e = threadIdx.x + n * 128;
      float qv = to_f32<T>(pq[n]), kv = to_f32<T>(pk[n]);
      // the activation's result is an activation of the model's element type (as in the chunked form, whose
      // tensor-core operands are bf16 values); silu(0) = 0: the padding stays zero
      if (P.act_silu) {
        qv = sizeof(T) == 2 ? silu_fast(qv) : silu_f(qv);
        kv = sizeof(T) == 2 ? silu_fast(kv) : silu_f(kv);
        qv = to_f32<T>(from_f32<T>(qv)), kv = to_f32<T>(from_f32<T>(kv));
      }
      if (e < kRecTok * KP) {
        sq[e] = qv;
        skk[e] = kv;
      }
    }
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      const int e = threadIdx.x + n * 128;
      float x = to_f32<TV>(pv[n]);
      if (P.act_silu) x = to_f32<TV>(from_f32<TV>(sizeof(TV) == 2 ? silu_fast(x) : silu_f(x)));
      sx[e] = x;
    }
    if (threadIdx.x < nt) {
      float a = a_const, step = 1.f;
      if (P.mode == 1) {
        step = softplus_f(to_f32<T>(pdt) + dt_b);
        a = expf(-rate * step);
      }
      sa[threadIdx.x] = a;
      sdt[threadIdx.x] = step;
    }
  };

  fetch(0);
  for (int t0 = 0; t0 < sp.q_len; t0 += kRecTok) {
    const int nt = min(kRecTok, sp.q_len - t0);
    __syncthreads();                                 // the previous batch has been consumed
    stage(t0);
    __syncthreads();
    if (t0 + kRecTok < sp.q_len) fetch(t0 + kRecTok);
    if (!warp_live) continue;
    float* outp = P.out + (int64_t)(sp.q_start + t0) * ((int64_t)P.H * vdim) + (int64_t)h * vdim + col;
    for (int tt = 0; tt < nt; ++tt) {
      const float a = sa[tt], x = sx[tt * CC + cl], vj = x * sdt[tt];
      const float4* q4 = reinterpret_cast<const float4*>(sq + tt * KP + ksl * KS);
      const float4* k4 = reinterpret_cast<const float4*>(skk + tt * KP + ksl * KS);
      float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;
      if (P.mode == 2) {                             // f S + (1 - f) v = v + f (S - v): the gate is the staged `k`
#pragma unroll
        for (int r4 = 0; r4 < KPT / 4; ++r4) {
          const float4 f4 = k4[r4], qq = q4[r4];
          S[r4 * 4 + 0] = fmaf(f4.x, S[r4 * 4 + 0] - vj, vj);
          o0 += S[r4 * 4 + 0] * qq.x;
          S[r4 * 4 + 1] = fmaf(f4.y, S[r4 * 4 + 1] - vj, vj);
          o1 += S[r4 * 4 + 1] * qq.y;
          S[r4 * 4 + 2] = fmaf(f4.z, S[r4 * 4 + 2] - vj, vj);
          o2 += S[r4 * 4 + 2] * qq.z;
          S[r4 * 4 + 3] = fmaf(f4.w, S[r4 * 4 + 3] - vj, vj);
          o3 += S[r4 * 4 + 3] * qq.w;
        }
      } else {
#pragma unroll
      for (int r4 = 0; r4 < KPT / 4; ++r4) {
        const float4 kq = k4[r4], qq = q4[r4];
        S[r4 * 4 + 0] = a * S[r4 * 4 + 0] + kq.x * vj;
        o0 += S[r4 * 4 + 0] * qq.x;
        S[r4 * 4 + 1] = a * S[r4 * 4 + 1] + kq.y * vj;
        o1 += S[r4 * 4 + 1] * qq.y;
        S[r4 * 4 + 2] = a * S[r4 * 4 + 2] + kq.z * vj;
        o2 += S[r4 * 4 + 2] * qq.z;
        S[r4 * 4 + 3] = a * S[r4 * 4 + 3] + kq.w * vj;
        o3 += S[r4 * 4 + 3] * qq.w;
      }
      }
      float o = (o0 + o1) + (o2 + o3);
#pragma unroll
      for (int off = 1; off < NS; off <<= 1) o += __shfl_xor_sync(0xffffffffu, o, off);
      if (ksl == 0 && col_ok) {
        if (P.mode == 1) o += d_skip * x;
        outp[(int64_t)tt * ((int64_t)P.H * vdim)] = o;
      }
    }
  }
  if (slot != nullptr && col_ok) {
#pragma unroll
    for (int r = 0; r < KPT; ++r) {
      const int i = ksl * KPT + r;
      if (i < kdim) slot[(int64_t)i * vdim + col] = S[r];
    }
  }
}

template <typename T, typename TV, int KPT, int NS>
static void recurrence_launch_as(const RecParams& P, int num_seqs, cudaStream_t stream) {
  constexpr int CC = 128 / NS;
  const dim3 grid((P.vdim + CC - 1) / CC, P.H, num_seqs);
  const size_t smem = (size_t)(2 * kRecTok * NS * KPT + kRecTok * CC + 2 * kRecTok) * sizeof(float);
  launch_pdl(linear_recurrence_kernel<T, TV, KPT, NS>, grid, dim3(128), smem, stream, P);
}

// ------------------------------------------------------------------ the same recurrence, 32 tokens at a time
// Prompt portions of bf16 models. With c_i = sum_{s<=i} log a_s inside a chunk of 32 tokens (S0 = state before it):
//   o_i = e^{c_i} S0^T q_i + sum_{j<=i} e^{c_i - c_j} b_j (q_i . k_j) v_j          S32 = e^{c_31} S0 + sum_j e^{c_31 - c_j} b_j k_j v_j^T
// -- three small matrix products per chunk on the tensor cores (mma.sync m16n8k16, fp32 accumulation). The
// 32-bit rule of the recurrence is kept: q, k, v are bf16 values already (exact operands), and every fp32 operand
// (the decayed scores, the state, the decayed values) enters the tensor core as the sum of three bf16 terms
// (hi + mid + lo, 24 bits), so each product is accurate to fp32 rounding. One CTA = one (sequence, head); warp w
// keeps rows 16w .. 16w+15 of S^T [vdim x kdim] as accumulator fragments, which are at the same time the A
// fragments of S^T q (the layout identity that flash attention uses for P V). Sizes are zero-padded to
// kdim <= D (template, 32 / 64 / 128) and vdim <= 128 in shared memory.
// Bound: latency and issue of a warp's chain per chunk (by their 255 registers an SM holds two CTAs of up to 4 warps for
// vdim <= 64, one of up to 8 warps above), so what
// counts is instructions: fragments come by ldmatrix (the A fragment of Q is also the B fragment of Q^T), the splits
// by packed conversions, every warp keeps the decays in its lanes (one CTA barrier per chunk) and stores its outputs
// straight from the accumulators; and the split and the scaling of the state are paid once per 32 tokens, not per 16.
// 16 x 1024 tokens, 32 heads of 128 x 64, selective: 673 us at first (1950 instructions per warp and 16 tokens), 419 us with
// chunks of 16 (1420), 328 us with chunks of 32. Chunks of 64 would need 10 more score tiles per warp than there are registers.
// The decays of a chunk are exponentials of sums over at most 16 tokens: across the two blocks they are multiplied, since a
// prefix sum over 32 loses a bit (error of the outputs against 64 bits 4.2e-7 with it, 2.5e-7 so).
constexpr int kChunk = 32;             // two 16-token blocks

// VEC: q, k, v rows start on 16-byte boundaries (strides, sizes and slice offsets % 8 == 0): the tiles of the next
// chunk are copied global -> shared with cp.async while the current chunk is computed (two sets of tiles).
// NW: warps that the shared-memory rows of V are sized for (vdim <= 16 NW); MODE, SILU: P.mode, P.act_silu; CTAS: how many of
// 4 warps an SM is to hold (chunk_recurrence_launch).
template <int D, int NW>
constexpr int chunk_recurrence_smem(bool vec) {
  return (vec ? 2 : 1) * kChunk * (2 * (D + 8) + 16 * NW + 8) * 2;
}
template <int D, int NW, bool VEC, int MODE, bool SILU, int CTAS>
__global__ void __launch_bounds__(32 * NW, CTAS * 4 / NW)
chunk_recurrence_kernel(const RecParams P) {
  using T = __nv_bfloat16;
  constexpr int QS = D + 8;                           // row stride (elements) of the q / k tiles: conflict-free
  constexpr int VS = 16 * NW + 8;
  constexpr int NB = VEC ? 2 : 1;
  extern __shared__ __align__(16) unsigned short s_tiles[];
  unsigned short* sQb = s_tiles;                      // [NB][kChunk][QS]
  unsigned short* sKb = sQb + NB * kChunk * QS;
  unsigned short* sVb = sKb + NB * kChunk * QS;       // [NB][kChunk][VS]
  pdl_wait();
  const int s = blockIdx.z, h = blockIdx.y;
  const SeqSpan sp = seq_span(P.cu_q, P.cu_k, P.ctx_lens, s);
  if (sp.q_len == 0) return;
  const int kdim = P.kdim, vdim = P.vdim;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nthreads = blockDim.x;
  const int g = lane >> 2, t = lane & 3;
  const int r0 = warp * 16;                           // first row (value channel) of this warp's slab of S^T
  const int grp = h / (P.H / P.groups);
  const T* q = (const T*)P.q + (int64_t)grp * kdim;
  const T* k = (const T*)P.k + (int64_t)grp * kdim;
  const T* v = (const T*)P.v + (int64_t)h * vdim;
  const T* dt = (const T*)P.dt;
  const float log_a_const = MODE == 0 ? fmaxf(logf(P.decay[h]), -60.f) : 0.f;   // e^-60: nothing survives a step
  const float rate = MODE == 1 ? expf(P.a_log[h]) : 0.f;
  const float dt_b = MODE == 1 ? P.dt_bias[h] : 0.f;
  const float d_skip = MODE == 1 ? P.d_skip[h] : 0.f;

  float* slot = P.state != nullptr
                    ? P.state + (((int64_t)P.state_slots[s] * P.H + h) * kdim) * (int64_t)vdim
                    : nullptr;
  const bool carried = slot != nullptr && sp.first_pos() > 0;
  if (D <= 64 && sp.q_len == 1) {
    // A single token (a decode row of a mixed step) of a small state is a rank-1 update: one pass over the state, in the order
    // it lies in memory, and no fragments. Thread = value channel x half of the key rows; the block has at least 2 vdim threads.
    // 200 of them beside a prompt of 256, 32 heads of 64 x 64: 134 us as chunks of 32, 98 as chunks of 16, 59 so; 16 heads of 64 x
    // 128 138 / 96 / 61. States of 128 key channels are no slower as chunks (181 / 184), and their registers are all taken.
    float* sq = reinterpret_cast<float*>(s_tiles);    // [D] q, [D] k, [vdim] partial outputs
    float *sk = sq + D, *so = sk + D;
    const int64_t tok = sp.q_start;
    for (int i = threadIdx.x; i < kdim; i += nthreads) {
      float qv = __bfloat162float(q[tok * P.q_stride + i]), kv = __bfloat162float(k[tok * P.k_stride + i]);
      if (SILU) qv = bits_f32(bf16_bits(silu_fast(qv))), kv = bits_f32(bf16_bits(silu_fast(kv)));
      sq[i] = qv, sk[i] = kv;
    }
    const int col = threadIdx.x % vdim, half = threadIdx.x / vdim;
    float x = __bfloat162float(v[tok * P.v_stride + col]), a = MODE == 0 ? P.decay[h] : 0.f, step = 1.f;
    if (SILU) x = bits_f32(bf16_bits(silu_fast(x)));
    if (MODE == 1) {
      step = softplus_f(__bfloat162float(dt[tok * P.dt_stride + h]) + dt_b);
      a = expf(-rate * step);
    }
    __syncthreads();
    const float bx = step * x;
    const int k_lo = half == 0 ? 0 : (kdim + 1) / 2, k_hi = half == 0 ? (kdim + 1) / 2 : half == 1 ? kdim : 0;
    float sum = 0.f;
    for (int i0 = k_lo; i0 < k_hi; i0 += 16) {        // 16 rows on their way at a time
      float row[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) row[i] = carried && i0 + i < k_hi ? slot[(int64_t)(i0 + i) * vdim + col] : 0.f;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        if (i0 + i >= k_hi) break;
        row[i] = fmaf(sk[i0 + i], bx, a * row[i]);
        if (slot != nullptr) slot[(int64_t)(i0 + i) * vdim + col] = row[i];
        sum = fmaf(sq[i0 + i], row[i], sum);
      }
    }
    if (half == 1) so[col] = sum;
    __syncthreads();
    if (half == 0) {
      sum += so[col];
      if (MODE == 1) sum = fmaf(d_skip, x, sum);
      P.out[tok * ((int64_t)P.H * vdim) + (int64_t)h * vdim + col] = sum;
    }
    return;
  }

  // S^T slab: n-tile n = key columns 8n .. 8n+7; [0],[1]: row r0+g, cols 8n+2t, +1; [2],[3]: row r0+g+8
  float S[D / 8][4];
#pragma unroll
  for (int n = 0; n < D / 8; ++n)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int row = r0 + g + (c >> 1) * 8, col = 8 * n + 2 * t + (c & 1);
      S[n][c] = (carried && row < vdim && col < kdim) ? slot[(int64_t)col * vdim + row] : 0.f;
    }

  // asynchronous copy of the raw tiles of chunk c0 into buffer `buf` (zero-filled past the chunk / the sizes)
  auto copy_async = [&](int c0, int buf) {
    const int nt = min(kChunk, sp.q_len - c0);
    const int64_t tok0 = sp.q_start + c0;
    for (int e = threadIdx.x; e < kChunk * (D / 8); e += nthreads) {
      const int j = e / (D / 8), i = (e % (D / 8)) * 8;
      const bool ok = j < nt && i < kdim;
      const int64_t tok = ok ? tok0 + j : sp.q_start;
      cp_async_16(smem_u32(&sQb[(buf * kChunk + j) * QS + i]), q + tok * P.q_stride + (ok ? i : 0), ok);
      cp_async_16(smem_u32(&sKb[(buf * kChunk + j) * QS + i]), k + tok * P.k_stride + (ok ? i : 0), ok);
    }
    for (int e = threadIdx.x; e < kChunk * 2 * NW; e += nthreads) {
      const int j = e / (2 * NW), i = (e % (2 * NW)) * 8;
      const bool ok = j < nt && i < vdim;
      const int64_t tok = ok ? tok0 + j : sp.q_start;
      cp_async_16(smem_u32(&sVb[(buf * kChunk + j) * VS + i]), v + tok * P.v_stride + (ok ? i : 0), ok);
    }
    cp_async_commit();
  };
  float dt_next = 0.f;                                // lane j: token j of the next chunk (every warp keeps its own copy)
  auto fetch_dt = [&](int c0) {
    dt_next = 0.f;
    if (MODE == 1 && c0 + lane < sp.q_len)
      dt_next = __bfloat162float(dt[(sp.q_start + c0 + lane) * P.dt_stride + h]);
  };
  // ldmatrix addresses inside a 16-row tile: rows in order of the lanes, the second 16 lanes 8 columns on (A operand from
  // [row][k], B operand from [k][n] transposed), or the second 8 lanes 8 columns on (B operand from [n][k], A from [k][m])
  const int r_a = lane & 15, c_a = (lane >> 4) * 8, r_b = (lane & 7) + (lane >> 4) * 8, c_b = ((lane >> 3) & 1) * 8;
  if (VEC) copy_async(0, 0);
  fetch_dt(0);

  for (int c0 = 0, it = 0; c0 < sp.q_len; c0 += kChunk, ++it) {
    const int nt = min(kChunk, sp.q_len - c0);
    const int64_t tok0 = sp.q_start + c0;
    const int buf = VEC ? (it & 1) : 0;
    unsigned short* sQ = sQb + buf * kChunk * QS;
    unsigned short* sK = sKb + buf * kChunk * QS;
    unsigned short* sV = sVb + buf * kChunk * VS;
    if (VEC) cp_async_wait<0>();
    __syncthreads();                                  // this chunk's tiles have landed; the previous chunk is consumed
    if (VEC) {
      if (c0 + kChunk < sp.q_len) copy_async(c0 + kChunk, buf ^ 1);
      if (SILU) {                                     // activation in place, 8 values per step
        constexpr int NQ = kChunk * (D / 8);
        for (int e = threadIdx.x; e < 2 * NQ + kChunk * 2 * NW; e += nthreads) {
          unsigned short* p;
          if (e < 2 * NQ) p = (e < NQ ? sQ : sK) + ((e % NQ) / (D / 8)) * QS + (e % (D / 8)) * 8;
          else p = sV + ((e - 2 * NQ) / (2 * NW)) * VS + ((e - 2 * NQ) % (2 * NW)) * 8;
          float f[8];
          load8<T>(reinterpret_cast<const T*>(p), f);
#pragma unroll
          for (int u = 0; u < 8; ++u) f[u] = silu_fast(f[u]);
          store8<T>(reinterpret_cast<T*>(p), f);
        }
      }
    } else {
      for (int e = threadIdx.x; e < kChunk * D; e += nthreads) {
        const int j = e / D, i = e % D;
        float qv = 0.f, kv = 0.f;
        if (j < nt && i < kdim) {
          qv = __bfloat162float(q[(tok0 + j) * P.q_stride + i]);
          kv = __bfloat162float(k[(tok0 + j) * P.k_stride + i]);
          if (SILU) qv = silu_fast(qv), kv = silu_fast(kv);
        }
        sQ[j * QS + i] = (unsigned short)bf16_bits(qv);
        sK[j * QS + i] = (unsigned short)bf16_bits(kv);
      }
      for (int e = threadIdx.x; e < kChunk * 16 * NW; e += nthreads) {
        const int j = e / (16 * NW), i = e % (16 * NW);
        float x = 0.f;
        if (j < nt && i < vdim) {
          x = __bfloat162float(v[(tok0 + j) * P.v_stride + i]);
          if (SILU) x = silu_fast(x);
        }
        sV[j * VS + i] = (unsigned short)bf16_bits(x);
      }
    }
    // log-decay of every token, its prefix sum inside each block of 16 (sums over 32 would lose a bit of the decays), step
    // sizes: lane j holds token j. A padded token neither decays nor adds
    float cum = 0.f, step = 1.f;
    if (lane < nt) {
      cum = log_a_const;
      if (MODE == 1) {
        step = softplus_f(dt_next + dt_b);
        cum = -rate * step;
      }
    }
#pragma unroll
    for (int off = 1; off < 16; off <<= 1) {
      const float up = __shfl_up_sync(0xffffffffu, cum, off, 16);
      if ((lane & 15) >= off) cum += up;
    }
    const float block_end = __shfl_sync(0xffffffffu, cum, 15, 16);
    const float e_blk = expf(cum);                    // decay from the block's start to and with the token
    const float f_blk = expf(block_end - cum) * step; // b_j times the decay from the token to its block's end
    const float through = expf(block_end);            // of the whole block
    const float through0 = __shfl_sync(0xffffffffu, through, 0), through1 = __shfl_sync(0xffffffffu, through, 16);
    fetch_dt(c0 + kChunk);
    if (!VEC || SILU) __syncthreads();                // tiles written by the CTA's threads themselves
    if (r0 >= vdim) continue;                         // (no warp of the CTA, by the launch's block size)
    // ---- 1. scores q_i . k_j (block m of 16 queries, tile n of 8 keys; rows 16 m + g, + 8; columns 8 n + 2 t, + 1; tiles
    //         above the diagonal left out) and the carried part S^T q_i: the A fragment of Q is the B fragment of Q^T
    float qk0[2][4], qk1[4][4], o[4][4];              // o: n-tile ni = tokens 8 ni .., rows r0 + g, + 8
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      qk0[0][c] = qk0[1][c] = 0.f;
#pragma unroll
      for (int n = 0; n < 4; ++n) qk1[n][c] = o[n][c] = 0.f;
    }
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) {
      uint32_t qa[2][4], kb[2][4], a0[3], a1[3], a2[3], a3[3];
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        ldsm_x4(smem_u32(sQ + (16 * m + r_a) * QS + 16 * ks + c_a), qa[m][0], qa[m][1], qa[m][2], qa[m][3]);
        ldsm_x4(smem_u32(sK + (16 * m + r_b) * QS + 16 * ks + c_b), kb[m][0], kb[m][1], kb[m][2], kb[m][3]);
      }
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const uint32_t b0 = kb[n >> 1][2 * (n & 1)], b1 = kb[n >> 1][2 * (n & 1) + 1];
        if (n < 2) mma_16816<T>(qk0[n], qa[0][0], qa[0][1], qa[0][2], qa[0][3], b0, b1);
        mma_16816<T>(qk1[n], qa[1][0], qa[1][1], qa[1][2], qa[1][3], b0, b1);
      }
      split3x2(S[2 * ks][0], S[2 * ks][1], a0);
      split3x2(S[2 * ks][2], S[2 * ks][3], a1);
      split3x2(S[2 * ks + 1][0], S[2 * ks + 1][1], a2);
      split3x2(S[2 * ks + 1][2], S[2 * ks + 1][3], a3);
#pragma unroll
      for (int p = 2; p >= 0; --p)                    // the small terms first
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          mma_16816<T>(o[2 * m], a0[p], a1[p], a2[p], a3[p], qa[m][0], qa[m][2]);
          mma_16816<T>(o[2 * m + 1], a0[p], a1[p], a2[p], a3[p], qa[m][1], qa[m][3]);
        }
    }
    // ---- 2. decayed, causal: p_ij = (j <= i) (decay from j to i) b_j (q_i . k_j)
    float cj[8], bj[8];                               // j = 8 n + 2 t, + 1
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      cj[u] = __shfl_sync(0xffffffffu, cum, 8 * (u >> 1) + 2 * t + (u & 1));
      bj[u] = __shfl_sync(0xffffffffu, step, 8 * (u >> 1) + 2 * t + (u & 1));
    }
    float f[8];                                       // f_blk of the tokens of this thread's columns
#pragma unroll
    for (int u = 0; u < 8; ++u) f[u] = __shfl_sync(0xffffffffu, f_blk, 8 * (u >> 1) + 2 * t + (u & 1));
    float ci[4], e1[2];                               // i = g, g + 8, g + 16, g + 24
#pragma unroll
    for (int u = 0; u < 4; ++u) ci[u] = __shfl_sync(0xffffffffu, cum, g + 8 * u);
#pragma unroll
    for (int u = 0; u < 2; ++u) e1[u] = __shfl_sync(0xffffffffu, e_blk, g + 16 + 8 * u);
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int u = 2 * n + (c & 1), i = g + (c >> 1) * 8, j = 8 * n + 2 * t + (c & 1);
        qk0[n][c] = j <= i ? qk0[n][c] * expf(ci[c >> 1] - cj[u]) * bj[u] : 0.f;
        qk1[n][c] *= e1[c >> 1] * f[u];               // keys of the first block, queries of the second
        qk1[2 + n][c] = j <= i ? qk1[2 + n][c] * expf(ci[2 + (c >> 1)] - cj[4 + u]) * bj[4 + u] : 0.f;
      }
    // ---- 3. o^T (rows: value channels, columns: tokens i) = e^{c_i} (S^T Q^T) + V^T P^T
    uint32_t va[2][4];                                // V^T fragment: rows r0+g / +8, k = tokens 16 b + 2t,2t+1 / 2t+8,2t+9
#pragma unroll
    for (int b = 0; b < 2; ++b)
      ldsm_x4_trans(smem_u32(sV + (16 * b + r_b) * VS + r0 + c_b), va[b][0], va[b][1], va[b][2], va[b][3]);
    const float e_i = lane < 16 ? e_blk : e_blk * through0;   // lane i: e^{c_i}
#pragma unroll
    for (int ni = 0; ni < 4; ++ni) {                  // token columns i = 8*ni + g  (B[k = j][n = i] = p_ij)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float e = __shfl_sync(0xffffffffu, e_i, 8 * ni + 2 * t + c);
        o[ni][c] *= e, o[ni][c + 2] *= e;
      }
      const int r = 2 * (ni & 1);
#pragma unroll
      for (int b = 0; b <= (ni >> 1); ++b) {
        uint32_t b0[3], b1[3];
        const float* x0 = ni < 2 ? qk0[2 * b] : qk1[2 * b];
        const float* x1 = ni < 2 ? qk0[(2 * b + 1) & 1] : qk1[2 * b + 1];
        split3x2(x0[r], x0[r + 1], b0);               // j = 16 b + 2t, 2t+1
        split3x2(x1[r], x1[r + 1], b1);               // j = 16 b + 2t+8, 2t+9
#pragma unroll
        for (int p = 2; p >= 0; --p) mma_16816<T>(o[ni], va[b][0], va[b][1], va[b][2], va[b][3], b0[p], b1[p]);
      }
    }
    // ---- 4. S^T <- e^{c_31} S^T + V'^T K,  v'_j = e^{c_31 - c_j} b_j v_j
    const float grow = through0 * through1;
    uint32_t wa[2][4][3];
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      float fb[4];                                    // j = 16 b + 2t, 2t+1, 2t+8, 2t+9
#pragma unroll
      for (int u = 0; u < 4; ++u) fb[u] = b == 0 ? f[u] * through1 : f[4 + u];
      split3x2(bits_f32(va[b][0] & 0xffffu) * fb[0], bits_f32(va[b][0] >> 16) * fb[1], wa[b][0]);
      split3x2(bits_f32(va[b][1] & 0xffffu) * fb[0], bits_f32(va[b][1] >> 16) * fb[1], wa[b][1]);
      split3x2(bits_f32(va[b][2] & 0xffffu) * fb[2], bits_f32(va[b][2] >> 16) * fb[3], wa[b][2]);
      split3x2(bits_f32(va[b][3] & 0xffffu) * fb[2], bits_f32(va[b][3] >> 16) * fb[3], wa[b][3]);
    }
#pragma unroll
    for (int n = 0; n < D / 8; n += 2) {              // B[k = token j][n = key column 8n + g] = k_j
      uint32_t kb[2][4];
#pragma unroll
      for (int b = 0; b < 2; ++b)
        ldsm_x4_trans(smem_u32(sK + (16 * b + r_a) * QS + 8 * n + c_a), kb[b][0], kb[b][1], kb[b][2], kb[b][3]);
#pragma unroll
      for (int m = 0; m < 2; ++m) {
#pragma unroll
        for (int c = 0; c < 4; ++c) S[n + m][c] *= grow;
#pragma unroll
        for (int p = 2; p >= 0; --p)
#pragma unroll
          for (int b = 0; b < 2; ++b)
            mma_16816<T>(S[n + m], wa[b][0][p], wa[b][1][p], wa[b][2][p], wa[b][3][p], kb[b][2 * m], kb[b][2 * m + 1]);
      }
    }
    // ---- 5. the chunk's output, straight from the fragments: 8 lanes write 8 neighbouring channels of a token (32 bytes)
    float* outp = P.out + tok0 * ((int64_t)P.H * vdim) + (int64_t)h * vdim;
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int i = 8 * ni + 2 * t + (c & 1), row = r0 + g + (c >> 1) * 8;
        float val = o[ni][c];
        if (MODE == 1) val += d_skip * bits_f32(sV[i * VS + row]);
        if (i < nt && row < vdim) outp[(int64_t)i * ((int64_t)P.H * vdim) + row] = val;
      }
  }
  if (slot != nullptr && r0 < vdim) {
#pragma unroll
    for (int n = 0; n < D / 8; ++n)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int row = r0 + g + (c >> 1) * 8, col = 8 * n + 2 * t + (c & 1);
        if (row < vdim && col < kdim) slot[(int64_t)col * vdim + row] = S[n][c];
      }
  }
}

// B200_CHUNK_RECURRENCE=0: every recurrence token by token
static bool recurrence_in_chunks() {
  static const bool off = [] {
    const char* e = getenv("B200_CHUNK_RECURRENCE");
    return e != nullptr && e[0] == '0';
  }();
  return !off;
}
static bool chunk_recurrence_ok(const RecParams& P, int dtype, int max_q) {
  return P.mode != 2 && dtype == B200_DTYPE_BF16 && P.cu_q != nullptr && max_q >= 16 && P.kdim <= 128 && P.vdim <= 128;
}

static int chunk_recurrence_launch(const RecParams& P, int num_seqs, cudaStream_t stream) {
  const dim3 grid(1, P.H, num_seqs);
  const dim3 block(32 * ((P.vdim + 15) / 16));
  const bool vec = P.kdim % 8 == 0 && P.vdim % 8 == 0 && P.q_stride % 8 == 0 && P.k_stride % 8 == 0 &&
                   P.v_stride % 8 == 0 && aligned16(P.q) && aligned16(P.k) && aligned16(P.v);
  // rows of V for 4 warps where the value size allows: less shared memory, and a register budget for two CTAs per SM (of 8
  // warps: one). Twice as many (at 128 registers, with some spilled) where there are that many and the state is small: what
  // counts then is how many states are on their way. 32 heads of 64 x 64, two / four: 256 prompts of 16 tokens 168 / 125 us, 16 of
  // 1024 260 / 239, 64 of 40 73.6 / 59.9; 4 of 100 14.7 / 17.5, 1 of 700 69 / 84.
  const bool many = (int64_t)P.H * num_seqs > (P.vdim <= 64 ? 2 : 1) * 148;
#define B200_CHUNK_REC_AT(DV, NW, VEC, M, SILU, CTAS)                                                               \
  do {                                                                                                              \
    auto kern = chunk_recurrence_kernel<DV, NW, VEC, M, SILU, CTAS>;                                                \
    constexpr int smem = chunk_recurrence_smem<DV, NW>(VEC);                                                        \
    static std::atomic<uint64_t> devices{0};                                                                        \
    const cudaError_t allowed = allow_smem(kern, smem, devices);                                                    \
    if (allowed != cudaSuccess) return (int)allowed;                                                                \
    launch_pdl(kern, grid, block, (size_t)smem, stream, P);                                                         \
  } while (0)
#define B200_CHUNK_REC_AS(DV, NW, VEC, M, SILU)                                            \
  do {                                                                                     \
    if (DV <= 64 && many) B200_CHUNK_REC_AT(DV, NW, VEC, M, SILU, (DV <= 64 ? 4 : 2));     \
    else B200_CHUNK_REC_AT(DV, NW, VEC, M, SILU, 2);                                       \
  } while (0)
#define B200_CHUNK_REC_V(DV, M, SILU)                                           \
  do {                                                                          \
    if (P.vdim <= 64 && vec) B200_CHUNK_REC_AS(DV, 4, true, M, SILU);           \
    else if (P.vdim <= 64) B200_CHUNK_REC_AS(DV, 4, false, M, SILU);            \
    else if (vec) B200_CHUNK_REC_AS(DV, 8, true, M, SILU);                      \
    else B200_CHUNK_REC_AS(DV, 8, false, M, SILU);                              \
  } while (0)
#define B200_CHUNK_REC(DV)                                             \
  do {                                                                 \
    if (P.mode == 1 && P.act_silu) B200_CHUNK_REC_V(DV, 1, true);      \
    else if (P.mode == 1) B200_CHUNK_REC_V(DV, 1, false);              \
    else if (P.act_silu) B200_CHUNK_REC_V(DV, 0, true);                \
    else B200_CHUNK_REC_V(DV, 0, false);                               \
  } while (0)
  if (P.kdim <= 32) B200_CHUNK_REC(32);
  else if (P.kdim <= 64) B200_CHUNK_REC(64);
  else B200_CHUNK_REC(128);
#undef B200_CHUNK_REC
#undef B200_CHUNK_REC_V
#undef B200_CHUNK_REC_AS
#undef B200_CHUNK_REC_AT
  return finish_launch();
}

template <typename T, typename TV = T>
static int recurrence_launch(const RecParams& P, int num_seqs, cudaStream_t stream) {
  if (P.kdim <= 16) recurrence_launch_as<T, TV, 16, 1>(P, num_seqs, stream);
  else if (P.kdim <= 32) recurrence_launch_as<T, TV, 32, 1>(P, num_seqs, stream);
  else if (P.kdim <= 64) recurrence_launch_as<T, TV, 64, 1>(P, num_seqs, stream);
  else if (P.kdim <= 128) recurrence_launch_as<T, TV, 64, 2>(P, num_seqs, stream);
  else recurrence_launch_as<T, TV, 64, 4>(P, num_seqs, stream);
  return finish_launch();
}

}  // namespace b200

using namespace b200;

extern "C" int b200_attn_generic_bounded(void* out, const void* q, int64_t q_stride, const void* k, int64_t k_stride,
                                 const void* v, int64_t v_stride, const int32_t* block_tables,
                                 int32_t bt_stride, int32_t block_size, const int32_t* cu_q,
                                 const int32_t* cu_k, const int32_t* ctx_lens, int32_t num_seqs, int32_t max_q,
                                 int32_t num_heads, int32_t num_kv_heads, int32_t dim, int32_t vdim,
                                 float scale, int32_t window, int32_t keep_first, int32_t chunk, float softcap,
                                 const float* sink, const void* gate, int64_t gate_stride, int32_t dtype, int64_t total_q, int64_t wait_ns,
                                 b200_stream_t stream) {
  B200_RETURN_IF(wait_ns < 0, B200_ERR_BAD_SHAPE);
  B200_RETURN_IF(num_seqs < 0 || max_q < 0 || num_heads <= 0 || num_kv_heads <= 0 || dim <= 0 || vdim <= 0 ||
                     num_heads % num_kv_heads != 0, B200_ERR_BAD_SHAPE);
  B200_RETURN_IF(vdim > 32 * kAttnMaxVChunks, B200_ERR_UNSUPPORTED);
  if (num_seqs == 0 || max_q == 0) return B200_OK;
  B200_RETURN_IF(!out || !q || !k || (cu_q == nullptr) == (ctx_lens == nullptr) || (cu_q && !cu_k),
                 B200_ERR_NULL_POINTER);
  B200_RETURN_IF(block_tables && block_size <= 0, B200_ERR_BAD_SHAPE);
  B200_RETURN_IF(window < 0 || keep_first < 0 || chunk < 0 || (window > 0 && chunk > 0) || (!v && vdim > dim), B200_ERR_BAD_SHAPE);
  B200_RETURN_IF(!block_tables && !cu_q, B200_ERR_NULL_POINTER);       // decode rows read the paged cache
  const int rep = num_heads / num_kv_heads;
  if (cu_q && attn_tiled_fits(max_q, rep, num_kv_heads, num_seqs, dim, vdim)) {              // prompt portions: 64 rows share every key tile
    AttnTiledParams A;
    A.out = out, A.q = q, A.k = k, A.v = v, A.q_stride = q_stride, A.k_stride = k_stride, A.v_stride = v_stride;
    A.block_tables = block_tables, A.bt_stride = bt_stride, A.block_size = block_size, A.cu_q = cu_q, A.cu_k = cu_k;
    A.H = num_heads, A.G = num_kv_heads, A.dim = dim, A.vdim = vdim, A.scale = scale, A.window = window;
    A.keep_first = keep_first, A.chunk = chunk, A.softcap = softcap, A.sink = sink, A.gate = gate, A.gate_stride = gate_stride;
    if (attn_split_fits(A, num_seqs, max_q, total_q, dtype)) return attn_split_launch(A, num_seqs, max_q, total_q, wait_ns, (cudaStream_t)stream);
    return attn_tiled_launch(A, num_seqs, max_q, dtype, (cudaStream_t)stream);
  }
  const dim3 grid((max_q * rep + kAttnRows - 1) / kAttnRows, num_kv_heads, num_seqs);
  const size_t smem = (size_t)(kAttnRows * dim + kAttnKeys * (dim + 1) + (v ? kAttnKeys * vdim : 0)) * sizeof(float);
  B200_RETURN_IF(smem > 200 * 1024, B200_ERR_UNSUPPORTED);
  B200_DISPATCH_3(dtype, T, {
    if (smem > 48 * 1024)
      cudaFuncSetAttribute(attn_generic_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    launch_pdl(attn_generic_kernel<T>, grid, dim3(kAttnRows * 32), smem, (cudaStream_t)stream, (T*)out,
               (const T*)q, q_stride, (const T*)k, k_stride, (const T*)v, v_stride, block_tables, bt_stride,
               block_size, cu_q, cu_k, ctx_lens, num_heads, num_kv_heads, dim, vdim, scale, window, keep_first, chunk,
               softcap, sink, (const T*)gate, gate_stride);
  });
  return finish_launch();
}

extern "C" int b200_attn_generic_step(void* out, const void* q, int64_t q_stride, const void* k, int64_t k_stride,
                                 const void* v, int64_t v_stride, const int32_t* block_tables,
                                 int32_t bt_stride, int32_t block_size, const int32_t* cu_q,
                                 const int32_t* cu_k, const int32_t* ctx_lens, int32_t num_seqs, int32_t max_q,
                                 int32_t num_heads, int32_t num_kv_heads, int32_t dim, int32_t vdim,
                                 float scale, int32_t window, int32_t keep_first, int32_t chunk, float softcap,
                                 const float* sink, const void* gate, int64_t gate_stride, int32_t dtype, int64_t total_q, b200_stream_t stream) {
  return b200_attn_generic_bounded(out, q, q_stride, k, k_stride, v, v_stride, block_tables, bt_stride, block_size, cu_q, cu_k,
          ctx_lens, num_seqs, max_q, num_heads, num_kv_heads, dim, vdim, scale, window, keep_first, chunk, softcap, sink, gate,
          gate_stride, dtype, total_q, kWaitNs, stream);
}

extern "C" int b200_attn_generic(void* out, const void* q, int64_t q_stride, const void* k, int64_t k_stride,
                                 const void* v, int64_t v_stride, const int32_t* block_tables,
                                 int32_t bt_stride, int32_t block_size, const int32_t* cu_q,
                                 const int32_t* cu_k, const int32_t* ctx_lens, int32_t num_seqs, int32_t max_q,
                                 int32_t num_heads, int32_t num_kv_heads, int32_t dim, int32_t vdim,
                                 float scale, int32_t window, int32_t keep_first, int32_t chunk, float softcap,
                                 const float* sink, const void* gate, int64_t gate_stride, int32_t dtype, b200_stream_t stream) {
  return b200_attn_generic_step(out, q, q_stride, k, k_stride, v, v_stride, block_tables, bt_stride, block_size, cu_q, cu_k, ctx_lens, num_seqs, max_q, num_heads, num_kv_heads, dim, vdim, scale, window, keep_first, chunk, softcap, sink, gate, gate_stride, dtype, 0, stream);
}

extern "C" int b200_linear_recurrence_bounded(float* out, const void* q, int64_t q_stride, const void* k,
                                      int64_t k_stride, const void* v, int64_t v_stride, float* state,
                                      const int32_t* state_slots, const int32_t* cu_q, const int32_t* cu_k,
                                      const int32_t* ctx_lens, int32_t num_seqs, int32_t max_q,
                                      int32_t num_heads, int32_t groups, int32_t kdim, int32_t vdim, int32_t mode,
                                      int32_t act_silu, const float* decay, const void* dt, int64_t dt_stride,
                                      const float* dt_bias, const float* a_log, const float* d_skip,
                                      int32_t qk_f32, int32_t dtype, int64_t total_q, int64_t wait_ns,
                                 b200_stream_t stream) {
  B200_RETURN_IF(wait_ns < 0, B200_ERR_BAD_SHAPE);
  B200_RETURN_IF(num_seqs < 0 || num_heads <= 0 || groups <= 0 || num_heads % groups != 0 || kdim <= 0 ||
                     vdim <= 0 || mode < 0 || mode > 2, B200_ERR_BAD_SHAPE);
  B200_RETURN_IF(kdim > 256, B200_ERR_UNSUPPORTED);
  if (num_seqs == 0) return B200_OK;
  B200_RETURN_IF(!out || !q || !k || !v || (cu_q == nullptr) == (ctx_lens == nullptr) || (cu_q && !cu_k) ||
                     (state && !state_slots), B200_ERR_NULL_POINTER);
  B200_RETURN_IF(mode == 0 ? !decay : (mode == 1 && (!dt || !dt_bias || !a_log || !d_skip)), B200_ERR_NULL_POINTER);
  B200_RETURN_IF(mode == 2 && !qk_f32 && dtype != B200_DTYPE_F32, B200_ERR_BAD_DTYPE);   // the gate is fp32
  RecParams P;
  P.q = q, P.k = k, P.v = v, P.q_stride = q_stride, P.k_stride = k_stride, P.v_stride = v_stride;
  P.out = out, P.state = state, P.state_slots = state_slots, P.cu_q = cu_q, P.cu_k = cu_k, P.ctx_lens = ctx_lens;
  P.H = num_heads, P.groups = groups, P.kdim = kdim, P.vdim = vdim, P.mode = mode, P.act_silu = act_silu;
  P.decay = decay, P.dt = dt, P.dt_stride = dt_stride, P.dt_bias = dt_bias, P.a_log = a_log, P.d_skip = d_skip;
  if (qk_f32 && dtype != B200_DTYPE_F32) {           // q, k already fp32 (rotated or normalised upstream), v as projected
    B200_RETURN_IF(mode == 1, B200_ERR_UNSUPPORTED);
    if (dtype == B200_DTYPE_BF16) return recurrence_launch<float, __nv_bfloat16>(P, num_seqs, (cudaStream_t)stream);
    if (dtype == B200_DTYPE_F16) return recurrence_launch<float, __half>(P, num_seqs, (cudaStream_t)stream);
    return B200_ERR_BAD_DTYPE;
  }
  if (recurrence_in_chunks()) {
    if (recurrence_umma_ok(P, dtype, num_seqs, max_q, total_q)) return recurrence_umma_launch(P, num_seqs, wait_ns, (cudaStream_t)stream);
    if (chunk_recurrence_ok(P, dtype, max_q)) return chunk_recurrence_launch(P, num_seqs, (cudaStream_t)stream);
  }
  B200_DISPATCH_3(dtype, T, return recurrence_launch<T>(P, num_seqs, (cudaStream_t)stream));
  return B200_OK;
}

extern "C" int b200_linear_recurrence_step(float* out, const void* q, int64_t q_stride, const void* k,
                                      int64_t k_stride, const void* v, int64_t v_stride, float* state,
                                      const int32_t* state_slots, const int32_t* cu_q, const int32_t* cu_k,
                                      const int32_t* ctx_lens, int32_t num_seqs, int32_t max_q,
                                      int32_t num_heads, int32_t groups, int32_t kdim, int32_t vdim, int32_t mode,
                                      int32_t act_silu, const float* decay, const void* dt, int64_t dt_stride,
                                      const float* dt_bias, const float* a_log, const float* d_skip,
                                      int32_t qk_f32, int32_t dtype, int64_t total_q, b200_stream_t stream) {
  return b200_linear_recurrence_bounded(out, q, q_stride, k, k_stride, v, v_stride, state, state_slots, cu_q, cu_k, ctx_lens,
          num_seqs, max_q, num_heads, groups, kdim, vdim, mode, act_silu, decay, dt, dt_stride, dt_bias, a_log, d_skip, qk_f32,
          dtype, total_q, kWaitNs, stream);
}

extern "C" int b200_linear_recurrence(float* out, const void* q, int64_t q_stride, const void* k,
                                      int64_t k_stride, const void* v, int64_t v_stride, float* state,
                                      const int32_t* state_slots, const int32_t* cu_q, const int32_t* cu_k,
                                      const int32_t* ctx_lens, int32_t num_seqs, int32_t max_q,
                                      int32_t num_heads, int32_t groups, int32_t kdim, int32_t vdim, int32_t mode,
                                      int32_t act_silu, const float* decay, const void* dt, int64_t dt_stride,
                                      const float* dt_bias, const float* a_log, const float* d_skip,
                                      int32_t qk_f32, int32_t dtype, b200_stream_t stream) {
  return b200_linear_recurrence_step(out, q, q_stride, k, k_stride, v, v_stride, state, state_slots, cu_q, cu_k, ctx_lens, num_seqs, max_q, num_heads, groups, kdim, vdim, mode, act_silu, decay, dt, dt_stride, dt_bias, a_log, d_skip, qk_f32, dtype, 0, stream);
}
