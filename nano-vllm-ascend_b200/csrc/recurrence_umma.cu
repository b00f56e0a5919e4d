// recurrence_umma.cu -- linear_recurrence (seq_mixers.cu) over prompts on the 5th-generation tensor cores, 64 tokens at a time.
//
// The mathematics is that of chunk_recurrence_kernel: bf16 tokens, an fp32 state that is split into three bf16 terms (24 bits)
// wherever it is an operand, decays that are exponentials of sums over at most 16 tokens and multiplied up beyond. Per chunk of 64
// tokens t and a CTA's 128 value channels c (two neighbouring heads of 64 that share q and k, or one head of 128):
//   SC[t, j]    = q_t . k_j                                exact operands              M128 (rows 64.. unused) N64 K = D
//   P[t, j]     = SC decay(j -> t) b_j, j <= t             registers -> three terms in shared memory
//   O2^T[c, t]  = sum_j x_j[c] P[t, j]                     3 products, for each head   M128 (half of the lanes written) N64 K64
//   O1^T[c, t]  = sum_n S[n, c] q_t[n]                     3 products, S from TMEM     M128 N64 K = D
//   dS^T[c, n]  = sum_t (decay(t -> end) b_t x_t[c]) k_t[n]  3 products                M128 N = D K64
//   S <- decay(chunk) S + dS;  o_t = decay(start -> t) O1 + O2                         fp32 registers, one rounding each
// with the products of the small terms accumulated first. S itself never is an accumulator: the tensor core adds up one chunk,
// the registers add chunks.
//
// What bounds it: the tensor pipe and its issue (D 128, two heads: SC 8 MMAs, O1 24, O2 24 of 64 columns, dS 12 of 128: 5500 of the
// 6400 cycles a chunk takes), as long as no chain is longer: load -> scaled values -> dS, SC -> P -> O2, S -> terms -> O1. So the
// order of issue is O2(i) | SC(i+1) | O1(i) | dS(i+1): the score warps work under O1 and dS, the state warps store outputs under
// dS(i+1) and turn S(i) into terms under O2(i+1), k and x come two chunks ahead. What also counts is code size: 24 warps of six
// roles run through their code once per chunk, and with everything unrolled (164 KB) instruction fetches took three quarters of
// the time (16 x 1024 tokens, 32 heads of 128 x 64: 265 us; 190 with short loops; 135 with the roles spread over 24 warps; 132 with an add per
// operand and MMA).
// Measured there (ten calls in a graph; 5 us more where the inputs change from call to call): 329 us (chunk_recurrence_kernel, mma.sync,
// chunks of 32) -> 132, 133 with the look at the values (see below); 8 heads of 128 x 128 195 -> 114; errors against 64 bits 2.1e-7 (2.5e-7).
// Warps: 0-7 state and outputs (a warp: 32 channels x half of the keys, then half of the tokens; D / 2 state registers a thread);
// 8, 9 and 12, 13 P of a head's diagonal blocks, 17 and 21 of the others (only warps w with w % 4 < 2 may read TMEM lanes 0-63);
// 10, 11, 14, 15 the scaled values; 16 issues; 20 decays; 18, 19 copy k and x, 22, 23 q. With one head of 128, 12 and 13 copy too.
// TMEM: dS 128 columns, S terms 192, O1 64, O2 64 (both heads: MMAs that write half of the lanes), SC 64. Shared memory: q, k two
// stages, x three (its last reader is O2), P and the scaled values one.
//
// A value x that is not finite must not reach the tokens before it (0 x inf): the warps that scale the values put a zero in its place,
// and the outputs of its channel from its token on are NaN (the state takes the value itself).
//
// Waits are bounded (mbar_warp_wait): one that runs out makes its role leave its loop, those that wait for that role run out as well, the
// products under way are waited for, the CTA sets the host's word and the library reports it.
#include <type_traits>

#include "recurrence.cuh"
#include "umma.cuh"

namespace b200 {

constexpr int kRuL = 64;                               // tokens per chunk
constexpr int kRuThreads = 768;
constexpr int kRuPanel = 64 * 128;                     // bytes of 64 rows x 64 elements
constexpr int kRuDec = 4;                              // stages of the decays

struct RuDecay {                                       // of one head and chunk; a block is 16 tokens
  float cum[kRuL];                                     // log decay from the block's start to and with the token
  float step[kRuL];                                    // b
  float head[kRuL];                                    // e^cum
  float tail[kRuL];                                    // decay from the token to its block's end, times b
  float from_start[kRuL];                              // decay from the chunk's start to and with the token
  float to_end[kRuL];                                  // decay from the token to the chunk's end, times b
  float block[4];                                      // decay of a whole block
  float all;                                           // of the chunk
  float pad[3];
};

struct RuParams {
  RecParams r;
  int wait_tries;                                      // of one wait
  int* wait_status;
};

template <int D, int NH>
constexpr int ru_smem() {
  return 1024 + 2 * 2 * (D / 64) * kRuPanel + 3 * 2 * kRuPanel + 3 * NH * kRuPanel + 3 * 2 * kRuPanel + kRuDec * NH * (int)sizeof(RuDecay) + 256;
}

template <int D, int NH, int MODE, bool SILU>
__global__ void __launch_bounds__(kRuThreads, 1)
recurrence_umma_kernel(const __grid_constant__ RuParams RP) {
  using T = __nv_bfloat16;
  const RecParams& P = RP.r;
  constexpr int VD = 128 / NH;                          // value channels per head
  constexpr int CP = D / 64;                            // panels of a q or k tile
  constexpr int kQK = CP * kRuPanel;
  constexpr uint32_t kTmD = 0, kTmS = 128, kTmO1 = 320, kTmO2 = 384, kTmSC = 448;
  extern __shared__ __align__(1024) uint8_t ru_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(ru_smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                                   // [2][CP panels][64 tokens]
  uint8_t* sK = sQ + 2 * kQK;                           // [2]
  uint8_t* sX = sK + 2 * kQK;                           // [3][2 panels of 64 channels][64 tokens]
  uint8_t* sP = sX + 3 * 2 * kRuPanel;                  // [3 terms][NH * 64 rows t][64 j]
  uint8_t* sW = sP + 3 * NH * kRuPanel;                 // [3 terms][2 panels][64 tokens]
  RuDecay* s_dec = reinterpret_cast<RuDecay*>(sW + 3 * 2 * kRuPanel);      // [kRuDec][NH]
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_dec + kRuDec * NH);
  uint64_t *k_full = bars, *k_empty = bars + 2, *q_full = bars + 23, *q_empty = bars + 25, *dec_full = bars + 4, *dec_empty = bars + 8, *sc_full = bars + 12,
           *sc_read = bars + 13, *p_ready = bars + 14, *w_ready = bars + 15, *d_done = bars + 16, *d_read = bars + 17,
           *s_ready = bars + 18, *o1_done = bars + 19, *o2_done = bars + 20, *o_read = bars + 21, *drained = bars + 22;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 27);
  volatile int *gave_up = reinterpret_cast<volatile int*>(tmem_slot + 1), *odd = gave_up + 1;

  pdl_wait();
  const int s = blockIdx.y, h0 = blockIdx.x * NH;
  const SeqSpan sp = seq_span(P.cu_q, P.cu_k, P.ctx_lens, s);
  if (sp.q_len == 0) return;
  const int kdim = P.kdim, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = h0 / (P.H / P.groups);
  const T* q = (const T*)P.q + (int64_t)grp * kdim;
  const T* k = (const T*)P.k + (int64_t)grp * kdim;
  const T* v = (const T*)P.v + (int64_t)h0 * VD;
  const T* dt = (const T*)P.dt;
  float* out = P.out + (int64_t)h0 * VD;
  const int64_t out_stride = (int64_t)P.H * VD;
  // state of channel c: head h0 + c / VD, column c % VD
  float* slot = P.state != nullptr ? P.state + ((int64_t)P.state_slots[s] * P.H + h0) * kdim * (int64_t)VD : nullptr;
  const bool carried = slot != nullptr && sp.first_pos() > 0;

  if (sp.q_len == 1) {
    // A single token (a decode row of a mixed step) is a rank-1 update: one pass over the state in the order it lies in memory.
    // Thread = channel x a quarter of the key rows.
    float* sq = reinterpret_cast<float*>(smem);         // [D] q, [D] k, [4][128] partial outputs
    float *sk = sq + D, *so = sk + D;
    const int64_t tok = sp.q_start;
    for (int i = threadIdx.x; i < kdim; i += kRuThreads) {
      float qv = __bfloat162float(q[tok * P.q_stride + i]), kv = __bfloat162float(k[tok * P.k_stride + i]);
      if (SILU) qv = bits_f32(bf16_bits(silu_fast(qv))), kv = bits_f32(bf16_bits(silu_fast(kv)));
      sq[i] = qv, sk[i] = kv;
    }
    const int c = threadIdx.x & 127, part = threadIdx.x >> 7, h = h0 + c / VD;
    float x = __bfloat162float(v[tok * P.v_stride + c]), a = MODE == 0 ? P.decay[h] : 0.f, step = 1.f;
    if (SILU) x = bits_f32(bf16_bits(silu_fast(x)));
    if (MODE == 1) {
      step = softplus_f(__bfloat162float(dt[tok * P.dt_stride + h]) + P.dt_bias[h]);
      a = expf(-expf(P.a_log[h]) * step);
    }
    __syncthreads();
    const float bx = step * x;
    const int64_t at = (int64_t)(c / VD) * kdim * VD + c % VD;
    const int per = (kdim + 3) / 4, k_lo = part * per, k_hi = part < 4 ? min(kdim, k_lo + per) : 0;
    float sum = 0.f;
    for (int i0 = k_lo; i0 < k_hi; i0 += 16) {
      float row[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) row[i] = carried && i0 + i < k_hi ? slot[at + (int64_t)(i0 + i) * VD] : 0.f;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        if (i0 + i >= k_hi) break;
        row[i] = fmaf(sk[i0 + i], bx, a * row[i]);
        if (slot != nullptr) slot[at + (int64_t)(i0 + i) * VD] = row[i];
        sum = fmaf(sq[i0 + i], row[i], sum);
      }
    }
    if (part < 4) so[part * 128 + c] = sum;
    __syncthreads();
    if (part == 0) {
      sum = (so[c] + so[128 + c]) + (so[256 + c] + so[384 + c]);
      if (MODE == 1) sum = fmaf(P.d_skip[h], x, sum);
      out[tok * out_stride + c] = sum;
    }
    return;
  }

  constexpr int kCopyK = NH == 1 ? 128 : 64, kCopyQ = 64;      // threads that copy k and x, and q
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) mbar_init(&k_full[i], kCopyK), mbar_init(&k_empty[i], 1), mbar_init(&q_full[i], kCopyQ), mbar_init(&q_empty[i], 1);
    for (int i = 0; i < kRuDec; ++i) mbar_init(&dec_full[i], 32), mbar_init(&dec_empty[i], 256);
    mbar_init(sc_full, 1), mbar_init(sc_read, NH * 96), mbar_init(p_ready, NH * 96), mbar_init(w_ready, 128);
    mbar_init(d_done, 1), mbar_init(d_read, 256), mbar_init(s_ready, 256);
    mbar_init(o1_done, 1), mbar_init(o2_done, 1), mbar_init(o_read, 256);
    mbar_init(drained, 1);
    mbar_fence_init();
    *gave_up = 0, *odd = 0;
  }
  if (warp == 16) umma::tmem_alloc(tmem_slot, 512);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  constexpr uint32_t tb = 0;                            // all 512 columns: they start at 0
  const int chunks = (sp.q_len + kRuL - 1) / kRuL;
  auto wait = [&](uint64_t* bar, int parity) { return mbar_warp_wait(bar, parity & 1, RP.wait_tries, gave_up); };
  // Copies: k and x of chunk j (kQ false) once the products of chunk j - 2 that read them have retired, or q; thread li of kThreads
  auto copies = [&](auto is_q, auto threads, int li) {
    constexpr bool kQ = decltype(is_q)::value;
    constexpr int kThreads = decltype(threads)::value;
    uint64_t *full = kQ ? q_full : k_full, *empty = kQ ? q_empty : k_empty;
    const int come = RP.wait_tries > 0 ? chunks : min(chunks, 2);     // (a limit of 0 tests the way out: nothing comes any more)
    for (int j = 0; j < come; ++j) {
      if (j >= 2 && !wait(&empty[j & 1], (j >> 1) - 1)) break;
      const int nt = min(kRuL, sp.q_len - j * kRuL);
      const int64_t tok0 = sp.q_start + j * kRuL;
      uint8_t *tk = (kQ ? sQ : sK) + (j & 1) * kQK, *tx = sX + (j % 3) * 2 * kRuPanel;
      // a thread's 16-byte column is the same in all of its rows
      auto each = [&](auto cols, auto f) {
        constexpr int C = decltype(cols)::value;       // 16-byte columns of a row
        const int cc = li % C;
        const uint32_t at = (cc >> 3) * kRuPanel;
#pragma unroll 2
        for (int row = li / C; row < kRuL; row += kThreads / C) f(row, cc, at + umma::sw128(row, cc & 7));
      };
      auto copy = [&](uint8_t* dst, const T* src, int64_t stride, auto cols, int width) {
        const uint32_t to = smem_u32(dst);
        each(cols, [&](int row, int cc, uint32_t at) {
          const bool ok = cc * 8 < width && row < nt;
          cp_async_16(to + at, ok ? src + (tok0 + row) * stride + cc * 8 : src, ok);
        });
      };
      auto activate = [&](uint8_t* dst, auto cols) {   // every thread what it copied
        each(cols, [&](int, int, uint32_t at) {
          T* p = reinterpret_cast<T*>(dst + at);
          float f[8];
          load8<T>(p, f);
#pragma unroll
          for (int u = 0; u < 8; ++u) f[u] = silu_fast(f[u]);
          store8<T>(p, f);
        });
      };
      constexpr std::integral_constant<int, D / 8> qk_cols{};
      constexpr std::integral_constant<int, 16> x_cols{};
      if (!kQ) copy(tx, v, P.v_stride, x_cols, 128);
      copy(tk, kQ ? q : k, kQ ? P.q_stride : P.k_stride, qk_cols, kdim);
      cp_async_commit();
      cp_async_wait<0>();
      if (SILU) {
        if (!kQ) activate(tx, x_cols);
        activate(tk, qk_cols);
      }
      fence_proxy_async_smem();
      mbar_arrive(&full[j & 1]);
    }
    cp_async_wait<0>();
  };
  auto store_p = [&](int row, int c16, const uint32_t (&y)[4][3]) {      // 8 columns of a row of P
#pragma unroll
    for (int p = 0; p < 3; ++p)
      *reinterpret_cast<uint4*>(sP + p * NH * kRuPanel + umma::sw128(row, c16)) = make_uint4(y[0][p], y[1][p], y[2][p], y[3][p]);
  };
  // Registers: 768 x 80 at launch = 256 x 112 (state) + 256 x 72 + 256 x 56
  if (warp < 8) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
    // =========================== state and outputs ===========================
    const int quarter = warp & 3, half = warp >> 2, c = quarter * 32 + lane, hh = NH == 2 ? quarter >> 1 : 0;
    const uint32_t base = tb + ((uint32_t)(quarter * 32) << 16);
    float S[D / 2];                                     // S[n][c], n = half * D / 2 + i
    float* mine = slot + (int64_t)hh * kdim * VD + c % VD;
    const int rows = min(D / 2, kdim - half * (D / 2)); // of this warp that exist
    mine += (int64_t)half * (D / 2) * VD;
#pragma unroll
    for (int i = 0; i < D / 2; ++i) S[i] = 0.f;
    if (carried) {
#pragma unroll
      for (int i = 0; i < D / 2; ++i) {
        if (i < rows) S[i] = mine[i * VD];
        if (i % 16 == 15) asm volatile("" ::: "memory");      // 16 on their way, no more registers
      }
    }
    for (int j = 0;; ++j) {                             // the terms of S(j - 1), for chunk j; the outputs of chunk j - 1
      const int d = j - 1;
      const RuDecay& dec = s_dec[(d & (kRuDec - 1)) * NH + hh];
      if (j > 0) {
        if (!wait(&dec_full[d & (kRuDec - 1)], d / kRuDec) || !wait(d_done, d)) break;
        umma::fence_after_sync();
        const float all = dec.all;
#pragma unroll
        for (int i0 = 0; i0 < D / 2; i0 += 16) {
          uint32_t w[16];
          umma::ld16(base + kTmD + half * (D / 2) + i0, w);
          umma::wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) S[i0 + i] = fmaf(all, S[i0 + i], __uint_as_float(w[i]));
        }
        umma::fence_before_sync();
        mbar_arrive(d_read);
        if (!wait(o1_done, d)) break;                   // the outputs of chunk d; the terms of the state before it are consumed
        umma::fence_after_sync();
        const int t0 = d * kRuL + half * 32;              // this warp's 32 tokens: a warp writes 128 bytes of each
        float* to = out + (sp.q_start + t0) * out_stride + c;
        const int left = sp.q_len - t0;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          uint32_t o1[16], o2[16];
          umma::ld16(base + kTmO1 + half * 32 + 16 * u, o1);
          umma::ld16(base + kTmO2 + half * 32 + 16 * u, o2);
          umma::wait_ld();
          if (u == 1) {
            umma::fence_before_sync();
            mbar_arrive(o_read);
          }
          const float* e = &dec.from_start[half * 32 + 16 * u];
          if (left >= 32) {                               // (stores under a predicate each took three times as long)
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
              const float4 e4 = *reinterpret_cast<const float4*>(e + i);
              const float ee[4] = {e4.x, e4.y, e4.z, e4.w};
#pragma unroll
              for (int x = 0; x < 4; ++x, to += out_stride) *to = fmaf(ee[x], __uint_as_float(o1[i + x]), __uint_as_float(o2[i + x]));
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i, to += out_stride)
              if (16 * u + i < left) *to = fmaf(e[i], __uint_as_float(o1[i]), __uint_as_float(o2[i]));
          }
        }
        mbar_arrive(&dec_empty[d & (kRuDec - 1)]);
      }
      if (j == chunks) break;
      // as the A operand: packed pairs along n
#pragma unroll
      for (int i0 = 0; i0 < D / 2; i0 += 16) {
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
      mbar_arrive(s_ready);
    }
    if (slot != nullptr) {
#pragma unroll
      for (int i = 0; i < D / 2; ++i)
        if (i < rows) mine[i * VD] = S[i];
    }
    if (*odd) {                                         // a value that is not finite: from its token on (beyond the chunk it is all NaN)
      int first = sp.q_len;
      for (int t = (*odd - 1) * kRuL; t < sp.q_len && first == sp.q_len; t += 16)
#pragma unroll
        for (int i = 15; i >= 0; --i) {                 // 16 on their way
          const float x = t + i < sp.q_len ? __bfloat162float(v[(sp.q_start + t + i) * P.v_stride + c]) : 0.f;
          if (!isfinite(SILU ? silu_fast(x) : x)) first = t + i;
        }
      for (int t = first; t < min(sp.q_len, (first / kRuL + 1) * kRuL); ++t)
        if ((t & 32) == 32 * half) out[(sp.q_start + t) * out_stride + c] = NAN;
    }
  } else if (warp < 16) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    const int wq = warp & 3, wg = (warp - 8) >> 2;
    if (wq >= 2) {
      // =========================== scaled values ===========================
      const int wi = (wg * 2 + wq - 2) * 32 + lane;     // 0 .. 127
      for (int j = 0; j < chunks; ++j) {
        const RuDecay* dec = s_dec + (j & (kRuDec - 1)) * NH;
        if (!wait(&dec_full[j & (kRuDec - 1)], j / kRuDec) || !wait(&k_full[j & 1], j >> 1)) break;
        if (j > 0 && !wait(d_done, j - 1)) break;       // the last chunk's are consumed
        uint8_t* x = sX + (j % 3) * 2 * kRuPanel;
        uint32_t seen = 0;                              // the largest magnitude of either half
#pragma unroll 1
        for (int e0 = 0; e0 < 8; ++e0) {
          const int e = e0 * 128 + wi, row = e >> 4, panel = (e >> 3) & 1;
          const uint32_t at = panel * kRuPanel + umma::sw128(row, e & 7);
          const uint4 u = *reinterpret_cast<const uint4*>(x + at);
          seen = __vimax3_u16x2(seen, u.x & 0x7fff7fffu, u.y & 0x7fff7fffu);
          seen = __vimax3_u16x2(seen, u.z & 0x7fff7fffu, u.w & 0x7fff7fffu);
          const float w = dec[NH == 2 ? panel : 0].to_end[row];
          const uint32_t in[4] = {u.x, u.y, u.z, u.w};
          uint32_t y[4][3];
#pragma unroll
          for (int i = 0; i < 4; ++i) split3cut(w * __uint_as_float(in[i] << 16), w * __uint_as_float(in[i] & 0xffff0000u), y[i]);
#pragma unroll
          for (int p = 0; p < 3; ++p)
            *reinterpret_cast<uint4*>(sW + p * 2 * kRuPanel + at) = make_uint4(y[0][p], y[1][p], y[2][p], y[3][p]);
        }
        if ((seen & 0xffffu) >= 0x7f80u || seen >= 0x7f800000u) {      // the tokens before see zero instead (0 x inf), see the outputs
          if (*odd == 0) *odd = j + 1;                  // the first chunk that has one
#pragma unroll 1
          for (int e = wi; e < 1024; e += 128) {
            uint16_t* h = reinterpret_cast<uint16_t*>(x + ((e >> 3) & 1) * kRuPanel + umma::sw128(e >> 4, e & 7));
            for (int i = 0; i < 8; ++i)
              if ((h[i] & 0x7f80u) == 0x7f80u) h[i] = 0;
          }
        }
        fence_proxy_async_smem();
        mbar_arrive(w_ready);
      }
    } else if (wg >= NH) {
      copies(std::false_type{}, std::integral_constant<int, kCopyK>{}, (2 + wq) * 32 + lane);
    } else {
      // =========================== scores, the diagonal's 32 x 32 ===========================
      // thread = row t = 32 wq + lane of head h0 + wg: blocks 2 wq (lanes 0-15: their own) and 2 wq + 1
      const uint32_t base = tb + ((uint32_t)(wq * 32) << 16) + kTmSC + 32 * wq;
      const float d_skip = MODE == 1 ? P.d_skip[h0 + wg] : 0.f;
      const bool hi = lane >= 16;
      const int t = 32 * wq + lane, row = wg * 64 + t;
      if (wq == 0) {                                    // nothing of the last 32 columns is seen
        const uint32_t zero[4][3] = {};
        for (int c16 = 4; c16 < 8; ++c16) store_p(row, c16, zero);
      }
      for (int j = 0; j < chunks; ++j) {
        const RuDecay& dec = s_dec[(j & (kRuDec - 1)) * NH + wg];
        if (!wait(&dec_full[j & (kRuDec - 1)], j / kRuDec) || !wait(sc_full, j)) break;
        umma::fence_after_sync();
        if (j > 0 && !wait(o2_done, j - 1)) break;      // the last chunk's P is consumed
        const float cum = dec.cum[t], head = dec.head[t];
        const int own0 = 32 * wq + (lane & 16);
#pragma unroll 1
        for (int c0 = 0; c0 < 16; c0 += 4) {            // columns c0 .. of both blocks (in a loop: see the note on code size)
          uint32_t w0[4], w1[4], y[2][3], z[2][3];
          umma::ld4(base + c0, w0);
          umma::ld4(base + 16 + c0, w1);
          const float4 cums = *reinterpret_cast<const float4*>(&dec.cum[own0 + c0]);
          const float4 steps = *reinterpret_cast<const float4*>(&dec.step[own0 + c0]);
          const float4 tails = *reinterpret_cast<const float4*>(&dec.tail[32 * wq + c0]);
          umma::wait_ld();
          const float cu[4] = {cums.x, cums.y, cums.z, cums.w}, st[4] = {steps.x, steps.y, steps.z, steps.w},
                      ta[4] = {tails.x, tails.y, tails.z, tails.w};
          float a[4], b[4];
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            const int c = c0 + x;
            float own = __uint_as_float(hi ? w1[x] : w0[x]) * expf(cum - cu[x]) * st[x];
            own = c <= (lane & 15) ? own : 0.f;
            if (MODE == 1 && c == (lane & 15)) own += d_skip;
            a[x] = hi ? __uint_as_float(w0[x]) * head * ta[x] : own;
            b[x] = hi ? own : 0.f;
          }
#pragma unroll
          for (int x = 0; x < 2; ++x) split3cut(a[2 * x], a[2 * x + 1], y[x]), split3cut(b[2 * x], b[2 * x + 1], z[x]);
          uint8_t* to = sP + umma::sw128(row, 4 * wq + (c0 >> 3)) + (c0 & 4) * 2;
          uint8_t* to2 = sP + umma::sw128(row, 4 * wq + 2 + (c0 >> 3)) + (c0 & 4) * 2;
#pragma unroll
          for (int p = 0; p < 3; ++p) {
            *reinterpret_cast<uint2*>(to + p * NH * kRuPanel) = make_uint2(y[0][p], y[1][p]);
            *reinterpret_cast<uint2*>(to2 + p * NH * kRuPanel) = make_uint2(z[0][p], z[1][p]);
          }
        }
        umma::fence_before_sync();
        mbar_arrive(sc_read);
        fence_proxy_async_smem();
        mbar_arrive(p_ready);
      }
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if ((warp & 3) == 1) {
      // =========================== scores, blocks 0 and 1 seen from blocks 2 (lanes 0-15) and 3 ===========================
      const int wg = (warp - 16) >> 2;
      if (wg < NH) {
        const uint32_t base = tb + (32u << 16) + kTmSC;
        const int t = 32 + lane, row = wg * 64 + t;
        for (int j = 0; j < chunks; ++j) {
          const RuDecay& dec = s_dec[(j & (kRuDec - 1)) * NH + wg];
          if (!wait(&dec_full[j & (kRuDec - 1)], j / kRuDec) || !wait(sc_full, j)) break;
          umma::fence_after_sync();
          if (j > 0 && !wait(o2_done, j - 1)) break;
          const float f1 = dec.head[t] * (lane >= 16 ? dec.block[2] : 1.f), f0 = f1 * dec.block[1];
#pragma unroll 1
          for (int c16 = 0; c16 < 4; ++c16) {
            uint32_t x[8], y[4][3];
            umma::ld8(base + 8 * c16, x);
            const float4 t0 = *reinterpret_cast<const float4*>(&dec.tail[8 * c16]), t1 = *reinterpret_cast<const float4*>(&dec.tail[8 * c16 + 4]);
            const float f = c16 < 2 ? f0 : f1;
            umma::wait_ld();
            split3cut(__uint_as_float(x[0]) * f * t0.x, __uint_as_float(x[1]) * f * t0.y, y[0]);
            split3cut(__uint_as_float(x[2]) * f * t0.z, __uint_as_float(x[3]) * f * t0.w, y[1]);
            split3cut(__uint_as_float(x[4]) * f * t1.x, __uint_as_float(x[5]) * f * t1.y, y[2]);
            split3cut(__uint_as_float(x[6]) * f * t1.z, __uint_as_float(x[7]) * f * t1.w, y[3]);
            store_p(row, c16, y);
          }
          umma::fence_before_sync();
          mbar_arrive(sc_read);
          fence_proxy_async_smem();
          mbar_arrive(p_ready);
        }
      }
    } else if (warp == 16) {
      // =========================== issue ===========================
      const uint32_t id_sc = umma::make_idesc<T>(128, 64, 0, 0), id_o2 = umma::make_idesc<T>(128, 64, 1, 0),
                     id_d = umma::make_idesc<T>(128, D, 1, 1);
      const uint32_t dq = umma::desc_low(smem_u32(sQ), 16), dk = umma::desc_low(smem_u32(sK), 16), dk_mn = umma::desc_low(smem_u32(sK), kRuPanel),
                     dx = umma::desc_low(smem_u32(sX), kRuPanel), dp = umma::desc_low(smem_u32(sP), 16), dw = umma::desc_low(smem_u32(sW), kRuPanel);
      const bool leader = umma::elect_one();
      auto issue_sc = [&](int j) {
        if (leader) {
          const uint32_t at = (j & 1) * (kQK >> 4), a0 = dq + at, b0 = dk + at;
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) {
            constexpr int kPanel = kRuPanel >> 4;
            umma::mma_ss_low(tb + kTmSC, a0 + (ks >> 2) * kPanel + (ks & 3) * 2, b0 + (ks >> 2) * kPanel + (ks & 3) * 2, id_sc, ks > 0);
          }
          umma::commit(sc_full);
        }
        __syncwarp();
      };
      auto issue_d = [&](int j) {
        if (leader) {
          const uint32_t b0 = dk_mn + (j & 1) * (kQK >> 4);
#pragma unroll
          for (int p = 2; p >= 0; --p)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma::mma_ss_low(tb + kTmD, dw + ((p * 2 * kRuPanel + ks * 2048) >> 4), b0 + (ks * 2048 >> 4), id_d, p < 2 || ks > 0);
          umma::commit(d_done);
          umma::commit(&k_empty[j & 1]);                // the last reader of k, and of x of chunk j - 1
        }
        __syncwarp();
      };
      auto issue_o1 = [&](int j) {
        if (leader) {
          const uint32_t b0 = dq + (j & 1) * (kQK >> 4);
#pragma unroll
          for (int p = 2; p >= 0; --p)
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks)
              umma::mma_ts_low(tb + kTmO1, tb + kTmS + p * (D / 2) + ks * 8, b0 + (((ks >> 2) * kRuPanel + (ks & 3) * 32) >> 4), id_sc, p < 2 || ks > 0);
          umma::commit(o1_done);
          umma::commit(&q_empty[j & 1]);                // their last reader
        }
        __syncwarp();
      };
      auto issue_o2 = [&](int j) {
        if (leader) {
          const uint32_t a0 = dx + (j % 3) * (2 * kRuPanel >> 4);
#pragma unroll
          for (int p = 2; p >= 0; --p)
#pragma unroll
            for (int hh = 0; hh < NH; ++hh)              // P of a head meets the values of both: half of the lanes are of use
#pragma unroll
              for (int ks = 0; ks < 4; ++ks) {
                const uint32_t a = a0 + (ks * 2048 >> 4), b = dp + (((p * NH + hh) * kRuPanel + ks * 32) >> 4);
                if (NH == 2) umma::mma_ss_half_low(tb + kTmO2, a, b, id_o2, p < 2 || ks > 0, hh);
                else umma::mma_ss_low(tb + kTmO2, a, b, id_o2, p < 2 || ks > 0);
              }
          umma::commit(o2_done);
        }
        __syncwarp();
      };
      for (int j = -1; j < chunks; ++j) {
        const bool more = j + 1 < chunks;
        if (j >= 0) {
          if (!wait(p_ready, j) || (j > 0 && !wait(o_read, j - 1))) break;
          umma::fence_after_sync();
          issue_o2(j);
        }
        if (more) {
          if (!wait(&k_full[(j + 1) & 1], (j + 1) >> 1) || !wait(&q_full[(j + 1) & 1], (j + 1) >> 1) || (j >= 0 && !wait(sc_read, j))) break;
          umma::fence_after_sync();
          issue_sc(j + 1);
        }
        if (j >= 0) {
          if (!wait(s_ready, j)) break;
          umma::fence_after_sync();
          issue_o1(j);
        }
        if (more) {
          if (!wait(w_ready, j + 1) || (j >= 0 && !wait(d_read, j))) break;
          umma::fence_after_sync();
          issue_d(j + 1);
        }
      }
      // products under way finish before the columns and the operands go
      if (leader) umma::commit(drained);
      __syncwarp();
      mbar_wait_bounded(drained, 0, nullptr, kDrainNs);
      __syncwarp();
    } else if (warp == 20) {
      // =========================== decays ===========================
      for (int j = 0; j < chunks; ++j) {
        // the step sizes of every part are on their way before the slot is waited for
        float raw[2 * NH];
#pragma unroll
        for (int u = 0; u < 2 * NH; ++u) {
          const int tok = j * kRuL + 32 * (u & 1) + lane;
          raw[u] = MODE == 1 && tok < sp.q_len ? __bfloat162float(dt[(sp.q_start + tok) * P.dt_stride + h0 + (u >> 1)]) : 0.f;
        }
        if (j >= kRuDec && !wait(&dec_empty[j & (kRuDec - 1)], j / kRuDec - 1)) break;
#pragma unroll 1
        for (int u = 0; u < 2 * NH; ++u) {              // 32 tokens of a head
          const int h = h0 + (u >> 1), half = u & 1, t = 32 * half + lane;
          RuDecay& dec = s_dec[(j & (kRuDec - 1)) * NH + (u >> 1)];
          float cum = 0.f, step = 1.f;                  // past the span: neither decays nor (its x is zero) adds
          if (j * kRuL + t < sp.q_len) {
            if (MODE == 1) {
              step = softplus_f(raw[0] + P.dt_bias[h]);
              cum = -expf(P.a_log[h]) * step;
            } else {
              cum = fmaxf(logf(P.decay[h]), -60.f);     // e^-60: nothing survives a step
            }
          }
#pragma unroll
          for (int i = 0; i + 1 < 2 * NH; ++i) raw[i] = raw[i + 1];
#pragma unroll
          for (int off = 1; off < 16; off <<= 1) {
            const float up = __shfl_up_sync(0xffffffffu, cum, off, 16);
            if ((lane & 15) >= off) cum += up;
          }
          const float end = __shfl_sync(0xffffffffu, cum, 15, 16);
          dec.cum[t] = cum, dec.step[t] = step, dec.head[t] = expf(cum), dec.tail[t] = expf(end - cum) * step;
          if ((lane & 15) == 0) dec.block[2 * half + (lane >> 4)] = expf(end);
          __syncwarp();
          if (half == 0) continue;
          const float b0 = dec.block[0], b1 = dec.block[1], b2 = dec.block[2], b3 = dec.block[3];
          const bool hi = lane >= 16;
          dec.from_start[lane] = dec.head[lane] * (hi ? b0 : 1.f);
          dec.from_start[t] = dec.head[t] * (hi ? b2 : 1.f) * (b0 * b1);
          dec.to_end[lane] = dec.tail[lane] * (hi ? 1.f : b1) * (b2 * b3);
          dec.to_end[t] = dec.tail[t] * (hi ? 1.f : b3);
          if (lane == 0) dec.all = (b0 * b1) * (b2 * b3);
        }
        mbar_arrive(&dec_full[j & (kRuDec - 1)]);
      }
    } else if (warp < 20) {
      copies(std::false_type{}, std::integral_constant<int, kCopyK>{}, (warp - 18) * 32 + lane);
    } else {
      copies(std::true_type{}, std::integral_constant<int, kCopyQ>{}, (warp - 22) * 32 + lane);
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 16) umma::tmem_dealloc(tb, 512);
  if (threadIdx.x == 0 && *gave_up) {
    *reinterpret_cast<volatile int*>(RP.wait_status) = 1;
    __threadfence_system();
  }
}

// bf16 rows that 16-byte copies can start on, value sizes that fill 128 lanes, and steps whose longest span has `from` tokens and
// whose spans have half of that on average: below, a chunk of 64 is mostly padding, and a CTA's start (tensor memory, barriers,
// the first chunk's way through all roles) is not paid back. us, chunk_recurrence_kernel / this one, one prompt and 16 of equal length:
//   32 heads of 128 x 64 selective:  64 tokens 11.3 / 11.3, 27.4 / 23.0;  72  15.0 / 15.8, 36.7 / 32.3;  96  15.2 / 15.5, 37.4 / 31.7;  160  22.5 / 18.9, 56.4 / 39.0
//   8 heads of 128 x 128 decay:      64 tokens 16.3 / 12.8, 17.0 / 14.3;  96  22.1 / 18.0, 23.1 / 20.0;  160  33.8 / 24.1, 34.9 / 26.2
//   32 heads of 64 x 64 selective:   96 tokens 10.7 / 13.3, 24.2 / 26.7;  160  15.1 / 16.6, 35.9 / 33.8; about 3.4 us per further 64 tokens of one prompt for 4.6
//   16 heads of 64 x 128 decay:      96 tokens 15.9 / 14.9, 26.3 / 30.7;  160  23.6 / 19.4, 40.5 / 40.0
// and steps of short spans, 32 heads of 128 x 64: 128 tokens beside 64 spans of 16 64.6 / 89.7, 200 beside 30 of 33 49.7 / 44.1; single tokens
// 256 beside 200 182 / 156, of 64 x 64 57.8 / 106.
bool recurrence_umma_ok(const RecParams& P, int dtype, int num_seqs, int max_q, int64_t total_q) {
  if (P.mode > 1 || dtype != B200_DTYPE_BF16 || P.cu_q == nullptr || num_seqs > 65535) return false;
  if (P.kdim > 128 || P.kdim % 8 != 0) return false;
  if (!(P.vdim == 128 || (P.vdim == 64 && (P.H / P.groups) % 2 == 0))) return false;
  if (P.q_stride % 8 != 0 || P.k_stride % 8 != 0 || P.v_stride % 8 != 0 || !aligned16(P.q) || !aligned16(P.k) || !aligned16(P.v)) return false;
  const int from = P.kdim > 64 ? 96 : 256;
  return max_q >= from && (num_seqs == 1 || total_q >= (int64_t)num_seqs * (from / 2));
}

template <int D, int NH, int MODE, bool SILU>
static int recurrence_umma_launch_as(const RecParams& P, int num_seqs, int64_t wait_ns, cudaStream_t stream) {
  auto kern = recurrence_umma_kernel<D, NH, MODE, SILU>;
  constexpr int smem = ru_smem<D, NH>();
  static_assert(smem <= 227 * 1024, "one CTA's shared memory");
  static std::atomic<uint64_t> devices{0};
  const cudaError_t allowed = allow_smem(kern, smem, devices);
  if (allowed != cudaSuccess) return (int)allowed;
  const RuParams RP{P, wait_tries(wait_ns), wait_status()};
  B200_RETURN_IF(RP.wait_status == nullptr, B200_ERR_DRIVER);
  launch_pdl(kern, dim3((unsigned)(P.H / NH), (unsigned)num_seqs), dim3(kRuThreads), (size_t)smem, stream, RP);
  return finish_launch();
}

int recurrence_umma_launch(const RecParams& P, int num_seqs, int64_t wait_ns, cudaStream_t stream) {
  B200_RETURN_IF(take_wait_status(), B200_ERR_WAIT);             // of an earlier call
#define B200_RU(D, NH)                                                                                                   \
  (P.mode == 1 ? (P.act_silu ? recurrence_umma_launch_as<D, NH, 1, true>(P, num_seqs, wait_ns, stream)                            \
                             : recurrence_umma_launch_as<D, NH, 1, false>(P, num_seqs, wait_ns, stream))                          \
               : (P.act_silu ? recurrence_umma_launch_as<D, NH, 0, true>(P, num_seqs, wait_ns, stream)                            \
                             : recurrence_umma_launch_as<D, NH, 0, false>(P, num_seqs, wait_ns, stream)))
  if (P.vdim == 128) return P.kdim <= 64 ? B200_RU(64, 1) : B200_RU(128, 1);
  return P.kdim <= 64 ? B200_RU(64, 2) : B200_RU(128, 2);
#undef B200_RU
}

}  // namespace b200
