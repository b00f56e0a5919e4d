// attn_split.cu -- prompt portions of attn_generic (seq_mixers.cu) for fp32 models, on the 5th-generation tensor cores.
//
// The same job as attn_tiled_kernel without a window, chunks or capped scores: causal softmax attention in 32 bits, packed or paged
// keys, sinks, output gates, values inside the key rows. Every fp32 operand is split into three bf16 terms, each the rounding of
// what the ones before it leave (24 bits and a sign), and a product of two is the six products of their terms that count, small
// ones first, accumulated in fp32; the three left out are below 2^-26 of it, of either sign. An accumulator never outlives a tile
// of 64 keys: a tile's P V is added to the rows' sums in registers, one rounding each, so what the tensor core's own additions
// lose does not grow with the length. Error against 64 bits (relative 2-norm, attn_tiled_kernel / this one): 4 prompts of 700-1024
// tokens, heads of 128 3.0e-7 / 1.9e-7; one of 64 1.7e-7 / 1.3e-7; heads of 64, one of 128 1.6e-7 / 1.3e-7. (With terms cut off
// instead of rounded, whose left-out products all have one sign, 2.4e-7 / 1.7e-7 / 1.8e-7.)
//
// CTA = 128 rows of one (sequence, kv head) -- row r is token r / rep, query head g * rep + r % rep -- and 64 keys at a time. Warps:
// 0-3 softmax (thread = row): S from TMEM, running maximum, P as three terms back into TMEM; 4-7 sums (thread = row): O <- O
// corr + P V, at the end O / l; 8-15 copy: a tile of K or V is loaded as fp32 into registers while the slot is still in use,
// split, and stored as three planes of SW128 panels (paging, row strides and padding of head sizes cost nothing more there); 16
// issues S(j+1) (6 x D/16 MMAs M128 N64 K16), then P V(j) (6 x 4 MMAs M128 N=vdim K16, A from TMEM). TMEM: S 2 x 64 columns, P
// 96, P V 2 x 128. Shared memory at 128: Q 96 KB, K 48, V 48: one CTA per SM.
// Bound: the tensor pipe (24 x 74 + 48 x 75 = 5376 cycles per tile of 64 keys at heads of 128, where the fp32 FMA pipes need 16384),
// and the copying warps' load -> split -> store beside it (a tile takes 6300). Measured: 4 ragged prompts of 700-1024 tokens, 8
// heads over 2 of 128, paged, 288 us (attn_tiled_kernel) -> 66 (20 calls in a graph; 68 where the inputs change from call to call;
// 10 more with 8 columns a lane, which read every sector twice, 7 with that but block ids looked up a step ahead); 4 of 600-1000, 32
// heads over 8 of 64, 490 -> 132.
//
// Few row tiles (attn_split_shared) have their keys shared by a cluster of two CTAs: each runs as above over its part, leaves its rows' maxima
// and sums in its shared memory, and the first one merges them, relative to the larger maximum.
//
// What the split cannot carry: what is not finite or close to the largest numbers (and 0 x inf would reach rows that do not see the key),
// and what is so small that a term of it would not be normal. Values come times 2^27, which leaves nothing too small, and go back
// at the end. A small element of Q or K (below 2^-100) is off by 2^-126 at most, which is nothing to a score unless it meets one of
// 2^70 or more. The copying warps look at the magnitudes; a CTA that met such values computes its rows once more in plain fp32,
// key by key as attn_generic_kernel does (4 prompts of 700-1024 tokens with an infinity in every head of each: 5.2 ms; attn_tiled_kernel 0.29).
// Waits are bounded as in recurrence_umma_kernel.
#include "attn_tiled.cuh"
#include "recurrence.cuh"
#include "umma.cuh"

namespace b200 {

constexpr int kAsM = 128, kAsN = 64, kAsThreads = 640, kAsCorr = 4;
constexpr int kAsPanel = 64 * 128;                     // bytes of 64 rows x 64 elements
constexpr int kAsParts = 2;                             // CTAs that share a row tile's keys, where they do

constexpr float kAsUp = 134217728.f;                    // 2^27: values come to the tensor core times it (see below)

struct AttnSplitParams {
  AttnTiledParams a;
  int wait_tries;                                      // of one wait
  int* wait_status;
};

template <int DK, int DV>
constexpr int as_smem() {
  return 1024 + 3 * (2 * (DK / 64) + DK / 64 + DV / 64) * kAsPanel + (kAsCorr + 3 + kAsParts) * kAsM * 4 + 256;
}

// four fp32 -> half a 16-byte chunk of each of three planes
__device__ __forceinline__ void store_split4(uint8_t* to, int plane, float4 x) {
  uint32_t w[2][3];
  split3x2(x.x, x.y, w[0]);
  split3x2(x.z, x.w, w[1]);
#pragma unroll
  for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(to + p * plane) = make_uint2(w[0][p], w[1][p]);
}
// two fp32 operations in one instruction: a b + c
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(reinterpret_cast<uint64_t&>(c)) : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)));
  return c;
}

// SHARED: a cluster of kAsParts CTAs takes a row tile, each a part of its keys; the first merges the results over distributed shared memory
template <int DK, int DV, bool SHARED>
__global__ void __launch_bounds__(kAsThreads, 1)
attn_split_kernel(const __grid_constant__ AttnSplitParams AP) {
  using T = __nv_bfloat16;
  const AttnTiledParams& P = AP.a;
  constexpr int CK = DK / 64, CV = DV / 64;
  constexpr int kQPlane = CK * 2 * kAsPanel, kKPlane = CK * kAsPanel, kVPlane = CV * kAsPanel;
  constexpr uint32_t kTmS = 0, kTmP = 128, kTmO = 256;
  extern __shared__ __align__(1024) uint8_t as_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(as_smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                                   // [3 terms][CK panels][128 rows]
  uint8_t* sK = sQ + 3 * kQPlane;                       // [3][CK][64 keys]
  uint8_t* sV = sK + 3 * kKPlane;                       // [3][CV][64 keys]
  float* s_corr = reinterpret_cast<float*>(sV + 3 * kVPlane);   // [kAsCorr][128], then [128] 1 / l
  float *s_m = s_corr + (kAsCorr + 1) * kAsM, *s_l = s_m + kAsM, *s_part = s_l + kAsM;   // keys shared: [128] m, l of this part; [kAsParts][128] what a part counts
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_part + kAsParts * kAsM);
  uint64_t *q_full = bars, *k_full = bars + 1, *k_empty = bars + 2, *v_full = bars + 3, *v_empty = bars + 4, *s_full = bars + 5,
           *p_ready = bars + 7, *o_full = bars + 8, *o_read = bars + 10, *done = bars + 12, *drained = bars + 13;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 14);
  volatile int* gave_up = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int *huge = gave_up + 1, *tiny = gave_up + 2, *large = gave_up + 3;
  int parts_met = 1;                                     // CTAs whose values count: set behind the meeting of a cluster's
  auto wild = [&] {
    bool any = *huge != 0 || (*tiny != 0 && *large != 0);
    for (int p = 1; p < parts_met; ++p)
      any = any || ld_peer_int(smem_u32(const_cast<int*>(huge)), p) != 0 ||
            (ld_peer_int(smem_u32(const_cast<int*>(tiny)), p) != 0 && ld_peer_int(smem_u32(const_cast<int*>(large)), p) != 0);
    return any;
  };

  auto peers_gave_up = [&] {
    bool any = false;
    for (int p = 1; p < parts_met; ++p) any = any || ld_peer_int(smem_u32(const_cast<int*>(gave_up)), p) != 0;
    return any;
  };

  pdl_wait();
  // the last row tiles see the most keys: those of every (sequence, kv head) start first
  constexpr int ctas = SHARED ? kAsParts : 1;
  const int part = SHARED ? (int)cluster_rank() : 0;
  const int units = P.G * P.num_seqs, index = blockIdx.x / ctas, tile = (int)(gridDim.x / ctas / units) - 1 - index / units, unit = index % units;
  const int s = unit / P.G, g = unit % P.G;
  const SeqSpan sp = seq_span(P.cu_q, P.cu_k, nullptr, s);
  const int rep = P.H / P.G, rows = sp.q_len * rep, r0 = tile * kAsM;
  if (r0 >= rows) return;
  const int dim = P.dim, vdim = P.vdim;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float* qb = reinterpret_cast<const float*>(P.q);
  const float* kb = reinterpret_cast<const float*>(P.k) + (int64_t)g * dim;
  const float* vb = P.v != nullptr ? reinterpret_cast<const float*>(P.v) + (int64_t)g * vdim : kb;
  const int64_t v_stride = P.v != nullptr ? P.v_stride : P.k_stride;
  const int64_t k_base = P.block_tables == nullptr ? P.cu_k[s] : 0;
  const int* table = P.block_tables != nullptr ? P.block_tables + (int64_t)s * P.bt_stride : nullptr;
  auto key_row = [&](int key) -> int64_t {
    return table != nullptr ? (int64_t)table[key / P.block_size] * P.block_size + key % P.block_size : k_base + key;
  };
  const int min_pos = sp.first_pos() + r0 / rep, max_pos = sp.first_pos() + (min(r0 + kAsM, rows) - 1) / rep;
  // this CTA's key tiles: of a cluster, each takes three at least, and those behind take none
  const int all_tiles = (max_pos + kAsN) / kAsN, parts = SHARED ? max(1, min(ctas, all_tiles / 3)) : 1, per = (all_tiles + parts - 1) / parts;
  if (SHARED && part >= parts) return;
  const int first_key = part * per * kAsN, tiles = min(per, all_tiles - part * per);

  if (threadIdx.x == 0) {
    mbar_init(q_full, 256), mbar_init(k_full, 256), mbar_init(k_empty, 1), mbar_init(v_full, 256), mbar_init(v_empty, 1);
    for (int b = 0; b < 2; ++b) mbar_init(&s_full[b], 1), mbar_init(&o_full[b], 1), mbar_init(&o_read[b], kAsM);
    mbar_init(p_ready, kAsM), mbar_init(done, kAsM), mbar_init(drained, 1);
    mbar_fence_init();
    *gave_up = 0, *huge = 0, *tiny = 0, *large = 0;
  }
  if (warp == 16) umma::tmem_alloc(tmem_slot, 512);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  constexpr uint32_t tb = 0;                            // all 512 columns: they start at 0
  auto wait = [&](uint64_t* bar, int parity) { return mbar_warp_wait(bar, parity & 1, AP.wait_tries, gave_up); };

  auto look = [&](float4 x, float& most, float& least) {
    asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(most) : "f"(x.x), "f"(x.y));
    asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(most) : "f"(x.z), "f"(x.w));
    asm("min.abs.f32 %0, %0, %1, %2;" : "+f"(least) : "f"(x.x), "f"(x.y));
    asm("min.abs.f32 %0, %0, %1, %2;" : "+f"(least) : "f"(x.z), "f"(x.w));
  };
  auto judge = [&](float most, float least) {           // of what was looked at in Q or K
    if (!(most < 0x1p127f)) *huge = 1;
    if (most >= 0x1p70f) *large = 1;
    if (least < 0x1p-100f) *tiny = 1;
  };
  auto fetch = [&](const float* row, int col, int width, bool there) {       // zero past the width (a multiple of 4)
    return there && col < width ? __ldg(reinterpret_cast<const float4*>(row + col)) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  // Q. Rows of 128: by the eight warps that have nothing else to do before the first scores, and registers for many loads; four rows at a time
  // by the copying warps, it held the first tiles up (graphs: 12 x 500 93.8 -> 79.5 us, 4 x 1000 84.2 -> 78.5, 4 x 700-1024 68.6 -> 67.2). Rows of 64 and
  // shared keys are up to 5 % better off with the copying warps.
  constexpr bool kEarlyQ = DK == 128 && !SHARED;
  auto copy_q = [&](int w8) {
    float most = 0.f, least = 1.f;
#pragma unroll (kEarlyQ ? 8 : 4)
    for (int row = DK == 128 ? w8 : 2 * w8 + (lane >> 4); row < kAsM; row += DK == 128 ? 8 : 16) {
      const int r = r0 + row, tok = r / rep, col = 4 * (DK == 128 ? lane : lane & 15);
      float4 y = fetch(qb + (int64_t)(sp.q_start + tok) * P.q_stride + (int64_t)(g * rep + r - tok * rep) * dim, col, dim, r < rows);
      look(y, most, least);
      if (P.scale < 0.f) y = make_float4(-y.x, -y.y, -y.z, -y.w);
      store_split4(sQ + (col >> 6) * 2 * kAsPanel + umma::sw128(row, (col >> 3) & 7) + (col & 4) * 2, kQPlane, y);
    }
    judge(most, least);
    fence_proxy_async_smem();
    mbar_arrive(q_full);
  };

  // Registers: 640 x 96 at launch = 128 x (112 softmax + 160 sums + 2 x 80 copies + 48)
  if (warp < 4) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
    // =========================== softmax ===========================
    if (kEarlyQ) copy_q(warp);
    const int row = warp * 32 + lane, r = min(r0 + row, rows - 1);
    const uint32_t base = tb + ((uint32_t)(warp * 32) << 16);
    const int pos = sp.first_pos() + r / rep;
    // A key's weight is 2^(x c - top), top = m c of the largest score so far, with c in two parts that are subtracted from top in one
    // rounding (with the rounded c alone the weights of short rows were off by a seventh more). Rows whose top has a spacing of 2^-7
    // or more count from the largest score itself: 2^((x - m) c). Hidden keys, and visible ones whose score has overflowed,
    // end at -FLT_MAX, which c turns into no weight and at which the small part stays finite (attn_split_fits); NaN stays NaN. Scores
    // of a negative scale have changed sign in q
    const float c = fabsf(P.scale) * kLog2e, c_low = fmaf(fabsf(P.scale), kLog2e, -c) + fabsf(P.scale) * 1.925963033500e-8f;
    float top = -INFINITY, less = 0.f;
    auto weights = [&](float& a, float& b) {                   // 2^(x c - less) of both
      float2 x = make_float2(a, b);
      asm("max.NaN.f32 %0, %0, %1;" : "+f"(x.x) : "f"(-3.4028234e38f));
      asm("max.NaN.f32 %0, %0, %1;" : "+f"(x.y) : "f"(-3.4028234e38f));
      const float2 e = fma2(x, make_float2(c, c), fma2(x, make_float2(c_low, c_low), make_float2(-less, -less)));
      a = ex2_approx(e.x), b = ex2_approx(e.y);
    };
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < tiles; ++j) {
      ok = wait(&s_full[j & 1], j >> 1);
      if (!ok) break;
      umma::fence_after_sync();
      float x[kAsN];
#pragma unroll
      for (int i0 = 0; i0 < kAsN; i0 += 32) {
        uint32_t w[32];
        umma::ld32(base + kTmS + (j & 1) * kAsN + i0, w);
        umma::wait_ld();
#pragma unroll
        for (int i = 0; i < 32; ++i) x[i0 + i] = __uint_as_float(w[i]);
      }
      if (first_key + j * kAsN + kAsN - 1 > min_pos) {
        const int last = pos - first_key - j * kAsN;
#pragma unroll
        for (int i = 0; i < kAsN; ++i) x[i] = i <= last ? x[i] : -INFINITY;
      }
      float mx[4] = {x[0], x[1], x[2], x[3]};
#pragma unroll
      for (int i = 4; i < kAsN; ++i) mx[i & 3] = fmaxf(mx[i & 3], x[i]);
      const float m_new = fmaxf(m, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])));
      const bool far = fabsf(m_new) * c >= 65536.f && m_new != -INFINITY;
      less = far || m_new == -INFINITY ? 0.f : m_new * c;      // (-inf: every score so far has overflowed)
      float corr = ex2_approx(top - less);
      if (far) {
        float none = 0.f;
        corr = m - m_new;
        weights(corr, none);
#pragma unroll
        for (int i = 0; i < kAsN; ++i) x[i] -= m_new;
      }
      top = m_new * c;
      m = m_new;
      s_corr[(j & (kAsCorr - 1)) * kAsM + row] = corr;
      if (j > 0) {
        ok = wait(&o_full[(j - 1) & 1], (j - 1) >> 1);   // the last tile's P is consumed
        if (!ok) break;
        umma::fence_after_sync();
      }
      float sum[2] = {0.f, 0.f};
#pragma unroll
      for (int i0 = 0; i0 < kAsN; i0 += 16) {
        uint32_t w[3][8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float a = x[i0 + 2 * i], b = x[i0 + 2 * i + 1];
          weights(a, b);
          sum[0] += a, sum[1] += b;
          uint32_t y[3];
          split3x2(a, b, y);
          w[0][i] = y[0], w[1][i] = y[1], w[2][i] = y[2];
        }
#pragma unroll
        for (int p = 0; p < 3; ++p) umma::st8(base + kTmP + p * 32 + i0 / 2, w[p]);
      }
      l = fmaf(l, corr, sum[0] + sum[1]);
      umma::wait_st();
      umma::fence_before_sync();
      mbar_arrive(p_ready);
    }
    if (SHARED && parts > 1) {                                    // the parts of the row's keys: what each counts, relative to the largest score of all
      s_m[row] = m, s_l[row] = l;
      cluster_arrive(), cluster_wait();
      if (part == 0) {
        float ms[kAsParts], m_all = m;
#pragma unroll
        for (int p = 0; p < kAsParts; ++p) {
          ms[p] = p < parts ? ld_peer(smem_u32(s_m + row), p) : -INFINITY;
          m_all = fmaxf(m_all, ms[p]);
        }
        const bool far = fabsf(m_all) * c >= 65536.f && m_all != -INFINITY;
        // (a part's weights count from the ROUNDED m c: with a product fused into the difference its residual would stay in the factor)
        less = 0.f, l = 0.f, top = __fmul_rn(m_all, c);
#pragma unroll
        for (int p = 0; p < kAsParts; ++p) {
          float f = ms[p] == -INFINITY ? 0.f : ex2_approx(__fmul_rn(ms[p], c) - top), none = 0.f;
          if (far && ms[p] != -INFINITY) f = ms[p] - m_all, weights(f, none);
          if (p < parts) l = fmaf(ld_peer(smem_u32(s_l + row), p), f, l);
          s_part[p * kAsM + row] = f;
        }
      }
    }
    // a sink is one more entry of the softmax that has a logit and no value (in units of log2, as top)
    float share = 1.f;
    if (P.sink != nullptr) {
      const float sink = P.sink[g * rep + r % rep] * kLog2e;
      if (sink > top) share = ex2_approx(top - sink), l = fmaf(l, share, 1.f);
      else l += top == -INFINITY ? 1.f : ex2_approx(sink - top);
    }
    float inv = share / l;
    if (P.gate != nullptr)
      inv *= sigmoid_f(reinterpret_cast<const float*>(P.gate)[(int64_t)(sp.q_start + r / rep) * P.gate_stride + g * rep + r % rep]);
    s_corr[kAsCorr * kAsM + row] = inv;
    mbar_arrive(done);
  } else if (warp < 8) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 160;");
    // =========================== sums ===========================
    if (kEarlyQ) copy_q(warp);
    const int quarter = warp - 4, row = quarter * 32 + lane, r = r0 + row;
    const uint32_t base = tb + ((uint32_t)(quarter * 32) << 16);
    float O[DV];
#pragma unroll
    for (int i = 0; i < DV; ++i) O[i] = 0.f;
    bool ok = true;
    for (int j = 0; j < tiles; ++j) {
      ok = wait(&o_full[j & 1], j >> 1);
      if (!ok) break;
      umma::fence_after_sync();
      const float corr = s_corr[(j & (kAsCorr - 1)) * kAsM + row];
#pragma unroll
      for (int i0 = 0; i0 < DV; i0 += 16) {
        uint32_t w[16];
        umma::ld16(base + kTmO + (j & 1) * 128 + i0, w);
        umma::wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) O[i0 + i] = fmaf(O[i0 + i], corr, __uint_as_float(w[i]));
      }
      umma::fence_before_sync();
      mbar_arrive(&o_read[j & 1]);
    }
    if (SHARED && parts > 1) {
      // other parts leave their sums where the operands were, which no product reads any more: [DV / 4][128 rows][4]
      if (part > 0) {
#pragma unroll
        for (int i = 0; i < DV; i += 4) reinterpret_cast<float4*>(smem)[(i / 4) * kAsM + row] = make_float4(O[i], O[i + 1], O[i + 2], O[i + 3]);
      }
      cluster_arrive(), cluster_wait();
    }
    parts_met = parts;
    ok = ok && part == 0 && wait(done, 0) && !peers_gave_up();     // (a part whose wait ran out has left nothing to merge)
    if (SHARED && ok && parts > 1) {
      const float own = s_part[row];
#pragma unroll
      for (int i = 0; i < DV; ++i) O[i] *= own;
#pragma unroll 1
      for (int p = 1; p < parts; ++p) {
        const float f = s_part[p * kAsM + row];
        const uint32_t from = smem_u32(smem) + row * 16;
#pragma unroll
        for (int i = 0; i < DV; i += 4) {
          const float4 x = ld_peer4(from + (i / 4) * kAsM * 16, p);
          O[i] = fmaf(x.x, f, O[i]), O[i + 1] = fmaf(x.y, f, O[i + 1]), O[i + 2] = fmaf(x.z, f, O[i + 2]), O[i + 3] = fmaf(x.w, f, O[i + 3]);
        }
      }
    }
    if (ok && r < rows && !wild()) {
      const float inv = s_corr[kAsCorr * kAsM + row];
      const int tok = r / rep;
      float* o = reinterpret_cast<float*>(P.out) + (int64_t)(sp.q_start + tok) * ((int64_t)P.H * vdim) + (int64_t)(g * rep + r - tok * rep) * vdim;
#pragma unroll
      for (int i = 0; i < DV; i += 4)
        if (i < vdim) *reinterpret_cast<float4*>(o + i) = make_float4(O[i] / kAsUp * inv, O[i + 1] / kAsUp * inv, O[i + 2] / kAsUp * inv, O[i + 3] / kAsUp * inv);
    }
  } else if (warp < 16) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
    // =========================== copies ===========================
    // A lane takes 4 columns, so that a warp reads whole rows (with 8, every 32-byte sector came twice); warp w of the eight takes
    // rows w, w + 8, .. of Q, K or V, for 64 columns two neighbouring rows at a time
    const int w8 = warp - 8;
    float most = 0.f, least = 1.f, most_v = 0.f;        // magnitudes met
    auto look_v = [&](float4 x) {
      asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(most_v) : "f"(x.x), "f"(x.y));
      asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(most_v) : "f"(x.z), "f"(x.w));
    };
    // steps: K0, K1, V0, K2, V1, .., the order in which the issuing warp takes them
    const int steps = 2 * tiles;
    auto is_key = [&](int st) { return st == 0 || ((st & 1) && st + 1 < steps); };
    auto tile_of = [&](int st) { return st == 0 ? 0 : is_key(st) ? (st + 1) >> 1 : st + 1 == steps ? tiles - 1 : (st >> 1) - 1; };
    // Under way at a time: the block id of step st + kAhead + 1, the values of the kAhead steps before, and step st's way to shared
    // memory. (Two steps of 128-wide rows are more registers than the role has: 72.9 -> 88.8 us.) A warp has 8 rows of a tile: lane i
    // looks up the i-th
    constexpr int kAhead = DK == 64 && DV == 64 ? 2 : 1, kItems = DK == 64 && DV == 64 ? 4 : 8;
    float4 x0[kItems], x1[kItems];
    int64_t own_row;
    auto row_of = [&](int i, int wide) { return wide ? w8 + 8 * i : 2 * (w8 + 8 * (i >> 1)) + (i & 1); };
    auto look_up = [&](int st) {
      own_row = key_row(min(first_key + tile_of(st) * kAsN + row_of(lane & 7, (is_key(st) ? DK : DV) == 128), max_pos));
    };
    auto each = [&](int wide, auto f) {                 // f(item, row of the tile, first column, which of the 8 rows)
#pragma unroll
      for (int i = 0; i < kItems; ++i) {
        if (wide) f(i, w8 + 8 * i, 4 * lane, i);
        else if (i < 4) f(i, 2 * (w8 + 8 * i) + (lane >> 4), 4 * (lane & 15), 2 * i + (lane >> 4));
      }
    };
    auto load = [&](int st, float4 (&x)[kItems]) {
      const bool key = is_key(st);
      const int j = tile_of(st), width = key ? dim : vdim;
      const float* from = key ? kb : vb;
      const int64_t stride = key ? P.k_stride : v_stride, offset = own_row * stride;
      each((key ? DK : DV) == 128, [&](int i, int row, int col, int nth) {
        x[i] = fetch(from + __shfl_sync(0xffffffffu, offset, nth), col, width, first_key + j * kAsN + row <= max_pos);
      });
    };
    look_up(0);
    load(0, x0);
    look_up(1);
    if (kAhead == 2) {
      load(1, x1);
      if (steps > 2) look_up(2);
    }
    if (!kEarlyQ) copy_q(w8);
    auto put = [&](int st, float4 (&x)[kItems]) -> bool {
      const bool key = is_key(st);
      const int j = tile_of(st), plane = key ? kKPlane : kVPlane;
      if (j > 0 && !wait(key ? k_empty : v_empty, j - 1)) return false;
      uint8_t* to = key ? sK : sV;
      each((key ? DK : DV) == 128, [&](int i, int row, int col, int) {
        if (key) look(x[i], most, least);
        else x[i] = make_float4(x[i].x * kAsUp, x[i].y * kAsUp, x[i].z * kAsUp, x[i].w * kAsUp), look_v(x[i]);
        store_split4(to + (col >> 6) * kAsPanel + umma::sw128(row, (col >> 3) & 7) + (col & 4) * 2, plane, x[i]);
      });
      if (!(most_v < 0x1p107f)) *huge = 1;
      judge(most, least);
      fence_proxy_async_smem();
      mbar_arrive(key ? k_full : v_full);
      if (st + kAhead < steps) load(st + kAhead, x);
      if (st + kAhead + 1 < steps) look_up(st + kAhead + 1);
      return true;
    };
    const int come = AP.wait_tries > 0 ? steps : min(steps, 4);       // (a limit of 0 tests the way out: nothing comes any more)
#pragma unroll 1
    for (int st = 0; st < come; st += kAhead) {         // (steps is even)
      if (!put(st, x0)) break;
      if (kAhead == 2 && !put(st + 1, x1)) break;
    }
    if (SHARED && parts > 1) cluster_arrive(), cluster_wait();
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
    if (warp == 16) {
      // =========================== issue ===========================
      const int nks = (dim + 15) >> 4, nv = (vdim + 15) & ~15;
      const uint32_t id_s = umma::make_idesc<T>(kAsM, kAsN, 0, 0), id_o = umma::make_idesc<T>(kAsM, nv, 0, 1);
      const uint32_t dq = umma::desc_low(smem_u32(sQ), 16), dk = umma::desc_low(smem_u32(sK), 16), dv = umma::desc_low(smem_u32(sV), kAsPanel);
      const bool leader = umma::elect_one();
      // products of terms (a of the first operand, b of the second), the smallest first
      constexpr int kA[6] = {1, 2, 0, 1, 0, 0}, kB[6] = {1, 0, 2, 0, 1, 0};
      auto issue_s = [&](int j) {
        if (leader) {
          const uint32_t to = tb + kTmS + (j & 1) * kAsN;
#pragma unroll
          for (int p = 0; p < 6; ++p)
#pragma unroll
            for (int ks = 0; ks < DK / 16; ++ks)
              if (ks < nks)
                umma::mma_ss_low(to, dq + ((kA[p] * kQPlane + (ks >> 2) * 2 * kAsPanel + (ks & 3) * 32) >> 4),
                                 dk + ((kB[p] * kKPlane + (ks >> 2) * kAsPanel + (ks & 3) * 32) >> 4), id_s, p > 0 || ks > 0);
          umma::commit(&s_full[j & 1]);
          umma::commit(k_empty);
        }
        __syncwarp();
      };
      bool ok = wait(q_full, 0) && wait(k_full, 0);
      umma::fence_after_sync();
      if (ok) issue_s(0);
      for (int j = 0; ok && j < tiles; ++j) {
        if (j + 1 < tiles) {
          ok = wait(k_full, j + 1);
          if (!ok) break;
          umma::fence_after_sync();
          issue_s(j + 1);
        }
        ok = wait(p_ready, j) && wait(v_full, j) && (j < 2 || wait(&o_read[j & 1], (j >> 1) - 1));
        if (!ok) break;
        umma::fence_after_sync();
        if (leader) {
          const uint32_t to = tb + kTmO + (j & 1) * 128;
#pragma unroll
          for (int p = 0; p < 6; ++p)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma::mma_ts_low(to, tb + kTmP + kA[p] * 32 + ks * 8, dv + ((kB[p] * kVPlane + ks * 2048) >> 4), id_o, p > 0 || ks > 0);
          umma::commit(&o_full[j & 1]);
          umma::commit(v_empty);
        }
        __syncwarp();
      }
      // products under way finish before the columns and the operands go
      if (leader) umma::commit(drained);
      __syncwarp();
      mbar_wait_bounded(drained, 0, nullptr, kDrainNs);
      __syncwarp();
    }
    if (SHARED && parts > 1) cluster_arrive(), cluster_wait();
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 16) umma::tmem_dealloc(tb, 512);
  if (threadIdx.x == 0 && *gave_up) {
    *reinterpret_cast<volatile int*>(AP.wait_status) = 1;
    __threadfence_system();
  }
  if (SHARED && part > 0) {                              // nobody leaves while the first part reads
    cluster_arrive(), cluster_wait();
    return;
  }
  parts_met = parts;
  const bool plain = wild() && !*gave_up && !peers_gave_up();
  if (SHARED && parts > 1) cluster_arrive(), cluster_wait();
  if (!plain) return;

  // ---- plain fp32, one warp per row, a lane per key of 32 and then a lane per value column of 32 (see above)
#pragma unroll 1
  for (int r = r0 + warp; r < min(r0 + kAsM, rows); r += kAsThreads / 32) {
    const int tok = r / rep, head = g * rep + r - tok * rep, pos = sp.first_pos() + tok;
    const float* q = qb + (int64_t)(sp.q_start + tok) * P.q_stride + (int64_t)head * dim;
    float m = P.sink != nullptr ? P.sink[head] : -INFINITY, l = P.sink != nullptr ? 1.f : 0.f, acc[DV / 32];
#pragma unroll
    for (int c = 0; c < DV / 32; ++c) acc[c] = 0.f;
#pragma unroll 1
    for (int j0 = 0; j0 <= pos; j0 += 32) {
      const bool seen = j0 + lane <= pos;
      float sc = -INFINITY;
      if (seen) {
        const float* k = kb + key_row(j0 + lane) * P.k_stride;
        float d = 0.f;
#pragma unroll 1
        for (int i = 0; i < dim; i += 4) {
          const float4 x = __ldg(reinterpret_cast<const float4*>(q + i)), y = __ldg(reinterpret_cast<const float4*>(k + i));
          d += x.x * y.x, d += x.y * y.y, d += x.z * y.z, d += x.w * y.w;
        }
        sc = d * P.scale;
      }
      const float m_new = fmaxf(m, warp_max(sc));
      if (m_new == -INFINITY) continue;
      const float corr = expf(m - m_new), p = sc == -INFINITY ? 0.f : expf(sc - m_new);
      l = l * corr + warp_sum(p);
      m = m_new;
#pragma unroll
      for (int c = 0; c < DV / 32; ++c) acc[c] *= corr;
#pragma unroll 1
      for (int j = 0; j < min(32, pos + 1 - j0); ++j) {
        const float pj = __shfl_sync(0xffffffffu, p, j);
        const float* v = vb + key_row(j0 + j) * v_stride;
#pragma unroll
        for (int c = 0; c < DV / 32; ++c)
          if (lane + 32 * c < vdim) acc[c] += pj * v[lane + 32 * c];
      }
    }
    float inv = 1.0f / l;
    if (P.gate != nullptr) inv *= sigmoid_f(reinterpret_cast<const float*>(P.gate)[(int64_t)(sp.q_start + tok) * P.gate_stride + head]);
    float* o = reinterpret_cast<float*>(P.out) + (int64_t)(sp.q_start + tok) * ((int64_t)P.H * vdim) + (int64_t)head * vdim;
#pragma unroll
    for (int c = 0; c < DV / 32; ++c)
      if (lane + 32 * c < vdim) o[lane + 32 * c] = acc[c] * inv;
  }
}

// fp32 rows that 16-byte loads can start on, and steps whose longest span has `least` rows (tokens x heads per group) and whose spans
// have half of that on average: below, most of a 128-row tile is padding. us, attn_tiled_kernel / this one, one prompt:
//   8 heads over 2 of 128 (4 rows a token)  33 tokens 15.7 / 16.6;  64  18.1 / 17.0;  128  30.2 / 20.5;  1000  196 / 66
//   32 heads over 8 of 64 (4)               17  12.0 / 9.3;  64  14.7 / 10.1;  200  32.9 / 15.2
//   8 heads of 48 (1)                       64  13.7 / 9.1;  128  22.1 / 12.3;  16 of 64  14.2 / 10.1
bool attn_split_fits(const AttnTiledParams& P, int num_seqs, int max_q, int64_t total_q, int dtype) {
  if (dtype != B200_DTYPE_F32 || P.window > 0 || P.chunk > 0 || P.softcap > 0.f || P.dim > 128 || P.vdim > 128) return false;
  if (P.dim % 4 != 0 || P.vdim % 4 != 0 || P.q_stride % 4 != 0 || P.k_stride % 4 != 0 || (P.v != nullptr && P.v_stride % 4 != 0)) return false;
  if (!aligned16(P.q) || !aligned16(P.k) || !aligned16(P.v) || !aligned16(P.out)) return false;
  if (!(fabsf(P.scale) > 1e-20f && fabsf(P.scale) < 1e6f)) return false;       // -FLT_MAX times c vanishes, times c_low stays finite
  const int rep = P.H / P.G;
  if (((int64_t)max_q * rep + kAsM - 1) / kAsM * P.G > 0x7fffffff / num_seqs) return false;
  const int64_t least = P.dim <= 64 && P.vdim <= 64 ? 64 : 192;
  return (int64_t)max_q * rep >= least && (num_seqs == 1 || total_q * rep >= num_seqs * least / 2);
}

template <int DK, int DV, bool SHARED>
static int attn_split_launch_as(const AttnTiledParams& P, dim3 grid, int64_t wait_ns, cudaStream_t stream) {
  auto kern = attn_split_kernel<DK, DV, SHARED>;
  constexpr int smem = as_smem<DK, DV>();
  static_assert(smem <= 227 * 1024, "one CTA's shared memory");
  static std::atomic<uint64_t> devices{0};
  const cudaError_t allowed = allow_smem(kern, smem, devices);
  if (allowed != cudaSuccess) return (int)allowed;
  const AttnSplitParams AP{P, wait_tries(wait_ns), wait_status()};
  B200_RETURN_IF(AP.wait_status == nullptr, B200_ERR_DRIVER);
  if (!SHARED) {
    launch_pdl(kern, grid, dim3(kAsThreads), (size_t)smem, stream, AP);
    return finish_launch();
  }
  constexpr unsigned ctas = kAsParts;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid.x * ctas), cfg.blockDim = dim3(kAsThreads), cfg.dynamicSmemBytes = smem, cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ctas, attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr, cfg.numAttrs = pdl_enabled() ? 2 : 1;
  cudaLaunchKernelEx(&cfg, kern, AP);
  return finish_launch();
}

// A CTA's time is 11 us and 3.6 for every tile of 64 keys at heads of 128, so two share a row tile's keys where both find an SM, from six
// tiles on, or where one of them does and there are many tiles. us, alone / shared, paged:
//   8 heads over 2 of 128: 1 x 200 25.0 / 25.2, x 500 41.6 / 32.1, x 1000 70 / 47.2, x 2000 124 / 88.2;  [4 x 500 41.6 / 57.0, x 1000 86.6 / 145.3]
//   8 of 48: 1 x 500 23.8 / 20.6, x 1000 39.0 / 27.4;  [32 over 8 of 64: 1 x 500 26.2 / 33.0, x 1000 49.0 / 75.9]
// (four CTAs: 33.5, 66.6, 157.8 and 21.2, 39.7 on what two gain from)
static bool attn_split_shared(int64_t row_tiles, int most_tiles) {
  const int sms = sm_count();
  return (row_tiles * 2 <= sms && most_tiles >= 6) || (row_tiles <= sms && most_tiles >= 24);
}

int attn_split_launch(AttnTiledParams P, int num_seqs, int max_q, int64_t total_q, int64_t wait_ns, cudaStream_t stream) {
  B200_RETURN_IF(take_wait_status(), B200_ERR_WAIT);             // of an earlier call
  P.num_seqs = num_seqs;
  const dim3 grid((unsigned)(((int64_t)max_q * (P.H / P.G) + kAsM - 1) / kAsM * P.G * num_seqs));
  const bool shared = total_q > 0 && attn_split_shared((total_q * (P.H / P.G) + kAsM - 1) / kAsM * P.G, (max_q + kAsN - 1) / kAsN);
#define B200_AS(DK, DV) (shared ? attn_split_launch_as<DK, DV, true>(P, grid, wait_ns, stream) : attn_split_launch_as<DK, DV, false>(P, grid, wait_ns, stream))
  if (P.dim <= 64) return P.vdim <= 64 ? B200_AS(64, 64) : B200_AS(64, 128);
  return P.vdim <= 64 ? B200_AS(128, 64) : B200_AS(128, 128);
#undef B200_AS
}

}  // namespace b200
