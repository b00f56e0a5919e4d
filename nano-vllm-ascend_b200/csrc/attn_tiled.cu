// attn_tiled.cu -- prompt portions of attn_generic (seq_mixers.cu) in true 32-bit arithmetic, as register-tiled products.
//
// What it computes is attn_generic_kernel's job to the letter: causal softmax attention for any element type (16-bit inputs
// are widened as they are staged), packed or paged keys, windows with kept first tokens, chunks, capped scores, sinks,
// output gates, values inside the key rows.
//
// Bound: the fp32 FMA pipes (128 per clock and SM; no TF32, no 16-bit split). The kernel that serves single tokens reads two
// shared-memory words per FMA, which bound it at 2.6 TFLOP/s of 74. Here CTA = 64 rows of one (sequence, kv head) -- row r is
// token r / rep, query head g * rep + r % rep, so all heads of a group share a key tile -- against 64 keys at a time, 256
// threads. A thread owns 4 x 4 scores (rows 4 ty .. 4 ty + 3, keys tx, tx + 16, ..: 8 16-byte shared loads per 64 FMAs) and 4
// rows x 4 VC output columns (1 + VC loads per 16 VC FMAs), both as packed fma.rn.f32x2, which halve the issue slots: the
// scores' pairs run along the head dimension (two partial sums per score), the outputs' along the columns. The 16
// threads of a row are the lanes of a half warp, so row maxima are four shuffles and row sums stay per thread until the end.
// K(j + 1) is copied (cp.async for fp32 rows) under the softmax and P V of tile j, V(j + 1) under the scores of tile j + 1.
// Rows of Q, K and P are unpadded with their 16-byte chunks XOR-swizzled, so that 64 x 64 tiles of 128-wide heads take 112 KB
// and two CTAs share an SM: one computes while the other waits at its barriers.
// Measured (4 ragged prompts of 700-1024 tokens, 8 heads over 2 of 128, fp32, paged): 2427 us -> 352 us with the row tiles of one
// sequence after the other, 298 us with the longest tiles of all first, 291 us (21.5 TFLOP/s) where warps whose rows lie past the
// span only copy and the last tile ends at its last key.
#include "seq_common.cuh"
#include "attn_tiled.cuh"

namespace b200 {

constexpr int kTM = 64, kTN = 64, kTThreads = 256;

// packed pair of fp32 (two registers); d = a * b + c per half
__device__ __forceinline__ void fma2(float2& c, const float2 a, const float2 b) {
  uint64_t& cc = reinterpret_cast<uint64_t&>(c);
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(cc) : "l"(reinterpret_cast<const uint64_t&>(a)), "l"(reinterpret_cast<const uint64_t&>(b)));
}

template <typename T, int VC, bool VEC>
__global__ void __launch_bounds__(kTThreads, VC <= 2 ? 2 : 1)
attn_tiled_kernel(const AttnTiledParams P) {
  extern __shared__ __align__(16) float smem[];
  pdl_wait();
  // the last row tiles see the most keys: those of every (sequence, kv head) start first
  const int units = P.G * P.num_seqs, tile = (int)(gridDim.x / units - 1 - blockIdx.x / units), unit = blockIdx.x % units;
  const int s = unit / P.G, g = unit % P.G;
  const SeqSpan sp = seq_span(P.cu_q, P.cu_k, nullptr, s);
  const int rep = P.H / P.G, rows = sp.q_len * rep;
  const int r0 = tile * kTM;
  if (r0 >= rows) return;
  const int dim = P.dim, vdim = P.vdim, QC = P.chunks;              // QC: 16-byte chunks per staged row, a multiple of 8
  float* sq = smem;                                                 // [64][QC] chunks
  float* sk = sq + kTM * QC * 4;                                    // [64][QC] chunks
  float* sv = sk + kTN * QC * 4;                                    // [64][64 VC] floats
  float* sp_ = sv + kTN * 64 * VC;                                  // [64 keys][16] chunks of 4 rows
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const T* kb = reinterpret_cast<const T*>(P.k) + (int64_t)g * dim;
  const T* vb = P.v != nullptr ? reinterpret_cast<const T*>(P.v) + (int64_t)g * vdim : kb;
  const int64_t v_stride = P.v != nullptr ? P.v_stride : P.k_stride;
  const int64_t k_base = P.block_tables == nullptr ? P.cu_k[s] : 0;
  const int* table = P.block_tables != nullptr ? P.block_tables + (int64_t)s * P.bt_stride : nullptr;
  auto key_row = [&](int key) -> int64_t {
    return table != nullptr ? (int64_t)table[key / P.block_size] * P.block_size + key % P.block_size : k_base + key;
  };
  auto swz = [&](int row, int c) { return (row * QC + (c ^ (row & 7))) * 4; };

  // ---- staging: nr rows of `width` columns as fp32, zero past them. Warp w copies rows 8 w .. 8 w + 7, a lane one 16-byte
  // chunk at a time; the eight row offsets (a division and a table look-up each) are found by eight lanes at once
  const int warp = tid >> 5, lane = tid & 31;
  const bool live = r0 + 8 * warp < rows;                           // warp-uniform: some row of this warp exists
  auto stage = [&](float* dst, bool swizzled, int chunks, int width, int nr, const T* base, auto row_offset) {
    const int mine = 8 * warp + (lane & 7);
    const int64_t offset = mine < nr ? row_offset(mine) : 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = 8 * warp + i;
      const T* from_row = base + __shfl_sync(0xffffffffu, offset, i);
      for (int c = lane; c < chunks; c += 32) {
        const int col = c * 4;
        float* to = dst + (swizzled ? swz(r, c) : (r * chunks + c) * 4);
        const bool ok = r < nr && col < width;
        if constexpr (VEC && sizeof(T) == 4) {
          cp_async_16(smem_u32(to), ok ? (const void*)(from_row + col) : (const void*)P.q, ok);
        } else {
          float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
          if (ok) {
            const T* from = from_row + col;
            if constexpr (VEC) {                                   // 16-bit rows, 8-byte aligned chunks
              const uint2 u = *reinterpret_cast<const uint2*>(from);
              const float2 a = unpack2<T>(u.x), b = unpack2<T>(u.y);
              x = make_float4(a.x, a.y, b.x, b.y);
            } else {
              x.x = to_f32<T>(from[0]);
              if (col + 1 < width) x.y = to_f32<T>(from[1]);
              if (col + 2 < width) x.z = to_f32<T>(from[2]);
              if (col + 3 < width) x.w = to_f32<T>(from[3]);
            }
          }
          *reinterpret_cast<float4*>(to) = x;
        }
      }
    }
    cp_async_commit();
  };
  stage(sq, true, QC, dim, min(kTM, rows - r0), reinterpret_cast<const T*>(P.q), [&](int r) -> int64_t {
    const int tok = (r0 + r) / rep;
    return (int64_t)(sp.q_start + tok) * P.q_stride + (int64_t)(g * rep + (r0 + r) - tok * rep) * dim;
  });

  auto seen_from = [&](int p) { return P.window > 0 ? max(0, p - P.window + 1) : P.chunk > 0 ? p / P.chunk * P.chunk : 0; };
  const int min_pos = sp.first_pos() + r0 / rep, max_pos = sp.first_pos() + (min(r0 + kTM, rows) - 1) / rep;
  const int first_key = seen_from(min_pos);
  const int kept = min(P.keep_first, first_key);
  auto next_tile = [&](int j0) { return (j0 < kept && j0 + kTN >= kept) ? first_key : j0 + kTN; };
  auto tile_keys = [&](int j0) { return min(kTN, (j0 < kept ? kept : max_pos + 1) - j0); };
  auto load_k = [&](int j0) {
    stage(sk, true, QC, dim, tile_keys(j0), kb, [&](int j) { return key_row(j0 + j) * P.k_stride; });
  };
  auto load_v = [&](int j0) {
    stage(sv, false, 16 * VC, vdim, tile_keys(j0), vb, [&](int j) { return key_row(j0 + j) * v_stride; });
  };

  int pos[4], lo[4];
  float m[4], l[4];
  float2 acc[4][2 * VC];                              // columns 64 c + 4 tx + {0, 1}, {2, 3}
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = min(r0 + 4 * ty + i, rows - 1);
    pos[i] = sp.first_pos() + r / rep;
    lo[i] = seen_from(pos[i]);
    // a sink is one more entry of the softmax that has a logit and no value: the running state starts from it
    m[i] = P.sink != nullptr ? P.sink[g * rep + r % rep] : -INFINITY;
    l[i] = P.sink != nullptr && tx == 0 ? 1.f : 0.f;
#pragma unroll
    for (int c = 0; c < 2 * VC; ++c) acc[i][c] = make_float2(0.f, 0.f);
  }

  int j0 = kept > 0 ? 0 : first_key;
  if (j0 <= max_pos) {
    load_k(j0);
    load_v(j0);
  }
  while (j0 <= max_pos) {
    const int nk = tile_keys(j0), j_next = next_tile(j0);
    cp_async_wait<1>();                               // Q and K(j) have landed (this thread's copies), V(j) may be under way
    __syncthreads();
    // ---- scores
    float2 d[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) d[i][j] = make_float2(0.f, 0.f);
    // the swizzle of a thread's keys (tx & 7, for all four) and rows ((4 ty + i) & 7 = 4 (ty & 1) + i) is an XOR of the chunk
    const int steps = (dim + 3) >> 2;
    const float4* kt = reinterpret_cast<const float4*>(sk) + tx * QC;
    const float4* qt = reinterpret_cast<const float4*>(sq) + 4 * ty * QC;
    if (live) {                                       // (warps whose rows all lie past the span only copy)
#pragma unroll 2
      for (int c = 0; c < steps; ++c) {
        float4 kk[4];
        const int ck = c ^ (tx & 7), cq = c ^ (4 * (ty & 1));
#pragma unroll
        for (int j = 0; j < 4; ++j) kk[j] = kt[16 * j * QC + ck];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 qq = qt[i * QC + (cq ^ i)];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            fma2(d[i][j], make_float2(qq.x, qq.y), make_float2(kk[j].x, kk[j].y));
            fma2(d[i][j], make_float2(qq.z, qq.w), make_float2(kk[j].z, kk[j].w));
          }
        }
      }
    }
    __syncthreads();                                  // K(j) is consumed
    if (j_next <= max_pos) load_k(j_next);
    else cp_async_commit();
    // ---- softmax. A masked pair's probability is stored as -0.0 (a visible one is never negative)
    const bool masked = j0 + nk - 1 > min_pos || nk < kTN || P.window > 0 || P.chunk > 0;
    if (live) {
      float p[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float mx = -INFINITY;
        bool seen[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int off = tx + 16 * j, key = j0 + off;
          float sc = (d[i][j].x + d[i][j].y) * P.scale;
          if (P.softcap > 0.f) sc = P.softcap * tanhf(sc / P.softcap);
          seen[j] = !masked || (off < nk && key <= pos[i] && (key >= lo[i] || key < P.keep_first));
          p[i][j] = seen[j] ? sc : -INFINITY;
          mx = fmaxf(mx, p[i][j]);
        }
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float m_new = fmaxf(m[i], mx);
        const float corr = m_new == -INFINITY ? 1.f : expf(m[i] - m_new);   // nothing visible so far: nothing to rescale
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float e = p[i][j] == -INFINITY ? 0.f : expf(p[i][j] - m_new);
          sum += e;
          p[i][j] = seen[j] ? e : -0.f;
        }
        l[i] = l[i] * corr + sum;
        m[i] = m_new;
#pragma unroll
        for (int c = 0; c < 2 * VC; ++c) acc[i][c].x *= corr, acc[i][c].y *= corr;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = tx + 16 * j;
        *reinterpret_cast<float4*>(sp_ + (key * 16 + (ty ^ (key & 7))) * 4) = make_float4(p[0][j], p[1][j], p[2][j], p[3][j]);
      }
    }
    cp_async_wait<1>();                               // V(j) has landed (K(j + 1) may be under way)
    // a value that is not finite must not reach rows that do not see its key (0 x inf): such tiles skip masked pairs
    bool wild = false;
    if (masked) {
      __syncthreads();
      for (int e = tid; e < nk * 16 * VC; e += kTThreads) {
        const float4 x = *reinterpret_cast<const float4*>(sv + e * 4);
        wild |= !(isfinite(x.x) && isfinite(x.y) && isfinite(x.z) && isfinite(x.w));
      }
    }
    wild = __syncthreads_or(wild) != 0;
    // ---- O += P V
    auto row_key = [&](int key, bool guard) {
      const float4 pp = *reinterpret_cast<const float4*>(sp_ + (key * 16 + (ty ^ (key & 7))) * 4);
      const float pr[4] = {pp.x, pp.y, pp.z, pp.w};
#pragma unroll
      for (int c = 0; c < VC; ++c) {
        const float4 vv = *reinterpret_cast<const float4*>(sv + key * 64 * VC + 64 * c + 4 * tx);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (guard && __float_as_uint(pr[i]) == 0x80000000u) continue;
          fma2(acc[i][2 * c], make_float2(pr[i], pr[i]), make_float2(vv.x, vv.y));
          fma2(acc[i][2 * c + 1], make_float2(pr[i], pr[i]), make_float2(vv.z, vv.w));
        }
      }
    };
    if (!live) {
    } else if (wild) {
      for (int key = 0; key < nk; ++key) row_key(key, true);
    } else {
#pragma unroll 4
      for (int key = 0, end = (nk + 3) & ~3; key < end; ++key) row_key(key, false);   // rows past nk are zero, their p too
    }
    __syncthreads();                                  // V(j) and P(j) are consumed
    if (j_next <= max_pos) load_v(j_next);
    else cp_async_commit();
    j0 = j_next;
  }
  cp_async_wait<0>();

#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], o);
    const int r = r0 + 4 * ty + i;
    if (r >= rows) continue;
    const int tok = r / rep, head = g * rep + r - tok * rep;
    float inv = 1.0f / l[i];
    if (P.gate != nullptr)
      inv *= sigmoid_f(to_f32<T>(reinterpret_cast<const T*>(P.gate)[(int64_t)(sp.q_start + tok) * P.gate_stride + head]));
    T* o = reinterpret_cast<T*>(P.out) + (int64_t)(sp.q_start + tok) * ((int64_t)P.H * vdim) + (int64_t)head * vdim;
#pragma unroll
    for (int c = 0; c < 4 * VC; ++c) {
      const int col = 64 * (c >> 2) + 4 * tx + (c & 3);
      const float x = (c & 1) ? acc[i][c >> 1].y : acc[i][c >> 1].x;
      if (col < vdim) o[col] = from_f32<T>(x * inv);
    }
  }
}

static size_t attn_tiled_smem(int dim, int vdim) {
  const int qc = ((dim + 3) / 4 + 7) / 8 * 8, vc = vdim <= 64 ? 1 : vdim <= 128 ? 2 : 4;
  return (size_t)(2 * kTM * qc * 4 + kTN * 64 * vc + kTN * kTM) * sizeof(float);
}

// Spans of at least 16 rows (tokens x heads per group) somewhere in the step: below that most of a 64-row tile would be
// padding (one token of 8 heads per group: 56 of 64 rows), and the 8-row kernel spreads over more CTAs. Values up to 256
// columns (the accumulators of a thread), rows that fit shared memory; everything else stays on the 8-row kernel.
// Which spans a step mixes does not count: a span's single token takes one warp of its CTA, and its keys come 64 at a time. us,
// 8-row kernel / this one, fp32, 8 heads of 128 over 8, 2 and 1 kv heads: a portion of 256 tokens and 200 single tokens on 1000
// keys 2414 / 872, 1038 / 304, 1109 / 177; 512 and 64 on 2000 1993 / 610, 1790 / 337, 1848 / 335; 16 spans of 16 tokens on 500
// keys 410 / 77, 287 / 101, 287 / 101; 64 of 16 on 16 32.8 / 26.4, 29.7 / 15.2, 28.9 / 15.0; one of 33, heads of 32, 10.1 / 10.6,
// 10.0 / 10.6, 10.9 / 10.4.
bool attn_tiled_fits(int max_q, int rep, int G, int num_seqs, int dim, int vdim) {
  const int64_t tiles = ((int64_t)max_q * rep + kTM - 1) / kTM;
  return (int64_t)max_q * rep >= 16 && max_q > 1 && vdim <= 256 && attn_tiled_smem(dim, vdim) <= 220 * 1024 &&
         tiles * G <= 0x7fffffff / num_seqs;                         // one grid dimension holds them all
}

template <typename T, int VC, bool VEC>
static int attn_tiled_launch_as(const AttnTiledParams& P, dim3 grid, size_t smem, cudaStream_t stream) {
  auto kern = attn_tiled_kernel<T, VC, VEC>;
  static std::atomic<uint64_t> devices{0};
  const cudaError_t allowed = allow_smem(kern, 220 * 1024, devices);
  if (allowed != cudaSuccess) return (int)allowed;
  launch_pdl(kern, grid, dim3(kTThreads), smem, stream, P);
  return finish_launch();
}

int attn_tiled_launch(AttnTiledParams P, int num_seqs, int max_q, int dtype, cudaStream_t stream) {
  const int rep = P.H / P.G;
  P.chunks = ((P.dim + 3) / 4 + 7) / 8 * 8;
  P.num_seqs = num_seqs;
  const dim3 grid((unsigned)(((int64_t)max_q * rep + kTM - 1) / kTM * P.G * num_seqs));
  const size_t smem = attn_tiled_smem(P.dim, P.vdim);
  B200_DISPATCH_3(dtype, T, {
    // vector form: 4-element chunks of every row lie on 4-element boundaries
    const uintptr_t bytes = 4 * sizeof(T) - 1;
    const bool vec = P.dim % 4 == 0 && P.vdim % 4 == 0 && P.q_stride % 4 == 0 && P.k_stride % 4 == 0 &&
                     (P.v == nullptr || P.v_stride % 4 == 0) &&
                     ((reinterpret_cast<uintptr_t>(P.q) | reinterpret_cast<uintptr_t>(P.k) | reinterpret_cast<uintptr_t>(P.v)) & bytes) == 0;
    if (P.vdim <= 64) return vec ? attn_tiled_launch_as<T, 1, true>(P, grid, smem, stream) : attn_tiled_launch_as<T, 1, false>(P, grid, smem, stream);
    if (P.vdim <= 128) return vec ? attn_tiled_launch_as<T, 2, true>(P, grid, smem, stream) : attn_tiled_launch_as<T, 2, false>(P, grid, smem, stream);
    return vec ? attn_tiled_launch_as<T, 4, true>(P, grid, smem, stream) : attn_tiled_launch_as<T, 4, false>(P, grid, smem, stream);
  });
  return B200_OK;
}

}  // namespace b200
