// decode_small.cu -- paged decode attention (decode_attn.cu) of few rows in one launch: a cluster of CTAs per (row, kv head).
//
// What bounds a step of one or a few rows is not bytes but the chain launch -> length -> block table -> keys -> merge, and a second launch
// that merges what CTAs leave in a workspace costs more than the keys do. Here the CTAs of a (row, kv head) are a cluster and merge over
// distributed shared memory. A warp works by itself: it copies units of 16 keys and values into buffers of its own (cp.async, two units under
// way, nothing that other warps wait for), and the mathematics of a unit is that of paged_decode_kernel.
#include "decode_common.cuh"

namespace b200 {

constexpr int kSmallWarps = 8;
template <bool FP8>
constexpr int kSmallStages = FP8 ? 3 : 2;                // units of a warp under way

struct DecodeSmallParams {
  DecodeParams p;
  const void *k, *v;                                    // [num_blocks * block_size][Hkv * D]
  int num_blocks;
  float v_scale;
};

template <typename T, int D, bool FP8>
__global__ void __launch_bounds__(kSmallWarps * 32, FP8 || D == 64 ? 2 : 1)
decode_small_kernel(const __grid_constant__ DecodeSmallParams S) {
  const DecodeParams& p = S.p;
  constexpr int KSTEPS = D / 16, NT = D / 8, kStages = kSmallStages<FP8>;
  constexpr int kRow = FP8 ? D : 2 * D, kUnit = 16 * kRow;             // bytes of a key, of 16 keys
  extern __shared__ __align__(128) uint8_t small_smem[]; // [warps][stages][K, V]; then the warps' results
  __shared__ float s_o[8][D], s_m[8], s_l[8];            // this CTA's
  __shared__ float w_m[kSmallWarps][8], w_l[kSmallWarps][8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int b = blockIdx.z, kv_head = blockIdx.y, G = p.G;
  const uint32_t rank = cluster_rank(), ctas = cluster_size();
  pdl_wait();
  const int len = p.context_lens[b];
  const int units = len > 0 ? (len + 15) / 16 : 0, step = (int)ctas * kSmallWarps;
  uint8_t* buf = small_smem + warp * (kStages * 2 * kUnit);
  const uint32_t buf_at = smem_u32(buf);
  const uint8_t* kc = reinterpret_cast<const uint8_t*>(S.k) + (int64_t)kv_head * kRow;
  const uint8_t* vc = reinterpret_cast<const uint8_t*>(S.v) + (int64_t)kv_head * kRow;
  const int64_t row_bytes = (int64_t)p.Hkv * kRow;
  const int first = (int)rank + (int)ctas * warp;        // this warp's units: first, first + step, ...
  int looked_up = 0, rows = -1;                          // first cache row of unit looked_up + lane (-1: keys of no block are zero)
  auto look_up = [&](int n) {                            // 32 units at a time: a table entry per unit would cost each a trip to L2
    const int u = first + (n + lane) * step;
    looked_up = n, rows = -1;
    if (u < units) {
      const int tok = u * 16, entry = tok / p.block_size;                      // (a unit lies inside one block)
      const int blk = p.block_tables[(int64_t)b * p.bt_stride + entry];
      if (blk >= 0 && blk < S.num_blocks) rows = blk * p.block_size + (tok - entry * p.block_size);
    }
  };
  auto load = [&](int n, int stage) {                    // the warp's n-th unit. Keys past the length are zero
    const int u = first + n * step;
    if (u < units) {
      if (n - looked_up >= 32) look_up(n);
      const int row0 = __shfl_sync(0xffffffffu, rows, n - looked_up);
      const int valid = row0 >= 0 ? len - u * 16 : 0;
      const int64_t at = (int64_t)max(row0, 0) * row_bytes;
      const uint32_t to = buf_at + stage * (2 * kUnit);
#pragma unroll
      for (int i = 0; i < kUnit / 512; ++i) {
        const int e = i * 32 + lane, row = e / (kRow / 16), c = e % (kRow / 16);
        const uint32_t dst = kRow == 64 ? row * 64 + ((c ^ ((row >> 1) & 3)) << 4) : (c >> 3) * 2048 + row * 128 + (((c & 7) ^ (row & 7)) << 4);
        const bool ok = row < valid;
        const int64_t src = ok ? at + row * row_bytes + c * 16 : 0;
        cp_async_16(to + dst, kc + src, ok);
        cp_async_16(to + kUnit + dst, vc + src, ok);
      }
    }
    cp_async_commit();
  };
  look_up(0);
#pragma unroll
  for (int i = 0; i < kStages; ++i) load(i, i);

  const bool capped = p.cap > 0.f;
  const float sl2 = capped ? kLog2e : p.scale_log2;
  uint32_t qa[KSTEPS][2];
  {
    const T* qrow = reinterpret_cast<const T*>(p.q) + (int64_t)b * p.q_stride + (int64_t)(kv_head * G + g) * D;
#pragma unroll
    for (int ks = 0; ks < KSTEPS; ++ks) {
      if constexpr (FP8) {                               // the order of paged_decode_fp8_kernel: a lane has D / 4 neighbouring elements
        uint2 w = make_uint2(0u, 0u);
        if (g < G) w = *reinterpret_cast<const uint2*>(qrow + t4 * (D / 4) + 4 * ks);
        qa[ks][0] = to_f16x2<T>(w.x), qa[ks][1] = to_f16x2<T>(w.y);
        continue;
      }
      qa[ks][0] = g < G ? *reinterpret_cast<const uint32_t*>(qrow + ks * 16 + 2 * t4) : 0u;
      qa[ks][1] = g < G ? *reinterpret_cast<const uint32_t*>(qrow + ks * 16 + 8 + 2 * t4) : 0u;
    }
  }
  float o_acc[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n) o_acc[n][0] = o_acc[n][1] = o_acc[n][2] = o_acc[n][3] = 0.f;
  float m_run = -INFINITY, l_run = 0.f;
  const int k_tok = ((lane >> 4) << 3) + (lane & 7), k_half = (lane >> 3) & 1;       // ldmatrix: as in paged_decode_kernel
  const int v_tok = (((lane >> 3) & 1) << 3) + (lane & 7), v_dt = lane >> 4;
  for (int n = 0, stage = 0; first + n * step < units; ++n, stage = stage + 1 == kStages ? 0 : stage + 1) {
    cp_async_wait<kStages - 1>();
    __syncwarp();
    const uint32_t kb = buf_at + stage * (2 * kUnit), vb = kb + kUnit;
    float s[2][4];
#pragma unroll
    for (int t = 0; t < 2; ++t) s[t][0] = s[t][1] = s[t][2] = s[t][3] = 0.f;
    if constexpr (FP8) {
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int i = 0; i < KSTEPS / 4; ++i) {
          const int c = t4 * (D / 64) + i;
          const uint4 x = lds128(kb + (t * 8 + g) * kRow + ((D == 64 ? c ^ ((g >> 1) & 3) : c ^ g) << 4));
          const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
          for (int y = 0; y < 4; ++y)
            mma_16816<__half>(s[t], qa[4 * i + y][0], 0u, qa[4 * i + y][1], 0u, e4m3x2_to_f16x2(w[y] & 0xffffu), e4m3x2_to_f16x2(w[y] >> 16));
        }
    } else {
#pragma unroll
      for (int ks = 0; ks < KSTEPS; ++ks) {
        const int c16 = ((ks & 3) << 1) + k_half;
        uint32_t r0, r1, r2, r3;
        ldsm_x4(kb + (ks >> 2) * 2048 + k_tok * 128 + ((c16 ^ (k_tok & 7)) << 4), r0, r1, r2, r3);
        mma_16816<T>(s[0], qa[ks][0], 0u, qa[ks][1], 0u, r0, r1);
        mma_16816<T>(s[1], qa[ks][0], 0u, qa[ks][1], 0u, r2, r3);
      }
    }
    const int valid = len - (first + n * step) * 16;
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        if (capped) s[t][e] = p.cap * tanh_ex2(s[t][e] * p.cap_pre);
        if (t * 8 + 2 * t4 + e >= valid) s[t][e] = -INFINITY;
      }
    float mx = fmaxf(fmaxf(s[0][0], s[0][1]), fmaxf(s[1][0], s[1][1]));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float m_new = fmaxf(m_run, mx), alpha = ex2_approx((m_run - m_new) * sl2), mb = m_new * sl2;
    const float p00 = ex2_approx(fmaf(s[0][0], sl2, -mb)), p01 = ex2_approx(fmaf(s[0][1], sl2, -mb));
    const float p10 = ex2_approx(fmaf(s[1][0], sl2, -mb)), p11 = ex2_approx(fmaf(s[1][1], sl2, -mb));
    l_run = fmaf(l_run, alpha, (p00 + p01) + (p10 + p11));
    m_run = m_new;
    if (alpha != 1.f) {
#pragma unroll
      for (int t = 0; t < NT; ++t) o_acc[t][0] *= alpha, o_acc[t][1] *= alpha, o_acc[t][2] *= alpha, o_acc[t][3] *= alpha;
    }
    if constexpr (FP8) {
      const uint32_t pa0 = pack2<__half>(p00, p01), pa2 = pack2<__half>(p10, p11);
#pragma unroll
      for (int jp = 0; jp < D / 32; ++jp) {
        const int c = 2 * jp + v_dt;
        uint32_t r0, r1, r2, r3;
        ldsm_x4_trans(vb + v_tok * kRow + ((D == 64 ? c ^ ((v_tok >> 1) & 3) : c ^ (v_tok & 7)) << 4), r0, r1, r2, r3);
        const uint32_t e0 = __byte_perm(r0, r1, 0x6420), o0 = __byte_perm(r0, r1, 0x7531);
        const uint32_t e1 = __byte_perm(r2, r3, 0x6420), o1 = __byte_perm(r2, r3, 0x7531);
        mma_16816<__half>(o_acc[4 * jp + 0], pa0, 0u, pa2, 0u, e4m3x2_to_f16x2(e0 & 0xffffu), e4m3x2_to_f16x2(e0 >> 16));
        mma_16816<__half>(o_acc[4 * jp + 1], pa0, 0u, pa2, 0u, e4m3x2_to_f16x2(o0 & 0xffffu), e4m3x2_to_f16x2(o0 >> 16));
        mma_16816<__half>(o_acc[4 * jp + 2], pa0, 0u, pa2, 0u, e4m3x2_to_f16x2(e1 & 0xffffu), e4m3x2_to_f16x2(e1 >> 16));
        mma_16816<__half>(o_acc[4 * jp + 3], pa0, 0u, pa2, 0u, e4m3x2_to_f16x2(o1 & 0xffffu), e4m3x2_to_f16x2(o1 >> 16));
      }
    } else {
      // two 16-bit terms of the probabilities, the second in the rows of the tile that the group does not use
      const uint32_t pa0 = pack2<T>(p00, p01), pa2 = pack2<T>(p10, p11);
      const float2 h0 = unpack2<T>(pa0), h1 = unpack2<T>(pa2);
      const uint32_t pa1 = pack2<T>(p00 - h0.x, p01 - h0.y), pa3 = pack2<T>(p10 - h1.x, p11 - h1.y);
#pragma unroll
      for (int jp = 0; jp < NT / 2; ++jp) {
        const int dt = 2 * jp + v_dt;
        uint32_t r0, r1, r2, r3;
        ldsm_x4_trans(vb + (dt >> 3) * 2048 + v_tok * 128 + (((dt & 7) ^ (v_tok & 7)) << 4), r0, r1, r2, r3);
        mma_16816<T>(o_acc[2 * jp], pa0, pa1, pa2, pa3, r0, r1);
        mma_16816<T>(o_acc[2 * jp + 1], pa0, pa1, pa2, pa3, r2, r3);
      }
    }
    __syncwarp();
    load(n + kStages, stage);
  }
  cp_async_wait<0>();
  if constexpr (!FP8) {
    // the second term is left out where an infinite value made it 0 x inf or inf - inf
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (fabsf(o_acc[n][2 + e]) < INFINITY) o_acc[n][e] += o_acc[n][2 + e];
  }
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
  // ---- the warps of this CTA: each into its own buffer
  float* mine = reinterpret_cast<float*>(buf);           // [8][D]
  static_assert(8 * D * 4 <= kStages * 2 * kUnit, "a warp's result fits its buffers");
  if (FP8 && g < G) {
#pragma unroll
    for (int c = 0; c < D / 16; ++c)
      *reinterpret_cast<float4*>(mine + g * D + 16 * c + 4 * t4) = make_float4(o_acc[2 * c][0], o_acc[2 * c + 1][0], o_acc[2 * c][1], o_acc[2 * c + 1][1]);
  } else if (g < G) {
#pragma unroll
    for (int n = 0; n < NT; ++n) *reinterpret_cast<float2*>(mine + g * D + n * 8 + 2 * t4) = make_float2(o_acc[n][0], o_acc[n][1]);
  }
  if (t4 == 0) w_m[warp][g] = m_run * sl2, w_l[warp][g] = l_run;       // running maximum in the exp2 domain
  __syncthreads();
  for (int e = threadIdx.x; e < G * D; e += kSmallWarps * 32) {
    const int r = e / D;
    float m = -INFINITY, l = 0.f, o = 0.f;
#pragma unroll
    for (int w = 0; w < kSmallWarps; ++w) m = fmaxf(m, w_m[w][r]);
#pragma unroll
    for (int w = 0; w < kSmallWarps; ++w) {
      const float x = w_m[w][r], f = x == -INFINITY ? 0.f : ex2_approx(x - m);
      l = fmaf(w_l[w][r], f, l);
      if (x != -INFINITY) o = fmaf(reinterpret_cast<const float*>(small_smem + w * (kStages * 2 * kUnit))[e], f, o);
    }
    s_o[0][e] = o;
    if (e % D == 0) s_m[r] = m, s_l[r] = l;
  }
  // ---- the CTAs of the cluster: each a share of the columns
  cluster_arrive();
  cluster_wait();
  const int total = G * D;
  for (int e0 = (int)rank * 2 + threadIdx.x * 2 * (int)ctas; e0 < total; e0 += kSmallWarps * 32 * 2 * (int)ctas) {
    const int r = e0 / D;
    const uint32_t am = smem_u32(&s_m[r]), al = smem_u32(&s_l[r]), ao = smem_u32(&s_o[0][e0]);
    float m = -INFINITY;
    for (uint32_t c = 0; c < ctas; ++c) m = fmaxf(m, ld_peer(am, c));
    float l = 0.f, o0 = 0.f, o1 = 0.f;
#pragma unroll 4
    for (uint32_t c = 0; c < ctas; ++c) {
      const float x = ld_peer(am, c), f = x == -INFINITY ? 0.f : ex2_approx(x - m);
      l = fmaf(ld_peer(al, c), f, l), o0 = fmaf(ld_peer(ao, c), f, o0), o1 = fmaf(ld_peer(ao + 4, c), f, o1);
    }
    if (p.sink != nullptr && len > 0) l += ex2_approx(p.sink[kv_head * G + r] * kLog2e - m);
    const float inv = len > 0 ? S.v_scale / l : 0.f;
    T* out = reinterpret_cast<T*>(p.out) + (int64_t)b * p.out_stride + (int64_t)kv_head * total + e0;
    *reinterpret_cast<uint32_t*>(out) = len > 0 ? pack2<T>(o0 * inv, o1 * inv) : 0u;
  }
  cluster_arrive();                                      // nobody leaves while others read
  cluster_wait();
}

template <typename T, int D, bool FP8>
static int decode_small_launch_as(const DecodeSmallParams& S, int ctas, cudaStream_t stream) {
  auto kern = decode_small_kernel<T, D, FP8>;
  constexpr int smem = kSmallWarps * kSmallStages<FP8> * 2 * 16 * D * (FP8 ? 1 : 2);
  static std::atomic<uint64_t> devices{0};
  cudaError_t e = allow_smem(kern, smem, devices);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)ctas, (unsigned)S.p.Hkv, (unsigned)S.p.batch);
  cfg.blockDim = dim3(kSmallWarps * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ctas, attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr, cfg.numAttrs = pdl_enabled() ? 2 : 1;
  cudaLaunchKernelEx(&cfg, kern, S);
  return finish_launch();
}

// us, paged_decode_kernel and its combine / this kernel, contexts of 40 to 100 % of the length named, launches of a graph (heads over kv heads of
// a size; the same number of pairs of other heads within 10 %):
//   16 / 8 of 128:  1 row x 100 6.7 / 4.3, x 500 7.8 / 4.9, x 1000 9.0 / 5.8, x 2000 9.9 / 7.2, x 4000 11.7 / 9.4;  2 x 1000 9.7 / 6.5, x 4000
//                   13.3 / 12.8;  4 x 1000 11.6 / 7.1, x 4000 16.5 / 14.3;  8 x 500 11.3 / 7.1, x 2000 16.2 / 14.2, [x 4000 22.8 / 22.9];  16 x 500
//                   12.9 / 9.4, x 1000 16.0 / 13.9, [x 2000 22.0 / 22.6];  [32 x 100 11.1 / 9.5, x 500 16.1 / 17.1]
//   8 / 2 of 128:   1 x 1000 8.3 / 6.2, x 4000 10.1 / 9.5, [x 8000 12.0 / 13.7]
//   32 / 8 of 64:   1 x 1000 8.4 / 5.1, x 8000 12.5 / 11.2;  4 x 1000 12.2 / 7.0, x 8000 18.6 / 15.1;  16 x 2000 18.1 / 14.1;  32 x 1000 18.0 / 13.8
//   8 / 8 of 64:    1 x 1000 7.7 / 4.5, x 8000 12.4 / 10.6;  8 x 4000 15.1 / 13.9, [x 8000 21.5 / 23.0];  32 x 1000 14.7 / 13.4, [x 2000 20.8 / 21.9]
// An SM takes about 70 bytes per ns, and one CTA (heads of 64: two), so what counts is the bytes per CTA: 131072 tokens of kv
// heads of 128 or 262144 of 64 in all, on up to 128 or 256 CTAs (clusters of 8 of 128 pack 64). More CTAs than eight warps' units of 16 keys
// only wait for one another (1 row x 100: 4.3 with one, 4.9 with eight).
// An e4m3 cache, two CTAs per SM: 16 / 8 of 128: 1 x 1000 9.3 / 5.7, x 4000 12.1 / 9.4;  4 x 4000 14.3 / 13.5;  8 x 2000 14.1 / 12.9, [x 4000 19.1 /
// 19.3];  16 x 1000 13.8 / 12.8, [x 2000 18.4 / 18.9];  32 x 500 13.9 / 12.0, [x 1000 18.4 / 18.4], [64 x 500 18.6 / 19.7];  32 / 8 of 64: 1 x 1000
// 10.7 / 4.7;  8 x 4000 16.1 / 11.6;  16 x 4000 20.0 / 17.2;  32 x 2000 20.0 / 16.5;  64 x 1000 21.3 / 19.2, [x 2000 29.2 / 29.0].
int decode_small_ctas(int64_t pairs, int64_t width, int dim, bool fp8) {
  const int64_t tokens = dim == 128 ? 128 << 10 : fp8 ? 512 << 10 : 256 << 10, most = !fp8 && dim == 128 ? 128 : fp8 && dim == 64 ? 512 : 256;
  if (width <= 0 || width > (dim == 128 ? 4096 : 8192) || pairs > most || pairs * width > tokens) return 0;
  const bool one = !fp8 && dim == 128;                   // CTA per SM
  int ctas = pairs <= (one ? 8 : 32) ? 8 : pairs <= (one ? 32 : 64) ? 4 : pairs <= (one ? 64 : 128) ? 2 : 1;
  while (ctas > 1 && (ctas / 2) * kSmallWarps * 16 >= width) ctas /= 2;
  return ctas;
}

template <bool FP8>
static int decode_small_launch_for(const DecodeSmallParams& S, int dim, int dtype, int ctas, cudaStream_t stream) {
  if (dtype == B200_DTYPE_BF16)
    return dim == 128 ? decode_small_launch_as<__nv_bfloat16, 128, FP8>(S, ctas, stream) : decode_small_launch_as<__nv_bfloat16, 64, FP8>(S, ctas, stream);
  return dim == 128 ? decode_small_launch_as<__half, 128, FP8>(S, ctas, stream) : decode_small_launch_as<__half, 64, FP8>(S, ctas, stream);
}
int decode_small_launch(const DecodeParams& p, const void* k, const void* v, int num_blocks, int dim, int dtype, int ctas, cudaStream_t stream) {
  return decode_small_launch_for<false>(DecodeSmallParams{p, k, v, num_blocks, 1.f}, dim, dtype, ctas, stream);
}
int decode_small_fp8_launch(const DecodeParams& p, const void* k, const void* v, int num_blocks, int dim, float v_scale, int dtype, int ctas,
                            cudaStream_t stream) {
  return decode_small_launch_for<true>(DecodeSmallParams{p, k, v, num_blocks, v_scale}, dim, dtype, ctas, stream);
}

}  // namespace b200
