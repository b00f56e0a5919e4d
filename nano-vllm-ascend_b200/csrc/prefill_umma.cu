// prefill_umma.cu -- K4/K5 on the 5th-generation tensor cores: varlen causal flash-attention with
// tcgen05.mma (UMMA), accumulators AND the probability tile in TMEM, operands staged by TMA.
//
// Replaces the same reference call sites as prefill_attn.cu (layers/attention.py:46-59,
// layers/attention_ori.py:63-70). Same semantics: bottom-right causal mask, packed K/V or paged K/V
// through block_tables.
//
// Shape of the kernel ("FA4 shape"; measured instruction costs on this part: SS M128 N64 K16 75
// cycles, SS N128 107, TS N128 74).
// Template parameter QT = 128-row query tiles per CTA, chosen per launch (prefill_query_tiles).
// QT = 2: two query tiles t = 0, 1 that ping-pong and share every K / V tile: 128 rows of two heads of one kv head, or (heads
//   that come alone) 256 rows of one head.
//   warps 0-3 / 4-7   softmax warpgroup of tile t, one thread per query row (= one TMEM lane): reads
//                     S[t] (128 fp32 columns) with tcgen05.ld, fp32 online softmax in the exp2 domain
//                     with lazy rescale of O (only when the row max grew by > 2^8), writes P as packed
//                     16-bit pairs OVER the first 64 columns of S[t] with tcgen05.st, in two halves of 64
//                     keys so that the PV product of the first half runs under the exponentials of the second
//   warp 8            TMA producers: lane 0 loads Q and runs a 2-stage K ring, lane 1 a 2-stage V ring
//                     (128-key tiles)
//   warp 9            MMA issuer (one elected lane):
//                       S[t]  = Q[t] K^T     8 x tcgen05.mma SS  (M128 N128 K16), K-major operands
//                       O[t] += P[t] V       8 x tcgen05.mma TS  (M128 N=D  K16), A = P from TMEM,
//                                            B = V MN-major straight from its [key][d] rows
//                     issue order  S0(0) S1(0) | PV0(0) S0(1) PV1(0) S1(1) | PV0(1) S0(2) ...
//                     so that the tensor pipe works on tile 1-t while warpgroup t is in its softmax.
//   warp 10           finds the work items of the softmax warps, one ahead
//   warp 11           gives its registers away (prefill_threads)
//   TMEM (512 columns): O[t] at 128 t, S[t] at 256 + 128 t, P[t] aliases S[t] columns [0, 64).
//   Shared memory: Q 2 x 32 KiB + K 2 x 32 KiB + V 2 x 32 KiB = 192 KiB at D = 128; one CTA per SM.
// QT = 1: one query tile per CTA: warps 0-3 softmax, warp 4 TMA, warp 5 MMA, warp 6 items; single-stage K / V rings; 256
//   TMEM columns (O at 0, S at 128), 105 KiB of shared memory -> two CTAs per SM.
// A CTA walks several work items (Q of the next one is loaded, and its first S computed, under the epilogue of the one
// before); a row's sizes live in shared memory, since 128 scores leave no registers for them. Sums and products of scores are
// packed fp32 pairs, row maxima four chains. What bounds it (16 x 1024 tokens, 16 heads over 8 of 128, inputs that rotate: 104.5 us =
// 657 TFLOP/s; 129 us with one item per CTA and one head): the chain S -> softmax -> P V -> S of a tile, 3300 to 3700 cycles of which
// the tensor pipe works 1448 for each of two tiles, and what goes with an item -- first loads, drain, epilogue -- at about 3 us
// (1024 items of 31 pair tiles per CTA against as many of 114).
// Hazards: S[t](j+1) overwrites the columns PV[t](j) reads P from -- both are tcgen05.mma of the same
// issuing thread and execute in issue order; softmax(j+1) of tile t starts only after S[t](j+1) has
// completed, hence after PV[t](j) has.
//
// Sliding window with kept first tokens (window > 0): position i sees j <= i with i - j < window or j < keep_first. A CTA
// visits the tiles of the kept keys, then those from its first row's window on; the tiles between are skipped by
// index (`kept`, `skip`), the borders are masked element by element. Chunks (chunk > 0: position i sees j <= i of its own
// chunk) run the same way, with the chunk's start in place of the window's.
// Keys and values may have different head sizes (DK in {64, 128, 192}, DV in {64, 128}; 192: one CTA per SM, single-stage
// rings); D below stands for the one that applies.
//
// Split-KV (few, long rows: the prefix-cache-hit form q_len << k_len): when the grid
// would leave most SMs idle, `kv_splits` CTAs share one (sequence, head, 256 rows), each takes a
// contiguous range of key tiles and writes un-normalised (O, m, l) partials to a caller-provided
// workspace; prefill_combine_kernel merges them. Flops: 4 * Lq * Lk * D per (sequence, head) before
// causal skipping; tensor-pipe bound.
#include "umma.cuh"

namespace b200 {

struct PrefillUmmaParams {
  const int32_t* cu_q;
  const int32_t* cu_k;
  const int32_t* block_tables;  // nullptr => packed K/V
  void* out;
  int64_t out_stride;
  int H, G, block_size, bt_stride;
  int kv_rows_box;   // rows per K/V TMA op (128 packed; min(block_size, 128) paged)
  int k_split, v_split;   // 1: each TMA op carries a single 64-wide chunk (paged, rows_box < 128)
  int pair;          // QT = 2: the two query tiles are 128 rows of two heads that share K and V, not 256 rows of one head
  int m_tiles, num_seqs;   // row tiles of the longest sequence, sequences: the items are m_tiles x kv_splits x H x num_seqs
  int ordered;       // the sequences are listed by length (several items per CTA), not in their own order
  int kv_splits;     // CTAs sharing one (sequence, head, 256 rows) along the keys; 1 = no split
  float* part_o;     // kv_splits > 1: [total_q][H][kv_splits][D] un-normalised O
  float* part_ml;    // kv_splits > 1: [total_q][H][kv_splits][2]  (row max in the exp2 domain, row sum)
  float scale_log2;
  // optional: scores capped by cap * tanh(scale * s / cap) (cap_pre = scale / cap; 0 = off), and a sink logit per
  // query head (fp32 [H], natural-log units) that joins the softmax denominator without a value
  float cap = 0.f, cap_pre = 0.f;
  // up to cap_short caps, the short polynomial (kCapShort) times cap_scale = cap * cap_pre. (The kernel makes its coefficients of these: 32 bytes of
  // them among the arguments cost every call 0.5 us of host time, 15.6 for 15.1)
  float cap_scale = 0.f, cap_short = -1.f;
  const float* sink = nullptr;
  int window = 0, keep_first = 0;   // window 0: every earlier key
  int chunk = 0;                    // chunk > 0: only keys of the row's own chunk (counted from position 0)

  __device__ __forceinline__ bool limited() const { return window > 0 || chunk > 0; }
  // first key that position `pos` sees besides the kept ones (window or chunk; may be negative)
  __device__ __forceinline__ int seen_from(int pos) const { return window > 0 ? pos - window + 1 : pos / chunk * chunk; }
};

constexpr int kUBM = 128, kUBN = 128;

// tanh(y) = y (1 + c1 y^2 + c2 y^4 + c3 y^6) up to y = kCapShortTo, off by 1.4e-10 at most: the minimax polynomial of its form (Remez exchange;
// cutting the series off after as many terms would leave 1.5e-8). In fp32, scores are off by 3.1e-8 (caps of 4 and 30) to 3.8e-8 (0.7) on
// average, like those of the long polynomial below (3.1e-8, 3.1e-8 and 3.9e-8)
constexpr double kCapShort[4] = {1., -0.33333323867490996, 0.13331341300491710, -0.05277317222556861};
constexpr float kCapShortTo = 0.17f;
constexpr int kOrderSeqs = 256;     // sequences that a launch orders by length
constexpr int kItems = 2;           // slots of work items: the one in hand and the next

// QT = query tiles per CTA. QT = 2: the layout described above (one CTA per SM, two tiles ping-pong, K/V
// tiles shared, 2-stage rings). QT = 1: one 128-row tile per CTA, single-stage K/V rings (K(j+1) is loaded
// under softmax(j) + PV(j), V(j+1) under S(j+1) + softmax(j+1) -- the chain leaves the time), 97 KB of
// shared memory, 256 TMEM columns, 192 threads -> TWO CTAs per SM: the two chains sharing the tensor pipe
// are independent CTAs, so one CTA's prologue (barrier init, TMEM alloc, Q load) and epilogue run under
// the other's main loop and the hardware balances 128-row items.
// K/V ring depth: QT stages; keys of 192 columns leave shared memory for one
// Registers: a row of 128 scores and what goes with it need about 200, the TMA and MMA warps a quarter of that. The CTA has
// QT softmax warpgroups and one more, of which two warps work and which gives registers to the others (setmaxnreg; the
// roles' code is compiled for those limits). QT = 1, two CTAs per SM: 256 threads x 128 = 128 x 200 + 128 x 56. QT = 2:
// 384 x 168 = 256 x 216 + 128 x 72. (Keys of 192 columns with one query tile: one CTA of 256 threads has enough.)
constexpr int prefill_threads(int qt) { return 128 * qt + 128; }
constexpr int prefill_stages(int dk, int qt) { return dk > 128 ? 1 : qt; }

// ---- packed fp32 pairs (one issue slot for two results; same rounding as the scalar forms) and row reductions. A softmax
// warp shares its scheduler with one or two others, so the length of its dependency chain per tile counts: four
// independent chains of maxima take 32 steps for 128 scores where one chain takes 127.
__device__ __forceinline__ uint64_t& bits2(float2& x) { return reinterpret_cast<uint64_t&>(x); }
__device__ __forceinline__ float2 both(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(bits2(r)) : "l"(bits2(a)), "l"(bits2(b)), "l"(bits2(c)));
  return r;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(bits2(r)) : "l"(bits2(a)), "l"(bits2(b)));
  return r;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(bits2(r)) : "l"(bits2(a)), "l"(bits2(b)));
  return r;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float2 score_pair(const uint32_t (&sr)[4][32], int c) {      // c even
  return make_float2(__uint_as_float(sr[c >> 5][c & 31]), __uint_as_float(sr[c >> 5][(c + 1) & 31]));
}
__device__ __forceinline__ float row_max(const uint32_t (&sr)[4][32]) {
  float m[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) m[i] = -INFINITY;
#pragma unroll
  for (int c = 0; c < 128; c += 2) {
    const float2 x = score_pair(sr, c);
    m[c & 3] = fmaxf(m[c & 3], x.x), m[(c + 1) & 3] = fmaxf(m[(c + 1) & 3], x.y);
  }
  return fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3]));
}
__device__ __forceinline__ float row_min(const uint32_t (&sr)[4][32]) {
  float m[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) m[i] = INFINITY;
#pragma unroll
  for (int c = 0; c < 128; c += 2) {
    const float2 x = score_pair(sr, c);
    m[c & 3] = fminf(m[c & 3], x.x), m[(c + 1) & 3] = fminf(m[(c + 1) & 3], x.y);
  }
  return fminf(fminf(m[0], m[1]), fminf(m[2], m[3]));
}

struct Item {
  int seq, head, split, q0, Lq, k0, Lk, m0, off, kept, skip, ntq, j_lo, NT;
  int n_tiles[2];
  bool ends_here[2];     // this split holds the last key tile of query tile t
  bool none;             // past the last item
};

template <typename T, int DK, int DV, int QT, bool CAP>
__global__ void __launch_bounds__(prefill_threads(QT), DK > 128 ? 1 : 3 - QT)
prefill_umma_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, const PrefillUmmaParams p) {
  constexpr int kUStages = prefill_stages(DK, QT);   // K/V ring depth
  constexpr int kTmaWarp = 4 * QT, kMmaWarp = 4 * QT + 1, kItemWarp = 4 * QT + 2;
  constexpr uint32_t kTmemCols = QT * 256;      // O[t] at 128 t, S[t] at QT * 128 + 128 t
  constexpr uint32_t kSBase = QT * 128;
  constexpr int CHK = DK / 64, CHV = DV / 64;   // 128-byte chunks per key / value head row
  constexpr int QPANEL = kUBM * 128;            // bytes of one Q panel (128 rows)
  constexpr int KPANEL = kUBN * 128;            // bytes of one K / V panel (128 rows)
  constexpr int QTILE = CHK * QPANEL;
  constexpr int KTILE = CHK * KPANEL;
  constexpr int VTILE = CHV * KPANEL;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  uint8_t* sQ = smem;                            // [QT][QTILE]
  uint8_t* sK = sQ + QT * QTILE;                  // [kUStages][KTILE]
  uint8_t* sV = sK + kUStages * KTILE;           // [kUStages][VTILE]
  uint8_t* s_out = sV + kUStages * VTILE;        // [4 QT warps][32 rows x 64 bytes]: the epilogue's way to whole sectors
  uint16_t* s_tiles = reinterpret_cast<uint16_t*>(s_out + 4 * QT * 2048);   // [kOrderSeqs] row tiles, most first
  uint16_t* s_order = s_tiles + kOrderSeqs;                                 // [kOrderSeqs] their sequences
  Item* s_items = reinterpret_cast<Item*>(s_order + kOrderSeqs);            // [kItems] for the softmax warps
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_items + kItems);
  uint64_t* q_full = bars;                       // [1]
  uint64_t* k_full = bars + 1;                   // [kUStages]
  uint64_t* v_full = k_full + kUStages;          // [kUStages]
  uint64_t* k_empty = v_full + kUStages;         // [kUStages] K stage consumed by both tiles' S(j)
  uint64_t* v_empty = k_empty + kUStages;        // [kUStages] V stage consumed by both tiles' PV(j)
  uint64_t* s_full = v_empty + kUStages;         // [2 tiles]  S[t](j) landed in TMEM
  uint64_t* p_full = s_full + 2;                 // [2 tiles][2 halves]  128 softmax threads stored 64 keys of P[t](j)
  uint64_t* o_full = p_full + 4;                 // [2 tiles]  PV[t](j) retired
  uint64_t* q_empty = o_full + 2;                // [1] the item's last S has retired: Q may be overwritten
  uint64_t* item_full = q_empty + 1;             // [kItems] the slot holds the next item
  uint64_t* item_empty = item_full + kItems;     // [kItems] the softmax warps are through with it
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(item_empty + kItems);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < kUStages; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    for (int t = 0; t < 2; ++t) {
      mbar_init(&s_full[t], 1);
      mbar_init(&p_full[2 * t], kUBM);
      mbar_init(&p_full[2 * t + 1], kUBM);
      mbar_init(&o_full[t], 1);
    }
    mbar_init(q_empty, 1);
    for (int i = 0; i < kItems; ++i) mbar_init(&item_full[i], 1), mbar_init(&item_empty[i], 4 * QT);
    mbar_fence_init();
  }
  if (warp == kTmaWarp && lane == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  // One query tile per CTA is the form of the smallest launches: its producer needs no columns and does not wait for them
  // before its first loads (us, 16 heads over 8 of 128: 1 x 17 tokens 6.6 -> 6.3, 1 x 300 10.2 -> 9.6). With two it made no difference, and the compiler spilled more.
  constexpr bool kEarly = QT == 1;
  if (kEarly) __syncthreads();                       // the barriers are initialised
  // The kernel before this one may still have CTAs on the SM that have yet to allocate their columns (it lets its dependents
  // in at its start): taking all 512 before it has finished could leave both waiting.
  pdl_wait();
  if (warp == kMmaWarp) umma::tmem_alloc(tmem_slot, kTmemCols);
  if (kEarly && warp == kTmaWarp) {
    named_bar_arrive(1, prefill_threads(QT));
  } else {
    umma::fence_before_sync();
    if (kEarly) named_bar_sync(1, prefill_threads(QT));
    else __syncthreads();
    umma::fence_after_sync();
  }
  const uint32_t tb = *tmem_slot;                    // (the early producer has no use for it)

  // Work items: (row tile, sequence, head, key split) in order of falling row tile, so that the longest come first and a
  // CTA's items have about the same number of key tiles as any other's; inside a row tile key
  // splits are neighbours, then the heads of a sequence (which share K and V in L2). The sequences that have a given row tile
  // are the first ones of the list sorted by length. Steps of more sequences than the list holds keep the sequences' own
  // order and pass over the row tiles that a sequence does not have; so do launches with a CTA for every item and those
  // whose sequences are all one row tile, where the order is nothing and the list a round trip to L2, three barriers and a
  // scan before the first load.
  const bool sorted = p.ordered;
  const bool pair = QT == 2 && p.pair;
  const int item_rows = pair ? kUBM : QT * kUBM, row_step = pair ? 0 : kUBM, head_step = pair ? 1 : 0;   // of query tile t
  const int per_seq = p.kv_splits * (pair ? p.H / 2 : p.H);
  if (sorted) {
    constexpr int kPer = (kOrderSeqs + prefill_threads(QT) - 1) / prefill_threads(QT);
    int mine[kPer], at[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int s = threadIdx.x + u * blockDim.x;
      mine[u] = s < p.num_seqs ? min((p.cu_q[s + 1] - p.cu_q[s] + item_rows - 1) / item_rows, 65535) : 0;
      at[u] = 0;
      if (s < kOrderSeqs) s_tiles[s] = (uint16_t)mine[u];             // 0 past the sequences: before nobody
    }
    __syncthreads();
    for (int o = 0; o < p.num_seqs; o += 8) {                         // 8 at a time: one by one it took 8 us of 256 sequences
      const uint4 eight = *reinterpret_cast<const uint4*>(s_tiles + o);
      const uint32_t w[4] = {eight.x, eight.y, eight.z, eight.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int other = (int)((w[i >> 1] >> (16 * (i & 1))) & 0xffffu);
#pragma unroll
        for (int u = 0; u < kPer; ++u)
          at[u] += other > mine[u] || (other == mine[u] && o + i < (int)(threadIdx.x + u * blockDim.x));
      }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int s = threadIdx.x + u * blockDim.x;
      if (s < p.num_seqs) s_tiles[at[u]] = (uint16_t)mine[u], s_order[at[u]] = (uint16_t)s;
    }
    __syncthreads();
  }
  // every role walks the same list with a cursor of its own: index, row tile (from the last one down), first index of it and
  // how many sequences have it
  struct Cursor {
    int round, i, rank, start, have;
  };
  // rounds run to and fro, so that no CTA gets the longest item of every round
  auto pick = [&](int round) { return round * (int)gridDim.x + ((round & 1) ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x); };
  auto sequences_with = [&](int m_tile) {             // how many have more than m_tile row tiles
    if (!sorted) return p.num_seqs;
    int lo = 0, hi = p.num_seqs;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if ((int)s_tiles[mid] > m_tile) lo = mid + 1;
      else hi = mid;
    }
    return lo;
  };
  auto begin = [&]() { return Cursor{0, pick(0), 0, 0, sequences_with(p.m_tiles - 1)}; };
  auto next_item = [&](Cursor& c, Item& it) -> bool {
    for (;; c.i = pick(++c.round)) {
      while (c.i - c.start >= c.have * per_seq) {
        c.start += c.have * per_seq;
        if (++c.rank == p.m_tiles) return false;
        c.have = sequences_with(p.m_tiles - 1 - c.rank);
      }
      const int in = c.i - c.start, k = in / per_seq, hs = in - k * per_seq;
      it.head = p.kv_splits == 1 ? hs : hs / p.kv_splits;
      it.split = hs - it.head * p.kv_splits;
      if (pair) it.head *= 2;
      it.seq = sorted ? (int)s_order[k] : k;
      it.m0 = (p.m_tiles - 1 - c.rank) * item_rows;
      it.q0 = p.cu_q[it.seq], it.Lq = p.cu_q[it.seq + 1] - it.q0;
      it.k0 = p.cu_k[it.seq], it.Lk = p.cu_k[it.seq + 1] - it.k0;
      if (it.m0 < it.Lq) break;
    }
    c.i = pick(++c.round);
    it.off = it.Lk - it.Lq;
    // tiles [0, kept) hold the kept first keys; the next `skip` tiles end before the window of this CTA's first row
    it.kept = p.window > 0 ? (min(p.keep_first, it.Lk) + kUBN - 1) / kUBN : 0;
    it.skip = p.limited() ? max(0, max(0, p.seen_from(it.m0 + it.off)) / kUBN - it.kept) : 0;
    it.n_tiles[0] = it.n_tiles[1] = 0;
#pragma unroll
    for (int t = 0; t < QT; ++t) {
      const int r0 = it.m0 + t * row_step;
      const int n_end = r0 < it.Lq ? min(it.Lk, r0 + kUBM + it.off) : 0;
      it.n_tiles[t] = n_end > 0 ? (n_end + kUBN - 1) / kUBN - it.skip : 0;
    }
    it.ntq = (QT == 2 && it.m0 + row_step < it.Lq) ? 2 : 1;
    // this item's share of the key tiles: [j_lo, j_lo + NT) of the tiles the later query tile needs
    const int nt_all = max(it.n_tiles[0], it.n_tiles[1]);
    int j_hi = nt_all;
    it.j_lo = 0;
    if (p.kv_splits > 1) {                            // (at most 8 splits: the products fit 32 bits)
      it.j_lo = nt_all * it.split / p.kv_splits;
      j_hi = nt_all * (it.split + 1) / p.kv_splits;
    }
    it.NT = j_hi - it.j_lo;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      it.ends_here[t] = it.n_tiles[t] > it.j_lo && it.n_tiles[t] <= j_hi;
      it.n_tiles[t] = max(0, min(it.n_tiles[t], j_hi) - it.j_lo);
    }
    return true;
  };
  // tile index = j_lo + j, past the kept tiles + skip
  auto first_key_of = [](const Item& it, int j) { return (it.j_lo + j + (it.j_lo + j >= it.kept ? it.skip : 0)) * kUBN; };

  constexpr bool kShift = DK <= 128 || QT == 2;
  if (kShift && warp >= 4 * QT) {
    if (QT == 1) asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
  }
  if (warp == kTmaWarp) {
    // =========================== TMA producer ===========================
    if (lane < 2) {
      const bool is_k = lane == 0;
      const CUtensorMap* tm = is_k ? &tmK : &tmV;
      uint64_t pol_keep;
      asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol_keep));
      const uint64_t pol_stream = l2_policy_evict_first();
      uint8_t* ring = is_k ? sK : sV;
      uint64_t* full = is_k ? k_full : v_full;
      uint64_t* empty = is_k ? k_empty : v_empty;
      const int CH = is_k ? CHK : CHV, TILE = is_k ? KTILE : VTILE;
      const int split_boxes = is_k ? p.k_split : p.v_split;
      int n = 0, jr = 0;                             // items and ring tiles so far
      Cursor cur = begin();
      Item it;
      while (next_item(cur, it)) {
        const int kvh = it.head / p.G;
        if (is_k) {
          mbar_wait(q_empty, (n & 1) ^ 1);
          mbar_expect_tx(q_full, it.ntq * QTILE);
          for (int t = 0; t < it.ntq; ++t)
            tma_load_3d(sQ + t * QTILE, &tmQ, q_full, 0, it.q0 + it.m0 + t * row_step, (it.head + t * head_step) * CHK, pol_stream);
        }
        ++n;
        for (int j = 0; j < it.NT; ++j, ++jr) {
          const int s = jr % kUStages;
          const int n0 = first_key_of(it, j);
          if (p.block_tables == nullptr) {
            mbar_wait(&empty[s], ((jr / kUStages) & 1) ^ 1);
            mbar_expect_tx(&full[s], TILE);
            tma_load_3d(ring + s * TILE, tm, &full[s], 0, it.k0 + n0, kvh * CH, pol_keep);
          } else {
            // The tile's block ids, up to 8 (blocks of 16 tokens), are all under way at once and while the ring slot is
            // still in use: looked up one by one between the copies they cost a trip to L2 each, the time of two tiles
            // (256 new tokens against 7936 cached ones, 32 heads over 8 of 64, blocks of 16: 51 -> 38 us).
            // Every op of the tile is issued: boxes past the end of the sequence use an out-of-range
            // row, which TMA zero-fills without touching memory -- P is exactly 0 there, but 0 x (stale
            // shared memory that happens to hold an Inf/NaN pattern) would poison O.
            const int rb = p.kv_rows_box;             // 16 .. 128: block_size where that is smaller than a tile
            const int nops = kUBN / rb;
            const int per_op = split_boxes ? CH : 1;
            const int op_bytes = rb * 128 * (split_boxes ? 1 : CH);
            const int entry = n0 / p.block_size, in_block = n0 - entry * p.block_size;   // in_block: 0 unless nops == 1
            const int32_t* table = p.block_tables + (int64_t)it.seq * p.bt_stride + entry;
            int blk[8];
#pragma unroll
            for (int o = 0; o < 8; ++o) blk[o] = o < nops && n0 + o * rb < it.Lk ? __ldg(table + o) : -1;
            mbar_wait(&empty[s], ((jr / kUStages) & 1) ^ 1);
            mbar_expect_tx(&full[s], nops * per_op * op_bytes);
#pragma unroll
            for (int o = 0; o < 8; ++o) {
              if (o >= nops) break;
              const int row = blk[o] < 0 ? -(1 << 30) : blk[o] * p.block_size + in_block;
              for (int c = 0; c < per_op; ++c) {
                const int dst = (split_boxes ? c * KPANEL : 0) + o * rb * 128;
                tma_load_3d(ring + s * TILE + dst, tm, &full[s], 0, row, kvh * CH + c, pol_keep);
              }
            }
          }
        }
      }
    }
  } else if (warp == kMmaWarp) {
    // =========================== MMA issuer ===========================
    // Warp-uniform control flow, loop-invariant descriptor bases + compile-time offsets, one elected
    // lane issues.
    const uint32_t idesc_s = umma::make_idesc<T>(kUBM, kUBN, 0, 0);   // S = Q K^T, both K-major
    const uint32_t idesc_o = umma::make_idesc<T>(kUBM, DV, 0, 1);      // O = P V, P from TMEM, V MN-major
    const uint64_t qd0 = umma::desc_kmajor(smem_u32(sQ));
    const uint64_t kd0 = umma::desc_kmajor(smem_u32(sK));
    const uint64_t vd0 = umma::desc_mnmajor(smem_u32(sV), KPANEL);
    const bool leader = umma::elect_one();
    // Descriptors are made where they are used: kept across the loop, the 4 to 12 of every operand were more than this role's
    // registers hold (keys of 192 columns, two query tiles: 652 bytes spilled, 104 so; 16 x 1024 tokens, 16 heads over 8 of 128,
    // 92.6 -> 83.5 us in a window of 300, 16 heads of 192 152 -> 141). Two query tiles of 64-wide keys have the room, and making
    // them again costs 2 %.
    constexpr bool kRemake = DK > 64 || QT == 1;
    // S[t] against K ring tile jr: the caller has waited for k_full of stage jr % kUStages
    auto issue_s = [&](int t, int jr) {
      if (leader) {
        uint64_t qd = qd0;
        if (kRemake) asm volatile("" : "+l"(qd));   // see kRemake
        const uint64_t kd = umma::desc_advance(kd0, (jr % kUStages) * KTILE);
        const uint32_t d = tb + kSBase + t * 128;
#pragma unroll
        for (int ks = 0; ks < DK / 16; ++ks) {
          const uint64_t ad = umma::desc_advance(qd, t * QTILE + (ks >> 2) * QPANEL + (ks & 3) * 32);
          const uint64_t bd = umma::desc_advance(kd, (ks >> 2) * KPANEL + (ks & 3) * 32);
          umma::mma_ss(d, ad, bd, idesc_s, ks > 0);
        }
        umma::commit(&s_full[t]);
      }
    };
    int n = 0, base = 0;                             // items and ring tiles so far
    int done[2] = {0, 0};                            // P[t] tiles so far
    Cursor cur = begin();
    Item it, ahead;
    for (bool live = next_item(cur, it); live; it = ahead) {
      live = next_item(cur, ahead);                  // looked up ahead: its loads and divisions are off the chain
      const int NT = it.NT;
      mbar_wait(q_full, n & 1);
      umma::fence_after_sync();
      if (NT > 0) {
        mbar_wait(&k_full[base % kUStages], (base / kUStages) & 1);
        umma::fence_after_sync();
#pragma unroll
        for (int t = 0; t < QT; ++t)
          if (it.n_tiles[t] > 0) issue_s(t, base);
        if (leader) umma::commit(&k_empty[base % kUStages]);
      }
      if (NT <= 1 && leader) umma::commit(q_empty);
      __syncwarp();
      // (O[t] of the item before has been read: the softmax group of tile t stores P of this one afterwards)
      for (int j = 0; j < NT; ++j) {
        const int jr = base + j, s = jr % kUStages, s1 = (jr + 1) % kUStages;
        mbar_wait(&v_full[s], (jr / kUStages) & 1);
        const bool more = j + 1 < NT;
        bool k_ready = false;
        umma::fence_after_sync();
        const uint64_t vd = umma::desc_advance(vd0, s * VTILE);
#pragma unroll
        for (int t = 0; t < QT; ++t) {
          if (j < it.n_tiles[t]) {
            const uint32_t pa = tb + kSBase + t * 128;                // P[t]: 16 keys = 8 packed columns
#pragma unroll
            for (int h = 0; h < 2; ++h) {                          // 64 keys at a time, as they are stored
              mbar_wait(&p_full[2 * t + h], (done[t] + j) & 1);
              umma::fence_after_sync();
              if (leader) {
                uint64_t vdh = vd;
                if (kRemake) asm volatile("" : "+l"(vdh));
#pragma unroll
                for (int kk = h * 4; kk < h * 4 + 4; ++kk)
                  umma::mma_ts(tb + t * 128, pa + kk * 8, umma::desc_advance(vdh, kk * 16 * 128), idesc_o,
                               (j > 0 || kk > 0) ? 1u : 0u);
              }
            }
            if (leader) umma::commit(&o_full[t]);
            if (j + 1 < it.n_tiles[t]) {                           // overwrites S[t]/P[t]: after PV[t](j)
              if (!k_ready) {
                mbar_wait(&k_full[s1], ((jr + 1) / kUStages) & 1);
                umma::fence_after_sync();
                k_ready = true;
              }
              issue_s(t, jr + 1);
            }
          }
        }
        if (leader) {
          umma::commit(&v_empty[s]);
          if (more) umma::commit(&k_empty[s1]);
          if (j + 2 == NT) umma::commit(q_empty);                  // the item's last S has been issued
        }
        __syncwarp();
      }
      base += NT;
      done[0] += it.n_tiles[0], done[1] += it.n_tiles[1];
      ++n;
    }
  } else if (warp < 4 * QT) {
    if (kShift) {
      if (QT == 1) asm volatile("setmaxnreg.inc.sync.aligned.u32 200;");
      else asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    }
    // =========================== softmax warpgroups ===========================
    const int t = warp >> 2;
    const int row = (warp & 3) * 32 + lane;          // row inside the 128-row tile == TMEM lane
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t s_addr = tb + lane_base + kSBase + t * 128;
    const uint32_t o_addr = tb + lane_base + t * 128;
    const float sl2 = CAP ? kLog2e : p.scale_log2;      // capped scores are already scaled
    constexpr float kLazy = 8.f;                     // lazy rescale threshold (exp2 domain): O is rescaled only when the max grew by > 2^8
    int n = 0, done = 0;                             // items and S[t] tiles so far
    for (;; ++n) {
    mbar_wait(&item_full[n % kItems], (n / kItems) & 1);
    const volatile Item& it = s_items[n % kItems];     // (in shared memory: a row of 128 scores leaves no registers for it)
    if (it.none) break;
    const int nt = it.n_tiles[t];
#define B200_QROW (it.m0 + t * row_step + row)             // row inside the sequence
    float m_ref = -INFINITY, l_run = 0.f;
    bool small = true;                               // capped scores: every tile so far was in the polynomial's range
    for (int j = 0; j < nt; ++j) {
      mbar_wait(&s_full[t], (done + j) & 1);
      umma::fence_after_sync();
      uint32_t sr[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) umma::ld32(s_addr + c * 32, sr[c]);
      umma::wait_ld();
      float mx = -INFINITY;
      bool found = false;                              // mx is the row's maximum
      if constexpr (CAP) {
        // tanh of small arguments is a short odd polynomial: while every score of the warp's rows stays below 0.35 caps, it
        // replaces the ex2 and the reciprocal per score that otherwise bind this loop to the special-function unit (3 of
        // its 16 results per clock for each score instead of 1). Truncation: 1.2e-8 of the score at 0.35, with terms up to x^11; below
        // 0.17 caps, where most scores are, four coefficients do (kCapShort), and their five packed operations a pair are what the loop has
        // most of otherwise (nine). The tests are warp-uniform (per-score selection would pay for both sides) and end with the first
        // tile that fails both. A capped maximum is the cap of the maximum: a tile without a mask needs no second search.
        // (12 ragged prompts of 37-1501 tokens, 32 heads of 64, cap 30: 232 us without polynomials, 162 with the long one, 145 with both.)
        float most = 0.f;
        if (small) {
          mx = row_max(sr);
          most = fmaxf(mx, -row_min(sr)) * fabsf(p.cap_pre);
          small = __all_sync(0xffffffffu, most <= 0.35f);
        }
        if (small && __all_sync(0xffffffffu, most <= p.cap_short)) {
          const float y2 = p.cap_pre * p.cap_pre, b0 = p.cap_scale, b1 = b0 * y2, b2 = b1 * y2;
          const float2 a0 = both(b0), a1 = both((float)kCapShort[1] * b1), a2 = both((float)kCapShort[2] * b2), a3 = both((float)kCapShort[3] * (b2 * y2));
#pragma unroll
          for (int c = 0; c < 128; c += 2) {
            const float2 x = score_pair(sr, c), x2 = mul2(x, x);
            const float2 t = mul2(x, fma2(x2, fma2(x2, fma2(x2, a3, a2), a1), a0));
            sr[c >> 5][c & 31] = __float_as_uint(t.x), sr[c >> 5][(c + 1) & 31] = __float_as_uint(t.y);
          }
          const float x2 = mx * mx;
          mx *= fmaf(x2, fmaf(x2, fmaf(x2, a3.x, a2.x), a1.x), a0.x);
          found = true;
        } else if (small) {
          const float2 pre = both(p.cap_pre), scale = both(p.cap * p.cap_pre);
#pragma unroll
          for (int c = 0; c < 128; c += 2) {
            const float2 x = score_pair(sr, c);
            const float2 y = mul2(x, pre), y2 = mul2(y, y);
            float2 t = fma2(y2, both(-1382.f / 155925.f), both(62.f / 2835.f));
            t = fma2(y2, t, both(-17.f / 315.f));
            t = fma2(y2, t, both(2.f / 15.f));
            t = fma2(y2, t, both(-1.f / 3.f));
            t = fma2(y2, t, both(1.f));
            t = mul2(t, mul2(x, scale));
            sr[c >> 5][c & 31] = __float_as_uint(t.x), sr[c >> 5][(c + 1) & 31] = __float_as_uint(t.y);
          }
        } else {                                       // cap tanh(y) = cap - 2 cap / (1 + e^2y)
          const float2 pre = both(p.cap_pre * 2.8853900817779268f), one = both(1.f), cap = both(p.cap), less = both(-2.f * p.cap);
#pragma unroll
          for (int c = 0; c < 128; c += 2) {
            const float2 x = mul2(score_pair(sr, c), pre);
            const float2 d = add2(make_float2(ex2_approx(x.x), ex2_approx(x.y)), one);
            const float2 t = fma2(make_float2(rcp_approx(d.x), rcp_approx(d.y)), less, cap);
            sr[c >> 5][c & 31] = __float_as_uint(t.x), sr[c >> 5][(c + 1) & 31] = __float_as_uint(t.y);
          }
        }
      }
      const int n0 = (it.j_lo + j + (it.j_lo + j >= it.kept ? it.skip : 0)) * kUBN;
      // mask (warp-uniform test: does this tile touch the diagonal or the end of the keys?)
      const int warp_row0 = it.m0 + t * row_step + (warp & 3) * 32, Lk = it.Lk, off = it.off;
      if (n0 + kUBN > Lk || n0 + kUBN - 1 > warp_row0 + off) {
        found = false;
        const int limit = min(Lk - 1, B200_QROW + off) - n0;   // last visible key (tile-relative)
        const int every = min(Lk - 1, warp_row0 + off) - n0;   // last key that all rows of the warp see
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (32 * k + 31 > every) {                      // warp-uniform: columns below the diagonal block need no test
#pragma unroll
            for (int c = 0; c < 32; ++c)
              if (32 * k + c > limit) sr[k][c] = 0xff800000u;      // -inf
          }
        }
      }
      if (p.limited() && n0 + kUBN > p.keep_first && n0 < p.seen_from(warp_row0 + 31 + off)) {
        found = false;
        const int low = p.seen_from(B200_QROW + off) - 1 - n0, keep = p.keep_first - n0;   // hidden: keep <= c <= low
#pragma unroll
        for (int c = 0; c < 128; ++c)
          if (c <= low && c >= keep) sr[c >> 5][c & 31] = 0xff800000u;
      }
      if (!CAP || !found) mx = row_max(sr);
      const bool grow = (mx - m_ref) * sl2 > kLazy;       // also true for the first finite max
      if (__any_sync(0xffffffffu, grow)) {
        const float m_new = grow ? mx : m_ref;
        const float alpha = (m_ref == -INFINITY) ? 0.f : ex2_approx((m_ref - m_new) * sl2);
        if (j > 0) {
          mbar_wait(&o_full[t], (done + j - 1) & 1);      // PV[t](j-1) landed
          umma::fence_after_sync();
#pragma unroll
          for (int c0 = 0; c0 < DV; c0 += 16) {    // 16 columns at a time: the S row stays in registers
            uint32_t orr[16];
            umma::ld16(o_addr + c0, orr);
            umma::wait_ld();
#pragma unroll
            for (int c = 0; c < 16; ++c) orr[c] = __float_as_uint(__uint_as_float(orr[c]) * alpha);
            umma::st16(o_addr + c0, orr);
          }
          umma::wait_st();
        }
        l_run *= alpha;
        m_ref = m_new;
      }
      const float mb = m_ref == -INFINITY ? 0.f : m_ref * sl2;
      const float2 scale2 = both(sl2), shift2 = both(-mb);
      float2 sum = make_float2(0.f, 0.f);
      // P(j): 128 keys -> 64 packed columns over S[t] columns [0, 64); this thread's S row is
      // already in registers, other rows live in other TMEM lanes. Packed in place: element i of
      // chunk 2h was consumed at iteration i/2.
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const int c = h * 64 + 2 * i;
          const float2 x = fma2(score_pair(sr, c), scale2, shift2);
          const float2 e = make_float2(ex2_approx(x.x), ex2_approx(x.y));
          sum = add2(sum, e);
          sr[2 * h][i] = pack2<T>(e.x, e.y);
        }
        umma::st32(s_addr + h * 32, sr[2 * h]);
        umma::wait_st();
        umma::fence_before_sync();
        mbar_arrive(&p_full[2 * t + h]);          // PV of these 64 keys may start
      }
      l_run += sum.x + sum.y;
    }
    // the sink joins the denominator once: in the split that holds the query tile's last keys (never an empty one)
    if (p.sink != nullptr && it.ends_here[t]) {
      const float sink2 = p.sink[it.head + t * head_step] * kLog2e;
      if (m_ref == -INFINITY) m_ref = sink2 / sl2, l_run = 1.f;      // no key of this split is visible to the row
      else l_run += ex2_approx(sink2 - m_ref * sl2);
    }
    // ---- epilogue: O / l -> global, or (split-KV) the un-normalised partial -> workspace
    if (nt > 0) mbar_wait(&o_full[t], (done + nt - 1) & 1);          // its own last product, not the other tile's
    umma::fence_after_sync();
    const int m0 = it.m0, Lq = it.Lq, q0 = it.q0, head = it.head + t * head_step, split = it.split, qrow = m0 + t * row_step + row;
    const int warp_row_base = m0 + t * row_step + (warp & 3) * 32;   // this warp's first row inside the sequence
    __syncwarp();
    if (lane == 0) mbar_arrive(&item_empty[n % kItems]);
    if (m0 + t * row_step < Lq) {
      T* orow = reinterpret_cast<T*>(p.out) + (int64_t)(q0 + qrow) * p.out_stride + (int64_t)head * DV;
      const int64_t pidx = ((int64_t)(q0 + qrow) * p.H + head) * p.kv_splits + split;
      float* prow = p.part_o + pidx * DV;
      const bool split_out = p.kv_splits > 1;
      if (split_out && qrow < Lq) {
        p.part_ml[pidx * 2] = (nt > 0 && m_ref != -INFINITY) ? m_ref * sl2 : -INFINITY;
        p.part_ml[pidx * 2 + 1] = nt > 0 ? l_run : 0.f;
      }
      if (nt > 0) {
        const float inv = split_out ? 1.f : (l_run > 0.f ? 1.f / l_run : 0.f);
        // A lane holds a whole row; stored straight from there, every 16-byte store of a warp touched 32 lines, and the
        // next item's first loads queued behind them (8-9 k cycles per item, measured). 32 rows x 64 bytes at a time pass
        // through shared memory (16-byte chunks XOR-swizzled by row / 2), 4 lanes write 64 contiguous bytes.
        uint8_t* stage = s_out + warp * 2048;
        const int rows = Lq - warp_row_base, sub = lane & 3, r8 = lane >> 2;
        auto pass = [&](const uint32_t (&w)[16], uint8_t* to, int64_t row_bytes) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
            *reinterpret_cast<uint4*>(stage + lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)) =
                make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int r = 8 * i + r8;
            const uint4 x = *reinterpret_cast<const uint4*>(stage + r * 64 + ((sub ^ ((r >> 1) & 3)) << 4));
            if (r < rows) *reinterpret_cast<uint4*>(to + r * row_bytes + sub * 16) = x;
          }
          __syncwarp();
        };
        if (split_out) {
          uint8_t* to = reinterpret_cast<uint8_t*>(p.part_o + (((int64_t)(q0 + warp_row_base) * p.H + head) * p.kv_splits + split) * DV);
          const int64_t row_bytes = (int64_t)p.H * p.kv_splits * DV * 4;
#pragma unroll
          for (int c0 = 0; c0 < DV; c0 += 16) {
            uint32_t w[16];
            umma::ld16(o_addr + c0, w);
            umma::wait_ld();
            pass(w, to + c0 * 4, row_bytes);
          }
        } else {
          uint8_t* to = reinterpret_cast<uint8_t*>(reinterpret_cast<T*>(p.out) + (int64_t)(q0 + warp_row_base) * p.out_stride + (int64_t)head * DV);
#pragma unroll
          for (int c0 = 0; c0 < DV; c0 += 32) {
            uint32_t orr[32], w[16];
            umma::ld32(o_addr + c0, orr);
            umma::wait_ld();
#pragma unroll
            for (int c = 0; c < 16; ++c)
              w[c] = pack2<T>(__uint_as_float(orr[2 * c]) * inv, __uint_as_float(orr[2 * c + 1]) * inv);
            pass(w, to + c0 * 2, p.out_stride * 2);
          }
        }
      } else if (qrow < Lq) {
        if (split_out) {
          for (int c = 0; c < DV; c += 4) *reinterpret_cast<uint4*>(prow + c) = make_uint4(0, 0, 0, 0);
        } else {
          for (int c = 0; c < DV; c += 8) *reinterpret_cast<uint4*>(orow + c) = make_uint4(0, 0, 0, 0);
        }
      }
    }
    umma::fence_before_sync();
    done += nt;
    }
  } else if (warp == kItemWarp) {
    // =========================== work items of the softmax warps ===========================
    // Found one ahead by a warp of its own: the loads and divisions took a softmax warp 1200 cycles of every item
    Cursor cur = begin();
    Item x;
    for (int n = 0;; ++n) {
      const bool found = next_item(cur, x);
      mbar_wait(&item_empty[n % kItems], ((n / kItems) & 1) ^ 1);
      if (lane == 0) {
        x.none = !found;
        s_items[n % kItems] = x;
        mbar_arrive(&item_full[n % kItems]);
      }
      if (!found) break;
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == kMmaWarp) umma::tmem_dealloc(tb, kTmemCols);
}

// Split-KV merge: one warp per (query row, head); lane = D/32 consecutive columns. Pieces are
// un-normalised (O, m, l) relative to their own reference max m (exp2 domain).
template <typename T, int D>
__global__ void __launch_bounds__(256)
prefill_combine_kernel(T* __restrict__ out, int64_t out_stride, const float* __restrict__ part_o,
                       const float* __restrict__ part_ml, int64_t rows_x_heads, int H, int splits) {
  constexpr int V = D / 32;
  pdl_wait();
  const int64_t item = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (item >= rows_x_heads) return;
  const int lane = threadIdx.x & 31;
  const int64_t row = item / H;
  const int head = (int)(item - row * H);
  const float* ml = part_ml + item * splits * 2;
  float m = -INFINITY;
  for (int s = 0; s < splits; ++s) m = fmaxf(m, ml[2 * s]);
  float l = 0.f, acc[V];
#pragma unroll
  for (int i = 0; i < V; ++i) acc[i] = 0.f;
  for (int s = 0; s < splits; ++s) {
    const float ms = ml[2 * s];
    if (ms == -INFINITY) continue;
    const float sc = ex2_approx(ms - m);
    l = fmaf(ml[2 * s + 1], sc, l);
    const float* po = part_o + (item * splits + s) * D + lane * V;
#pragma unroll
    for (int i = 0; i < V; ++i) acc[i] = fmaf(po[i], sc, acc[i]);
  }
  const float inv = l > 0.f ? 1.f / l : 0.f;
  T* orow = out + row * out_stride + (int64_t)head * D + lane * V;
#pragma unroll
  for (int i = 0; i < V; i += 2) *reinterpret_cast<uint32_t*>(orow + i) = pack2<T>(acc[i] * inv, acc[i + 1] * inv);
}

template <typename T, int DK, int DV, int QT, bool CAP>
static int prefill_umma_launch_c(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                                 PrefillUmmaParams p, int num_seqs, int max_seqlen_q, int total_q,
                                 cudaStream_t stream) {
  constexpr int CHK = DK / 64, CHV = DV / 64;
  constexpr size_t smem =
      1024 + QT * CHK * kUBM * 128 + prefill_stages(DK, QT) * (CHK + CHV) * kUBN * 128 + 4 * QT * 2048 + kOrderSeqs * 4 + kItems * sizeof(Item) + 36 * 8 + 16;
  static_assert(kItems * sizeof(Item) % 8 == 0, "barriers on 8-byte boundaries");
  auto kern = prefill_umma_kernel<T, DK, DV, QT, CAP>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    attr_set = true;
  }
  const int item_rows = QT == 2 && p.pair ? kUBM : QT * kUBM;
  p.m_tiles = (max_seqlen_q + item_rows - 1) / item_rows, p.num_seqs = num_seqs;
  const int64_t items = (int64_t)p.m_tiles * p.kv_splits * (QT == 2 && p.pair ? p.H / 2 : p.H) * num_seqs;
  if (items > 0x7fffffff) return B200_ERR_UNSUPPORTED;
  const int slots = 148 * (DK > 128 ? 1 : 3 - QT);
  p.ordered = num_seqs <= kOrderSeqs && p.m_tiles > 1 && items > slots;
  launch_pdl(kern, dim3((unsigned)(items < slots ? items : slots)), dim3(prefill_threads(QT)), smem, stream, mq, mk, mv, p);
  if (p.kv_splits > 1) {
    const int64_t rows = (int64_t)total_q * p.H;
    launch_pdl(prefill_combine_kernel<T, DV>, dim3((unsigned)((rows + 7) / 8)), dim3(256), 0, stream,
               reinterpret_cast<T*>(p.out), p.out_stride, (const float*)p.part_o, (const float*)p.part_ml,
               rows, p.H, p.kv_splits);
  }
  return finish_launch(p.kv_splits > 1 ? 2 : 1);
}

template <typename T, int DK, int DV, int QT>
static int prefill_umma_launch_t(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                                 const PrefillUmmaParams& p, int num_seqs, int max_seqlen_q, int total_q, cudaStream_t stream) {
  return p.cap > 0.f ? prefill_umma_launch_c<T, DK, DV, QT, true>(mq, mk, mv, p, num_seqs, max_seqlen_q, total_q, stream)
                     : prefill_umma_launch_c<T, DK, DV, QT, false>(mq, mk, mv, p, num_seqs, max_seqlen_q, total_q, stream);
}

// Key splits for a launch: only when its items -- `rows` rows of one head, or of a pair of heads, of one sequence -- would
// leave more than half of the co-resident CTA slots idle, at least two 128-key tiles per split, at most 8, and only if the
// workspace holds them.
int prefill_kv_splits(int num_seqs, int H, int max_seqlen_q, int max_seqlen_k, int total_q, int D,
                      int64_t workspace_bytes, int qt, int pair) {
  const int slots = 148 * (3 - qt);            // co-resident CTAs: one per SM at QT = 2, two at QT = 1
  const int rows = pair ? kUBM : qt * kUBM;
  const int64_t ctas = (int64_t)((max_seqlen_q + rows - 1) / rows) * (pair ? H / 2 : H) * num_seqs;
  if (ctas * 2 > slots) return 1;
  const int key_tiles = (max_seqlen_k + kUBN - 1) / kUBN;
  int splits = (int)(slots / ctas);
  if (splits > 8) splits = 8;
  if (splits > key_tiles / 2) splits = key_tiles / 2;
  while (splits > 1 && (int64_t)total_q * H * splits * (D + 2) * 4 > workspace_bytes) --splits;
  return splits < 1 ? 1 : splits;
}

// Query tiles per CTA for a launch. Measured, us, QT = 1 / QT = 2 as 128 rows of two heads:
//   D 128, 16 heads over 8:  4 x 2000  83.5 / 75.5;  1 x 8192  256 / 233;  12 x 37-1483  68 / 65;  512 x 20  148 / 138;  256 x 16  77 / 72;
//                            64 x 128  28.4 / 29.7;  16 x 1024 in a window of 300  96 / 84, in chunks of 200  87 / 77
//   D 64, 32 heads over 8:   4 x 2000  129 / 121;  1 x 8192  419 / 389;  12 x 37-1483  102 / 97;  256 x 16  112 / 121;  64 x 128  34 / 36
// and QT = 1 / QT = 2 as 256 rows of a head, where heads come alone:
//   D 128, 8 heads over 8:   2 x 4096  77 / 67;  16 x 1024  60 / 58;  12 x 37-1483  45 / 46;  32 x 300  33 / 37;  64 x 100  17 / 21
//          24 heads over 8:  2 x 4096  203 / 183;  16 x 1024  152 / 141;  12 x 37-1483  96 / 97;  32 x 300  72 / 82;  64 x 100  38 / 49
//   D 64, 16 heads over 16:  2 x 4096  118 / 112;  16 x 1024  85 / 87;  12 x 37-1483  55 / 64;  32 x 300  44 / 49;  64 x 100  20 / 29
// What decides is how often K and V cross from L2 (QT = 1 reads every tile for 128 rows of one head,
// and its one-stage rings wait for them), then the rows that a 256-row tile computes for nothing. So: two heads that share
// K and V wherever heads come in pairs; otherwise 256 rows of one head from 512 rows on (D 128) or 2048 (D 64, whose
// tiles are cheaper), and where the grid is so small that keys are split across CTAs anyway.
// b200_prefill_set_query_tiles(1|2) forces one layout (A/B runs, parity tests of both instantiations).
// Launches whose 128-row tiles of one head find a CTA slot each (`slots`), with at most four key tiles, take QT = 1 in any
// case: nothing is read often enough for sharing to count, and a CTA's start, two chains and end are shorter than those of a
// pair (us, QT = 1 / pair, 16 heads over 8: D 128, 1 x 17 6.3 / 7.1, 1 x 300 9.6 / 11.2, 2 x 129 8.1 / 9.2; keys of 192, 1 x 300 8.9 / 11.1).
static bool prefill_small(int num_seqs, int H, int max_seqlen_q, int max_seqlen_k, int slots) {
  return (int64_t)((max_seqlen_q + kUBM - 1) / kUBM) * H * num_seqs <= slots && max_seqlen_k <= 4 * kUBN;
}
static int g_forced_query_tiles = 0;
void prefill_force_query_tiles(int qt) { g_forced_query_tiles = qt; }

int prefill_query_tiles(int num_seqs, int H, int rep, int max_seqlen_q, int max_seqlen_k, int D, int span) {
  if (g_forced_query_tiles) return g_forced_query_tiles;
  if (prefill_small(num_seqs, H, max_seqlen_q, max_seqlen_k, 2 * 148)) return 1;
  if (rep % 2 == 0) return 2;
  const int64_t ctas2 = (int64_t)((max_seqlen_q + 2 * kUBM - 1) / (2 * kUBM)) * H * num_seqs;
  if (ctas2 * 2 <= 148) return 2;                 // key-split territory (prefill_kv_splits)
  const int least = D == 128 ? 512 : 2048;
  return max_seqlen_q >= least && span >= 512 ? 2 : 1;   // span: tokens along the keys a row walks over
}

// Entry used by b200_prefill_varlen_attn (prefill_attn.cu). Returns B200_ERR_UNSUPPORTED when the
// strides cannot be described by a TMA map (caller falls back to the mma.sync kernel).
int prefill_umma_launch(void* out, const void* q, const void* k, const void* v,
                         const int32_t* cu_q, const int32_t* cu_k, int num_seqs, int total_q,
                         int total_k, int max_seqlen_q, int H, int Hkv, int DK, int DV, int64_t q_stride,
                         int64_t k_stride, int64_t v_stride, int64_t out_stride,
                        const int32_t* block_tables, int bt_stride, int num_blocks, int block_size,
                        float scale, int dtype, void* workspace, int64_t workspace_bytes, int max_seqlen_k,
                        cudaStream_t stream, float softcap, const float* sink, int window, int keep_first, int chunk) {
  if (q_stride % 8 != 0 || out_stride % 8 != 0 || !aligned16(out)) return B200_ERR_UNSUPPORTED;
  if (total_q <= 0) return B200_ERR_UNSUPPORTED;
  const int CHK = DK / 64, CHV = DV / 64;
  CUtensorMap mq, mk, mv;
  int rc = get_panel_map(q, total_q, q_stride * 2, H * CHK, kUBM, CHK, dtype, &mq);
  if (rc != B200_OK) return rc;
  PrefillUmmaParams p;
  p.cu_q = cu_q, p.cu_k = cu_k, p.block_tables = block_tables;
  p.out = out, p.out_stride = out_stride;
  p.H = H, p.G = H / Hkv, p.block_size = block_size, p.bt_stride = bt_stride;
  p.scale_log2 = scale * 1.4426950408889634f;
  if (softcap > 0.f) {
    p.cap = softcap, p.cap_pre = scale / softcap;
    // (coefficients and squares of scores have to be normal numbers: others leave it to the long polynomial, whose powers are of the quotient)
    if (scale >= 0x1p-20f && scale <= 0x1p20f && p.cap_pre >= 0x1p-14f && p.cap_pre <= 0x1p14f) p.cap_scale = scale, p.cap_short = kCapShortTo;
  }
  p.sink = sink;
  p.window = window, p.keep_first = window > 0 ? keep_first : 0, p.chunk = chunk;
  const int span = window > 0 ? window : chunk;
  // keys that a 128-row query tile can see at most: what the choice of layout and of key splits is made on
  if (span > 0 && max_seqlen_k > span + p.keep_first + 3 * kUBM) max_seqlen_k = span + p.keep_first + 3 * kUBM;
  // one CTA per SM either way with keys of 192 columns: two ping-pong tiles wherever a sequence has them
  const int qt = DK > 128 ? (max_seqlen_q > kUBM && !prefill_small(num_seqs, H, max_seqlen_q, max_seqlen_k, 148) ? 2 : 1)
                          : prefill_query_tiles(num_seqs, H, p.G, max_seqlen_q, max_seqlen_k, DV,
                                                span > 0 ? max_seqlen_k : max_seqlen_q);
  p.pair = qt == 2 && p.G % 2 == 0;
  p.kv_splits = (workspace != nullptr && (reinterpret_cast<uintptr_t>(workspace) & 15) == 0)
                    ? prefill_kv_splits(num_seqs, H, max_seqlen_q, max_seqlen_k, total_q, DV, workspace_bytes, qt, p.pair)
                    : 1;
  p.part_o = reinterpret_cast<float*>(workspace);
  p.part_ml = p.part_o + (int64_t)total_q * H * p.kv_splits * DV;
  if (block_tables == nullptr) {
    if (k_stride % 8 != 0 || v_stride % 8 != 0 || total_k <= 0) return B200_ERR_UNSUPPORTED;
    p.kv_rows_box = kUBN, p.k_split = p.v_split = 0;
    rc = get_panel_map(k, total_k, k_stride * 2, Hkv * CHK, kUBN, CHK, dtype, &mk);
    if (rc != B200_OK) return rc;
    rc = get_panel_map(v, total_k, v_stride * 2, Hkv * CHV, kUBN, CHV, dtype, &mv);
    if (rc != B200_OK) return rc;
  } else {
    if (block_size % 16 != 0 || (block_size < kUBN && kUBN % block_size != 0) ||
        (block_size > kUBN && block_size % kUBN != 0))
      return B200_ERR_UNSUPPORTED;
    p.kv_rows_box = block_size < kUBN ? block_size : kUBN;
    p.k_split = p.v_split = p.kv_rows_box < kUBN ? 1 : 0;
    const int64_t rows = (int64_t)num_blocks * block_size;
    rc = get_panel_map(k, rows, (int64_t)Hkv * DK * 2, Hkv * CHK, p.kv_rows_box, p.k_split ? 1 : CHK, dtype, &mk);
    if (rc != B200_OK) return rc;
    rc = get_panel_map(v, rows, (int64_t)Hkv * DV * 2, Hkv * CHV, p.kv_rows_box, p.v_split ? 1 : CHV, dtype, &mv);
    if (rc != B200_OK) return rc;
  }
#define B200_PREFILL_QT(T, K, V)                                                                          \
  (qt == 2 ? prefill_umma_launch_t<T, K, V, 2>(mq, mk, mv, p, num_seqs, max_seqlen_q, total_q, stream) \
           : prefill_umma_launch_t<T, K, V, 1>(mq, mk, mv, p, num_seqs, max_seqlen_q, total_q, stream))
#define B200_PREFILL_DISPATCH(T)                                                      \
  (DK == 192   ? (DV == 128 ? B200_PREFILL_QT(T, 192, 128) : B200_PREFILL_QT(T, 192, 64)) \
   : DK == 128 ? (DV == 128 ? B200_PREFILL_QT(T, 128, 128) : B200_PREFILL_QT(T, 128, 64)) \
             : (DV == 128 ? B200_PREFILL_QT(T, 64, 128) : B200_PREFILL_QT(T, 64, 64)))
  return dtype == B200_DTYPE_BF16 ? B200_PREFILL_DISPATCH(__nv_bfloat16) : B200_PREFILL_DISPATCH(__half);
#undef B200_QROW
#undef B200_PREFILL_DISPATCH
#undef B200_PREFILL_QT
}

}  // namespace b200
