// bf16 GEMM on tcgen05 with CTA pairs (cta_group::2): two CTAs of a cluster share one 256 x 256 output tile.
//
//   C[M, N] (+)= A[M, K] * B[N, K]^T (+ bias[N])
//
// Each CTA of the pair holds 128 rows of A and 128 of the 256 rows of the B tile; one thread of the leader CTA
// issues tcgen05.mma.cta_group::2 (M 256 x N 256 x K 16), the hardware reads both CTAs' shared memory and each
// CTA's tensor memory receives its 128 accumulator rows.  Per SM that halves the shared-memory traffic of B, which
// is what bounds the single-CTA kernel.  Roles per CTA: warp 0 TMA producer (both CTAs' loads complete on the
// leader's "full" barrier), warp 1 MMA issuer (leader only; commits are multicast to both CTAs' barriers),
// the other warps (four or eight) epilogue.  Bounded waits everywhere; a CTA that gives up still joins the final cluster barrier.
// Operands may be K-major or MN-major as in gemm_tcgen05.cu.
#include "act_common.cuh"
#include "launch.cuh"
#include "pair_common.cuh"
#include "tmap_util.cuh"
#include "xent_common.cuh"

namespace {

using namespace tc;

constexpr int BM2 = 128;          // rows per CTA (256 per pair)
// N extent of the pair tile: 256 (default) or 128 (for outputs whose 256-wide tiles quantise badly over the 74 CTA
// pairs, e.g. 96 tiles = 1.3 waves); each CTA holds BN / 2 rows of the B tile.
constexpr int BK2 = 64;
template <int BN> struct PairCfg {
  static constexpr int BNH = BN / 2;
  static constexpr int STAGES = (BN >= 192) ? 6 : 8;
  static constexpr int TMEM_COLS = (2 * BN <= 256) ? 256 : 512;        // two accumulators; the allocation is a power of two
  static constexpr int STAGE_BYTES = 128 * 64 * 2 + BNH * 64 * 2;      // A rows of this CTA + its half of B
};
constexpr int MAX_SPLITS = 3;      // K slices per output tile at most
// Epilogue warps: one per 32 rows, or two of them (one for each half of the columns) where the epilogue has arithmetic to do
// (bias, activation): a warp alone on its scheduler waits out the latency of everything it does, and with a K of 768 the
// epilogue of a tile then takes longer than the products of the next one.  Without arithmetic the second warp costs more than it
// hides.  us, one / two warps, with a pass over 64 MB before each launch (so that operands come from memory):
//   8192 x 3072 x 768   plain 37.8 / 39.9   with bias 46.0 / 41.9   with bias and activation 60.3 / 50.2
//   8192 x 2304 x 768   plain 29.7 / 31.7   with bias 35.7 / 31.8   1024 x 768 x 3072 with bias 27.4 / 25.5
// (with bias and activation 67.5 with the bias read as described at bias_pair).
constexpr int EPI_STAGE_BYTES = 8 * 4096;          // boxes of [32 rows][64 bf16] for the TMA store: two per warp, or one
template <int BN> constexpr int pair_smem_bytes() { return PairCfg<BN>::STAGES * PairCfg<BN>::STAGE_BYTES + EPI_STAGE_BYTES + 1024 + 256; }

__device__ int g_gemm2_error = 0;

// One GEMM of a launch.  A launch runs up to MAX_GROUP of them (same operand layouts) as ONE list of output tiles over
// the persistent clusters: small products that each fill the clusters badly (the four weight gradients of a
// transformer layer: 27 + 9 + 36 + 36 tiles on 74 clusters) then share rounds, and the fixed cost of a launch
// (pipeline fill, last epilogue) is paid once.
constexpr int MAX_GROUP = 6;
struct GemmProblem {
  CUtensorMap ta, tb, tc;
  CUtensorMap tb_half;              // K-major B in boxes of half as many rows, for units of half a tile
  void* C;
  const void* bias;
  int M, N, K, ldc;
  int out_fp32, accumulate;
  int n_store;                      // columns that a bf16 output may be written in: N, or more (zeros)
  int tma_store;                    // bf16 output written through shared memory and TMA stores (full lines, async)
  int num_m_pairs, num_n_tiles;
  int group_m;                      // tile order: blocks of group_m tile rows, all their columns, rows fastest (see pick_group_m)
  int tile_start;                   // index of this product's first tile in the launch's list
};
struct GemmGroup {
  GemmProblem pr[MAX_GROUP];
  int n, num_tiles;                 // products, tiles of all of them
  // split-K (one product only): a work unit is (output tile, K slice).  Every unit stores its fp32 partial tile in
  // `ws`; per 32 rows and epilogue warp a counter tells the last unit to arrive, which sums the slices in slice order and
  // writes the output; with two slices and a TMA-stored output the slices exchange half an accumulator each instead.
  int splits, kb_per_split;
  // tail split (splits == 1): the last `tail` tiles of the list, the ones of the launch's final, partly filled wave
  // of clusters, run as two units each, side by side in that wave: with tail_k two K halves that exchange half an
  // accumulator each (the two-slice TMA-store path), else two halves of the columns; 0 = every tile is one unit
  int tail, tail_k;
  float* ws;                        // [slices * tiles][2 CTAs][8 column chunks][8 float4 of a row][128 rows] float4:
                                    // consecutive lanes (rows) are consecutive in memory, so a warp's store covers whole lines
  int* counters;                    // [tiles][2 CTAs][4 row groups][2 column halves or slices], zero between launches
  // Activation in the epilogue (one product, whole tiles): act = 1 + its mode (act_common.cuh), 0 = none.  The activated tile goes
  // out through `tact`, the product itself only with keep_c.
  CUtensorMap tact;
  int act, keep_c;
  // Statistics for a cross-entropy over the output's columns (one product, whole tiles): see epilogue_loss
  const int64_t* labels;
  float2* part;
  float* target;
  int part_ld;
  float cap;
  // Rows beyond the last whole 256 (one product, K-major A, whole tiles): see narrow_rows.  `narrow` columns of the transposed tiles, a
  // multiple of 32; ta_narrow: these rows of A in boxes of half as many
  CUtensorMap ta_narrow;
  int narrow, narrow_first;
};
enum Epilogue { EPI_STORE, EPI_ACT, EPI_LOSS, EPI_LOSS_CAP, EPI_STORE_NARROW };

// The units of one cluster, in order.  With narrow tiles (one per tile column, index num_tiles + column): whole tiles go round;
// narrow ones go to the clusters that have one whole tile less, narrow_first times, then round from the first of these.  Both
// lists are merged by column, so that the weights of a column are read at about the same time.
template <bool NARROW>
struct Units {
  int at, step, end;
  __device__ Units(const GemmGroup&, int cluster, int clusters, int num_units) : at(cluster), step(clusters), end(num_units) {}
  __device__ __forceinline__ bool more() const { return at < end; }
  __device__ __forceinline__ int unit() const { return at; }
  __device__ __forceinline__ void advance() { at += step; }
};
template <>
struct Units<true> {
  int whole, nar, step, tiles, cols, per_col, idle, first, turn;
  __device__ Units(const GemmGroup& g, int cluster, int clusters, int)
      : whole(cluster), step(clusters), tiles(g.num_tiles), cols(g.pr[0].num_n_tiles), per_col(g.pr[0].num_m_pairs) {
    const int rem = tiles % clusters;
    idle = clusters - rem;
    first = idle * (rem ? g.narrow_first : 0);
    turn = cluster >= rem ? cluster - rem : cluster - rem + clusters;       // place in the order of the narrow tiles
    nar = turn < idle && first > 0 ? turn : first + turn;
  }
  __device__ __forceinline__ bool take_narrow() const { return nar < cols && (whole >= tiles || nar <= whole / per_col); }
  __device__ __forceinline__ bool more() const { return whole < tiles || nar < cols; }
  __device__ __forceinline__ int unit() const { return take_narrow() ? tiles + nar : whole; }
  __device__ __forceinline__ void advance() {
    if (!take_narrow()) whole += step;
    else if (nar < first) nar = nar + idle < first ? nar + idle : first + turn;
    else nar += step;
  }
};

// One unit of work of a cluster: an output tile, one K slice of it, or half of its columns.
struct Unit {
  int pi, tile, lt, ks, kb0, kb1;   // product, tile in the launch's list, tile within the product, K slice and its blocks
  int part;                         // columns: 0 all, 1 first half, 2 second half
  int wtile, wtiles;                // index of the tile among those cut along K and their number (workspace / flag addressing)
  bool split;                       // one of several K slices
};
__device__ __forceinline__ Unit decode_unit(const GemmGroup& g, int unit) {
  Unit u;
  const int T = g.num_tiles, whole = T - g.tail;
  u.ks = u.part = 0;
  u.wtile = u.tile = unit;
  u.wtiles = T;
  u.split = g.splits > 1;
  if (g.splits > 1) {
    u.wtile = u.tile = unit % T;
    u.ks = unit / T;
  } else if (unit >= whole) {
    const int second = unit - whole >= g.tail ? 1 : 0;
    u.wtile = unit - whole - second * g.tail;
    u.wtiles = g.tail;
    u.tile = whole + u.wtile;
    u.split = g.tail_k != 0;
    if (g.tail_k) u.ks = second;
    else u.part = 1 + second;
  }
  u.pi = 0;
#pragma unroll
  for (int i = 1; i < MAX_GROUP; ++i)
    if (i < g.n && u.tile >= g.pr[i].tile_start) u.pi = i;
  u.lt = u.tile - g.pr[u.pi].tile_start;
  const int nkb = (g.pr[u.pi].K + BK2 - 1) / BK2;
  const int per = u.split && g.splits == 1 ? (nkb + 1) / 2 : g.kb_per_split;
  u.kb0 = u.ks * per;
  u.kb1 = min(nkb, u.kb0 + per);
  return u;
}

__device__ __forceinline__ void tile_coords(const GemmProblem& p, int lt, int& tm, int& tn) {
  const int block = p.group_m * p.num_n_tiles, gi = lt / block, w = lt - gi * block;
  const int gm = min(p.group_m, p.num_m_pairs - gi * p.group_m);
  tn = w / gm;
  tm = gi * p.group_m + w - tn * gm;
}

// TMA load whose completion is signalled on the pair leader's barrier (same offset, CTA-rank bit cleared).
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1) {
  const uint32_t bar_leader = smem_u32(bar) & 0xFEFFFFFFu;
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(bar_leader), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, const void* src, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(map), "r"(smem_u32(src)), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// Bias of a warp's boxes (64 columns each): lane l holds columns 2 l and 2 l + 1 of a box, fetched before the wait for the
// products, and hands them round by shuffles.  (Every lane reading every column, 256 two-byte loads a tile, cost 3.3 us per
// tile: 8192 x 2304 x 768 launched back to back 38 us with a bias against 25 without; now 24.3 against 23.1.)
__device__ __forceinline__ uint32_t bias_pair(const GemmProblem& p, int col, int lane) {
  const unsigned short* bp = reinterpret_cast<const unsigned short*>(p.bias);
  const int c = col + 2 * lane;
  if (!bp) return 0u;
  return (c < p.N ? (uint32_t)bp[c] : 0u) | (c + 1 < p.N ? (uint32_t)bp[c + 1] << 16 : 0u);
}
__device__ __forceinline__ void add_bias(uint32_t (&ra)[32], uint32_t (&rb)[32], uint32_t pair) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const uint32_t wa = __shfl_sync(0xffffffffu, pair, i), wb = __shfl_sync(0xffffffffu, pair, 16 + i);
    ra[2 * i] = __float_as_uint(__uint_as_float(ra[2 * i]) + __uint_as_float(wa << 16));
    ra[2 * i + 1] = __float_as_uint(__uint_as_float(ra[2 * i + 1]) + __uint_as_float(wa & 0xffff0000u));
    rb[2 * i] = __float_as_uint(__uint_as_float(rb[2 * i]) + __uint_as_float(wb << 16));
    rb[2 * i + 1] = __float_as_uint(__uint_as_float(rb[2 * i + 1]) + __uint_as_float(wb & 0xffff0000u));
  }
}
// One box of 32 rows and 64 columns: `w` = the lane's row, packed bf16, through the warp's staging buffer `st` to `map`.
template <int EW>
__device__ __forceinline__ void store_box(const CUtensorMap* map, unsigned char* st, uint32_t& buf, const uint32_t (&w)[32], int col, int row0, bool inside, int lane) {
  st += buf;
  if (EW == 4) buf ^= 4096;
  if (lane == 0) bulk_wait_read<EW == 4 ? 1 : 0>();    // the store that read this buffer last is done
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 8; ++q) *reinterpret_cast<uint4*>(st + swz128(lane, q * 8)) = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
  fence_async_smem();
  __syncwarp();
  if (lane == 0) {
    if (inside) tma_store_2d(map, st, col, row0);
    bulk_commit();
  }
}
__device__ __forceinline__ void pack_box(const uint32_t (&ra)[32], const uint32_t (&rb)[32], uint32_t (&w)[32]) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    w[i] = pack_bf16(__uint_as_float(ra[2 * i]), __uint_as_float(ra[2 * i + 1]));
    w[16 + i] = pack_bf16(__uint_as_float(rb[2 * i]), __uint_as_float(rb[2 * i + 1]));
  }
}

// Output of boxes [cb_lo, cb_hi) of one tile with an activation: the product itself (with keep_c) and the activated values.  The
// activation reads the rounded values, as a kernel of its own would.
// (A gate and its factor in one tile, 128 columns of each, was slower than two kernels: 777 x 16 384 x 3072 80 -> 105 us, the
// two halves of the weight lie a power of two apart and share memory channels.)
template <int EW>
__device__ __forceinline__ void epilogue_act(const GemmGroup& gg, const GemmProblem& p, unsigned char* stg, uint32_t& buf, uint32_t taddr0, int n0, int row0,
                                             int cb_lo, int cb_hi, uint32_t bias, int lane) {
  const int mode = gg.act - 1;
#pragma unroll 1
  for (int cb = cb_lo; cb < cb_hi; ++cb) {
    const int col = n0 + cb * 64;
    const bool inside = col < p.N && row0 < p.M;
    const uint32_t next = bias_pair(p, col + 64, lane);
    uint32_t x[32];
    {
      uint32_t ra[32], rb[32];
      tmem_ld32_nowait(taddr0 + cb * 64, ra);
      tmem_ld32_nowait(taddr0 + cb * 64 + 32, rb);
      tmem_wait_ld();
      if (p.bias) add_bias(ra, rb, bias);
      bias = next;
      pack_box(ra, rb, x);
    }
    if (gg.keep_c) store_box<EW>(&p.tc, stg, buf, x, col, row0, inside, lane);
#pragma unroll
    for (int i = 0; i < 32; ++i)
      x[i] = pack_bf16(zen_act::value(mode, __uint_as_float(x[i] << 16), 0.f), zen_act::value(mode, __uint_as_float(x[i] & 0xffff0000u), 0.f));
    store_box<EW>(&gg.tact, stg, buf, x, col, row0, inside, lane);
  }
}

// Output of two boxes of one tile as logits: the product itself (with keep_c) and, for each row, the maximum of these up to 128
// columns and the sum of exponentials of what they lie below it, part[columns / 128][row]; the label's logit of a row goes to target[row]
// from whoever meets it.  CAP: of the soft-capped values cap tanh(x / cap); target is the value before.  Everything is made of
// the values as rounded for the store, so that a gradient taken from the stored ones belongs to the same distribution.  The
// products leave the special-function units idle: 8192 x 50 257 x 768 takes 463 us without and 470 with the statistics.
template <int EW, bool CAP>
__device__ __forceinline__ void epilogue_loss(const GemmGroup& gg, const GemmProblem& p, unsigned char* stg, uint32_t& buf, uint32_t taddr0, int n0, int row0,
                                              int cb_lo, int cb_hi, int lane) {
  typedef __nv_bfloat16 T;
  using zen_xe::ex2_fast;
  constexpr float L2E = zen_xe::L2E;
  const int row = row0 + lane;
  const float k2 = CAP ? 2.f * L2E / gg.cap : 0.f;
  const int64_t label = row < p.M ? gg.labels[row] : -1;
  float m = -INFINITY, s = 0.f;
#pragma unroll 1
  for (int cb = cb_lo; cb < cb_hi; ++cb) {
    const int col = n0 + cb * 64;
    if (col >= p.N) break;
    uint32_t w[32];
    {
      uint32_t ra[32], rb[32];
      tmem_ld32_nowait(taddr0 + cb * 64, ra);
      tmem_ld32_nowait(taddr0 + cb * 64 + 32, rb);
      tmem_wait_ld();
      pack_box(ra, rb, w);
    }
    if (gg.keep_c) store_box<EW>(&p.tc, stg, buf, w, col, row0, row0 < p.M, lane);
    auto at = [&](int i) { return __uint_as_float((i & 1) ? w[i >> 1] & 0xffff0000u : w[i >> 1] << 16); };
    const int64_t rel = label - col;
    if (__any_sync(0xffffffffu, rel >= 0 && rel < 64)) {
      float mine = 0.f;
#pragma unroll
      for (int i = 0; i < 64; ++i) mine = rel == i ? at(i) : mine;
      if (rel >= 0 && rel < 64 && label < p.N) gg.target[row] = mine;
    }
    if (col + 64 > p.N) {                                // the matrix ends in this box: columns beyond count for nothing
#pragma unroll
      for (int i = 0; i < 64; ++i)
        if (col + i >= p.N) w[i >> 1] = (i & 1) ? (w[i >> 1] & 0xffffu) | 0xff800000u : (w[i >> 1] & 0xffff0000u) | 0xff80u;
    }
    float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int i = 0; i < 64; ++i) mx[i & 3] = fmaxf(mx[i & 3], at(i));
    float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
    if (CAP) top = zen_xe::xent_cap<T, CAP>(top, gg.cap, k2);                      // monotonic; -inf becomes -cap (a box has columns inside)
    const float nm = fmaxf(m, top), ref = nm == -INFINITY ? 0.f : nm;
    float add[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 64; ++i) {
      const float y = zen_xe::xent_cap<T, CAP>(at(i), gg.cap, k2);
      const float e = ex2_fast((y - ref) * L2E);
      add[i & 3] += CAP && col + i >= p.N ? 0.f : e;     // (a soft-capped -inf is -cap)
    }
    s = s * ex2_fast((m - ref) * L2E) + ((add[0] + add[1]) + (add[2] + add[3]));
    m = nm;
  }
  if (row < p.M) gg.part[(size_t)((n0 + cb_lo * 64) / 128) * gg.part_ld + row] = make_float2(m, s);
}

// A transposed tile: the lane's column of the output, `narrow` rows of it in the columns of tensor memory.  Columns from N on are zero
// there, as B is filled up with zeros.
template <int HALVES>
__device__ __forceinline__ void store_narrow(const GemmGroup& gg, uint32_t taddr, int col, int half) {
  const GemmProblem& p = gg.pr[0];
  const float bias = p.bias && col < p.N ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.bias)[col]) : 0.f;
#pragma unroll 1
  for (int ch = half; ch < gg.narrow / 32; ch += HALVES) {
    uint32_t r[32];
    tmem_ld32(taddr + ch * 32, r);
    const int row = p.num_m_pairs * 256 + ch * 32;
    __nv_bfloat16* c = reinterpret_cast<__nv_bfloat16*>(p.C) + (size_t)row * p.ldc + col;
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (row + i < p.M && col < p.n_store) c[(size_t)i * p.ldc] = __float2bfloat16_rn(__uint_as_float(r[i]) + bias);
  }
}

template <bool A_MN, bool B_MN, int BN2, int EW, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(64 + EW * 32, 1)
gemm_bf16_2cta_kernel(const __grid_constant__ GemmGroup gg) {
  constexpr int BNH = PairCfg<BN2>::BNH, STAGES2 = PairCfg<BN2>::STAGES, STAGE_BYTES2 = PairCfg<BN2>::STAGE_BYTES;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* epi_stage = smem + STAGES2 * STAGE_BYTES2;              // 1024-byte aligned
  uint64_t* bars = reinterpret_cast<uint64_t*>(epi_stage + EPI_STAGE_BYTES);
  uint64_t* full = bars;                       // [STAGES2]   used on the leader
  uint64_t* empty = bars + STAGES2;            // [STAGES2]   one copy per CTA
  uint64_t* tfull = bars + 2 * STAGES2;        // [2]         one copy per CTA
  uint64_t* tempty = bars + 2 * STAGES2 + 2;   // [2]         used on the leader, one arrival per epilogue warp of the pair
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES2 + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  constexpr bool NARROW = EPI == EPI_STORE_NARROW;
  constexpr uint32_t IDESC = make_idesc(256, BN2, A_MN, B_MN), IDESC_HALF = make_idesc(256, BN2 / 2, A_MN, B_MN);
  constexpr int A_BYTES = BM2 * BK2 * 2;

  const int warp = (int)uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank();
  const int cluster_id = blockIdx.x >> 1, num_clusters = gridDim.x >> 1;
  const int num_tiles = gg.num_tiles;
  const int num_units = gg.tail ? num_tiles + gg.tail : num_tiles * gg.splits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES2; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&tfull[a], 1); mbar_init(&tempty[a], 2 * EW); }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, PairCfg<BN2>::TMEM_COLS);
  fence_before();
  __syncthreads();
  cluster_sync_all();                            // both CTAs' barriers exist before anyone signals them
  fence_after();
  zen_pdl::enter();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      // ---------------------------------------------------------------- TMA producer (both CTAs)
      uint32_t it = 0;
      bool ok = true;
      for (Units<NARROW> w(gg, cluster_id, num_clusters, num_units); w.more() && ok; w.advance()) {
        if (NARROW && w.unit() >= num_tiles) {
          const GemmProblem& p = gg.pr[0];
          const int n0 = (w.unit() - num_tiles) * 256 + (int)cta * BM2, m0 = p.num_m_pairs * 256 + (int)cta * (gg.narrow / 2);
          const uint32_t bytes = 2 * (A_BYTES + gg.narrow / 2 * (BK2 * 2));
          for (int kb = 0; kb < gg.kb_per_split; ++kb, ++it) {
            const int s = it % STAGES2;
            if (!mbar_wait(&empty[s], ((it / STAGES2) & 1) ^ 1, abort_flag, 1, &g_gemm2_error)) { ok = false; break; }
            unsigned char* sa = smem + s * STAGE_BYTES2;
            if (cta == 0) mbar_expect_tx(&full[s], bytes);
            const int k0 = kb * BK2;
            if (!B_MN) {
              tma_load_2d_pair(sa, &p.tb, &full[s], k0, n0);
            } else {
#pragma unroll
              for (int j = 0; j < BM2 / 64; ++j) tma_load_2d_pair(sa + j * 8192, &p.tb, &full[s], n0 + 64 * j, k0);
            }
            tma_load_2d_pair(sa + A_BYTES, &gg.ta_narrow, &full[s], k0, m0);
          }
          continue;
        }
        const Unit u = decode_unit(gg, w.unit());
        const GemmProblem& p = gg.pr[u.pi];
        int tm, tn;
        tile_coords(p, u.lt, tm, tn);
        const int nh = u.part ? BNH / 2 : BNH;               // rows of B that this CTA holds
        const int m0 = tm * 256 + (int)cta * BM2, n0 = tn * BN2 + (u.part == 2 ? BNH : 0) + (int)cta * nh;
        const uint32_t bytes = 2 * (A_BYTES + nh * (BK2 * 2));
        for (int kb = u.kb0; kb < u.kb1; ++kb, ++it) {
          const int s = it % STAGES2;
          const uint32_t ph = (it / STAGES2) & 1;
          if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, 1, &g_gemm2_error)) { ok = false; break; }
          unsigned char* sa = smem + s * STAGE_BYTES2;
          unsigned char* sb = sa + A_BYTES;
          if (cta == 0) mbar_expect_tx(&full[s], bytes);
          const int k0 = kb * BK2;
          if (!A_MN) {
            tma_load_2d_pair(sa, &p.ta, &full[s], k0, m0);
          } else {
#pragma unroll
            for (int j = 0; j < BM2 / 64; ++j) tma_load_2d_pair(sa + j * 8192, &p.ta, &full[s], m0 + 64 * j, k0);
          }
          if (!B_MN) {
            tma_load_2d_pair(sb, u.part ? &p.tb_half : &p.tb, &full[s], k0, n0);
          } else {
#pragma unroll
            for (int j = 0; j < BNH / 64; ++j)
              if (64 * j < nh) tma_load_2d_pair(sb + j * 8192, &p.tb, &full[s], n0 + 64 * j, k0);
          }
        }
      }
    }
  } else if (warp == 1) {
    if (cta == 0) {
      // ---------------------------------------------------------------- MMA issuer (leader CTA only; converged warp)
      const bool leader = elect_one();
      const uint32_t tmem_u = uniform(tmem_base);
      uint32_t it = 0, tcount = 0;
      bool ok = true;
      for (Units<NARROW> w(gg, cluster_id, num_clusters, num_units); w.more() && ok; w.advance(), ++tcount) {
        const uint32_t acc = tcount & 1, aph = (tcount >> 1) & 1;
        if (!mbar_wait(&tempty[acc], aph ^ 1, abort_flag, 2, &g_gemm2_error)) { ok = false; break; }
        fence_after();
        const uint32_t d_tmem = tmem_u + acc * BN2;
        const bool narrow = NARROW && w.unit() >= num_tiles;
        const Unit u = decode_unit(gg, narrow ? 0 : w.unit());           // (whole tiles share their blocks of K)
        const int kb0 = u.kb0, kb1 = u.kb1;
        const uint32_t idesc = narrow ? make_idesc(256, gg.narrow, B_MN, A_MN) : u.part ? IDESC_HALF : IDESC;
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % STAGES2;
          const uint32_t ph = (it / STAGES2) & 1;
          if (!mbar_wait(&full[s], ph, abort_flag, 3, &g_gemm2_error)) { ok = false; break; }
          fence_after();
          const uint32_t sa = smem_u32(smem + s * STAGE_BYTES2);
          const uint32_t sb = sa + A_BYTES;
          const bool a_mn = NARROW && narrow ? B_MN : A_MN, b_mn = NARROW && narrow ? A_MN : B_MN;
          const uint64_t adesc = a_mn ? make_desc(sa, 8192, 1024) : make_desc(sa, 16, 1024);
          const uint64_t bdesc = b_mn ? make_desc(sb, 8192, 1024) : make_desc(sb, 16, 1024);
          if (leader) {
#pragma unroll
            for (int j = 0; j < BK2 / 16; ++j) {
              const uint64_t astep = (uint64_t)((a_mn ? j * 2048 : j * 32) >> 4);
              const uint64_t bstep = (uint64_t)((b_mn ? j * 2048 : j * 32) >> 4);
              umma_bf16_pair(d_tmem, adesc + astep, bdesc + bstep, idesc, (kb != kb0 || j != 0) ? 1u : 0u);
            }
            umma_commit_pair(&empty[s]);
          }
        }
        if (ok && leader) umma_commit_pair(&tfull[acc]);
      }
    }
  } else {
    // -------------------------------------------------------------------- epilogue (warps 2.., both CTAs)
    constexpr int HALVES = EW / 4;
    const int grp = warp & 3, half = HALVES == 2 ? (warp - 2) >> 2 : 0;        // 32 rows, and which half of the tile's 64-column boxes
    constexpr int BOXES = BN2 / 64;
    unsigned char* stg = epi_stage + (warp - 2) * (EPI_STAGE_BYTES / EW);
    uint32_t buf = 0;
    uint32_t tcount = 0;
    bool ok = true;
    for (Units<NARROW> w(gg, cluster_id, num_clusters, num_units); w.more() && ok; w.advance(), ++tcount) {
      if (NARROW && w.unit() >= num_tiles) {
        if (!mbar_wait(&tfull[tcount & 1], (tcount >> 1) & 1, abort_flag, 4, &g_gemm2_error)) { ok = false; break; }
        fence_after();
        store_narrow<HALVES>(gg, tmem_base + ((uint32_t)(grp * 32) << 16) + (tcount & 1) * BN2,
                             (w.unit() - num_tiles) * 256 + (int)cta * BM2 + grp * 32 + lane, half);
        fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_leader(&tempty[tcount & 1]);
        continue;
      }
      const Unit u = decode_unit(gg, w.unit());
      const GemmProblem& p = gg.pr[u.pi];
      const int tile = u.tile, ks = u.ks;
      int tm, tn;
      tile_coords(p, u.lt, tm, tn);
      const int m0 = tm * 256 + (int)cta * BM2, n0 = tn * BN2 + (u.part == 2 ? BNH : 0);
      const uint32_t acc = tcount & 1, aph = (tcount >> 1) & 1;
      const bool split = BN2 == 256 && u.split;
      // this warp's boxes: half of the tile's, or with two K slices half of what its slice finishes
      const int boxes = u.part ? BOXES / 2 : BOXES;
      int cb_lo = half ? (boxes + 1) / 2 : 0, cb_hi = half || HALVES == 1 ? boxes : (boxes + 1) / 2;
      if (split && p.tma_store) { cb_lo = ks * 2 + half; cb_hi = cb_lo + 2 / HALVES; }
      uint32_t bias = bias_pair(p, n0 + cb_lo * 64, lane);
      if (!mbar_wait(&tfull[acc], aph, abort_flag, 4, &g_gemm2_error)) { ok = false; break; }
      fence_after();
      const int row = m0 + grp * 32 + lane;
      const uint32_t taddr0 = tmem_base + ((uint32_t)(grp * 32) << 16) + acc * BN2;
      if constexpr (EPI != EPI_STORE && EPI != EPI_STORE_NARROW) {
        if constexpr (EPI == EPI_ACT) epilogue_act<EW>(gg, p, stg, buf, taddr0, n0, m0 + grp * 32, cb_lo, cb_hi, bias, lane);
        else epilogue_loss<EW, EPI == EPI_LOSS_CAP>(gg, p, stg, buf, taddr0, n0, m0 + grp * 32, cb_lo, cb_hi, lane);
        fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_leader(&tempty[acc]);
        continue;
      }
      if (split && !p.tma_store) {
        // store this K slice's partial tile and count in.  Every slice but the last to arrive for these 32 rows is
        // done then; the last one adds the others' partials to its own accumulator, in slice order, below.
        float4* wp = reinterpret_cast<float4*>(gg.ws + ((size_t)(ks * num_tiles + tile) * 2 + cta) * (BM2 * BN2)) + (grp * 32 + lane);
#pragma unroll 1
        for (int ch = half * (BN2 / 64); ch < (half + 1) * (BN2 / 32 / HALVES); ch += 2) {
          uint32_t r[32], r2[32];
          tmem_ld32_nowait(taddr0 + ch * 32, r);
          tmem_ld32_nowait(taddr0 + ch * 32 + 32, r2);
          tmem_wait_ld();
          float4* dst = wp + (size_t)ch * (8 * BM2);
          float4* dst2 = wp + (size_t)(ch + 1) * (8 * BM2);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            dst[i * BM2] = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
            dst2[i * BM2] = make_float4(__uint_as_float(r2[4 * i]), __uint_as_float(r2[4 * i + 1]), __uint_as_float(r2[4 * i + 2]), __uint_as_float(r2[4 * i + 3]));
          }
        }
        __threadfence();
        __syncwarp();
        int* cnt = gg.counters + ((tile * 2 + (int)cta) * 4 + grp) * 2 + half;
        int old = 0;
        if (lane == 0) {
          old = atomicAdd(cnt, 1);
          if (old == gg.splits - 1) *cnt = 0;           // every slice has arrived: ready for the next launch
        }
        old = __shfl_sync(0xffffffffu, old, 0);
        if (old != gg.splits - 1) {
          fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_leader(&tempty[acc]);
          continue;
        }
        __threadfence();
      }
      if (p.tma_store) {
        // bf16 output: each warp turns its 32 rows into [32][64] boxes in shared memory (the swizzled layout of the
        // tensor map) and one lane stores each box with TMA: whole lines, clipped at the matrix edge, no waiting.
        // With two K slices each slice finishes half of the columns: it hands the other half of its accumulator to
        // the peer through the workspace, waits (bounded) for the peer's half and adds it to its own.
        const float4* peer = nullptr;
        if (split) {
          const int other = 1 - ks;
          float4* wp = reinterpret_cast<float4*>(gg.ws + ((size_t)(ks * u.wtiles + u.wtile) * 2 + cta) * (BM2 * BN2)) + (grp * 32 + lane);
#pragma unroll 1
          for (int give = other * 2 + half; give < other * 2 + half + 2 / HALVES; ++give) {      // the boxes that the peer finishes
            uint32_t r[32], r2[32];
            tmem_ld32_nowait(taddr0 + give * 64, r);
            tmem_ld32_nowait(taddr0 + give * 64 + 32, r2);
            tmem_wait_ld();
            float4* dst = wp + (size_t)(2 * give) * (8 * BM2);
            float4* dst2 = wp + (size_t)(2 * give + 1) * (8 * BM2);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              dst[i * BM2] = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
              dst2[i * BM2] = make_float4(__uint_as_float(r2[4 * i]), __uint_as_float(r2[4 * i + 1]), __uint_as_float(r2[4 * i + 2]), __uint_as_float(r2[4 * i + 3]));
            }
          }
          __threadfence();
          __syncwarp();
          // flags[..][ks], bit `half`: "slice ks has published this warp's box"; the consumer clears it for the next launch
          int* flags = gg.counters + ((u.wtile * 2 + (int)cta) * 4 + grp) * 2;
          int got = 1;
          if (lane == 0) {
            const int bit = 1 << half;
            atomicOr(flags + ks, bit);
            const uint64_t t0 = gtimer();
            while ((atomicAdd(flags + other, 0) & bit) == 0) {
              if (*abort_flag || gtimer() - t0 > WAIT_NS) { got = 0; break; }
            }
            if (got) atomicAnd(flags + other, ~bit);
            else { *abort_flag = 5; atomicCAS(&g_gemm2_error, 0, 5); }
          }
          got = __shfl_sync(0xffffffffu, got, 0);
          if (!got) { ok = false; break; }
          __threadfence();
          peer = reinterpret_cast<const float4*>(gg.ws + ((size_t)(other * u.wtiles + u.wtile) * 2 + cta) * (BM2 * BN2)) + (grp * 32 + lane);
        }
#pragma unroll 1
        for (int cb = cb_lo; cb < cb_hi; ++cb) {
          uint32_t ra[32], rb[32];
          const uint32_t next = bias_pair(p, n0 + cb * 64 + 64, lane);
          tmem_ld32_nowait(taddr0 + cb * 64, ra);
          tmem_ld32_nowait(taddr0 + cb * 64 + 32, rb);
          if (split) {
            float4 oa[8], ob[8];
            const float4* qa = peer + (size_t)(2 * cb) * (8 * BM2);
            const float4* qb = peer + (size_t)(2 * cb + 1) * (8 * BM2);
#pragma unroll
            for (int i = 0; i < 8; ++i) { oa[i] = __ldcg(qa + i * BM2); ob[i] = __ldcg(qb + i * BM2); }
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              ra[4 * i] = __float_as_uint(__uint_as_float(ra[4 * i]) + oa[i].x);
              ra[4 * i + 1] = __float_as_uint(__uint_as_float(ra[4 * i + 1]) + oa[i].y);
              ra[4 * i + 2] = __float_as_uint(__uint_as_float(ra[4 * i + 2]) + oa[i].z);
              ra[4 * i + 3] = __float_as_uint(__uint_as_float(ra[4 * i + 3]) + oa[i].w);
              rb[4 * i] = __float_as_uint(__uint_as_float(rb[4 * i]) + ob[i].x);
              rb[4 * i + 1] = __float_as_uint(__uint_as_float(rb[4 * i + 1]) + ob[i].y);
              rb[4 * i + 2] = __float_as_uint(__uint_as_float(rb[4 * i + 2]) + ob[i].z);
              rb[4 * i + 3] = __float_as_uint(__uint_as_float(rb[4 * i + 3]) + ob[i].w);
            }
          } else {
            tmem_wait_ld();
          }
          const int col0 = n0 + cb * 64;
          if (p.bias) add_bias(ra, rb, bias);
          bias = next;
          uint32_t w[32];
          pack_box(ra, rb, w);
          store_box<EW>(&p.tc, stg, buf, w, col0, m0 + grp * 32, col0 < p.N && m0 + grp * 32 < p.M, lane);
        }
        fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_leader(&tempty[acc]);
        continue;
      }
      // 32-column chunks of this warp: as many as its boxes of 64 would be (192-wide tiles: three of six)
      const int chunks = (u.part ? BN2 / 64 : BN2 / 32) / HALVES;
#pragma unroll 1
      for (int ch = half * chunks; ch < (half + 1) * chunks; ++ch) {
        uint32_t r[32];
        if (split) {
          // the sum runs over slice indices whichever slice arrived last; one slice's partials in flight at a time (all of
          // them do not fit in the registers)
          const float4* src = reinterpret_cast<const float4*>(gg.ws + ((size_t)tile * 2 + cta) * (BM2 * BN2)) + (size_t)ch * (8 * BM2) + (grp * 32 + lane);
          tmem_ld32(taddr0 + ch * 32, r);
          float a[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) a[i] = 0.f;
#pragma unroll 1
          for (int sidx = 0; sidx < gg.splits; ++sidx) {
            if (sidx == ks) {
#pragma unroll
              for (int i = 0; i < 32; ++i) a[i] += __uint_as_float(r[i]);
            } else {
              const float4* q = src + (size_t)sidx * num_tiles * 2 * (BM2 * BN2 / 4);
              float4 buf[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) buf[i] = __ldcg(q + i * BM2);
#pragma unroll
              for (int i = 0; i < 8; ++i) { a[4 * i] += buf[i].x; a[4 * i + 1] += buf[i].y; a[4 * i + 2] += buf[i].z; a[4 * i + 3] += buf[i].w; }
            }
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(a[i]);
        } else {
          tmem_ld32(taddr0 + ch * 32, r);
        }
        const int col0 = n0 + ch * 32;
        if (row < p.M && col0 < p.N) {
          float v[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
          const bool fullw = (col0 + 32 <= p.N);
          if (p.bias) {
            const __nv_bfloat16* bp = reinterpret_cast<const __nv_bfloat16*>(p.bias) + col0;
#pragma unroll
            for (int i = 0; i < 32; ++i) if (fullw || col0 + i < p.N) v[i] += __bfloat162float(bp[i]);
          }
          if (p.out_fp32) {
            float* cp = reinterpret_cast<float*>(p.C) + (size_t)row * p.ldc + col0;
            if (fullw && (p.ldc % 4 == 0)) {
#pragma unroll
              for (int i = 0; i < 32; i += 4) {
                float4 o = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                if (p.accumulate) { const float4 c = *reinterpret_cast<const float4*>(cp + i); o.x += c.x; o.y += c.y; o.z += c.z; o.w += c.w; }
                *reinterpret_cast<float4*>(cp + i) = o;
              }
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (col0 + i < p.N) cp[i] = p.accumulate ? cp[i] + v[i] : v[i];
            }
          } else {
            __nv_bfloat16* cp = reinterpret_cast<__nv_bfloat16*>(p.C) + (size_t)row * p.ldc + col0;
            if (fullw && (p.ldc % 8 == 0)) {
#pragma unroll
              for (int i = 0; i < 32; i += 8) {
                if (p.accumulate) {
                  const uint4 c = *reinterpret_cast<const uint4*>(cp + i);
                  const uint32_t w[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
                  for (int q = 0; q < 4; ++q) { v[i + 2 * q] += __uint_as_float(w[q] << 16); v[i + 2 * q + 1] += __uint_as_float(w[q] & 0xffff0000u); }
                }
                *reinterpret_cast<uint4*>(cp + i) = make_uint4(pack_bf16(v[i], v[i + 1]), pack_bf16(v[i + 2], v[i + 3]),
                                                               pack_bf16(v[i + 4], v[i + 5]), pack_bf16(v[i + 6], v[i + 7]));
              }
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                if (col0 + i < p.N) {
                  const float o = p.accumulate ? __bfloat162float(cp[i]) + v[i] : v[i];
                  cp[i] = __float2bfloat16_rn(o);
                }
              }
            }
          }
        }
      }
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_leader(&tempty[acc]);
    }
    if (lane == 0) bulk_wait_all();                    // shared memory stays valid until the last store has read it
  }

  // ---------------------------------------------------------------------- teardown
  fence_before();
  __syncthreads();
  if (*abort_flag) {
    const uint64_t t0 = gtimer();
    while (gtimer() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  cluster_sync_all();                            // the peer may still be reading this CTA's shared memory / barriers
  if (warp == 1) {
    fence_after();
    tmem_dealloc_pair(tmem_base, PairCfg<BN2>::TMEM_COLS);
  }
}

template <bool A_MN, bool B_MN, int BN2, int EW, int EPI = EPI_STORE>
int launch2_as(const GemmGroup& g, cudaStream_t st) {
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(gemm_bf16_2cta_kernel<A_MN, B_MN, BN2, EW, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, pair_smem_bytes<BN2>());
    if (e != cudaSuccess) return (int)e;
    attr_set = true;
  }
  const int units = EPI == EPI_STORE_NARROW ? g.num_tiles + g.pr[0].num_n_tiles : g.tail ? g.num_tiles + g.tail : g.num_tiles * g.splits;
  int clusters = zen_tmap::sm_count() / 2;
  if (units < clusters) clusters = units;
  zen_pdl::launch(gemm_bf16_2cta_kernel<A_MN, B_MN, BN2, EW, EPI>, clusters * 2, 64 + EW * 32, pair_smem_bytes<BN2>(), st, g);
  return (int)cudaGetLastError();
}

template <bool A_MN, bool B_MN, int BN2>
int launch2(const GemmGroup& g, cudaStream_t st) {
  return g.pr[0].bias ? launch2_as<A_MN, B_MN, BN2, 8>(g, st) : launch2_as<A_MN, B_MN, BN2, 4>(g, st);   // a group has no bias
}

int launch2_layout(const GemmGroup& g, int a_mn, int b_mn, int bn, cudaStream_t st) {
#define LAUNCH2(BN_)                                                   \
  do {                                                                 \
    if (!a_mn && !b_mn) return launch2<false, false, BN_>(g, st);      \
    if (!a_mn && b_mn) return launch2<false, true, BN_>(g, st);        \
    if (a_mn && !b_mn) return launch2<true, false, BN_>(g, st);        \
    return launch2<true, true, BN_>(g, st);                            \
  } while (0)
  if (bn == 128) LAUNCH2(128);
  if (bn == 192) {                                             // K-major B only (see pick_pair_bn)
    if (!a_mn) return launch2<false, false, 192>(g, st);
    return launch2<true, false, 192>(g, st);
  }
  LAUNCH2(256);
#undef LAUNCH2
}

// Order of the output tiles.  All 74 clusters walk K side by side, so a wave fetches one panel of A per tile row and one of
// B per tile column it touches.  When one operand fits in half of the L2 beside the stream of the other, that operand stays
// and the other is read once: rows fastest over all of A, or columns fastest over all of B.  When neither fits (a weight
// gradient or an input gradient of a wide MLP: K = 8 192 tokens or 32 768 columns), blocks of 8 tile rows make a wave about
// as high as wide.  32768 x 2048 x 8192 with rows fastest fetched each of 128 A panels (4 MB) for every one of 8 columns,
// 4.3 GB for 0.6 GB of operands.
int pick_group_m(int M, int N, int K, int num_m) {
  constexpr uint64_t kHalfL2 = 60ull << 20;
  if ((uint64_t)M * K * 2 <= kHalfL2) return num_m;
  if ((uint64_t)N * K * 2 <= kHalfL2) return 1;
  return num_m < 8 ? num_m : 8;
}

// Tensor maps, tile counts and the output path of one product.  n_store: 0, or a width in [N, ldc] that the kernel may
// write (columns N.. receive zeros); max_slices: K slices that will write this output (the TMA-store path sums at most two).
int fill_problem(GemmProblem& q, const void* A, const void* B, void* C, const void* bias, int M, int N, int K, int lda,
                 int ldb, int ldc, int a_mn, int b_mn, int out_fp32, int accumulate, int n_store, int bn, int max_slices) {
  if (M <= 0 || N <= 0 || K <= 0) return -1;
  if ((lda % 8) || (ldb % 8) || (reinterpret_cast<uintptr_t>(A) % 16) || (reinterpret_cast<uintptr_t>(B) % 16)) return -2;
  int rc;
  if (!a_mn) rc = zen_tmap::get(A, (uint64_t)K, (uint64_t)M, (uint64_t)lda, 64, 128, &q.ta);
  else rc = zen_tmap::get(A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, 64, 64, &q.ta);
  if (rc) return rc;
  if (!b_mn) rc = zen_tmap::get(B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb, 64, (uint32_t)(bn / 2), &q.tb);
  else rc = zen_tmap::get(B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, 64, 64, &q.tb);
  if (rc) return rc;
  q.tb_half = q.tb;
  if (!b_mn && bn == 256 && (rc = zen_tmap::get(B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb, 64, 64, &q.tb_half))) return rc;
  // Plain bf16 output with a TMA-compatible layout: store through shared memory.  The stored width must be a
  // multiple of 8 columns (16 bytes); a caller whose buffer has spare columns after N may allow them to be written
  // (with zeros) by passing n_store = N rounded up.
  if (n_store < N || n_store > ldc) n_store = N;
  q.tma_store = (C && !out_fp32 && !accumulate && max_slices <= 2 && (ldc % 8) == 0 && (n_store % 8) == 0 &&
                 (reinterpret_cast<uintptr_t>(C) % 16) == 0) ? 1 : 0;
  q.tc = q.ta;
  if (q.tma_store) {
    rc = zen_tmap::get(C, (uint64_t)n_store, (uint64_t)M, (uint64_t)ldc, 64, 32, &q.tc);
    if (rc) return rc;
  }
  q.n_store = n_store;
  q.C = C; q.bias = bias; q.M = M; q.N = N; q.K = K; q.ldc = ldc; q.out_fp32 = out_fp32; q.accumulate = accumulate;
  q.num_m_pairs = (M + 255) / 256;
  q.num_n_tiles = (N + bn - 1) / bn;
  q.group_m = pick_group_m(M, N, K, q.num_m_pairs);
  q.tile_start = 0;
  return 0;
}

}  // namespace

int g_force_bn = 0;
int g_tail_min_kb = 1;             // fewest 64-wide K blocks for which the tiles of the last wave are cut in two; 0 = never

// The tiles of the last, partly filled wave of clusters run as two units each when both units of all of them fit in that wave.
// Halves of 128 columns need nothing from each other and sum every element in the order of a whole tile, but each reads its
// rows of A again, and what bounds a tile is what its SMs draw from L2: three quarters of a tile's time.  K halves take half
// of it, and about 4 us to exchange half an accumulator each through memory (and need the TMA store and a workspace).  us, K halves /
// column halves: the 108 tiles of a GPT-2 layer's weight gradients, K = 8192, 75 / 80; 8192 x 768 x 3072 40.9 / 40.9;
// 8192 x 768 x 2304 34.7 / 32.7; 8192 x 3072 x 768 38.8 (whole) / 36.8; 700 x 2304 x 9216 without a workspace 55.1 (whole) / 47.0.
// By time the line would lie near K = 4096.  It lies at 1024, where the sum of a tile's two halves has been taken since K was
// first cut, and for single products not in outputs of one round, which split_k_choice cuts where that pays (no plan sees the tiles of
// a group): another order of summation in one tile of ten moves the logits of a four-layer Llama by up to 1.2 % (2 x 600 and 1 x 2048
// tokens), as much as any rounding there, and scores should not change by that for 2 us.
// Groups of less than a round have no last round to balance, so time alone decides: from K = 2304 on.  us, K halves / column halves: 12
// tiles (a layer 256 wide) of K = 1024 11.8 / 9.5, 2048 14.3 / 13.9, 4096 19.2 / 22.6, 8192 29.2 / 39.9; 36 tiles 12.4 / 9.7, 14.9 / 14.4,
// 20.1 / 23.5, 32.4 / 41.4.
constexpr int TAIL_K_MIN_KB = 16, ONE_ROUND_K_MIN_KB = 36;
// ws_floats, n_counters: what the caller's workspace holds; one_round: K also where all tiles fit one round.
static void cut_tail(GemmGroup& g, int min_kb, uint64_t ws_floats = 0, int n_counters = 0, bool one_round = false) {
  const int clusters = zen_tmap::sm_count() / 2, rem = g.num_tiles % clusters;
  g.tail = g_tail_min_kb > 0 && min_kb >= g_tail_min_kb && 2 * rem <= clusters ? rem : 0;
  const bool room = g.ws && g.counters && reinterpret_cast<uintptr_t>(g.ws) % 16 == 0 && ws_floats >= (uint64_t)g.tail * 2 * 2 * BM2 * 256 &&
                    n_counters >= g.tail * 16;
  g.tail_k = g.tail > 0 && room && (g.num_tiles > clusters ? min_kb >= TAIL_K_MIN_KB : one_round && min_kb >= ONE_ROUND_K_MIN_KB);
  for (int i = 0; i < g.n && g.tail_k; ++i) {
    const int end = g.pr[i].tile_start + g.pr[i].num_m_pairs * g.pr[i].num_n_tiles;
    if (end > g.num_tiles - g.tail && !g.pr[i].tma_store) g.tail_k = 0;
  }
}
// Rows beyond the last whole 256: up to 128 of them as transposed tiles, 256 columns of the output (rows of B) as the
// rows of the MMA and these rows of A, rounded up to 32, as its columns.  Such a tile draws half as much from L2 and takes about
// 0.78 of a whole one's time (its stages are as many, and half as full).  Taken where the rounds, so weighed, come out shorter by
// 3 %; the clusters that would be idle in the last round take up to three.  In practice that is an output many rounds long: us, whole tiles /
// with transposed ones, 777 x 128256 x 3072 494 / 454, 1300 x 16384 x 2048 71.7 / 68.6, 300 x 50257 x 768 41.0 / 40.0; but
// 777 x 16384 x 3072 70.6 / 73.3, 2100 x 2304 x 768 19.0 / 20.0 and 3100 x 7680 x 2560 86 / 89, which the weights leave whole.
// last: no product reads the output (logits), so the order of summation may change with it, see cut_tail.
static bool narrow_rows(GemmGroup& g, const void* A, int lda, int min_kb, bool last) {
  GemmProblem& p = g.pr[0];
  const int clusters = zen_tmap::sm_count() / 2, rows = p.M % 256;
  if (g_tail_min_kb <= 0 || min_kb < g_tail_min_kb || p.M < 256 || rows == 0 || rows > 128 || !p.tma_store) return false;
  if (g.tail_k && !last) return false;
  const int width = (rows + 31) / 32 * 32, cols = p.num_n_tiles, tiles = (p.num_m_pairs - 1) * cols;
  const double cost = 0.75 + width / 1024.0;
  const int now_rem = g.num_tiles % clusters;
  const double now = g.num_tiles / clusters + (now_rem == 0 ? 0.0 : g.tail ? (g.tail_k ? 0.6 : 0.75) : 1.0);
  const int rounds = tiles / clusters, rem = tiles % clusters, idle = clusters - rem;
  double best = now * 0.97;
  int first = -1;
  for (int k = 0; k <= (rem ? 3 : 0); ++k) {
    const int head = k * idle < cols ? k * idle : cols, rest = cols - head, after = rest > idle ? rest - idle : 0;
    const double early = rounds + ((head + idle - 1) / idle + (rest + clusters - 1) / clusters) * cost;
    const double late = rounds + (rem ? 1 : 0) + (after + clusters - 1) / clusters * cost;
    const double t = early > late ? early : late;
    if (t < best) { best = t; first = k; }
  }
  if (first < 0) return false;
  if (zen_tmap::get(A, (uint64_t)p.K, (uint64_t)p.M, (uint64_t)lda, 64, (uint32_t)(width / 2), &g.ta_narrow)) return false;
  g.narrow = width;
  g.narrow_first = first;
  --p.num_m_pairs;
  p.group_m = pick_group_m(p.M, p.N, p.K, p.num_m_pairs);
  g.num_tiles = tiles;
  g.tail = g.tail_k = 0;
  return true;
}

// 256-wide pair tiles.  The narrower ones exist for outputs whose 256-wide tiles fill the 74 CTA pairs unevenly: 8192 x 768 is
// 96 tiles of 256, 1.3 rounds, or 128 tiles of 192 (K-major B only: its half of 96 rows is one TMA box; an MN-major half would
// need one and a half 64-column boxes).  Back to back on a B200, us with tiles of 256 / 192 / 128 columns:
//   8192 x 768 x 768    14.4 / 14.5 / 14.9      8192 x 768 x 3072   33.5 / 33.4 / 38.3
//   8192 x 3072 x 768   32.2 / 32.7 / 40.2      4096 x 3072 x 8192   143 / 150 / 186
// With half the columns the A rows are fetched twice as often.  192 columns gain nothing where they even out the rounds (with a
// cold L2, 8192 x 768 x 768 takes 18.7 us instead of 20.5) and lose 2 to 5 % elsewhere.  Both are taken only when forced.
int pick_pair_bn(int M, int N, int b_mn, int splits) {
  (void)M; (void)N;
  if (g_force_bn == 192) return (!b_mn && splits == 1) ? 192 : 256;
  return g_force_bn ? g_force_bn : 256;
}

extern "C" {

// Same contract as zen_gemm_bf16 (without the tile choice): C[M,N] (+)= A * B^T (+ bias), CTA-pair kernel.
// splits > 1 cuts K into that many slices per output tile (for outputs with too few tiles to fill the GPU and a
// long K, the weight-gradient shape): `ws` must hold splits * tiles * 2 * 128 * 256 floats and `counters`
// tiles * 16 ints that are zero on entry (the kernel leaves them zero); both are caller-owned and used in stream
// order.  The slices are summed in slice order, so the result does not depend on timing.
// With splits == 1 a caller may still pass `ws` and `counters` (as for two slices of the tiles of a partly filled last wave): these may
// then be cut along K (cut_tail).
// n_store: 0, or a width in [N, ldc] that the kernel may write (columns N.. receive zeros).  last: no product reads the output.
int zen_gemm_bf16_2cta_splitk(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, int lda,
                              int ldb, int ldc, int a_mn, int b_mn, int out_fp32, int accumulate, int splits, float* ws,
                              uint64_t ws_floats, int* counters, int n_counters, int n_store, int last, void* stream);

int zen_gemm_bf16_2cta(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, int lda, int ldb,
                       int ldc, int a_mn, int b_mn, int out_fp32, int accumulate, void* stream) {
  return zen_gemm_bf16_2cta_splitk(A, B, C, bias, M, N, K, lda, ldb, ldc, a_mn, b_mn, out_fp32, accumulate, 1, nullptr, 0,
                                   nullptr, 0, 0, 0, stream);
}

int zen_gemm_bf16_2cta_splitk(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, int lda,
                              int ldb, int ldc, int a_mn, int b_mn, int out_fp32, int accumulate, int splits, float* ws,
                              uint64_t ws_floats, int* counters, int n_counters, int n_store, int last, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0) return -1;
  const int nkb = (K + BK2 - 1) / BK2;
  if (splits < 1) splits = 1;
  if (splits > MAX_SPLITS) splits = MAX_SPLITS;
  if (splits > nkb) splits = nkb;
  int kb_per = (nkb + splits - 1) / splits;
  splits = (nkb + kb_per - 1) / kb_per;                     // no empty slice
  if (splits > 1) {
    // The two slices of a tile hand each other half of the columns and wait for it: both must be resident at the
    // same time, i.e. every (tile, slice) unit needs its own cluster in the one wave that the launch has.
    const uint64_t units = (uint64_t)((M + 255) / 256) * ((N + 255) / 256) * (uint64_t)splits;
    if (units > (uint64_t)(zen_tmap::sm_count() / 2)) { splits = 1; kb_per = nkb; }
  }
  const int bn = (splits > 1) ? 256 : pick_pair_bn(M, N, b_mn, splits);
  if (splits > 1) {
    const uint64_t tiles = (uint64_t)((M + 255) / 256) * ((N + 255) / 256);
    if (!ws || !counters || ws_floats < tiles * splits * 2 * BM2 * 256 || (uint64_t)n_counters < tiles * 16) return -4;
    if (reinterpret_cast<uintptr_t>(ws) % 16) return -2;
  }
  GemmGroup g;
  g.act = g.keep_c = 0;
  int rc = fill_problem(g.pr[0], A, B, C, bias, M, N, K, lda, ldb, ldc, a_mn, b_mn, out_fp32, accumulate, n_store, bn, splits);
  if (rc) return rc;
  g.n = 1;
  g.num_tiles = g.pr[0].num_m_pairs * g.pr[0].num_n_tiles;
  g.splits = splits;
  g.kb_per_split = kb_per;
  g.ws = ws;
  g.counters = counters;
  g.tail = g.tail_k = 0;
  if (splits == 1 && bn == 256) {
    cut_tail(g, nkb, ws_floats, n_counters);
    if (!a_mn && narrow_rows(g, A, lda, nkb, last != 0)) {
      if (bias) return b_mn ? launch2_as<false, true, 256, 8, EPI_STORE_NARROW>(g, (cudaStream_t)stream) : launch2_as<false, false, 256, 8, EPI_STORE_NARROW>(g, (cudaStream_t)stream);
      return b_mn ? launch2_as<false, true, 256, 4, EPI_STORE_NARROW>(g, (cudaStream_t)stream) : launch2_as<false, false, 256, 4, EPI_STORE_NARROW>(g, (cudaStream_t)stream);
    }
  }
  return launch2_layout(g, a_mn, b_mn, bn, (cudaStream_t)stream);
}

// Product and activation in one launch: act_out [M, N] (row stride ld_act) = activation of C = A B' (+ bias), `mode` 0 or 1 as in
// zen_act_fwd.  C (row stride ldc) is written only with keep_c.  K-major A.
int zen_gemm_bf16_2cta_act(const void* A, const void* B, void* C, const void* bias, void* act_out, int M, int N, int K, int lda, int ldb,
                           int ldc, int b_mn, int mode, int ld_act, int keep_c, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || mode < 0 || mode > 1) return -1;
  if (N % 8 || ld_act % 8 || reinterpret_cast<uintptr_t>(act_out) % 16) return -2;
  GemmGroup g;
  int rc = fill_problem(g.pr[0], A, B, C, bias, M, N, K, lda, ldb, ldc, 0, b_mn, 0, 0, 0, 256, 1);
  if (!rc && !g.pr[0].tma_store) rc = -2;
  if (!rc) rc = zen_tmap::get(act_out, (uint64_t)N, (uint64_t)M, (uint64_t)ld_act, 64, 32, &g.tact);
  if (rc) return rc;
  g.n = 1;
  g.num_tiles = g.pr[0].num_m_pairs * g.pr[0].num_n_tiles;
  g.splits = 1;
  g.kb_per_split = (K + BK2 - 1) / BK2;
  g.ws = nullptr; g.counters = nullptr;
  cut_tail(g, g.kb_per_split);
  g.act = mode + 1; g.keep_c = keep_c;
  return b_mn ? launch2_as<false, true, 256, 8, EPI_ACT>(g, (cudaStream_t)stream) : launch2_as<false, false, 256, 8, EPI_ACT>(g, (cudaStream_t)stream);
}

// Logits C[M, N] = A[M, K] B[N, K]' (bf16, K-major operands; C null: not written) and what a cross-entropy needs of them:
// part [2 * ceil(N / 256)][part_ld] (maximum, sum of exponentials) of 128 columns of each row, target[row] the label's logit of rows
// whose label lies in [0, N) (others are left alone).  softcap > 0: of the soft-capped logits, with target as stored.
int zen_gemm_bf16_2cta_loss(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc, int n_store,
                            const int64_t* labels, void* part, int part_ld, float* target, float softcap, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || part_ld < M || !labels || !part || !target) return -1;
  GemmGroup g;
  int rc = fill_problem(g.pr[0], A, B, C, nullptr, M, N, K, lda, ldb, ldc, 0, 0, 0, 0, n_store, 256, 1);
  if (!rc && C && !g.pr[0].tma_store) rc = -2;
  if (rc) return rc;
  g.n = 1;
  g.num_tiles = g.pr[0].num_m_pairs * g.pr[0].num_n_tiles;
  g.splits = 1;
  g.kb_per_split = (K + BK2 - 1) / BK2;
  g.ws = nullptr; g.counters = nullptr;
  g.tail = g.tail_k = 0;                                 // a piece of 128 columns belongs to one warp
  g.act = 0; g.keep_c = C != nullptr;
  g.labels = labels; g.part = (float2*)part; g.part_ld = part_ld; g.target = target; g.cap = softcap;
  return softcap > 0.f ? launch2_as<false, false, 256, 8, EPI_LOSS_CAP>(g, (cudaStream_t)stream)
                       : launch2_as<false, false, 256, 8, EPI_LOSS>(g, (cudaStream_t)stream);
}

// Several products with the same operand layouts in ONE launch (see GemmProblem): the tiles of all of them form one
// list that the persistent clusters walk, and the tiles of the last, partly filled wave are cut in two (cut_tail).  `descs`: n
// records of ZenGemmDesc; every product follows the contract of zen_gemm_bf16_2cta (no bias).  ws / counters as for
// zen_gemm_bf16_2cta_splitk (may be null: K is not cut).
struct ZenGemmDesc {
  const void* A;
  const void* B;
  void* C;
  int32_t M, N, K, lda, ldb, ldc;
  int32_t out_fp32, accumulate;
};
int zen_gemm_desc_size() { return (int)sizeof(ZenGemmDesc); }
int zen_gemm_group_max() { return MAX_GROUP; }

int zen_gemm_bf16_2cta_group(const ZenGemmDesc* descs, int n, int a_mn, int b_mn, float* ws, uint64_t ws_floats,
                             int* counters, int n_counters, void* stream) {
  if (!descs || n < 1 || n > MAX_GROUP) return -1;
  GemmGroup g;
  g.act = g.keep_c = 0;
  int tiles = 0, min_kb = 1 << 30;
  for (int i = 0; i < n; ++i) {
    const ZenGemmDesc& d = descs[i];
    int rc = fill_problem(g.pr[i], d.A, d.B, d.C, nullptr, d.M, d.N, d.K, d.lda, d.ldb, d.ldc, a_mn, b_mn, d.out_fp32,
                          d.accumulate, 0, 256, 2);
    if (rc) return rc;
    g.pr[i].tile_start = tiles;
    tiles += g.pr[i].num_m_pairs * g.pr[i].num_n_tiles;
    const int nkb = (d.K + BK2 - 1) / BK2;
    if (nkb < min_kb) min_kb = nkb;
  }
  g.n = n;
  g.num_tiles = tiles;
  g.splits = 1;
  g.kb_per_split = 1 << 30;
  g.ws = ws;
  g.counters = counters;
  cut_tail(g, min_kb, ws_floats, n_counters, true);
  return launch2_layout(g, a_mn, b_mn, 256, (cudaStream_t)stream);
}

// 0 = choose the N tile per call, 128 / 256 = force it (tests, measurements); returns the previous setting.
int zen_gemm2_force_bn(int bn) {
  const int old = g_force_bn;
  if (bn == 0 || bn == 128 || bn == 192 || bn == 256) g_force_bn = bn;
  return old;
}

// Fewest K blocks (of 64) from which the tiles of a launch's last, partly filled wave run as two units; 0 switches
// that off.  Returns the previous setting.
int zen_gemm2_tail_split(int min_kb) {
  const int old = g_tail_min_kb;
  if (min_kb >= 0) g_tail_min_kb = min_kb;
  return old;
}

int zen_gemm2_error() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_gemm2_error, sizeof(int)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(g_gemm2_error, &zero, sizeof(int));
  return v;
}

}  // extern "C"
