// Causal self-attention for head sizes up to 128 (any multiple of 8) and any sequence length, forward and backward, on
// tcgen05 tensor cores with P and dS kept in tensor memory (sm_100a).
//
// Operands are read through 4-D tensor maps (head_dim, heads, sequence, batch) over the fused projection
// qkv[B*S, (Hq + 2*Hkv) * hd], so a head size that is not a multiple of 64 and a sequence that is not a multiple of 128
// are zero-filled by TMA on the way into shared memory: nothing is padded or copied in memory, and the tensor core
// multiplies hd / 16 (not 128 / 16) steps.
//
// What bounds it: per 128 x 128 score tile the tensor core needs 512 cycles per product (hd 128) and the MUFU 1024
// cycles for the exponentials (16 per SM and cycle), so a kernel whose softmax and products run one after the other
// leaves both idle half of the time.  Two things follow.
//  * P (forward, dK / dV) and dS (both backward kernels) go from the softmax warps straight into tensor memory, where
//    they are the A operand of the next product: no shared-memory round trip, no proxy fence, and 32 KB of shared
//    memory less.
//  * The products of one tile run while the softmax warps are busy with another: two query tiles per CTA take turns in
//    the forward kernel; the next scores are issued ahead of the accumulating product in the backward kernels.
//
// Backward, no atomics, results do not depend on the schedule:
//  * with scratch for dS (zen_flash_ds_bytes): D = rowsum(dO * O), then the dK / dV kernel, which also leaves dS as bf16 tiles in the
//    layout that the tensor core reads, then dQ as one product per tile over them;
//  * else dQ kernel (also computes D), then dK / dV kernel: two products and the exponentials of every tile twice.
//  All mbarrier waits are bounded.
#include "attention_common.cuh"
#include "launch.cuh"
#include "tmap_util.cuh"

namespace {

using namespace tc;

__device__ int g_flash_error = 0;

struct FlashParams {
  __nv_bfloat16* out;            // forward: O [B*S, Hq*hd]
  float* lse2;                   // [B*Hq, Sp] base-2 log-sum-exp of the scaled scores; +inf beyond S
  const __nv_bfloat16* o_in;     // backward: O and dO, row stride ld_o
  const __nv_bfloat16* dout;
  __nv_bfloat16* dqkv;           // backward: [B*S, (Hq + 2*Hkv)*hd], row stride ld_dqkv
  float* stat;                   // backward: [2][B*Hq, Sp]: -lse2 and -D, made before the dK / dV kernel
  unsigned char* ds;             // backward: dS tiles (see flash_bwd_dq_tiles_kernel), or null
  int B, S, Sp, Hq, Hkv, hd;
  int ld_o, ld_dqkv;
  float scale_log2, scale;
};

// D [128 x N] (+)= A B' over `ksteps` steps of 16, both operands K-major tiles ([64-column atom][row] of 128 bytes).
__device__ __forceinline__ void umma_tile_ss(uint32_t d, uint32_t a, uint32_t b, int ksteps, uint32_t idesc) {
  const uint64_t ad = make_desc(a, 16, 1024), bd = make_desc(b, 16, 1024);
#pragma unroll
  for (int kk = 0; kk < 8; ++kk)
    if (kk < ksteps) {
      const uint64_t off = (uint64_t)(((kk >> 2) * 16384 + (kk & 3) * 32) >> 4);
      umma_bf16(d, ad + off, bd + off, idesc, kk > 0 ? 1u : 0u);
    }
}
// D [128 x N] (+)= A B over 64 rows of B (MN-major tile, rows of 128 bytes), A in tensor memory.
__device__ __forceinline__ void umma_tile_ts(uint32_t d, uint32_t ta, uint32_t b, uint32_t idesc, bool first) {
  const uint64_t bd = make_desc(b, 16384, 1024);
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) umma_bf16_ts(d, ta + kk * 8, bd + (uint64_t)(kk * 128), idesc, (first && kk == 0) ? 0u : 1u);
}
// Byte offset of a dS tile: 128 queries x 128 keys as [16 pieces of 8 queries][128 keys][8 queries] (32 KB), the tiles of a query tile
// in key order, query tiles of a head in order.
constexpr int DS_TILE = 32768;
__device__ __forceinline__ size_t ds_tile(size_t head, int qi, int kt, int nq) {
  return (head * (size_t)(nq * (nq + 1) / 2) + (size_t)(qi * (qi + 1) / 2 + kt)) * DS_TILE;
}
__device__ __forceinline__ void leave(volatile int* abort_flag, bool owner, uint32_t tmem_base, uint32_t cols = 512) {
  fence_before();
  __syncthreads();
  if (*abort_flag) {                                   // copies and products in flight are given time to land
    const uint64_t t0 = gtimer();
    while (gtimer() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (owner) {
    fence_after();
    tmem_dealloc(tmem_base, cols);
  }
}

// ============================================================================================ forward
// One CTA per (128-query tile or pair of adjacent ones, head, batch); four softmax warps per query tile (thread = query row), a
// TMA and an MMA warp.  Tensor memory: scores of the QT tiles (P of a tile overwrites the first half of its scores), then
// their O accumulators.  P V of the first 64 keys starts while the exponentials of the last 64 are under way.  (Score buffers of
// 64 columns, two per tile, would let S run ahead of P V, but an M 128 x N 64 product takes as long as an N 128 one.)
//
// The products of one query tile have to run while the softmax warps of another work.  Head sizes above 64: two tiles per
// CTA, the tensor core alternates P0 V, S0 = Q0 K', P1 V, S1 = Q1 K'; they share their K and V loads, without which L2
// traffic would bound it.  Up to 64: one tile per CTA, two CTAs per SM, which also overlap each other's start and output:
// 35.6 -> 32.5 us at 8 x 1024 x 12 heads, 162 -> 150 us at 1 x 8192, 22.5 -> 19.7 us at 32 x 256.
template <int ATOMS>
struct FwdCfg {
  static constexpr int QT = ATOMS == 1 ? 1 : 2;
  static constexpr int TILE = ATOMS * 16384;
  static constexpr int STAGES = QT == 1 ? 3 : 2;
  static constexpr int THREADS = QT * 128 + 64;
  static constexpr uint32_t TCOLS = QT == 1 ? 256 : 512;
  // no slack for aligning the base: without static shared memory the window starts 1024-byte aligned (checked)
  static constexpr int SMEM = QT * TILE + 2 * STAGES * TILE + 256;
};

template <int ATOMS>
__global__ void __launch_bounds__(FwdCfg<ATOMS>::THREADS, 3 - FwdCfg<ATOMS>::QT)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tm, const FlashParams p) {
  using C = FwdCfg<ATOMS>;
  constexpr int QT = C::QT;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  if ((smem_u32(smem_raw) & 1023u) != 0u) {                        // uniform over the CTA: nothing has been allocated yet
    if (threadIdx.x == 0) atomicCAS(&g_flash_error, 0, 98);
    return;
  }
  unsigned char* q_s = smem_raw;                                   // [QT]
  unsigned char* k_s = q_s + QT * C::TILE;                         // [STAGES]
  unsigned char* v_s = k_s + C::STAGES * C::TILE;                  // [STAGES]
  uint64_t* bars = reinterpret_cast<uint64_t*>(v_s + C::STAGES * C::TILE);
  uint64_t *q_full = bars, *k_full = bars + 1, *k_empty = bars + 5, *v_full = bars + 9, *v_empty = bars + 13;
  uint64_t *s_full = bars + 17, *p_half = bars + 19, *p_ready = bars + 21, *o_done = bars + 23;    // [query tile]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 25);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = (int)uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  constexpr int W_TMA = QT * 4, W_MMA = QT * 4 + 1;
  const int pair = gridDim.z - 1 - blockIdx.z;                     // heavy (late) query tiles of every head first
  const int h = blockIdx.x, b = blockIdx.y;
  const int g = h / (p.Hq / p.Hkv);
  const int nq = (p.S + 127) >> 7;
  const int n0 = QT * pair + 1, n1 = QT == 2 && 2 * pair + 1 < nq ? 2 * pair + 2 : 0;   // key tiles of the query tiles
  const int n = n1 ? n1 : n0;
  const int ksteps = (p.hd + 15) >> 4;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < C::STAGES; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], 1); mbar_init(&p_half[i], 4); mbar_init(&p_ready[i], 4); mbar_init(&o_done[i], 1); }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == W_MMA) tmem_alloc(tmem_slot, C::TCOLS);
  fence_before();
  __syncthreads();
  fence_after();
  zen_pdl::enter();
  const uint32_t tm0 = *tmem_slot;

  if (warp == W_TMA) {
    if (lane == 0) {
      mbar_expect_tx(q_full, (n1 ? 2 : 1) * C::TILE);
      for (int t = 0; t < (n1 ? 2 : 1); ++t)
#pragma unroll
        for (int a = 0; a < ATOMS; ++a) tma_load_4d(q_s + t * C::TILE + a * 16384, &tm, q_full, a * 64, h, (QT * pair + t) * 128, b);
      for (int j = 0; j < n; ++j) {
        const int st = j % C::STAGES;
        const uint32_t ph = (j / C::STAGES) & 1;
        if (!mbar_wait(&k_empty[st], ph ^ 1, abort_flag, 1, &g_flash_error)) break;
        mbar_expect_tx(&k_full[st], C::TILE);
#pragma unroll
        for (int a = 0; a < ATOMS; ++a) tma_load_4d(k_s + st * C::TILE + a * 16384, &tm, &k_full[st], a * 64, p.Hq + g, j * 128, b);
        if (!mbar_wait(&v_empty[st], ph ^ 1, abort_flag, 2, &g_flash_error)) break;
        mbar_expect_tx(&v_full[st], C::TILE);
#pragma unroll
        for (int a = 0; a < ATOMS; ++a) tma_load_4d(v_s + st * C::TILE + a * 16384, &tm, &v_full[st], a * 64, p.Hq + p.Hkv + g, j * 128, b);
      }
    }
  } else if (warp == W_MMA) {
    const bool leader = elect_one();
    const uint32_t tmu = uniform(tm0);
    const uint32_t idesc_s = make_idesc(128, 128, false, false);
    const uint32_t idesc_o = make_idesc(128, ksteps * 16, false, true);
    auto scores = [&](int t, int j) {
      if (leader) {
        umma_tile_ss(tmu + t * 128, smem_u32(q_s + t * C::TILE), smem_u32(k_s + (j % C::STAGES) * C::TILE), ksteps, idesc_s);
        umma_commit(&s_full[t]);
      }
    };
    bool ok = mbar_wait(q_full, 0, abort_flag, 3, &g_flash_error) && mbar_wait(&k_full[0], 0, abort_flag, 4, &g_flash_error);
    fence_after();
    if (ok) {
      scores(0, 0);
      if (n1) scores(1, 0);
      if (leader && C::STAGES < n) umma_commit(&k_empty[0]);       // only where a later load waits for it
    }
    for (int j = 0; j < n && ok; ++j) {
      const int st = j % C::STAGES, sn = (j + 1) % C::STAGES;
      if (!mbar_wait(&v_full[st], (j / C::STAGES) & 1, abort_flag, 5, &g_flash_error)) break;
      if (j + 1 < n && !mbar_wait(&k_full[sn], ((j + 1) / C::STAGES) & 1, abort_flag, 6, &g_flash_error)) break;
      for (int t = 0; t < QT && ok; ++t) {
        const int nt = t ? n1 : n0;
        if (j >= nt) continue;
        const uint32_t va = smem_u32(v_s + st * C::TILE);
        ok = mbar_wait(&p_half[t], j & 1, abort_flag, 12, &g_flash_error);
        if (!ok) break;
        fence_after();
        if (leader) umma_tile_ts(tmu + QT * 128 + t * 128, tmu + t * 128, va, idesc_o, j == 0);
        ok = mbar_wait(&p_ready[t], j & 1, abort_flag, 7, &g_flash_error);
        if (!ok) break;
        fence_after();
        if (leader) {
          umma_tile_ts(tmu + QT * 128 + t * 128, tmu + t * 128 + 32, va + 8192, idesc_o, false);
          umma_commit(&o_done[t]);
        }
        if (j + 1 < nt) scores(t, j + 1);
      }
      if (!ok) break;
      if (leader) {
        if (j + C::STAGES < n) umma_commit(&v_empty[st]);
        if (j + 1 + C::STAGES < n) umma_commit(&k_empty[sn]);
      }
    }
  } else {
    const int t = QT == 2 ? warp >> 2 : 0;
    const int nt = t ? n1 : n0;
    const int row = threadIdx.x & 127;                              // also the tensor-memory lane
    const int qrow = (QT * pair + t) * 128 + row;
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tS = tm0 + t * 128 + lane_addr, tO = tm0 + QT * 128 + t * 128 + lane_addr;
    const uint64_t cs2 = pk2(p.scale_log2, p.scale_log2);
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < nt; ++j) {
      if (!mbar_wait(&s_full[t], j & 1, abort_flag, 8, &g_flash_error)) { ok = false; break; }
      fence_after();
      uint32_t s[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32_nowait(tS + c * 32, s[c]);
      tmem_wait_ld();
      if (j == nt - 1) {                                            // diagonal tile: keys after the query
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i > row) s[c][i] = 0xff800000u;
      }
      float x[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < 32; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) x[c] = fmaxf(x[c], __uint_as_float(s[c][i]));
      const float mx = fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3])) * p.scale_log2;
      // lazy maximum: the old reference stays unless the row maximum grew by more than 2^8; P stays below 256, the final
      // normalisation is exact either way, and O is rescaled only on such jumps
      const bool need = mx > m + 8.f;
      const float m_new = need ? mx : m;
      if (j > 0 && __any_sync(0xffffffffu, need)) {
        if (!mbar_wait(&o_done[t], (j - 1) & 1, abort_flag, 9, &g_flash_error)) { ok = false; break; }
        fence_after();
        const float alpha = need ? ex2f(m - m_new) : 1.f;
        l *= alpha;
#pragma unroll 1
        for (int c = 0; c < ksteps; ++c) {
          uint32_t r[16];
          tmem_ld16(tO + c * 16, r);
#pragma unroll
          for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
          tmem_st16(tO + c * 16, r);
        }
      }
      m = m_new;
      const uint64_t nm2 = pk2(-m_new, -m_new);
      uint64_t sum0 = 0ull, sum1 = 0ull;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t pk[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const uint32_t* sp = &s[half * 2 + (i >> 4)][(i & 15) * 2];
          float y0, y1;
          exp2_pair(fma2(pk2(__uint_as_float(sp[0]), __uint_as_float(sp[1])), cs2, nm2), y0, y1);
          if (i & 1) sum1 = add2(sum1, pk2(y0, y1)); else sum0 = add2(sum0, pk2(y0, y1));
          pk[i] = pack_bf16(y0, y1);
        }
        tmem_st32_nowait(tS + half * 32, pk);
        tmem_wait_st();
        fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(half ? &p_ready[t] : &p_half[t]);
      }
      float a0, a1, b0, b1;
      unpk2(sum0, a0, a1);
      unpk2(sum1, b0, b1);
      l += (a0 + a1) + (b0 + b1);
    }
    if (nt > 0 && ok && mbar_wait(&o_done[t], (nt - 1) & 1, abort_flag, 10, &g_flash_error)) {
      fence_after();
      const bool live = qrow < p.S;
      store_rows(tO, 0, ksteps * 16, p.hd, 1.f / l, p.out + (size_t)(b * p.S + qrow) * p.ld_o + h * p.hd, live);
      p.lse2[((size_t)b * p.Hq + h) * p.Sp + qrow] = live ? m + log2f(l) : INFINITY;
    }
  }
  leave(abort_flag, warp == W_MMA, tm0, C::TCOLS);
}

// ============================================================================================ backward: dQ
// One CTA per (128-query tile, head, batch).  The two softmax warpgroups (warps 0-3, 4-7; thread = query row) take the
// 128-key tiles in turn, each with its own score buffer, so that the exponentials of one group run beside the products and
// the dS arithmetic of the other.  Tensor memory: scores [0, 256) with dS over them, dP [256, 384), dQ [384, 512).  dP of
// tile j + 1 is issued as soon as dP of tile j is in registers, the scores of tile j + 2 behind dQ += dS K of tile j.  K
// stays in shared memory from its scores to its dQ product: three stages; V only for dP: two.
template <int ATOMS>
struct DqCfg {
  static constexpr int TILE = ATOMS * 16384;
  static constexpr int KST = 3, VST = 2;
  static constexpr int SMEM = 2 * TILE + (KST + VST) * TILE + 1024 + 1024 + 256;
};

template <int ATOMS>
__global__ void __launch_bounds__(320, 1)
flash_bwd_dq_kernel(const __grid_constant__ CUtensorMap tm, const __grid_constant__ CUtensorMap tm_do, const FlashParams p) {
  using C = DqCfg<ATOMS>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char *q_s = smem, *do_s = q_s + C::TILE, *k_s = do_s + C::TILE, *v_s = k_s + C::KST * C::TILE;
  float* red = reinterpret_cast<float*>(v_s + C::VST * C::TILE);   // [2][128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(red + 256);
  uint64_t *q_full = bars, *k_full = bars + 1, *k_empty = bars + 4, *v_full = bars + 7, *v_empty = bars + 9;
  uint64_t *s_full = bars + 11, *ds_ready = bars + 13, *dp_full = bars + 15, *dp_free = bars + 17, *dq_done = bars + 18;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 19);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = (int)uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int qi = gridDim.z - 1 - blockIdx.z;
  const int h = blockIdx.x, b = blockIdx.y;
  const int g = h / (p.Hq / p.Hkv);
  const int n = qi + 1;
  const int ksteps = (p.hd + 15) >> 4;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < C::KST; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); }
    for (int i = 0; i < C::VST; ++i) { mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], 1); mbar_init(&dp_full[i], 1); mbar_init(&ds_ready[i], 4); }
    mbar_init(dp_free, 4); mbar_init(dq_done, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 9) tmem_alloc(tmem_slot, 512);
  fence_before();
  __syncthreads();
  fence_after();
  zen_pdl::enter();
  const uint32_t tm0 = *tmem_slot, tDP = tm0 + 256, tDQ = tm0 + 384;

  if (warp == 8) {
    if (lane == 0) {
      mbar_expect_tx(q_full, 2 * C::TILE);
#pragma unroll
      for (int a = 0; a < ATOMS; ++a) {
        tma_load_4d(q_s + a * 16384, &tm, q_full, a * 64, h, qi * 128, b);
        tma_load_4d(do_s + a * 16384, &tm_do, q_full, a * 64, h, qi * 128, b);
      }
      for (int j = 0; j < n; ++j) {
        const int ks = j % C::KST, vs = j % C::VST;
        if (!mbar_wait(&k_empty[ks], ((j / C::KST) & 1) ^ 1, abort_flag, 21, &g_flash_error)) break;
        mbar_expect_tx(&k_full[ks], C::TILE);
#pragma unroll
        for (int a = 0; a < ATOMS; ++a) tma_load_4d(k_s + ks * C::TILE + a * 16384, &tm, &k_full[ks], a * 64, p.Hq + g, j * 128, b);
        if (!mbar_wait(&v_empty[vs], ((j / C::VST) & 1) ^ 1, abort_flag, 22, &g_flash_error)) break;
        mbar_expect_tx(&v_full[vs], C::TILE);
#pragma unroll
        for (int a = 0; a < ATOMS; ++a) tma_load_4d(v_s + vs * C::TILE + a * 16384, &tm, &v_full[vs], a * 64, p.Hq + p.Hkv + g, j * 128, b);
      }
    }
  } else if (warp == 9) {
    const bool leader = elect_one();
    const uint32_t tmu = uniform(tm0);
    const uint32_t idesc_s = make_idesc(128, 128, false, false);
    const uint32_t idesc_q = make_idesc(128, ksteps * 16, false, true);
    const uint32_t qa = smem_u32(q_s), da = smem_u32(do_s);
    auto scores = [&](int j) -> bool {
      const int ks = j % C::KST;
      if (!mbar_wait(&k_full[ks], (j / C::KST) & 1, abort_flag, 23, &g_flash_error)) return false;
      fence_after();
      if (leader) {
        umma_tile_ss(tmu + (j & 1) * 128, qa, smem_u32(k_s + ks * C::TILE), ksteps, idesc_s);
        umma_commit(&s_full[j & 1]);
      }
      return true;
    };
    auto dprobs = [&](int j) -> bool {
      const int vs = j % C::VST;
      if (!mbar_wait(&v_full[vs], (j / C::VST) & 1, abort_flag, 24, &g_flash_error)) return false;
      fence_after();
      if (leader) {
        umma_tile_ss(tmu + 256, da, smem_u32(v_s + vs * C::TILE), ksteps, idesc_s);
        umma_commit(&dp_full[j & 1]);
        if (j + C::VST < n) umma_commit(&v_empty[vs]);
      }
      return true;
    };
    bool ok = mbar_wait(q_full, 0, abort_flag, 25, &g_flash_error) && scores(0) && dprobs(0) && (n < 2 || scores(1));
    for (int j = 0; j < n && ok; ++j) {
      const int e = j & 1;
      if (j + 1 < n) {
        ok = mbar_wait(dp_free, j & 1, abort_flag, 26, &g_flash_error);
        if (!ok) break;
        fence_after();
        if (!dprobs(j + 1)) break;
      }
      ok = mbar_wait(&ds_ready[e], (j >> 1) & 1, abort_flag, 27, &g_flash_error);
      if (!ok) break;
      fence_after();
      if (leader) {
        const uint32_t ka = smem_u32(k_s + (j % C::KST) * C::TILE);
        umma_tile_ts(tmu + 384, tmu + e * 128, ka, idesc_q, j == 0);
        umma_tile_ts(tmu + 384, tmu + e * 128 + 64, ka + 8192, idesc_q, false);
        if (j + C::KST < n) umma_commit(&k_empty[j % C::KST]);
      }
      if (j + 2 < n && !scores(j + 2)) break;
    }
    if (ok && leader) umma_commit(dq_done);
  } else {
    const int w = warp >> 2, row = threadIdx.x & 127;
    const int qrow = qi * 128 + row;
    const bool live = qrow < p.S;
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    // D of this row: the two threads of a row take every other 8-column piece of dO * O
    float d = 0.f;
    if (live) {
      const size_t off = (size_t)(b * p.S + qrow) * p.ld_o + h * p.hd + w * 8;
      d = row_dot<ATOMS * 4>(p.dout + off, p.o_in + off, p.hd - w * 8);
    }
    red[w * 128 + row] = d;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    const float nd = -(red[row] + red[128 + row]);
    const size_t stat = ((size_t)b * p.Hq + h) * p.Sp + qrow;
    const float nl = -p.lse2[stat];
    if (w == 0) {
      p.stat[stat] = nl;
      p.stat[(size_t)p.B * p.Hq * p.Sp + stat] = nd;
    }
    const uint64_t cs2 = pk2(p.scale_log2, p.scale_log2), nl2 = pk2(nl, nl), nd2 = pk2(nd, nd);
    const uint32_t tS = tm0 + w * 128 + lane_addr;
    bool ok = true;
    for (int j = w; j < n && ok; j += 2) {
      if (!mbar_wait(&s_full[w], (j >> 1) & 1, abort_flag, 28, &g_flash_error)) { ok = false; break; }
      fence_after();
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t s[2][32];
        tmem_ld32_nowait(tS + half * 64, s[0]);
        tmem_ld32_nowait(tS + half * 64 + 32, s[1]);
        tmem_wait_ld();
        if (j == n - 1) {                                           // diagonal tile: keys after the query
          const int lim = row - half * 64;
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (c * 32 + i > lim) s[c][i] = 0xff800000u;
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          uint32_t* sp = &s[i >> 4][(i & 15) * 2];
          float y0, y1;
          exp2_pair(fma2(pk2(__uint_as_float(sp[0]), __uint_as_float(sp[1])), cs2, nl2), y0, y1);
          sp[0] = __float_as_uint(y0);
          sp[1] = __float_as_uint(y1);
        }
        if (half == 0) {
          if (!mbar_wait(&dp_full[w], (j >> 1) & 1, abort_flag, 29, &g_flash_error)) { ok = false; break; }
          fence_after();
        }
        uint32_t dp[2][32];
        tmem_ld32_nowait(tDP + half * 64 + lane_addr, dp[0]);
        tmem_ld32_nowait(tDP + half * 64 + 32 + lane_addr, dp[1]);
        tmem_wait_ld();
        if (half == 1) {
          fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(dp_free);
        }
        uint32_t pk[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const uint32_t *sp = &s[i >> 4][(i & 15) * 2], *dq = &dp[i >> 4][(i & 15) * 2];
          float y0, y1;
          unpk2(mul2(add2(pk2(__uint_as_float(dq[0]), __uint_as_float(dq[1])), nd2), pk2(__uint_as_float(sp[0]), __uint_as_float(sp[1]))), y0, y1);
          pk[i] = pack_bf16(y0, y1);
        }
        tmem_st32_nowait(tS + half * 64, pk);
      }
      if (!ok) break;
      tmem_wait_st();
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ds_ready[w]);
    }
    if (ok && mbar_wait(dq_done, 0, abort_flag, 30, &g_flash_error)) {
      fence_after();
      const int mid = ((ksteps + 1) >> 1) * 16;                     // the two warps of a lane quarter share the columns
      store_rows(tDQ + lane_addr, w ? mid : 0, w ? ksteps * 16 : mid, p.hd, p.scale,
                 p.dqkv + (size_t)(b * p.S + qrow) * p.ld_dqkv + h * p.hd, live);
    }
  }
  leave(abort_flag, warp == 9, tm0);
}

// ============================================================================================ backward: dK and dV
// One CTA per (128-key tile, KV head, batch); walks the query tiles at or after the diagonal of every query head of the
// group.  Transposed scores S' = K Q' and dP' = V dO', so that P' and dS' have the keys in the lanes and are the A operands
// of dV += P' dO and dK += dS' Q out of tensor memory.  Warp w of the eight softmax warps: keys of lane quarter w % 4,
// queries of half w / 4.  With two accumulators of 128 columns (ATOMS 2) tensor memory is full: S' [0, 128) with P' over
// it, dP' [128, 256) with dS' over it, dV [256, 384), dK [384, 512); the order dV(i), S'(i + 1), dK(i), dP'(i + 1) lets the
// exponentials of tile i + 1 run beside dK(i) and dP'(i + 1), and dS'(i) beside dV(i) and S'(i + 1).  With accumulators of
// 64 columns there is room for a second score buffer (at 384, dK at 320): S'(i + 1) is issued ahead of everything else of
// tile i.  -lse and -D of the query tile ride in with dO and Q.
template <int ATOMS>
struct DkvCfg {
  static constexpr int TILE = ATOMS * 16384;
  static constexpr int QST = 3, DST = 2, SB = ATOMS == 1 ? 2 : 1;
  static constexpr uint32_t S1 = SB == 2 ? 384 : 0, DV = 256, DK = SB == 2 ? 320 : 384;
  // no slack for aligning the base: without static shared memory the window starts 1024-byte aligned (checked)
  static constexpr int SMEM = 2 * TILE + (QST + DST) * TILE + (QST + DST) * 512 + 256;
};

template <int ATOMS>
__global__ void __launch_bounds__(320, 1)
flash_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tm, const __grid_constant__ CUtensorMap tm_do, const FlashParams p) {
  using C = DkvCfg<ATOMS>;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  if ((smem_u32(smem_raw) & 1023u) != 0u) {                        // uniform over the CTA: nothing has been allocated yet
    if (threadIdx.x == 0) atomicCAS(&g_flash_error, 0, 99);
    return;
  }
  unsigned char *k_s = smem_raw, *v_s = k_s + C::TILE, *q_s = v_s + C::TILE, *do_s = q_s + C::QST * C::TILE;
  float* nl_s = reinterpret_cast<float*>(do_s + C::DST * C::TILE);  // [DST][128] -lse, released with dO (after P' is there)
  float* nd_s = nl_s + C::DST * 128;                                // [QST][128] -D, released with Q (after dS' is there)
  uint64_t* bars = reinterpret_cast<uint64_t*>(nd_s + C::QST * 128);
  uint64_t *kv_full = bars, *q_full = bars + 1, *q_empty = bars + 4, *d_full = bars + 7, *d_empty = bars + 9;
  uint64_t *s_full = bars + 11, *dp_full = bars + 13, *p_ready = bars + 14, *ds_ready = bars + 15, *done = bars + 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 17);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = (int)uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int kt = blockIdx.z;                                       // early key tiles see the most queries
  const int g = blockIdx.x, b = blockIdx.y;
  const int rep = p.Hq / p.Hkv;
  const int nq = (p.S + 127) >> 7;
  const int per = nq - kt, n = rep * per;
  const int ksteps = (p.hd + 15) >> 4;
  const size_t stat_d = (size_t)p.B * p.Hq * p.Sp;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int i = 0; i < C::QST; ++i) { mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1); }
    for (int i = 0; i < C::DST; ++i) { mbar_init(&d_full[i], 1); mbar_init(&d_empty[i], 1); }
    mbar_init(&s_full[0], 1); mbar_init(&s_full[1], 1); mbar_init(dp_full, 1); mbar_init(p_ready, 8); mbar_init(ds_ready, 8);
    mbar_init(done, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 9) tmem_alloc(tmem_slot, 512);
  fence_before();
  __syncthreads();
  fence_after();
  zen_pdl::enter();
  const uint32_t tm0 = *tmem_slot, tDP = tm0 + 128;

  if (warp == 8) {
    if (lane == 0) {
      mbar_expect_tx(kv_full, 2 * C::TILE);
#pragma unroll
      for (int a = 0; a < ATOMS; ++a) {
        tma_load_4d(k_s + a * 16384, &tm, kv_full, a * 64, p.Hq + g, kt * 128, b);
        tma_load_4d(v_s + a * 16384, &tm, kv_full, a * 64, p.Hq + p.Hkv + g, kt * 128, b);
      }
      int h = g * rep, qi = kt;
      for (int i = 0; i < n; ++i) {
        const int qs = i % C::QST, ds = i % C::DST;
        const float* src = p.stat + ((size_t)b * p.Hq + h) * p.Sp + qi * 128;
        if (!mbar_wait(&q_empty[qs], ((i / C::QST) & 1) ^ 1, abort_flag, 41, &g_flash_error)) break;
        mbar_expect_tx(&q_full[qs], C::TILE + 512);
#pragma unroll
        for (int a = 0; a < ATOMS; ++a) tma_load_4d(q_s + qs * C::TILE + a * 16384, &tm, &q_full[qs], a * 64, h, qi * 128, b);
        bulk_load_1d(nd_s + qs * 128, src + stat_d, 512, &q_full[qs]);
        if (!mbar_wait(&d_empty[ds], ((i / C::DST) & 1) ^ 1, abort_flag, 42, &g_flash_error)) break;
        mbar_expect_tx(&d_full[ds], C::TILE + 512);
        bulk_load_1d(nl_s + ds * 128, src, 512, &d_full[ds]);
#pragma unroll
        for (int a = 0; a < ATOMS; ++a) tma_load_4d(do_s + ds * C::TILE + a * 16384, &tm_do, &d_full[ds], a * 64, h, qi * 128, b);
        if (++qi == nq) { qi = kt; ++h; }
      }
    }
  } else if (warp == 9) {
    const bool leader = elect_one();
    const uint32_t tmu = uniform(tm0);
    const uint32_t idesc_s = make_idesc(128, 128, false, false);
    const uint32_t idesc_g = make_idesc(128, ksteps * 16, false, true);
    const uint32_t ka = smem_u32(k_s), va = smem_u32(v_s);
    auto scores = [&](int i) -> bool {
      const int qs = i % C::QST, e = i % C::SB;
      if (!mbar_wait(&q_full[qs], (i / C::QST) & 1, abort_flag, 43, &g_flash_error)) return false;
      fence_after();
      if (leader) {
        umma_tile_ss(tmu + (e ? C::S1 : 0), ka, smem_u32(q_s + qs * C::TILE), ksteps, idesc_s);
        umma_commit(&s_full[e]);
      }
      return true;
    };
    auto dprobs = [&](int i) -> bool {
      const int ds = i % C::DST;
      if (!mbar_wait(&d_full[ds], (i / C::DST) & 1, abort_flag, 44, &g_flash_error)) return false;
      fence_after();
      if (leader) {
        umma_tile_ss(tmu + 128, va, smem_u32(do_s + ds * C::TILE), ksteps, idesc_s);
        umma_commit(dp_full);
      }
      return true;
    };
    bool ok = mbar_wait(kv_full, 0, abort_flag, 45, &g_flash_error) && scores(0) && dprobs(0);
    for (int i = 0; i < n && ok; ++i) {
      if (C::SB == 2 && i + 1 < n && !scores(i + 1)) break;        // its buffer was last read by dV(i - 1)
      ok = mbar_wait(p_ready, i & 1, abort_flag, 46, &g_flash_error);
      if (!ok) break;
      fence_after();
      if (leader) {
        const uint32_t da = smem_u32(do_s + (i % C::DST) * C::TILE), ta = tmu + (i % C::SB ? C::S1 : 0);
        umma_tile_ts(tmu + C::DV, ta, da, idesc_g, i == 0);
        umma_tile_ts(tmu + C::DV, ta + 64, da + 8192, idesc_g, false);
        if (i + C::DST < n) umma_commit(&d_empty[i % C::DST]);
      }
      if (C::SB == 1 && i + 1 < n && !scores(i + 1)) break;
      ok = mbar_wait(ds_ready, i & 1, abort_flag, 47, &g_flash_error);
      if (!ok) break;
      fence_after();
      if (leader) {
        const uint32_t qa = smem_u32(q_s + (i % C::QST) * C::TILE);
        umma_tile_ts(tmu + C::DK, tmu + 128, qa, idesc_g, i == 0);
        umma_tile_ts(tmu + C::DK, tmu + 192, qa + 8192, idesc_g, false);
        if (i + C::QST < n) umma_commit(&q_empty[i % C::QST]);
      }
      if (i + 1 < n) ok = dprobs(i + 1);
      else if (leader) umma_commit(done);
    }
  } else {
    const int w = warp >> 2, row = threadIdx.x & 127;                // key row, also the tensor-memory lane
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tP = tDP + w * 64 + lane_addr;
    const uint64_t cs2 = pk2(p.scale_log2, p.scale_log2);
    bool ok = true;
    int qi = kt, h = g * rep;
    for (int i = 0; i < n; ++i) {
      const int e = i % C::SB;
      const uint32_t tS = tm0 + (e ? C::S1 : 0) + w * 64 + lane_addr;
      const float *lp = nl_s + (i % C::DST) * 128 + w * 64, *ndp = nd_s + (i % C::QST) * 128 + w * 64;
      if (!mbar_wait(&s_full[e], (i / C::SB) & 1, abort_flag, 48, &g_flash_error)) { ok = false; break; }
      // the statistics (copied with Q and dO)
      if (!mbar_wait(&q_full[i % C::QST], (i / C::QST) & 1, abort_flag, 49, &g_flash_error)) { ok = false; break; }
      if (!mbar_wait(&d_full[i % C::DST], (i / C::DST) & 1, abort_flag, 52, &g_flash_error)) { ok = false; break; }
      fence_after();
      uint32_t s[2][32];
      tmem_ld32_nowait(tS, s[0]);
      tmem_ld32_nowait(tS + 32, s[1]);
      tmem_wait_ld();
      if (qi == kt) {                                                // diagonal tile: queries before the key
#pragma unroll
        for (int c = 0; c < 64; ++c)
          if (w * 64 + c < row) s[c >> 5][c & 31] = 0xff800000u;
      }
      {
        uint32_t pk[32];
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          const float4 nl = *reinterpret_cast<const float4*>(lp + q * 4);
#pragma unroll
          for (int e2 = 0; e2 < 2; ++e2) {
            const int c = q * 4 + e2 * 2;
            uint32_t* sp = &s[c >> 5][c & 31];
            float y0, y1;
            exp2_pair(fma2(pk2(__uint_as_float(sp[0]), __uint_as_float(sp[1])), cs2, e2 ? pk2(nl.z, nl.w) : pk2(nl.x, nl.y)), y0, y1);
            sp[0] = __float_as_uint(y0);
            sp[1] = __float_as_uint(y1);
            pk[q * 2 + e2] = pack_bf16(y0, y1);
          }
        }
        tmem_st32_nowait(tS, pk);
        tmem_wait_st();
      }
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready);
      if (!mbar_wait(dp_full, i & 1, abort_flag, 50, &g_flash_error)) { ok = false; break; }
      fence_after();
      uint32_t dp[2][32];
      tmem_ld32_nowait(tP, dp[0]);
      tmem_ld32_nowait(tP + 32, dp[1]);
      tmem_wait_ld();
      {
        uint32_t pk[32];
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          const float4 nd = *reinterpret_cast<const float4*>(ndp + q * 4);
#pragma unroll
          for (int e2 = 0; e2 < 2; ++e2) {
            const int c = q * 4 + e2 * 2;
            const uint32_t *sp = &s[c >> 5][c & 31], *dq = &dp[c >> 5][c & 31];
            float y0, y1;
            unpk2(mul2(add2(pk2(__uint_as_float(dq[0]), __uint_as_float(dq[1])), e2 ? pk2(nd.z, nd.w) : pk2(nd.x, nd.y)),
                       pk2(__uint_as_float(sp[0]), __uint_as_float(sp[1]))), y0, y1);
            pk[q * 2 + e2] = pack_bf16(y0, y1);
          }
        }
        tmem_st32_nowait(tP, pk);
        if (p.ds) {                                                  // 16 bytes = 8 queries of the key; a warp's stores are 512 in a row
          uint4* dst = reinterpret_cast<uint4*>(p.ds + ds_tile((size_t)b * p.Hq + h, qi, kt, nq)) + w * 1024 + row;
#pragma unroll
          for (int c = 0; c < 8; ++c) dst[c * 128] = make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
        }
        tmem_wait_st();
      }
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_ready);
      if (++qi == nq) { qi = kt; ++h; }
    }
    if (ok && mbar_wait(done, 0, abort_flag, 51, &g_flash_error)) {
      fence_after();
      const int krow = kt * 128 + row;
      const bool live = krow < p.S;
      __nv_bfloat16* dst = p.dqkv + (size_t)(b * p.S + krow) * p.ld_dqkv;
      // one of the two warps of a lane quarter writes dK, the other dV
      if (w == 0) store_rows(tm0 + C::DK + lane_addr, 0, ksteps * 16, p.hd, p.scale, dst + (p.Hq + g) * p.hd, live);
      else store_rows(tm0 + C::DV + lane_addr, 0, ksteps * 16, p.hd, 1.f, dst + (p.Hq + p.Hkv + g) * p.hd, live);
    }
  }
  leave(abort_flag, warp == 9, tm0);
}

// ============================================================================================ backward with dS kept: D, then dQ
// stat = -lse2 and -D of every row (rows beyond S: -inf, 0).  CTA = 128 rows of a head; L lanes to a row (8 up to 64 columns, else 16),
// L / 2 rows of a group under way.  It streams O and dO, so it starts early only as a small grid (launch.cuh): the whole op at 1 x 8192, 32
// heads of 128, 2 118 us, with this kernel early 2 129.
template <int L>
__global__ void __launch_bounds__(256)
flash_stat_kernel(const FlashParams p) {
  zen_pdl::enter();
  constexpr int R = L / 2;
  const int l = threadIdx.x % L, h = blockIdx.y, b = blockIdx.z, s0 = blockIdx.x * 128 + threadIdx.x / L * R;
  uint4 x[R], y[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const bool in = s0 + i < p.S && l * 8 < p.hd;
    const size_t at = (size_t)(b * p.S + s0 + i) * p.ld_o + h * p.hd + l * 8;
    x[i] = in ? *reinterpret_cast<const uint4*>(p.dout + at) : make_uint4(0u, 0u, 0u, 0u);
    y[i] = in ? *reinterpret_cast<const uint4*>(p.o_in + at) : make_uint4(0u, 0u, 0u, 0u);
  }
  const size_t at = ((size_t)b * p.Hq + h) * p.Sp + s0 + l;          // Sp is a multiple of 128
  const float lse = l < R ? p.lse2[at] : 0.f;
  float mine = 0.f;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const uint32_t xw[4] = {x[i].x, x[i].y, x[i].z, x[i].w}, yw[4] = {y[i].x, y[i].y, y[i].z, y[i].w};
    float d = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      d += __uint_as_float(xw[k] << 16) * __uint_as_float(yw[k] << 16);
      d += __uint_as_float(xw[k] & 0xffff0000u) * __uint_as_float(yw[k] & 0xffff0000u);
    }
#pragma unroll
    for (int o = L / 2; o; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o, L);
    if (l == i) mine = d;
  }
  if (l < R) {
    p.stat[at] = -lse;
    p.stat[(size_t)p.B * p.Hq * p.Sp + at] = -mine;
  }
}

// dQ = dS K over the tiles that the dK / dV kernel left: a plain product, one CTA per (128-query tile, head, batch).  The tiles are the
// A operand as they lie in memory (queries contiguous, 8 x 8 core matrices, no swizzle), one 32 KB bulk copy each.
// What bounds it: reading dS (1 x 8192, 32 heads: 2.2 GB in 403 us, 5.4 TB/s; working the scores out again took 669 us).
template <int ATOMS>
struct DqtCfg {
  static constexpr int KT = ATOMS * 16384, STAGE = DS_TILE + KT;
  static constexpr int STAGES = ATOMS == 1 ? 2 : 3;               // up to 64 columns two CTAs fit an SM
  static constexpr int SMEM = STAGES * STAGE + 128;
};
template <int ATOMS>
__global__ void __launch_bounds__(192, ATOMS == 1 ? 2 : 1)
flash_bwd_dq_tiles_kernel(const __grid_constant__ CUtensorMap tm, const FlashParams p) {
  using C = DqtCfg<ATOMS>;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  if ((smem_u32(smem_raw) & 1023u) != 0u) {                        // uniform over the CTA: nothing has been allocated yet
    if (threadIdx.x == 0) atomicCAS(&g_flash_error, 0, 97);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + C::STAGES * C::STAGE);
  uint64_t *full = bars, *empty = bars + 3, *done = bars + 6;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 7);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = (int)uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int qi = gridDim.z - 1 - blockIdx.z;                       // heavy query tiles first
  const int h = blockIdx.x, b = blockIdx.y, g = h / (p.Hq / p.Hkv), n = qi + 1, nq = (p.S + 127) >> 7;
  const int ksteps = (p.hd + 15) >> 4;
  if (threadIdx.x == 0) {
    for (int i = 0; i < C::STAGES; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    mbar_init(done, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, 128);
  fence_before();
  __syncthreads();
  fence_after();
  zen_pdl::enter();
  const uint32_t tm0 = *tmem_slot;
  if (warp == 0) {
    if (lane == 0) {
      const unsigned char* src = p.ds + ds_tile((size_t)b * p.Hq + h, qi, 0, nq);
      for (int j = 0; j < n; ++j) {
        const int st = j % C::STAGES;
        if (!mbar_wait(&empty[st], ((j / C::STAGES) & 1) ^ 1, abort_flag, 61, &g_flash_error)) break;
        unsigned char* dst = smem_raw + st * C::STAGE;
        mbar_expect_tx(&full[st], C::STAGE);
        bulk_load_1d(dst, src + (size_t)j * DS_TILE, DS_TILE, &full[st]);
#pragma unroll
        for (int a = 0; a < ATOMS; ++a) tma_load_4d(dst + DS_TILE + a * 16384, &tm, &full[st], a * 64, p.Hq + g, j * 128, b);
      }
    }
  } else if (warp == 1) {
    const bool leader = elect_one();
    const uint32_t tmu = uniform(tm0), idesc = make_idesc(128, ksteps * 16, true, true);
    bool ok = true;
    for (int j = 0; j < n; ++j) {
      const int st = j % C::STAGES;
      ok = mbar_wait(&full[st], (j / C::STAGES) & 1, abort_flag, 62, &g_flash_error);
      if (!ok) break;
      fence_after();
      if (leader) {
        const uint32_t sa = smem_u32(smem_raw + st * C::STAGE);
        // no swizzle, queries contiguous: core matrices 2048 bytes apart along the queries, 128 along the keys
        const uint64_t ad = make_desc_plain(sa, 128, 2048), bd = make_desc(sa + DS_TILE, 16384, 1024);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) umma_bf16(tmu, ad + (uint64_t)(kk * 16), bd + (uint64_t)(kk * 128), idesc, (j > 0 || kk > 0) ? 1u : 0u);
        if (j + C::STAGES < n) umma_commit(&empty[st]);            // only where a later load waits for it
      }
    }
    if (ok && leader) umma_commit(done);
  } else if (mbar_wait(done, 0, abort_flag, 63, &g_flash_error)) {
    fence_after();
    const int row = (warp & 3) * 32 + lane, qrow = qi * 128 + row;
    store_rows(tm0 + ((uint32_t)((warp & 3) * 32) << 16), 0, ksteps * 16, p.hd, p.scale,
               p.dqkv + (size_t)(b * p.S + qrow) * p.ld_dqkv + h * p.hd, qrow < p.S);
  }
  leave(abort_flag, warp == 1, tm0, 128);
}

template <typename F>
int opt_in(F* f, int bytes) {
  return (int)cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

template <int ATOMS>
int flash_attrs() {
  static const int rc = [] {
    int r = opt_in(flash_fwd_kernel<ATOMS>, FwdCfg<ATOMS>::SMEM);
    if (!r) r = opt_in(flash_bwd_dq_kernel<ATOMS>, DqCfg<ATOMS>::SMEM);
    if (!r) r = opt_in(flash_bwd_dkv_kernel<ATOMS>, DkvCfg<ATOMS>::SMEM);
    if (!r) r = opt_in(flash_bwd_dq_tiles_kernel<ATOMS>, DqtCfg<ATOMS>::SMEM);
    return r;
  }();
  return rc;
}

bool flash_shape_ok(const void* a, const void* b, int S, int Hq, int Hkv, int hd, int ld_a, int ld_b) {
  return S > 0 && Hkv > 0 && Hq % Hkv == 0 && hd >= 8 && hd <= 128 && hd % 8 == 0 && ld_a % 8 == 0 && ld_b % 8 == 0 &&
         reinterpret_cast<uintptr_t>(a) % 16 == 0 && reinterpret_cast<uintptr_t>(b) % 16 == 0;
}

}  // namespace

extern "C" {

// Causal attention forward, hd <= 128 (multiple of 8), any S.  qkv: bf16 [B*S, (Hq + 2*Hkv)*hd], row stride ld_qkv; out: bf16
// [B*S, Hq*hd], row stride ld_out; lse2: fp32 [B, Hq, Sp] with Sp = S rounded up to a multiple of 128 (+inf beyond S).
int zen_flash_fwd(const void* qkv, void* out, float* lse2, int B, int S, int Hq, int Hkv, int hd, int ld_qkv, int ld_out, float scale,
                  void* stream) {
  if (!flash_shape_ok(qkv, out, S, Hq, Hkv, hd, ld_qkv, ld_out)) return -2;
  CUtensorMap tm;
  int rc = zen_tmap::get_heads(qkv, hd, Hq + 2 * Hkv, S, B, ld_qkv, &tm);
  if (rc) return rc;
  const int nq = (S + 127) / 128;
  FlashParams p{};
  p.out = (__nv_bfloat16*)out; p.lse2 = lse2;
  p.B = B; p.S = S; p.Sp = nq * 128; p.Hq = Hq; p.Hkv = Hkv; p.hd = hd; p.ld_o = ld_out;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  cudaStream_t st = (cudaStream_t)stream;
  if (hd <= 64) {
    if ((rc = flash_attrs<1>())) return rc;
    zen_pdl::launch(flash_fwd_kernel<1>, dim3(Hq, B, nq), FwdCfg<1>::THREADS, FwdCfg<1>::SMEM, st, tm, p);
  } else {
    if ((rc = flash_attrs<2>())) return rc;
    zen_pdl::launch(flash_fwd_kernel<2>, dim3(Hq, B, (nq + 1) / 2), FwdCfg<2>::THREADS, FwdCfg<2>::SMEM, st, tm, p);
  }
  return (int)cudaGetLastError();
}

// Scratch for which the backward keeps dS between its kernels: 32 KB per pair of a query and a key tile at or below the diagonal.  0: not
// kept, the scores are worked out twice.
//  * Fewer than DS_MIN_TILES tiles: the third launch costs more than the scores (1 x 512, 12 heads of 64, 120 tiles: 20 us worked out
//    twice, 23 kept; 8 x 256, 288 tiles: 25.3 / 24.0; 2 x 512, 24 heads of 128, 480 tiles: 51 / 45).
//  * Head sizes up to 96 leave a tile in half the time that one of 128 takes, so that dS has to stay in L2 to pay: 8 x 1024, 12 heads of
//    64 (113 MB) 116 / 110, 1 x 4096 (208 MB) 132 / 138; 3 x 1000, 32 heads of 80 (113 MB) 140 / 127, 1 x 8192 1444 / 1478.
//  * Above that up to DS_MOST (1 x 4096, 24 heads of 128, 415 MB: 324 / 294; 1 x 8192, 32 heads, 2.2 GB: 1680 / 1575).
int zen_flash_ds_bytes(int B, int S, int Hq, int hd, int64_t* bytes) {
  constexpr int64_t DS_MIN_TILES = 256, DS_IN_L2 = (int64_t)128 << 20, DS_MOST = (int64_t)3 << 30;
  const int64_t nq = (S + 127) / 128, tiles = (int64_t)B * Hq * nq * (nq + 1) / 2;
  *bytes = nq < 2 || tiles < DS_MIN_TILES || tiles * DS_TILE > (hd > 96 ? DS_MOST : DS_IN_L2) ? 0 : tiles * DS_TILE;
  return 0;
}

// Backward of the above.  dout / out: bf16 [B*S, Hq*hd] (row stride ld_o); lse2 from the forward; stat: fp32 scratch
// [2][B, Hq, Sp]; dqkv: bf16 [B*S, (Hq + 2*Hkv)*hd] (row stride ld_dqkv), fully overwritten.  ds: null, or scratch of
// zen_flash_ds_bytes (16-byte aligned) where that is not 0.
int zen_flash_bwd(const void* qkv, const void* out, const void* dout, const float* lse2, float* stat, void* dqkv, int B, int S, int Hq,
                  int Hkv, int hd, int ld_qkv, int ld_o, int ld_dqkv, float scale, void* ds, void* stream) {
  if (!flash_shape_ok(qkv, out, S, Hq, Hkv, hd, ld_qkv, ld_o) || !flash_shape_ok(dout, dqkv, S, Hq, Hkv, hd, ld_o, ld_dqkv)) return -2;
  if (reinterpret_cast<uintptr_t>(stat) % 16 || reinterpret_cast<uintptr_t>(ds) % 16) return -3;
  CUtensorMap tm, tm_do;
  int rc = zen_tmap::get_heads(qkv, hd, Hq + 2 * Hkv, S, B, ld_qkv, &tm);
  if (!rc) rc = zen_tmap::get_heads(dout, hd, Hq, S, B, ld_o, &tm_do);
  if (rc) return rc;
  const int nq = (S + 127) / 128;
  FlashParams p{};
  p.lse2 = const_cast<float*>(lse2); p.o_in = (const __nv_bfloat16*)out; p.dout = (const __nv_bfloat16*)dout;
  p.dqkv = (__nv_bfloat16*)dqkv; p.stat = stat; p.ds = (unsigned char*)ds;
  p.B = B; p.S = S; p.Sp = nq * 128; p.Hq = Hq; p.Hkv = Hkv; p.hd = hd; p.ld_o = ld_o; p.ld_dqkv = ld_dqkv;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  const dim3 gq(Hq, B, nq), gk(Hkv, B, nq);
  cudaStream_t st = (cudaStream_t)stream;
  if (hd <= 64) {
    if ((rc = flash_attrs<1>())) return rc;
    if (ds) zen_pdl::launch_small(flash_stat_kernel<8>, dim3(nq, Hq, B), 256, 0, st, p);
    else zen_pdl::launch(flash_bwd_dq_kernel<1>, gq, 320, DqCfg<1>::SMEM, st, tm, tm_do, p);
    zen_pdl::launch(flash_bwd_dkv_kernel<1>, gk, 320, DkvCfg<1>::SMEM, st, tm, tm_do, p);
    if (ds) zen_pdl::launch(flash_bwd_dq_tiles_kernel<1>, gq, 192, DqtCfg<1>::SMEM, st, tm, p);
  } else {
    if ((rc = flash_attrs<2>())) return rc;
    if (ds) zen_pdl::launch_small(flash_stat_kernel<16>, dim3(nq, Hq, B), 256, 0, st, p);
    else zen_pdl::launch(flash_bwd_dq_kernel<2>, gq, 320, DqCfg<2>::SMEM, st, tm, tm_do, p);
    zen_pdl::launch(flash_bwd_dkv_kernel<2>, gk, 320, DkvCfg<2>::SMEM, st, tm, tm_do, p);
    if (ds) zen_pdl::launch(flash_bwd_dq_tiles_kernel<2>, gq, 192, DqtCfg<2>::SMEM, st, tm, p);
  }
  return (int)cudaGetLastError();
}

int zen_flash_error() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_flash_error, sizeof(int)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(g_flash_error, &zero, sizeof(int));
  return v;
}

}  // extern "C"
