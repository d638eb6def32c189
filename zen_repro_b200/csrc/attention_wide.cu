// Causal self-attention for head sizes above 128 (up to 256, any multiple of 8) and for soft-capped scores of any head size,
// any sequence length, forward and backward, on tcgen05 tensor cores with CTA pairs (cta_group::2, sm_100a).
//
// A pair of CTAs owns 256 adjacent rows (queries, or keys in the dK / dV kernels), 128 each, and walks the other side in
// tiles of 128.  What bounds it: at head size 256 one 128-row tile of an operand is 64 KB and an accumulator takes half of
// tensor memory.  A CTA of its own would fetch 128 KB per 2048 tensor-core cycles, all that an SM can draw from L2, with
// room for one stage; of a pair each CTA holds half of every streamed tile (64 of its rows for the score products, 128 of
// its 256 columns for the accumulating one), so the traffic halves and the stages fit.  P and dS go from the softmax warps
// into tensor memory as A operands of the accumulating products (csrc/attention_flash.cu has the reasons).
//
//   kernel  resident    streamed, score products     A operand   accumulator
//   fwd     Q           K                 S = Q K'    P           O  += P V      (online softmax)
//   dV      K           Q                 S' = K Q'   P'          dV += P' dO
//   dQ      Q, dO       K, V   S = Q K', dP = dO V'   dS          dQ += dS K
//   dK      K, V        Q, dO  S' = K Q', dP' = V dO' dS'         dK += dS' Q
//
// dK and dV together would need all of tensor memory for their accumulators, hence two kernels and the scores twice: eight
// products of 1024 cycles per tile pair in the backward instead of seven.  The kernels with two products per tile keep
// two score buffers, so S of the next tile runs while the softmax warps work; those with three have one buffer each for S and dP,
// and the order S(i + 1), accumulate(i), dP(i + 1) hides the exponentials behind two products and dS behind one.
//
// The reference runs eager attention (matmul + softmax + matmul, train.py:155), which materialises the scores.
//
// Measured against one-CTA kernels with P and dS in shared memory and 64-row streamed tiles: 4 x 2048, 8 heads, 1 KV head of 256:
// forward 152 -> 87 us, backward 763 -> 356 us; 1 x 8192, 8 heads: forward 238 us (1160 TFLOP/s), backward 935 us.
#include "attention_common.cuh"
#include "launch.cuh"
#include "pair_common.cuh"
#include "tmap_util.cuh"

namespace {

using namespace tc;

__device__ int g_attn_error = 0;

struct WideParams {
  __nv_bfloat16* out;            // forward: O [B*S, Hq*hd], row stride ld_o
  float* lse2;                   // [B*Hq, Sp] base-2 log-sum-exp of the scaled scores; +inf beyond S
  const __nv_bfloat16* o_in;     // backward: O and dO, row stride ld_o
  const __nv_bfloat16* dout;
  __nv_bfloat16* dqkv;           // backward: [B*S, (Hq + 2*Hkv)*hd], row stride ld_dqkv
  float* stat;                   // backward: [2][B*Hq, Sp]: -lse2 and -D, left by the dQ kernel for dK / dV
  float* part;                   // hsplit > 1: fp32 partial dK | dV, each [hsplit][B*S][Hkv*hd]
  int B, S, Sp, Hq, Hkv, hd;
  int ld_o, ld_dqkv, hsplit;
  float scale_log2, scale;
  float cap_a;                   // soft-capping, cap * tanh(s * scale / cap): scale / cap
};

// Soft-capped raw score: the value x' with x' * scale = cap * tanh(x * scale / cap), so that everything after it
// (maximum, exponentials, the saved log-sum-exp) goes on as for plain scores.  a = scale / cap.
__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// ---- pair helpers of this file
__device__ __forceinline__ void tma_pair_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2, int c3) {
  const uint32_t bar_leader = smem_u32(bar) & 0xFEFFFFFFu;         // the barrier at this offset in the pair's leader
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(bar_leader), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void umma_pair_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Wait of the MMA warp for arrivals that come from both CTAs.
__device__ __forceinline__ bool test_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool wait_pair(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int code) {
  if (test_cluster(bar, parity)) return true;
  const uint64_t t0 = gtimer();
  for (;;) {
    for (int i = 0; i < 256; ++i)
      if (test_cluster(bar, parity)) return true;
    if (*abort_flag) return false;
    if (gtimer() - t0 > WAIT_NS) {
      *abort_flag = code;
      atomicCAS(&g_attn_error, 0, code);
      return false;
    }
  }
}
__device__ __forceinline__ bool wait_own(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int code) {
  return mbar_wait(bar, parity, abort_flag, code, &g_attn_error);
}

constexpr uint32_t IDESC_S = make_idesc(256, 128, false, false);
constexpr uint32_t IDESC_ACC = make_idesc(256, 256, false, true);
constexpr int RES = 65536;                       // resident operand: four atoms of [128 rows][64 columns]
constexpr int STR = 32768;                       // half of a streamed tile: four atoms of [64][64], or two of [128][64]

// S [256 x 128] = A B': A own 128 rows (atoms of 16 KB), B own 64 of the 128 rows (atoms of 8 KB)
__device__ __forceinline__ void pair_scores(uint32_t d, uint32_t a, uint32_t b, int ksteps) {
  const uint64_t ad = make_desc(a, 16, 1024), bd = make_desc(b, 16, 1024);
#pragma unroll
  for (int kk = 0; kk < 16; ++kk)
    if (kk < ksteps)
      umma_bf16_pair(d, ad + (uint64_t)(((kk >> 2) * 16384 + (kk & 3) * 32) >> 4), bd + (uint64_t)(((kk >> 2) * 8192 + (kk & 3) * 32) >> 4),
                     IDESC_S, kk > 0 ? 1u : 0u);
}
// acc [256 x 256] (+)= A B over 128 rows of B (MN-major, own 128 of the 256 columns), A in tensor memory: two pieces of 64
__device__ __forceinline__ void pair_accumulate(uint32_t acc, uint32_t ta, uint32_t b, bool first) {
  const uint64_t bd = make_desc(b, 16384, 1024);
#pragma unroll
  for (int kk = 0; kk < 8; ++kk)
    umma_pair_ts(acc, ta + (kk >> 2) * 64 + (kk & 3) * 8, bd + (uint64_t)(kk * 128), IDESC_ACC, (first && kk == 0) ? 0u : 1u);
}

struct Bars {
  uint64_t r_full, t_full[2], t_empty[2], c_full[2], c_empty[2], s_full[2], w_ready[2], acc_done, st_full[2];
  uint64_t u_full, u_empty, dp_full, s_free, done;
  uint32_t tmem;
  int abort_flag;
};

// Everything before the roles: barriers, tensor memory, the pair's first meeting.
__device__ __forceinline__ uint32_t enter(Bars* bs, int warp) {
  if (threadIdx.x == 0) {
    mbar_init(&bs->r_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bs->t_full[i], 1); mbar_init(&bs->t_empty[i], 1);
      mbar_init(&bs->c_full[i], 1); mbar_init(&bs->c_empty[i], 1);
      mbar_init(&bs->s_full[i], 1); mbar_init(&bs->w_ready[i], 16);
      mbar_init(&bs->st_full[i], 1);
    }
    mbar_init(&bs->acc_done, 1); mbar_init(&bs->u_full, 1); mbar_init(&bs->u_empty, 1); mbar_init(&bs->dp_full, 1);
    mbar_init(&bs->s_free, 16); mbar_init(&bs->done, 1);
    bs->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 9) tmem_alloc_pair(&bs->tmem, 512);
  fence_before();
  __syncthreads();
  cluster_sync_all();                                  // both CTAs' barriers exist before anyone signals them
  fence_after();
  zen_pdl::enter();
  return bs->tmem;
}
__device__ __forceinline__ void leave(Bars* bs, int warp, uint32_t tm0) {
  fence_before();
  __syncthreads();
  if (*(volatile int*)&bs->abort_flag) {               // copies and products in flight are given time to land
    const uint64_t t0 = gtimer();
    while (gtimer() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  cluster_sync_all();                                  // the peer's products read this CTA's memory
  if (warp == 9) {
    fence_after();
    tmem_dealloc_pair(tm0, 512);
  }
}

// Own rows x columns [w * 128, w * 128 + 128) of the accumulator (w: which of the two warps of a lane quarter).
__device__ __forceinline__ void store_half(uint32_t tacc, int w, int hd, float mul, __nv_bfloat16* dst, bool live) {
  const int hi = (hd + 15) / 16 * 16;
  store_rows(tacc, w * 128, hi < w * 128 + 128 ? hi : w * 128 + 128, hd, mul, dst, live);
}
__device__ __forceinline__ void store_half_f32(uint32_t tacc, int w, int hd, float mul, float* dst, bool live) {
#pragma unroll 1
  for (int c = w * 128; c < w * 128 + 128 && c < hd; c += 16) {
    uint32_t r[16];
    tmem_ld16(tacc + c, r);
    if (!live) continue;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (c + q * 4 < hd)
        *reinterpret_cast<float4*>(dst + c + q * 4) = make_float4(__uint_as_float(r[4 * q]) * mul, __uint_as_float(r[4 * q + 1]) * mul,
                                                                  __uint_as_float(r[4 * q + 2]) * mul, __uint_as_float(r[4 * q + 3]) * mul);
  }
}

// What a CTA walks: FWD / dQ the key tiles up to the pair's later query tile, dK / dV the query tiles from the pair's first key
// tile on, of every query head of its share of the group.
struct Walk {
  int pair, own, b, h0, g, part;                       // tile pair, own 128-row tile, batch, first query head, KV head, head share
  int first, per, n;                                   // first streamed tile, tiles per head, tiles in all
};
template <bool QSIDE>
__device__ __forceinline__ Walk walk_of(const WideParams& p, int cta) {
  Walk k;
  const int nq = (p.S + 127) >> 7, rep = p.Hq / p.Hkv, x = blockIdx.x >> 1;
  k.b = blockIdx.y;
  if (QSIDE) {
    k.pair = gridDim.z - 1 - blockIdx.z;               // heavy (late) query tiles of every head first
    k.h0 = x; k.g = x / rep; k.part = 0;
    k.first = 0;
    k.per = k.n = min(2 * k.pair + 2, nq);
  } else {
    k.pair = blockIdx.z;                               // early key tiles see the most queries
    k.g = x / p.hsplit; k.part = x - k.g * p.hsplit;
    const int heads = rep / p.hsplit;
    k.h0 = k.g * rep + k.part * heads;
    k.first = 2 * k.pair;
    k.per = nq - k.first;
    k.n = heads * k.per;
  }
  k.own = 2 * k.pair + cta;
  return k;
}

// Scores of 64 columns of a row, masked: FWD / dQ columns are keys (hide those after the query), dK / dV queries (those before
// the key).  lim = own row minus first column.
template <bool QSIDE>
__device__ __forceinline__ void mask_scores(uint32_t (&s)[2][32], int lim) {
#pragma unroll
  for (int c = 0; c < 64; ++c)
    if (QSIDE ? c > lim : c < lim) s[c >> 5][c & 31] = 0xff800000u;
}
template <bool CAP>
__device__ __forceinline__ void cap_scores(uint32_t (&s)[2][32], float a) {
  if (!CAP) return;
  const float ia = 1.f / a;
#pragma unroll
  for (int c = 0; c < 64; ++c) s[c >> 5][c & 31] = __float_as_uint(tanh_fast(__uint_as_float(s[c >> 5][c & 31]) * a) * ia);
}

// ============================================================================================ forward, and dV
// 320 threads: warps 0-7 softmax (thread = row of lane quarter warp % 4, columns of half warp / 4), warp 8 TMA, warp 9 MMA (on
// the pair's leader).  Tensor memory: two score buffers [0, 256), P over the first half of each 64 columns; accumulator [256, 512).
constexpr int TWO_SMEM = RES + 4 * STR + 2048 + 512;

template <bool FWD, bool CAP>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(320, 1)
wide_two_kernel(const __grid_constant__ CUtensorMap tm128, const __grid_constant__ CUtensorMap tm64, const __grid_constant__ CUtensorMap tmc,
                const WideParams p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  if ((smem_u32(smem) & 1023u) != 0u) {                // uniform over the grid: nothing has been allocated yet
    if (threadIdx.x == 0) atomicCAS(&g_attn_error, 0, 99);
    return;
  }
  unsigned char *a_s = smem, *t_s = a_s + RES, *c_s = t_s + 2 * STR;
  float* aux = reinterpret_cast<float*>(c_s + 2 * STR);               // FWD: row maxima [2 tiles][2 halves][128]; dV: -lse [2][128]
  Bars* bs = reinterpret_cast<Bars*>(aux + 512);
  volatile int* abort_flag = &bs->abort_flag;
  const int warp = (int)uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int cta = (int)cluster_ctarank();
  const Walk k = walk_of<FWD>(p, cta);
  const int ksteps = (p.hd + 15) >> 4, n = k.n;
  const uint32_t tm0 = enter(bs, warp), tACC = tm0 + 256;

  if (warp == 8) {
    if (lane == 0) {
      if (cta == 0) mbar_expect_tx(&bs->r_full, 2 * RES);
#pragma unroll
      for (int a = 0; a < 4; ++a) tma_pair_4d(a_s + a * 16384, &tm128, &bs->r_full, a * 64, FWD ? k.h0 : p.Hq + k.g, k.own * 128, k.b);
      int h = k.h0, t = k.first;
      for (int i = 0; i < n; ++i) {
        const int e = i & 1;
        const uint32_t ph = ((i >> 1) & 1) ^ 1;
        if (!wait_own(&bs->t_empty[e], ph, abort_flag, 1)) break;
        if (cta == 0) mbar_expect_tx(&bs->t_full[e], 2 * STR);
#pragma unroll
        for (int a = 0; a < 4; ++a)
          tma_pair_4d(t_s + e * STR + a * 8192, &tm64, &bs->t_full[e], a * 64, FWD ? p.Hq + k.g : h, t * 128 + cta * 64, k.b);
        if (!wait_own(&bs->c_empty[e], ph, abort_flag, 2)) break;
        if (cta == 0) mbar_expect_tx(&bs->c_full[e], 2 * STR);
#pragma unroll
        for (int a = 0; a < 2; ++a)
          tma_pair_4d(c_s + e * STR + a * 16384, &tmc, &bs->c_full[e], cta * 128 + a * 64, FWD ? p.Hq + p.Hkv + k.g : h, t * 128, k.b);
        if (!FWD) {                                     // P' of tile i - 2 has been used: so have its statistics
          mbar_expect_tx(&bs->st_full[e], 512);
          bulk_load_1d(aux + e * 128, p.stat + ((size_t)k.b * p.Hq + h) * p.Sp + t * 128, 512, &bs->st_full[e]);
        }
        if (++t == k.first + k.per) { t = k.first; ++h; }
      }
    }
  } else if (warp == 9) {
    if (cta == 0) {
      const bool leader = elect_one();
      const uint32_t tmu = uniform(tm0);
      auto scores = [&](int i) -> bool {
        const int e = i & 1;
        if (!wait_pair(&bs->t_full[e], (i >> 1) & 1, abort_flag, 3)) return false;
        fence_after();
        if (leader) {
          pair_scores(tmu + e * 128, smem_u32(a_s), smem_u32(t_s + e * STR), ksteps);
          umma_commit_pair(&bs->s_full[e]);
          if (i + 2 < n) umma_commit_pair(&bs->t_empty[e]);
        }
        return true;
      };
      bool ok = wait_pair(&bs->r_full, 0, abort_flag, 4) && scores(0);
      for (int i = 0; i < n && ok; ++i) {
        const int e = i & 1;
        if (i + 1 < n && !scores(i + 1)) break;         // its buffer was last read by the accumulating product of tile i - 1
        ok = wait_pair(&bs->c_full[e], (i >> 1) & 1, abort_flag, 5) && wait_pair(&bs->w_ready[e], (i >> 1) & 1, abort_flag, 6);
        if (!ok) break;
        fence_after();
        if (leader) {
          pair_accumulate(tmu + 256, tmu + e * 128, smem_u32(c_s + e * STR), i == 0);
          if (FWD) umma_commit_pair(&bs->acc_done);
          if (i + 2 < n) umma_commit_pair(&bs->c_empty[e]);
          if (i + 1 == n) umma_commit_pair(&bs->done);   // of its own: a wait on acc_done could be two phases behind here
        }
      }
    }
  } else {
    const int w = warp >> 2, row = threadIdx.x & 127;   // row: also the tensor-memory lane
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const uint64_t cs2 = pk2(p.scale_log2, p.scale_log2);
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    int t = k.first;
    for (int i = 0; i < n; ++i) {
      const int e = i & 1;
      const uint32_t tS = tm0 + e * 128 + w * 64 + lane_addr;
      if (!wait_own(&bs->s_full[e], (i >> 1) & 1, abort_flag, 7)) { ok = false; break; }
      if (!FWD && !wait_own(&bs->st_full[e], (i >> 1) & 1, abort_flag, 8)) { ok = false; break; }
      fence_after();
      uint32_t s[2][32];
      tmem_ld32_nowait(tS, s[0]);
      tmem_ld32_nowait(tS + 32, s[1]);
      tmem_wait_ld();
      cap_scores<CAP>(s, p.cap_a);
      if (FWD ? t >= k.own : t <= k.own) mask_scores<FWD>(s, (k.own - t) * 128 + row - w * 64);
      float m_new = 0.f;
      if (FWD) {
        float x0 = -INFINITY, x1 = -INFINITY, x2 = -INFINITY, x3 = -INFINITY;
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          x0 = fmaxf(x0, __uint_as_float(s[0][c])); x1 = fmaxf(x1, __uint_as_float(s[0][16 + c]));
          x2 = fmaxf(x2, __uint_as_float(s[1][c])); x3 = fmaxf(x3, __uint_as_float(s[1][16 + c]));
        }
        float mx = fmaxf(fmaxf(x0, x1), fmaxf(x2, x3));
        // the other 64 columns of the row are with warp (warp ^ 4); buffers alternate, so one meeting per tile is enough
        aux[(e * 2 + w) * 128 + row] = mx;
        asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp & 3)) : "memory");
        mx = fmaxf(mx, aux[(e * 2 + (w ^ 1)) * 128 + row]) * p.scale_log2;
        // lazy maximum: the old reference stays unless the row maximum grew by more than 2^8; P stays below 256, the final
        // normalisation is exact either way, and O is rescaled only on such jumps
        const bool need = mx > m + 8.f;
        m_new = need ? mx : m;
        if (i > 0 && __any_sync(0xffffffffu, need)) {
          if (!wait_own(&bs->acc_done, (i - 1) & 1, abort_flag, 9)) { ok = false; break; }
          fence_after();
          const float alpha = need ? ex2f(m - m_new) : 1.f;
          l *= alpha;
#pragma unroll 1
          for (int c = w * 128; c < w * 128 + 128; c += 16) {
            uint32_t r[16];
            tmem_ld16(tACC + lane_addr + c, r);
#pragma unroll
            for (int q = 0; q < 16; ++q) r[q] = __float_as_uint(__uint_as_float(r[q]) * alpha);
            tmem_st16(tACC + lane_addr + c, r);
          }
        }
        m = m_new;
      }
      const uint64_t nm2 = pk2(-m_new, -m_new);
      const float* lp = aux + e * 128 + w * 64;
      uint64_t sum0 = 0ull, sum1 = 0ull;
      uint32_t pk[32];
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        float4 nl;
        if (!FWD) nl = *reinterpret_cast<const float4*>(lp + q * 4);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int c = q * 4 + u * 2;
          const uint32_t* sp = &s[c >> 5][c & 31];
          float y0, y1;
          exp2_pair(fma2(pk2(__uint_as_float(sp[0]), __uint_as_float(sp[1])), cs2, FWD ? nm2 : (u ? pk2(nl.z, nl.w) : pk2(nl.x, nl.y))), y0, y1);
          if (FWD) {
            if (u) sum1 = add2(sum1, pk2(y0, y1)); else sum0 = add2(sum0, pk2(y0, y1));
          }
          pk[q * 2 + u] = pack_bf16(y0, y1);
        }
      }
      tmem_st32_nowait(tS, pk);
      tmem_wait_st();
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_leader(&bs->w_ready[e]);
      if (FWD) {
        float a0, a1, b0, b1;
        unpk2(sum0, a0, a1);
        unpk2(sum1, b0, b1);
        l += (a0 + a1) + (b0 + b1);
      }
      if (++t == k.first + k.per) t = k.first;
    }
    if (ok && wait_own(&bs->done, 0, abort_flag, 10)) {
      fence_after();
      const int r = k.own * 128 + row;
      const bool live = r < p.S;
      if (FWD) {
        aux[((n & 1) * 2 + w) * 128 + row] = l;         // the buffer that the last tile did not use
        asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp & 3)) : "memory");
        l += aux[((n & 1) * 2 + (w ^ 1)) * 128 + row];
        store_half(tACC + lane_addr, w, p.hd, 1.f / l, p.out + (size_t)(k.b * p.S + r) * p.ld_o + k.h0 * p.hd, live);
        if (w == 0 && r < p.Sp) p.lse2[((size_t)k.b * p.Hq + k.h0) * p.Sp + r] = live ? m + log2f(l) : INFINITY;
      } else if (p.hsplit > 1) {
        const size_t rows = (size_t)p.B * p.S, wid = (size_t)p.Hkv * p.hd;
        store_half_f32(tACC + lane_addr, w, p.hd, 1.f, p.part + ((size_t)(p.hsplit + k.part) * rows + (size_t)k.b * p.S + r) * wid + (size_t)k.g * p.hd, live);
      } else {
        store_half(tACC + lane_addr, w, p.hd, 1.f, p.dqkv + (size_t)(k.b * p.S + r) * p.ld_dqkv + (p.Hq + p.Hkv + k.g) * p.hd, live);
      }
    }
  }
  leave(bs, warp, tm0);
}

// ============================================================================================ dQ, and dK
// Roles as above.  Tensor memory: S [0, 128), dP [128, 256) with dS over the first half of each 64 columns, accumulator
// [256, 512).  One stage for each streamed operand: each is in use for one product in three, the next copy has the time of the
// other two.  The dQ kernel also computes D = rowsum(dO * O) and leaves the statistics for dK / dV.
constexpr int THREE_SMEM = 2 * RES + 3 * STR + 2048 + 512;

template <bool DQ, bool CAP>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(320, 1)
wide_three_kernel(const __grid_constant__ CUtensorMap tm128, const __grid_constant__ CUtensorMap tm64, const __grid_constant__ CUtensorMap tmd128,
                  const __grid_constant__ CUtensorMap tmd64, const WideParams p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  if ((smem_u32(smem) & 1023u) != 0u) {                // uniform over the grid: nothing has been allocated yet
    if (threadIdx.x == 0) atomicCAS(&g_attn_error, 0, 99);
    return;
  }
  unsigned char *a1_s = smem, *a2_s = a1_s + RES, *t_s = a2_s + RES, *u_s = t_s + STR, *c_s = u_s + STR;
  float* aux = reinterpret_cast<float*>(c_s + STR);                   // dQ: partial D [2][128]; dK: -lse | -D, [2 tiles][2][128]
  Bars* bs = reinterpret_cast<Bars*>(aux + 512);
  volatile int* abort_flag = &bs->abort_flag;
  const int warp = (int)uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int cta = (int)cluster_ctarank();
  const Walk k = walk_of<DQ>(p, cta);
  const int ksteps = (p.hd + 15) >> 4, n = k.n;
  const size_t stat_d = (size_t)p.B * p.Hq * p.Sp;
  const uint32_t tm0 = enter(bs, warp), tDP = tm0 + 128, tACC = tm0 + 256;

  if (warp == 8) {
    if (lane == 0) {
      if (cta == 0) mbar_expect_tx(&bs->r_full, 4 * RES);
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        tma_pair_4d(a1_s + a * 16384, &tm128, &bs->r_full, a * 64, DQ ? k.h0 : p.Hq + k.g, k.own * 128, k.b);
        if (DQ) tma_pair_4d(a2_s + a * 16384, &tmd128, &bs->r_full, a * 64, k.h0, k.own * 128, k.b);
        else tma_pair_4d(a2_s + a * 16384, &tm128, &bs->r_full, a * 64, p.Hq + p.Hkv + k.g, k.own * 128, k.b);
      }
      const int last = k.first + k.per;
      auto load_t = [&](int i, int h, int t) -> bool {  // streamed operand of S (and the statistics of its queries)
        if (!wait_own(&bs->t_empty[0], (i & 1) ^ 1, abort_flag, 21)) return false;
        if (cta == 0) mbar_expect_tx(&bs->t_full[0], 2 * STR);
#pragma unroll
        for (int a = 0; a < 4; ++a) tma_pair_4d(t_s + a * 8192, &tm64, &bs->t_full[0], a * 64, DQ ? p.Hq + k.g : h, t * 128 + cta * 64, k.b);
        return true;
      };
      auto load_u = [&](int i, int h, int t) -> bool {  // of dP
        if (!wait_own(&bs->u_empty, (i & 1) ^ 1, abort_flag, 22)) return false;
        if (cta == 0) mbar_expect_tx(&bs->u_full, 2 * STR);
#pragma unroll
        for (int a = 0; a < 4; ++a)
          tma_pair_4d(u_s + a * 8192, DQ ? &tm64 : &tmd64, &bs->u_full, a * 64, DQ ? p.Hq + p.Hkv + k.g : h, t * 128 + cta * 64, k.b);
        return true;
      };
      auto load_c = [&](int i, int h, int t) -> bool {  // of the accumulating product
        if (!wait_own(&bs->c_empty[0], (i & 1) ^ 1, abort_flag, 23)) return false;
        if (cta == 0) mbar_expect_tx(&bs->c_full[0], 2 * STR);
#pragma unroll
        for (int a = 0; a < 2; ++a) tma_pair_4d(c_s + a * 16384, &tm128, &bs->c_full[0], cta * 128 + a * 64, DQ ? p.Hq + k.g : h, t * 128, k.b);
        return true;
      };
      auto load_stat = [&](int i, int h, int t) {       // dS of tile i - 2 has been used: so have the statistics in this buffer
        if (DQ) return;
        const float* src = p.stat + ((size_t)k.b * p.Hq + h) * p.Sp + t * 128;
        mbar_expect_tx(&bs->st_full[i & 1], 1024);
        bulk_load_1d(aux + (i & 1) * 256, src, 512, &bs->st_full[i & 1]);
        bulk_load_1d(aux + (i & 1) * 256 + 128, src + stat_d, 512, &bs->st_full[i & 1]);
      };
      int h = k.h0, t = k.first, hn = h, tn = t;        // tile i, tile i + 1
      if (++tn == last) { tn = k.first; ++hn; }
      load_stat(0, h, t);
      bool ok = load_t(0, h, t) && load_u(0, h, t);
      for (int i = 0; i < n && ok; ++i) {
        // in the order in which the products free the stages: S(i), accumulate(i - 1), dP(i)
        if (i + 1 < n && !load_t(i + 1, hn, tn)) break;
        if (!load_c(i, h, t)) break;
        if (i + 1 < n) {
          load_stat(i + 1, hn, tn);                     // accumulate(i - 1) is over
          if (!load_u(i + 1, hn, tn)) break;
        }
        h = hn; t = tn;
        if (++tn == last) { tn = k.first; ++hn; }
      }
    }
  } else if (warp == 9) {
    if (cta == 0) {
      const bool leader = elect_one();
      const uint32_t tmu = uniform(tm0);
      auto scores = [&](int i) -> bool {
        if (!wait_pair(&bs->t_full[0], i & 1, abort_flag, 24)) return false;
        fence_after();
        if (leader) {
          pair_scores(tmu, smem_u32(a1_s), smem_u32(t_s), ksteps);
          umma_commit_pair(&bs->s_full[0]);
          if (i + 1 < n) umma_commit_pair(&bs->t_empty[0]);
        }
        return true;
      };
      auto dprobs = [&](int i) -> bool {
        if (!wait_pair(&bs->u_full, i & 1, abort_flag, 25)) return false;
        fence_after();
        if (leader) {
          pair_scores(tmu + 128, smem_u32(a2_s), smem_u32(u_s), ksteps);
          umma_commit_pair(&bs->dp_full);
          if (i + 1 < n) umma_commit_pair(&bs->u_empty);
        }
        return true;
      };
      bool ok = wait_pair(&bs->r_full, 0, abort_flag, 26) && scores(0) && dprobs(0);
      for (int i = 0; i < n && ok; ++i) {
        if (i + 1 < n) {
          ok = wait_pair(&bs->s_free, i & 1, abort_flag, 27);
          if (!ok) break;
          fence_after();
          if (!scores(i + 1)) break;
        }
        ok = wait_pair(&bs->c_full[0], i & 1, abort_flag, 28) && wait_pair(&bs->w_ready[0], i & 1, abort_flag, 29);
        if (!ok) break;
        fence_after();
        if (leader) {
          pair_accumulate(tmu + 256, tmu + 128, smem_u32(c_s), i == 0);
          if (i + 1 < n) umma_commit_pair(&bs->c_empty[0]);
          else umma_commit_pair(&bs->done);
        }
        if (i + 1 < n && !dprobs(i + 1)) break;
      }
    }
  } else {
    const int w = warp >> 2, row = threadIdx.x & 127;
    const int r = k.own * 128 + row;
    const bool live = r < p.S;
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tS = tm0 + w * 64 + lane_addr, tD = tDP + w * 64 + lane_addr;
    const uint64_t cs2 = pk2(p.scale_log2, p.scale_log2);
    uint64_t nl_row = 0ull, nd_row = 0ull;
    if (DQ) {
      // D of this row: the two threads of a row take every other 8-column piece of dO * O
      float d = 0.f;
      if (live) {
        const size_t off = (size_t)(k.b * p.S + r) * p.ld_o + k.h0 * p.hd + w * 8;
        d = row_dot<16>(p.dout + off, p.o_in + off, p.hd - w * 8);
      }
      aux[w * 128 + row] = d;
      asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp & 3)) : "memory");
      const float nd = -(aux[row] + aux[128 + row]);
      float nl = -INFINITY;
      if (r < p.Sp) {
        const size_t stat = ((size_t)k.b * p.Hq + k.h0) * p.Sp + r;
        nl = -p.lse2[stat];
        if (w == 0) {
          p.stat[stat] = nl;
          p.stat[stat_d + stat] = nd;
        }
      }
      nl_row = pk2(nl, nl);
      nd_row = pk2(nd, nd);
    }
    bool ok = true;
    int t = k.first;
    for (int i = 0; i < n; ++i) {
      const float *lp = aux + (i & 1) * 256 + w * 64, *dp_ = lp + 128;
      if (!wait_own(&bs->s_full[0], i & 1, abort_flag, 30)) { ok = false; break; }
      if (!DQ && !wait_own(&bs->st_full[i & 1], (i >> 1) & 1, abort_flag, 31)) { ok = false; break; }
      fence_after();
      uint32_t s[2][32];
      tmem_ld32_nowait(tS, s[0]);
      tmem_ld32_nowait(tS + 32, s[1]);
      tmem_wait_ld();
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_leader(&bs->s_free);
      cap_scores<CAP>(s, p.cap_a);
      if (DQ ? t >= k.own : t <= k.own) mask_scores<DQ>(s, (k.own - t) * 128 + row - w * 64);
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        float4 nl;
        if (!DQ) nl = *reinterpret_cast<const float4*>(lp + q * 4);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int c = q * 4 + u * 2;
          uint32_t* sp = &s[c >> 5][c & 31];
          float y0, y1;
          exp2_pair(fma2(pk2(__uint_as_float(sp[0]), __uint_as_float(sp[1])), cs2, DQ ? nl_row : (u ? pk2(nl.z, nl.w) : pk2(nl.x, nl.y))), y0, y1);
          if (CAP) {
            // chain rule through cap * tanh(.): 1 - tanh^2, with tanh = capped score * a (masked entries: factor 0)
            const float t0 = fminf(fabsf(__uint_as_float(sp[0]) * p.cap_a), 1.f), t1 = fminf(fabsf(__uint_as_float(sp[1]) * p.cap_a), 1.f);
            y0 *= 1.f - t0 * t0;
            y1 *= 1.f - t1 * t1;
          }
          sp[0] = __float_as_uint(y0);
          sp[1] = __float_as_uint(y1);
        }
      }
      if (!wait_own(&bs->dp_full, i & 1, abort_flag, 32)) { ok = false; break; }
      fence_after();
      uint32_t d[2][32];
      tmem_ld32_nowait(tD, d[0]);
      tmem_ld32_nowait(tD + 32, d[1]);
      tmem_wait_ld();
      uint32_t pk[32];
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        float4 nd;
        if (!DQ) nd = *reinterpret_cast<const float4*>(dp_ + q * 4);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int c = q * 4 + u * 2;
          const uint32_t *sp = &s[c >> 5][c & 31], *dd = &d[c >> 5][c & 31];
          float y0, y1;
          unpk2(mul2(add2(pk2(__uint_as_float(dd[0]), __uint_as_float(dd[1])), DQ ? nd_row : (u ? pk2(nd.z, nd.w) : pk2(nd.x, nd.y))),
                     pk2(__uint_as_float(sp[0]), __uint_as_float(sp[1]))), y0, y1);
          pk[q * 2 + u] = pack_bf16(y0, y1);
        }
      }
      tmem_st32_nowait(tD, pk);
      tmem_wait_st();
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_leader(&bs->w_ready[0]);
      if (++t == k.first + k.per) t = k.first;
    }
    if (ok && wait_own(&bs->done, 0, abort_flag, 33)) {
      fence_after();
      if (DQ) {
        store_half(tACC + lane_addr, w, p.hd, p.scale, p.dqkv + (size_t)(k.b * p.S + r) * p.ld_dqkv + k.h0 * p.hd, live);
      } else if (p.hsplit > 1) {
        const size_t rows = (size_t)p.B * p.S, wid = (size_t)p.Hkv * p.hd;
        store_half_f32(tACC + lane_addr, w, p.hd, p.scale, p.part + ((size_t)k.part * rows + (size_t)k.b * p.S + r) * wid + (size_t)k.g * p.hd, live);
      } else {
        store_half(tACC + lane_addr, w, p.hd, p.scale, p.dqkv + (size_t)(k.b * p.S + r) * p.ld_dqkv + (p.Hq + k.g) * p.hd, live);
      }
    }
  }
  leave(bs, warp, tm0);
}

// dK and dV of a backward whose heads are shared out: sum the hsplit fp32 partials in order, write bf16 into dqkv.
__global__ void __launch_bounds__(256)
wide_reduce_kernel(const float* part, __nv_bfloat16* __restrict__ dqkv, int rows, int Hq, int Hkv, int hd, int hsplit, int ld) {
  zen_pdl::enter();
  const size_t wid = (size_t)Hkv * hd, per = (size_t)rows * wid;
  const size_t nvec = 2 * per / 8;
  for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < nvec; v += (size_t)gridDim.x * blockDim.x) {
    const size_t e = v * 8;
    const int which = (int)(e / per);                      // 0 = dK, 1 = dV
    const size_t off = e % per;
    const size_t row = off / wid;
    const int col = (int)(off % wid);
    float a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int sidx = 0; sidx < hsplit; ++sidx) {
      const float4* q = reinterpret_cast<const float4*>(part + ((size_t)which * hsplit + sidx) * per + off);
      const float4 x = __ldcs(q), y = __ldcs(q + 1);
      a[0] += x.x; a[1] += x.y; a[2] += x.z; a[3] += x.w; a[4] += y.x; a[5] += y.y; a[6] += y.z; a[7] += y.w;
    }
    __nv_bfloat16* dst = dqkv + row * ld + (size_t)(Hq + which * Hkv) * hd + col;
    *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16(a[0], a[1]), pack_bf16(a[2], a[3]), pack_bf16(a[4], a[5]), pack_bf16(a[6], a[7]));
  }
}

template <typename F>
int opt_in(F* f, int bytes) {
  return (int)cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}
template <bool CAP>
int wide_attrs() {
  static const int rc = [] {
    int r = opt_in(wide_two_kernel<true, CAP>, TWO_SMEM);
    if (!r) r = opt_in(wide_two_kernel<false, CAP>, TWO_SMEM);
    if (!r) r = opt_in(wide_three_kernel<true, CAP>, THREE_SMEM);
    if (!r) r = opt_in(wide_three_kernel<false, CAP>, THREE_SMEM);
    return r;
  }();
  return rc;
}
bool wide_shape_ok(const void* a, const void* b, int S, int Hq, int Hkv, int hd, int ld_a, int ld_b) {
  return S > 0 && Hkv > 0 && Hq % Hkv == 0 && hd >= 8 && hd <= 256 && hd % 8 == 0 && ld_a % 8 == 0 && ld_b % 8 == 0 &&
         reinterpret_cast<uintptr_t>(a) % 16 == 0 && reinterpret_cast<uintptr_t>(b) % 16 == 0;
}

template <bool CAP>
void launch_bwd(const CUtensorMap& t128, const CUtensorMap& t64, const CUtensorMap& d128, const CUtensorMap& d64, const WideParams& p, int np,
                cudaStream_t st) {
  const dim3 gq(2 * p.Hq, p.B, np), gk(2 * p.Hkv * p.hsplit, p.B, np);
  zen_pdl::launch(wide_three_kernel<true, CAP>, gq, 320, THREE_SMEM, st, t128, t64, d128, d64, p);
  zen_pdl::launch(wide_three_kernel<false, CAP>, gk, 320, THREE_SMEM, st, t128, t64, d128, d64, p);
  zen_pdl::launch(wide_two_kernel<false, CAP>, gk, 320, TWO_SMEM, st, t128, t64, d128, p);
}

}  // namespace

extern "C" {

// CTA pairs that share the query heads of one KV head in the dK / dV kernels (a divisor of Hq / Hkv).  Few KV heads leave
// pairs idle (4 x 2048, one KV head: 32 pairs of work for 74), more shares cost fp32 partials: the time of both kernels is
// about 2.8 us per tile and pair, of the busiest pair the average load plus half of the longest share; a share's partials go
// out and come back at 5.5 TB/s.
int zen_attn_hsplit(int B, int S, int Hq, int Hkv, int hd) {
  const int rep = Hkv > 0 ? Hq / Hkv : 1, nq = (S + 127) / 128;
  double tiles = 0, best = 0;
  for (int k = 0; k < nq; k += 2) tiles += nq - k;
  tiles *= (double)B * Hq;
  int pick = 1;
  for (int d = 1; d <= rep; ++d) {
    if (rep % d) continue;
    const double longest = (double)rep / d * nq, load = tiles / 74 + longest / 2;
    double us = 2.8 * (load > longest ? load : longest);
    if (d > 1) us += 4.0 * d * (double)B * S * Hkv * hd * 4 / 5.5e6 + 3;
    if (d == 1 || us < best) { best = us; pick = d; }
  }
  return pick;
}

// Causal attention forward, hd <= 256 (multiple of 8), any S.  qkv: bf16 [B*S, (Hq + 2*Hkv)*hd], row stride ld_qkv; out: bf16
// [B*S, Hq*hd], row stride ld_out; lse2: fp32 [B, Hq, Sp] with Sp = S rounded up to a multiple of 128 (+inf beyond S).
// softcap > 0: scores are soft-capped, cap * tanh(s * scale / cap), before the softmax (0 = none).
int zen_attn_fwd(const void* qkv, void* out, float* lse2, int B, int S, int Hq, int Hkv, int hd, int ld_qkv, int ld_out,
                 float scale, float softcap, void* stream) {
  if (!wide_shape_ok(qkv, out, S, Hq, Hkv, hd, ld_qkv, ld_out)) return -2;
  CUtensorMap t128, t64;
  int rc = zen_tmap::get_heads(qkv, hd, Hq + 2 * Hkv, S, B, ld_qkv, &t128);
  if (!rc) rc = zen_tmap::get_heads(qkv, hd, Hq + 2 * Hkv, S, B, ld_qkv, &t64, 64);
  if (rc) return rc;
  const int nq = (S + 127) / 128;
  WideParams p{};
  p.out = (__nv_bfloat16*)out; p.lse2 = lse2;
  p.B = B; p.S = S; p.Sp = nq * 128; p.Hq = Hq; p.Hkv = Hkv; p.hd = hd; p.ld_o = ld_out; p.hsplit = 1;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f; p.cap_a = softcap > 0.f ? scale / softcap : 0.f;
  const dim3 grid(2 * Hq, B, (nq + 1) / 2);
  cudaStream_t st = (cudaStream_t)stream;
  if (softcap > 0.f) {
    if ((rc = wide_attrs<true>())) return rc;
    zen_pdl::launch(wide_two_kernel<true, true>, grid, 320, TWO_SMEM, st, t128, t64, t128, p);
  } else {
    if ((rc = wide_attrs<false>())) return rc;
    zen_pdl::launch(wide_two_kernel<true, false>, grid, 320, TWO_SMEM, st, t128, t64, t128, p);
  }
  return (int)cudaGetLastError();
}

// Backward of the above.  dout / out: bf16 [B*S, Hq*hd] (row stride ld_o); lse2 from the forward; stat: fp32 scratch
// [2][B, Hq, Sp]; dqkv: bf16 [B*S, (Hq + 2*Hkv)*hd] (row stride ld_dqkv), fully overwritten.
// part / hsplit: with hsplit > 1 the query heads of a KV head are shared out over hsplit pairs of CTAs whose fp32 partial dK / dV
// go to `part` (2 * hsplit * B*S * Hkv*hd floats) and are summed by a last kernel; hsplit divides Hq / Hkv.
int zen_attn_bwd(const void* qkv, const void* out, const void* dout, const float* lse2, float* stat, void* dqkv, int B,
                 int S, int Hq, int Hkv, int hd, int ld_qkv, int ld_o, int ld_dqkv, float scale, float softcap, float* part, int hsplit,
                 void* stream) {
  if (!wide_shape_ok(qkv, out, S, Hq, Hkv, hd, ld_qkv, ld_o) || !wide_shape_ok(dout, dqkv, S, Hq, Hkv, hd, ld_o, ld_dqkv)) return -2;
  if (reinterpret_cast<uintptr_t>(stat) % 16) return -3;
  if (hsplit < 1 || !part) hsplit = 1;
  if ((Hq / Hkv) % hsplit) return -2;
  CUtensorMap t128, t64, d128, d64;
  int rc = zen_tmap::get_heads(qkv, hd, Hq + 2 * Hkv, S, B, ld_qkv, &t128);
  if (!rc) rc = zen_tmap::get_heads(qkv, hd, Hq + 2 * Hkv, S, B, ld_qkv, &t64, 64);
  if (!rc) rc = zen_tmap::get_heads(dout, hd, Hq, S, B, ld_o, &d128);
  if (!rc) rc = zen_tmap::get_heads(dout, hd, Hq, S, B, ld_o, &d64, 64);
  if (rc) return rc;
  const int nq = (S + 127) / 128;
  WideParams p{};
  p.lse2 = const_cast<float*>(lse2); p.o_in = (const __nv_bfloat16*)out; p.dout = (const __nv_bfloat16*)dout;
  p.dqkv = (__nv_bfloat16*)dqkv; p.stat = stat; p.part = part; p.hsplit = hsplit;
  p.B = B; p.S = S; p.Sp = nq * 128; p.Hq = Hq; p.Hkv = Hkv; p.hd = hd; p.ld_o = ld_o; p.ld_dqkv = ld_dqkv;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f; p.cap_a = softcap > 0.f ? scale / softcap : 0.f;
  cudaStream_t st = (cudaStream_t)stream;
  if ((rc = softcap > 0.f ? wide_attrs<true>() : wide_attrs<false>())) return rc;
  if (softcap > 0.f) launch_bwd<true>(t128, t64, d128, d64, p, (nq + 1) / 2, st);
  else launch_bwd<false>(t128, t64, d128, d64, p, (nq + 1) / 2, st);
  if (hsplit > 1) {
    const size_t nvec = (size_t)2 * B * S * Hkv * hd / 8;
    size_t nb = (nvec + 255) / 256;
    if (nb > 148 * 8) nb = 148 * 8;
    zen_pdl::launch_small(wide_reduce_kernel, (int)nb, 256, 0, st, part, (__nv_bfloat16*)dqkv, B * S, Hq, Hkv, hd, hsplit, ld_dqkv);
  }
  return (int)cudaGetLastError();
}

int zen_attn_error() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_attn_error, sizeof(int)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(g_attn_error, &zero, sizeof(int));
  return v;
}

}  // extern "C"
