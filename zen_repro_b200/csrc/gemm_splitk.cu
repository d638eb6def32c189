// bf16 GEMM for outputs with too few tiles to cover the GPU (few tokens: decoding, scoring a short prompt, small batches):
//
//   C[M, N] (+)= A[M, K] * B[N, K]^T (+ bias[N])
//
// A cluster of S CTAs (S = 2..8) shares one 128 x {64, 128} output tile and cuts K into S slices.  Each CTA runs the usual
// TMA -> tcgen05 pipeline over its slice (warp 0 TMA, warp 1 MMA), parks its fp32 accumulator in its own shared memory,
// and after a cluster barrier CTA r sums rows [128 r / S, 128 (r + 1) / S) over all S slices, in slice order, through
// distributed shared memory and writes them.  One launch, no workspace, the same bits every time.
//
// What bounds it: a tile walks K at about 0.25 us per 64-wide block (the latency of loads from HBM over the stages in
// flight), whatever the other SMs do, so the time is the length of that chain; S slices cut it by S and let S times as
// many SMs pull the weights.  64 tokens, 50264 -> 768 (input gradient of an LM head, 77 MB of weights): 208 us on the 6 CTAs of
// the plain kernel.  When it is taken, with how many slices: cluster_split and _plan in ops/gemm.py, by a time model.
#include "launch.cuh"
#include "tc_common.cuh"
#include "tmap_util.cuh"

namespace {

using namespace tc;

__device__ int g_splitk_error = 0;

struct SplitKParams {
  void* C;
  const __nv_bfloat16* bias;
  int M, N, K, ldc, out_fp32, accumulate;
  int num_m, num_n;
};

template <int BN>
struct SkCfg {
  static constexpr int A_BYTES = 128 * 64 * 2, B_BYTES = BN * 64 * 2, STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = BN == 64 ? 8 : 6;                  // 192 KB of loads in flight
  static constexpr int LD = BN + 4;                                // floats per parked row: 16-byte rows without bank conflicts
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 + 256;   // the parked tile reuses the stages
  static_assert(128 * LD * 4 <= STAGES * STAGE_BYTES, "parked tile");
};

__device__ __forceinline__ uint32_t ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_peer_f4(uint32_t local, uint32_t rank) {
  uint32_t remote;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
  return v;
}

template <int BN, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(192, 1)
gemm_splitk_kernel(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb, const SplitKParams p, int S) {
  using C = SkCfg<BN>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::STAGES * C::STAGE_BYTES);
  uint64_t *full = bars, *empty = bars + C::STAGES, *done = bars + 2 * C::STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = (int)uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int rank = (int)ctarank();
  const int tile = blockIdx.x / S;
  const int m0 = (tile % p.num_m) * 128, n0 = (tile / p.num_m) * BN;
  const int nkb = (p.K + 63) / 64;
  const int kb0 = (int)((long)nkb * rank / S), kb1 = (int)((long)nkb * (rank + 1) / S);   // never empty: S <= nkb

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(done, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, BN);
  fence_before();
  __syncthreads();
  fence_after();
  zen_pdl::enter();
  const uint32_t tm0 = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      for (int kb = kb0; kb < kb1; ++kb) {
        const int it = kb - kb0, s = it % C::STAGES;
        if (!mbar_wait(&empty[s], ((it / C::STAGES) & 1) ^ 1, abort_flag, 1, &g_splitk_error)) break;
        unsigned char *sa = smem + s * C::STAGE_BYTES, *sb = sa + C::A_BYTES;
        mbar_expect_tx(&full[s], C::STAGE_BYTES);
        if (!A_MN) {
          tma_load_2d(sa, &ta, &full[s], kb * 64, m0);
        } else {
#pragma unroll
          for (int j = 0; j < 2; ++j) tma_load_2d(sa + j * 8192, &ta, &full[s], m0 + 64 * j, kb * 64);
        }
        if (!B_MN) {
          tma_load_2d(sb, &tb, &full[s], kb * 64, n0);
        } else {
#pragma unroll
          for (int j = 0; j < BN / 64; ++j) tma_load_2d(sb + j * 8192, &tb, &full[s], n0 + 64 * j, kb * 64);
        }
      }
    }
  } else if (warp == 1) {
    const bool leader = elect_one();
    const uint32_t tmu = uniform(tm0);
    constexpr uint32_t IDESC = make_idesc(128, BN, A_MN, B_MN);
    bool ok = true;
    for (int kb = kb0; kb < kb1; ++kb) {
      const int it = kb - kb0, s = it % C::STAGES;
      ok = mbar_wait(&full[s], (it / C::STAGES) & 1, abort_flag, 2, &g_splitk_error);
      if (!ok) break;
      fence_after();
      if (leader) {
        const uint32_t sa = smem_u32(smem + s * C::STAGE_BYTES), sb = sa + C::A_BYTES;
        const uint64_t ad = A_MN ? make_desc(sa, 8192, 1024) : make_desc(sa, 16, 1024);
        const uint64_t bd = B_MN ? make_desc(sb, 8192, 1024) : make_desc(sb, 16, 1024);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          umma_bf16(tmu, ad + (uint64_t)((A_MN ? j * 2048 : j * 32) >> 4), bd + (uint64_t)((B_MN ? j * 2048 : j * 32) >> 4), IDESC, (it > 0 || j > 0) ? 1u : 0u);
        if (kb + C::STAGES < kb1) umma_commit(&empty[s]);          // only where a later load waits for it
      }
    }
    if (ok && leader) umma_commit(done);
  } else {
    // the accumulator to shared memory: row = tensor-memory lane.  All loads have landed and been read when `done` completes.
    if (mbar_wait(done, 0, abort_flag, 3, &g_splitk_error)) {
      fence_after();
      const int grp = warp & 3;
      float* row = reinterpret_cast<float*>(smem) + (grp * 32 + lane) * C::LD;
#pragma unroll 1
      for (int c = 0; c < BN; c += 32) {
        uint32_t r[32];
        tmem_ld32(tm0 + ((uint32_t)(grp * 32) << 16) + c, r);
#pragma unroll
        for (int i = 0; i < 32; i += 4)
          *reinterpret_cast<float4*>(row + c + i) = make_float4(__uint_as_float(r[i]), __uint_as_float(r[i + 1]), __uint_as_float(r[i + 2]), __uint_as_float(r[i + 3]));
      }
    }
  }
  fence_before();
  cluster_sync();                                      // every slice is parked (or its CTA has given up)
  if (!*abort_flag) {
    const int r0 = 128 * rank / S, r1 = 128 * (rank + 1) / S;
    constexpr int V = BN / 4;
    const bool vec = p.ldc % 4 == 0;                  // four elements of either type
    for (int v = threadIdx.x; v < (r1 - r0) * V; v += 192) {
      const int r = r0 + v / V, c = (v % V) * 4;
      if (m0 + r >= p.M || n0 + c >= p.N) continue;
      const uint32_t at = smem_u32(smem) + (uint32_t)(r * C::LD + c) * 4u;
      float4 part[8];
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s < S) part[s] = ld_peer_f4(at, s);
      float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s < S) { o[0] += part[s].x; o[1] += part[s].y; o[2] += part[s].z; o[3] += part[s].w; }
      const size_t off = (size_t)(m0 + r) * p.ldc + n0 + c;
      const bool whole = vec && n0 + c + 4 <= p.N;
      if (p.bias) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (n0 + c + i < p.N) o[i] += __bfloat162float(p.bias[n0 + c + i]);
      }
      if (p.out_fp32) {
        float* cp = reinterpret_cast<float*>(p.C) + off;
        if (whole) {
          if (p.accumulate) { const float4 x = *reinterpret_cast<const float4*>(cp); o[0] += x.x; o[1] += x.y; o[2] += x.z; o[3] += x.w; }
          *reinterpret_cast<float4*>(cp) = make_float4(o[0], o[1], o[2], o[3]);
        } else {
          for (int i = 0; i < 4; ++i)
            if (n0 + c + i < p.N) cp[i] = p.accumulate ? cp[i] + o[i] : o[i];
        }
      } else {
        __nv_bfloat16* cp = reinterpret_cast<__nv_bfloat16*>(p.C) + off;
        if (whole) {
          if (p.accumulate) {
            const uint2 x = *reinterpret_cast<const uint2*>(cp);
            o[0] += __uint_as_float(x.x << 16); o[1] += __uint_as_float(x.x & 0xffff0000u);
            o[2] += __uint_as_float(x.y << 16); o[3] += __uint_as_float(x.y & 0xffff0000u);
          }
          *reinterpret_cast<uint2*>(cp) = make_uint2(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]));
        } else {
          for (int i = 0; i < 4; ++i)
            if (n0 + c + i < p.N) cp[i] = __float2bfloat16_rn(p.accumulate ? __bfloat162float(cp[i]) + o[i] : o[i]);
        }
      }
    }
  }
  __syncthreads();
  if (*abort_flag) {
    const uint64_t t0 = gtimer();
    while (gtimer() - t0 < 200000ull) __nanosleep(1000);
  }
  cluster_sync();                                      // peers may still be reading this CTA's shared memory
  if (warp == 1) {
    fence_after();
    tmem_dealloc(tm0, BN);
  }
}

template <int BN, bool A_MN, bool B_MN>
int launch_splitk(const CUtensorMap& ta, const CUtensorMap& tb, const SplitKParams& p, int S, cudaStream_t st) {
  static const cudaError_t attr = cudaFuncSetAttribute(gemm_splitk_kernel<BN, A_MN, B_MN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SkCfg<BN>::SMEM);
  if (attr != cudaSuccess) return (int)attr;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(p.num_m * p.num_n * S);
  cfg.blockDim = dim3(192);
  cfg.dynamicSmemBytes = SkCfg<BN>::SMEM;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;            // see launch.cuh
  at[1].val.programmaticStreamSerializationAllowed = 1;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = S;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  return zen_pdl::counted(cudaLaunchKernelEx(&cfg, gemm_splitk_kernel<BN, A_MN, B_MN>, ta, tb, p, S));
}

}  // namespace

extern "C" {

// C[M,N] (+)= A * B^T (+ bias): operands, strides and output as for zen_gemm_bf16; bn = 64 or 128 columns per tile, S = 2..8
// slices of K (at most one per 64-wide block).
int zen_gemm_bf16_cluster_splitk(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, int lda, int ldb,
                                 int ldc, int a_mn, int b_mn, int out_fp32, int accumulate, int bn, int S, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0) return -1;
  if ((lda % 8) || (ldb % 8) || (reinterpret_cast<uintptr_t>(A) % 16) || (reinterpret_cast<uintptr_t>(B) % 16)) return -2;
  if ((bn != 64 && bn != 128) || S < 2 || S > 8 || S > (K + 63) / 64) return -3;
  CUtensorMap ta, tb;
  int rc = a_mn ? zen_tmap::get(A, M, K, lda, 64, 64, &ta) : zen_tmap::get(A, K, M, lda, 64, 128, &ta);
  if (!rc) rc = b_mn ? zen_tmap::get(B, N, K, ldb, 64, 64, &tb) : zen_tmap::get(B, K, N, ldb, 64, bn, &tb);
  if (rc) return rc;
  // the vector stores need rows that start on the vector's boundary
  const bool aligned = reinterpret_cast<uintptr_t>(C) % (out_fp32 ? 16 : 8) == 0;
  SplitKParams p{C, (const __nv_bfloat16*)bias, M, N, K, ldc, out_fp32, accumulate, (M + 127) / 128, (N + bn - 1) / bn};
  if (!aligned) return -2;
  cudaStream_t st = (cudaStream_t)stream;
#define SK(BN_)                                                                   \
  do {                                                                            \
    if (!a_mn && !b_mn) return launch_splitk<BN_, false, false>(ta, tb, p, S, st); \
    if (!a_mn && b_mn) return launch_splitk<BN_, false, true>(ta, tb, p, S, st);   \
    if (a_mn && !b_mn) return launch_splitk<BN_, true, false>(ta, tb, p, S, st);   \
    return launch_splitk<BN_, true, true>(ta, tb, p, S, st);                       \
  } while (0)
  if (bn == 64) SK(64);
  SK(128);
#undef SK
}

int zen_gemm_splitk_error() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_splitk_error, sizeof(int)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(g_splitk_error, &zero, sizeof(int));
  return v;
}

}  // extern "C"
