// Sparse all-reduce kernels (element granule) for sm_100a.
//
// Pipeline per bucket, one launch each, all on one stream, no host sync:
//   zen_partition_push  : stream the flat bucket through a shared-memory ring filled by bulk
//                         asynchronous copies (cp.async.bulk + mbarrier), hash 64-element blocks to
//                         owners, stage (slot, value) records per owner in shared memory and push
//                         them in large contiguous runs straight into the owner's receive region
//                         over NVLink (P2P stores).
//   zen_owner_reduce    : bounded wait on every source's mailbox at once; with many records, sort them by bucket of the
//                         owner's slots (K2b).
//   zen_gather_push     : add up a bucket's records in shared memory, compact the touched slots chunk by chunk, reserve
//                         room in the payload with one atomic per bucket and push bitmap|COO + values to every peer
//                         (P2P stores, or one multimem store through the NVSwitch when a multicast alias of the region
//                         exists).  (K3b; owners of more than 2^25 slots keep sums and bitmap in global memory, K2 + K3.)
//   zen_densify         : bounded wait on each owner's mailbox, one pass over the output that
//                         writes zeros and values together.
//
// Record slots and their mailboxes exist twice and alternate with the parity of the call number, so a
// rank that is one call ahead never writes into records that a slower peer is still reading.
//
// Replaces, in the reference: the three sparse_balance kernels and the
// boolean-mask compaction after them (functions_cuda_kernel.cu:97-167,
// tensor_load_balance.py:24-51), both all_to_all calls and the scatter_add /
// nonzero between them (comm.py:117-127), encode_bitmap / decode_bitmap and the
// padded all_gathers (comm.py:59-99, 128-145).
#include <type_traits>

#include "launch.cuh"
#include "tc_common.cuh"
#include "zen_common.cuh"

struct ZenSparseCtx {
  int32_t rank;
  int32_t nranks;
  uint32_t epoch;
  uint32_t fmt_mode;        // 0 auto, ZEN_FMT_COO, ZEN_FMT_BITMAP
  uint64_t wait_ns;
  char* sym[ZEN_MAX_RANKS]; // base of every rank's symmetric region
  uint64_t off_rec_mail;    // ZenMail[2][ZEN_MAX_RANKS], indexed by call parity and source
  uint64_t off_g_mail;      // ZenMail[ZEN_MAX_RANKS], indexed by owner
  uint64_t off_rec;         // uint2[2][P][cap_rec], indexed by call parity and source
  uint64_t off_g_idx;       // uint32[P][g_idx_words]: bitmap words or COO slots
  uint64_t off_g_off;       // uint32[P][nchunks + 1]: value offset of every 1024-slot chunk
  uint64_t off_g_val;       // T[P][cap_g] (stride in bytes: cap_g * 4)
  uint32_t cap_rec;
  uint32_t cap_g;
  uint32_t g_idx_words;
  uint32_t nchunks;
  float* acc;               // [S] local
  uint32_t* bitmap;         // [nwords] local
  uint32_t* seg;            // [buckets][P * tiles] runs of a bucket in the sorted record tiles (K2b)
  uint32_t* cursors;        // [P] record cursors, [MAX] done counter K1, [MAX+1] done counter K3, [MAX+2] payload cursor, [MAX+3] what K2 / K2b tells the gather
  uint32_t* status;         // status word
  uint64_t numel;           // N
  uint32_t nslots;          // S = sb * G
  uint32_t nwords;          // ceil(S / 32)
  ZenPerm perm;
  const uint32_t* epoch_dev;  // optional: call counter on the device (zen_sparse_epoch_bump); overrides `epoch`
  char* mc;                   // optional: multicast alias of the symmetric region (stores reach every rank)
  uint32_t k1_density_ppm;    // nonzeros per million elements that the plan was sized for (0 = unknown)
  uint32_t seg_words;         // what `seg` holds
};

// Contexts, inputs and outputs of the ranks that one launch works for: one, or all ranks of a call that runs on one device
// (blockIdx.y = rank), where launching rank by rank left most of the GPU idle for small buckets (50 000 elements on two ranks:
// 8 launches of 4 to 12 us each).
template <int NB>
struct ZenSparseBatch {
  ZenSparseCtx c[NB];
  const void* in[NB];
  void* out[NB];
};

// The context of this CTA's rank.  With several in the parameters the index is dynamic and every field read would be a
// load from parameter memory: they are copied to shared memory once.
template <int NB>
__device__ __forceinline__ const ZenSparseCtx& zen_ctx(const ZenSparseBatch<NB>& b, ZenSparseCtx& s) {
  if constexpr (NB == 1) {
    return b.c[0];
  } else {
    static_assert(sizeof(ZenSparseCtx) % 4 == 0, "copied by words");
    const uint32_t* src = reinterpret_cast<const uint32_t*>(&b.c[blockIdx.y]);
    for (uint32_t i = threadIdx.x; i < sizeof(ZenSparseCtx) / 4; i += blockDim.x) reinterpret_cast<uint32_t*>(&s)[i] = src[i];
    __syncthreads();
    return s;
  }
}

// Orders this CTA's stores before its arrival at the counter whose last CTA publishes them.  All ranks on one device: GPU scope
// (a system-scope fence in every CTA costs 4 to 5 us of a launch).  Peers on other devices: by the memory model GPU scope would do
// here too, since the last CTA's system-scope release is cumulative over what it has seen, but that form has not run between GPUs.
template <int NB>
__device__ __forceinline__ void arrive_fence() {
  if constexpr (NB > 1) __threadfence();
  else __threadfence_system();
}
// The last CTA's side of it: what the others arrived with is visible after the fence; `epoch` goes to the mail last.  All ranks on one
// device: the consumer is a later kernel of the stream, so the stores need no release and the fence no system scope (each costs
// the last CTA, and with it a small call, one to three microseconds: 50 000 elements on two ranks 27.1 -> 20.3 us).
template <int NB>
__device__ __forceinline__ void publish_fence() {
  if constexpr (NB > 1) __threadfence();
  else __threadfence_system();
}
template <int NB>
__device__ __forceinline__ void publish_epoch(uint32_t* p, uint32_t v) {
  if constexpr (NB > 1) *reinterpret_cast<volatile uint32_t*>(p) = v;
  else zen_st_release_sys(p, v);
}

__device__ __forceinline__ uint32_t zen_epoch(const ZenSparseCtx& c) { return c.epoch_dev ? *c.epoch_dev : c.epoch; }
__device__ __forceinline__ uint2* zen_rec_slots(const ZenSparseCtx& c, int at_rank, int src, uint32_t epoch) {
  return reinterpret_cast<uint2*>(c.sym[at_rank] + c.off_rec) + ((uint64_t)(epoch & 1u) * c.nranks + src) * c.cap_rec;
}
__device__ __forceinline__ ZenMail* zen_rec_mail(const ZenSparseCtx& c, int at_rank, int src, uint32_t epoch) {
  return reinterpret_cast<ZenMail*>(c.sym[at_rank] + c.off_rec_mail) + (epoch & 1u) * ZEN_MAX_RANKS + src;
}

#define K1_THREADS 288                                  // eight consumer warps and the producer warp
#define K1_WARPS 8
// Records of a queue: a longer queue is drained less often (every drain stops the consumer warps twice), as long as three CTAs still fit
// an SM.  us with 256 / 512: four ranks of 4 M bf16 at 10 % 30.8 / 25.9, two of 13 M fp32 at 2 % 32.8 / 29.6, eight of 64 M at 1 % 207 / 228.
__host__ __device__ __forceinline__ uint32_t k1_qcap(int queues) { return queues <= 4 ? 512u : 256u; }
#define K1_FLUSH_MIN 128
#define K1_STAGE_BYTES 16384
#define K1_NS 2
#define K1_LIST 64                                      // listed vectors per warp (a ring)

// 32 consecutive bytes of the bucket as raw bits: 8 fp32 or 16 16-bit elements, all in one 64-element block.
template <typename T>
struct RawV {
  static constexpr int E = 32 / sizeof(T);
  uint32_t w[8];

  __device__ __forceinline__ void load(const T* g, uint64_t e0, uint64_t n) {     // guarded element by element
    if constexpr (sizeof(T) == 4) {
#pragma unroll
      for (int i = 0; i < 8; ++i) w[i] = (e0 + i < n) ? reinterpret_cast<const uint32_t*>(g)[e0 + i] : 0u;
    } else {
      const unsigned short* gs = reinterpret_cast<const unsigned short*>(g);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t lo = (e0 + 2 * i < n) ? gs[e0 + 2 * i] : 0u, hi = (e0 + 2 * i + 1 < n) ? gs[e0 + 2 * i + 1] : 0u;
        w[i] = lo | (hi << 16);
      }
    }
  }
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = 0u;
  }
  __device__ __forceinline__ bool any() const {
    return ((w[0] | w[1] | w[2] | w[3] | w[4] | w[5] | w[6] | w[7]) & (sizeof(T) == 4 ? 0x7fffffffu : 0x7fff7fffu)) != 0u;
  }
  // cheap test "some element may reach the threshold" (keep_mask decides): magnitudes compared as integers, for bf16 the
  // largest of each half by the packed maximum (t16 = the threshold's bits rounded up to 16)
  __device__ __forceinline__ bool hit(uint32_t tbits, uint32_t t16) const {
    if constexpr (sizeof(T) == 4) {
      uint32_t m = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) m = max(m, w[i] & 0x7fffffffu);
      return m >= tbits;
    } else {
      uint32_t m = w[0] & 0x7fff7fffu;
#pragma unroll
      for (int i = 1; i < 8; ++i) m = __vmaxu2(m, w[i] & 0x7fff7fffu);
      return max(m & 0xffffu, m >> 16) >= t16;
    }
  }
};
// Bit i set when element i of a vector (words at `w` in shared memory) is kept: |x| >= threshold, as an integer compare of the
// magnitude bits (monotonic for non-negative floats); tbits = 1 keeps every nonzero; NaNs are dropped when a real threshold
// is in force.
template <typename T>
__device__ __forceinline__ uint32_t keep_mask(const uint32_t* w, uint32_t tbits, bool use_thr, float thr) {
  uint32_t m = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t v = w[k];
    if constexpr (sizeof(T) == 4) {
      const uint32_t a = v & 0x7fffffffu;
      m |= (a >= tbits && (!use_thr || a <= 0x7f800000u)) ? (1u << k) : 0u;
    } else if constexpr (std::is_same<T, __nv_bfloat16>::value) {
      const uint32_t lo = (v & 0x7fffu) << 16, hi = v & 0x7fff0000u;           // magnitudes as fp32 bit patterns
      m |= (lo >= tbits && (!use_thr || lo <= 0x7f800000u)) ? (1u << (2 * k)) : 0u;
      m |= (hi >= tbits && (!use_thr || hi <= 0x7f800000u)) ? (2u << (2 * k)) : 0u;
    } else {
      const __half2 h = *reinterpret_cast<const __half2*>(&v);
      const float x = fabsf(__low2float(h)), y = fabsf(__high2float(h));
      m |= ((v & 0x7fffu) != 0u && (!use_thr || x >= thr)) ? (1u << (2 * k)) : 0u;
      m |= ((v & 0x7fff0000u) != 0u && (!use_thr || y >= thr)) ? (2u << (2 * k)) : 0u;
    }
  }
  return m;
}

// ---------------------------------------------------------------------------------------------
// K1: partition + compact + push.  The bucket streams through a ring of K1_NS shared-memory stages:
// a producer warp keeps them filled with bulk asynchronous copies (full / empty mbarriers per stage),
// eight consumer warps scan them.  Every lane owns 32 consecutive bytes at a time (all in one
// 64-element block, hence one owner); vectors that hold a kept element are first compacted into a per-warp
// list, and the expensive part -- owner lookup, queue reservation, record writes -- runs on 32 listed
// vectors at a time with every lane busy.  Records go to per-owner queues in shared memory; every
// `batch` stages the consumer warps meet at a named barrier and warp w drains queue w to the owner's
// receive region in runs of at least K1_FLUSH_MIN records (a queue that fills up earlier spills
// straight to the destination).  kBroadcast = true is the method-1 variant: one queue of
// (global index, value) records pushed to every peer.  kRing = false reads the bucket with plain
// loads instead (a base pointer that is not 16-byte aligned).
//
// What bounds it: instruction issue.  With 16-byte vectors and a three-operation test per word it ran 85 instructions per warp
// and 512 bytes, 39 us for 2^26 bf16 elements at 1 % (20.5 us of memory time); 32-byte vectors halve the ballots and list
// stores, the packed maximum (or one OR chain without a threshold) replaces the per-word test, and a stage carries two
// vectors per lane.
#define K1_CONSUMERS 256
__device__ __forceinline__ void k1_consumer_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

struct K1Entry { uint32_t w[8]; };

template <typename T, bool kBroadcast, bool kRing, int NB>
__global__ void __launch_bounds__(K1_THREADS, 3)
zen_partition_push_kernel(const __grid_constant__ ZenSparseBatch<NB> bt, const float* thr_ptr, int batch) {
  zen_pdl::enter();
  __shared__ ZenSparseCtx s_ctx;
  const ZenSparseCtx& c = zen_ctx(bt, s_ctx);
  const T* g = reinterpret_cast<const T*>(bt.in[NB > 1 ? blockIdx.y : 0]);
  extern __shared__ __align__(128) unsigned char smem_raw[];
  constexpr uint32_t VB = 32;                                         // bytes of one vector
  constexpr uint32_t VE = RawV<T>::E;                                 // its elements
  constexpr uint32_t EPS = K1_STAGE_BYTES / sizeof(T);                // elements per stage
  constexpr int VPL = K1_STAGE_BYTES / VB / K1_CONSUMERS;             // vectors per lane per stage
  static_assert(VPL >= 1, "stage too small");
  const int nq = kBroadcast ? 1 : c.nranks;
  const uint32_t qcap = k1_qcap(nq);
  unsigned char* ring = smem_raw;                                     // [K1_NS][K1_STAGE_BYTES] (kRing)
  uint2* q = reinterpret_cast<uint2*>(smem_raw + (kRing ? K1_NS * K1_STAGE_BYTES : 0));   // [nq][qcap]
  __shared__ uint64_t full[K1_NS], empty[K1_NS];
  __shared__ uint32_t qn[ZEN_MAX_RANKS];
  __shared__ uint32_t qvalid[ZEN_MAX_RANKS];
  __shared__ uint32_t s_last;
  __shared__ int s_abort;
  __shared__ __align__(16) K1Entry wdat[K1_WARPS][K1_LIST];           // per-warp list of vectors with a kept element (a ring)
  __shared__ uint32_t wel[K1_WARPS][K1_LIST];                         // ... and their first element index

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool use_thr = thr_ptr != nullptr;
  const float thr = use_thr ? fmaxf(*thr_ptr, 0.f) : 0.f;
  const uint32_t tbits = use_thr ? max(__float_as_uint(thr), 1u) : 1u; // magnitude bits an element must reach to be kept
  // the same threshold for the cheap per-vector test of 16-bit types, rounded up to 16 bits; any nonzero for fp16, where the
  // threshold is applied in keep_mask
  const uint32_t t16 = std::is_same<T, __half>::value ? 1u : max((tbits + 0xffffu) >> 16, 1u);
  const bool plain = tbits <= 1u || std::is_same<T, __half>::value;
  const uint64_t N = c.numel;
  const uint32_t nst = (uint32_t)((N + EPS - 1) / EPS);               // stages of the whole bucket
  const uint64_t copy_end = (N * sizeof(T)) & ~15ull;                 // bytes that bulk copies may fetch
  const uint32_t full_stages = (uint32_t)(copy_end / K1_STAGE_BYTES);
  const uint32_t epoch = zen_epoch(c);
  const uint64_t rec_base = ((uint64_t)(epoch & 1u) * c.nranks + c.rank) * c.cap_rec;
  const ZenPerm perm = c.perm;
  uint32_t local_status = 0;
  if (batch < 1) batch = 1;

  if (tid < ZEN_MAX_RANKS) { qn[tid] = 0; qvalid[tid] = 0; }
  if (tid == 0) {
    s_abort = 0;
    if (kRing) {
      for (int s = 0; s < K1_NS; ++s) { tc::mbar_init(&full[s], 1); tc::mbar_init(&empty[s], K1_WARPS); }
      tc::fence_barrier_init();
    }
  }
  __syncthreads();

  auto stage_bytes = [&](uint32_t it) -> uint32_t {
    if (it < full_stages) return K1_STAGE_BYTES;
    const uint64_t b0 = (uint64_t)it * K1_STAGE_BYTES;
    return b0 >= copy_end ? 0u : (uint32_t)(copy_end - b0);
  };
  // bounded wait on an mbarrier phase; gives up at once when the CTA has already aborted
  auto wait_phase = [&](uint64_t* bar, uint32_t parity) -> bool {
    if (tc::mbar_test(bar, parity)) return true;
    const uint64_t t0 = zen_globaltimer();
    for (;;) {
      for (int i = 0; i < 128; ++i)
        if (tc::mbar_test(bar, parity)) return true;
      if (*(volatile int*)&s_abort || zen_globaltimer() - t0 > c.wait_ns) { s_abort = 1; return false; }
    }
  };

  if (warp == K1_WARPS) {
    // ---- producer warp: one lane keeps the ring full
    if (kRing && lane == 0) {
      uint32_t issued[K1_NS] = {};
      uint32_t k = 0;
      for (uint32_t it = blockIdx.x; it < nst; it += gridDim.x, ++k) {
        const int s = k % K1_NS;
        if (k >= K1_NS && !wait_phase(&empty[s], ((k / K1_NS) - 1u) & 1u)) break;
        const uint32_t b = stage_bytes(it);
        tc::mbar_expect_tx(&full[s], b);
        if (b) tc::bulk_load_1d(ring + s * K1_STAGE_BYTES, reinterpret_cast<const unsigned char*>(g) + (uint64_t)it * K1_STAGE_BYTES, b, &full[s]);
        ++issued[s];
      }
      if (*(volatile int*)&s_abort) {
        // give the copies that are still in flight a bounded chance to land before the CTA (and its shared memory) goes
        const uint64_t t0 = zen_globaltimer();
        for (int s = 0; s < K1_NS; ++s) {
          if (!issued[s]) continue;
          while (!tc::mbar_test(&full[s], (issued[s] - 1u) & 1u) && zen_globaltimer() - t0 < c.wait_ns) {}
        }
      }
    }
  } else {
    // ---- consumer warps
    uint32_t wtail = 0, whead = 0;                                    // list entries appended / consumed (warp-uniform)

    // Records of the listed vector `idx`: choose the owner, reserve queue space, write them.
    auto emit = [&](uint32_t idx) {
      const K1Entry& en = wdat[warp][idx & (K1_LIST - 1u)];
      const uint32_t e32 = wel[warp][idx & (K1_LIST - 1u)];
      uint32_t wv[8];
      *reinterpret_cast<uint4*>(&wv[0]) = *reinterpret_cast<const uint4*>(&en.w[0]);
      *reinterpret_cast<uint4*>(&wv[4]) = *reinterpret_cast<const uint4*>(&en.w[4]);
      uint32_t m = keep_mask<T>(wv, tbits, use_thr, thr);
      if (!m) return;
      uint32_t owner = 0, slot0 = e32;
      if (!kBroadcast) {
        const uint32_t pb = zen_perm_fwd(perm, e32 >> perm.lg);
        owner = zen_owner_of(perm, pb, c.nranks);
        slot0 = ((pb - owner * perm.sb) << perm.lg) + (e32 & (perm.block - 1u));
      }
      const uint32_t cnt = __popc(m);
      uint32_t k = atomicAdd(&qn[owner], cnt);
      bool direct = false;
      if (k + cnt > qcap) {
        if (k <= qcap) qvalid[owner] = k;                          // exactly one lane per overflow sees this
        direct = true;
        k = atomicAdd(&c.cursors[owner], cnt);                        // reserve directly in the destination
      }
      while (m) {
        const int i = __ffs(m) - 1;
        m &= m - 1;
        const uint2 rec = make_uint2(slot0 + i, sizeof(T) == 4 ? en.w[i] : (uint32_t)reinterpret_cast<const unsigned short*>(en.w)[i]);
        if (!direct) {
          q[owner * qcap + k] = rec;
        } else if (k < c.cap_rec) {
          if (kBroadcast) {
            for (int p = 0; p < c.nranks; ++p)
              (reinterpret_cast<uint2*>(c.sym[p] + c.off_rec) + rec_base)[k] = rec;
          } else {
            (reinterpret_cast<uint2*>(c.sym[owner] + c.off_rec) + rec_base)[k] = rec;
          }
        } else {
          local_status |= ZEN_REC_OVERFLOW;
        }
        ++k;
      }
    };
    // warp w drains queue w when it holds a worthwhile run (or at the end)
    auto flush = [&](bool final_flush) {
      if (warp < nq) {
        uint32_t n = qn[warp];
        const bool overflowed = n > qcap;
        if (overflowed) n = qvalid[warp];
        if (n > 0 && (n >= K1_FLUSH_MIN || final_flush || overflowed)) {
          uint32_t gbase = 0;
          if (lane == 0) gbase = atomicAdd(&c.cursors[warp], n);
          gbase = __shfl_sync(0xffffffffu, gbase, 0);
          const uint32_t fit = (gbase >= c.cap_rec) ? 0u : min(n, c.cap_rec - gbase);
          if (fit < n) local_status |= ZEN_REC_OVERFLOW;
          const uint2* src = q + warp * qcap;
          if (kBroadcast) {
            for (int p = 0; p < c.nranks; ++p) {
              uint2* dst = reinterpret_cast<uint2*>(c.sym[p] + c.off_rec) + rec_base + gbase;
              for (uint32_t i = lane; i < fit; i += 32) dst[i] = src[i];
            }
          } else {
            uint2* dst = reinterpret_cast<uint2*>(c.sym[warp] + c.off_rec) + rec_base + gbase;
            for (uint32_t i = lane; i < fit; i += 32) dst[i] = src[i];
          }
          __syncwarp();
          if (lane == 0) { qn[warp] = 0; qvalid[warp] = 0; }
        } else if (overflowed && lane == 0) {
          qn[warp] = 0; qvalid[warp] = 0;
        }
      }
    };

    uint32_t kk = 0;
    int since = 0;
    const uint32_t lt_mask = (1u << lane) - 1u;
    for (uint32_t it = blockIdx.x; it < nst; it += gridDim.x, ++kk) {
      const int s = kk % K1_NS;
      RawV<T> v[VPL];
      const uint32_t ebase = it * EPS + tid * VE;                      // first element of this lane's first vector
      if (kRing) {
        const bool ok = wait_phase(&full[s], (kk / K1_NS) & 1u);
        const unsigned char* st = ring + s * K1_STAGE_BYTES + tid * VB;
        if (ok && it < full_stages) {                                  // a whole stage: no bounds to look at
#pragma unroll
          for (int u = 0; u < VPL; ++u) {
            const uint4* p4 = reinterpret_cast<const uint4*>(st + u * K1_CONSUMERS * VB);
            *reinterpret_cast<uint4*>(&v[u].w[0]) = p4[0];
            *reinterpret_cast<uint4*>(&v[u].w[4]) = p4[1];
          }
        } else {
          const uint32_t sb = ok ? stage_bytes(it) : 0u;
#pragma unroll
          for (int u = 0; u < VPL; ++u) {
            const uint32_t vi = u * K1_CONSUMERS + tid;
            const uint64_t e0 = (uint64_t)it * EPS + (uint64_t)vi * VE;
            if ((vi + 1) * VB <= sb) {
              const uint4* p4 = reinterpret_cast<const uint4*>(st + u * K1_CONSUMERS * VB);
              *reinterpret_cast<uint4*>(&v[u].w[0]) = p4[0];
              *reinterpret_cast<uint4*>(&v[u].w[4]) = p4[1];
            } else if (ok && e0 < N) {
              v[u].load(g, e0, N);                                     // ragged end of the bucket: guarded plain loads
            } else {
              v[u].zero();
            }
          }
        }
      } else {
#pragma unroll
        for (int u = 0; u < VPL; ++u) {
          const uint64_t e0 = (uint64_t)it * EPS + (uint64_t)(u * K1_CONSUMERS + tid) * VE;
          if (e0 < N) v[u].load(g, e0, N); else v[u].zero();
        }
      }
      const bool last_it = (it + gridDim.x >= nst);
      bool hit[VPL];
      uint32_t bals[VPL];
#pragma unroll
      for (int u = 0; u < VPL; ++u) {
        hit[u] = plain ? v[u].any() : v[u].hit(tbits, t16);            // most vectors of a bucket stop here
        bals[u] = __ballot_sync(0xffffffffu, hit[u]);
      }
      if (kRing) {
        // This warp is done with the stage.  Not before the ballots, which need every word that was read: a load that has only
        // been issued may still be queued when the arrival (of another unit) lets the next copy into the stage, and then returns
        // the wrong stage's data (seen in one call of fifty at 8 x 3 M bf16: sixteen bytes of a lane's second vector).
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&empty[s]);
      }
#pragma unroll
      for (int u = 0; u < VPL; ++u) {
        const uint32_t bal = bals[u];
        if (!bal) continue;
        if (hit[u]) {
          const uint32_t idx = (wtail + __popc(bal & lt_mask)) & (K1_LIST - 1u);
          wel[warp][idx] = ebase + (uint32_t)u * (K1_CONSUMERS * VE);
          uint4* p4 = reinterpret_cast<uint4*>(&wdat[warp][idx]);
          p4[0] = make_uint4(v[u].w[0], v[u].w[1], v[u].w[2], v[u].w[3]);
          p4[1] = make_uint4(v[u].w[4], v[u].w[5], v[u].w[6], v[u].w[7]);
        }
        wtail += __popc(bal);
        if (wtail - whead >= 32) {
          __syncwarp();
          emit(whead + lane);
          whead += 32;
          __syncwarp();
        }
      }
      if (last_it && wtail != whead) {                     // leftovers of this warp: drain with the lanes that have one
        __syncwarp();
        if ((uint32_t)lane < wtail - whead) emit(whead + lane);
        whead = wtail;
      }
      if (++since >= batch || last_it) {
        since = 0;
        k1_consumer_sync();                                // every consumer's records are in the queues
        flush(last_it);
        k1_consumer_sync();                                // queues drained before the next records arrive
      }
    }
  }

  if (s_abort) local_status |= ZEN_TIMEOUT;
  if (local_status) atomicOr(c.status, local_status);
  // completion: the last CTA to arrive publishes counts and epochs to the consumers.  Every thread's stores are
  // ordered before thread 0's fence by the barrier (the fence is cumulative).
  __syncthreads();
  if (tid == 0) {
    arrive_fence<NB>();
    const uint32_t prev = atomicAdd(&c.cursors[ZEN_MAX_RANKS], 1u);
    s_last = (prev == gridDim.x - 1) ? 1u : 0u;
  }
  __syncthreads();
  if (s_last) {
    publish_fence<NB>();
    if (tid < c.nranks) {
      const int p = tid;
      const uint32_t raw = atomicAdd(&c.cursors[kBroadcast ? 0 : p], 0u);
      const uint32_t st = atomicOr(c.status, 0u);
      ZenMail* mail = zen_rec_mail(c, p, c.rank, epoch);
      mail->count = min(raw, c.cap_rec);
      mail->info = ((raw > c.cap_rec) || (st & ZEN_REC_OVERFLOW)) ? 1u : 0u;
      mail->aux = 0;
      publish_epoch<NB>(&mail->epoch, epoch);
    }
    __syncthreads();
    if (tid < ZEN_MAX_RANKS + 1) c.cursors[tid] = 0;                  // ready for the next call
  }
}

// Records received from sources [src_begin, src_end), s_n[source - src_begin], after a bounded wait for each one's mail; one thread per
// source.  Returns the calling thread's part of the status.  Every CTA waits for itself and one may give up on a mail that another
// still saw, so every CTA has to report what it got: its records are missing from the result.
__device__ __forceinline__ uint32_t records_wait(const ZenSparseCtx& c, uint32_t epoch, int src_begin, int src_end, uint32_t* s_n) {
  uint32_t status = 0;
  if ((int)threadIdx.x < src_end - src_begin) {
    const ZenMail* mail = zen_rec_mail(c, c.rank, src_begin + threadIdx.x, epoch);
    uint32_t n = 0;
    if (zen_wait_epoch(&mail->epoch, epoch, c.wait_ns)) {
      // count and info were written before the epoch's release store: plain loads after the acquire above see them
      n = min(*reinterpret_cast<const volatile uint32_t*>(&mail->count), c.cap_rec);
      if (*reinterpret_cast<const volatile uint32_t*>(&mail->info) & 1u) status = ZEN_PEER_OVERFLOW;
    } else {
      status = ZEN_TIMEOUT;
    }
    s_n[threadIdx.x] = n;
  }
  __syncthreads();
  return status;
}

// ---------------------------------------------------------------------------------------------
// K2: owner-side reduce of sources [src_begin, src_end).  One launch over all sources is the fast
// mode; one launch per source gives a fixed accumulation order.  The waits on the sources' mailboxes
// run side by side (one thread each); the sources' records are read side by side too (CTA b takes source b mod ns: one
// source after the other left three threads of four without a record), two per 16-byte load, four loads in flight.
#define K2_DENSE 4                                        // no bitmap with more than one record per this many slots
template <typename T, int NB>
__global__ void __launch_bounds__(256)
zen_owner_reduce_kernel(const __grid_constant__ ZenSparseBatch<NB> bt, int src_begin, int src_end, int allow_dense) {
  zen_pdl::enter();
  __shared__ ZenSparseCtx s_ctx;
  const ZenSparseCtx& c = zen_ctx(bt, s_ctx);
  __shared__ uint32_t s_n[ZEN_MAX_RANKS];
  const uint32_t epoch = zen_epoch(c);
  const int ns = src_end - src_begin;
  uint32_t local_status = records_wait(c, epoch, src_begin, src_end, s_n);
  // With many records the occupancy bitmap is not kept: the gather then reads every slot anyway and takes "touched" to mean
  // "sum is not zero" (a slot whose sum is exactly zero need not travel), which halves the number of atomics here.  At 24 % of
  // the slots reduce + gather take the same time both ways (16 M x 8 bf16: 126 us), at 20 % the scan costs 6 us of 33 more (4 M x 2
  // fp32).  The choice is published for the gather kernel of this call.
  uint64_t total = 0;
  for (int k = 0; k < ns; ++k) total += s_n[k];
  const bool dense_mode = allow_dense && total * (uint64_t)allow_dense > (uint64_t)c.nslots;
  if (blockIdx.x == 0 && threadIdx.x == 0) c.cursors[ZEN_MAX_RANKS + 3] = dense_mode ? 1u : 0u;
  const uint32_t nslots = c.nslots;
  float* acc = c.acc;
  uint32_t* bitmap = c.bitmap;
  auto apply = [&](uint32_t slot, uint32_t bits) {
    if (slot < nslots) {
      atomicAdd(&acc[slot], ZenVal<T>::unbits(bits));
      if (!dense_mode) atomicOr(&bitmap[slot >> 5], 1u << (slot & 31));
    } else {
      local_status |= ZEN_BAD_ARG;
    }
  };
  // the CTAs of source k: b = k, k + ns, ... (with fewer CTAs than sources, a CTA walks several)
  for (int k = blockIdx.x % ns; k < ns; k += gridDim.x) {
    const uint32_t rank_in = blockIdx.x / ns, nctas = max(1u, ((uint32_t)gridDim.x - k + ns - 1) / ns);
    const uint32_t n = s_n[k];
    const uint2* rec = zen_rec_slots(c, c.rank, src_begin + k, epoch);
    const uint4* rec4 = reinterpret_cast<const uint4*>(rec);
    const uint32_t npair = n >> 1, stride = nctas * 256u;
    for (uint32_t i = rank_in * 256u + threadIdx.x; i < npair; i += 4 * stride) {
      uint4 r[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t j = i + u * stride;
        r[u] = (j < npair) ? rec4[j] : make_uint4(0xffffffffu, 0u, 0xffffffffu, 0u);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (i + u * stride < npair) { apply(r[u].x, r[u].y); apply(r[u].z, r[u].w); }
      }
    }
    if ((n & 1u) && rank_in == 0 && threadIdx.x == 0) { const uint2 r = rec[n - 1]; apply(r.x, r.y); }
  }
  if (local_status) atomicOr(c.status, local_status);
}

// ---------------------------------------------------------------------------------------------
// K3: a warp takes one or two pairs of 1024-slot chunks per step (lane = 64 slots of a pair), compacts their touched slots in
// shared memory and pushes them as one run -- values, and COO slots or bitmap words, + the chunks' value offsets -- to every
// peer.  Room in this owner's payload is reserved per CTA step with one atomic (one per warp, 4096 on one address, made the
// kernel 30 % slower); chunks start on 8-value boundaries, so every push is a 16-byte vector store.  Chunks may land in the
// payload in any order: the consumer finds a chunk's values (and COO slots) through the chunk's offset.
//
// What bounds it: latency.  The chain is bitmap words -> slots -> push, a few round trips for a few hundred values per warp, so
// all slots of a warp are listed first (bit walks, no memory) and fetched eight at a time per lane, the reservation is made
// meanwhile, and the launcher sizes the steps so that one wave of CTAs takes them all.
#define K3_WARPS 8
#define K3_RUN_ALIGN 8u
#define K3_EMPTY 0xffffffffu                              // value offset of a chunk without values (COO)
#define K3_STAGE 1032                                     // staged entries per warp: one full chunk, rounded up to a whole run
#define K3_PPW 2                                          // pairs per warp and step at most
#define K3_LIST_MAX 1024u                                 // touched slots (padded) that are listed one by one at a time
__device__ __forceinline__ uint32_t k3_pad(uint32_t n) { return (n + K3_RUN_ALIGN - 1) & ~(K3_RUN_ALIGN - 1u); }

__device__ __forceinline__ void zen_multimem_st16(void* mc_addr, const uint4& v) {
  asm volatile("multimem.st.relaxed.sys.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(mc_addr), "f"(__uint_as_float(v.x)),
               "f"(__uint_as_float(v.y)), "f"(__uint_as_float(v.z)), "f"(__uint_as_float(v.w)) : "memory");
}
__device__ __forceinline__ void zen_multimem_st4(void* mc_addr, uint32_t v) {
  asm volatile("multimem.st.relaxed.sys.global.b32 [%0], %1;" ::"l"(mc_addr), "r"(v) : "memory");
}

// End of a gather: the last CTA of a rank publishes its payload to the consumers.
template <int NB>
__device__ __forceinline__ void publish_gather(const ZenSparseCtx& c, uint32_t fmt, uint32_t epoch, uint32_t& s_last) {
  const int tid = threadIdx.x;
  __syncthreads();
  if (tid == 0) {
    arrive_fence<NB>();
    const uint32_t prev = atomicAdd(&c.cursors[ZEN_MAX_RANKS + 1], 1u);
    s_last = (prev == gridDim.x - 1) ? 1u : 0u;
  }
  __syncthreads();
  if (s_last) {
    publish_fence<NB>();
    if (tid < c.nranks) {
      const uint32_t total = atomicAdd(&c.cursors[ZEN_MAX_RANKS + 2], 0u);
      const uint32_t st = atomicOr(c.status, 0u);
      const bool overflow = total > c.cap_g || (st & ZEN_GATHER_OVERFLOW);
      ZenMail* mail = reinterpret_cast<ZenMail*>(c.sym[tid] + c.off_g_mail) + c.rank;
      mail->count = overflow ? 0u : total;
      mail->info = ((overflow || (st & (ZEN_REC_OVERFLOW | ZEN_PEER_OVERFLOW | ZEN_TIMEOUT))) ? 1u : 0u) | (fmt << 8);
      mail->aux = 0;
      publish_epoch<NB>(&mail->epoch, epoch);
    }
    __syncthreads();
    if (tid == 0) { c.cursors[ZEN_MAX_RANKS + 1] = 0; c.cursors[ZEN_MAX_RANKS + 2] = 0; }
  }
}

template <typename T, int NB>
__global__ void __launch_bounds__(K3_WARPS * 32, sizeof(T) == 2 ? 4 : 3)
zen_gather_push_kernel(const __grid_constant__ ZenSparseBatch<NB> bt, int ppw) {
  zen_pdl::enter();
  __shared__ ZenSparseCtx s_ctx;
  const ZenSparseCtx& c = zen_ctx(bt, s_ctx);
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, hl = lane & 15, hf = lane >> 4;
  uint32_t* s_idx = reinterpret_cast<uint32_t*>(smem_raw) + warp * K3_STAGE;
  T* s_val = reinterpret_cast<T*>(smem_raw + K3_WARPS * K3_STAGE * 4) + warp * K3_STAGE;
  __shared__ uint32_t s_last, s_fmt, s_base, s_tot[2][K3_WARPS];
  const uint32_t epoch = zen_epoch(c);
  if (warp == 0) {
    // index format: bitmap when more than one slot in 32 is expected to be touched.  The estimate is the number of
    // records received (an upper bound of the union), which every CTA reads from the same mails.
    uint32_t fmt = c.fmt_mode;
    uint64_t recs = lane < c.nranks ? min(zen_rec_mail(c, c.rank, lane, epoch)->count, c.cap_rec) : 0u;
#pragma unroll
    for (int d = 4; d; d >>= 1) recs += __shfl_xor_sync(0xffffffffu, recs, d);   // lanes 0 .. 7 hold the sources
    if (fmt == 0) fmt = (recs * 32ull > (uint64_t)c.nslots) ? ZEN_FMT_BITMAP : ZEN_FMT_COO;
    // a COO list (touched slots plus the padding between runs) must fit the index region
    if (fmt == ZEN_FMT_COO && min(recs, (uint64_t)c.nslots) + K3_RUN_ALIGN * (uint64_t)c.nchunks > (uint64_t)c.g_idx_words) fmt = ZEN_FMT_BITMAP;
    if (lane == 0) s_fmt = fmt;
  }
  __syncthreads();
  const uint32_t fmt = s_fmt;
  constexpr uint32_t VPV = 16 / sizeof(T);                               // values per 16-byte vector
  uint32_t local_status = 0;
  char* mc = c.mc;
  const bool no_bitmap = c.cursors[ZEN_MAX_RANKS + 3] != 0u;            // the reduce kept no bitmap: touched = nonzero sum
  const uint32_t nchunks = c.nchunks, npairs = (nchunks + 1) >> 1, nwords = c.nwords;
  float* const acc = c.acc;
  uint32_t* const bitmap = c.bitmap;
  const int npeer = mc ? 1 : c.nranks;

  // the 64 slots of this lane in a pair: their bits (nwords is even: slots come in blocks of 64 and more)
  auto fetch = [&](uint32_t pair) -> uint2 {
    const uint32_t wi = pair * 64 + lane * 2;
    if (pair >= npairs) return make_uint2(0u, 0u);
    if (!no_bitmap) return wi < nwords ? *reinterpret_cast<const uint2*>(bitmap + wi) : make_uint2(0u, 0u);
    // one word per coalesced line of the slots; the words of this lane are 2 lane and 2 lane + 1
    uint32_t w[2] = {0u, 0u};
    const uint32_t at = pair * 2048 + lane, left = c.nslots - pair * 2048;
#pragma unroll 16
    for (int i = 0; i < 64; ++i) {
      const uint32_t v = (uint32_t)(i * 32 + lane) < left ? __float_as_uint(acc[at + i * 32]) : 0u;
      const uint32_t m = __ballot_sync(0xffffffffu, (v & 0x7fffffffu) != 0u);
      if (lane == (i >> 1)) w[i & 1] = m;
    }
    return make_uint2(w[0], w[1]);
  };
  // `n` staged entries (a multiple of the run alignment) to place `at` of the payload of every peer
  auto push = [&](uint32_t n, uint32_t at) {
    const uint32_t nvec = n / VPV, nvi = n / 4;
    const uint64_t val_off = c.off_g_val + (uint64_t)c.rank * c.cap_g * 4ull + (uint64_t)at * sizeof(T);
    const uint64_t idx_off = c.off_g_idx + ((uint64_t)c.rank * c.g_idx_words + at) * 4ull;
    const uint4* sv4 = reinterpret_cast<const uint4*>(s_val);
    const uint4* si4 = reinterpret_cast<const uint4*>(s_idx);
    if (mc) {                                                            // one store, replicated by the switch
      for (uint32_t i = lane; i < nvec; i += 32) zen_multimem_st16(mc + val_off + (uint64_t)i * 16, sv4[i]);
      if (fmt == ZEN_FMT_COO)
        for (uint32_t i = lane; i < nvi; i += 32) zen_multimem_st16(mc + idx_off + (uint64_t)i * 16, si4[i]);
    } else {
      for (uint32_t i = lane; i < nvec; i += 32) {
        const uint4 v = sv4[i];
        for (int p = 0; p < npeer; ++p) *reinterpret_cast<uint4*>(c.sym[p] + val_off + (uint64_t)i * 16) = v;
      }
      if (fmt == ZEN_FMT_COO) {
        for (uint32_t i = lane; i < nvi; i += 32) {
          const uint4 v = si4[i];
          for (int p = 0; p < npeer; ++p) *reinterpret_cast<uint4*>(c.sym[p] + idx_off + (uint64_t)i * 16) = v;
        }
      }
    }
  };

  const uint32_t spw = K3_WARPS * (uint32_t)ppw, nsteps = (npairs + spw - 1) / spw;
  uint32_t par = 0;
  for (uint32_t step = blockIdx.x; step < nsteps; step += gridDim.x, par ^= 1) {
    const uint32_t pair0 = step * spw + warp * ppw;
    uint2 word[K3_PPW];
    uint32_t first[K3_PPW], n_mine[K3_PPW], run[K3_PPW];                 // lane's first entry; touched slots and first entry of its half's chunk
#pragma unroll
    for (int j = 0; j < K3_PPW; ++j) word[j] = j < ppw ? fetch(pair0 + j) : make_uint2(0u, 0u);
    uint32_t total = 0;
#pragma unroll
    for (int j = 0; j < K3_PPW; ++j) {
      if (!no_bitmap && (word[j].x | word[j].y))
        *reinterpret_cast<uint2*>(bitmap + (pair0 + j) * 64 + lane * 2) = make_uint2(0u, 0u);   // clean for the next call
      const uint32_t own = __popc(word[j].x) + __popc(word[j].y);
      uint32_t incl = own;
#pragma unroll
      for (int d = 1; d < 16; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d, 16);
        if (hl >= d) incl += t;
      }
      n_mine[j] = __shfl_sync(0xffffffffu, incl, 15, 16);
      const uint32_t n_pad = k3_pad(n_mine[j]), n0 = __shfl_sync(0xffffffffu, n_pad, 0), n1 = __shfl_sync(0xffffffffu, n_pad, 16);
      run[j] = total + (hf ? n0 : 0u);
      first[j] = run[j] + incl - own;
      total += n0 + n1;
    }
    if (lane == 0) s_tot[par][warp] = total;
    __syncthreads();
    uint32_t base = (lane & 7) < K3_WARPS ? s_tot[par][lane & 7] : 0u;   // inclusive prefix over the warps, in every group of 8 lanes
#pragma unroll
    for (int d = 1; d < K3_WARPS; d <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, base, d, 8);
      if ((lane & 7) >= d) base += t;
    }
    const uint32_t cta_total = __shfl_sync(0xffffffffu, base, K3_WARPS - 1);
    base = __shfl_sync(0xffffffffu, base, warp) - total;
    if (tid == 0) s_base = cta_total ? atomicAdd(&c.cursors[ZEN_MAX_RANKS + 2], cta_total) : 0u;
    // slots of pairs [j0, j1), entries [e0, e0 + n) of the warp: listed (bit walks, no memory), then fetched and cleared
    auto collect = [&](int j0, int j1, uint32_t e0, uint32_t n) {
#pragma unroll
      for (int j = 0; j < K3_PPW; ++j) {
        if (j < j0 || j >= j1) continue;
        uint32_t r = first[j] - e0;
        const uint32_t slot0 = (pair0 + j) * 2048 + lane * 64;
        for (uint32_t w = word[j].x; w; w &= w - 1) s_idx[r++] = slot0 + __ffs(w) - 1;
        for (uint32_t w = word[j].y; w; w &= w - 1) s_idx[r++] = slot0 + __ffs(w) + 31;
        if ((uint32_t)hl < k3_pad(n_mine[j]) - n_mine[j]) s_idx[run[j] - e0 + n_mine[j] + hl] = 0xffffffffu;   // padding: skipped by the consumer
      }
      __syncwarp();
      for (uint32_t i0 = lane; i0 < n; i0 += 256) {
        uint32_t sl[8];
        float f[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) sl[u] = i0 + u * 32 < n ? s_idx[i0 + u * 32] : 0xffffffffu;
#pragma unroll
        for (int u = 0; u < 8; ++u) f[u] = sl[u] != 0xffffffffu ? acc[sl[u]] : 0.f;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          if (sl[u] != 0xffffffffu) acc[sl[u]] = 0.f;
          if (i0 + u * 32 < n) s_val[i0 + u * 32] = ZenVal<T>::from_f(f[u]);
        }
      }
    };
    const bool listed = total <= K3_LIST_MAX;
    if (listed) collect(0, K3_PPW, 0, total);
    __syncthreads();
    const uint32_t cta_base = s_base;
    const bool fits = cta_base + cta_total <= c.cap_g && (fmt != ZEN_FMT_COO || cta_base + cta_total <= c.g_idx_words);
    if (cta_total && !fits) local_status |= ZEN_GATHER_OVERFLOW;
    base += cta_base;
    if (listed) {
      __syncwarp();
      if (fits) push(total, base);
    } else {
#pragma unroll
      for (int j = 0; j < K3_PPW; ++j) {
        if (j >= ppw) continue;
        const uint32_t e0 = __shfl_sync(0xffffffffu, run[j], 0), e1 = __shfl_sync(0xffffffffu, run[j] + k3_pad(n_mine[j]), 16);
        if (e1 - e0 <= K3_LIST_MAX) {                                    // one pair at a time fits
          collect(j, j + 1, e0, e1 - e0);
          __syncwarp();
          if (fits) push(e1 - e0, base + e0);
          __syncwarp();                                                  // the staging area is free again
          continue;
        }
        // most slots: chunk by chunk, all slots streamed as vectors of four, four of them in flight per lane
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          const uint32_t n = __shfl_sync(0xffffffffu, n_mine[j], h * 16), run0 = __shfl_sync(0xffffffffu, run[j], h * 16);
          if (n == 0) continue;
          const uint32_t chunk0 = ((pair0 + j) * 2 + h) * 1024;
#pragma unroll 1
          for (int q0 = 0; q0 < 8; q0 += 4) {
            float4 v[4];
            uint32_t nib[4], at[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int wq = (q0 + q) * 4 + (lane >> 3), src = h * 16 + (wq >> 1);   // the lane's word of the chunk, and who holds it
              const uint32_t wx = __shfl_sync(0xffffffffu, word[j].x, src), wy = __shfl_sync(0xffffffffu, word[j].y, src);
              at[q] = __shfl_sync(0xffffffffu, first[j] - run0, src) + ((wq & 1) ? __popc(wx) : 0);
              const uint32_t w = (wq & 1) ? wy : wx, sh = (lane & 7) * 4;
              nib[q] = (w >> sh) & 15u;
              at[q] += __popc(w & ((1u << sh) - 1u));
              v[q] = nib[q] ? *reinterpret_cast<const float4*>(acc + chunk0 + (q0 + q) * 128 + lane * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              if (!nib[q]) continue;
              const uint32_t slot = chunk0 + (q0 + q) * 128 + lane * 4;
              *reinterpret_cast<float4*>(acc + slot) = make_float4(0.f, 0.f, 0.f, 0.f);
              const float f[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
              uint32_t r = at[q];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                if ((nib[q] >> i) & 1u) {
                  s_val[r] = ZenVal<T>::from_f(f[i]);
                  if (fmt == ZEN_FMT_COO) s_idx[r] = slot + i;
                  ++r;
                }
              }
            }
          }
          if (fmt == ZEN_FMT_COO && (uint32_t)lane < k3_pad(n) - n) s_idx[n + lane] = 0xffffffffu;
          __syncwarp();
          if (fits) push(k3_pad(n), base + run0);
          __syncwarp();                                                  // the staging area is free again
        }
      }
    }
    if (fits) {
      // bitmap words, and where each chunk's values begin
#pragma unroll
      for (int j = 0; j < K3_PPW; ++j) {
        if (j >= ppw) continue;
        const uint32_t wi = (pair0 + j) * 64 + lane * 2, my_ch = (pair0 + j) * 2 + hf;
        const uint32_t at = (fmt == ZEN_FMT_COO && n_mine[j] == 0) ? K3_EMPTY : base + run[j];
        const uint64_t bm = c.off_g_idx + ((uint64_t)c.rank * c.g_idx_words + wi) * 4ull;
        const uint64_t of = c.off_g_off + ((uint64_t)c.rank * (nchunks + 1) + my_ch) * 4ull;
        const bool words = fmt != ZEN_FMT_COO && wi < nwords, offset = hl == 0 && my_ch < nchunks;
        if (mc) {
          if (words) { zen_multimem_st4(mc + bm, word[j].x); zen_multimem_st4(mc + bm + 4, word[j].y); }
          if (offset) zen_multimem_st4(mc + of, at);
        } else {
          for (int p = 0; p < npeer; ++p) {
            if (words) *reinterpret_cast<uint2*>(c.sym[p] + bm) = word[j];
            if (offset) *reinterpret_cast<uint32_t*>(c.sym[p] + of) = at;
          }
        }
      }
    }
    __syncwarp();                                                        // the staging area is free again
  }

  if (local_status) atomicOr(c.status, local_status);
  publish_gather<NB>(c, fmt, epoch, s_last);
}

// ---------------------------------------------------------------------------------------------
// K2b + K3b: the owner's sums in shared memory.  The slot space of an owner is cut into buckets of 16 384 slots (32 768 from
// 2^24 slots on); one CTA adds up all records of a bucket in shared memory and gathers and pushes from there, so neither sums nor
// occupancy bitmap exist in global memory.  For that the records of a bucket have to be found:
//   * few records: every CTA reads all of its owner's records and keeps its bucket's (no kernel before K3b at all);
//   * else K2b sorts them by bucket first, tile by tile (4096 records of one source) and in place, and notes where the
//     bucket's run of each tile begins and ends: seg[bucket][tile].
//
// What bounds K2 + K3, which this replaces: the scattered atomics of K2, two a record, 38 per clock over the whole GPU however
// they are arranged, and in K3 the round trips from bitmap to slots to push.  Here a record costs one more trip through L2
// (K2b) and one shared-memory atomic; what is left is the chain of a bucket (words, records, adds, count, reservation, push), about
// 10 us with 24 warps to an SM, of which the stores to eight peers are a quarter.  us, K2 + K3 / K2b + K3b: 8 ranks of 2^26 bf16
// elements at 1 % 170 + 121 / 34 + 100, 4 of 13 M 20 + 20 / 7 + 19, 2 of 50 000 (fp32) 4 + 11 / 0 + 8.
// (Tried: one CTA per bucket, not persistent, 120 us for the first; the next bucket's runs fetched ahead 195, in spills and waits.)
// K2 and K3 remain for owners of more than 2^25 slots, whose tiles would leave less than four records to a run, and for calls of
// less than one bucket over all owners, which the host's side bounds (3 x 10 000: 26 us as four
// kernels, 25 to 28 in buckets).
#define SB_MIN_SLOTS (1u << 14)
#define SB_TILE 4096
#define SB_MAX_BUCKETS 1024
#define SB_SORT_THREADS 512
#define SB_WINDOW 512                                     // list entries per warp
#define SB_FILTER_RECORDS 65536                           // most record slots of an owner that every CTA reads for itself

struct SbShape { uint32_t lg, nbuckets, tiles, lg_lanes; bool on, sorted; };      // tiles: per source; lanes to a run
__host__ __device__ __forceinline__ SbShape sb_shape(uint32_t nslots, uint32_t cap_rec, int nranks) {
  SbShape s;
  s.lg = nslots <= (SB_MAX_BUCKETS << 14) ? 14u : 15u;
  s.nbuckets = (nslots + (1u << s.lg) - 1) >> s.lg;
  s.tiles = (cap_rec + SB_TILE - 1) / SB_TILE;
  s.lg_lanes = s.nbuckets > 384 ? 3u : s.nbuckets > 160 ? 4u : 5u;      // a full tile's runs: 4096 / buckets records
  s.on = s.nbuckets <= SB_MAX_BUCKETS && (uint64_t)nslots * nranks >= SB_MIN_SLOTS;
  s.sorted = s.nbuckets > 1 && (uint64_t)cap_rec * nranks > SB_FILTER_RECORDS;
  return s;
}

template <int NB>
__global__ void __launch_bounds__(SB_SORT_THREADS, 2)
zen_record_sort_kernel(const __grid_constant__ ZenSparseBatch<NB> bt, int deterministic, int by_index) {
  zen_pdl::enter();
  __shared__ ZenSparseCtx s_ctx;
  const ZenSparseCtx& c = zen_ctx(bt, s_ctx);
  __shared__ uint32_t s_n[ZEN_MAX_RANKS];
  __shared__ uint32_t hist[SB_MAX_BUCKETS + 1], s_warp[SB_SORT_THREADS / 32];
  __shared__ __align__(16) uint2 sorted[SB_TILE];
  const uint32_t epoch = zen_epoch(c);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t local_status = records_wait(c, epoch, 0, c.nranks, s_n);
  if (blockIdx.x == 0 && tid == 0) c.cursors[ZEN_MAX_RANKS + 3] = deterministic ? 2u : 0u;     // for a K3b that is launched without being told
  const uint32_t nslots = by_index ? (uint32_t)c.numel : c.nslots;       // method 1: records carry element indices
  const SbShape sh = sb_shape(nslots, c.cap_rec, c.nranks);
  if (sh.on && sh.sorted) {
    const uint32_t nb = sh.nbuckets, stride = sh.tiles * c.nranks;
    uint32_t* seg = c.seg;
    for (uint32_t t = blockIdx.x; t < stride; t += gridDim.x) {
      const uint32_t src = t / sh.tiles, first = (t - src * sh.tiles) * SB_TILE;
      if (first >= s_n[src]) continue;
      const uint32_t n = min((uint32_t)SB_TILE, s_n[src] - first);
      uint2* rec = zen_rec_slots(c, c.rank, src, epoch) + first;
      for (uint32_t b = tid; b <= nb; b += SB_SORT_THREADS) hist[b] = 0;
      constexpr int PAIRS = SB_TILE / 2 / SB_SORT_THREADS;
      uint4 r[PAIRS];
#pragma unroll
      for (int u = 0; u < PAIRS; ++u) {
        const uint32_t i = (uint32_t)(u * SB_SORT_THREADS + tid) * 2;
        r[u] = i + 1 < n ? reinterpret_cast<const uint4*>(rec)[i / 2] : make_uint4(0xffffffffu, 0u, 0xffffffffu, 0u);
        if (i + 1 == n) { const uint2 x = rec[i]; r[u].x = x.x; r[u].y = x.y; }
      }
      __syncthreads();
      // a slot that does not exist goes to the bucket after the last, which nobody reads
      uint32_t at[2 * PAIRS];
      auto bucket = [&](uint32_t slot) { return slot < nslots ? slot >> sh.lg : nb; };
#pragma unroll
      for (int u = 0; u < PAIRS; ++u) {
        const uint32_t i = (uint32_t)(u * SB_SORT_THREADS + tid) * 2;
        if (i < n) { at[2 * u] = atomicAdd(&hist[bucket(r[u].x)], 1u); if (r[u].x >= nslots) local_status |= ZEN_BAD_ARG; }
        if (i + 1 < n) { at[2 * u + 1] = atomicAdd(&hist[bucket(r[u].z)], 1u); if (r[u].z >= nslots) local_status |= ZEN_BAD_ARG; }
      }
      __syncthreads();
      // exclusive prefix sums over the buckets, two per thread
      const uint32_t b0 = tid * 2, h0 = b0 < nb ? hist[b0] : 0u, h1 = b0 + 1 < nb ? hist[b0 + 1] : 0u;
      uint32_t incl = h0 + h1;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += x;
      }
      if (lane == 31) s_warp[warp] = incl;
      __syncthreads();
      uint32_t before = 0;
#pragma unroll
      for (int k = 0; k < SB_SORT_THREADS / 32; ++k) before += k < warp ? s_warp[k] : 0u;
      const uint32_t e0 = before + incl - h0 - h1, e1 = e0 + h0;
      if (b0 < nb) { hist[b0] = e0; seg[(size_t)b0 * stride + t] = e0 | h0 << 16; }
      if (b0 + 1 < nb) { hist[b0 + 1] = e1; seg[(size_t)(b0 + 1) * stride + t] = e1 | h1 << 16; }
      if (tid == SB_SORT_THREADS - 1) hist[nb] = e1 + h1;
      __syncthreads();
#pragma unroll
      for (int u = 0; u < PAIRS; ++u) {
        const uint32_t i = (uint32_t)(u * SB_SORT_THREADS + tid) * 2;
        if (i < n) sorted[hist[bucket(r[u].x)] + at[2 * u]] = make_uint2(r[u].x, r[u].y);
        if (i + 1 < n) sorted[hist[bucket(r[u].z)] + at[2 * u + 1]] = make_uint2(r[u].z, r[u].w);
      }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < PAIRS; ++u) {
        const uint32_t i = (uint32_t)(u * SB_SORT_THREADS + tid) * 2;
        if (i + 1 < n) reinterpret_cast<uint4*>(rec)[i / 2] = *reinterpret_cast<const uint4*>(&sorted[i]);
        else if (i < n) rec[i] = sorted[i];
      }
      __syncthreads();                                     // hist and the tile are free
    }
  }
  if (local_status) atomicOr(c.status, local_status);
}

template <int W> constexpr size_t sb_smem() { return (size_t)W * (2048 * 4 + 256 + SB_WINDOW * 2); }

// The records of one bucket from sources [s_lo, s_hi), each handed to apply(slot, value bits).
template <int W, typename Apply>
__device__ __forceinline__ void sb_records(const ZenSparseCtx& c, const SbShape& sh, uint32_t nslots, uint32_t bucket, int s_lo, int s_hi,
                                           const uint32_t* s_n, uint32_t epoch, uint32_t& status, Apply apply) {
  const int tid = threadIdx.x, lane = tid & 31;
  if (!sh.sorted) {
    for (int s = s_lo; s < s_hi; ++s) {
      const uint2* rec = zen_rec_slots(c, c.rank, s, epoch);
      const uint32_t n = s_n[s], npair = (n + 1) >> 1;
      for (uint32_t i = tid; i < npair; i += 4 * W * 32) {
        uint4 r[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint32_t j = i + u * W * 32;
          r[u] = j < npair ? reinterpret_cast<const uint4*>(rec)[j] : make_uint4(0u, 0u, 0u, 0u);   // cap_rec is even
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint32_t j = (i + u * W * 32) * 2;
          if (j < n) {
            if (r[u].x >= nslots) status |= ZEN_BAD_ARG;
            else if ((r[u].x >> sh.lg) == bucket) apply(r[u].x, r[u].y);
          }
          if (j + 1 < n) {
            if (r[u].z >= nslots) status |= ZEN_BAD_ARG;
            else if ((r[u].z >> sh.lg) == bucket) apply(r[u].z, r[u].w);
          }
        }
      }
    }
  } else {
    // 8, 16 or 32 lanes to a run, at least half of what a full tile's runs hold; a group stays with one source and has U runs, two
    // records of each per lane, under way together: words, then records, two trips to L2 for most buckets
    constexpr int U = 6;
    const uint32_t* seg = c.seg + (size_t)bucket * (sh.tiles * c.nranks);
    const uint2* rec0 = zen_rec_slots(c, c.rank, 0, epoch);
    const uint32_t lanes = 1u << sh.lg_lanes, l = lane & (lanes - 1u), group = tid >> sh.lg_lanes, ns = s_hi - s_lo;
    const uint32_t per_src = ((W * 32u) >> sh.lg_lanes) / ns, k0 = group / ns, src = s_lo + group - k0 * ns;
    const uint32_t rec_end = c.cap_rec * (uint32_t)c.nranks, ntiles = k0 < per_src ? (s_n[src] + SB_TILE - 1) / SB_TILE : 0u;
    for (uint32_t k = k0; k < ntiles; k += U * per_src) {
      uint32_t n[U], at[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t t = k + u * per_src;
        n[u] = t < ntiles ? seg[src * sh.tiles + t] : 0u;
        at[u] = src * c.cap_rec + t * SB_TILE;
      }
      uint2 x[U], y[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t first = n[u] & 0xffffu;
        n[u] >>= 16;
        at[u] += first;
        // (K2b may have given up its wait for a source and left another call's runs: kept inside the tile and the region)
        if (first + n[u] > SB_TILE || at[u] + n[u] > rec_end) n[u] = 0;
        if (l < n[u]) x[u] = rec0[at[u] + l];
        if (l + lanes < n[u]) y[u] = rec0[at[u] + l + lanes];
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (l < n[u]) apply(x[u].x, x[u].y);
        if (l + lanes < n[u]) apply(y[u].x, y[u].y);
        for (uint32_t i = l + 2 * lanes; i < n[u]; i += 4 * lanes) {   // long runs
          uint2 z[4];
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (i + q * lanes < n[u]) z[q] = rec0[at[u] + i + q * lanes];
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (i + q * lanes < n[u]) apply(z[q].x, z[q].y);
        }
      }
    }
  }
}

// det: 1 rank order, 0 any order, -1 as K2b left it
template <typename T, int W, int NB>
__global__ void __launch_bounds__(W * 32, W == 8 ? 3 : 1)
zen_reduce_gather_kernel(const __grid_constant__ ZenSparseBatch<NB> bt, int det) {
  zen_pdl::enter();
  __shared__ ZenSparseCtx s_ctx;
  const ZenSparseCtx& c = zen_ctx(bt, s_ctx);
  extern __shared__ __align__(128) unsigned char smem_raw[];
  constexpr uint32_t BS = W * 2048;
  float* acc = reinterpret_cast<float*>(smem_raw);                       // [BS]
  uint32_t* bm = reinterpret_cast<uint32_t*>(acc + BS);                  // [BS / 32]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, hl = lane & 15, hf = lane >> 4;
  unsigned short* list = reinterpret_cast<unsigned short*>(bm + BS / 32) + warp * SB_WINDOW;    // pair-local slots
  __shared__ uint32_t s_n[ZEN_MAX_RANKS], s_last, s_fmt, s_base, s_tot[W];
  const uint32_t epoch = zen_epoch(c);
  const SbShape sh = sb_shape(c.nslots, c.cap_rec, c.nranks);
  for (uint32_t i = tid; i < (BS + BS / 32) / 4; i += W * 32) reinterpret_cast<uint4*>(smem_raw)[i] = make_uint4(0u, 0u, 0u, 0u);
  uint32_t local_status = records_wait(c, epoch, 0, c.nranks, s_n);
  uint64_t recs = 0;
  for (int k = 0; k < c.nranks; ++k) recs += s_n[k];
  // With many records the occupancy bitmap is not kept while they are added up: "touched" then means "sum is not zero" (a slot
  // whose sum is exactly zero need not travel).
  const bool dense_mode = recs * K2_DENSE > (uint64_t)c.nslots;
  if (tid == 0) {
    // index format: bitmap when more than one slot in 32 is expected to be touched; the estimate is the number of records
    // received (an upper bound of the union), which every CTA reads from the same mails
    uint32_t fmt = c.fmt_mode;
    if (fmt == 0) fmt = (recs * 32ull > (uint64_t)c.nslots) ? ZEN_FMT_BITMAP : ZEN_FMT_COO;
    // a COO list (touched slots plus the padding between runs) must fit the index region
    if (fmt == ZEN_FMT_COO && min(recs, (uint64_t)c.nslots) + K3_RUN_ALIGN * (uint64_t)c.nchunks > (uint64_t)c.g_idx_words) fmt = ZEN_FMT_BITMAP;
    s_fmt = fmt;
  }
  const bool in_order = det < 0 ? c.cursors[ZEN_MAX_RANKS + 3] == 2u : det != 0;
  __syncthreads();
  auto apply = [&](uint32_t slot, uint32_t bits) {                       // a slot of this bucket
    const uint32_t at = slot & (BS - 1);
    atomicAdd(&acc[at], ZenVal<T>::unbits(bits));
    if (!dense_mode) atomicOr(&bm[at >> 5], 1u << (at & 31));
  };
  const uint32_t fmt = s_fmt, nchunks = c.nchunks, nwords = c.nwords;
  char* const mc = c.mc;
  const int npeer = mc ? 1 : c.nranks;
  constexpr uint32_t VPV = 16 / sizeof(T);                               // values per 16-byte vector
  float* const pacc = acc + warp * 2048;                                 // gather: warp = one pair of chunks, lane = 64 of its slots
  for (uint32_t bucket = blockIdx.x; bucket < sh.nbuckets; bucket += gridDim.x) {
    for (int s_lo = 0; s_lo < c.nranks;) {
      const int s_hi = in_order ? s_lo + 1 : c.nranks;
      sb_records<W>(c, sh, c.nslots, bucket, s_lo, s_hi, s_n, epoch, local_status, apply);
      __syncthreads();                                                     // in order: the next source's adds come after these
      s_lo = s_hi;
    }

    const uint32_t pair = bucket * W + warp;
    uint2 word;
    if (!dense_mode) {
      uint2* at = reinterpret_cast<uint2*>(bm + warp * 64 + lane * 2);
      word = *at;
      *at = make_uint2(0u, 0u);
    } else {
      uint32_t w[2] = {0u, 0u};
#pragma unroll 16
      for (int i = 0; i < 64; ++i) {
        const uint32_t m = __ballot_sync(0xffffffffu, (__float_as_uint(pacc[i * 32 + lane]) & 0x7fffffffu) != 0u);
        if (lane == (i >> 1)) w[i & 1] = m;
      }
      word = make_uint2(w[0], w[1]);
    }
    const uint32_t own = __popc(word.x) + __popc(word.y);
    uint32_t incl = own;
#pragma unroll
    for (int d = 1; d < 16; d <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d, 16);
      if (hl >= d) incl += t;
    }
    const uint32_t n_mine = __shfl_sync(0xffffffffu, incl, 15, 16), n_pad = k3_pad(n_mine);
    const uint32_t n0 = __shfl_sync(0xffffffffu, n_pad, 0), total = n0 + __shfl_sync(0xffffffffu, n_pad, 16);
    const uint32_t run0 = hf ? n0 : 0u, first = run0 + incl - own;         // the half's first entry, and the lane's
    if (lane == 0) s_tot[warp] = total;
    __syncthreads();
    uint32_t base = 0, cta_total = 0;
#pragma unroll
    for (int k = 0; k < W; ++k) { const uint32_t x = s_tot[k]; base += k < warp ? x : 0u; cta_total += x; }
    if (tid == 0) s_base = cta_total ? atomicAdd(&c.cursors[ZEN_MAX_RANKS + 2], cta_total) : 0u;
    __syncthreads();
    const uint32_t cta_base = s_base;
    const bool fits = cta_base + cta_total <= c.cap_g && (fmt != ZEN_FMT_COO || cta_base + cta_total <= c.g_idx_words);
    if (!fits) {
      if (cta_total) local_status |= ZEN_GATHER_OVERFLOW;
      for (int i = lane; i < 512; i += 32) reinterpret_cast<float4*>(pacc)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    base += cta_base;
    if (fits) {
      for (uint32_t e0 = 0; e0 < total; e0 += SB_WINDOW) {                 // a window of the warp's entries at a time
        const uint32_t n = min((uint32_t)SB_WINDOW, total - e0);
        if (first < e0 + n && first + own > e0) {
          uint32_t r = first - e0;                                         // wraps below the window: not stored
          for (uint32_t w = word.x; w; w &= w - 1, ++r) if (r < n) list[r] = (unsigned short)(lane * 64 + __ffs(w) - 1);
          for (uint32_t w = word.y; w; w &= w - 1, ++r) if (r < n) list[r] = (unsigned short)(lane * 64 + __ffs(w) + 31);
        }
        const uint32_t pad = run0 + n_mine + hl - e0;
        if ((uint32_t)hl < n_pad - n_mine && pad < n) list[pad] = 0xffffu; // padding: skipped by the consumer
        __syncwarp();
        const uint64_t val_off = c.off_g_val + (uint64_t)c.rank * c.cap_g * 4ull + (uint64_t)(base + e0) * sizeof(T);
        for (uint32_t i = lane; i < n / VPV; i += 32) {
          uint32_t bits[VPV];
#pragma unroll
          for (int q = 0; q < (int)VPV; q += 4) {
            const uint2 l4 = *reinterpret_cast<const uint2*>(list + i * VPV + q);
            const uint32_t at[4] = {l4.x & 0xffffu, l4.x >> 16, l4.y & 0xffffu, l4.y >> 16};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              bits[q + k] = 0u;
              if (at[k] == 0xffffu) continue;
              bits[q + k] = ZenVal<T>::bits(ZenVal<T>::from_f(pacc[at[k]]));
              pacc[at[k]] = 0.f;                                           // clean for the next bucket
            }
          }
          uint4 v;
          if constexpr (VPV == 4) v = make_uint4(bits[0], bits[1], bits[2], bits[3]);
          else v = make_uint4(bits[0] | bits[1] << 16, bits[2] | bits[3] << 16, bits[VPV - 4] | bits[VPV - 3] << 16, bits[VPV - 2] | bits[VPV - 1] << 16);
          if (mc) zen_multimem_st16(mc + val_off + (uint64_t)i * 16, v);   // one store, replicated by the switch
          else
            for (int p = 0; p < npeer; ++p) *reinterpret_cast<uint4*>(c.sym[p] + val_off + (uint64_t)i * 16) = v;
        }
        if (fmt == ZEN_FMT_COO) {
          const uint64_t idx_off = c.off_g_idx + ((uint64_t)c.rank * c.g_idx_words + base + e0) * 4ull;
          for (uint32_t i = lane; i < n / 4; i += 32) {
            uint32_t sl[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) { const uint32_t at = list[i * 4 + q]; sl[q] = at != 0xffffu ? pair * 2048 + at : 0xffffffffu; }
            const uint4 v = make_uint4(sl[0], sl[1], sl[2], sl[3]);
            if (mc) zen_multimem_st16(mc + idx_off + (uint64_t)i * 16, v);
            else
              for (int p = 0; p < npeer; ++p) *reinterpret_cast<uint4*>(c.sym[p] + idx_off + (uint64_t)i * 16) = v;
          }
        }
        __syncwarp();                                                      // the list is free again
      }
      // bitmap words, and where each chunk's values begin
      const uint32_t wi = pair * 64 + lane * 2, my_ch = pair * 2 + hf;
      const uint32_t at = (fmt == ZEN_FMT_COO && n_mine == 0) ? K3_EMPTY : base + run0;
      const uint64_t bmo = c.off_g_idx + ((uint64_t)c.rank * c.g_idx_words + wi) * 4ull;
      const uint64_t ofo = c.off_g_off + ((uint64_t)c.rank * (nchunks + 1) + my_ch) * 4ull;
      const bool words = fmt != ZEN_FMT_COO && wi < nwords, offset = hl == 0 && my_ch < nchunks;
      if (mc) {
        if (words) { zen_multimem_st4(mc + bmo, word.x); zen_multimem_st4(mc + bmo + 4, word.y); }
        if (offset) zen_multimem_st4(mc + ofo, at);
      } else {
        for (int p = 0; p < npeer; ++p) {
          if (words) *reinterpret_cast<uint2*>(c.sym[p] + bmo) = word;
          if (offset) *reinterpret_cast<uint32_t*>(c.sym[p] + ofo) = at;
        }
      }
    }
    __syncthreads();                                                     // sums and bitmap are clean
  }

  if (local_status) atomicOr(c.status, local_status);
  publish_gather<NB>(c, fmt, epoch, s_last);
}

// ---------------------------------------------------------------------------------------------
// K4: densify.  Walks every owner's slot space two chunks at a time (2048 slots, one 64-slot block per lane); every output
// element is written once (zeros included), so the output needs no memset.  A chunk's COO list (slots in order, padding at its
// end) is turned into the chunk's bitmap words, so both formats take the same path.
//
// A warp works on three of its chunk pairs at a time: the bitmap words and the value offsets of the one after next are being
// fetched, the values of the next one travel to shared memory with 16-byte asynchronous copies, and the current one is
// assembled in shared memory (zeros, then the values at their slots) and written with full 16-byte vectors: the memory system
// sees whole lines, however few or many values there are.  What bounds it now is where the lines go: for eight ranks of 2^26 bf16
// elements at 1 % it takes 300 us (164 us of memory time), of which plain stores of 128-byte blocks in the same places take 235.
// Before, instruction issue did: with one chunk at a time (lane = 32 slots) a chunk took 383 instructions per warp, 312 us; with
// two, the prefix sum, the walk of the permutation and the bookkeeping are shared and every lane finds the output place of its
// own block.
#define K4_WARPS 8
#define K4_VCAP 256                                       // values of a chunk that are staged; with more, the pair is read in place
template <typename T>
struct K4Smem {
  uint4 tile[2048 * sizeof(T) / 16];                      // the pair's elements
  T vals[2][2][K4_VCAP];                                  // read up to 32 past a chunk's last value: `words` follows
  uint32_t words[64];                                     // bitmap words rebuilt from COO lists
};

template <typename T, int NB>
__global__ void __launch_bounds__(K4_WARPS * 32, sizeof(T) == 2 ? 4 : 2)
zen_densify_kernel(const __grid_constant__ ZenSparseBatch<NB> bt) {
  zen_pdl::enter();
  __shared__ ZenSparseCtx s_ctx;
  const ZenSparseCtx& c = zen_ctx(bt, s_ctx);
  T* __restrict__ out = reinterpret_cast<T*>(bt.out[NB > 1 ? blockIdx.y : 0]);
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ uint32_t s_fmt[ZEN_MAX_RANKS], s_cnt[ZEN_MAX_RANKS];
  const int tid = threadIdx.x, lane = tid & 31, hl = lane & 15, hf = lane >> 4;
  K4Smem<T>& sm = reinterpret_cast<K4Smem<T>*>(smem_raw)[tid >> 5];
  const uint32_t epoch = zen_epoch(c);
  uint32_t local_status = 0;
  if (tid < c.nranks) {
    const ZenMail* mail = reinterpret_cast<const ZenMail*>(c.sym[c.rank] + c.off_g_mail) + tid;
    uint32_t f = 0;
    if (zen_wait_epoch(&mail->epoch, epoch, c.wait_ns)) {
      const uint32_t info = zen_ld_acquire_sys(&mail->info);
      f = (info >> 8) & 0xffu;
      if (info & 1u) { local_status |= ZEN_PEER_OVERFLOW; f = 0; }
      s_cnt[tid] = min(zen_ld_acquire_sys(&mail->count), min(c.cap_g, c.g_idx_words));     // COO entries
    } else {
      local_status |= ZEN_TIMEOUT;
    }
    s_fmt[tid] = f;
  }
  __syncthreads();
  const uint64_t N = c.numel;
  const uint32_t gw = (blockIdx.x * blockDim.x + tid) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  const uint32_t nchunks = c.nchunks, npairs = (nchunks + 1) >> 1, nranks = (uint32_t)c.nranks, nunits = nranks * npairs;
  const uint32_t nblk = c.nslots >> 6, lg6 = c.perm.lg - 6;
  const char* base = c.sym[c.rank];
  const uint32_t* gidx = reinterpret_cast<const uint32_t*>(base + c.off_g_idx);
  const uint32_t* goff = reinterpret_cast<const uint32_t*>(base + c.off_g_off);
  const char* gval = base + c.off_g_val;
  const uint32_t stride_o = nw / npairs, stride_p = nw % npairs;
  // units are (owner, pair of chunks) walked with a fixed stride, advanced without divisions.  off, n and at (this lane's first
  // value, counted from off) belong to the lane's chunk: the first one's for lanes 0 - 15, the second one's for 16 - 31.
  struct Unit { uint32_t o, pr, w0, w1, off, n, at; };
  auto fetch = [&](Unit& u) {                             // issue the loads of a unit's index
    u.w0 = u.w1 = 0; u.off = K3_EMPTY;
    if (u.o >= nranks) return;
    const uint32_t f = s_fmt[u.o], ch = u.pr * 2 + hf;
    if (f == 0u || ch >= nchunks) return;
    u.off = goff[(size_t)u.o * (nchunks + 1) + ch];
    const uint32_t wi = u.pr * 64 + lane * 2;             // nwords is even: the slots come in blocks of 64 and more
    if (f == ZEN_FMT_BITMAP && wi < c.nwords) {
      const uint2 w = *reinterpret_cast<const uint2*>(gidx + (size_t)u.o * c.g_idx_words + wi);
      u.w0 = w.x; u.w1 = w.y;
    }
  };
  auto after = [&](const Unit& u) {
    Unit v;
    v.o = u.o + stride_o; v.pr = u.pr + stride_p;
    if (v.pr >= npairs) { v.pr -= npairs; ++v.o; }
    return v;
  };
  auto values_of = [&](const Unit& u) { return reinterpret_cast<const T*>(gval + (uint64_t)u.o * c.cap_g * 4ull) + u.off; };
  // where the chunks' values lie, and the copies of them into staging buffer `b`
  auto stage = [&](Unit& u, int b) {
    u.n = 0; u.at = 0;
    if (u.o < nranks) {
      if (s_fmt[u.o] == ZEN_FMT_COO) {
        const uint32_t* gi = gidx + (size_t)u.o * c.g_idx_words;
        const uint32_t total = s_cnt[u.o], ch = u.pr * 2 + hf;
        sm.words[lane] = 0; sm.words[32 + lane] = 0;
        __syncwarp();
        bool go = u.off != K3_EMPTY;
        for (uint32_t k = u.off; __any_sync(0xffffffffu, go); k += 16) {   // a run ends at padding, another chunk's slots or the list's end
          const uint32_t slot = (go && k < total && hl < total - k) ? gi[k + hl] : K3_EMPTY;
          const bool in = (slot >> 10) == ch;
          if (in) atomicOr(&sm.words[(slot >> 5) & 63u], 1u << (slot & 31u));
          go = __shfl_sync(0xffffffffu, in, hf * 16 + 15);
        }
        __syncwarp();
        u.w0 = sm.words[lane * 2]; u.w1 = sm.words[lane * 2 + 1];
        __syncwarp();
      }
      uint32_t incl = __popc(u.w0) + __popc(u.w1);
      const uint32_t own = incl;
#pragma unroll
      for (int d = 1; d < 16; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d, 16);
        if (hl >= d) incl += t;
      }
      u.n = __shfl_sync(0xffffffffu, incl, 15, 16);
      u.at = incl - own;
      if (u.off == K3_EMPTY || (uint64_t)u.off + u.n > c.cap_g) { u.n = 0; u.w0 = u.w1 = 0; }
      if (u.n <= K4_VCAP) {
        const char* src = reinterpret_cast<const char*>(values_of(u));
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&sm.vals[b][hf][0]), bytes = u.n * (uint32_t)sizeof(T);
        for (uint32_t i = hl * 16; i < bytes; i += 256)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i), "l"(src + i) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  Unit cur, nxt;
  cur.o = gw / npairs; cur.pr = gw % npairs;
  fetch(cur);
  nxt = after(cur);
  fetch(nxt);
  stage(cur, 0);
  constexpr int NV = 2048 * sizeof(T) / 16 / 32;          // 16-byte vectors per lane in the tile (8 or 16)
  constexpr int VPB = 64 * sizeof(T) / 16;                // vectors per block (8 or 16)
  constexpr int EPV = 16 / sizeof(T);                     // elements per vector
  uint32_t it = 0;
  for (uint32_t unit = gw; unit < nunits; unit += nw, ++it) {
    Unit nn = after(nxt);
    fetch(nn);
    stage(nxt, (it + 1) & 1);
    // where this lane's block lives in the output, in units of 64 elements
    uint32_t blk = 0xffffffffu;
    const uint32_t sblk = cur.pr * 32 + lane;
    if (sblk < nblk) {
      blk = (zen_perm_inv(c.perm, cur.o * c.perm.sb + (sblk >> lg6)) << lg6) + (sblk & ((1u << lg6) - 1u));
      if ((uint64_t)blk * 64 >= N) blk = 0xffffffffu;
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");  // the current pair's values
    if (__any_sync(0xffffffffu, cur.n > K4_VCAP)) {
      // Many values: block by block, two slots per lane, straight from the payload to the output, eight values in flight per
      // lane (bit by bit through the tile, each read in place, 8 M x 8 bf16 with 80 % of the slots took 185 us).
      const T* vals = reinterpret_cast<const T*>(gval + (uint64_t)cur.o * c.cap_g * 4ull);
      const uint32_t at0 = cur.off + cur.at;
#pragma unroll 1
      for (int b0 = 0; b0 < 32; b0 += 4) {
        T lo[4], hi[4];
        uint32_t at_blk[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint32_t x = __shfl_sync(0xffffffffu, cur.w0, b0 + u), y = __shfl_sync(0xffffffffu, cur.w1, b0 + u);
          at_blk[u] = __shfl_sync(0xffffffffu, blk, b0 + u);
          const uint32_t w = hf ? y : x, sh = hl * 2, bits = (w >> sh) & 3u;
          const uint32_t at = __shfl_sync(0xffffffffu, at0, b0 + u) + (hf ? __popc(x) : 0) + __popc(w & ((1u << sh) - 1u));
          lo[u] = (bits & 1u) ? vals[at] : ZenVal<T>::from_bits(0u);
          hi[u] = (bits & 2u) ? vals[at + (bits & 1u)] : ZenVal<T>::from_bits(0u);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint64_t e = (uint64_t)at_blk[u] * 64 + lane * 2;
          if (at_blk[u] == 0xffffffffu || e >= N) continue;
          if (e + 2 > N) {
            out[e] = lo[u];
          } else if constexpr (sizeof(T) == 2) {
            *reinterpret_cast<uint32_t*>(out + e) = ZenVal<T>::bits(lo[u]) | (ZenVal<T>::bits(hi[u]) << 16);
          } else {
            *reinterpret_cast<uint2*>(out + e) = make_uint2(ZenVal<T>::bits(lo[u]), ZenVal<T>::bits(hi[u]));
          }
        }
      }
      cur = nxt; nxt = nn;
      continue;
    }
    const bool some = __any_sync(0xffffffffu, cur.n != 0);
    if (some) {
      // Vector v of block b lies at v ^ (b & 7): the lanes drop their values a block apart, which would otherwise meet in the
      // same four banks.
#pragma unroll
      for (int k = 0; k < NV; ++k) sm.tile[k * 32 + lane] = make_uint4(0u, 0u, 0u, 0u);
      __syncwarp();
      T* mine = reinterpret_cast<T*>(sm.tile) + lane * 64;
      const uint32_t sw = (lane & 7u) * EPV;
      // both words at once: half the rounds, two reads in flight
      const T *v0 = sm.vals[it & 1][hf] + cur.at, *v1 = v0 + __popc(cur.w0);
      uint32_t w0 = cur.w0, w1 = cur.w1;
      while (w0 | w1) {
        const T a = *v0++, b = *v1++;                     // past a word's last value: a neighbour, not used
        if (w0) mine[(uint32_t)(__ffs(w0) - 1) ^ sw] = a;
        if (w1) mine[(uint32_t)(__ffs(w1) + 31) ^ sw] = b;
        w0 &= w0 - 1; w1 &= w1 - 1;
      }
      __syncwarp();
    }
    uint4* out16 = reinterpret_cast<uint4*>(out) + (lane % VPB);
    // whole blocks need no look at the end of the output
    if (__all_sync(0xffffffffu, blk != 0xffffffffu && (uint64_t)blk * 64 + 64 <= N)) {
#pragma unroll
      for (int k = 0; k < NV; ++k) {
        const int v = k * 32 + lane;
        const uint32_t at_blk = __shfl_sync(0xffffffffu, blk, v / VPB);
        out16[(uint64_t)at_blk * VPB] = some ? sm.tile[v ^ ((v / VPB) & 7)] : make_uint4(0u, 0u, 0u, 0u);
      }
    } else {
#pragma unroll 1
      for (int k = 0; k < NV; ++k) {
        const int v = k * 32 + lane;
        const uint32_t at_blk = __shfl_sync(0xffffffffu, blk, v / VPB);
        if (at_blk == 0xffffffffu) continue;
        const uint4 x = some ? sm.tile[v ^ ((v / VPB) & 7)] : make_uint4(0u, 0u, 0u, 0u);
        const uint64_t e = (uint64_t)at_blk * 64 + (uint64_t)(v % VPB) * EPV;
        if (e + EPV <= N) {
          *reinterpret_cast<uint4*>(out + e) = x;
        } else {
          const uint32_t xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
          for (int i = 0; i < EPV; ++i) {
            const uint32_t bits = sizeof(T) == 2 ? (xs[i / 2] >> ((i & 1) * 16)) & 0xffffu : xs[i % 4];
            if (e + i < N) out[e + i] = ZenVal<T>::from_bits(bits);
          }
        }
      }
    }
    __syncwarp();                                          // the tile and the staged values are free for the next pair
    cur = nxt; nxt = nn;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (local_status) atomicOr(c.status, local_status);
}

// Method 1 consumer: out[idx] += val for one source, read-modify-write in T (indices are unique
// within a source, and sources are applied by separate launches in rank order).
template <typename T, int NB>
__global__ void __launch_bounds__(256)
zen_scatter_source_kernel(const __grid_constant__ ZenSparseBatch<NB> bt, int src) {
  zen_pdl::enter();
  __shared__ ZenSparseCtx s_ctx;
  const ZenSparseCtx& c = zen_ctx(bt, s_ctx);
  T* __restrict__ out = reinterpret_cast<T*>(bt.out[NB > 1 ? blockIdx.y : 0]);
  __shared__ uint32_t s_ok;
  const uint32_t epoch = zen_epoch(c);
  const ZenMail* mail = zen_rec_mail(c, c.rank, src, epoch);
  if (threadIdx.x == 0) s_ok = zen_wait_epoch(&mail->epoch, epoch, c.wait_ns) ? 1u : 0u;
  __syncthreads();
  if (!s_ok) { if (threadIdx.x == 0) atomicOr(c.status, ZEN_TIMEOUT); return; }
  if ((mail->info & 1u) && threadIdx.x == 0) atomicOr(c.status, ZEN_PEER_OVERFLOW);
  const uint32_t n = min(mail->count, c.cap_rec);
  const uint2* rec = zen_rec_slots(c, c.rank, src, epoch);
  // records, then targets, four at a time per thread: each is a dependent trip to memory
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += 4 * stride) {
    uint2 r[4];
    T o[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) r[u] = i + u * stride < n ? rec[i + u * stride] : make_uint2(0xffffffffu, 0u);
#pragma unroll
    for (int u = 0; u < 4; ++u) if (r[u].x < c.numel) o[u] = out[r[u].x];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (r[u].x < c.numel) out[r[u].x] = ZenVal<T>::from_f(ZenVal<T>::to_f(o[u]) + ZenVal<T>::unbits(r[u].y));
  }
}

// Method 1 in buckets: the elements of the output are cut up as the slots of an owner are for K2b and K3b.  One CTA adds up a bucket's
// elements in shared memory, source after source, rounding to T after each as the scatter above does, and writes them out, zeros
// included: one or two launches instead of a clearing pass a rank and a launch a source (from a bucket's size on).  That is what bounds small calls; from
// IB_MAX elements on the scatter's traffic costs less than the sort's.  us, scatter / buckets: 2 x 20 000 bf16 at 2 % 47 / 34, 8 x
// 200 000 fp32 at 10 % 140 / 80, 8 x 500 000 bf16 at 10 % 133 / 112; 8 x 1 M at 10 % 152 / 178, 2 x 2 M at 1 % 34 / 41.
#define IB_MAX (1u << 19)
template <typename T, int NB>
__global__ void __launch_bounds__(256, 3)
zen_index_buckets_kernel(const __grid_constant__ ZenSparseBatch<NB> bt) {
  zen_pdl::enter();
  __shared__ ZenSparseCtx s_ctx;
  const ZenSparseCtx& c = zen_ctx(bt, s_ctx);
  T* __restrict__ out = reinterpret_cast<T*>(bt.out[NB > 1 ? blockIdx.y : 0]);
  extern __shared__ __align__(128) unsigned char smem_raw[];
  constexpr int W = 8;
  constexpr uint32_t BS = W * 2048, EPV = 16 / sizeof(T);
  float* acc = reinterpret_cast<float*>(smem_raw);                       // [BS]
  __shared__ uint32_t s_n[ZEN_MAX_RANKS];
  const uint32_t epoch = zen_epoch(c), tid = threadIdx.x;
  for (uint32_t i = tid; i < BS / 4; i += W * 32) reinterpret_cast<float4*>(acc)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  uint32_t local_status = records_wait(c, epoch, 0, c.nranks, s_n);
  const uint32_t N = (uint32_t)c.numel;
  const SbShape sh = sb_shape(N, c.cap_rec, c.nranks);
  // an element occurs once in a source
  auto apply = [&](uint32_t e, uint32_t bits) {
    float* a = acc + (e & (BS - 1));
    *a = ZenVal<T>::to_f(ZenVal<T>::from_f(*a + ZenVal<T>::unbits(bits)));
  };
  for (uint32_t bucket = blockIdx.x; bucket < sh.nbuckets; bucket += gridDim.x) {
    for (int s = 0; s < c.nranks; ++s) {
      sb_records<W>(c, sh, N, bucket, s, s + 1, s_n, epoch, local_status, apply);
      __syncthreads();
    }
    const uint32_t e0 = bucket << sh.lg, n = min(BS, N - e0);
    for (uint32_t i = tid * EPV; i < n; i += W * 32 * EPV) {
      float v[EPV];
#pragma unroll
      for (uint32_t q = 0; q < EPV; q += 4) {
        const float4 x = *reinterpret_cast<const float4*>(acc + i + q);
        *reinterpret_cast<float4*>(acc + i + q) = make_float4(0.f, 0.f, 0.f, 0.f);      // clean for the next bucket
        v[q] = x.x; v[q + 1] = x.y; v[q + 2] = x.z; v[q + 3] = x.w;
      }
      if (i + EPV <= n) {
        uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (uint32_t q = 0; q < EPV; ++q) w[q * sizeof(T) / 4] |= ZenVal<T>::bits(ZenVal<T>::from_f(v[q])) << (sizeof(T) == 2 ? (q & 1) * 16 : 0);
        *reinterpret_cast<uint4*>(out + e0 + i) = make_uint4(w[0], w[1], w[2], w[3]);
      } else {
#pragma unroll
        for (uint32_t q = 0; q < EPV; ++q)
          if (i + q < n) out[e0 + i + q] = ZenVal<T>::from_f(v[q]);
      }
    }
    __syncthreads();
  }
  if (local_status) atomicOr(c.status, local_status);
}

__global__ void zen_sparse_epoch_bump_kernel(uint32_t* e) { *e += 1u; }

// ---------------------------------------------------------------------------------------------
// Owner map (API parity with hash_index, functions_cuda_kernel.cu:169-177): out[i] = owner(i).
// mode 0: block permutation; mode 1: the reference's cubic polynomial, owner = (h % M) / (M / P).
__device__ __forceinline__ uint32_t zen_poly3(uint32_t k, uint32_t seed) {
  return 573729859u * k * k * k + 0xcc9e2d51u * k * k + 0x1b873593u * k + seed;
}

__global__ void __launch_bounds__(256)
zen_owner_map_kernel(int32_t* __restrict__ out, uint64_t n, ZenPerm perm, int mode, uint32_t table, int parts) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    if (mode == 0) {
      out[i] = (int32_t)zen_owner_of(perm, zen_perm_fwd(perm, (uint32_t)(i >> perm.lg)), parts);
    } else {
      const uint32_t per = table / parts;
      out[i] = (int32_t)((zen_poly3((uint32_t)i, 10001861u) % table) / per);
    }
  }
}

// Reference-compatible balancer (sparse_balance, functions_cuda_kernel.cu:97-167): open-addressing
// table of element indices with up to `rehash` probes inside the partition chosen by the first
// probe, overflow appended per partition.  Differences: slots are claimed with atomicCAS (no lost
// indices), indices are stored +1 so that element 0 is representable, the overflow cursor is bounded.
template <typename T>
__global__ void __launch_bounds__(256)
zen_sparse_balance_kernel(const T* __restrict__ in, uint64_t n, int32_t* __restrict__ table, uint32_t table_size,
                          int32_t* __restrict__ serial, uint32_t serial_per_part, uint32_t* __restrict__ cursors,
                          int parts, int rehash, uint32_t* __restrict__ status) {
  const uint32_t per = table_size / parts;
  const uint32_t seeds[3] = {10001861u, 100703u, 5002639u};
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    if (ZenVal<T>::to_f(in[i]) == 0.f) continue;
    const uint32_t first = zen_poly3((uint32_t)i, seeds[0]) % table_size;
    const uint32_t part = first / per, start = part * per;
    bool placed = atomicCAS(&table[first], 0, (int32_t)i + 1) == 0;
    for (int r = 1; r < rehash && r < 3 && !placed; ++r) {
      const uint32_t s = start + zen_poly3((uint32_t)i, seeds[r]) % per;
      placed = atomicCAS(&table[s], 0, (int32_t)i + 1) == 0;
    }
    if (!placed) {
      const uint32_t k = atomicAdd(&cursors[part], 1u);
      if (k < serial_per_part) serial[(uint64_t)part * serial_per_part + k] = (int32_t)i + 1;
      else atomicOr(status, ZEN_REC_OVERFLOW);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Host launchers (C ABI, called with raw pointers and the caller's stream).
static inline int grid_for(uint64_t work_items, int per_cta, int max_ctas) {
  uint64_t g = (work_items + per_cta - 1) / per_cta;
  if (g < 1) g = 1;
  if (g > (uint64_t)max_ctas) g = max_ctas;
  return (int)g;
}

static int g_sm_count = 0;
static int sm_count() {
  if (!g_sm_count) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sm_count, cudaDevAttrMultiProcessorCount, dev);
    if (g_sm_count <= 0) g_sm_count = 148;
  }
  return g_sm_count;
}

// Resident CTAs per SM of a kernel at a dynamic shared-memory size, asked once per device and size: the two calls cost more host
// time than the launch itself.  `limit`: the largest size that the kernel is ever launched with, which its attribute is set to.
template <typename K>
static int resident(K kernel, int threads, size_t smem, size_t limit, int (&known)[16][ZEN_MAX_RANKS + 1], int slot) {
  int dev = 0;
  cudaGetDevice(&dev);
  int* k = dev < 16 ? &known[dev][slot] : nullptr;
  if (k && *k > 0) return *k;
  int per_sm = 0;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess || per_sm < 1) return 0;
  if (k) *k = per_sm;
  return per_sm;
}

// Ranks of one launch: the first `n` contexts of a batch.
template <int NB> static dim3 batch_grid(int per_rank, int n) { return dim3(per_rank, NB > 1 ? n : 1); }
// Kernels for all ranks of one device start under their predecessor (launch.cuh) when the call does not fill the GPU; kernels of
// one rank may wait for other GPUs.
static bool small_call(const ZenSparseCtx& c, int n) { return c.numel * (uint64_t)n <= (1u << 20); }
template <int NB, typename K, typename... A>
static void start(bool small, K kernel, dim3 grid, int threads, size_t smem, cudaStream_t st, const A&... args) {
  if constexpr (NB > 1) zen_pdl::launch_if(small, kernel, grid, dim3(threads), smem, st, args...);
  else zen_pdl::plain(kernel, grid, threads, smem, st, args...);
}
// CTAs of one rank when `total` of them are wanted for the launch
static int share_of(int total, int n) { return total / n > 0 ? total / n : 1; }

template <typename T, bool kBroadcast, bool kRing, int NB>
static int launch_partition_as(const ZenSparseBatch<NB>& b, int n, const float* thr, cudaStream_t st) {
  constexpr uint32_t EPS = K1_STAGE_BYTES / sizeof(T);
  const ZenSparseCtx& c = b.c[0];
  const uint64_t nst = (c.numel + EPS - 1) / EPS;
  const int nq = kBroadcast ? 1 : c.nranks;
  constexpr size_t kRingBytes = kRing ? (size_t)K1_NS * K1_STAGE_BYTES : 0, kQueue = sizeof(uint2);
  const size_t smem = nq * k1_qcap(nq) * kQueue + kRingBytes;
  static int known[16][ZEN_MAX_RANKS + 1];
  const int per_sm = resident(zen_partition_push_kernel<T, kBroadcast, kRing, NB>, K1_THREADS, smem, 2048 * kQueue + kRingBytes, known, nq);
  if (per_sm < 1) return (int)cudaErrorInvalidConfiguration;
  // every CTA takes a fixed share of the stages, so the grid is exactly what is resident at once
  const int grid = grid_for(nst, 1, share_of(sm_count() * per_sm, n));
  // stages between two drains of the queues: as many as keep a queue below half of its capacity at the density the
  // plan was sized for (c.k1_density_ppm nonzeros per million elements; 0 = unknown)
  int batch = 2;
  if (c.k1_density_ppm) {
    const double per_stage = (double)EPS * c.k1_density_ppm * 1e-6 / nq;
    batch = per_stage > 0 ? (int)((k1_qcap(nq) / 2) / per_stage) : 16;
    if (batch < 1) batch = 1;
    if (batch > 16) batch = 16;
  }
  start<NB>(small_call(c, n), zen_partition_push_kernel<T, kBroadcast, kRing, NB>, batch_grid<NB>(grid, n), K1_THREADS, smem, st, b, thr, batch);
  return (int)cudaGetLastError();
}

template <typename T, int NB>
static int launch_partition(const ZenSparseBatch<NB>& b, int n, const float* thr, int broadcast, cudaStream_t st) {
  // bulk copies need 16-byte aligned sources: ranks without one go into a launch of their own
  ZenSparseBatch<NB> plain;
  const ZenSparseBatch<NB>* ring = &b;
  ZenSparseBatch<NB> some;
  int np = 0, nr = 0;
  for (int i = 0; i < n; ++i) np += reinterpret_cast<uintptr_t>(b.in[i]) % 16 != 0;
  if (np == 0) {
    nr = n;
  } else {
    np = 0;
    for (int i = 0; i < n; ++i) {
      const bool al = reinterpret_cast<uintptr_t>(b.in[i]) % 16 == 0;
      ZenSparseBatch<NB>& to = al ? some : plain;
      int& k = al ? nr : np;
      to.c[k] = b.c[i]; to.in[k] = b.in[i]; to.out[k] = b.out[i];
      ++k;
    }
    ring = &some;
  }
  int rc = 0;
  if (nr) rc = broadcast ? launch_partition_as<T, true, true, NB>(*ring, nr, thr, st) : launch_partition_as<T, false, true, NB>(*ring, nr, thr, st);
  if (!rc && np) rc = broadcast ? launch_partition_as<T, true, false, NB>(plain, np, thr, st) : launch_partition_as<T, false, false, NB>(plain, np, thr, st);
  return rc;
}

template <typename T, int NB>
static int launch_reduce(const ZenSparseBatch<NB>& b, int n, int deterministic, cudaStream_t st) {
  const ZenSparseCtx& c = b.c[0];
  const int ns = deterministic ? 1 : c.nranks;
  // four 16-byte loads (eight records) per thread when every source fills its slots, at most four CTAs per SM
  int grid = grid_for((uint64_t)ns * c.cap_rec, 256 * 8, share_of(sm_count() * 4, n));
  if (grid < ns) grid = ns;
  for (int s = 0; s < c.nranks; s += ns)
    start<NB>(small_call(c, n), zen_owner_reduce_kernel<T, NB>, batch_grid<NB>(grid, n), 256, 0, st, b, s, s + ns, deterministic ? 0 : K2_DENSE);
  return (int)cudaGetLastError();
}

template <typename T, int NB>
static int launch_gather(const ZenSparseBatch<NB>& b, int n, cudaStream_t st) {
  const ZenSparseCtx& c = b.c[0];
  const size_t smem = (size_t)K3_WARPS * K3_STAGE * (4 + sizeof(T));
  static int known[16][ZEN_MAX_RANKS + 1];
  const int per_sm = resident(zen_gather_push_kernel<T, NB>, K3_WARPS * 32, smem, smem, known, 0);
  if (per_sm < 1) return (int)cudaErrorInvalidConfiguration;
  // two pairs of chunks per warp and step where one would not fit one wave of CTAs
  const int wave = share_of(sm_count() * per_sm, n), npairs = (int)((c.nchunks + 1) / 2);
  const int ppw = npairs > K3_WARPS * wave ? K3_PPW : 1;
  const int grid = grid_for(npairs, K3_WARPS * ppw, wave);
  start<NB>(small_call(c, n), zen_gather_push_kernel<T, NB>, batch_grid<NB>(grid, n), K3_WARPS * 32, smem, st, b, ppw);
  return (int)cudaGetLastError();
}

template <typename T, int NB>
static int launch_densify(const ZenSparseBatch<NB>& b, int n, cudaStream_t st) {
  const ZenSparseCtx& c = b.c[0];
  const size_t smem = K4_WARPS * sizeof(K4Smem<T>);
  static int known[16][ZEN_MAX_RANKS + 1];
  const int per_sm = resident(zen_densify_kernel<T, NB>, K4_WARPS * 32, smem, smem, known, 0);
  if (per_sm < 1) return (int)cudaErrorInvalidConfiguration;
  const int grid = grid_for((uint64_t)c.nranks * ((c.nchunks + 1) / 2), K4_WARPS, share_of(sm_count() * per_sm, n));
  start<NB>(small_call(c, n), zen_densify_kernel<T, NB>, batch_grid<NB>(grid, n), K4_WARPS * 32, smem, st, b);
  return (int)cudaGetLastError();
}

// K2b; for owners whose CTAs read all records themselves it only waits and reports.
template <int NB>
static int launch_sort(const ZenSparseBatch<NB>& b, int n, int deterministic, int by_index, cudaStream_t st) {
  const ZenSparseCtx& c = b.c[0];
  const SbShape sh = sb_shape(by_index ? (uint32_t)c.numel : c.nslots, c.cap_rec, c.nranks);
  const int grid = sh.sorted ? grid_for((uint64_t)sh.tiles * c.nranks, 1, share_of(sm_count() * 2, n)) : 1;
  start<NB>(small_call(c, n), zen_record_sort_kernel<NB>, batch_grid<NB>(grid, n), SB_SORT_THREADS, 0, st, b, deterministic, by_index);
  return (int)cudaGetLastError();
}

// Words of `seg` for outputs of `numel` elements by method 1 in buckets; -1 where they are not taken.
static int64_t index_bucket_words(uint64_t numel, uint32_t cap_rec, int nranks) {
  if (numel > IB_MAX || numel < SB_MIN_SLOTS) return -1;
  const SbShape sh = sb_shape((uint32_t)numel, cap_rec, nranks);
  return sh.sorted ? (int64_t)sh.nbuckets * sh.tiles * nranks : 0;
}
// Method 1 in buckets: only where the plan's `seg` holds the runs (a plan that was not made for method 1 may hold fewer) and the
// output takes 16-byte stores.
static bool by_buckets(const ZenSparseCtx& c, const void* out) {
  const int64_t words = index_bucket_words(c.numel, c.cap_rec, c.nranks);
  return words >= 0 && words <= (int64_t)c.seg_words && reinterpret_cast<uintptr_t>(out) % 16 == 0;
}
template <typename T, int NB>
static int launch_scatter(const ZenSparseBatch<NB>& b, int n, cudaStream_t st) {
  const ZenSparseCtx& c = b.c[0];
  bool buckets = true;
  for (int i = 0; i < n; ++i) buckets = buckets && by_buckets(b.c[i], b.out[i]);
  if (buckets) {
    const SbShape sh = sb_shape((uint32_t)c.numel, c.cap_rec, c.nranks);
    int rc = 0;
    if (sh.sorted && (rc = launch_sort<NB>(b, n, 0, 1, st))) return rc;
    constexpr size_t smem = 8 * 2048 * 4;
    static int known[16][ZEN_MAX_RANKS + 1];
    const int per_sm = resident(zen_index_buckets_kernel<T, NB>, 256, smem, smem, known, 0);
    if (per_sm < 1) return (int)cudaErrorInvalidConfiguration;
    start<NB>(small_call(c, n), zen_index_buckets_kernel<T, NB>, batch_grid<NB>(grid_for(sh.nbuckets, 1, share_of(sm_count() * per_sm, n)), n), 256, smem, st, b);
    return (int)cudaGetLastError();
  }
  for (int i = 0; i < n; ++i) ZEN_CUDA_CHECK_RET(cudaMemsetAsync(b.out[i], 0, c.numel * sizeof(T), st));
  const int grid = grid_for(c.cap_rec, 256 * 4, share_of(sm_count() * 8, n));
  for (int s = 0; s < c.nranks; ++s) start<NB>(small_call(c, n), zen_scatter_source_kernel<T, NB>, batch_grid<NB>(grid, n), 256, 0, st, b, s);
  return (int)cudaGetLastError();
}

// K3b
template <typename T, int W, int NB>
static int launch_reduce_gather_as(const ZenSparseBatch<NB>& b, int n, uint32_t buckets, int det, cudaStream_t st) {
  static int known[16][ZEN_MAX_RANKS + 1];
  const int per_sm = resident(zen_reduce_gather_kernel<T, W, NB>, W * 32, sb_smem<W>(), sb_smem<W>(), known, 0);
  if (per_sm < 1) return (int)cudaErrorInvalidConfiguration;
  const int grid = grid_for(buckets, 1, share_of(sm_count() * per_sm, n));
  start<NB>(small_call(b.c[0], n), zen_reduce_gather_kernel<T, W, NB>, batch_grid<NB>(grid, n), W * 32, sb_smem<W>(), st, b, det);
  return (int)cudaGetLastError();
}
template <typename T, int NB>
static int launch_reduce_gather(const ZenSparseBatch<NB>& b, int n, int det, cudaStream_t st) {
  const SbShape sh = sb_shape(b.c[0].nslots, b.c[0].cap_rec, b.c[0].nranks);
  return sh.lg == 14 ? launch_reduce_gather_as<T, 8, NB>(b, n, sh.nbuckets, det, st) : launch_reduce_gather_as<T, 16, NB>(b, n, sh.nbuckets, det, st);
}
static bool in_buckets(const ZenSparseCtx& c) { return sb_shape(c.nslots, c.cap_rec, c.nranks).on; }

static ZenSparseBatch<1> one_rank(const ZenSparseCtx* c, const void* in, void* out) {
  ZenSparseBatch<1> b;
  b.c[0] = *c; b.in[0] = in; b.out[0] = out;
  return b;
}

#define DISPATCH_DTYPE(dtype, ...)                                       \
  switch (dtype) {                                                       \
    case ZEN_DTYPE_F32: { using T = float; __VA_ARGS__; } break;         \
    case ZEN_DTYPE_BF16: { using T = __nv_bfloat16; __VA_ARGS__; } break; \
    case ZEN_DTYPE_F16: { using T = __half; __VA_ARGS__; } break;        \
    default: return -1;                                                  \
  }

extern "C" {

int zen_sparse_ctx_size() { return (int)sizeof(ZenSparseCtx); }

// Advance a device-resident call counter by one (first launch of a call whose kernels read `epoch_dev`).
int zen_sparse_epoch_bump(uint32_t* epoch_dev, void* stream) {
  zen_pdl::plain(zen_sparse_epoch_bump_kernel, 1, 1, 0, (cudaStream_t)stream, epoch_dev);
  return (int)cudaGetLastError();
}

// K1.  `thr` may be null (keep every nonzero) or point at a device float threshold on |g|.
int zen_partition_push(const ZenSparseCtx* c, const void* g, const float* thr, int dtype, int broadcast, void* stream) {
  int rc = 0;
  DISPATCH_DTYPE(dtype, rc = (launch_partition<T, 1>(one_rank(c, g, nullptr), 1, thr, broadcast, (cudaStream_t)stream)));
  return rc;
}

// Buckets in shared memory where the owner's slots allow it (K2b + K3b), K2 + K3 otherwise: what `seg` has to hold, in words, and
// whether `acc` and `bitmap` are used.
// method1_numel: the elements of the output where method 1 is to be served, else 0.
int zen_sparse_scratch(uint32_t nslots, uint32_t cap_rec, int nranks, uint32_t method1_numel, int64_t* out) {
  const SbShape sh = sb_shape(nslots, cap_rec, nranks);
  out[0] = sh.on && sh.sorted ? (int64_t)sh.nbuckets * sh.tiles * nranks : 1;
  const int64_t m1 = index_bucket_words(method1_numel, cap_rec, nranks);
  if (m1 > out[0]) out[0] = m1;
  out[1] = sh.on ? 0 : 1;
  return 0;
}

// K2 or K2b.  deterministic != 0: sums in rank order (K2: one launch per source).
int zen_owner_reduce(const ZenSparseCtx* c, int dtype, int deterministic, void* stream) {
  int rc = 0;
  if (in_buckets(*c)) return launch_sort<1>(one_rank(c, nullptr, nullptr), 1, deterministic, 0, (cudaStream_t)stream);
  DISPATCH_DTYPE(dtype, rc = (launch_reduce<T, 1>(one_rank(c, nullptr, nullptr), 1, deterministic, (cudaStream_t)stream)));
  return rc;
}

// K3 or K3b (compact + push in one launch).
int zen_gather_push(const ZenSparseCtx* c, int dtype, void* stream) {
  int rc = 0;
  if (in_buckets(*c)) {
    DISPATCH_DTYPE(dtype, rc = (launch_reduce_gather<T, 1>(one_rank(c, nullptr, nullptr), 1, -1, (cudaStream_t)stream)));
    return rc;
  }
  DISPATCH_DTYPE(dtype, rc = (launch_gather<T, 1>(one_rank(c, nullptr, nullptr), 1, (cudaStream_t)stream)));
  return rc;
}

// K4.
int zen_densify(const ZenSparseCtx* c, void* out, int dtype, void* stream) {
  int rc = 0;
  DISPATCH_DTYPE(dtype, rc = (launch_densify<T, 1>(one_rank(c, nullptr, out), 1, (cudaStream_t)stream)));
  return rc;
}

// Whether method 1 takes its buckets for this context and output; else it clears the output and scatters.
int zen_sparse_method1_buckets(const ZenSparseCtx* c, const void* out) { return by_buckets(*c, out) ? 1 : 0; }

// Method 1 consumer: every source added in rank order, in buckets or into the cleared `out`.
int zen_scatter_sources(const ZenSparseCtx* c, void* out, int dtype, void* stream) {
  int rc = 0;
  DISPATCH_DTYPE(dtype, rc = (launch_scatter<T, 1>(one_rank(c, nullptr, out), 1, (cudaStream_t)stream)));
  return rc;
}

// One whole call from a single entry (one crossing from the host language instead of five): optional bump of the
// device call counter, partition + push, then scatter (method 1) or reduce + gather + densify (methods 2 / 3 / auto;
// `c->fmt_mode` carries the format).  `out` may be `x`: the scan of `x` ends before the first write.
int zen_sparse_allreduce(const ZenSparseCtx* c, const void* x, const float* thr, void* out, int dtype, int method1,
                         int deterministic, void* stream) {
  int rc = 0;
  if (c->epoch_dev && (rc = zen_sparse_epoch_bump(const_cast<uint32_t*>(c->epoch_dev), stream))) return rc;
  if ((rc = zen_partition_push(c, x, thr, dtype, method1 ? 1 : 0, stream))) return rc;
  if (method1) return zen_scatter_sources(c, out, dtype, stream);
  if (in_buckets(*c)) {
    const cudaStream_t st = (cudaStream_t)stream;
    if (sb_shape(c->nslots, c->cap_rec, c->nranks).sorted && (rc = launch_sort<1>(one_rank(c, nullptr, nullptr), 1, deterministic, 0, st))) return rc;
    DISPATCH_DTYPE(dtype, rc = (launch_reduce_gather<T, 1>(one_rank(c, nullptr, nullptr), 1, deterministic ? 1 : 0, st)));
    if (rc) return rc;
    return zen_densify(c, out, dtype, stream);
  }
  if ((rc = zen_owner_reduce(c, dtype, deterministic, stream))) return rc;
  if ((rc = zen_gather_push(c, dtype, stream))) return rc;
  return zen_densify(c, out, dtype, stream);
}

// All `n` ranks of a call that runs on one device, phase by phase: no kernel starts before everything it would wait for
// has been written.  `io` = n input pointers, then n output pointers.  All ranks go in one launch a phase.  Only the sums of owners of
// more than 2^25 slots, which are not cut into buckets, take more than the L2 holds (134 MB): K2 and K3 of such a rank go over
// them at random, one rank after the other.
int zen_sparse_allreduce_local(const ZenSparseCtx* c, int n, void* const* io, const float* thr, uint32_t epoch, uint32_t fmt,
                               int dtype, int method1, int deterministic, void* stream) {
  if (n < 1 || n > ZEN_MAX_RANKS) return -1;
  cudaStream_t st = (cudaStream_t)stream;
  ZenSparseBatch<ZEN_MAX_RANKS> b;
  for (int i = 0; i < n; ++i) {
    b.c[i] = c[i]; b.c[i].epoch = epoch; b.c[i].fmt_mode = fmt;
    b.in[i] = io[i]; b.out[i] = io[n + i];
  }
  int rc = 0;
  DISPATCH_DTYPE(dtype, {
    if ((rc = launch_partition<T, ZEN_MAX_RANKS>(b, n, thr, method1, st))) return rc;
    if (method1) return launch_scatter<T, ZEN_MAX_RANKS>(b, n, st);
    if (in_buckets(*c)) {
      if (sb_shape(c->nslots, c->cap_rec, c->nranks).sorted && (rc = launch_sort<ZEN_MAX_RANKS>(b, n, deterministic, 0, st))) return rc;
      if ((rc = launch_reduce_gather<T, ZEN_MAX_RANKS>(b, n, deterministic ? 1 : 0, st))) return rc;
      return launch_densify<T, ZEN_MAX_RANKS>(b, n, st);
    }
    const int group = c->nslots < SB_MIN_SLOTS ? n : 1;      // (in between, in_buckets)
    for (int i = 0; i < n; i += group) {
      ZenSparseBatch<ZEN_MAX_RANKS> part = b;
      if (group == 1) { part.c[0] = b.c[i]; part.in[0] = b.in[i]; part.out[0] = b.out[i]; }
      if ((rc = launch_reduce<T, ZEN_MAX_RANKS>(part, group, deterministic, st))) return rc;
      if ((rc = launch_gather<T, ZEN_MAX_RANKS>(part, group, st))) return rc;
    }
    rc = launch_densify<T, ZEN_MAX_RANKS>(b, n, st);
  });
  return rc;
}

int zen_owner_map(int32_t* out, uint64_t n, const ZenPerm* perm, int mode, uint32_t table, int parts, void* stream) {
  ZenPerm p = *perm;
  zen_pdl::plain(zen_owner_map_kernel, grid_for(n, 256 * 8, sm_count() * 8), 256, 0, (cudaStream_t)stream, out, n, p, mode, table, parts);
  return (int)cudaGetLastError();
}

int zen_sparse_balance(const void* in, uint64_t n, int dtype, int32_t* table, uint32_t table_size, int32_t* serial,
                       uint32_t serial_per_part, uint32_t* cursors, int parts, int rehash, uint32_t* status,
                       void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  const int grid = grid_for(n, 256 * 4, sm_count() * 8);
  DISPATCH_DTYPE(dtype, zen_pdl::plain(zen_sparse_balance_kernel<T>, grid, 256, 0, st, (const T*)in, n, table, table_size, serial,
                                                                           serial_per_part, cursors, parts, rehash,
                                                                           status));
  return (int)cudaGetLastError();
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------
// Sampled top-k threshold (the sparsifier of train.py:56-73 without a sort and without leaving the device):
//   zen_sample_abs       |x| at `nsamples` pseudo-random positions (counter-based hash, with replacement)
//   zen_select_kth       k-th largest of the (gathered) samples by a three-pass radix select on the float bits
// The result is one device float that zen_partition_push consumes as its threshold.
__device__ __forceinline__ uint32_t zen_mix32(uint32_t x) {
  x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
  return x;
}

template <typename T>
__global__ void __launch_bounds__(256)
zen_sample_abs_kernel(const T* __restrict__ x, uint64_t n, float* __restrict__ out, uint32_t nsamples, uint32_t seed) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nsamples; i += gridDim.x * blockDim.x) {
    const uint64_t r = ((uint64_t)zen_mix32(i * 2u + seed) << 32) | zen_mix32(i * 2u + 1u + seed * 0x9e3779b9u);
    out[i] = fabsf(ZenVal<T>::to_f(x[r % n]));
  }
}

// Histogram of bits [shift, shift + nbits) of the samples whose higher bits equal `prefix` (prefix_bits of them).
__global__ void __launch_bounds__(256)
zen_select_hist_kernel(const float* __restrict__ v, uint32_t n, uint32_t* __restrict__ hist, const uint32_t* __restrict__ state,
                       int pass) {
  __shared__ uint32_t sh[2048];
  for (int i = threadIdx.x; i < 2048; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  // state[0] = prefix found so far (high bits), state[1] = remaining rank k (1-based among the candidates)
  const uint32_t prefix = state[0];
  const int shift = pass == 0 ? 21 : (pass == 1 ? 10 : 0);
  const int nbits = pass == 2 ? 10 : 11;
  const int hi_shift = shift + nbits;                                  // bits above the current digit
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t b = __float_as_uint(v[i]) & 0x7fffffffu;
    if (pass == 0 || (b >> hi_shift) == prefix) atomicAdd(&sh[(b >> shift) & ((1u << nbits) - 1u)], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2048; i += blockDim.x)
    if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

// One CTA: walk the histogram from the top bin down to the bin holding the k-th largest; update state; clear hist.
__global__ void __launch_bounds__(1024)
zen_select_pick_kernel(uint32_t* __restrict__ hist, uint32_t* __restrict__ state, float* __restrict__ out, int pass) {
  __shared__ uint32_t cnt[2048];
  const int nbins = pass == 2 ? 1024 : 2048;
  for (int i = threadIdx.x; i < 2048; i += blockDim.x) { cnt[i] = i < nbins ? hist[i] : 0u; hist[i] = 0u; }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t k = state[1], acc = 0;
    int bin = 0;
    for (int i = nbins - 1; i >= 0; --i) {
      if (acc + cnt[i] >= k) { bin = i; break; }
      acc += cnt[i];
    }
    const int nbits = pass == 2 ? 10 : 11;
    state[0] = (state[0] << nbits) | (uint32_t)bin;
    state[1] = k - acc;
    if (pass == 2) *out = __uint_as_float(state[0]);
  }
}

__global__ void zen_select_init_kernel(uint32_t* state, uint32_t k) { state[0] = 0u; state[1] = k; }

extern "C" {

int zen_sample_abs(const void* x, uint64_t n, float* out, uint32_t nsamples, uint32_t seed, int dtype, void* stream) {
  if (n == 0 || nsamples == 0) return -1;
  const int grid = grid_for(nsamples, 256, sm_count() * 4);
  DISPATCH_DTYPE(dtype, zen_pdl::plain(zen_sample_abs_kernel<T>, grid, 256, 0, (cudaStream_t)stream, (const T*)x, n, out, nsamples, seed));
  return (int)cudaGetLastError();
}

// k-th largest (1-based) of v[0..n) (non-negative floats) -> *out.  hist: 2048 zeroed uint32 (left zeroed),
// state: 2 uint32 scratch.  Seven small launches, no host synchronisation.
int zen_select_kth(const float* v, uint32_t n, uint32_t k, uint32_t* hist, uint32_t* state, float* out, void* stream) {
  if (n == 0 || k == 0 || k > n) return -1;
  cudaStream_t st = (cudaStream_t)stream;
  zen_pdl::plain(zen_select_init_kernel, 1, 1, 0, st, state, k);
  const int grid = grid_for(n, 256 * 8, sm_count() * 2);
  for (int pass = 0; pass < 3; ++pass) {
    zen_pdl::plain(zen_select_hist_kernel, grid, 256, 0, st, v, n, hist, state, pass);
    zen_pdl::plain(zen_select_pick_kernel, 1, 1024, 0, st, hist, state, out, pass);
  }
  return (int)cudaGetLastError();
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------
// Exchange of the threshold samples among the ranks of a tensor-parallel group (every shard of a replica must use one
// threshold: train.py:62-63 all-gathers the samples with NCCL).  Every rank stores its `ns` samples into slot `rank` of
// every peer's buffer with P2P stores, the last CTA publishes a flag per peer and then waits (bounded) for the flags of
// all peers: when the kernel ends, this rank's buffer holds the samples of the whole group.  Buffers and flags exist
// twice and alternate with the call parity, so a rank that is one call ahead writes where nobody reads.
struct ZenSampleXchg {
  int32_t rank;
  int32_t nranks;
  uint32_t epoch;
  uint32_t ns;                       // samples per rank
  uint64_t wait_ns;
  float* buf[ZEN_MAX_RANKS];         // per rank: float [2][nranks][ns]
  uint32_t* flags[ZEN_MAX_RANKS];    // per rank: uint32 [2][ZEN_MAX_RANKS]
  uint32_t* status;
  uint32_t* done;                    // CTA arrival counter (left at zero)
  const uint32_t* epoch_dev;         // optional device-resident call counter
};

__global__ void __launch_bounds__(256)
zen_sample_exchange_kernel(const ZenSampleXchg c, const float* __restrict__ mine) {
  __shared__ uint32_t s_last;
  const uint32_t epoch = c.epoch_dev ? *c.epoch_dev : c.epoch;
  const uint32_t par = epoch & 1u;
  const size_t slot = ((size_t)par * c.nranks + c.rank) * c.ns;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < c.ns; i += gridDim.x * blockDim.x) {
    const float v = mine[i];
    for (int p = 0; p < c.nranks; ++p) c.buf[p][slot + i] = v;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence_system();
    s_last = (atomicAdd(c.done, 1u) == gridDim.x - 1) ? 1u : 0u;
  }
  __syncthreads();
  if (s_last) {
    __threadfence_system();
    if ((int)threadIdx.x < c.nranks) {
      zen_st_release_sys(c.flags[threadIdx.x] + par * ZEN_MAX_RANKS + c.rank, epoch);
      if (!zen_wait_epoch(c.flags[c.rank] + par * ZEN_MAX_RANKS + threadIdx.x, epoch, c.wait_ns)) atomicOr(c.status, ZEN_TIMEOUT);
    }
    if (threadIdx.x == 0) *c.done = 0u;
  }
}

// The gathered samples of this call (the half of the buffer that its parity selects) copied to a fixed place, so that
// a captured consumer reads the same address at every replay.
__global__ void __launch_bounds__(256)
zen_sample_collect_kernel(const ZenSampleXchg c, float* __restrict__ out) {
  const uint32_t epoch = c.epoch_dev ? *c.epoch_dev : c.epoch;
  const size_t n = (size_t)c.nranks * c.ns;
  const float* src = c.buf[c.rank] + (size_t)(epoch & 1u) * n;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) out[i] = src[i];
}

extern "C" {

int zen_sample_xchg_size() { return (int)sizeof(ZenSampleXchg); }

// out: nranks * ns floats (slot r = rank r's samples), valid when the two kernels have run.
int zen_sample_exchange(const ZenSampleXchg* c, const float* mine, float* out, void* stream) {
  if (!c || c->nranks < 1 || c->nranks > ZEN_MAX_RANKS || c->ns == 0) return -1;
  const int grid = grid_for(c->ns, 256 * 8, 16);
  zen_pdl::plain(zen_sample_exchange_kernel, grid, 256, 0, (cudaStream_t)stream, *c, mine);
  zen_pdl::plain(zen_sample_collect_kernel, grid_for((uint64_t)c->nranks * c->ns, 256 * 4, sm_count()), 256, 0, (cudaStream_t)stream, *c, out);
  return (int)cudaGetLastError();
}

}  // extern "C"
