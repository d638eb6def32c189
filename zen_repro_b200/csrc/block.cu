// A whole decoder block, forward or backward, from one host call.
//
// A block is 7 to 11 launches forward and 16 to 22 backward.  Launched op by op from Python, each paid for a tensor allocation, an
// autograd node and the wrapper around the call, 15 to 40 us, against kernels of 3 to 10 us for few tokens: a 64-token step of
// two GPT-2 layers took 3.0 ms of host time for 1.1 ms of kernels.  Here the host work per launch is the launch (about 2 us);
// activations live in one buffer per block whose layout is computed in this file.
//
// The kernels are the library's own entry points; only their order and the buffers are decided here.  Weight gradients with
// few tiles go out as one grouped launch at the end, with the bias and norm-parameter reductions of the block in another.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

extern "C" {
int zen_norm_fwd(const void*, const void*, const void*, const void*, void*, void*, float*, float*, int, int, float, int, int, int, void*);
int zen_norm_bwd_sums(const void*, const void*, const void*, const float*, const float*, const void*, void*, float*, float*, float*, void*, void*,
                      int, int, int, int, int, int, int, void*);
int zen_norm_bwd_parts_used(int, int);
int zen_colsum_partial(const void*, float*, int, int, int, void*);
int zen_colsum_parts(int);
int zen_act_fwd(const void*, const void*, void*, int, int, int, int, int, int, void*);
int zen_act_bwd(const void*, const void*, const void*, void*, void*, int, int, int, int, int, int, void*);
int zen_act_bwd_colsum(const void*, const void*, void*, float*, int, int, int, int, void*);
int zen_act_colsum_parts(int);
int zen_rope(void*, int, int, int, int, int, int, float, int, int, void*);
int zen_colreduce_multi(const void*, int, int, void*);
int zen_flash_fwd(const void*, void*, float*, int, int, int, int, int, int, int, float, void*);
int zen_flash_bwd(const void*, const void*, const void*, const float*, float*, void*, int, int, int, int, int, int, int, int, float, void*, void*);
int zen_flash_ds_bytes(int, int, int, int, int64_t*);
int zen_attn_fwd(const void*, void*, float*, int, int, int, int, int, int, int, float, float, void*);
int zen_attn_bwd(const void*, const void*, const void*, const float*, float*, void*, int, int, int, int, int, int, int, int, float, float,
                 float*, int, void*);
int zen_attn_hsplit(int B, int S, int Hq, int Hkv, int hd);
int zen_gemm_bf16_2cta_act(const void*, const void*, void*, const void*, void*, int, int, int, int, int, int, int, int, int, int, void*);
int zen_gemm_bf16(const void*, const void*, void*, const void*, int, int, int, int, int, int, int, int, int, int, int, void*);
int zen_gemm_bf16_2cta_splitk(const void*, const void*, void*, const void*, int, int, int, int, int, int, int, int, int, int, int, float*,
                              uint64_t, int*, int, int, int, void*);
int zen_gemm_bf16_cluster_splitk(const void*, const void*, void*, const void*, int, int, int, int, int, int, int, int, int, int, int, int,
                                 void*);
struct ZenGemmDesc {
  const void* A;
  const void* B;
  void* C;
  int32_t M, N, K, lda, ldb, ldc;
  int32_t out_fp32, accumulate;
};
int zen_gemm_bf16_2cta_group(const ZenGemmDesc*, int, int, int, float*, uint64_t, int*, int, void*);
}

namespace {

constexpr int BF16 = 1;

// Kernel of one product, chosen by the caller's time model: 0 single CTA (p0 = tile columns), 1 CTA pair (p0 = K slices),
// 2 cluster split-K (p0 = tile columns, p1 = K slices), 3 part of the grouped launch (weight gradients).
struct GemmPick { int32_t kind, p0, p1, pad; };

enum Param { NORM1_W, NORM1_B, NORM2_W, NORM2_B, POST1_W, POST2_W, QKV_W, QKV_B, O_W, O_B, UP_W, UP_B, DOWN_W, DOWN_B, NPARAMS };
enum Proj { QKV, OUT, UP, DOWN, NPROJ };

}  // namespace

extern "C" {

struct ZenBlock {
  int32_t d, hq, hkv, hd, inner;
  int32_t layer_norm, unit_offset, act_mode, gated, rope, w_in_out;      // w_in_out: weights stored [in, out]
  float eps, theta, scale, softcap;
  int32_t pad;
  const void* w[14];                                                      // by Param; null where the family has none
  GemmPick fwd[4], dx[4], dw[4], fwd_only[4];                             // by Proj, for the token count of the call; fwd_only: no backward
};
struct ZenBlockGrads {
  void* g[14];                                                            // gradient of each parameter (bf16), or null: not wanted
  int32_t acc[14];                                                        // add to what is there instead of overwriting it
};
struct ZenWorkspace { float* ws; uint64_t n_ws; int* cnt; int32_t n_cnt, pad; };

int zen_block_size() { return (int)sizeof(ZenBlock); }
int zen_block_grads_size() { return (int)sizeof(ZenBlockGrads); }

}  // extern "C"

namespace {

size_t up(size_t n) { return (n + 255) & ~size_t(255); }

// Buffer layouts.  Offsets in bytes; a null base gives the sizes.
struct Layout {
  char* base;
  size_t at = 0;
  template <typename T>
  T* take(size_t n) {
    T* p = reinterpret_cast<T*>(base + at);
    at += up(n * sizeof(T));
    return p;
  }
};

struct Saved {
  void *h1, *y1, *qkv, *a, *o, *y2, *u, *m, *dn;
  float *r1, *m1, *r2, *m2, *rp1, *rp2, *lse;
  size_t bytes;
};
struct Shape {
  int T, B, S, Sp, d, Q, H, U, inner;
  bool post1, post2;
};
Shape shape_of(const ZenBlock& z, int B, int S) {
  Shape s;
  s.B = B; s.S = S; s.T = B * S; s.Sp = (S + 127) / 128 * 128;
  s.d = z.d; s.H = z.hq * z.hd; s.Q = (z.hq + 2 * z.hkv) * z.hd; s.inner = z.inner; s.U = z.inner * (z.gated ? 2 : 1);
  s.post1 = z.w[POST1_W] != nullptr; s.post2 = z.w[POST2_W] != nullptr;
  return s;
}
Saved saved_of(const Shape& s, void* base, bool has_res) {
  Layout l{(char*)base};
  typedef uint16_t bf;
  const size_t td = (size_t)s.T * s.d;
  Saved v{};
  if (has_res) v.h1 = l.take<bf>(td);
  v.y1 = l.take<bf>(td);
  v.qkv = l.take<bf>((size_t)s.T * s.Q);
  v.a = l.take<bf>((size_t)s.T * s.H);
  v.y2 = l.take<bf>(td);
  v.u = l.take<bf>((size_t)s.T * s.U);
  v.m = l.take<bf>((size_t)s.T * s.inner);
  if (s.post1) { v.o = l.take<bf>(td); v.rp1 = l.take<float>(s.T); }
  if (s.post2) { v.dn = l.take<bf>(td); v.rp2 = l.take<float>(s.T); }
  v.r1 = l.take<float>(s.T); v.m1 = l.take<float>(s.T);
  v.r2 = l.take<float>(s.T); v.m2 = l.take<float>(s.T);
  v.bytes = l.at;
  return v;
}

struct Call {
  const ZenBlock& z;
  const ZenWorkspace& w;
  void* st;
  bool record = true;
  int rc = 0;

  const GemmPick& forward(Proj pr) const { return record ? z.fwd[pr] : z.fwd_only[pr]; }

  void gemm(const GemmPick& k, const void* A, int lda, int a_mn, const void* B, int ldb, int b_mn, void* C, int ldc, const void* bias,
            int M, int N, int K, int acc) {
    if (rc) return;
    if (k.kind == 1)                                       // p1: no workspace to cut the last round's K with
      rc = zen_gemm_bf16_2cta_splitk(A, B, C, bias, M, N, K, lda, ldb, ldc, a_mn, b_mn, 0, acc, k.p0, k.p1 ? nullptr : w.ws, k.p1 ? 0 : w.n_ws,
                                     k.p1 ? nullptr : w.cnt, k.p1 ? 0 : w.n_cnt, 0, 0, st);
    else if (k.kind == 2 && reinterpret_cast<uintptr_t>(C) % 16 == 0)
      rc = zen_gemm_bf16_cluster_splitk(A, B, C, bias, M, N, K, lda, ldb, ldc, a_mn, b_mn, 0, acc, k.p0, k.p1, st);
    else
      rc = zen_gemm_bf16(A, B, C, bias, M, N, K, lda, ldb, ldc, a_mn, b_mn, 0, acc, k.kind == 0 ? k.p0 : 0, st);
  }
  // y[T, out] = x[T, in] W (+ bias)
  void project(Proj pr, const void* x, int in, const void* W, void* y, int out, const void* bias, int T) {
    gemm(forward(pr), x, in, 0, W, z.w_in_out ? out : in, z.w_in_out, y, out, bias, T, out, in, 0);
  }
  // u = y W (+ bias) and m = activation of u.  In one launch where the CTA-pair kernel runs whole tiles and there is no gate;
  // `record`: u is needed later.
  void up(const void* y, void* u, void* m, int T) {
    const int U = z.inner * (z.gated ? 2 : 1);
    if (rc) return;
    if (!z.gated && forward(UP).kind == 1 && forward(UP).p0 <= 1) {
      rc = zen_gemm_bf16_2cta_act(y, z.w[UP_W], u, z.w[UP_B], m, T, U, z.d, z.d, z.w_in_out ? U : z.d, U, z.w_in_out, z.act_mode, U, record, st);
      return;
    }
    project(UP, y, z.d, z.w[UP_W], u, U, z.w[UP_B], T);
    if (!rc) rc = zen_act_fwd(u, z.gated ? (const char*)u + (size_t)z.inner * 2 : nullptr, m, T, z.inner, U, U, z.act_mode, BF16, st);
  }
  // dx[T, in] = dy[T, out] W'
  void project_back(Proj pr, const void* dy, int out, const void* W, void* dx, int in, int T) {
    gemm(z.dx[pr], dy, out, 0, W, z.w_in_out ? out : in, !z.w_in_out, dx, in, nullptr, T, in, out, 0);
  }
  void norm(const void* x, const void* res, int wi, int bi, void* y, void* h, float* rstd, float* mean, int T, int layer) {
    if (!rc) rc = zen_norm_fwd(x, res, z.w[wi], bi >= 0 ? z.w[bi] : nullptr, y, h, rstd, layer ? mean : nullptr, T, z.d, z.eps, layer,
                               z.unit_offset, BF16, st);
  }
};

// head sizes up to 128 without soft-capping: csrc/attention_flash.cu, everything else csrc/attention_wide.cu
bool wide_attention(const ZenBlock& z) { return z.hd > 128 || z.softcap > 0.f; }

struct ReduceJob {
  const float* part;
  void* out;
  const float* part2;
  void* out2;
  int nparts, cols, accumulate, pad;
};

struct BwdTemp {
  void *dm, *du, *dy, *dres, *da, *dqkv, *dpost;
  float *stat, *part256;
  void* ds;
  float *p_n1w, *p_n1b, *p_n2w, *p_n2b, *p_p1, *p_p2, *p_qkv, *p_o, *p_up, *p_down;
  size_t bytes;
};
size_t lse_floats(const ZenBlock& z, const Shape& s) { return (size_t)s.B * z.hq * s.Sp; }

// keep_ds: with room for dS between the kernels of the attention backward, where they would keep it.
BwdTemp bwd_temp_of(const ZenBlock& z, const Shape& s, void* base, bool keep_ds) {
  Layout l{(char*)base};
  typedef uint16_t bf;
  BwdTemp t{};
  const size_t td = (size_t)s.T * s.d;
  t.dm = l.take<bf>((size_t)s.T * s.inner);
  t.du = l.take<bf>((size_t)s.T * s.U);
  t.dy = l.take<bf>(td);
  t.dres = l.take<bf>(td);
  t.da = l.take<bf>((size_t)s.T * s.H);
  t.dqkv = l.take<bf>((size_t)s.T * s.Q);
  if (s.post1 || s.post2) t.dpost = l.take<bf>(td);
  t.stat = l.take<float>(2 * lse_floats(z, s));
  if (!wide_attention(z)) {
    int64_t need = 0;
    if (keep_ds) zen_flash_ds_bytes(s.B, s.S, z.hq, z.hd, &need);
    if (need) t.ds = l.take<char>((size_t)need);
  } else {
    const int hs = zen_attn_hsplit(s.B, s.S, z.hq, z.hkv, z.hd);
    if (hs > 1) t.part256 = l.take<float>((size_t)2 * hs * s.T * z.hkv * z.hd);
  }
  const size_t np = (size_t)zen_norm_bwd_parts_used(s.T, s.d) * s.d;
  t.p_n1w = l.take<float>(np); t.p_n2w = l.take<float>(np);
  if (z.layer_norm) { t.p_n1b = l.take<float>(np); t.p_n2b = l.take<float>(np); }
  if (s.post1) t.p_p1 = l.take<float>(np);
  if (s.post2) t.p_p2 = l.take<float>(np);
  if (z.w[QKV_B]) {
    const size_t cp = zen_colsum_parts(s.T);
    t.p_qkv = l.take<float>(cp * s.Q);
    t.p_o = l.take<float>(np);
    t.p_down = l.take<float>(cp * s.d);
    t.p_up = l.take<float>((size_t)(z.gated ? cp : zen_act_colsum_parts(s.T)) * s.U);
  }
  t.bytes = l.at;
  return t;
}

}  // namespace

extern "C" {

// Bytes of the saved buffer (with and without a residual input), of the forward temporaries and of the backward ones (with dS kept
// and without).
int zen_block_bytes(const ZenBlock* z, int B, int S, int64_t* out) {
  const Shape s = shape_of(*z, B, S);
  const size_t lse = up(lse_floats(*z, s) * 4);
  out[0] = (int64_t)(saved_of(s, nullptr, false).bytes + lse);
  out[1] = (int64_t)(saved_of(s, nullptr, true).bytes + lse);
  out[2] = (int64_t)(2 * up((size_t)s.T * s.d * 2));
  out[3] = (int64_t)bwd_temp_of(*z, s, nullptr, true).bytes;
  out[4] = (int64_t)bwd_temp_of(*z, s, nullptr, false).bytes;
  return 0;
}

// (dn, h2) = block(x, res): h1 = x + res (x itself when res is null) and h2 are the residual stream before and after the
// attention branch, dn the output of the MLP branch.  saved: kept for the backward; temp: free again when the call's work is done.
// record: a backward will follow (0: what only it needs is not written).
int zen_block_fwd(const ZenBlock* zb, int B, int S, const void* x, const void* res, void* saved, void* temp, void* dn, void* h2, int record,
                  const ZenWorkspace* ws, void* stream) {
  const ZenBlock& z = *zb;
  const Shape s = shape_of(z, B, S);
  Saved v = saved_of(s, saved, res != nullptr);
  v.lse = reinterpret_cast<float*>((char*)saved + v.bytes);
  Call c{z, *ws, stream, record != 0};
  const int T = s.T, d = s.d;
  void* o = s.post1 ? v.o : temp;
  void* o2 = (char*)temp + up((size_t)T * d * 2);
  c.norm(x, res, NORM1_W, NORM1_B, v.y1, v.h1, v.r1, v.m1, T, z.layer_norm);
  c.project(QKV, v.y1, d, z.w[QKV_W], v.qkv, s.Q, z.w[QKV_B], T);
  if (!c.rc && z.rope) c.rc = zen_rope(v.qkv, T, z.hq + z.hkv, z.hd, s.Q, S, 0, z.theta, 0, BF16, stream);
  if (!c.rc) {
    if (!wide_attention(z)) c.rc = zen_flash_fwd(v.qkv, v.a, v.lse, B, S, z.hq, z.hkv, z.hd, s.Q, s.H, z.scale, stream);
    else c.rc = zen_attn_fwd(v.qkv, v.a, v.lse, B, S, z.hq, z.hkv, z.hd, s.Q, s.H, z.scale, z.softcap, stream);
  }
  c.project(OUT, v.a, s.H, z.w[O_W], o, d, z.w[O_B], T);
  if (s.post1) c.norm(o, nullptr, POST1_W, -1, o2, nullptr, v.rp1, nullptr, T, z.layer_norm);
  c.norm(s.post1 ? o2 : o, res ? v.h1 : x, NORM2_W, NORM2_B, v.y2, h2, v.r2, v.m2, T, z.layer_norm);
  c.up(v.y2, v.u, v.m, T);
  c.project(DOWN, v.m, s.inner, z.w[DOWN_W], s.post2 ? v.dn : dn, d, z.w[DOWN_B], T);
  if (s.post2) c.norm(v.dn, nullptr, POST2_W, -1, dn, nullptr, v.rp2, nullptr, T, z.layer_norm);
  return c.rc;
}

// Gradient of x (which is also the gradient of res) into dx and of the parameters into gr, from the gradients of dn and of h2
// (null: none).  x, res, h2, saved: as in the forward.  keep_ds: which of the two sizes temp has.
int zen_block_bwd(const ZenBlock* zb, int B, int S, const void* x, const void* res, const void* h2, void* saved, void* temp, int keep_ds,
                  const void* d_dn, const void* d_h2, void* dx, const ZenBlockGrads* gr, const ZenWorkspace* ws, void* stream) {
  const ZenBlock& z = *zb;
  const Shape s = shape_of(z, B, S);
  Saved v = saved_of(s, saved, res != nullptr);
  v.lse = reinterpret_cast<float*>((char*)saved + v.bytes);
  BwdTemp t = bwd_temp_of(z, s, temp, keep_ds != 0);
  Call c{z, *ws, stream};
  const int T = s.T, d = s.d, L = z.layer_norm;
  ReduceJob jobs[8];
  int njobs = 0;
  auto reduce = [&](const float* p, int gi, const float* p2, int gi2, int nparts, int cols) {
    void *g1 = gr->g[gi], *g2 = gi2 >= 0 ? gr->g[gi2] : nullptr;
    if (g1) {
      const bool both = g2 && gr->acc[gi2] == gr->acc[gi];
      jobs[njobs++] = ReduceJob{p, g1, both ? p2 : nullptr, both ? g2 : nullptr, nparts, cols, gr->acc[gi], 0};
      if (both) g2 = nullptr;
    }
    if (g2) jobs[njobs++] = ReduceJob{p2, g2, nullptr, nullptr, nparts, cols, gr->acc[gi2], 0};
  };
  auto norm_back = [&](const void* dy, const void* h, int wi, int bi, const float* rstd, const float* mean, const void* dres, void* dh, float* pw,
                       float* pb, int sum_gi = -1, float* psum = nullptr) {       // sum_gi: the bias whose gradient the column sums of dh are
    const bool sum = sum_gi >= 0 && z.w[sum_gi] && gr->g[sum_gi];
    const int parts = zen_norm_bwd_parts_used(T, d);
    if (!c.rc) c.rc = zen_norm_bwd_sums(dy, h, z.w[wi], rstd, L ? mean : nullptr, dres, dh, pw, L ? pb : nullptr, sum ? psum : nullptr, nullptr, nullptr,
                                        T, d, L, z.unit_offset, 0, BF16, 1, stream);
    reduce(pw, wi, pb, bi, parts, d);
    if (sum) reduce(psum, sum_gi, nullptr, -1, parts, d);
  };
  auto bias_back = [&](const void* dy, int cols, int gi, float* part) {
    if (!z.w[gi] || !gr->g[gi]) return;
    if (!c.rc) c.rc = zen_colsum_partial(dy, part, T, cols, BF16, stream);
    reduce(part, gi, nullptr, -1, zen_colsum_parts(T), cols);
  };
  // MLP branch
  const void* ddn = d_dn;
  if (s.post2) {
    norm_back(d_dn, v.dn, POST2_W, -1, v.rp2, nullptr, nullptr, t.dpost, t.p_p2, nullptr);
    ddn = t.dpost;
  }
  c.project_back(DOWN, ddn, d, z.w[DOWN_W], t.dm, s.inner, T);
  bias_back(ddn, d, DOWN_B, t.p_down);
  if (!c.rc) {
    if (z.gated) {
      const size_t half = (size_t)s.inner * 2;
      c.rc = zen_act_bwd(v.u, (const char*)v.u + half, t.dm, t.du, (char*)t.du + half, T, s.inner, s.U, s.U, z.act_mode, BF16, stream);
      bias_back(t.du, s.U, UP_B, t.p_up);
    } else if (z.w[UP_B] && gr->g[UP_B]) {
      c.rc = zen_act_bwd_colsum(v.u, t.dm, t.du, t.p_up, T, s.inner, z.act_mode, BF16, stream);
      reduce(t.p_up, UP_B, nullptr, -1, zen_act_colsum_parts(T), s.U);
    } else {
      c.rc = zen_act_bwd(v.u, nullptr, t.dm, t.du, nullptr, T, s.inner, s.U, s.U, z.act_mode, BF16, stream);
    }
  }
  c.project_back(UP, t.du, s.U, z.w[UP_W], t.dy, d, T);
  // (its result goes to the output projection as it is, unless a norm lies between)
  norm_back(t.dy, h2, NORM2_W, NORM2_B, v.r2, v.m2, d_h2, t.dres, t.p_n2w, t.p_n2b, s.post1 ? -1 : O_B, t.p_o);
  // weight gradients of the MLP before its scratch is needed no more (post2 and post1 share dpost)
  ZenGemmDesc group[4];
  int ngroup = 0;
  auto weight = [&](Proj pr, int gi, const void* in_act, int in, const void* dy, int out) {
    if (!gr->g[gi] || c.rc) return;
    const void *A = z.w_in_out ? in_act : dy, *Bm = z.w_in_out ? dy : in_act;
    const int M = z.w_in_out ? in : out, N = z.w_in_out ? out : in;
    if (z.dw[pr].kind == 3) group[ngroup++] = ZenGemmDesc{A, Bm, gr->g[gi], M, N, T, M, N, N, 0, gr->acc[gi]};
    else c.gemm(z.dw[pr], A, M, 1, Bm, N, 1, gr->g[gi], N, nullptr, M, N, T, gr->acc[gi]);
  };
  auto flush = [&]() {
    if (ngroup && !c.rc) c.rc = zen_gemm_bf16_2cta_group(group, ngroup, 1, 1, ws->ws, ws->n_ws, ws->cnt, ws->n_cnt, stream);
    ngroup = 0;
  };
  weight(DOWN, DOWN_W, v.m, s.inner, ddn, d);
  weight(UP, UP_W, v.y2, d, t.du, s.U);
  // attention branch
  const void* d_o = t.dres;
  if (s.post1) {
    if (s.post2) flush();                                  // the group may still read dpost
    norm_back(t.dres, v.o, POST1_W, -1, v.rp1, nullptr, nullptr, t.dpost, t.p_p1, nullptr, O_B, t.p_o);
    d_o = t.dpost;
  }
  c.project_back(OUT, d_o, d, z.w[O_W], t.da, s.H, T);
  if (!c.rc) {
    if (!wide_attention(z))
      c.rc = zen_flash_bwd(v.qkv, v.a, t.da, v.lse, t.stat, t.dqkv, B, S, z.hq, z.hkv, z.hd, s.Q, s.H, s.Q, z.scale, t.ds, stream);
    else
      c.rc = zen_attn_bwd(v.qkv, v.a, t.da, v.lse, t.stat, t.dqkv, B, S, z.hq, z.hkv, z.hd, s.Q, s.H, s.Q, z.scale, z.softcap, t.part256,
                          zen_attn_hsplit(B, S, z.hq, z.hkv, z.hd), stream);
  }
  if (!c.rc && z.rope) c.rc = zen_rope(t.dqkv, T, z.hq + z.hkv, z.hd, s.Q, S, 0, z.theta, 1, BF16, stream);
  c.project_back(QKV, t.dqkv, s.Q, z.w[QKV_W], t.dy, d, T);
  bias_back(t.dqkv, s.Q, QKV_B, t.p_qkv);
  norm_back(t.dy, res ? v.h1 : x, NORM1_W, NORM1_B, v.r1, v.m1, t.dres, dx, t.p_n1w, t.p_n1b);
  weight(OUT, O_W, v.a, s.H, d_o, d);
  weight(QKV, QKV_W, v.y1, d, t.dqkv, s.Q);
  flush();
  if (njobs && !c.rc) c.rc = zen_colreduce_multi(jobs, njobs, BF16, stream);
  return c.rc;
}

}  // extern "C"
