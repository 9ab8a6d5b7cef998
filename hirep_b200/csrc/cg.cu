// cg.cu -- multi-shift CG on the device (LibHR/Inverters/cg_mshift.c) and its
// mixed-precision defect-correction driver (LibHR/Inverters/cg_mshift_flt.c).
//
// The recursion is HiRep's, term for term, but every scalar (alpha, omega,
// gamma, delta and the per-shift z1/z2/z3 and flags) lives in device memory and
// is updated by one-block "fold" kernels, so an iteration never waits for the
// host.  One iteration with the even-odd H^2 is
//   H k (two hops, the last with the |H k|^2 = <k, H^2 k> partials) ->
//   fold_alpha, beside the first hop of the second H -> its last hop, which adds
//   omega H^2 k to r instead of writing it and leaves the |r|^2 partials ->
//   fold_lambda -> k = gamma k + r
// and the shifted systems (x_i += c_i p_i, p_i = d_i p_i + z3_i r), which only follow
// the recursion, are brought up to date once per CG_CHUNK iterations.
// With another operator the products and r += omega M k are kernels of their own.
// The host launches several iterations at a time (a captured CUDA graph), one chunk
// ahead of the state that it reads.  When fold_lambda finds the stopping condition it marks the
// state; the remaining kernels of that iteration finish it exactly as HiRep's
// loop body would, and every kernel of later iterations returns at once, so the
// solution and the iteration count are those of HiRep's loop.
#include <cstddef>
#include <type_traits>
#include <vector>

#include "dirac.cuh"
#include "linalg.cuh"

namespace hrgpu {

constexpr int MAXS = 64;
constexpr int CG_CHUNK = 4;
constexpr int CG_HARD_LIMIT = 200000;  // iterations, when the caller sets no max_iter

struct CGState {
  double omega, oldomega, gamma, alpha, lambda, delta, innorm2, err2;
  int n, state, iter, max_iter, notconv, flt;
  int bad;  // <k, Mk> was zero or not finite (k_cg_fold_alpha; k_cg_fold_lambda ends the solve)
  double shift[MAXS], z1[MAXS], z2[MAXS], z3[MAXS];
  int flag[MAXS];
  // the last iterations' coefficients of the shifted systems, not yet applied to the fields:
  // x_i += cx p_i, then p_i = cp p_i + pz r where pf is set
  int pend;  // how many
  double cx[CG_CHUNK][MAXS], cp[CG_CHUNK][MAXS], pz[CG_CHUNK][MAXS];
  int pf[CG_CHUNK][MAXS];
};

constexpr int FOLD_THREADS = 512;

// sum of the partials in a fixed order, eight loads in flight per thread
__device__ double fold_partials(const double *partials, int nblocks, int stride) {
  double s = 0;
  int b = threadIdx.x;
  for (; b + 7 * (int)blockDim.x < nblocks; b += 8 * blockDim.x) {
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = partials[(long)(b + k * (int)blockDim.x) * stride];
#pragma unroll
    for (int k = 0; k < 8; k++) s += v[k];
  }
  for (; b < nblocks; b += blockDim.x) s += partials[(long)b * stride];
  return block_sum(s);
}

// alpha = <k, Mk>; omega = -delta/alpha; z3 and the solution coefficients
// (cg_mshift.c:82-91), one thread per shift.  It may run beside the first hop of the second
// H, whose threads read the state to decide whether to leave ahead of a barrier, so it only
// reads the state and leaves a breakdown in bad.
// slot: the iteration's place among those kept for the shifted systems.
__global__ void __launch_bounds__(FOLD_THREADS) k_cg_fold_alpha(CGState *S, const double *partials, int nblocks, int stride,
                                                                int slot) {
  if (slot == 0 && threadIdx.x == 0) S->pend = 0;
  if (S->state != 0) return;
  const double alpha = fold_partials(partials, nblocks, stride);
  const bool bad = !isfinite(alpha) || alpha == 0.0;  // breakdown (non-positive operator or NaN input)
  const double omega = -S->delta / alpha, oldomega = S->omega, gamma = S->gamma;
  const int i = threadIdx.x;
  if (!bad && i < S->n) {
    if (S->flag[i]) {
      const double z1 = S->z1[i], z2 = S->z2[i];
      const double z3 = oldomega * z1 * z2 / (omega * gamma * (z1 - z2) + z1 * oldomega * (1. + S->shift[i] * omega));
      S->z3[i] = z3;
      S->cx[slot][i] = -omega * z3 / z2;
    } else {
      S->cx[slot][i] = 0.0;
    }
  }
  __syncthreads();
  if (i == 0) {
    S->alpha = alpha;
    S->bad = bad;
    if (!bad) {
      S->oldomega = oldomega;
      S->omega = omega;
    }
  }
}

// lambda = |r|^2, gamma, convergence flags (cg_mshift.c:92-111; cg_mshift_flt.c:96-118).
// The only kernel that changes the state, when nothing runs beside it: 1 in the iteration that
// converged, whose updates still follow, 2 in the one after it, 3 in one that broke down
// (its residual, made with the iteration before's omega, is not used).
__global__ void __launch_bounds__(FOLD_THREADS) k_cg_fold_lambda(CGState *S, const double *partials, int nblocks, int slot) {
  pdl_enter();
  const int state = S->state, bad = S->bad;
  __syncthreads();
  if (state != 0 || bad) {
    if (threadIdx.x == 0) S->state = state == 0 ? 3 : (state == 1 ? 2 : state);
    return;
  }
  const double lambda = fold_partials(partials, nblocks, 1);
  const double gamma = lambda / S->delta;
  const int i = threadIdx.x;
  int open = 0;
  if (i < S->n) {
    const double z3 = S->z3[i], lim = S->err2 * S->innorm2;
    int flag = S->flag[i];
    if (S->flt) {
      open = lambda * z3 * z3 > lim;
    } else {
      if (lambda * z3 * z3 < lim) S->flag[i] = flag = 0;
      open = flag;
    }
    // a shift that converged in this iteration keeps its z's, and gets its last x in the update
    S->pf[slot][i] = flag;
    if (flag) {
      const double z2 = S->z2[i];
      S->cp[slot][i] = gamma * z3 * z3 / (z2 * z2);
      S->pz[slot][i] = z3;
      S->z1[i] = z2;
      S->z2[i] = z3;
    }
  }
  const int notconv = __syncthreads_count(open);
  if (i == 0) {
    S->lambda = lambda;
    S->gamma = gamma;
    S->delta = lambda;
    S->notconv = notconv;
    S->iter++;
    if (isfinite(lambda)) S->pend = slot + 1;
    if (!isfinite(lambda)) S->state = 3;
    else if (notconv == 0 || (S->max_iter != 0 && S->iter >= S->max_iter)) S->state = 1;
  }
}

// rn = r + omega Mk (rn may be r) with |rn|^2 partials, for the operators whose last hop does not do it
template <typename V>
__global__ void __launch_bounds__(RED_THREADS) k_cg_update_r(CGState *S, V *rn, const V *r, const V *Mk, long n,
                                                             double *partials) {
  if (S->state != 0) return;
  const double omega = S->omega;
  double nrm = 0.0;
  long stride = (long)gridDim.x * blockDim.x;
  for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += stride) {
    V rv = r[e];
    rmac(rv, (decltype(rv.x))omega, Mk[e]);
    rn[e] = rv;
    nrm += (double)rv.x * rv.x + (double)rv.y * rv.y;
  }
  nrm = block_sum(nrm);
  if (threadIdx.x == 0) partials[blockIdx.x] = nrm;
}

// one 16-byte word of a field: one FP64 complex number or two FP32 ones
__device__ __forceinline__ double2 fma_r(double a, double2 x, double2 y) { return make_double2(fma(a, x.x, y.x), fma(a, x.y, y.y)); }
__device__ __forceinline__ float4 fma_r(float a, float4 x, float4 y) {
  return make_float4(fmaf(a, x.x, y.x), fmaf(a, x.y, y.y), fmaf(a, x.z, y.z), fmaf(a, x.w, y.w));
}
__device__ __forceinline__ double2 mul_r(double a, double2 x) { return make_double2(a * x.x, a * x.y); }
__device__ __forceinline__ float4 mul_r(float a, float4 x) { return make_float4(a * x.x, a * x.y, a * x.z, a * x.w); }

// k = gamma k + r.  one: a single unshifted system, whose p_0 is k (every z is 1): x_0 += cx_0 k
// as well, and p_0 is not touched.
// W: 16-byte words.  (FP32 solves run on the library's own fields only; an FP64
// complex number is one word, so a caller's field needs no more than its own alignment.)
template <typename W, typename R, bool PDL>
__global__ void __launch_bounds__(RED_THREADS) k_cg_update(const CGState *S, W *const *x, W *k, const W *r, long n, int one) {
  if (PDL) pdl_enter();
  if (S->state >= 2) return;
  const R gamma = (R)S->gamma, cx = (R)S->cx[0][0];
  W *x0 = x[0];
  const long stride = (long)gridDim.x * blockDim.x;
  for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += stride) {
    const W rv = r[e], kv = k[e];
    if (one) x0[e] = fma_r(cx, kv, x0[e]);
    k[e] = fma_r(gamma, kv, rv);
  }
}

template <typename W>
struct CGRing {
  const W *r[CG_CHUNK];
};

// The iterations kept in S (pend of them, their residuals in ring) applied to every shifted
// system: x_i += cx p_i, p_i = cp p_i + pz r, one after the other in registers, so the
// results are bit for bit those of an update in each iteration.  Such an update is bound by HBM:
// 4n + 1 vectors in each; this is 4n + CG_CHUNK per CG_CHUNK iterations.  The solve with 10
// shifts on 16^4 with NF = 6 in FP64 takes 17.5 ms, and 23.5 ms with an update in each iteration
// (516 MB, part of it still in L2).
template <typename W, typename R>
__global__ void __launch_bounds__(RED_THREADS) k_cg_shifts(const CGState *S, W *const *x, W *const *p, CGRing<W> ring, long n) {
  const int pend = S->pend;
  if (pend == 0) return;
  __shared__ R cx[CG_CHUNK][MAXS], cp[CG_CHUNK][MAXS], pz[CG_CHUNK][MAXS];
  __shared__ int pf[CG_CHUNK][MAXS], act[MAXS];  // act: 0 converged before, 1 x only, 2 x and p
  __shared__ W *px[MAXS], *pp[MAXS];
  const int ns = S->n;
  for (int i = threadIdx.x; i < ns; i += blockDim.x) {
    int a = 0;
    for (int c = 0; c < CG_CHUNK; c++) {
      const bool in = c < pend;
      cx[c][i] = in ? (R)S->cx[c][i] : (R)0;
      pf[c][i] = in && cx[c][i] != (R)0 ? S->pf[c][i] : 0;
      cp[c][i] = pf[c][i] ? (R)S->cp[c][i] : (R)0;
      pz[c][i] = pf[c][i] ? (R)S->pz[c][i] : (R)0;
      if (pf[c][i]) a = 2;
      else if (cx[c][i] != (R)0 && a == 0) a = 1;
    }
    act[i] = a;
    px[i] = x[i];
    pp[i] = p[i];
  }
  __syncthreads();
  const long stride = (long)gridDim.x * blockDim.x;
  for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += stride) {
    W rv[CG_CHUNK];
#pragma unroll
    for (int c = 0; c < CG_CHUNK; c++) rv[c] = ring.r[c < pend ? c : 0][e];
#pragma unroll 2
    for (int i = 0; i < ns; i++) {
      if (act[i] == 0) continue;
      W pv = pp[i][e], xv = px[i][e];
#pragma unroll
      for (int c = 0; c < CG_CHUNK; c++) {
        if (cx[c][i] == (R)0) continue;
        xv = fma_r(cx[c][i], pv, xv);
        if (pf[c][i]) pv = fma_r(pz[c][i], rv[c], mul_r(cp[c][i], pv));
      }
      px[i][e] = xv;
      if (act[i] == 2) pp[i][e] = pv;
    }
  }
}

// <k, Mk> partials (re, im per block) for the fold; stops with the state
template <typename V>
__global__ void __launch_bounds__(RED_THREADS) k_cg_dot(const CGState *S, const V *a, const V *b, long n, double *partials) {
  if (S->state != 0) return;
  double re = 0.0;
  long stride = (long)gridDim.x * blockDim.x;
  for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += stride) {
    V u = a[e], v = b[e];
    re += (double)u.x * v.x + (double)u.y * v.y;
  }
  re = block_sum(re);
  if (threadIdx.x == 0) {
    partials[2 * blockIdx.x] = re;
    partials[2 * blockIdx.x + 1] = 0.0;
  }
}

// ---------------------------------------------------------------------------
// workspace (cached between calls, grown on demand)
// ---------------------------------------------------------------------------
// The padding of the work fields (components are L.ld >= VH sites apart) is kept at zero: the
// hops write the sites alone, but the updates and the norms run over whole fields.
struct CGWork {
  std::vector<void *> bufs;  // p[0..n-1], k, r, Mk, and where memory allows CG_CHUNK - 1 more residuals
  size_t bytes = 0;
  CGState *S = nullptr;
  CGState *hS = nullptr;  // pinned host copies of the last two chunks' states
  cudaEvent_t ev[2] = {nullptr, nullptr};
  void **d_ptrs = nullptr;  // device arrays of pointers: x[MAXS], p[MAXS]
};
static CGWork W[2];  // [prec]

// work fields of the defect-correction driver: FP64 res, res2, tmp; FP32 res_flt, out_flt[n]
struct FltWork {
  void *dres = nullptr, *dres2 = nullptr, *dtmp = nullptr;
  std::vector<void *> fbuf;
  size_t bd = 0, bf = 0;
};
static FltWork FW;

static int cg_workspace(int prec, int nvec, size_t bytes) {
  CGWork &w = W[prec];
  if (w.bytes != bytes) {
    for (void *b : w.bufs) cudaFree(b);
    w.bufs.clear();
    w.bytes = bytes;
  }
  while ((int)w.bufs.size() < nvec) {
    void *b = nullptr;
    HR_CUDA(cudaMalloc(&b, bytes));
    w.bufs.push_back(b);
    HR_CUDA(cudaMemsetAsync(b, 0, bytes, L.stream));
  }
  if (!w.S) {
    HR_CUDA(cudaMalloc(&w.S, sizeof(CGState)));
    HR_CUDA(cudaMallocHost(&w.hS, 2 * sizeof(CGState)));
    for (cudaEvent_t &ev : w.ev) HR_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    HR_CUDA(cudaMalloc(&w.d_ptrs, sizeof(void *) * 2 * MAXS));
  }
  return 0;
}

// CG_CHUNK - 1 more residuals behind the first nvec fields, where they leave as much again
// free: true if they are there.  Without them the solve runs as well, updating every iteration.
static bool cg_more_residuals(CGWork &w, int nvec) {
  if (!optional_allowed()) return false;
  while ((int)w.bufs.size() < nvec + CG_CHUNK - 1) {
    void *b = nullptr;
    if (!optional_room((CG_CHUNK - 1) * w.bytes)) return false;
    if (cudaMalloc(&b, w.bytes) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    if (cudaMemsetAsync(b, 0, w.bytes, L.stream) != cudaSuccess) {
      cudaGetLastError();
      cudaFree(b);
      return false;
    }
    w.bufs.push_back(b);
  }
  return true;
}

// The chunk of iterations as a CUDA graph, captured once per (operator, mass,
// work buffers, kernel variants, link storage) and replayed: seven launches per
// iteration (one more every CG_CHUNK with shifted systems), most of them small, cost more in launch gaps than in work.  The
// graph reads the links and clover blocks at replay; the clover blocks (for
// this mass) and the BF16 link copy are brought up to date before each replay.
// (Folding the partials in the last block of the kernel that wrote them, with
// an atomic ticket, instead of one-block fold kernels was measured slower: the
// per-block fence outweighs the launches it saves inside a graph.)
struct CGGraph {
  int op = -1;
  double mass = 0;
  const void *ptrs[9 + CG_CHUNK] = {};
  int v[3] = {-1, -1, -1}, force = -1, flt_links = -1, pdl = -1, recon = -1, one = -1, keep = -1, both = -1;
  unsigned long mvm = 0;  // hop launches in one replay (the MVM counter)
  cudaGraphExec_t exec = nullptr;
};
static CGGraph CGG[2];  // [prec]
static cudaStream_t cg_cap = nullptr, cg_cap2 = nullptr;  // capture streams: the iteration, the fold beside a hop
static cudaEvent_t cg_ev[2] = {nullptr, nullptr};

static void drop_cg_graph(CGGraph &c) {
  if (c.exec) cudaGraphExecDestroy(c.exec);
  c = CGGraph();
}

void cg_drop_work() {
  for (int q = 0; q < 2; q++) {
    for (cudaEvent_t ev : W[q].ev)  // a solve leaves a chunk in flight behind its last one
      if (ev) cudaEventSynchronize(ev);
    drop_cg_graph(CGG[q]);
    for (void *b : W[q].bufs) cudaFree(b);
    W[q].bufs.clear();
    W[q].bytes = 0;
  }
}

void cg_release() {
  batch_release();
  qmr_release();
  hmc_release();
  hostop_release();
  cudaFree(FW.dres); cudaFree(FW.dres2); cudaFree(FW.dtmp);
  for (void *b : FW.fbuf) cudaFree(b);
  FW = FltWork();
  cg_drop_work();
  if (cg_cap) cudaStreamDestroy(cg_cap);
  if (cg_cap2) cudaStreamDestroy(cg_cap2);
  for (cudaEvent_t &ev : cg_ev) {
    if (ev) cudaEventDestroy(ev);
    ev = nullptr;
  }
  cg_cap = cg_cap2 = nullptr;
  for (int q = 0; q < 2; q++) {
    if (W[q].S) cudaFree(W[q].S);
    if (W[q].hS) cudaFreeHost(W[q].hS);
    for (cudaEvent_t &ev : W[q].ev) {
      if (ev) cudaEventDestroy(ev);
      ev = nullptr;
    }
    if (W[q].d_ptrs) cudaFree(W[q].d_ptrs);
    W[q].S = nullptr;
    W[q].hS = nullptr;
    W[q].d_ptrs = nullptr;
  }
}

static unsigned red_grid(long n) {
  long b = (n + RED_THREADS - 1) / RED_THREADS;
  return (unsigned)(b < RED_MAX_BLOCKS ? b : RED_MAX_BLOCKS);
}

// CG_CHUNK iterations, launched one kernel at a time.  side: a second stream of the
// capture in progress for the fold beside a hop, or nullptr.  r: the residual after iteration
// c is r[c % keep]; the shifted systems are updated when keep of them are there.
template <typename R>
static int cg_iterations(int op, int prec, double mass, CGWork &w, void *k, void *const *r, int keep, void *Mk, long ne,
                         unsigned g, int one, cudaStream_t side) {
  typedef typename C2<R>::T V;
  typedef typename std::conditional<sizeof(R) == 8, double2, float4>::type W;
  const long nw = ne * (long)sizeof(V) / (long)sizeof(W);
  W *const *dx = (W *const *)w.d_ptrs;
  W *const *dp = (W *const *)(w.d_ptrs + MAXS);
  const bool eo = op == HRGPU_OP_G5DPHI_EOPRE_SQ || op == HRGPU_OP_G5CPHI_EOPRE_SQ;
  const bool clover = op == HRGPU_OP_G5CPHI_EOPRE_SQ;
  const bool small = eo && L.hop_pdl && hop_small(clover, prec);
  double *part2 = L.partials + L.npart / 2;  // |r|^2, while the |Hk|^2 ones may still be read
  CGRing<W> ring;
  for (int c = 0; c < CG_CHUNK; c++) ring.r[c] = (const W *)r[c % keep];
  for (int c = 0; c < CG_CHUNK; c++) {
    unsigned nlam = g;
    const int slot = c % keep;
    const void *r0 = r[(slot + keep - 1) % keep];
    void *r1 = r[slot];
    if (eo) {
      // alpha = <k, H^2 k> = |H k|^2 from the first H's partials
      void *tmp = eo_tmp(prec);
      if (!tmp) return HRGPU_E_CUDA;
      if (int q = apply_eo(clover, prec, mass, tmp, k, 1, L.partials, nullptr)) return q;
      const int nb = hop_red_blocks(clover, prec);  // tuned by now
      const bool tail = hop_tail_settled(clover, prec);
      cudaStream_t fs = tail && side ? side : L.stream;
      if (fs != L.stream) {
        HR_CUDA(cudaEventRecord(cg_ev[0], L.stream));
        HR_CUDA(cudaStreamWaitEvent(fs, cg_ev[0], 0));
      }
      k_cg_fold_alpha<<<1, FOLD_THREADS, 0, fs>>>(w.S, L.partials, nb, 1, slot);
      if (fs != L.stream) HR_CUDA(cudaEventRecord(cg_ev[1], fs));
      if (tail) {
        HopTail t;
        t.racc = r0;
        t.omega = &w.S->omega;
        t.no_pdl = fs != L.stream;
        // the second H, joined by the fold before its last hop
        if (int q = eo_stage<R>(clover, mass, 0, HRGPU_EVEN, Mk, tmp, 1, nullptr, 0, -1)) return q;
        if (fs != L.stream) HR_CUDA(cudaStreamWaitEvent(L.stream, cg_ev[1], 0));
        if (int q = eo_stage<R>(clover, mass, 1, HRGPU_EVEN, r1, tmp, 1, part2, 0, -1, &t)) return q;
        nlam = (unsigned)nb;
      } else {
        if (int q = apply_eo(clover, prec, mass, Mk, tmp, 1, nullptr, nullptr)) return q;
        k_cg_update_r<V><<<g, RED_THREADS, 0, L.stream>>>(w.S, (V *)r1, (const V *)r0, (const V *)Mk, ne, part2);
      }
    } else {
      if (int q = apply_op(op, prec, mass, Mk, k)) return q;
      k_cg_dot<V><<<g, RED_THREADS, 0, L.stream>>>(w.S, (const V *)k, (const V *)Mk, ne, L.partials);
      k_cg_fold_alpha<<<1, FOLD_THREADS, 0, L.stream>>>(w.S, L.partials, g, 2, slot);
      k_cg_update_r<V><<<g, RED_THREADS, 0, L.stream>>>(w.S, (V *)r1, (const V *)r0, (const V *)Mk, ne, part2);
    }
    // on a small lattice, where the launches count, these start while the kernel before ends
    const bool pdl = side && small;
    HR_CUDA(launch_after(pdl, k_cg_fold_lambda, 1u, (unsigned)FOLD_THREADS, w.S, part2, (int)nlam, slot));
    HR_CUDA(launch_after(pdl, pdl ? k_cg_update<W, R, true> : k_cg_update<W, R, false>, red_grid(nw), (unsigned)RED_THREADS,
                         w.S, dx, (W *)k, (const W *)r1, nw, one));
    if (!one && slot == keep - 1)
      k_cg_shifts<W, R><<<red_grid(nw), RED_THREADS, 0, L.stream>>>(w.S, dx, dp, ring, nw);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail_cuda(e, "cg iteration", __FILE__, __LINE__);
  }
  return 0;
}
static bool op_is_clover(int op) {
  return op == HRGPU_OP_G5CPHI_EOPRE_SQ || op == HRGPU_OP_G5CPHI_SQ || op == HRGPU_OP_CPHI_EOPRE ||
         op == HRGPU_OP_G5CPHI_EOPRE || op == HRGPU_OP_CPHI;
}
// *mvm: the hops of the chunk launched, for the caller to count when it is known that they ran
template <typename R>
static int cg_chunk(int op, int prec, double mass, CGWork &w, void *k, void *const *r, int keep, void *Mk, long ne,
                    unsigned g, int one, unsigned long *mvm) {
  if (op_is_clover(op))
    if (int rc = clover_prepare(mass, prec)) return rc;
  if (prec == HRGPU_FLOAT && L.flt_links == HRGPU_LINKS_BF16)
    if (int rc = ensure_links_bf16()) return rc;
  const int pi = prec == HRGPU_DOUBLE ? 0 : (L.flt_links == HRGPU_LINKS_BF16 ? 2 : 1);
  if (!op_tuned(op, prec)) {  // tunes the hopping kernels
    const unsigned long m0 = mvm_count();
    const int rc = cg_iterations<R>(op, prec, mass, w, k, r, keep, Mk, ne, g, one, nullptr);
    *mvm = mvm_count() - m0;
    mvm_restore(m0);
    return rc;
  }
  const void *links = prec == HRGPU_DOUBLE ? (const void *)L.U
                                           : (L.flt_links == HRGPU_LINKS_BF16 ? (const void *)L.Ubf : (const void *)L.Uf);
  const void *ptrs[9 + CG_CHUNK] = {k, Mk, w.S, w.d_ptrs, L.partials, links, L.cur_stop,
                          prec == HRGPU_DOUBLE ? L.tmp_e : L.tmp_e_f, prec == HRGPU_DOUBLE ? L.tmp_o : L.tmp_o_f};
  for (int c = 0; c < CG_CHUNK; c++) ptrs[9 + c] = r[c % keep];
  CGGraph &c = CGG[prec];
  const int recon = L.recon_allow ? L.recon12 : 0;
  const int both = L.hop_both[pi][op_is_clover(op) ? EP_CLOV : EP_AXPY];
  bool same = c.exec && c.op == op && c.mass == mass && c.force == L.hop_force && c.flt_links == L.flt_links &&
              c.both == both && c.pdl == (int)L.hop_pdl && c.recon == recon && c.one == one && c.keep == keep;
  for (int i = 0; i < 3 && same; i++) same = c.v[i] == L.hop_variant[pi][i];
  for (int i = 0; i < 9 + CG_CHUNK && same; i++) same = c.ptrs[i] == ptrs[i];
  if (!same) {
    drop_cg_graph(c);
    if (!cg_cap) {
      HR_CUDA(cudaStreamCreateWithFlags(&cg_cap, cudaStreamNonBlocking));
      HR_CUDA(cudaStreamCreateWithFlags(&cg_cap2, cudaStreamNonBlocking));
      for (cudaEvent_t &ev : cg_ev) HR_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    }
    const unsigned long m0 = mvm_count();
    cudaGraph_t graph = nullptr;
    cudaStream_t saved = L.stream;
    HR_CUDA(cudaStreamBeginCapture(cg_cap, cudaStreamCaptureModeRelaxed));
    L.stream = cg_cap;
    int rc = cg_iterations<R>(op, prec, mass, w, k, r, keep, Mk, ne, g, one, cg_cap2);
    L.stream = saved;
    cudaError_t e = cudaStreamEndCapture(cg_cap, &graph);
    const unsigned long dm = mvm_count() - m0;
    mvm_restore(m0);  // nothing ran yet
    if (rc) {
      if (graph) cudaGraphDestroy(graph);
      return rc;
    }
    if (e != cudaSuccess) return fail_cuda(e, "cg capture", __FILE__, __LINE__);
    e = cudaGraphInstantiate(&c.exec, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) {
      c.exec = nullptr;
      return fail_cuda(e, "cg graph instantiate", __FILE__, __LINE__);
    }
    c.op = op;
    c.mass = mass;
    c.force = L.hop_force;
    c.flt_links = L.flt_links;
    c.pdl = (int)L.hop_pdl;
    c.recon = recon;
    c.one = one;
    c.keep = keep;
    c.both = both;
    for (int i = 0; i < 3; i++) c.v[i] = L.hop_variant[pi][i];
    for (int i = 0; i < 9 + CG_CHUNK; i++) c.ptrs[i] = ptrs[i];
    c.mvm = dm;
  }
  HR_CUDA(cudaGraphLaunch(c.exec, L.stream));
  *mvm = c.mvm;
  return 0;
}

// cg_mshift_core (cg_mshift.c:24-145) / cg_mshift_flt_core (cg_mshift_flt.c:22-140).
// out[i] are fields of precision `prec`; flags[i] in/out (flt: read only).
// Returns the iteration count, or a negative status.
template <typename R>
static int cg_core(int op, double mass, int n, const double *shift, double err2, int max_iter, const void *in,
                   void *const *out, int *flags, int flt, int *iters) {
  typedef typename C2<R>::T V;
  const int prec = sizeof(R) == 8 ? HRGPU_DOUBLE : HRGPU_FLOAT;
  const int par = op_parity(op);
  const size_t bytes = spinor_bytes(par, prec);
  const long ne = (long)spinor_elems(par);
  if (int rc = cg_workspace(prec, n + 3, bytes)) return rc;
  CGWork &w = W[prec];
  void *k = w.bufs[n], *r = w.bufs[n + 1], *Mk = w.bufs[n + 2];
  int cgiter = 0;
  double innorm2;
  if (int rc = la_dot(2, par, prec, in, nullptr, &innorm2)) return rc;
  if (!isfinite(innorm2)) {
    *iters = 0;
    set_error("cg_mshift: the source norm is not finite (%g)", innorm2);
    return HRGPU_E_BREAKDOWN;
  }
  if (innorm2 == 0.0) {  // (M - s_i) x = 0: every solution is zero, nothing to iterate
    for (int i = 0; i < n; i++) HR_CUDA(cudaMemsetAsync(out[i], 0, bytes, L.stream));
    *iters = 0;
    return 0;
  }
  if (n == 1) {
    // out[0] is the initial guess
    if (int rc = apply_op(op, prec, mass, Mk, out[0])) return rc;
    ++cgiter;
    if (int rc = la_op(LA_MUL_ADD_ASSIGN, par, prec, Mk, out[0], nullptr, -shift[0], 0, 0, 0)) return rc;
    if (int rc = la_op(LA_SUB, par, prec, r, in, Mk, 0, 0, 0, 0)) return rc;
  } else {
    HR_CUDA(cudaMemcpyAsync(r, in, bytes, cudaMemcpyDeviceToDevice, L.stream));
  }
  HR_CUDA(cudaMemcpyAsync(k, r, bytes, cudaMemcpyDeviceToDevice, L.stream));
  double delta;
  if (int rc = la_dot(2, par, prec, r, nullptr, &delta)) return rc;
  for (int i = 0; i < n; i++) {
    HR_CUDA(cudaMemcpyAsync(w.bufs[i], r, bytes, cudaMemcpyDeviceToDevice, L.stream));
    if (n != 1) HR_CUDA(cudaMemsetAsync(out[i], 0, bytes, L.stream));
  }
  // (la_dot above has waited for the stream, so no copy into hS is in flight)
  CGState &h0 = w.hS[0];
  memset(&h0, 0, sizeof(CGState));
  h0.omega = 1.0;
  h0.gamma = 0.0;
  h0.delta = delta;
  h0.innorm2 = innorm2;
  h0.err2 = err2;
  h0.n = n;
  h0.state = 0;
  h0.iter = 0;
  h0.max_iter = max_iter == 0 ? CG_HARD_LIMIT : (max_iter > cgiter ? max_iter - cgiter : 1);
  h0.flt = flt;
  for (int i = 0; i < n; i++) {
    h0.shift[i] = shift[i];
    h0.z1[i] = h0.z2[i] = 1.0;
    h0.z3[i] = 0.0;
    h0.flag[i] = flt ? flags[i] : 1;
  }
  HR_CUDA(cudaMemcpyAsync(w.S, &h0, sizeof(CGState), cudaMemcpyHostToDevice, L.stream));
  void *ptrs[2 * MAXS];
  for (int i = 0; i < n; i++) {
    ptrs[i] = out[i];
    ptrs[MAXS + i] = w.bufs[i];
  }
  HR_CUDA(cudaMemcpyAsync(w.d_ptrs, ptrs, sizeof(void *) * 2 * MAXS, cudaMemcpyHostToDevice, L.stream));
  const unsigned g = red_grid(ne);
  const int one = n == 1 && shift[0] == 0.0;
  // residuals of the last CG_CHUNK iterations where the shifted systems can wait for them
  void *ring[CG_CHUNK] = {r, r, r, r};
  const int keep = !one && cg_more_residuals(w, n + 3) ? CG_CHUNK : 1;
  if (keep > 1)
    for (int c = 0; c < CG_CHUNK - 1; c++) ring[c] = w.bufs[n + 3 + c];  // the first is in ring[CG_CHUNK - 1] = r
  L.cur_stop = &w.S->state;
  int rc = 0;
  // one chunk is in flight behind the one whose state is read; the kernels of a
  // chunk that follows the last iteration return at once and its hops are not counted
  unsigned long mvm[2] = {0, 0};
  auto launch = [&](int b) -> int {
    if (int q = cg_chunk<R>(op, prec, mass, w, k, ring, keep, Mk, ne, g, one, &mvm[b])) return q;
    HR_CUDA(cudaMemcpyAsync(&w.hS[b], w.S, offsetof(CGState, cx), cudaMemcpyDeviceToHost, L.stream));
    HR_CUDA(cudaEventRecord(w.ev[b], L.stream));
    return 0;
  };
  rc = launch(0);
  int cur = 0;
  while (!rc) {
    rc = launch(cur ^ 1);
    if (rc) break;
    cudaError_t e = cudaEventSynchronize(w.ev[cur]);
    if (e != cudaSuccess) {
      rc = fail_cuda(e, "cg state readback", __FILE__, __LINE__);
      break;
    }
    add_mvm(mvm[cur]);
    if (w.hS[cur].state != 0) break;
    cur ^= 1;
  }
  L.cur_stop = nullptr;
  if (rc) return rc;
  const CGState &h = w.hS[cur];
  cgiter += h.iter;
  // coefficients that were not finite may have reached the padding
  auto clear_padding = [&]() -> int {
    for (void *b : w.bufs) HR_CUDA(cudaMemsetAsync(b, 0, bytes, L.stream));
    return 0;
  };
  if (h.state == 3) {
    if (int q = clear_padding()) return q;
    *iters = cgiter;
    set_error("cg_mshift: breakdown at iteration %d (alpha=%g, |r|^2=%g)", cgiter, h.alpha, h.lambda);
    return HRGPU_E_BREAKDOWN;
  }
  if (!flt) {
    // true residual of every shift (cg_mshift.c:122-137)
    for (int i = 0; i < n; i++) {
      if (int q = apply_op(op, prec, mass, Mk, out[i])) return q;
      ++cgiter;
      if (int q = la_op(LA_MUL_ADD_ASSIGN, par, prec, Mk, out[i], nullptr, -shift[i], 0, 0, 0)) return q;
      if (int q = la_op(LA_SUB_ASSIGN, par, prec, Mk, in, nullptr, 0, 0, 0, 0)) return q;
      double nr;
      if (int q = la_dot(2, par, prec, Mk, nullptr, &nr)) return q;
      if (!isfinite(nr)) {
        if (int q = clear_padding()) return q;
        *iters = cgiter;
        set_error("cg_mshift: the true residual of shift %d is not finite (%g)", i, nr);
        return HRGPU_E_BREAKDOWN;
      }
      flags[i] = (fabs(nr / innorm2) > err2) ? 0 : 1;
    }
  }
  *iters = cgiter;
  return 0;
}

static int cg_check(int op, int n, const double *shift, const void *in, void *const *out, int *iters) {
  HR_REQUIRE(L.ready, HRGPU_E_STATE, "cg_mshift: lattice not initialised");
  HR_REQUIRE(op >= 0 && op <= 3, HRGPU_E_ARG, "cg_mshift: unknown operator %d", op);
  HR_REQUIRE(n > 0 && n <= MAXS, HRGPU_E_ARG, "cg_mshift: n = %d shifts (1..%d supported)", n, MAXS);
  HR_REQUIRE(shift && in && out && iters, HRGPU_E_ARG, "cg_mshift: NULL argument");
  for (int i = 0; i < n; i++) HR_REQUIRE(out[i] != nullptr && out[i] != in, HRGPU_E_ARG, "cg_mshift: bad output field");
  return 0;
}

}  // namespace hrgpu

using namespace hrgpu;

extern "C" {

int hrgpu_cg_mshift(int op, double mass, int n, const double *shift, double err2, int max_iter, const void *in,
                    void *const *out, int *iters) {
  if (int rc = cg_check(op, n, shift, in, out, iters)) return rc;
  std::vector<int> flags(n, 1);
  int total = 0, it = 0;
  if (int rc = cg_core<double>(op, mass, n, shift, err2, max_iter, in, out, flags.data(), 0, &it)) return rc;
  total += it;
  // unconverged shifts are solved again one at a time from their current solution
  // (cg_mshift.c:170-179); bounded here so a hopeless system returns instead of looping
  int status = 0;
  for (int i = 0; i < n; i++) {
    int rep = 0;
    while (flags[i] == 0) {
      if (++rep > 20) {
        status = HRGPU_E_NOCONV;
        set_error("cg_mshift: shift %d did not reach err2=%g after %d restarts", i, err2, rep - 1);
        break;
      }
      void *o[1] = {out[i]};
      if (int rc = cg_core<double>(op, mass, 1, shift + i, err2, max_iter, in, o, &flags[i], 0, &it)) return rc;
      total += it;
    }
  }
  *iters = total;
  return status;
}

// cg_mshift_flt (cg_mshift_flt.c:144-276)
int hrgpu_cg_mshift_flt(int op, double mass, int n, const double *shift, double err2, int max_iter, const void *in,
                        void *const *out, int *iters) {
  if (int rc = cg_check(op, n, shift, in, out, iters)) return rc;
  HR_REQUIRE(op != HRGPU_OP_G5CPHI_SQ, HRGPU_E_ARG, "cg_mshift_flt: no float version of g5Cphi_sq");
  const int par = op_parity(op);
  const size_t bd = spinor_bytes(par, HRGPU_DOUBLE), bf = spinor_bytes(par, HRGPU_FLOAT);
  if (FW.bd != bd) {
    cudaFree(FW.dres); cudaFree(FW.dres2); cudaFree(FW.dtmp);
    HR_CUDA(cudaMalloc(&FW.dres, bd));
    HR_CUDA(cudaMalloc(&FW.dres2, bd));
    HR_CUDA(cudaMalloc(&FW.dtmp, bd));
    for (void *b : {FW.dres, FW.dres2, FW.dtmp}) HR_CUDA(cudaMemsetAsync(b, 0, bd, L.stream));
    FW.bd = bd;
  }
  if (FW.bf != bf) {
    for (void *b : FW.fbuf) cudaFree(b);
    FW.fbuf.clear();
    FW.bf = bf;
  }
  while ((int)FW.fbuf.size() < n + 1) {
    void *b;
    HR_CUDA(cudaMalloc(&b, bf));
    FW.fbuf.push_back(b);
    HR_CUDA(cudaMemsetAsync(b, 0, bf, L.stream));
  }
  void *dres = FW.dres, *dres2 = FW.dres2, *dtmp = FW.dtmp;
  std::vector<void *> &fbuf = FW.fbuf;
  void *res_flt = fbuf[0];
  std::vector<void *> out_flt(fbuf.begin() + 1, fbuf.begin() + 1 + n);
  std::vector<int> sflags(n, 1), loc(n);
  std::vector<double> norm(n, 0.0);
  for (int i = 0; i < n; i++)
    if (n != 1) HR_CUDA(cudaMemsetAsync(out[i], 0, bd, L.stream));
  double innorm2;
  if (int rc = la_dot(2, par, HRGPU_DOUBLE, in, nullptr, &innorm2)) return rc;
  if (!isfinite(innorm2)) {
    *iters = 0;
    set_error("cg_mshift_flt: the source norm is not finite (%g)", innorm2);
    return HRGPU_E_BREAKDOWN;
  }
  if (innorm2 == 0.0) {
    for (int i = 0; i < n; i++) HR_CUDA(cudaMemsetAsync(out[i], 0, bd, L.stream));
    *iters = 0;
    return 0;
  }
  int siter = 0, diter = 0, notconverged, rounds = 0;
  const double mass_d = mass;
  do {
    int first = 1;
    notconverged = 0;
    double local_err2 = err2;
    for (int i = 0; i < n; i++) {
      if (!sflags[i]) continue;
      if (int rc = apply_op(op, HRGPU_DOUBLE, mass_d, dtmp, out[i])) return rc;
      ++diter;
      if (int rc = la_op(LA_SUB, par, HRGPU_DOUBLE, dres2, in, dtmp, 0, 0, 0, 0)) return rc;
      if (int rc = la_op(LA_MUL_ADD_ASSIGN, par, HRGPU_DOUBLE, dres2, out[i], nullptr, shift[i], 0, 0, 0)) return rc;
      if (int rc = la_dot(2, par, HRGPU_DOUBLE, dres2, nullptr, &norm[i])) return rc;
      if (!isfinite(norm[i])) {
        *iters = siter + diter;
        set_error("cg_mshift_flt: the residual of shift %d is not finite (%g)", i, norm[i]);
        return HRGPU_E_BREAKDOWN;
      }
      if (norm[i] < innorm2 * err2) {
        sflags[i] = 0;
        norm[i] /= innorm2;
      } else {
        ++notconverged;
        if (first) {
          first = 0;
          local_err2 = norm[i] / innorm2;
          norm[i] = sqrt(norm[i]);
          if (int rc = la_op(LA_MUL, par, HRGPU_DOUBLE, dres, dres2, nullptr, 1. / norm[i], 0, 0, 0)) return rc;
        } else {
          double pr[2];
          if (int rc = la_dot(0, par, HRGPU_DOUBLE, dres, dres2, pr)) return rc;
          norm[i] = pr[0];
        }
      }
    }
    if (notconverged) {
      if (int rc = hrgpu_assign_sd2s(res_flt, dres, par)) return rc;
      local_err2 = err2 / local_err2 * 0.9;
      if (local_err2 < 1.e-10) local_err2 = 1.e-10;
      for (int i = 0; i < n; i++) loc[i] = sflags[i];
      // a single shift starts the inner solve from out_flt[0]: start from zero
      if (n == 1) HR_CUDA(cudaMemsetAsync(out_flt[0], 0, bf, L.stream));
      int it = 0;
      if (int rc = cg_core<float>(op, mass_d, n, shift, local_err2, max_iter, res_flt, out_flt.data(), loc.data(), 1, &it))
        return rc;
      siter += it;
      for (int i = 0; i < n; i++)
        if (sflags[i]) {
          if (int rc = hrgpu_assign_s2sd(dres2, out_flt[i], par)) return rc;
          if (int rc = la_op(LA_MUL_ADD_ASSIGN, par, HRGPU_DOUBLE, out[i], dres2, nullptr, norm[i], 0, 0, 0)) return rc;
        }
    }
    if (++rounds > 200) {
      *iters = siter + diter;
      set_error("cg_mshift_flt: no convergence to err2=%g after %d defect-correction rounds", err2, rounds);
      return HRGPU_E_NOCONV;
    }
  } while (notconverged);
  *iters = siter + diter;
  return 0;
}

}  // extern "C"
