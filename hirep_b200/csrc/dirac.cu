// dirac.cu -- Wilson / clover Dirac operators on the device (LibHR/Update/Dphi.c,
// Dphi_flt.c, D_update.c), built from the fused hopping kernel in hop.cuh.
#include "dirac.cuh"
#include "hop_dir.cuh"

namespace hrgpu {

template <typename R, int EP>
int launch_ep(HopArgs<R> &a);  // hop_launch.cuh, instantiated in dirac_{d,f}_ep*.cu

template <typename R>
int launch_hop(int ep, HopArgs<R> &a) {
  if (ep == EP_AXPY) return launch_ep<R, EP_AXPY>(a);
  if (ep == EP_CLOV_INV) return launch_ep<R, EP_CLOV_INV>(a);
  return launch_ep<R, EP_CLOV>(a);
}
template int launch_hop<double>(int, HopArgs<double> &);
template int launch_hop<float>(int, HopArgs<float> &);

static unsigned long g_mvm = 0;
static double g_static_mass = 0.0;

template <typename R>
static const void *links() {
  if (sizeof(R) == 8) return L.U;
  return L.flt_links == HRGPU_LINKS_BF16 ? L.Ubf : L.Uf;
}

template <typename R>
static int hop_args(HopArgs<R> &a, int outp, void *out, const void *in, double cacc, const void *aux, double caux, int g5,
                    double *red, const R *cdg, const typename C2<R>::T *cod, int cb0, int cb1, const HopTail *tail) {
  a.cb0 = cb0;
  a.cb1 = cb1;
  a.in = in;
  a.out = out;
  a.U = links<R>();
  a.aux = aux;
  a.cdg = cdg;
  a.cod = cod;
  a.red = red;
  a.cacc = (R)cacc;
  a.caux = (R)caux;
  a.outp = outp;
  a.g5 = g5;
  a.stop = L.cur_stop;
  a.err = nullptr;
  a.both = 0;
  a.pre = tail ? tail->pre : 0;
  a.racc = tail ? tail->racc : nullptr;
  a.omega = tail ? tail->omega : nullptr;
  a.red_g5 = tail ? tail->red_g5 : 0;
  a.no_pdl = tail ? tail->no_pdl : 0;
  a.Ug = sizeof(R) == 8 ? (const void *)L.Ug : (const void *)L.Ugf;
  if (sizeof(R) == 4 && L.flt_links == HRGPU_LINKS_BF16) {
    if (int rc = ensure_links_bf16()) return rc;
    a.U = L.Ubf;
  }
  return 0;
}

// one hop onto parity outp with the given epilogue; fields are parity fields
template <typename R>
int hop(int outp, void *out, const void *in, int ep, double cacc, const void *aux, double caux, int g5, double *red,
        const R *cdg, const typename C2<R>::T *cod, int cb0, int cb1, const HopTail *tail) {
  HopArgs<R> a;
  if (cb1 < 0) cb1 = (int)L.VH;
  if (cb1 <= cb0) return 0;
  if (int rc = hop_args<R>(a, outp, out, in, cacc, aux, caux, g5, red, cdg, cod, cb0, cb1, tail)) return rc;
  if (cb0 == 0 && cb1 == (int)L.VH) g_mvm++;  // partial launches are counted by their caller
  return launch_hop<R>(ep, a);
}
template int hop<double>(int, void *, const void *, int, double, const void *, double, int, double *, const double *,
                         const double2 *, int, int, const HopTail *);
template int hop<float>(int, void *, const void *, int, double, const void *, double, int, double *, const float *,
                        const float2 *, int, int, const HopTail *);

static int tune_slot(int prec) { return prec == HRGPU_DOUBLE ? 0 : (L.flt_links == HRGPU_LINKS_BF16 ? 2 : 1); }

static int last_hop_variant(int ep, int prec) { return L.hop_force >= 0 ? L.hop_force : L.hop_variant[tune_slot(prec)][ep]; }

// whether candidates may be timed now: nothing is forced, and no stream capture is on
static bool can_tune() {
  if (L.hop_force >= 0) return false;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(L.stream, &cs) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return cs == cudaStreamCaptureStatusNone;
}

// milliseconds of run() on the GPU: the launches queue up behind a delay, since they cost the
// host as much as the hops of a small lattice take.  The events resolve half a microsecond, so
// a short run is repeated more often.
template <typename F>
static int time_launches(F &&run, float *ms) {
  cudaEvent_t e[2] = {nullptr, nullptr};
  int rc = 0;
  if (cudaEventCreate(&e[0]) != cudaSuccess || cudaEventCreate(&e[1]) != cudaSuccess)
    rc = fail_cuda(cudaGetLastError(), "cudaEventCreate", __FILE__, __LINE__);
  for (int reps = 3; !rc; reps = 10) {
    rc = stream_delay(reps == 3 ? 30.0 : 80.0);
    if (!rc) rc = run();
    if (!rc && cudaEventRecord(e[0], L.stream) != cudaSuccess) rc = fail_cuda(cudaGetLastError(), "cudaEventRecord", __FILE__, __LINE__);
    for (int r = 0; r < reps && !rc; r++) rc = run();
    if (!rc && (cudaEventRecord(e[1], L.stream) != cudaSuccess || cudaEventSynchronize(e[1]) != cudaSuccess ||
                cudaEventElapsedTime(ms, e[0], e[1]) != cudaSuccess))
      rc = fail_cuda(cudaGetLastError(), "hop timing", __FILE__, __LINE__);
    *ms /= reps;
    if (reps > 3 || *ms > 0.05f) break;
  }
  for (cudaEvent_t ev : e)
    if (ev) cudaEventDestroy(ev);
  return rc;
}

// run() timed with each variant for epilogue ep's hop (and too's, where not negative):
// milliseconds, -1 where a variant is not built or not applicable
template <typename F>
static int time_variants(int pi, int ep, int too, F &&run) {
  float *t = L.hop_tune_ms[pi][ep];
  for (int v = 0; v < HOP_VARIANTS; v++) {
    t[v] = -1.0f;
    // 5 is slower in every measured case, 6 runs as 0 while the links are not known to come from the fundamental ones
    if (v == 5 || (v == 6 && (L.recon12 < 3 || !L.recon_allow))) continue;
    L.hop_variant[pi][ep] = v;
    if (too >= 0) L.hop_variant[pi][too] = v;
    int rc = run();
    if (rc == HRGPU_E_NF && v > 0) continue;  // not built for this NF
    if (!rc) rc = time_launches(run, &t[v]);
    if (rc) return rc;
  }
  return 0;
}

// The variants of an even-odd operator's two hops by the time run(), which launches both, takes:
// how well a hop follows another (what the blocks of the next launch find free, what the
// second hop reads before the first has ended) differs between variants.  The same variant
// for both hops first: 0 unless another one saves 2 % (a step with the operands out of L2
// favours it slightly over the register-capped ones), and the spin split (3) only where it saves
// 6 % over the rest (inside a solve it gains less: g5QMR with clover, SU(4) on 6x10x12x16,
// took 2 % more with it than with 1 where the pair read less).  A second one beside it only where that saves 2 % (sextet clover at
// 48x24^3: 763 us with 6 and 1, 860 and 868 with one of them), or 8 % of less than 100 us: the
// gaps between short launches are others behind other kernels than back to back (g5QMR
// with clover, SU(3) on 12x6x14x10: 1 and 3 read 6 % faster than 1 and 1, and the solve took
// 2 % more).
template <typename F>
static int tune_pair(int pi, int ep0, int ep1, F &&run) {
  int &v0 = L.hop_variant[pi][ep0], &v1 = L.hop_variant[pi][ep1];
  const float *t0 = L.hop_tune_ms[pi][ep0], *t1 = L.hop_tune_ms[pi][ep1];
  auto best_of = [](const float *t, int from, float f) {
    int b = from;
    for (int c : {0, 1, 2, 4, 6, 3})
      if (t[c] > 0.0f && t[c] < t[b]) b = c;
    return t[b] < f * t[from] ? b : from;
  };
  if (int rc = time_variants(pi, ep1, ep0, run)) return rc;
  int u = 0;
  for (int c : {1, 2, 4, 6})
    if (t1[c] > 0.0f && t1[c] < t1[u]) u = c;
  if (t1[u] > 0.98f * t1[0]) u = 0;
  if (t1[3] > 0.0f && t1[3] < 0.94f * t1[u]) u = 3;
  v0 = v1 = u;
  if (ep0 == ep1) return 0;
  if (int rc = time_variants(pi, ep1, -1, run)) return rc;
  const float f = t1[u] > 0.1f ? 0.98f : 0.92f;
  v1 = best_of(t1, u, f);
  if (int rc = time_variants(pi, ep0, -1, run)) return rc;
  v0 = best_of(t0, u, v1 == u ? f : 0.98f);
  return 0;
}

// the hop onto both parities of a full field: one launch of variant 1, which takes both (a
// small lattice then fills twice the SMs), or one per parity, whichever took less time
template <typename R>
static int hop_full(void *out, const void *in, int ep, double cacc, const void *aux, double caux, int g5, const R *cdg,
                    const typename C2<R>::T *cod) {
  const int prec = sizeof(R) == 8 ? HRGPU_DOUBLE : HRGPU_FLOAT, pi = tune_slot(prec);
  const size_t half = (size_t)4 * L.nf * L.ld * sizeof(typename C2<R>::T);
  auto one_launch = [&]() -> int {
    HopArgs<R> a;
    if (int rc = hop_args<R>(a, HRGPU_EVEN, out, in, cacc, aux, caux, g5, nullptr, cdg, cod, 0, (int)L.VH, nullptr)) return rc;
    a.both = 1;
    g_mvm += 2;
    const int force = L.hop_force;
    L.hop_force = 1;
    const int rc = launch_hop<R>(ep, a);
    L.hop_force = force;
    return rc;
  };
  auto two_launches = [&]() -> int {
    for (int p = 0; p < 2; p++)
      if (int rc = hop<R>(p, (char *)out + p * half, (const char *)in + (p ^ 1) * half, ep, cacc,
                          aux ? (const char *)aux + p * half : nullptr, caux, g5, nullptr, cdg, cod))
        return rc;
    return 0;
  };
  if (L.nf > 6) return two_launches();
  int &both = L.hop_both[pi][ep];
  if (both < 0 && can_tune()) {
    const unsigned long m0 = g_mvm;
    float t1 = 0, t2 = 0;
    int rc = two_launches();  // tunes the hop onto one parity
    if (!rc) rc = time_launches(two_launches, &t2);
    if (!rc) rc = time_launches(one_launch, &t1);
    g_mvm = m0;
    if (rc) return rc;
    both = t1 < t2;
  }
  const bool b = L.hop_force >= 0 || both < 0 ? last_hop_variant(ep, prec) == 1 : both == 1;
  return b ? one_launch() : two_launches();
}

int check_gauge(int prec) {
  HR_REQUIRE(L.ready, HRGPU_E_STATE, "lattice not initialised");
  if (prec == HRGPU_DOUBLE) HR_REQUIRE(L.have_gauge, HRGPU_E_STATE, "no gauge field set");
  else HR_REQUIRE(L.have_gauge_flt, HRGPU_E_STATE, "no float gauge field set");
  return 0;
}

// Dphi_ on parity or full fields
template <typename R>
int Dphi_hop(void *out, int out_par, const void *in) {
  if (int rc = check_gauge(sizeof(R) == 8 ? HRGPU_DOUBLE : HRGPU_FLOAT)) return rc;
  HR_REQUIRE(out && in && out != in, HRGPU_E_ARG, "Dphi_: input and output fields must be different");
  HR_REQUIRE(out_par >= 0 && out_par <= 2, HRGPU_E_ARG, "Dphi_: bad parity");
  if (out_par == HRGPU_FULL) {
    if (int rc = hop_full<R>(out, in, EP_AXPY, -0.5, nullptr, 0.0, 0, nullptr, nullptr)) return rc;
    g_mvm++;  // a full-lattice application counts twice (Dphi.c:205-207)
    return 0;
  }
  return hop<R>(out_par, out, in, EP_AXPY, -0.5, nullptr, 0.0, 0, nullptr, nullptr, nullptr);
}

// full lattice: out = -1/2 H in + (4+m) in, optionally gamma_5 (Dphi / g5Dphi)
template <typename R>
int Dphi_full(double m0, void *out, const void *in, int g5) {
  if (int rc = check_gauge(sizeof(R) == 8 ? HRGPU_DOUBLE : HRGPU_FLOAT)) return rc;
  HR_REQUIRE(out && in && out != in, HRGPU_E_ARG, "Dphi: input and output fields must be different");
  return hop_full<R>(out, in, EP_AXPY, -0.5, in, 4.0 + m0, g5, nullptr, nullptr);
}

// one hop of an even-odd preconditioned operator with output parity p, on the
// output sites cb0 <= cb < cb1 of its parity:
//   stage 0: tmp = D_qp in on parity q = 1-p (clover: times D_qq^-1)
//   stage 1: out = rho in + 1/2 D_pq tmp with rho = (4+m)^2 (Wilson), or
//            D_pp in + 1/2 D_pq tmp (clover), optionally times gamma_5.
// Stage 1 on a range needs stage 0 done on the neighbouring range (one site
// further in every direction).
//
// The variants of the two hops are chosen (tune_pair) when the second one first runs on the
// whole parity.
template <typename R>
int eo_stage(int clover, double mass, int stage, int outp, void *out, const void *in, int g5, double *red, int cb0,
             int cb1, const HopTail *tail) {
  void **tmp = sizeof(R) == 8 ? &L.tmp_o : &L.tmp_o_f;
  if (int rc = ensure_tmp(tmp, spinor_bytes(HRGPU_EVEN, sizeof(R) == 8 ? HRGPU_DOUBLE : HRGPU_FLOAT))) return rc;
  const int pi = tune_slot(sizeof(R) == 8 ? HRGPU_DOUBLE : HRGPU_FLOAT);
  const int ep0 = clover ? EP_CLOV_INV : EP_AXPY, ep1 = clover ? EP_CLOV : EP_AXPY;
  bool &tuned = L.hop_pair_tuned[pi][clover ? 1 : 0];
  if (!tuned && !tail && cb0 == 0 && (cb1 < 0 || cb1 == (int)L.VH) && can_tune()) {
    if (stage == 0) {
      if (L.hop_variant[pi][ep0] < 0) L.hop_variant[pi][ep0] = 0;  // until the second hop
    } else {
      const unsigned long m0 = g_mvm;
      tuned = true;
      auto pair = [&]() -> int {
        if (int rc = eo_stage<R>(clover, mass, 0, outp, out, in, g5, nullptr, cb0, cb1, nullptr)) return rc;
        return eo_stage<R>(clover, mass, 1, outp, out, in, g5, red, cb0, cb1, nullptr);
      };
      int rc = tune_pair(pi, ep0, ep1, pair);
      if (!rc) rc = eo_stage<R>(clover, mass, 0, outp, out, in, g5, nullptr, cb0, cb1, nullptr);
      g_mvm = m0;
      if (rc) {
        tuned = false;
        L.hop_variant[pi][ep0] = L.hop_variant[pi][ep1] = -1;
        return rc;
      }
    }
  }
  // the second hop follows the first, which has waited for whatever made the links,
  // the clover blocks and in
  HopTail ht;
  if (tail) ht = *tail;
  ht.pre = 1;
  tail = stage ? &ht : nullptr;
  if (clover) {
    const R *idg, *ddg;
    const typename C2<R>::T *iod, *dod;
    clover_blocks<R>(&ddg, &dod, &idg, &iod);
    if (stage == 0) return hop<R>(outp ^ 1, *tmp, in, EP_CLOV_INV, -0.5, nullptr, 0.0, 0, nullptr, idg, iod, cb0, cb1);
    return hop<R>(outp, out, *tmp, EP_CLOV, 0.5, in, 0.0, g5, red, ddg, dod, cb0, cb1, tail);
  }
  if (stage == 0) return hop<R>(outp ^ 1, *tmp, in, EP_AXPY, -0.5, nullptr, 0.0, 0, nullptr, nullptr, nullptr, cb0, cb1);
  double rho = 4.0 + mass;
  if (sizeof(R) == 4) {
    float r = 4.f + (float)mass;
    rho = (double)(r * r);
  } else {
    rho = rho * rho;
  }
  return hop<R>(outp, out, *tmp, EP_AXPY, 0.5, in, rho, g5, red, nullptr, nullptr, cb0, cb1, tail);
}
template int eo_stage<double>(int, double, int, int, void *, const void *, int, double *, int, int, const HopTail *);
template int eo_stage<float>(int, double, int, int, void *, const void *, int, double *, int, int, const HopTail *);

// even-odd: out = (4+m)^2 in - D_pq D_qp in on parity p, optionally gamma_5
template <typename R>
int Dphi_eo(double m0, void *out, const void *in, int outp, int g5, double *red, const HopTail *tail) {
  if (int rc = check_gauge(sizeof(R) == 8 ? HRGPU_DOUBLE : HRGPU_FLOAT)) return rc;
  HR_REQUIRE(out && in && out != in, HRGPU_E_ARG, "Dphi_eopre: input and output fields must be different");
  if (int rc = eo_stage<R>(0, m0, 0, outp, out, in, g5, nullptr, 0, -1)) return rc;
  return eo_stage<R>(0, m0, 1, outp, out, in, g5, red, 0, -1, tail);
}

template int Dphi_eo<double>(double, void *, const void *, int, int, double *, const HopTail *);
template int Dphi_eo<float>(double, void *, const void *, int, int, double *, const HopTail *);

// ------------------------------------------------------------------ clover
template <typename R>
int Cphi_eo(double mass, void *out, const void *in, int g5, double *red, const HopTail *tail) {
  if (int rc = check_gauge(sizeof(R) == 8 ? HRGPU_DOUBLE : HRGPU_FLOAT)) return rc;
  HR_REQUIRE(L.clover, HRGPU_E_STATE, "Cphi_eopre: no clover term (hrgpu_clover_init)");
  HR_REQUIRE(out && in && out != in, HRGPU_E_ARG, "Cphi_eopre: input and output fields must be different");
  if (int rc = clover_prepare(mass, sizeof(R) == 8 ? HRGPU_DOUBLE : HRGPU_FLOAT)) return rc;
  if (int rc = eo_stage<R>(1, mass, 0, HRGPU_EVEN, out, in, g5, nullptr, 0, -1)) return rc;
  return eo_stage<R>(1, mass, 1, HRGPU_EVEN, out, in, g5, red, 0, -1, tail);
}
template int Cphi_eo<double>(double, void *, const void *, int, double *, const HopTail *);
template int Cphi_eo<float>(double, void *, const void *, int, double *, const HopTail *);

static int Cphi_full(double mass, void *out, const void *in, int g5) {
  if (int rc = check_gauge(HRGPU_DOUBLE)) return rc;
  HR_REQUIRE(L.clover, HRGPU_E_STATE, "Cphi: no clover term (hrgpu_clover_init)");
  HR_REQUIRE(out && in && out != in, HRGPU_E_ARG, "Cphi: input and output fields must be different");
  if (int rc = clover_prepare(mass, HRGPU_DOUBLE)) return rc;
  const double *idg, *ddg;
  const double2 *iod, *dod;
  clover_blocks<double>(&ddg, &dod, &idg, &iod);
  return hop_full<double>(out, in, EP_CLOV, -0.5, in, 0.0, g5, ddg, dod);
}

template <typename R>
static int sq(int (*op)(double, void *, const void *, int), double m, void *out, const void *in, int par) {
  void **tmp = par == HRGPU_FULL ? (sizeof(R) == 8 ? &L.tmp_full : &L.tmp_full_f) : (sizeof(R) == 8 ? &L.tmp_e : &L.tmp_e_f);
  if (int rc = ensure_tmp(tmp, spinor_bytes(par, sizeof(R) == 8 ? HRGPU_DOUBLE : HRGPU_FLOAT))) return rc;
  if (int rc = op(m, *tmp, in, 1)) return rc;
  return op(m, out, *tmp, 1);
}

static int op_Dfull_d(double m, void *o, const void *i, int g5) { return Dphi_full<double>(m, o, i, g5); }
static int op_Dfull_f(double m, void *o, const void *i, int g5) { return Dphi_full<float>(m, o, i, g5); }
static int op_eo_d(double m, void *o, const void *i, int g5) { return Dphi_eo<double>(m, o, i, HRGPU_EVEN, g5, nullptr); }
static int op_eo_f(double m, void *o, const void *i, int g5) { return Dphi_eo<float>(m, o, i, HRGPU_EVEN, g5, nullptr); }
static int op_ceo_d(double m, void *o, const void *i, int g5) { return Cphi_eo<double>(m, o, i, g5, nullptr); }
static int op_ceo_f(double m, void *o, const void *i, int g5) { return Cphi_eo<float>(m, o, i, g5, nullptr); }
static int op_cfull_d(double m, void *o, const void *i, int g5) { return Cphi_full(m, o, i, g5); }

// operator used by the inverters: M = op(mass) on fields of the returned parity
int apply_op(int op, int prec, double mass, void *out, const void *in) {
  if (prec == HRGPU_DOUBLE) {
    switch (op) {
      case HRGPU_OP_G5DPHI_SQ: return sq<double>(op_Dfull_d, mass, out, in, HRGPU_FULL);
      case HRGPU_OP_G5DPHI_EOPRE_SQ: return sq<double>(op_eo_d, mass, out, in, HRGPU_EVEN);
      case HRGPU_OP_G5CPHI_EOPRE_SQ: return sq<double>(op_ceo_d, mass, out, in, HRGPU_EVEN);
      case HRGPU_OP_G5CPHI_SQ: return sq<double>(op_cfull_d, mass, out, in, HRGPU_FULL);
      case HRGPU_OP_DPHI_EOPRE: return op_eo_d(mass, out, in, 0);
      case HRGPU_OP_G5DPHI_EOPRE: return op_eo_d(mass, out, in, 1);
      case HRGPU_OP_CPHI_EOPRE: return op_ceo_d(mass, out, in, 0);
      case HRGPU_OP_G5CPHI_EOPRE: return op_ceo_d(mass, out, in, 1);
      case HRGPU_OP_DPHI: return op_Dfull_d(mass, out, in, 0);
      case HRGPU_OP_CPHI: return op_cfull_d(mass, out, in, 0);
    }
  } else {
    switch (op) {
      case HRGPU_OP_G5DPHI_SQ: return sq<float>(op_Dfull_f, mass, out, in, HRGPU_FULL);
      case HRGPU_OP_G5DPHI_EOPRE_SQ: return sq<float>(op_eo_f, mass, out, in, HRGPU_EVEN);
      case HRGPU_OP_G5CPHI_EOPRE_SQ: return sq<float>(op_ceo_f, mass, out, in, HRGPU_EVEN);
      default: break;
    }
  }
  set_error("operator %d has no %s version", op, prec == HRGPU_DOUBLE ? "double" : "float");
  return HRGPU_E_ARG;
}

int hop_red_blocks(bool clover, int prec) {
  int v = last_hop_variant(clover ? EP_CLOV : EP_AXPY, prec);
  if (v == 6 && L.hop_force < 0 && (L.recon12 < 3 || !L.recon_allow)) v = 0;  // what the launcher then runs
  return v < 0 ? 0 : hop_blocks(v, L.VH, L.nf);
}

bool op_tuned(int op, int prec) {
  if (L.hop_force >= 0) return true;
  const bool clover = op == HRGPU_OP_G5CPHI_EOPRE_SQ || op == HRGPU_OP_G5CPHI_SQ || op == HRGPU_OP_CPHI_EOPRE ||
                      op == HRGPU_OP_G5CPHI_EOPRE || op == HRGPU_OP_CPHI;
  const int pi = tune_slot(prec), ep = clover ? EP_CLOV : EP_AXPY;
  if (op_parity(op) == HRGPU_EVEN) return L.hop_pair_tuned[pi][clover];
  return L.hop_variant[pi][ep] >= 0 && (L.nf > 6 || L.hop_both[pi][ep] >= 0);
}

bool hop_tail_settled(bool clover, int prec) {
  const int v = last_hop_variant(clover ? EP_CLOV : EP_AXPY, prec);
  return v >= 0 && (L.hop_force >= 0 || L.hop_pair_tuned[tune_slot(prec)][clover]) && hop_tail_ok(v, L.nf, prec == HRGPU_FLOAT && L.flt_links == HRGPU_LINKS_BF16);
}

int apply_eo(bool clover, int prec, double mass, void *out, const void *in, int g5, double *red, const HopTail *tail) {
  if (prec == HRGPU_DOUBLE)
    return clover ? Cphi_eo<double>(mass, out, in, g5, red, tail) : Dphi_eo<double>(mass, out, in, HRGPU_EVEN, g5, red, tail);
  return clover ? Cphi_eo<float>(mass, out, in, g5, red, tail) : Dphi_eo<float>(mass, out, in, HRGPU_EVEN, g5, red, tail);
}

bool hop_small(bool clover, int prec) { return L.nf <= 6 && last_hop_variant(clover ? EP_CLOV : EP_AXPY, prec) == 1; }

void *eo_tmp(int prec) {
  void **tmp = prec == HRGPU_DOUBLE ? &L.tmp_e : &L.tmp_e_f;
  return ensure_tmp(tmp, spinor_bytes(HRGPU_EVEN, prec)) ? nullptr : *tmp;
}

int op_parity(int op) {
  return (op == HRGPU_OP_G5DPHI_SQ || op == HRGPU_OP_G5CPHI_SQ || op == HRGPU_OP_DPHI || op == HRGPU_OP_CPHI)
             ? HRGPU_FULL
             : HRGPU_EVEN;
}

double static_mass() { return g_static_mass; }

void add_mvm(unsigned long n) { g_mvm += n; }
unsigned long mvm_count() { return g_mvm; }
void mvm_restore(unsigned long n) { g_mvm = n; }

}  // namespace hrgpu

using namespace hrgpu;

extern "C" {

int hrgpu_Dphi_(void *out, int out_par, const void *in) { return Dphi_hop<double>(out, out_par, in); }
int hrgpu_Dphi(double m0, void *out, const void *in) { return Dphi_full<double>(m0, out, in, 0); }
int hrgpu_g5Dphi(double m0, void *out, const void *in) { return Dphi_full<double>(m0, out, in, 1); }
int hrgpu_g5Dphi_sq(double m0, void *out, const void *in) { return sq<double>(op_Dfull_d, m0, out, in, HRGPU_FULL); }
int hrgpu_Dphi_eopre(double m0, void *out, const void *in) { return Dphi_eo<double>(m0, out, in, HRGPU_EVEN, 0, nullptr); }
int hrgpu_Dphi_oepre(double m0, void *out, const void *in) { return Dphi_eo<double>(m0, out, in, HRGPU_ODD, 0, nullptr); }
int hrgpu_g5Dphi_eopre(double m0, void *out, const void *in) { return Dphi_eo<double>(m0, out, in, HRGPU_EVEN, 1, nullptr); }
int hrgpu_g5Dphi_eopre_sq(double m0, void *out, const void *in) { return sq<double>(op_eo_d, m0, out, in, HRGPU_EVEN); }

int hrgpu_Dphi_flt_(void *out, int out_par, const void *in) { return Dphi_hop<float>(out, out_par, in); }
int hrgpu_Dphi_flt(double m0, void *out, const void *in) { return Dphi_full<float>(m0, out, in, 0); }
int hrgpu_g5Dphi_flt(double m0, void *out, const void *in) { return Dphi_full<float>(m0, out, in, 1); }
int hrgpu_g5Dphi_sq_flt(double m0, void *out, const void *in) { return sq<float>(op_Dfull_f, m0, out, in, HRGPU_FULL); }
int hrgpu_Dphi_eopre_flt(double m0, void *out, const void *in) { return Dphi_eo<float>(m0, out, in, HRGPU_EVEN, 0, nullptr); }
int hrgpu_g5Dphi_eopre_flt(double m0, void *out, const void *in) { return Dphi_eo<float>(m0, out, in, HRGPU_EVEN, 1, nullptr); }
int hrgpu_g5Dphi_eopre_sq_flt(double m0, void *out, const void *in) { return sq<float>(op_eo_f, m0, out, in, HRGPU_EVEN); }

int hrgpu_set_hop_variant(int variant) {
  HR_REQUIRE(variant >= -1 && variant < HOP_VARIANTS, HRGPU_E_ARG, "set_hop_variant: variant must be -1..%d",
             HOP_VARIANTS - 1);
  L.hop_force = variant;
  return 0;
}

int hrgpu_hop_tuning(int prec, int epilogue, int *chosen, float *ms) {
  HR_REQUIRE(prec >= 0 && prec <= 2 && epilogue >= 0 && epilogue <= 2 && chosen && ms, HRGPU_E_ARG,
             "hop_tuning: bad arguments");
  *chosen = L.hop_variant[prec][epilogue];
  for (int v = 0; v < HOP_VARIANTS; v++) ms[v] = L.hop_tune_ms[prec][epilogue][v];
  return 0;
}

int hrgpu_set_hop_pdl(int on) {
  L.hop_pdl = on != 0;
  return 0;
}

unsigned long hrgpu_getMVM(void) {
  unsigned long r = g_mvm >> 1;
  g_mvm = 0;
  return r;
}

int hrgpu_Cphi(double mass, void *out, const void *in) { return Cphi_full(mass, out, in, 0); }
int hrgpu_g5Cphi(double mass, void *out, const void *in) { return Cphi_full(mass, out, in, 1); }
int hrgpu_g5Cphi_sq(double mass, void *out, const void *in) { return sq<double>(op_cfull_d, mass, out, in, HRGPU_FULL); }
int hrgpu_Cphi_eopre(double mass, void *out, const void *in) { return Cphi_eo<double>(mass, out, in, 0, nullptr); }
int hrgpu_g5Cphi_eopre(double mass, void *out, const void *in) { return Cphi_eo<double>(mass, out, in, 1, nullptr); }
int hrgpu_g5Cphi_eopre_sq(double mass, void *out, const void *in) { return sq<double>(op_ceo_d, mass, out, in, HRGPU_EVEN); }
int hrgpu_g5Cphi_eopre_flt(double mass, void *out, const void *in) { return Cphi_eo<float>(mass, out, in, 1, nullptr); }
int hrgpu_g5Cphi_eopre_sq_flt(double mass, void *out, const void *in) { return sq<float>(op_ceo_f, mass, out, in, HRGPU_EVEN); }

int hrgpu_set_flt_link_storage(int kind) {
  HR_REQUIRE(kind == HRGPU_LINKS_F32 || kind == HRGPU_LINKS_BF16, HRGPU_E_ARG,
             "set_flt_link_storage: kind must be HRGPU_LINKS_F32 or HRGPU_LINKS_BF16");
  L.flt_links = kind;
  return 0;
}

int hrgpu_set_dirac_mass(double mass) {
  g_static_mass = mass;
  return 0;
}
double hrgpu_get_dirac_mass(void) { return g_static_mass; }

// H2, H, D of D_update.c:41-95 in the UPDATE_EO build
int hrgpu_H2(void *out, const void *in) {
  return L.clover ? hrgpu_g5Cphi_eopre_sq(g_static_mass, out, in) : hrgpu_g5Dphi_eopre_sq(g_static_mass, out, in);
}
int hrgpu_H(void *out, const void *in) {
  return L.clover ? hrgpu_g5Cphi_eopre(g_static_mass, out, in) : hrgpu_g5Dphi_eopre(g_static_mass, out, in);
}
int hrgpu_D(void *out, const void *in) {
  return L.clover ? hrgpu_Cphi_eopre(g_static_mass, out, in) : hrgpu_Dphi_eopre(g_static_mass, out, in);
}

}  // extern "C"
