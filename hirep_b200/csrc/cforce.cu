// cforce.cu -- the clover part of fermion_force_end (LibHR/Update/force_fermion_core.c:282-379)
// through the fundamental links.
//
// cl_force holds an anti-Hermitian matrix Z per site and plane in the fermion
// representation R; the force is the derivative of
//   sum over planes, sites y and the loops L_y of the plane's plaquettes that start
//   at y, of Re Tr(Z_y R(L_y)),
// and the reference takes it by carrying Z around every loop as NF x NF products.
// R(L) is a fixed function of the NG x NG loop L, so one step of the chain rule
// brings it down to the fundamental matrices first:
//   d/de Re Tr(Z R(L (1 + e X))) = Re Tr(E X) for X in su(NG),
// with E the anti-Hermitian part of G L, G_ji = d Tr(Z R(L)) / d L_ij (the
// two-index representations: four terms per element of Z), or the su(2) vector of
// Z R(L) for the SU(2) adjoint.  E and S (X at the loop's start, G L -> L G) are
// then carried around the plaquette with NG x NG products.
//
// At 24x12^3 SU(3) sextet the force took 8.34 ms as NF x NF products in local memory
// and takes 0.13 + 0.05 + 0.02 ms in the three kernels here; one thread doing the four
// corners of a plaquette (Z read four times, 255 registers) took 0.19 ms, and spilled
// 20 KB per thread for SU(4).
// Three kernels: k_cforce_corner forms E and S of the four loops that start at a
// site (Z is read once), k_cforce_plaq carries the seven that a plaquette needs to
// its links, one thread per (plaquette, plane), and k_cforce_gather adds the six
// contributions to each link in a fixed order, so the result does not depend on
// scheduling.  The corners and link forces take 42 NG^2 + 24 (NG^2 - 1) doubles per site
// (3.0 GB for SU(3) at 48x24^3), kept for the next force; they are only taken where
// as much again stays free.
#include "suN.cuh"

namespace hrgpu {

// G_ji = d Tr(Z R(L)) / d L_ij; Z read from its planes, lower triangle only
template <int NG, int RP>
__device__ __forceinline__ void z_contract(double2 (&G)[NG][NG], const double2 *z, long lp, const double2 (&u)[NG][NG]) {
  typedef Rep<NG, RP> P;
  constexpr int NF = P::NF;
  mzero<NG>(G);
#pragma unroll
  for (int A = 0; A < NF; A++)
#pragma unroll
    for (int C = 0; C < NF; C++) {
      if (C > A) continue;
      const double2 zr = __ldg(z + (long)(A * NF + C) * lp);
      if constexpr (RP == HRGPU_FUND) {
        G[A][C] = zr;
        if (C < A) G[C][A] = make_double2(-zr.x, zr.y);
      } else {
        const double w = P::w(A) * P::w(C);
#pragma unroll
        for (int m = 0; m < 2; m++) {
          if (m && A == C) continue;
          // element (a2, c2) of Z: zr, or by anti-Hermiticity -conj(zr) for the mirrored one
          const int ra = m ? C : A, rc = m ? A : C;
          const double2 y = m ? make_double2(-w * zr.x, w * zr.y) : make_double2(w * zr.x, w * zr.y);
          const int a = P::hi(ra), b = P::lo(ra), c = P::hi(rc), e = P::lo(rc);
          if (RP == HRGPU_SYM) {  // R_CA = w (u_ea u_cb + u_eb u_ca)
            cmac(G[a][e], y, u[c][b]);
            cmac(G[b][c], y, u[e][a]);
            cmac(G[b][e], y, u[c][a]);
            cmac(G[a][c], y, u[e][b]);
          } else {  // R_CA = u_ca u_eb - u_cb u_ea
            const double2 n = make_double2(-y.x, -y.y);
            cmac(G[a][c], y, u[e][b]);
            cmac(G[b][e], y, u[c][a]);
            cmac(G[b][c], n, u[e][a]);
            cmac(G[a][e], n, u[c][b]);
          }
        }
      }
    }
}

// E (X at the end of the loop) and S (X at its start) of one loop
template <int NG, int RP>
__device__ __forceinline__ void corner(AH<NG> &E, AH<NG> &S, const double2 *z, long lp, const double2 (&u)[NG][NG]) {
  if constexpr (RP == HRGPU_ADJ) {
    double r[3][3], zr[3][3];
    su2_adjoint(r, u);
    zr[0][0] = zr[1][1] = zr[2][2] = 0.0;
#pragma unroll
    for (int i = 1; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++)
        if (j < i) {
          zr[i][j] = __ldg(z + (long)(i * 3 + j) * lp).x;
          zr[j][i] = -zr[i][j];
        }
    // p_A = Tr(M rho(iT_A)) = M_CB - M_BC for (A, B, C) cyclic; P = -2i sum p_A T_A
    auto vec = [](AH<NG> &o, const double (&m)[3][3]) {
      const double p0 = m[2][1] - m[1][2], p1 = m[0][2] - m[2][0], p2 = m[1][0] - m[0][1];
      o.d[0] = -p2;
      o.d[1] = p2;
      o.o[1][0] = make_double2(-p1, p0);  // T_0 = -s2/2, T_1 = s1/2: element (1, 0) of -2 (p0 T_0 + p1 T_1)
    };
    double m[3][3];
    {
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) m[i][j] = zr[i][0] * r[0][j] + zr[i][1] * r[1][j] + zr[i][2] * r[2][j];
      vec(E, m);
    }
    {
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) m[i][j] = r[i][0] * zr[0][j] + r[i][1] * zr[1][j] + r[i][2] * zr[2][j];
      vec(S, m);
    }
  } else {
    double2 G[NG][NG];
    z_contract<NG, RP>(G, z, lp, u);
    E.from_product(G, u);
    S.from_product(u, G);
  }
}

template <int N>
__device__ __forceinline__ void ah_store(double *p, long lp, const AH<N> &a) {
#pragma unroll
  for (int i = 0; i < N; i++) {
    p[(long)(i * N + i) * lp] = a.d[i];
#pragma unroll
    for (int j = 0; j < N; j++)
      if (j < i) {
        p[(long)(i * N + j) * lp] = a.o[i][j].x;
        p[(long)(j * N + i) * lp] = a.o[i][j].y;
      }
  }
}
template <int N>
__device__ __forceinline__ void ah_load(AH<N> &a, const double *p, long lp) {
#pragma unroll
  for (int i = 0; i < N; i++) {
    a.d[i] = __ldg(p + (long)(i * N + i) * lp);
#pragma unroll
    for (int j = 0; j < N; j++)
      if (j < i) a.o[i][j] = make_double2(__ldg(p + (long)(i * N + j) * lp), __ldg(p + (long)(j * N + i) * lp));
  }
}

// slots of the corner buffer [plane][slot][N*N][2ld]: E of corner k, S of corners 0, 1, 3
constexpr int CF_SLOTS = 7;
__host__ __device__ constexpr int cf_slot_s(int k) { return k == 3 ? 6 : 4 + k; }

// The products with U^+ that carry a force around the plaquette stand for U^-1, so a link
// that is unitary up to an error of this size changes the force by about as much.
// update_gauge_field's links are off by at most 1.4e-14 when they are made unitary
// again after 17 steps (16^4, SU(2) to SU(4)).
constexpr double CF_UNITARY = 4e-14;

// E and S of the four loops that start at a site.  Bound by FP64 latency at 12 warps
// per SM (168 registers) and the Z loads from L2.  A link that is not unitary to
// CF_UNITARY sets *bad.
template <int NG, int RP>
__global__ void __launch_bounds__(192, NG < 4 ? 2 : 1)
    k_cforce_corner(double *C, const double2 *Ul, const double2 *clf, Geo g, int *bad) {
  constexpr int NF2 = Rep<NG, RP>::NF * Rep<NG, RP>::NF, N2 = NG * NG;
  const long d = (long)blockIdx.x * 32 + (threadIdx.x & 31);
  const int q = threadIdx.x >> 5;  // cl_force's plane: (0,1) (0,2) (1,2) (0,3) (1,3) (2,3)
  if ((d >= g.ld ? d - g.ld : d) >= g.VH) return;
  const int nu = q < 1 ? 1 : (q < 3 ? 2 : 3), mu = q - nu * (nu - 1) / 2;
  const long lp = 2L * g.ld;
  int t, x, y, z;
  dev_coords(g, (int)d, t, x, y, z);
  if (q < 4) {  // warp q checks direction q
    const LinkPtr<NG> u = link_at<NG>(Ul, q, d, lp);
    double2 m[NG][NG];
    mul_ll<NG, false, true>(m, u, u);
    bool ok = true;
#pragma unroll
    for (int i = 0; i < NG; i++)
#pragma unroll
      for (int j = 0; j < NG; j++)
        if (j <= i) ok = ok && fabs(m[i][j].x - (i == j ? 1.0 : 0.0)) <= CF_UNITARY && fabs(m[i][j].y) <= CF_UNITARY;
    if (!ok) atomicOr(bad, 1);
  }
  const double2 *Z = clf + (long)q * NF2 * lp + d;
  double *Co = C + (long)q * CF_SLOTS * N2 * lp + d;
#pragma unroll 1
  for (int k = 0; k < 4; k++) {
    double2 l[NG][NG];
    leaf_loop<NG>(l, Ul, g, lp, t, x, y, z, mu, nu, k);
    AH<NG> E, S;
    corner<NG, RP>(E, S, Z, lp, l);
    ah_store<NG>(Co + (long)k * N2 * lp, lp, E);
    if (k != 2) ah_store<NG>(Co + (long)cf_slot_s(k) * N2 * lp, lp, S);
  }
}

// The force on the four links of the plaquette x0 -> x1 = x+mu -> x2 = x+mu+nu ->
// x3 = x+nu, u1 = U_mu(x0), u2 = U_nu(x1), u3 = U_mu(x3), u4 = U_nu(x0), each of
// which lies in the four loops around it.  With t = u2 E2 u2^+, e = u1 (E1 + t) u1^+,
// s = u4 S3 u4^+ the forces are
//   u1: S0 + e + s                       u4: -(E0 + e + s)               (at x0)
//   u2: S1 + t + u1^+ (S0 + s) u1 (x1)   u3: -(E3 + u4^+ (E0 + e) u4)    (at x3)
// (the loop that starts at a link's base gives S where the link is the loop's
// first and E where it is its last).
template <int NG>
__global__ void __launch_bounds__(192, NG < 4 ? 2 : 1) k_cforce_plaq(double *F, const double *C, const double2 *Ul, Geo g, const int *bad) {
  constexpr int N2 = NG * NG, DG = N2 - 1;
  if (*bad) return;
  const long d = (long)blockIdx.x * 32 + (threadIdx.x & 31);
  const int q = threadIdx.x >> 5;
  if ((d >= g.ld ? d - g.ld : d) >= g.VH) return;
  const int nu = q < 1 ? 1 : (q < 3 ? 2 : 3), mu = q - nu * (nu - 1) / 2;
  const long lp = 2L * g.ld;
  int t, x, y, z;
  dev_coords(g, (int)d, t, x, y, z);
  const long x1 = site_at(g, t, x, y, z, mu, 1, nu, 0), x3 = site_at(g, t, x, y, z, mu, 0, nu, 1);
  const long x2 = site_at(g, t, x, y, z, mu, 1, nu, 1);
  const LinkPtr<NG> u1 = link_at<NG>(Ul, mu, d, lp), u2 = link_at<NG>(Ul, nu, x1, lp), u4 = link_at<NG>(Ul, nu, d, lp);
  const double *Cq = C + (long)q * CF_SLOTS * N2 * lp;
  auto slot = [&](int k, long site) { return Cq + (long)k * N2 * lp + site; };
  double *Fo = F + (long)q * 4 * DG * lp + d;
  AH<NG> a, b, c, e;
  ah_load<NG>(a, slot(2, x2), lp);
  a.template transport<false>(u2);  // t
  ah_load<NG>(e, slot(1, x1), lp);
  e.add(a);
  e.template transport<false>(u1);  // e
  ah_load<NG>(b, slot(cf_slot_s(3), x3), lp);
  b.template transport<false>(u4);  // s
  ah_load<NG>(c, slot(cf_slot_s(1), x1), lp);
  c.add(a);                         // S1 + t
  ah_load<NG>(a, slot(cf_slot_s(0), d), lp);
  a.add(b);                         // S0 + s
  b.add(e);                         // e + s
  AH<NG> w;
  ah_load<NG>(w, slot(0, d), lp);   // E0
  e.add(w);                         // E0 + e
  w.add(b);                         // E0 + e + s
  w.project([&](int A, double f) { Fo[(long)(3 * DG + A) * lp] = -f; });
  ah_load<NG>(w, slot(cf_slot_s(0), d), lp);
  w.add(b);                         // S0 + e + s
  w.project([&](int A, double f) { Fo[(long)A * lp] = f; });
  a.template transport<true>(u1);
  a.add(c);
  a.project([&](int A, double f) { Fo[(long)(DG + A) * lp] = f; });
  e.template transport<true>(u4);
  ah_load<NG>(c, slot(3, x3), lp);
  e.add(c);
  e.project([&](int A, double f) { Fo[(long)(2 * DG + A) * lp] = -f; });
}

// force_sum(x, mu) += coeff times the contributions of the six plaquettes of the link
__global__ void k_cforce_gather(double *fsum, const double *F, Geo g, int DG, double coeff, const int *bad) {
  if (*bad) return;
  const long d = (long)blockIdx.x * 32 + (threadIdx.x & 31);
  const int mu = threadIdx.x >> 5;
  if ((d >= g.ld ? d - g.ld : d) >= g.VH) return;
  const long lp = 2L * g.ld;
  int t, x, y, z;
  dev_coords(g, (int)d, t, x, y, z);
  const double *src[6];
#pragma unroll
  for (int i = 1; i < 4; i++) {
    const int nu = (mu + i) & 3;
    const long xd = site_at(g, t, x, y, z, nu, -1, nu, 0);
    const int q = mu < nu ? nu * (nu - 1) / 2 + mu : mu * (mu - 1) / 2 + nu;
    // as the plane's first direction: u1 here, u3 of the plaquette below; as its second: u4 here, u2 below
    src[2 * i - 2] = F + (long)(4 * q + (mu < nu ? 0 : 3)) * DG * lp + d;
    src[2 * i - 1] = F + (long)(4 * q + (mu < nu ? 2 : 1)) * DG * lp + xd;
  }
  double *o = fsum + (long)mu * DG * lp + d;
  for (int A = 0; A < DG; A++) {
    double f = 0.0;
#pragma unroll
    for (int k = 0; k < 6; k++) f += __ldg(src[k] + (long)A * lp);
    o[(long)A * lp] += coeff * f;
  }
}

// The clover force through the fundamental links: 0 done (unless *bad is set on
// the device, when force_sum is untouched), -1 where it does not apply (the
// represented links are not known to come from the fundamental ones held, or a
// larger group), else an error status.
int clover_force_fund(double coeff, int **bad_out) {
  const double2 *Ul = nullptr;
  if (L.repr == HRGPU_FUND) Ul = (const double2 *)L.U;  // the boundary sign enters a loop twice or not at all
  else if (L.fund_current) Ul = L.Ug;
  const bool built = (L.repr == HRGPU_FUND && L.ng <= 4) || (L.repr == HRGPU_ADJ && L.ng == 2) ||
                     (L.repr == HRGPU_SYM && L.ng <= 3) || (L.repr == HRGPU_ASYM && (L.ng == 3 || L.ng == 4));
  if (!Ul || !built) return -1;
  const long lp = 2L * L.ld;
  const int N2 = L.ng * L.ng;
  const size_t nc = (size_t)6 * CF_SLOTS * N2 * lp, nf = (size_t)24 * L.dimg * lp;  // corners, link forces
  const size_t bytes = sizeof(double) * (nc + nf + 1);
  if (!L.cl_plaq && (!optional_room(bytes) || cudaMalloc(&L.cl_plaq, bytes) != cudaSuccess)) {
    cudaGetLastError();  // no room for the workspace: the representation's kernel needs none
    L.cl_plaq = nullptr;
    return -1;
  }
  double *C = L.cl_plaq, *F = C + nc;
  int *bad = (int *)(F + nf);
  HR_CUDA(cudaMemsetAsync(bad, 0, sizeof(int), L.stream));
  const Geo g = make_geo();
  const unsigned grid = (unsigned)(lp / 32);
#define HR_CF(NGV, RPV)                                                                    \
  do {                                                                                     \
    k_cforce_corner<NGV, RPV><<<grid, 192, 0, L.stream>>>(C, Ul, L.cl_force, g, bad);       \
    k_cforce_plaq<NGV><<<grid, 192, 0, L.stream>>>(F, C, Ul, g, bad);                       \
  } while (0)
  switch (L.repr) {
    case HRGPU_FUND:
      if (L.ng == 2) HR_CF(2, HRGPU_FUND);
      else if (L.ng == 3) HR_CF(3, HRGPU_FUND);
      else HR_CF(4, HRGPU_FUND);
      break;
    case HRGPU_ADJ: HR_CF(2, HRGPU_ADJ); break;
    case HRGPU_SYM:
      if (L.ng == 2) HR_CF(2, HRGPU_SYM);
      else HR_CF(3, HRGPU_SYM);
      break;
    default:
      if (L.ng == 3) HR_CF(3, HRGPU_ASYM);
      else HR_CF(4, HRGPU_ASYM);
      break;
  }
#undef HR_CF
  HR_LAUNCH_CHECK();
  // the reference projects with 1 / C(R), and its sum runs with the opposite sign
  k_cforce_gather<<<grid, 128, 0, L.stream>>>(L.force_sum, F, g, L.dimg, -coeff / L.repr_norm2, bad);
  HR_LAUNCH_CHECK();
  *bad_out = bad;
  return 0;
}

}  // namespace hrgpu
