// cterm.cu -- compute_clover_term (LibHR/Update/clover_tools.c:161-206) from the
// fundamental links.
//
// The clover term is made of the anti-Hermitian parts of the four-leaf loops.  A
// product of represented links is the represented product, and a loop crosses the
// antiperiodic boundary twice or not at all, so each loop is multiplied out in the
// fundamental representation (NG x NG instead of NF x NF) and represented once, and
// only its anti-Hermitian part is formed and summed (NF^2 reals in registers).
// One thread per (site, plane), a block of 32 sites x 6 planes; the planes' sums
// meet in shared memory, where each warp combines one element of the four blocks
// for the block's sites, so that the stores are whole runs of sites.
#include "suN.cuh"

namespace hrgpu {

// element (C, A) of the represented link of u
template <int NG, int RP>
__device__ __forceinline__ double2 rep_elem(const double2 (&u)[NG][NG], int C, int A) {
  typedef Rep<NG, RP> P;
  if (RP == HRGPU_FUND) return u[C < NG ? C : 0][A < NG ? A : 0];
  const int c = P::hi(C), e = P::lo(C), a = P::hi(A), b = P::lo(A);
  double2 r = make_double2(0.0, 0.0);
  if (RP == HRGPU_SYM) {
    cmac(r, u[e][a], u[c][b]);
    cmac(r, u[e][b], u[c][a]);
    const double w = P::w(C) * P::w(A);
    return w == 1.0 ? r : make_double2(w * r.x, w * r.y);
  }
  cmac(r, u[c][a], u[e][b]);
  cmac(r, make_double2(-u[c][b].x, -u[c][b].y), u[e][a]);
  return r;
}

// K = R^+ - R of one plane: [i][i] the imaginary part of K_ii, [i][j], j < i, Re K_ij, [j][i] Im K_ij
template <int NG, int RP>
__device__ __forceinline__ void add_antiherm(double (&k)[Rep<NG, RP>::NF][Rep<NG, RP>::NF], const double2 (&u)[NG][NG]) {
  constexpr int NF = Rep<NG, RP>::NF;
  if constexpr (RP == HRGPU_ADJ) {
    double r[3][3];
    su2_adjoint(r, u);
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++)
        if (j < i) k[i][j] += r[j][i] - r[i][j];
  } else {
#pragma unroll
    for (int i = 0; i < NF; i++) {
      k[i][i] -= 2.0 * rep_elem<NG, RP>(u, i, i).y;
#pragma unroll
      for (int j = 0; j < NF; j++)
        if (j < i) {
          const double2 a = rep_elem<NG, RP>(u, i, j), b = rep_elem<NG, RP>(u, j, i);
          k[i][j] += b.x - a.x;
          k[j][i] -= b.y + a.y;
        }
    }
  }
}

// Bound by FP64 latency at 12 warps per SM (168 registers) and the link loads from
// L1/L2 (16 NG^2 complex per thread): 0.14 ms at 24x12^3 SU(3) sextet, against 2.55 ms
// with the loops multiplied out in the representation (k_clover_term_r).
template <int NG, int RP>
__global__ void __launch_bounds__(192, NG < 4 ? 2 : 1) k_clover_term_fund(double2 *cl, const double2 *Ul, Geo g, double csw) {
  constexpr int NF = Rep<NG, RP>::NF;
  extern __shared__ double ct_k[];  // [plane][NF*NF][32]
  const int lane = threadIdx.x & 31, q = threadIdx.x >> 5;
  const long d = (long)blockIdx.x * 32 + lane;
  const bool on = (d >= g.ld ? d - g.ld : d) < g.VH;
  const long lp = 2L * g.ld;
  double k[NF][NF];
#pragma unroll
  for (int i = 0; i < NF; i++)
#pragma unroll
    for (int j = 0; j < NF; j++) k[i][j] = 0.0;
  if (on) {
    int t, x, y, z;
    dev_coords(g, (int)d, t, x, y, z);
    // planes (0,1) (0,2) (0,3) (1,2) (1,3) (2,3)
    const int mu = q < 3 ? 0 : (q < 5 ? 1 : 2), nu = q < 3 ? q + 1 : (q < 5 ? q - 1 : 3);
#pragma unroll 1
    for (int m = 0; m < 4; m++) {
      double2 l[NG][NG];
      leaf_loop<NG>(l, Ul, g, lp, t, x, y, z, mu, nu, m);
      add_antiherm<NG, RP>(k, l);
    }
  }
#pragma unroll
  for (int i = 0; i < NF; i++)
#pragma unroll
    for (int j = 0; j < NF; j++) ct_k[((q * NF + i) * NF + j) * 32 + lane] = k[i][j];
  __syncthreads();
  if (!on) return;
  const double c = -csw / 16.0;
  for (int o = q; o < NF * NF; o += 6) {
    const int i = o / NF, j = o % NF;
    auto K = [&](int p) {
      const double a = ct_k[((p * NF + i) * NF + j) * 32 + lane], b = ct_k[((p * NF + j) * NF + i) * 32 + lane];
      if (i == j) return make_double2(0.0, a);
      return i > j ? make_double2(a, b) : make_double2(-b, a);
    };
    const double2 k0 = K(0), k1 = K(1), k2 = K(2), k3 = K(3), k4 = K(4), k5 = K(5);
    const double2 a = make_double2(-k2.y, k2.x), b = make_double2(-k3.y, k3.x);
    const double2 e = make_double2(-k0.y + k1.x, k0.x + k1.y), f = make_double2(-k5.y - k4.x, k5.x - k4.y);
    double2 *p = cl + (long)o * lp + d;
    const long s = (long)NF * NF * lp;
    p[0] = make_double2(c * (a.x - b.x), c * (a.y - b.y));
    p[s] = make_double2(c * (e.x - f.x), c * (e.y - f.y));
    p[2 * s] = make_double2(-c * (a.x + b.x), -c * (a.y + b.y));
    p[3 * s] = make_double2(-c * (e.x + f.x), -c * (e.y + f.y));
  }
}

template <int NG, int RP>
static int launch_term(const double2 *Ul) {
  constexpr int NF = Rep<NG, RP>::NF;
  constexpr int smem = (int)sizeof(double) * 6 * NF * NF * 32;
  if (smem > 48 * 1024)
    if (int rc = allow_smem((const void *)k_clover_term_fund<NG, RP>, smem)) return rc;
  k_clover_term_fund<NG, RP><<<(unsigned)(2L * L.ld / 32), 192, smem, L.stream>>>(L.cl_term, Ul, make_geo(), L.csw);
  HR_LAUNCH_CHECK();
  return 0;
}

// -1 where the clover term is not formed this way: the represented links are not
// known to come from the fundamental ones held, a larger group, or SU(2) adjoint
// links that did not pass the row check (the adjoint of a product is the product of
// the adjoints for unitary links only)
int clover_term_fund() {
  const double2 *Ul = nullptr;
  if (L.repr == HRGPU_FUND) Ul = (const double2 *)L.U;
  else if (L.fund_current && (L.repr != HRGPU_ADJ || L.recon12 == 1 || L.recon12 == 2)) Ul = L.Ug;
  if (!Ul) return -1;
  switch (L.repr * 16 + L.ng) {
    case HRGPU_FUND * 16 + 2: return launch_term<2, HRGPU_FUND>(Ul);
    case HRGPU_FUND * 16 + 3: return launch_term<3, HRGPU_FUND>(Ul);
    case HRGPU_FUND * 16 + 4: return launch_term<4, HRGPU_FUND>(Ul);
    case HRGPU_ADJ * 16 + 2: return launch_term<2, HRGPU_ADJ>(Ul);
    case HRGPU_SYM * 16 + 2: return launch_term<2, HRGPU_SYM>(Ul);
    case HRGPU_SYM * 16 + 3: return launch_term<3, HRGPU_SYM>(Ul);
    case HRGPU_ASYM * 16 + 3: return launch_term<3, HRGPU_ASYM>(Ul);
    case HRGPU_ASYM * 16 + 4: return launch_term<4, HRGPU_ASYM>(Ul);
    default: return -1;
  }
}

}  // namespace hrgpu
