// suN.cuh -- fundamental-representation matrices held in registers (NG <= 4):
// products whose operands stream from the link planes element by element, the
// algebra projection with the generators written out, and the index pairs of
// the two-index representations for any NG.  Every loop is unrolled, so no
// array is indexed at run time and nothing goes to local memory.
#pragma once
#include "dirac.cuh"

namespace hrgpu {

constexpr int SUN_MAX = 4;  // largest NG of the register kernels (16 complex FP64 = 64 registers a matrix)

// element k of the link plane base p (already at its site)
template <int N>
struct LinkPtr {
  const double2 *p;
  long lp;
  __device__ __forceinline__ double2 operator()(int i, int j) const { return __ldg(p + (long)(i * N + j) * lp); }
};

template <int N>
__device__ __forceinline__ LinkPtr<N> link_at(const double2 *Ug, int mu, long site, long lp) {
  LinkPtr<N> l;
  l.p = Ug + (long)mu * N * N * lp + site;
  l.lp = lp;
  return l;
}

template <int N>
__device__ __forceinline__ void mzero(double2 (&c)[N][N]) {
#pragma unroll
  for (int i = 0; i < N; i++)
#pragma unroll
    for (int j = 0; j < N; j++) c[i][j] = make_double2(0.0, 0.0);
}

__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }

// C = op(A) op(B), both operands streamed: one row or column of each is held at a time
template <int N, bool DA, bool DB, typename LA, typename LB>
__device__ __forceinline__ void mul_ll(double2 (&c)[N][N], const LA &a, const LB &b) {
  mzero<N>(c);
#pragma unroll
  for (int k = 0; k < N; k++) {
    double2 ac[N], br[N];
#pragma unroll
    for (int i = 0; i < N; i++) {
      ac[i] = DA ? cconj(a(k, i)) : a(i, k);
      br[i] = DB ? cconj(b(i, k)) : b(k, i);
    }
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
      for (int j = 0; j < N; j++) cmac(c[i][j], ac[i], br[j]);
  }
}

// S += T op(B), B streamed
template <int N, bool DB, typename LB>
__device__ __forceinline__ void mac_rl(double2 (&s)[N][N], const double2 (&t)[N][N], const LB &b) {
#pragma unroll
  for (int k = 0; k < N; k++) {
    double2 br[N];
#pragma unroll
    for (int j = 0; j < N; j++) br[j] = DB ? cconj(b(j, k)) : b(k, j);
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
      for (int j = 0; j < N; j++) cmac(s[i][j], t[i][k], br[j]);
  }
}

// index of the generator T_A of the pair (a, b) in build_generators' order
// (a > b: symmetric, a < b: antisymmetric, a == b > 0: diagonal)
template <int N>
__host__ __device__ constexpr int gen_index(int a, int b) { return a * N + b - 1; }

// f_A = 2 Re Tr((i T_A)^+ w) with the generators written out
template <int N, typename F>
__device__ __forceinline__ void algebra_project(const double2 (&w)[N][N], F &&put) {
#pragma unroll
  for (int a = 0; a < N; a++)
#pragma unroll
    for (int b = 0; b < N; b++) {
      if (a == 0 && b == 0) continue;
      double f;
      if (a > b) {
        f = w[a][b].y + w[b][a].y;
      } else if (a < b) {
        f = w[b][a].x - w[a][b].x;
      } else {
        f = -(double)a * w[a][a].y;
#pragma unroll
        for (int k = 0; k < N; k++)
          if (k < a) f += w[k][k].y;
        f *= sqrt(2.0 / ((double)a * (a + 1.0)));
      }
      put(gen_index<N>(a, b), f);
    }
}

// device site of (t, x, y, z) shifted by da along direction a and db along b (each -1, 0 or 1)
__device__ __forceinline__ long site_at(const Geo &g, int t, int x, int y, int z, int a, int da, int b, int db) {
  t += (a == 0 ? da : 0) + (b == 0 ? db : 0);
  x += (a == 1 ? da : 0) + (b == 1 ? db : 0);
  y += (a == 2 ? da : 0) + (b == 2 ? db : 0);
  z += (a == 3 ? da : 0) + (b == 3 ? db : 0);
  // sizes are at least 2, so a shift of one in each of two different directions wraps once
  t = t < 0 ? t + g.T : (t >= g.T ? t - g.T : t);
  x = x < 0 ? x + g.X : (x >= g.X ? x - g.X : x);
  y = y < 0 ? y + g.Y : (y >= g.Y ? y - g.Y : y);
  z = z < 0 ? z + g.Z : (z >= g.Z ? z - g.Z : z);
  return (long)((t + x + y + z) & 1) * g.ld + coords_to_cb(g, t, x, y, z);
}

// C = op(A) op(B) of matrices in registers
template <int N, bool DA, bool DB>
__device__ __forceinline__ void mul_rr(double2 (&c)[N][N], const double2 (&a)[N][N], const double2 (&b)[N][N]) {
#pragma unroll
  for (int i = 0; i < N; i++)
#pragma unroll
    for (int j = 0; j < N; j++) {
      double2 s = make_double2(0.0, 0.0);
#pragma unroll
      for (int k = 0; k < N; k++) cmac(s, DA ? cconj(a[k][i]) : a[i][k], DB ? cconj(b[j][k]) : b[k][j]);
      c[i][j] = s;
    }
}

// An anti-Hermitian N x N matrix i H by its Hermitian H: real diagonal d, lower triangle o[i][j], j < i
template <int N>
struct AH {
  double d[N];
  double2 o[N][N];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < N; i++) {
      d[i] = 0.0;
#pragma unroll
      for (int j = 0; j < N; j++)
        if (j < i) o[i][j] = make_double2(0.0, 0.0);
    }
  }
  __device__ __forceinline__ void add(const AH<N> &b) {
#pragma unroll
    for (int i = 0; i < N; i++) {
      d[i] += b.d[i];
#pragma unroll
      for (int j = 0; j < N; j++)
        if (j < i) o[i][j] = cadd(o[i][j], b.o[i][j]);
    }
  }
  // the anti-Hermitian part (M - M^+) / 2 of M = A B
  __device__ __forceinline__ void from_product(const double2 (&a)[N][N], const double2 (&b)[N][N]) {
    double2 m[N][N];
    mul_rr<N, false, false>(m, a, b);
#pragma unroll
    for (int i = 0; i < N; i++) {
      d[i] = m[i][i].y;
#pragma unroll
      for (int j = 0; j < N; j++)  // (m_ij - conj(m_ji)) / (2 i)
        if (j < i) o[i][j] = make_double2(0.5 * (m[i][j].y + m[j][i].y), -0.5 * (m[i][j].x - m[j][i].x));
    }
  }
  __device__ __forceinline__ double2 h(int i, int j) const {
    return i == j ? make_double2(d[i], 0.0) : (j < i ? o[i][j] : cconj(o[j][i]));
  }
  // this <- U this U^+ (DAG: U^+ this U), U streamed
  template <bool DAG>
  __device__ __forceinline__ void transport(LinkPtr<N> u) {
    double2 w[N][N], t[N][N];
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
      for (int j = 0; j < N; j++) w[i][j] = DAG ? cconj(u(j, i)) : u(i, j);
    transport_r(w, t);
  }
  __device__ __forceinline__ void transport_r(const double2 (&w)[N][N], double2 (&t)[N][N]) {
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
      for (int j = 0; j < N; j++) {
        double2 s = make_double2(0.0, 0.0);
#pragma unroll
        for (int k = 0; k < N; k++) cmac(s, w[i][k], h(k, j));
        t[i][j] = s;
      }
#pragma unroll
    for (int i = 0; i < N; i++) {
#pragma unroll
      for (int j = 0; j < N; j++)
        if (j <= i) {
          double2 s = make_double2(0.0, 0.0);
#pragma unroll
          for (int k = 0; k < N; k++) cmac(s, t[i][k], cconj(w[j][k]));
          if (i == j) d[i] = s.x;
          else o[i][j] = s;
        }
    }
  }
  // f_A = Re Tr(i T_A (i H)) = -Tr(T_A H)
  template <typename F>
  __device__ __forceinline__ void project(F &&put) const {
#pragma unroll
    for (int a = 0; a < N; a++)
#pragma unroll
      for (int b = 0; b < N; b++) {
        if (a == 0 && b == 0) continue;
        double f;
        if (a > b) {
          f = -o[a][b].x;
        } else if (a < b) {
          f = o[b][a].y;
        } else {
          f = (double)a * d[a];
#pragma unroll
          for (int k = 0; k < N; k++)
            if (k < a) f -= d[k];
          f *= 0.5 * sqrt(2.0 / ((double)a * (a + 1.0)));
        }
        put(gen_index<N>(a, b), f);
      }
  }
};

// A link or its dagger, chosen at run time by the strides
template <int N>
struct DagLink {
  const double2 *p;
  long ro, co;  // row and column strides
  double sg;    // sign of the imaginary part
  __device__ __forceinline__ double2 operator()(int i, int j) const {
    const double2 v = __ldg(p + i * ro + j * co);
    return make_double2(v.x, sg * v.y);
  }
};

// The loop k = 0..3 of the four-leaf loop around (t, x, y, z) in the plane
// (mu, nu) (clover_tools.c:59-95): it runs around the plaquette whose corner k is
// the site (base shifted by (0,0), (-1,0), (-1,-1), (0,-1)), starting there, along
// w_0 = U_mu(b), w_1 = U_nu(b+mu), w_2 = U_mu(b+nu)^+, w_3 = U_nu(b)^+ cyclically.
// k is a run-time value so that one copy of the code serves the four loops.
template <int N>
__device__ __forceinline__ void leaf_loop(double2 (&l)[N][N], const double2 *Ul, const Geo &g, long lp, int t, int x, int y,
                                          int z, int mu, int nu, int k) {
  const int da = (k == 1 || k == 2) ? -1 : 0, db = k >= 2 ? -1 : 0;
  auto w = [&](int m) {
    const int j = (k + m) & 3, dir = (j & 1) ? nu : mu;
    const long site = site_at(g, t, x, y, z, mu, da + (j == 1), nu, db + (j == 2));
    DagLink<N> q;
    q.p = Ul + (long)dir * N * N * lp + site;
    q.ro = j >= 2 ? lp : N * lp;
    q.co = j >= 2 ? N * lp : lp;
    q.sg = j >= 2 ? -1.0 : 1.0;
    return q;
  };
  double2 a[N][N];
  mul_ll<N, false, false>(l, w(0), w(1));
  mzero<N>(a);
  mac_rl<N, false>(a, l, w(2));
  mzero<N>(l);
  mac_rl<N, false>(l, a, w(3));
}

// The representations whose links the register kernels form from the
// fundamental ones: all four, by NG and HRGPU_*.
template <int NG, int RP>
struct Rep {
  static constexpr int NF = RP == HRGPU_FUND ? NG
                            : RP == HRGPU_ADJ ? NG * NG - 1
                            : RP == HRGPU_SYM ? NG * (NG + 1) / 2 : NG * (NG - 1) / 2;
  // basis element k of a two-index representation is the index pair (hi, lo)
  __host__ __device__ static constexpr int hi(int k) {
    return RP == HRGPU_SYM ? (k < 1 ? 0 : (k < 3 ? 1 : (k < 6 ? 2 : 3))) : (k < 1 ? 1 : (k < 3 ? 2 : 3));
  }
  __host__ __device__ static constexpr int lo(int k) {
    return RP == HRGPU_SYM ? k - hi(k) * (hi(k) + 1) / 2 : k - hi(k) * (hi(k) - 1) / 2;
  }
  // weight of a symmetric diagonal pair: R_CA = w_C w_A (u_ea u_cb + u_eb u_ca)
  __host__ __device__ static constexpr double w(int k) {
    return (RP == HRGPU_SYM && hi(k) == lo(k)) ? 0.70710678118654752440 : 1.0;
  }
};

// The SU(2) adjoint: R_CA(u) = 2 Re Tr(T_C u T_A u^+), real 3 x 3, T = (-s2, s1, s3) / 2
__device__ __forceinline__ void su2_adjoint(double (&r)[3][3], const double2 (&u)[2][2]) {
  auto mc = [](double2 p, double2 q) {  // p conj(q)
    return make_double2(p.x * q.x + p.y * q.y, p.y * q.x - p.x * q.y);
  };
  const double2 ab = mc(u[0][0], u[0][1]), cd = mc(u[1][0], u[1][1]);
  const double2 ad = mc(u[0][0], u[1][1]), bc = mc(u[0][1], u[1][0]);
  const double2 z3 = csub(mc(u[0][0], u[1][0]), mc(u[0][1], u[1][1]));
  // the column A is (Im z, Re z, (p - s) / 2) of u (2 T_A) u^+ = [[p, z], [conj z, s]]
  r[0][0] = ad.x - bc.x;
  r[1][0] = bc.y - ad.y;
  r[2][0] = cd.y - ab.y;
  r[0][1] = ad.y + bc.y;
  r[1][1] = ad.x + bc.x;
  r[2][1] = ab.x - cd.x;
  r[0][2] = z3.y;
  r[1][2] = z3.x;
  r[2][2] = 0.5 * (mc(u[0][0], u[0][0]).x - mc(u[0][1], u[0][1]).x - mc(u[1][0], u[1][0]).x + mc(u[1][1], u[1][1]).x);
}

}  // namespace hrgpu
