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
template <int N, bool DA, bool DB>
__device__ __forceinline__ void mul_ll(double2 (&c)[N][N], LinkPtr<N> a, LinkPtr<N> b) {
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
template <int N, bool DB>
__device__ __forceinline__ void mac_rl(double2 (&s)[N][N], const double2 (&t)[N][N], LinkPtr<N> b) {
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

}  // namespace hrgpu
