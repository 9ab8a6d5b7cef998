// hop_dir.cuh -- the hopping kernel with the eight directions of a site on eight warps.
//
// A block works on 32 consecutive sites.  Warp w takes direction w >> 1 forward
// (w & 1 = 0) or backward: each thread projects one neighbour's spinor, multiplies
// it by one link and puts the two NF-vectors in shared memory.  The loads of all
// eight neighbours and links are then in flight at once, where k_hop's thread walks
// through them with the registers that four spins' accumulators leave it (8 warps
// per SM).  The components of the result are summed from shared memory, one
// (spin, colour) per warp at a time, in a fixed order.  The clover blocks' elements
// are loaded by the eight warps while the sums are formed and meet the spinor in
// shared memory, one row of the packed matrix per warp at a time.
//
// It serves small lattices, which get eight times the warps of one thread per site
// (8^4 has 16 blocks of 128 sites for 148 SMs), and the NF = 6 clover hop, whose
// 144 clover numbers per site it loads by eight warps.  A large NF = 3 lattice is bound
// by HBM and L2, where 128 consecutive sites per block share their y neighbours in L1
// and 32 do not.  Per operator, FP64, in a CUDA graph of many, against the best of the others:
//   8^4 SU(3) Dphi_eopre                        5.2 us, 6.7 (two threads per site)
//   14x6x10x12 SU(4) antisymmetric g5Dphi_sq   28.4 us, 38.2
//   48x24^3 SU(3) sextet Cphi_eopre             868 us, 839 (links built from the fundamental
//                                                ones, as here); 769 with that hop first
//   32x16^3 SU(3) Cphi_eopre                   75.7 us, 39 (the autotuner keeps the others)
// What bounds it: the latency of one load from L2, two barriers and the launch.  Of two
// hops of an operator the second reads its links, clover blocks and diagonal-term field
// while the first still runs (programmatic dependent launch), and waits for it only
// before the neighbour spinors.  (Several groups of 32 sites per block, for L1 hits
// between them, were slower at every size.)
#pragma once
#include "hop.cuh"

namespace hrgpu {

constexpr int HD_SITES = 32, HD_THREADS = 256;

template <int NFT, typename R, int EP>
struct HopDirLayout {
  typedef typename C2<R>::T V;
  static constexpr int NO = NFT * (2 * NFT - 1);  // off-diagonal elements of a chiral block
  static constexpr int C_BYTES = 8 * 2 * NFT * HD_SITES * (int)sizeof(V);
  static constexpr int CL_BYTES = EP == EP_AXPY ? 0 : 2 * NO * HD_SITES * (int)sizeof(V) + 4 * NFT * HD_SITES * (int)sizeof(R);
  static constexpr int MAIN = C_BYTES > CL_BYTES ? C_BYTES : CL_BYTES;  // products, then the clover blocks
  static constexpr int SMEM = MAIN + (EP == EP_AXPY ? 0 : 4 * NFT * HD_SITES * (int)sizeof(V));
};

// built for the representations whose products and clover blocks fit in shared memory
template <int N>
struct HopDirOK {
  static constexpr bool v = N <= 6;
};

// thread blocks of a whole-lattice launch of a single-field hop variant (the length
// of its |out|^2 partials)
inline int hop_blocks(int variant, long nsites, int nf) {
  if (variant == 1 && nf <= 6) return (int)((nsites + HD_SITES - 1) / HD_SITES);
  const long threads = (variant == 1 || variant == 3) ? 2 * nsites : nsites;
  return (int)((threads + HOP_THREADS - 1) / HOP_THREADS);
}

// the variants whose epilogue has the inverters' forms (HopArgs::racc, red_g5)
inline bool hop_tail_ok(int variant, int nf, bool bf16) {
  return (!bf16 && (variant == 0 || variant == 2 || variant == 6 || (variant == 3 && nf <= 6))) || (variant == 1 && nf <= 6);
}

__device__ __forceinline__ float hd_elem(const __nv_bfloat16 *p) { return __bfloat162float(__ldg(p)); }
__device__ __forceinline__ float2 hd_elem(const __nv_bfloat162 *p) { return __bfloat1622float2(__ldg(p)); }
template <typename E>
__device__ __forceinline__ E hd_elem(const E *p) { return ld_u(p); }

template <bool DAG, typename V>
__device__ __forceinline__ void hd_mac(V &a, V u, V h) {
  if (DAG) cmacc(a, u, h);
  else cmac(a, u, h);
}
template <bool DAG>
__device__ __forceinline__ void hd_mac(double2 &a, double u, double2 h) { rmac(a, u, h); }
template <bool DAG>
__device__ __forceinline__ void hd_mac(float2 &a, float u, float2 h) { rmac(a, u, h); }

// A link as it is read: NF x NF stored elements, rows 0 and 1 (RC), or the fundamental
// link (FR); loaded early where it fits in registers beside a neighbour's spinor.
template <int NFT, bool REAL, typename R, typename LE, bool RC, int FR>
struct HdLink {
  typedef typename C2<R>::T V;
  static constexpr bool bf16 = std::is_same<LE, __nv_bfloat162>::value || std::is_same<LE, __nv_bfloat16>::value;
  static constexpr int NG = FR ? TwoIdx<FR ? FR : 1>::NG : 0;
  static constexpr bool rc = RC && NFT == 3 && !bf16;
  static constexpr int NE = FR ? NG * NG : NFT * NFT;
  static constexpr bool EARLY = NE <= 16;
  typedef typename std::conditional<FR != 0, V, typename std::conditional<bf16, typename std::conditional<REAL, R, V>::type, LE>::type>::type E;
  E u[EARLY ? NE : 1];
  const LE *U;
  long plane;
  R sg;
  // flip: the link crosses the time boundary
  __device__ __forceinline__ void load(const HopArgs<R> &a, int mu, long site, bool flip) {
    plane = 2L * a.g.ld;
    if constexpr (FR != 0) {
      const V *Ug = (const V *)a.Ug + (long)mu * NE * plane + site;
#pragma unroll
      for (int k = 0; k < NE; k++) u[k] = ld_u(Ug + (long)k * plane);
      sg = (a.recon == 4 && flip) ? (R)-1 : (R)1;
    } else {
      U = (const LE *)a.U + (long)mu * NFT * NFT * plane + site;
      if constexpr (rc) {
#pragma unroll
        for (int e = 0; e < 6; e++) u[e] = ld_u(U + (long)e * plane);
        sg = (a.recon == 2 && flip) ? (R)-1 : (R)1;
      } else if constexpr (EARLY) {
#pragma unroll
        for (int e = 0; e < NE; e++) u[e] = hd_elem(U + (long)e * plane);
      }
    }
  }
  __device__ __forceinline__ void ready() {
    if constexpr (rc) {
      if constexpr (REAL) so3_row2(u, sg);
      else su3_row2(u, sg);
    }
  }
  __device__ __forceinline__ E operator()(int i, int j) const {
    if constexpr (FR != 0) return two_idx_elem<FR>(u, i, j, sg);
    else if constexpr (EARLY) return u[i * NFT + j];
    else return hd_elem(U + (long)(i * NFT + j) * plane);
  }
};

// the two products of one link, row by row into shared memory
template <int NFT, bool DAG, typename LK, typename V>
__device__ __forceinline__ void hd_link(const LK &link, V *c0, V *c1, const V (&h0)[NFT], const V (&h1)[NFT]) {
#pragma unroll
  for (int i = 0; i < NFT; i++) {
    V a0 = cmk<V>(0.0, 0.0), a1 = cmk<V>(0.0, 0.0);
#pragma unroll
    for (int j = 0; j < NFT; j++) {
      const auto u = DAG ? link(j, i) : link(i, j);
      hd_mac<DAG>(a0, u, h0[j]);
      hd_mac<DAG>(a1, u, h1[j]);
    }
    c0[i * HD_SITES] = a0;
    c1[i * HD_SITES] = a1;
  }
}

template <int NFT, bool REAL, typename R, int EP, int MINB, typename LE = typename LinkE<REAL, R>::T, bool RC = false,
          int FR = 0>
__global__ void __launch_bounds__(HD_THREADS, MINB) k_hop_dir(HopArgs<R> a) {
  typedef typename C2<R>::T V;
  typedef HopDirLayout<NFT, R, EP> LAY;
  constexpr int NS = 4 * NFT, KC = (NS + 7) / 8;  // components; at most KC per warp
  constexpr int NO2 = 2 * LAY::NO, KO = (NO2 + 7) / 8;
  extern __shared__ __align__(16) unsigned char hd_sm[];
  V *sc = (V *)hd_sm;                       // [8 warps][2][NFT][32]
  V *so = (V *)hd_sm;                       // clover off-diagonal [2 NO][32] ...
  R *sd = (R *)(so + NO2 * HD_SITES);       // ... and diagonal [4 NFT][32], over the products
  V *sx = (V *)(hd_sm + LAY::MAIN);         // the vector the clover blocks act on [NS][32]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, mu = w >> 1, bw = w & 1;
  const Geo g = a.g;
  const long ld = g.ld, lp = 2L * ld;
  const int outp = a.both ? (int)blockIdx.y : a.outp, inp = outp ^ 1;
  const long half = a.both ? (long)NS * ld : 0;  // from the even to the odd half of a full field
  const V *fin = (const V *)a.in + inp * half, *faux = (const V *)a.aux + outp * half;
  V *fout = (V *)a.out + outp * half;
  const R sgn = bw ? (R)-1 : (R)1, ca = a.cacc, g5 = a.g5 ? (R)-1 : (R)1;
  double nrm = 0.0;
  const int base = a.cb0 + blockIdx.x * HD_SITES;
  const bool on = base + lane < a.cb1;
  const int cb = on ? base + lane : a.cb1 - 1;
  int t, x, y, z;
  cb_to_coords(g, cb, outp, t, x, y, z);
  bool flip = t == 0;  // the link crosses the time boundary (mu = 0)
  if (mu == 0) t = bw ? (t == 0 ? g.T - 1 : t - 1) : (t + 1 == g.T ? 0 : t + 1);
  if (mu == 1) x = bw ? (x == 0 ? g.X - 1 : x - 1) : (x + 1 == g.X ? 0 : x + 1);
  if (mu == 2) y = bw ? (y == 0 ? g.Y - 1 : y - 1) : (y + 1 == g.Y ? 0 : y + 1);
  if (mu == 3) z = bw ? (z == 0 ? g.Z - 1 : z - 1) : (z + 1 == g.Z ? 0 : z + 1);
  if (bw) flip = t == 0;
  flip = flip && mu == 0;
  const int cn = coords_to_cb(g, t, x, y, z);
  const long site = (long)outp * ld + cb;
  if (!a.pre) pdl_enter();
  typedef HdLink<NFT, REAL, R, LE, RC, FR> LK;
  LK link;
  link.load(a, mu, bw ? (long)inp * ld + cn : site, flip);
  // what the epilogue reads from memory: with the link where the registers allow it,
  // else on its way while the sums are formed
  constexpr bool EARLY_EP = NFT <= 3;
  V ax[KC], rr[KC];
  V co[EP == EP_AXPY ? 1 : KO];
  R cd[KC];
  const bool axpy = EP == EP_AXPY && a.aux != nullptr && a.caux != (R)0;
  // the inverters' <gamma_5 aux, result> needs aux whether or not it enters the result (m = -4)
  const bool use_aux = EP == EP_CLOV || axpy || (EP == EP_AXPY && a.red_g5);
  auto load_epilogue = [&]() {
#pragma unroll
    for (int k = 0; k < KC; k++)
      if (use_aux && w + 8 * k < NS) ax[k] = ld_c(faux + cb + (long)(w + 8 * k) * ld);
    if constexpr (EP != EP_AXPY) {
      const unsigned long long pol = l2_evict_first();
#pragma unroll
      for (int k = 0; k < KO; k++)
        if (w + 8 * k < NO2) co[k] = ld_ef(a.cod + (long)(w + 8 * k) * lp + site, pol);
#pragma unroll
      for (int k = 0; k < KC; k++)
        if (w + 8 * k < NS) cd[k] = ld_ef(a.cdg + (long)(w + 8 * k) * lp + site, pol);
    }
  };
  if (EARLY_EP) load_epilogue();
  if (a.pre) pdl_enter();
  if (a.stop && *a.stop) return;
  const bool tail = EP != EP_CLOV_INV && a.racc != nullptr;
  {
    const V *s = fin + cn;
    V h0[NFT], h1[NFT];
    // (1 -+ gamma_mu): spins 0 and 1 plus sgn times the partner's
    const int pa = (mu == 0 || mu == 3) ? 2 : 3;
#pragma unroll
    for (int i = 0; i < NFT; i++) {
      const V s0 = ld_c(s + (long)i * ld), s1 = ld_c(s + (long)(NFT + i) * ld);
      V p0 = ld_c(s + (long)(pa * NFT + i) * ld), p1 = ld_c(s + (long)((5 - pa) * NFT + i) * ld);
      p0 = cscale(sgn, p0);
      p1 = cscale(sgn, p1);
      if (mu == 0) { h0[i] = cadd(s0, p0); h1[i] = cadd(s1, p1); }
      else if (mu == 1) { h0[i] = caddi(s0, p0); h1[i] = caddi(s1, p1); }
      else if (mu == 2) { h0[i] = cadd(s0, p0); h1[i] = csub(s1, p1); }
      else { h0[i] = caddi(s0, p0); h1[i] = csubi(s1, p1); }
    }
    V *c0 = sc + (long)(2 * w) * NFT * HD_SITES + lane, *c1 = c0 + NFT * HD_SITES;
    link.ready();
    if (!bw) hd_link<NFT, false>(link, c0, c1, h0, h1);
    else hd_link<NFT, true>(link, c0, c1, h0, h1);
  }
  if (!EARLY_EP) load_epilogue();
  const R om = tail ? (R)*a.omega : (R)0;
#pragma unroll
  for (int k = 0; k < KC; k++)
    if (tail && w + 8 * k < NS) rr[k] = ((const V *)a.racc)[cb + (long)(w + 8 * k) * ld];
  {
    __syncthreads();
    V acc[KC];
#pragma unroll
    for (int k = 0; k < KC; k++) {
      const int comp = w + 8 * k;
      if (comp >= NS) break;
      const int sp = comp / NFT, i = comp % NFT;
      auto C = [&](int m, int b, int h) { return sc[(((2 * m + b) * 2 + h) * NFT + i) * HD_SITES + lane]; };
      V r;
      if (sp < 2) {
        r = cadd(C(0, 0, sp), C(0, 1, sp));
#pragma unroll
        for (int m = 1; m < 4; m++) r = cadd(r, cadd(C(m, 0, sp), C(m, 1, sp)));
      } else if (sp == 2) {
        r = csub(C(0, 0, 0), C(0, 1, 0));
        r = csubi(r, csub(C(1, 0, 1), C(1, 1, 1)));
        r = csub(r, csub(C(2, 0, 1), C(2, 1, 1)));
        r = csubi(r, csub(C(3, 0, 0), C(3, 1, 0)));
      } else {
        r = csub(C(0, 0, 1), C(0, 1, 1));
        r = csubi(r, csub(C(1, 0, 0), C(1, 1, 0)));
        r = cadd(r, csub(C(2, 0, 0), C(2, 1, 0)));
        r = caddi(r, csub(C(3, 0, 1), C(3, 1, 1)));
      }
      r = cscale(ca, r);
      if constexpr (EP == EP_AXPY) {
        if (axpy) rmac(r, a.caux, ax[k]);
      }
      acc[k] = r;
    }
    if constexpr (EP != EP_AXPY) {
#pragma unroll
      for (int k = 0; k < KC; k++)
        if (w + 8 * k < NS) sx[(w + 8 * k) * HD_SITES + lane] = EP == EP_CLOV_INV ? acc[k] : ax[k];
      __syncthreads();  // the products have been read
#pragma unroll
      for (int k = 0; k < KO; k++)
        if (w + 8 * k < NO2) so[(w + 8 * k) * HD_SITES + lane] = co[k];
#pragma unroll
      for (int k = 0; k < KC; k++)
        if (w + 8 * k < NS) sd[(w + 8 * k) * HD_SITES + lane] = cd[k];
      __syncthreads();
#pragma unroll
      for (int k = 0; k < KC; k++) {
        const int comp = w + 8 * k;
        if (comp >= NS) break;
        const int b = comp / (2 * NFT), i = comp % (2 * NFT);
        const V *x = sx + (long)b * 2 * NFT * HD_SITES + lane, *o = so + (long)b * LAY::NO * HD_SITES + lane;
        V y = cscale(sd[comp * HD_SITES + lane], x[i * HD_SITES]);
#pragma unroll
        for (int j = 0; j < 2 * NFT; j++) {
          if (j == i) continue;
          if (j < i) cmac(y, o[(i * (i - 1) / 2 + j) * HD_SITES], x[j * HD_SITES]);
          else cmacc(y, o[(j * (j - 1) / 2 + i) * HD_SITES], x[j * HD_SITES]);
        }
        acc[k] = EP == EP_CLOV ? cadd(acc[k], y) : y;
      }
    }
    V *out = fout + cb;
#pragma unroll
    for (int k = 0; k < KC; k++) {
      const int comp = w + 8 * k;
      if (comp >= NS || !on) break;
      V r = acc[k];
      if (comp >= 2 * NFT) r = cscale(g5, r);
      if (tail) {
        rmac(rr[k], om, r);
        r = rr[k];
      }
      out[(long)comp * ld] = r;
      if (EP != EP_CLOV_INV && a.red_g5) {
        const double q = (double)ax[k].x * r.x + (double)ax[k].y * r.y;
        nrm += comp >= 2 * NFT ? -q : q;
      } else if (a.red) {
        nrm += (double)r.x * r.x + (double)r.y * r.y;
      }
    }
  }
  if (a.red) {
    nrm = block_sum(nrm);
    if (threadIdx.x == 0) a.red[blockIdx.y * gridDim.x + blockIdx.x] = nrm;
  }
}

}  // namespace hrgpu
