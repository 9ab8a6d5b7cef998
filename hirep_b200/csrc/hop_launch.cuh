// hop_launch.cuh -- host-side dispatch of the hopping kernel over NF and the
// epilogue; instantiated once per precision (dirac_d.cu, dirac_f.cu) so the two
// compile in parallel.
#pragma once
#include "dirac.cuh"
#include "hop_async.cuh"
#include "hop_dir.cuh"
#include "hop_tma.cuh"

namespace hrgpu {

// A whole-lattice FP64 hop is launched with programmatic stream serialisation
// (the kernels wait on their predecessor with griddepcontrol.wait before
// reading memory), so its blocks fill the SMs the previous hop's last wave
// leaves idle: Cphi_eopre 62.5 -> 60.4 us at 16^3x32 (alternating A/B in one
// process), the FP64 CG unchanged.  small: variant 1, whose launches overlap in FP32
// as well.  Without it: the other FP32 hops (inside the mixed
// solve's graphs it cost 3 %: 18.7 -> 19.3 ms) and launches over a few time
// slabs (the host-field pipeline, where the early, waiting blocks held SMs
// that the copy-stream kernels beside them needed: 0.47 -> 0.69 ms).
template <typename R>
static inline cudaError_t launch_pdl(void (*kernel)(HopArgs<R>), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                     HopArgs<R> &a, bool small = false) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (L.hop_pdl && !a.no_pdl && (sizeof(R) == 8 || small) && a.cb0 == 0 && a.cb1 == (int)L.VH) ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, a);
}

template <int N, bool RL, typename R, int EP>
int launch_async(HopArgs<R> &a, dim3 grid, dim3 block, cudaStream_t s) {
  if constexpr (AsyncOK<N, RL>::v) {
    constexpr int smem = AsyncLayout<N, RL, R>::SMEM;
    static bool attr = false;
    if (!attr) {
      HR_CUDA(cudaFuncSetAttribute(k_hop_async<N, RL, R, EP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      attr = true;
    }
    HR_CUDA(launch_pdl<R>(k_hop_async<N, RL, R, EP>, grid, block, smem, s, a));
    return 0;
  } else {
    return -1;  // not built for this NF
  }
}

// variant 5: the time halo staged by bulk copies, for the small representations
// and where blocks of HOP_THREADS sites tile the time slabs of the launch
template <int N, bool RL, typename R, int EP>
int launch_tma(HopArgs<R> &a, dim3 grid, dim3 block, cudaStream_t s) {
  if constexpr (AsyncOK<N, RL>::v) {
    const int S = a.g.Xh * a.g.Y * a.g.Z;
    if (S % HOP_THREADS != 0 || a.cb0 % HOP_THREADS != 0 || (a.cb1 - a.cb0) % HOP_THREADS != 0) return -1;
    constexpr int smem = TmaLayout<N, R>::SMEM;
    static bool attr = false;
    if (!attr) {
      HR_CUDA(cudaFuncSetAttribute(k_hop_tma<N, RL, R, EP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      attr = true;
    }
    HR_CUDA(launch_pdl<R>(k_hop_tma<N, RL, R, EP>, grid, block, smem, s, a));
    return 0;
  } else {
    return -1;  // not built for this NF
  }
}

// k_hop for variants 0 and 2: the instantiation that rebuilds row 2 of the
// 3x3 links (SU(3) fundamental, SU(2) adjoint) when the links passed the
// check, else the one reading full links
template <int N, bool RL, typename R, int EP, int MINB>
static inline void (*hop_kernel(int recon, bool tail))(HopArgs<R>) {
  typedef typename LinkE<RL, R>::T LE;
  constexpr bool T = EP != EP_CLOV_INV;  // the first hop of a clover operator has no inverters' form
  if constexpr (N == 3) {
    if (recon) return tail ? k_hop<N, RL, R, EP, MINB, LE, true, 0, T> : k_hop<N, RL, R, EP, MINB, LE, true>;
  }
  return tail ? k_hop<N, RL, R, EP, MINB, LE, false, 0, T> : k_hop<N, RL, R, EP, MINB>;
}

// variant 1: one warp per direction (k_hop_dir) for NF <= 6, two threads per site
// (k_hop2) for larger NF.  Links are built from the fundamental ones where variant 6
// would do so.  Row 2 of a 3 x 3 link is rebuilt in FP32 only: in FP64 that saves nothing on
// the lattices that lie in L2, and its roundings raised the operator's error at 8^4 from
// 1.0e-16 to 1.3e-16; in FP32, whose operator the variants 0 and 2 apply with rebuilt rows as
// well, it takes 7.8 us instead of 11.5 on 10x14x12x20.
template <int N, bool RL, typename R, int EP, typename LE = typename LinkE<RL, R>::T>
int launch_dir(HopArgs<R> &a, long nsites, cudaStream_t s) {
  if constexpr (HopDirOK<N>::v) {
    constexpr bool stored = std::is_same<LE, typename LinkE<RL, R>::T>::value;  // not BF16
    void (*f)(HopArgs<R>) = k_hop_dir<N, RL, R, EP, 2, LE>;
    if constexpr (stored && N == 3 && sizeof(R) == 4) {
      if (a.recon) f = k_hop_dir<N, RL, R, EP, 2, LE, true>;
    }
    if constexpr (stored && N == 6 && !RL) {
      if (a.recon >= 3 && a.Ug) f = L.repr == HRGPU_SYM ? k_hop_dir<N, RL, R, EP, 2, LE, false, 1> : k_hop_dir<N, RL, R, EP, 2, LE, false, 2>;
    }
    constexpr int smem = HopDirLayout<N, R, EP>::SMEM;
    if (smem > 40 * 1024)  // with the static part of the norm's sum, at NF = 6
      if (int rc = allow_smem((const void *)f, smem)) return rc;
    const dim3 grid((unsigned)((nsites + HD_SITES - 1) / HD_SITES), a.both ? 2 : 1);
    HR_CUDA(launch_pdl<R>(f, grid, dim3(HD_THREADS), smem, s, a, true));
  } else {
    const dim3 grid((unsigned)((2 * nsites + HOP_THREADS - 1) / HOP_THREADS));
    HR_CUDA(launch_pdl<R>(k_hop2<N, RL, R, EP, 1, LE>, grid, dim3(HOP_THREADS), 0, s, a));
  }
  return 0;
}

// variant 3: two threads per site.  For NF <= 6 with the registers that it takes: capped for
// 4 blocks per SM it was slower than that, or than variants 0 and 2, at every size from
// 4^3 x 8 to 24^4 (2 to 6 colours, FP64 and FP32, with and without clover), while uncapped it
// is the best one between the sizes of variant 1 and of variant 0: 20.4 us per operator against
// 25.9 for g5Cphi of SU(4) on 10x14x12x20, 28.7 against 34.9 for the FP32 clover operator of
// SU(4) antisymmetric.  Larger NF has it uncapped as variant 1.
template <int N, bool RL, typename R, int EP, typename LE = typename LinkE<RL, R>::T>
static inline void (*hop2_kernel(bool tail))(HopArgs<R>) {
  constexpr bool T = HopDirOK<N>::v && EP != EP_CLOV_INV && std::is_same<LE, typename LinkE<RL, R>::T>::value;
  constexpr int MINB = HopDirOK<N>::v ? 1 : 4;
  return tail ? k_hop2<N, RL, R, EP, MINB, LE, T> : k_hop2<N, RL, R, EP, MINB, LE>;
}

// variant 6: k_hop (variant 0's register budget) building the NF = 6
// two-index links from the fundamental ones (FP64 from L.Ug, FP32 from its
// float copy L.Ugf) while the fundamental links are those the represented
// field was made from (link modes 3 and 4); -1 otherwise
template <int N, bool RL, typename R, int EP>
int launch_fund(HopArgs<R> &a, dim3 grid, dim3 block, cudaStream_t s) {
  if constexpr (N == 6 && !RL) {
    if (a.recon < 3 || !a.Ug) return -1;
    typedef typename LinkE<RL, R>::T LE;
    constexpr bool T = EP != EP_CLOV_INV;
    const bool tail = a.racc || a.red_g5;
    void (*f)(HopArgs<R>);
    if (L.repr == HRGPU_SYM) f = tail ? k_hop<N, RL, R, EP, 1, LE, false, 1, T> : k_hop<N, RL, R, EP, 1, LE, false, 1>;
    else f = tail ? k_hop<N, RL, R, EP, 1, LE, false, 2, T> : k_hop<N, RL, R, EP, 1, LE, false, 2>;
    HR_CUDA(launch_pdl<R>(f, grid, block, 0, s, a));
    return 0;
  } else {
    return -1;
  }
}

template <typename R, int EP>
int launch_ep_variant(HopArgs<R> &a, int variant) {
  a.g = make_geo();
  a.nf = L.nf;
  a.recon = L.recon_allow ? L.recon12 : 0;
  // variants: 0 one thread per site, 1 one warp per direction (NF <= 6; else two threads
  // per site, spin split), 2 as 0 with the register budget capped for 4 resident blocks
  // per SM, 3 the spin split (NF > 6: capped likewise),
  // 4 one thread per site with the per-direction loads pipelined through shared memory,
  // 5 one thread per site with the time halo staged by bulk (TMA) copies,
  // 6 one thread per site building the NF = 6 two-index links from the fundamental ones
  const long nsites = a.cb1 - a.cb0;
  dim3 grid((unsigned)((nsites + HOP_THREADS - 1) / HOP_THREADS)), block(HOP_THREADS);
  dim3 grid2((unsigned)((2 * nsites + HOP_THREADS - 1) / HOP_THREADS));
  const bool tail = a.racc || a.red_g5;
  cudaStream_t s = L.stream;
#define HOPV(N, RL)                                                                    \
  case N:                                                                              \
    switch (variant) {                                                                 \
      case 0: HR_CUDA(launch_pdl<R>(hop_kernel<N, RL, R, EP, 1>(a.recon, tail), grid, block, 0, s, a)); break; \
      case 1:                                                                          \
        if (int rc_ = launch_dir<N, RL, R, EP>(a, nsites, s)) return rc_;              \
        break;                                                                         \
      case 3: HR_CUDA(launch_pdl<R>(hop2_kernel<N, RL, R, EP>(tail), grid2, block, 0, s, a)); break; \
      case 2: HR_CUDA(launch_pdl<R>(hop_kernel<N, RL, R, EP, 4>(a.recon, tail), grid, block, 0, s, a)); break; \
      case 4:                                                                          \
        if (int rc_ = launch_async<N, RL, R, EP>(a, grid, block, s)) return rc_;       \
        break;                                                                         \
      case 5:                                                                          \
        if (int rc_ = launch_tma<N, RL, R, EP>(a, grid, block, s)) return rc_;         \
        break;                                                                         \
      default:                                                                         \
        if (int rc_ = launch_fund<N, RL, R, EP>(a, grid, block, s)) return rc_;        \
        break;                                                                         \
    }                                                                                  \
    break;
#define HOPC(N) HOPV(N, false)
#define HOPR(N) HOPV(N, true)
  // FP32 operator with BF16 link storage: variants 0-3 (no cp.async form)
#define HOPVB(N, RL)                                                                            \
  case N:                                                                                       \
    switch (variant) {                                                                          \
      case 0: HR_CUDA(launch_pdl<float>(k_hop<N, RL, float, EP, 1, typename LinkBF16<RL>::T>, grid, block, 0, s, a)); break;  \
      case 1:                                                                                   \
        if (int rc_ = launch_dir<N, RL, float, EP, typename LinkBF16<RL>::T>(a, nsites, s)) return rc_; \
        break;                                                                                  \
      case 3: HR_CUDA(launch_pdl<float>(hop2_kernel<N, RL, float, EP, typename LinkBF16<RL>::T>(false), grid2, block, 0, s, a)); break; \
      case 2: HR_CUDA(launch_pdl<float>(k_hop<N, RL, float, EP, 4, typename LinkBF16<RL>::T>, grid, block, 0, s, a)); break;  \
      default: return -1;                                                                       \
    }                                                                                           \
    break;
  if constexpr (std::is_same<R, float>::value) {
    if (L.flt_links == HRGPU_LINKS_BF16) {
      if (!L.real) {
        switch (L.nf) {
          HOPVB(2, false) HOPVB(3, false) HOPVB(4, false) HOPVB(5, false) HOPVB(6, false) HOPVB(10, false)
          default: set_error("no hopping kernel instantiated for complex NF=%d", L.nf); return HRGPU_E_NF;
        }
      } else {
        switch (L.nf) {
          HOPVB(3, true) HOPVB(8, true) HOPVB(15, true)
          default: set_error("no hopping kernel instantiated for real NF=%d", L.nf); return HRGPU_E_NF;
        }
      }
      HR_LAUNCH_CHECK();
      return 0;
    }
  }
#undef HOPVB
  if (!L.real) {
    switch (L.nf) {
      HOPC(2) HOPC(3) HOPC(4) HOPC(5) HOPC(6) HOPC(10)
      default: set_error("no hopping kernel instantiated for complex NF=%d", L.nf); return HRGPU_E_NF;
    }
  } else {
    switch (L.nf) {
      HOPR(3) HOPR(8) HOPR(15)
      default: set_error("no hopping kernel instantiated for real NF=%d", L.nf); return HRGPU_E_NF;
    }
  }
#undef HOPC
#undef HOPR
#undef HOPV
  HR_LAUNCH_CHECK();
  return 0;
}

// variant 5 (pinned with hrgpu_set_hop_variant): the launch gets the device
// error word, and outside a stream capture the word is read back at once, so a
// bounded wait that gave up (copies possibly still in flight into shared
// memory) is reported as an error status instead of passing silently
template <typename R, int EP>
int launch_tma_checked(HopArgs<R> &a) {
  if (!L.hop_err) {
    HR_CUDA(cudaMalloc(&L.hop_err, sizeof(unsigned)));
    HR_CUDA(cudaMemsetAsync(L.hop_err, 0, sizeof(unsigned), L.stream));
  }
  a.err = L.hop_err;
  int rc = launch_ep_variant<R, EP>(a, 5);
  a.err = nullptr;
  if (rc < 0) {
    set_error("hopping-kernel variant 5 is not built for NF=%d (or this lattice)", L.nf);
    return HRGPU_E_NF;
  }
  if (rc) return rc;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  HR_CUDA(cudaStreamIsCapturing(L.stream, &cs));
  if (cs != cudaStreamCaptureStatusNone) return 0;
  unsigned h = 0;
  HR_CUDA(cudaMemcpyAsync(&h, L.hop_err, sizeof(unsigned), cudaMemcpyDeviceToHost, L.stream));
  HR_CUDA(cudaStreamSynchronize(L.stream));
  if (h) {
    HR_CUDA(cudaMemsetAsync(L.hop_err, 0, sizeof(unsigned), L.stream));
    set_error("hopping-kernel variant 5: a bounded wait for the staged time halo gave up (error word %u)", h);
    return HRGPU_E_CUDA;
  }
  return 0;
}

// Autotuner: the first launch of each (precision, epilogue) on a lattice times
// every variant on the real arguments (3 or 16 launches each, CUDA events on the
// library stream) and keeps the faster one.  The output is rewritten by the
// final launch, so tuning does not change results.  (The even-odd operators choose
// by their two hops together, see eo_stage.)  hrgpu_set_hop_variant forces
// a variant (tests use it to check both).
template <typename R, int EP>
int launch_ep(HopArgs<R> &a) {
  // tuning slots: FP64, FP32, FP32 with BF16 links
  const int pi = sizeof(R) == 8 ? 0 : (L.flt_links == HRGPU_LINKS_BF16 ? 2 : 1);
  int &v = L.hop_variant[pi][EP];
  if (L.hop_force >= 0) {
    if (L.hop_force == 5) return launch_tma_checked<R, EP>(a);
    int rc = launch_ep_variant<R, EP>(a, L.hop_force);
    if (rc < 0) {
      set_error("hopping-kernel variant %d is not built for NF=%d", L.hop_force, L.nf);
      return HRGPU_E_NF;
    }
    return rc;
  }
  if (v < 0 && (a.cb0 != 0 || a.cb1 != L.VH || a.racc)) {
    // a launch over part of the lattice is no measure for the full operator, and
    // one that accumulates cannot be repeated: run the default variant and leave
    // tuning to the first full launch
    return launch_ep_variant<R, EP>(a, 0);
  }
  if (v < 0) {
    // nothing can be timed while the stream is being captured into a CUDA
    // graph: run the default variant and leave tuning to an uncaptured launch
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    HR_CUDA(cudaStreamIsCapturing(L.stream, &cs));
    if (cs != cudaStreamCaptureStatusNone) return launch_ep_variant<R, EP>(a, 0);
  }
  if (v < 0) {
    float best = 1e30f;
    int bestv = 0;
    cudaEvent_t e0, e1;
    HR_CUDA(cudaEventCreate(&e0));
    if (cudaError_t err = cudaEventCreate(&e1)) {
      cudaEventDestroy(e0);
      return fail_cuda(err, "cudaEventCreate(&e1)", __FILE__, __LINE__);
    }
    // milliseconds per launch.  A launch costs the host 2.4 to 2.8 us, as long as a hop of a
    // small lattice takes: the launches queue up behind a delay, so that what is timed is the
    // GPU (without it the best variant of 8 x 12 x 10 x 12 SU(2) adjoint, 3.4 us per hop, was
    // read as 7.5 and passed over for one of 6.2).  A short hop is timed over more launches
    // than a long one: the events resolve half a microsecond.
    auto timed = [&](int cand, int reps, float *ms) -> int {
      if (int rc = stream_delay(reps < 16 ? 30.0 : 80.0)) return rc;
      if (int rc = launch_ep_variant<R, EP>(a, cand)) return rc;
      HR_CUDA(cudaEventRecord(e0, L.stream));
      for (int r = 0; r < reps; r++)
        if (int rc = launch_ep_variant<R, EP>(a, cand)) return rc;
      HR_CUDA(cudaEventRecord(e1, L.stream));
      HR_CUDA(cudaEventSynchronize(e1));
      HR_CUDA(cudaEventElapsedTime(ms, e0, e1));
      *ms /= reps;
      return 0;
    };
    // the events are destroyed on every way out of the loop
    auto tune = [&]() -> int {
      for (int cand = 0; cand < HOP_VARIANTS; cand++) {
        if (cand == 5) {  // the TMA-staged variant: slower in every measured case, pinned only
          L.hop_tune_ms[pi][EP][cand] = -1.0f;
          continue;
        }
        int rc0 = launch_ep_variant<R, EP>(a, cand);  // warm-up
        if (rc0 < 0) {  // variant not built for this NF
          L.hop_tune_ms[pi][EP][cand] = -1.0f;
          continue;
        }
        if (rc0) return rc0;
        float ms = 0;
        if (int rc = timed(cand, 3, &ms)) return rc;
        if (ms < 0.03f)
          if (int rc = timed(cand, 16, &ms)) return rc;
        L.hop_tune_ms[pi][EP][cand] = ms;
        if (ms < best) {
          best = ms;
          bestv = cand;
        }
      }
      return 0;
    };
    const int trc = tune();
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (trc) return trc;
    // the candidates are timed on back-to-back launches with the operands
    // warm in L2, which favours the register-capped variants slightly over a
    // cold step (16^3x32 FP64: variant 2 1.5 % ahead warm, variant 0 1.5 %
    // ahead with L2 flushed): another variant replaces variant 0 only when it
    // is at least 3 % faster
    const float t0 = L.hop_tune_ms[pi][EP][0];
    if (bestv != 0 && t0 > 0.0f && best > 0.97f * t0) bestv = 0;
    v = bestv;
  }
  int rc = launch_ep_variant<R, EP>(a, v);
  // variant 6 chosen while the links could be built from the fundamental ones,
  // and the fundamental links written since: the stored links, variant 0
  if (rc < 0 && v == 6) rc = launch_ep_variant<R, EP>(a, 0);
  if (rc < 0) {
    set_error("hopping-kernel variant %d is not built for NF=%d", v, L.nf);
    return HRGPU_E_NF;
  }
  return rc;
}




}  // namespace hrgpu
