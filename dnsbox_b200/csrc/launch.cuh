// Launchers of the size-templated pass kernels.  Each (precision, N) pair is
// explicitly instantiated in its own translation unit (inst.cu built once per
// pair), so the library compiles in parallel; api.cu sees declarations only.
#pragma once

#include <type_traits>

#include "kernels.cuh"
#include "kernels_tc.cuh"
#include "kernels_tma.cuh"

namespace dnsbox {

// Launches a kernel that begins with pdl_launch / pdl_wait so that it may start
// while its predecessor in the stream ends.
template <typename... KA, typename... A>
static inline cudaError_t launch_pdl(void (*kernel)(KA...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, KA(args)...);
}

template <typename T, int N> struct Launcher {
  static cudaError_t strided(const StridedArgs<T> &a, bool inv, int ntiles, cudaStream_t st);
  static int strided_threads();   // of a block
  // tensor-core split-precision form of `strided` (FP32, N = 128 .. 1024);
  // adft: the four DFT-64 operands, status: set to 1 if an MMA wait gave up
  static cudaError_t strided_tc(const StridedArgs<T> &a, bool inv, int nother, const void *adft, int *status,
                                int nctas, cudaStream_t st);
  static bool has_tc();
  // TMA-staged tensor-core pass of the right-hand side (FP32, N = 128 .. 512)
  static cudaError_t strided_tma(const TmaArgs &a, bool inv, const void *adft, int *status, int nctas,
                                 cudaStream_t st);
  static bool has_tma();
  // variant: at lines whose fields fit a warp's registers (XReg) there is one kernel; at 512 in FP64
  // 1 is the block kernel and anything else the warp kernel; at 1024 the block kernel
  static cudaError_t xline_nl(const XlineNLArgs<T> &a, int variant, cudaStream_t st);
  static bool has_xline_warp();
  static bool has_xline_vjp();
  static cudaError_t xline_vjp(const XlineVjpArgs<T> &a, cudaStream_t st);
  static cudaError_t xline_c2r(const XlineArgs<T> &a, int nf, cudaStream_t st);
  static cudaError_t xline_r2c(const XlineArgs<T> &a, int nf, cudaStream_t st);
};

#define DNSBOX_SIZES(X) X(8) X(12) X(16) X(24) X(32) X(48) X(64) X(96) X(128) X(192) X(256) X(512) X(1024)

#ifdef DNSBOX_LAUNCH_IMPL
// Opts the kernel in to `bytes` of dynamic shared memory where the 48 KB every
// kernel may use (static + dynamic; no kernel here has 4 KB of static) does
// not cover them; refuses sizes over the 227 KB per-CTA limit.
template <typename K>
static cudaError_t set_smem(K kernel, size_t bytes) {
  if (bytes > 227 * 1024) return cudaErrorInvalidConfiguration;
  if (bytes <= 44 * 1024) return cudaSuccess;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <typename T, int N, bool INV, int MODE>
static cudaError_t strided_launch(const StridedArgs<T> &a, dim3 nb, cudaStream_t st) {
  using SH = StridedShape<T, N>;
  const cudaError_t e = set_smem(k_strided<T, N, INV, MODE>, SH::smem(INV));
  if (e != cudaSuccess) return e;
  return launch_pdl(k_strided<T, N, INV, MODE>, nb, SH::NT, SH::smem(INV), st, a);
}

template <typename T, int N>
cudaError_t Launcher<T, N>::strided(const StridedArgs<T> &a, bool inv, int ntiles, cudaStream_t st) {
  const bool tail = a.band.n || a.cfl.on;   // one more block per box
  const dim3 nb((unsigned)ntiles * a.njobs + (tail ? 1 : 0), (unsigned)(a.nbatch > 0 ? a.nbatch : 1));
  // the workspace modes of the passes that use them (inverse: state or
  // workspace to workspace, forward: workspace to either); pruned columns need
  // the compact workspace
  const int ws = a.kcol.a && !a.compact ? 0 : a.ws;
  if ((a.band.n && !(inv && ws == 2 && strided_threads() >= 32)) || (a.cfl.on && (inv || ws != 3))) return cudaErrorInvalidValue;
  if (inv) {
    if (ws == 3) return strided_launch<T, N, true, ST_WS>(a, nb, st);
    if (ws == 2) return strided_launch<T, N, true, ST_TO_WS>(a, nb, st);
    return strided_launch<T, N, true, ST_ANY>(a, nb, st);
  }
  if (ws == 3) return strided_launch<T, N, false, ST_WS>(a, nb, st);
  if (ws == 1) return strided_launch<T, N, false, ST_FROM_WS>(a, nb, st);
  return strided_launch<T, N, false, ST_ANY>(a, nb, st);
}

template <typename T, int N> int Launcher<T, N>::strided_threads() { return StridedShape<T, N>::NT; }

template <typename T, int N> bool Launcher<T, N>::has_tc() {
  return std::is_same<T, float>::value && TcPlan<N>::on;
}

template <typename T, int N>
cudaError_t Launcher<T, N>::strided_tc(const StridedArgs<T> &a, bool inv, int nother, const void *adft,
                                       int *status, int nctas, cudaStream_t st) {
  if constexpr (std::is_same<T, float>::value && TcPlan<N>::on) {
    using PL = TcPlan<N>;
    TcArgs g;
    g.ntx = strided_ntx(a, PL::TCW);   // column tiles of the (possibly pruned) grid
    g.nother = nother;
    const long long total = (long long)a.njobs * g.ntx * nother * (a.nbatch > 0 ? a.nbatch : 1);
    if (total == 0) return cudaSuccess;
    if (total + 2LL * nctas >= (1LL << 31)) return cudaErrorInvalidValue;
    if ((long long)N * a.rowstride >= (1LL << 31) || (long long)N * out_rowstride(a) >= (1LL << 31))
      return cudaErrorInvalidValue;   // 32-bit row offsets
    g.total = (int)total;
    g.per_box.init((unsigned)(a.njobs * g.ntx * nother));
    g.njobs.init((unsigned)a.njobs);
    g.ntxd.init((unsigned)g.ntx);
    const unsigned nb = (unsigned)(g.total < nctas ? g.total : nctas);
    const __half *A = reinterpret_cast<const __half *>(adft) + (inv ? 2 * 128 * 64 : 0);
    cudaError_t e;
    // two 96 KB CTAs per SM: ask for the largest shared-memory carveout
    if ((e = cudaFuncSetAttribute(inv ? k_strided_tc<N, true> : k_strided_tc<N, false>,
                                  cudaFuncAttributePreferredSharedMemoryCarveout, 100)) != cudaSuccess)
      return e;
    if (inv) {
      if ((e = set_smem(k_strided_tc<N, true>, PL::SMEM)) != cudaSuccess) return e;
      k_strided_tc<N, true><<<nb, PL::THREADS, PL::SMEM, st>>>(a, g, A, status);
    } else {
      if ((e = set_smem(k_strided_tc<N, false>, PL::SMEM)) != cudaSuccess) return e;
      k_strided_tc<N, false><<<nb, PL::THREADS, PL::SMEM, st>>>(a, g, A, status);
    }
    return cudaGetLastError();
  } else {
    (void)a, (void)inv, (void)nother, (void)adft, (void)status, (void)nctas, (void)st;
    return cudaErrorInvalidValue;
  }
}

template <typename T, int N> bool Launcher<T, N>::has_tma() {
  return std::is_same<T, float>::value && TmaPlan<N>::on;
}

template <typename T, int N>
cudaError_t Launcher<T, N>::strided_tma(const TmaArgs &a, bool inv, const void *adft, int *status, int nctas,
                                        cudaStream_t st) {
  if constexpr (std::is_same<T, float>::value && TmaPlan<N>::on) {
    using PL = TmaPlan<N>;
    if (a.total == 0) return cudaSuccess;
    const unsigned nb = (unsigned)(a.total < nctas ? a.total : nctas);
    const __half *A = reinterpret_cast<const __half *>(adft) + (inv ? 2 * 128 * 64 : 0);
    cudaError_t e;
    if (inv) {
      if ((e = set_smem(k_strided_tma<N, true>, PL::SMEM)) != cudaSuccess) return e;
      k_strided_tma<N, true><<<nb, PL::THREADS, PL::SMEM, st>>>(a, A, status);
    } else {
      if ((e = set_smem(k_strided_tma<N, false>, PL::SMEM)) != cudaSuccess) return e;
      k_strided_tma<N, false><<<nb, PL::THREADS, PL::SMEM, st>>>(a, A, status);
    }
    return cudaGetLastError();
  } else {
    (void)a, (void)inv, (void)adft, (void)status, (void)nctas, (void)st;
    return cudaErrorInvalidValue;
  }
}

template <typename T, int N> bool Launcher<T, N>::has_xline_warp() { return XlineWarp<T, N>::on; }

// Threads of an x-line block of up to nt, P to a sequence: smaller blocks where
// the sequences are few, so that each of the 148 SMs gets four, for sequences of
// up to 8 threads.  Halved against not, us: step 32^3 FP32 39.1 / 40.2, 48^3 57.0 / 58.7;
// transposed term 48^3 35.6 / 37.2, 64^3 FP64 38.6 / 38.7; C2R 24^3 5.6 / 6.4, 64^3 6.4 /
// 7.0.  With 16 and 32 threads a sequence it loses: step 256 x 16 x 16 48.4 / 45.6,
// 128 x 32 x 32 FP64 59.1 / 58.4, 512 x 16 x 16 57.2 / 56.4.
static inline int xline_threads(int P, int nt, long long sequences) {
  while (P <= 8 && nt > 32 && sequences * P < 148LL * 4 * nt) nt >>= 1;
  return nt;
}

template <typename T, int N>
cudaError_t Launcher<T, N>::xline_nl(const XlineNLArgs<T> &a, int variant, cudaStream_t st) {
  using C = typename CT<T>::type;
  cudaError_t e;
  if constexpr (SplitPlan<N>::on && (sizeof(T) == 4 || N == 192)) {
    // by the lines of one box, so that a box runs the same arithmetic whatever
    // other boxes or ranks share its launch.  Split against equal shares, us:
    // 192 points 9216 lines FP32 23.8 / 25.3, FP64 43.5 / 46.3, 36864 lines 68 / 77,
    // 148 / 165; 96 points FP32 8192 lines 14.9 / 14.6, 18432 25.9 / 27.3, 36864
    // 43.1 / 48.7, 32 boxes of 9216 255 / 290.  Below, its barriers cost more than
    // they save (192 points, 4608 lines, FP32: 19.5 / 17.0); at 96 points in FP64
    // it gains nothing (9216 lines 26.8 / 25.7, 36864 84.8 / 86.2).
    using SH = XSplit<T, N>;
    if (a.box_lines >= 8192) {
      const unsigned blocks = (unsigned)((a.nlines + SH::L - 1) / SH::L);
      if ((e = set_smem(k_xline_nl_s<T, N>, SH::smem)) != cudaSuccess) return e;
      return launch_pdl(k_xline_nl_s<T, N>, blocks, SH::NT, SH::smem, st, a);
    }
  }
  if constexpr (XReg<T, N>::on) {   // whatever the choice
    using SH = XReg<T, N>;
    const int nt = xline_threads(SH::PL::P, SH::NT, a.nlines);
    const int lpb = nt / SH::PL::P;
    if ((e = set_smem(k_xline_nl_g<T, N>, SH::smem(nt))) != cudaSuccess) return e;
    return launch_pdl(k_xline_nl_g<T, N>, (unsigned)((a.nlines + lpb - 1) / lpb), nt, SH::smem(nt), st, a);
  } else {
    if constexpr (XlineWarp<T, N>::on) {
      if (variant != 1) {   // one warp per line pair
        constexpr int WPB = XlineWarp<T, N>::wpb;
        constexpr int LDC = N + N / XlineWarp<T, N>::Plan::R[0];
        const size_t smem = (size_t)WPB * 6 * LDC * sizeof(C);
        const long long pairs = (a.nlines + 1) / 2;
        if ((e = set_smem(k_xline_nl_w<T, N>, smem)) != cudaSuccess) return e;
        k_xline_nl_w<T, N><<<(unsigned)((pairs + WPB - 1) / WPB), 32 * WPB, smem, st>>>(a);
        return cudaGetLastError();
      }
    }
    constexpr int B = XlineB<T, N>::v;
    const size_t smem = (size_t)N * (3 * B + 1) * sizeof(C);
    const int nt = round32(3 * B * (N / FftPlan<N>::E));
    if ((e = set_smem(k_xline_nl<T, N>, smem)) != cudaSuccess) return e;
    k_xline_nl<T, N><<<(unsigned)((a.nlines + B - 1) / B), nt, smem, st>>>(a);
  }
  return cudaGetLastError();
}

template <typename T, int N> bool Launcher<T, N>::has_xline_vjp() { return XReg<T, N>::on; }
template <typename T, int N>
cudaError_t Launcher<T, N>::xline_vjp(const XlineVjpArgs<T> &a, cudaStream_t st) {
  if constexpr (XReg<T, N>::on) {
    using SH = XReg<T, N>;
    const int nt = xline_threads(SH::PL::P, SH::NT, a.nlines);   // an even number of lines
    const int lpb = nt / SH::PL::P;
    const cudaError_t e = set_smem(k_xline_vjp<T, N>, SH::smem(nt));
    if (e != cudaSuccess) return e;
    return launch_pdl(k_xline_vjp<T, N>, (unsigned)((a.nlines + lpb - 1) / lpb), nt, SH::smem(nt), st, a);
  } else {
    (void)a, (void)st;
    return cudaErrorInvalidValue;
  }
}

template <typename T, int N>
cudaError_t Launcher<T, N>::xline_c2r(const XlineArgs<T> &a, int nf, cudaStream_t st) {
  using SH = XPlain<T, N>;
  const int nt = xline_threads(SH::PL::P, SH::NT, (long long)nf * a.nlines / 2), lpb = 2 * (nt / SH::PL::P);
  const cudaError_t e = set_smem(k_xline_c2r<T, N>, SH::smem(nt));
  if (e != cudaSuccess) return e;
  return launch_pdl(k_xline_c2r<T, N>, dim3((unsigned)((a.nlines + lpb - 1) / lpb), (unsigned)nf), nt, SH::smem(nt), st, a);
}

template <typename T, int N>
cudaError_t Launcher<T, N>::xline_r2c(const XlineArgs<T> &a, int nf, cudaStream_t st) {
  using SH = XPlain<T, N>;
  const int nt = xline_threads(SH::PL::P, SH::NT, (long long)nf * a.nlines / 2), lpb = 2 * (nt / SH::PL::P);
  const cudaError_t e = set_smem(k_xline_r2c<T, N>, SH::smem(nt));
  if (e != cudaSuccess) return e;
  return launch_pdl(k_xline_r2c<T, N>, dim3((unsigned)((a.nlines + lpb - 1) / lpb), (unsigned)nf), nt, SH::smem(nt), st, a);
}

#endif

}  // namespace dnsbox
