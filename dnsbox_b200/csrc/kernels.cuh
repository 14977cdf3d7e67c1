// Pass kernels of the dnsbox B200 pseudospectral step.
//
// Every spectral or mixed-space array is [nz][ny][nxh] complex with the kx
// (half-axis) index fastest; physical arrays are [nz][ny][nx] real.  A 3D
// transform is three passes, one per axis:
//   z and y : k_strided  -- tiles of TC consecutive kx columns x N rows along
//             the axis; each CTA runs one "job" (one output field) whose input
//             is in1*(a1 + i b1 k) + in2*(a2 + i b2 k), which fuses the spectral
//             curl into the inverse transforms;
//   x       : k_xline_*  -- whole lines along x, two real lines per complex FFT.
// The nonlinear term fuses the last inverse x pass, the u x omega product, the
// max|u_i| (CFL) reduction and the first forward x pass (k_xline_nl_g, ..); after
// the last forward z pass (k_strided, in place) one streaming kernel applies
// dealiasing, pressure projection, band forcing, the integrating-factor
// stepper and the energy/dissipation row sums (k_finish_rows).
#pragma once

#include <cmath>
#include <type_traits>

#include "../../include/dnsbox.h"
#include "common.cuh"
#include "fft.cuh"
#include "fftv.cuh"

namespace dnsbox {

// Blocks are launched with a multiple of 32 threads (full warps for the
// shuffle reductions); threads beyond the FFT's own count only take part in
// the strided element loops and barriers.
__host__ __device__ constexpr int round32(int x) { return (x + 31) / 32 * 32; }
// Resident CTAs to ask the register allocator for: `want` for blocks of up
// to 256 threads, one for larger blocks (which hold enough warps alone).
__host__ __device__ constexpr int min_ctas(int threads, int want) { return threads <= 256 ? want : 1; }

// Host/device step bookkeeping kept in device memory (one per context).
struct StepState {
  double dt;        // step size of the current step
  double t;         // time at the start of the current step
  double t_prev;    // time at the start of the previous step (AB2 history)
  double eband;     // rhs_Eband of the current RHS input
  double umax[3];   // max |u_i| of the current RHS input (atomic max)
  double courant;   // io_Courant of the step's initial state with dt
  double eband1;    // eband of the step's first RHS (for the diagnostics)
  double step;      // step counter
  unsigned rec_done, pad0;   // planes of the step record that are through (0 between launches)
  double pad[5];
};

// Programmatic dependent launch: a kernel launched with launch_pdl may start
// while its predecessor's last blocks run, so its launch and its prologue
// (indices, twiddle tables) are hidden; it waits for the predecessor's end
// before it touches memory any kernel writes.  Every kernel so launched lets
// its own successor start early too, and waits before anything else it does
// on global memory but read constant tables.
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// io_Courant (io.f90:664-676) on the fused max|u_i| of one box and, when
// control is on, set_time_step (dnsboxheun.f90:153-157, 227-246).  The maxima
// are consumed: they start the next right-hand side at zero.
struct CflArgs {
  int on, control, force, ring_cap;
  double dx, dy, dz, cmin, cmax, dtmax;
  dnsbox_diag *ring;
};
__device__ __forceinline__ void cfl_update(const CflArgs &c, StepState *st, int box, int nbatch) {
  const double umax[3] = {st->umax[0], st->umax[1], st->umax[2]};
  dnsbox_diag *drec = c.ring ? c.ring + ((long long)st->step % c.ring_cap) * nbatch + box : nullptr;
  double dt = st->dt;
  double C = umax[0] * dt / c.dx + umax[1] * dt / c.dy + umax[2] * dt / c.dz;
  if (c.control && (c.force || C > c.cmax || (C < c.cmin && dt < c.dtmax))) {
    double nd = ((c.cmax + c.cmin) / (2.0 * C)) * dt;
    if (nd > c.dtmax) nd = c.dtmax;
    C = C * nd / dt;
    st->dt = nd;
    dt = nd;
  }
  st->courant = C;
  st->eband1 = st->eband;
  if (drec) {
    drec->courant = C;
    drec->umax[0] = umax[0];
    drec->umax[1] = umax[1];
    drec->umax[2] = umax[2];
    drec->eband = st->eband;
    drec->dt = dt;
  }
  st->umax[0] = st->umax[1] = st->umax[2] = 0.0;   // for the next right-hand side that takes the maxima
}

// The band modes of rhs_Eband, (offset lo, offset hi, kx) triples.
struct BandArgs {
  const int *modes;
  int n;            // 0: none
  double s2;
  StepState *st;
  const void *u;    // the right-hand side's input, components nh apart, boxes bstride apart
  long long nh, bstride;
};
// rhs_Eband (rhs.f90:137-168) of box `box` by a block of NT threads, a power of
// two from 32 on (red: a double per 32 sums); optionally resets the CFL maxima.
// 256 partial sums (modes j, j + 256, ..) and a fixed tree over them, whatever the
// number of threads: the band energy is one number, of a block of its own and of
// a tail block of any pass A.
constexpr int kBandRed = 256;
template <typename C, int NT>
__device__ __forceinline__ void eband_block(const BandArgs &b, int nx, int box, bool reset_umax, double *red) {
  const C *u = reinterpret_cast<const C *>(b.u) + (long long)box * b.bstride;
  StepState *st = b.st + box;
  auto energy = [&](int i) {
    const long long off = (long long)(unsigned)b.modes[3 * i] | ((long long)b.modes[3 * i + 1] << 32);
    const double w = (k_half(b.modes[3 * i + 2], nx, 1.0) == 0.0) ? 0.5 : 1.0;   // rhs.f90:151-155
    double e = 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const C v = u[c * b.nh + off];
      e = fma(fma((double)v.x, (double)v.x, __dmul_rn(v.y, v.y)), w, e);   // one rounding in every kernel
    }
    return e;
  };
  // thread t of P owns the sums t, t + P, .., in registers; a warp's shuffles add
  // 32 neighbouring ones
  constexpr int P = NT < kBandRed ? NT : kBandRed, M = kBandRed / P, Q = M < 4 ? M : 4;   // Q modes in flight
  static_assert(P >= 32 && kBandRed % P == 0, "whole warps");
  const int t = threadIdx.x;
  if (t < P) {
    double s[M];
#pragma unroll
    for (int m = 0; m < M; ++m) s[m] = 0.0;
    for (int i = t; i < b.n; i += kBandRed)
#pragma unroll
      for (int q = 0; q < M; q += Q) {
        if (i - t + q * P >= b.n) break;
        double e[Q];
#pragma unroll
        for (int m = 0; m < Q; ++m) e[m] = energy(min(i + (q + m) * P, b.n - 1));
#pragma unroll
        for (int m = 0; m < Q; ++m)
          if (i + (q + m) * P < b.n) s[q + m] += e[m];
      }
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int g = t / 32 + m * (P / 32);
      if (32 * g < b.n) s[m] = warp_sum(s[m]);   // else zeros
      if (t % 32 == 0) red[g] = s[m];
    }
  }
  __syncthreads();
  if (t == 0) {
    for (int o = kBandRed / 64; o; o >>= 1)
      for (int j = 0; j < o; ++j) red[j] += red[j + o];
    st->eband = red[0] * b.s2;
    if (reset_umax) st->umax[0] = st->umax[1] = st->umax[2] = 0.0;
  }
}

// Pruning of the 2/3-rule zeros.  On an axis of length n the dealiasing mask
// (rhs.f90:74-88) keeps index i when |k_i| < (n/2)(2/3) alpha, i.e. i < a, the
// Nyquist index n/2 (whose wavenumber is 0) and, on full axes, i > n - a.  A
// state that vanishes outside the kept set keeps doing so under the stepper,
// so the transforms may skip loading those zeros, skip outputs the mask
// discards, and skip whole tiles; results are bit-identical.  a = 0: no pruning.
struct AxisKeep {
  int a, n, full;
  __host__ __device__ __forceinline__ bool keep(int i) const {
    return a == 0 || i < a || i == (n >> 1) || (full && i > n - a);
  }
  // kept indices of a full axis in order: [0, a), n/2, (n - a, n)
  __host__ __device__ __forceinline__ int count() const { return a == 0 ? n : 2 * a; }
  __host__ __device__ __forceinline__ int map(int o) const {
    return (a == 0 || o < a) ? o : (o == a ? (n >> 1) : n - 2 * a + o);
  }
};

// Tile width (kx columns) of the strided passes: 128 B per row segment.
template <typename T> struct TileCols;
template <> struct TileCols<double> { static constexpr int v = 8; };
template <> struct TileCols<float> { static constexpr int v = 16; };

template <typename T> struct StridedJob {
  using C = typename CT<T>::type;
  const C *in1;
  const C *in2;
  C *out;
  double a1, b1, a2, b2;   // multiplier a + i b k
  int ks1, ks2;            // k: 0 kx of the column, 1 the row index's, 2 the tile's other-axis index's
};

template <typename T> struct StridedArgs {
  using C = typename CT<T>::type;
  StridedJob<T> job[9];
  const C *tw;             // exp(-2 pi i j / N), j < N
  int njobs;
  int ncols;               // nxh
  int nx;
  int pad0;
  long long rowstride;     // elements between consecutive rows of the axis
  long long otherstride;   // elements between consecutive tiles of the other axis
  double alpha_row, alpha_x;
  int n_other;             // length of the other axis (for ks = 2)
  int nbatch;              // boxes (blockIdx.y), each job pointer advanced by bstride per box
  double alpha_other;
  long long bstride;
  // pruning (all zero when off, so zero-initialised arguments run the full
  // grid): kept kx columns, kept other-axis indices (the tile grid covers only
  // these), kept input rows (others read as 0) and kept output rows (others
  // not stored).  Column tiles: all ceil(ncols / width) when ntx_lo = 0, else
  // [0, ntx_lo) followed by tile nyq_tile when nyq_tile > 0; nyq_tile < 0
  // places the Nyquist column in the free slot kx = kcol.a of the last low
  // tile (see strided_col).
  AxisKeep kcol, koth, krin, krout;
  int ntx_lo, nyq_tile;
  // strides of the output when its row pitch differs from the input's (the
  // padded workspace fields of a right-hand side); 0: the input's
  long long rowstride_o, otherstride_o, bstride_o;
  // which sides are padded workspace fields (1: input, 2: output), whose rows
  // of nslot columns start on 128-byte boundaries; with column pruning the
  // workspace is compact: slot kcol.a holds the Nyquist column (compact = 1)
  int ws, compact, nslot, pad;
  BandArgs band;   // band.n: one more block per box (the last) computes the band energy
  CflArgs cfl;     // cfl.on: likewise (forward passes), the CFL update of the box
  StepState *st;   // step states, with cfl.on
};

// Output strides of a strided launch (the input's where unset).
template <typename T> __host__ __device__ __forceinline__ long long out_rowstride(const StridedArgs<T> &a) {
  return a.rowstride_o ? a.rowstride_o : a.rowstride;
}
template <typename T> __host__ __device__ __forceinline__ long long out_otherstride(const StridedArgs<T> &a) {
  return a.otherstride_o ? a.otherstride_o : a.otherstride;
}
template <typename T> __host__ __device__ __forceinline__ long long out_bstride(const StridedArgs<T> &a) {
  return a.bstride_o ? a.bstride_o : a.bstride;
}

// Column tiles of the grid of a strided launch with tile width tcw.
template <typename T>
__host__ __device__ __forceinline__ int strided_ntx(const StridedArgs<T> &a, int tcw) {
  return a.ntx_lo ? a.ntx_lo + (a.nyq_tile > 0 ? 1 : 0) : (a.ncols + tcw - 1) / tcw;
}

// Half-axis index held by tile column kx0 + c: the identity, except in the
// merged layout (nyq_tile < 0), where the first column past the cut holds the
// Nyquist column kcol.n / 2.
template <typename T>
__host__ __device__ __forceinline__ int strided_col(const StridedArgs<T> &a, int kx) {
  return (a.nyq_tile < 0 && kx == a.kcol.a) ? (a.kcol.n >> 1) : kx;
}

// Shape of a strided block: 8 threads across the columns, each with one 16-byte
// element per row (a complex double, or two neighbouring single-precision
// columns), so a row segment of a tile is 128 bytes; P threads along the rows.
template <typename T, int N> struct StridedShape {
  using PL = VPlan<N>;
  static constexpr int W = 8;
  static constexpr int NT = W * PL::P;
  static constexpr size_t tile = PL::NST > 1 ? (size_t)N * W * 16 : 0;
  static constexpr size_t smem(bool inv) {   // tile, twiddles and (inverse) row multipliers
    const size_t n = tile + (size_t)vtw_size<PL>() * 16 + (inv ? 2 * N * sizeof(T) : 0);
    return n < kBandRed / 32 * sizeof(double) ? kBandRed / 32 * sizeof(double) : n;   // the band block's sums
  }
  // Resident CTAs asked of the register allocator: 16 warps per SM where a
  // thread holds 16 values (128 registers), 20 at 12 (96), 24 at 8 (80).  The
  // 256-row pass with 8 values, three stages and 32 warps measured the same
  // (57.7 against 56.7 us for pass D: the loads in flight per SM are equal);
  // at 512, whose 8-value plan spills at the 64 registers of 32 warps, 16
  // values take passes A / D / E1 from 553 / 355 / 261 to 516 / 326 / 236 us
  // (512^3 FP32); at 96, 24 values in two stages take pass B from 224 to 252.
  static constexpr int warps = PL::E >= 16 ? 16 : PL::E == 12 ? 20 : 24;
  static constexpr int wcta = round32(NT) / 32;
  static constexpr int minb = warps / wcta < 1 ? 1 : warps / wcta;
};

// Column origin and other-axis index of tile t of the (possibly pruned) grid.
template <typename T>
__device__ __forceinline__ void strided_tile(const StridedArgs<T> &a, int tile, int tcw, int &kx0, int &other) {
  const int ntk = strided_ntx(a, tcw);
  const int o = tile / ntk, kt = tile - o * ntk;
  kx0 = (a.ntx_lo == 0 || kt < a.ntx_lo ? kt : a.nyq_tile) * tcw;
  other = a.koth.map(o);
}

// Tile addressing: rows of 8 elements of 16 bytes (128 bytes), so the eight
// lanes of a quarter warp, one row's columns, cover all banks once.
struct AddrRows8 {
  __device__ static __forceinline__ int at(int row, int col) { return row * 8 + col; }
};

// One 16-byte element from / to memory (zero where !on): an aligned 16-byte
// word, or (single precision) two columns one by one.  The loads are volatile,
// so that a thread's rows are all requested before the first is used.
template <typename C> struct StridedIO;
template <> struct StridedIO<double2> {
  using Raw = VC<double>;
  __device__ static __forceinline__ Raw load(const double2 *p, bool on) {
    Raw x{0.0, 0.0};
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\t@q ld.global.v2.f64 {%0, %1}, [%2];\n\t}"
                 : "+d"(x.re), "+d"(x.im)
                 : "l"(p), "r"((unsigned)on));
    return x;
  }
  __device__ static __forceinline__ void store(double2 *p, Raw v) { *p = make_double2(v.re, v.im); }
  // x (a + i b)
  __device__ static __forceinline__ Raw mul(Raw x, double a, double b, double) {
    return Raw{x.re * a - x.im * b, x.im * a + x.re * b};
  }
  __device__ static __forceinline__ Raw add(Raw x, Raw y) { return Raw{x.re + y.re, x.im + y.im}; }
};
template <> struct StridedIO<float2> {
  using Raw = Raw2;
  __device__ static __forceinline__ Raw load(const float2 *p, bool on) {
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %5, 0;\n\t@q ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
        : "+f"(x.x), "+f"(x.y), "+f"(x.z), "+f"(x.w)
        : "l"(p), "r"((unsigned)on));
    return Raw{x};
  }
  __device__ static __forceinline__ Raw load2(const float2 *p0, const float2 *p1, bool v0, bool v1) {
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\t@q ld.global.v2.f32 {%0, %1}, [%2];\n\t}"
                 : "+f"(x.x), "+f"(x.y)
                 : "l"(p0), "r"((unsigned)v0));
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\t@q ld.global.v2.f32 {%0, %1}, [%2];\n\t}"
                 : "+f"(x.z), "+f"(x.w)
                 : "l"(p1), "r"((unsigned)v1));
    return Raw{x};
  }
  __device__ static __forceinline__ void store(float2 *p, Raw v) { *reinterpret_cast<float4 *>(p) = v.q; }
  __device__ static __forceinline__ void store2(float2 *p0, float2 *p1, Raw v, bool v0, bool v1) {
    if (v0) *p0 = make_float2(v.q.x, v.q.y);
    if (v1) *p1 = make_float2(v.q.z, v.q.w);
  }
  // x (a + i b0), y (a + i b1) of the two columns
  __device__ static __forceinline__ Raw mul(Raw x, float a, float b0, float b1) {
    return Raw{make_float4(x.q.x * a - x.q.y * b0, x.q.y * a + x.q.x * b0, x.q.z * a - x.q.w * b1, x.q.w * a + x.q.z * b1)};
  }
  __device__ static __forceinline__ Raw add(Raw x, Raw y) {
    return Raw{make_float4(x.q.x + y.q.x, x.q.y + y.q.y, x.q.z + y.q.z, x.q.w + y.q.w)};
  }
};

// Bit q is set when row p + P q of the axis is kept (q < E).
template <class PL> __device__ __forceinline__ unsigned keep_mask(const AxisKeep &k, int p) {
  constexpr int P = PL::P, E = PL::E, N = PL::N;
  constexpr unsigned all = E == 32 ? 0xffffffffu : (1u << E) - 1u;
  if (k.a == 0) return all;
  const int lo = (k.a - p + P - 1) / P;                    // rows below a: q < lo (a >= 1, p < P)
  unsigned m = lo >= E ? all : (1u << lo) - 1u;
  if (k.full) {
    const int t = N - k.a - p;                             // rows above N - a: P q > t
    const int hi = t < 0 ? 0 : t / P + 1;
    if (hi < E) m |= all & ~((1u << hi) - 1u);
  }
  if ((N / 2 - p) % P == 0 && N / 2 >= p) m |= 1u << ((N / 2 - p) / P);   // the Nyquist row
  return m;
}

// Layouts of a strided pass's two sides.  A workspace side is read and
// written in whole 16-byte elements over its nslot columns, padding included,
// so that every 32-byte sector is written whole (a sector written in part
// costs a read of it when it leaves L2: 57 MB of 219 in pass B at 256^3 FP32);
// a state side column by column, kept columns only.
enum StridedMode : int {
  ST_ANY = 0,      // columns of any layout, one by one
  ST_TO_WS = 1,    // state -> workspace
  ST_WS = 2,       // workspace -> workspace
  ST_FROM_WS = 3,  // workspace -> state
};

// One strided pass.  A thread holds E rows of one 16-byte element (VPlan), so
// a row segment of 8 threads is 128 bytes, loads, stores and exchanges are
// 16-byte instructions, and in single precision the transform runs on packed
// pairs (fftv.cuh).  Row pruning and the jobs' multipliers concern the inputs
// of the inverse passes and the outputs of the forward ones only.  With its
// instructions halved the pass is bound by DRAM and its latency: without the
// FFT the same loads and stores take 67 / 125 / 56 / 35 us (A, B, D, E1,
// 256^3 FP32, padded rows with the kept columns first) and the pass takes
// 76 / 135 / 57 / 39; compact rows, written in whole sectors, bring it to
// 61 / 109 / 45 / 31 (one 8-byte column per thread: 77 / 148 / 63 / 43), FP64
// from 111 / 248 / 94 / 67 to 99 / 191 / 74 / 54.
template <typename T, int N, bool INV, int MODE>
__global__ void __launch_bounds__(StridedShape<T, N>::NT, StridedShape<T, N>::minb)
    k_strided(const __grid_constant__ StridedArgs<T> a) {
  using C = typename CT<T>::type;
  using SH = StridedShape<T, N>;
  using PL = typename SH::PL;
  using EN = VEnds<PL>;
  using IO = StridedIO<C>;
  using Raw = typename IO::Raw;
  using V = VC<typename VecOf<T>::R>;
  constexpr int E = PL::E, P = PL::P, CPT = VecOf<T>::cols;
  constexpr bool PAIR = CPT == 2;
  constexpr bool WSI = MODE == ST_WS || MODE == ST_FROM_WS, WSO = MODE == ST_WS || MODE == ST_TO_WS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V *s = reinterpret_cast<V *>(smem_raw);
  V *twt = reinterpret_cast<V *>(smem_raw + SH::tile);
  T *bks = reinterpret_cast<T *>(smem_raw + SH::tile + (size_t)vtw_size<PL>() * 16);
  pdl_launch();
  if constexpr (INV && MODE == ST_TO_WS && SH::NT >= 32) {
    if (a.band.n && blockIdx.x == gridDim.x - 1) {
      pdl_wait();
      eband_block<C, SH::NT>(a.band, a.nx, blockIdx.y, false, reinterpret_cast<double *>(smem_raw));
      return;
    }
  }
  if constexpr (!INV && MODE == ST_WS) {
    if (a.cfl.on && blockIdx.x == gridDim.x - 1) {
      pdl_wait();
      if (threadIdx.x == 0) cfl_update(a.cfl, a.st + blockIdx.y, blockIdx.y, gridDim.y);
      return;
    }
  }
  const int job = blockIdx.x % a.njobs;
  const int tile = blockIdx.x / a.njobs;
  int kx0, other;
  strided_tile(a, tile, TileCols<T>::v, kx0, other);
  const StridedJob<T> &jb = a.job[job];
  const int col = threadIdx.x % SH::W, p = threadIdx.x / SH::W;
  // the thread's slot(s) and the modes they hold; v0, v1: kept columns
  const int s0 = kx0 + CPT * col;
  const int c0 = strided_col(a, s0), c1 = PAIR ? strided_col(a, s0 + 1) : c0;
  const bool v0 = c0 < a.ncols && a.kcol.keep(c0);
  const bool v1 = PAIR && c1 < a.ncols && a.kcol.keep(c1);
  const bool vs = s0 < a.nslot;
  const long long base = (long long)other * a.otherstride + (long long)blockIdx.y * a.bstride + (long long)p * a.rowstride +
                         (WSI ? s0 : c0);
  const long long step = (long long)P * a.rowstride;
  const unsigned rin = INV ? keep_mask<PL>(a.krin, p) : 0u;
  // rows p + P q, q in [Q0, Q0 + QN), of one input into x[0 .. QN)
  auto load = [&](const C *in, Raw *x, int Q0, int QN) {
    const C *q0 = in + base + Q0 * step;
#pragma unroll
    for (int q = Q0; q < Q0 + QN; ++q, q0 += step) {
      const bool k = INV ? (rin >> q & 1) : true;
      if constexpr (WSI || !PAIR) x[q - Q0] = IO::load(q0, (WSI ? vs : v0) && k);
      else x[q - Q0] = IO::load2(q0, q0 + (c1 - c0), v0 && k, v1 && k);
    }
  };
  // twiddles: read before the wait, stored once the rows are on their way
  constexpr int NTW = (vtw_size<PL>() + SH::NT - 1) / SH::NT;
  C tws[NTW > 0 ? NTW : 1];
  if constexpr (NTW > 0) {
#pragma unroll
    for (int i = 0; i < NTW; ++i)
      if ((int)threadIdx.x + i * SH::NT < vtw_size<PL>()) tws[i] = vtw_entry<PL>(a.tw, threadIdx.x + i * SH::NT);
  }
  pdl_wait();
  Raw v[E];   // row p + P q in v[in_i(q)]
  {
    Raw x[E];
    load(jb.in1, x, 0, E);
#pragma unroll
    for (int q = 0; q < E; ++q) v[EN::in_i(q)] = x[q];
  }
  // second inputs: a part of the rows at a time, so that their loads in flight
  // fit beside the first input's values; the first part right away
  constexpr int QN = E <= 8 ? E : E / 2;
  const C *const in2p = INV ? jb.in2 : nullptr;
  Raw w[INV ? QN : 1];
  if (INV && in2p) load(in2p, w, 0, QN);
  // with the rows on their way: the twiddle tables (read after the exchange's
  // barrier) and the job's row multipliers T(b k_row(n)) (ks == 1)
  if constexpr (NTW > 0) {
#pragma unroll
    for (int i = 0; i < NTW; ++i)
      if ((int)threadIdx.x + i * SH::NT < vtw_size<PL>()) twt[threadIdx.x + i * SH::NT] = VtwOf<V>::of(tws[i]);
  }
  if constexpr (INV) {
    const bool mult1 = !(jb.a1 == 1.0 && jb.b1 == 0.0);
    const bool rows1 = mult1 && jb.ks1 == 1, rows2 = in2p && jb.ks2 == 1;
    if (rows1 || rows2) {
      for (int n = threadIdx.x; n < N; n += SH::NT) {
        const double k = k_full(n, N, a.alpha_row);
        bks[n] = T(jb.b1 * k);
        bks[N + n] = T(jb.b2 * k);
      }
      __syncthreads();
    }
    // the factor b k of a column (ks 0) or of the tile's other-axis index (ks 2)
    auto colmul = [&](int ks, double b, int c) {
      return T(b * (ks == 2 ? (a.n_other ? k_full(other, a.n_other, a.alpha_other) : 0.0) : k_half(c, a.nx, a.alpha_x)));
    };
    if (mult1) {   // v (a + i b k)
      const T aa = T(jb.a1), m0 = colmul(jb.ks1, jb.b1, c0), m1 = colmul(jb.ks1, jb.b1, c1);
#pragma unroll
      for (int q = 0; q < E; ++q) {
        const T br = rows1 ? bks[p + P * q] : m0;
        v[EN::in_i(q)] = IO::mul(v[EN::in_i(q)], aa, br, rows1 ? br : m1);
      }
    }
    if (in2p) {
      const T aa = T(jb.a2), m0 = colmul(jb.ks2, jb.b2, c0), m1 = colmul(jb.ks2, jb.b2, c1);
#pragma unroll
      for (int h = 0; h < E / QN; ++h) {
        if (h) load(in2p, w, h * QN, QN);
#pragma unroll
        for (int i = 0; i < QN; ++i) {
          const T br = rows2 ? bks[N + p + P * (h * QN + i)] : m0;
          Raw &x = v[EN::in_i(h * QN + i)];
          x = IO::add(x, IO::mul(w[i], aa, br, rows2 ? br : m1));
        }
      }
    }
  }
  Raw x[E];   // row p + P q in x[out_i(q)]
  vfft<PL, INV, AddrRows8>(v, x, s, col, p, twt, []() { __syncthreads(); });
  const unsigned rout = INV ? 0u : keep_mask<PL>(a.krout, p);
  const long long rso = out_rowstride(a), so = (long long)P * rso;
  C *o0 = jb.out + (long long)other * out_otherstride(a) + (long long)blockIdx.y * out_bstride(a) + (long long)p * rso +
          (WSO ? s0 : c0);
#pragma unroll
  for (int q = 0; q < E; ++q, o0 += so) {
    const bool k = INV ? true : (rout >> q & 1);
    if constexpr (WSO || !PAIR) {
      if ((WSO ? vs : v0) && k) IO::store(o0, x[EN::out_i(q)]);
    } else {
      IO::store2(o0, o0 + (c1 - c0), x[EN::out_i(q)], v0 && k, v1 && k);
    }
  }
}

// ------------------------------------------------------------------ x lines
template <typename T> struct XlineNLArgs {
  using C = typename CT<T>::type;
  const C *U, *V, *W, *OX, *OY, *OZ;  // (kx, y, z) space, rows of nxh; omega scaled by 1/N^3
  C *NX, *NY, *NZ;                     // forward x transforms of (omega x u) * s
  const C *tw;
  StepState *st;                       // per-box step state: umax[3] gets max |u_i| (true scale)
  int nlines, nxh;
  int lines_per_box;                   // ny * nz, of the planes of this launch
  int box_lines;                       // ny * nz of the whole box
  int kxa;                             // pruning: only kx < kxa and kx = N/2 are read and written (0: all)
  int pin, pout;                       // row pitch (complex elements) of the inputs / outputs; 0: nxh
  int npad;                            // compact rows: slots after nyq that complete its 32-byte sector (written as 0)
  int nyq;                             // slot of the Nyquist column in a row (kxa in compact workspace rows); 0: N/2
  double s;                            // scalemodes
};

// kept half-axis index under the x-line pruning rule
__device__ __forceinline__ bool xkeep(int kxa, int k, int n) { return kxa == 0 || k < kxa || k == (n >> 1); }

// Slot of half-axis index k in a row whose Nyquist column lies at nyq (0: N/2).
__device__ __forceinline__ int xslot(int nyq, int k, int n) { return nyq && k == (n >> 1) ? nyq : k; }

// Lines per CTA of the block x kernel (even; 3B columns in shared memory).
template <typename T, int N> struct XlineB {
  static constexpr int v = 2;
};

// Full-length sequence value at row n of Z = X1 + i X2, where X1, X2 are the
// half spectra (nxh values) of two real lines: rows above N/2 are the
// Hermitian mirror; the imaginary parts of the kx = 0 and Nyquist bins are
// dropped, as a C2R does.
template <typename C, int N>
__device__ __forceinline__ C pack_pair(int n, C X1, C X2) {
  if (n == 0 || n == N / 2) return mkc<C>(X1.x, X2.x);
  if (n < N / 2) return mkc<C>(X1.x - X2.y, X1.y + X2.x);
  return mkc<C>(X1.x + X2.y, X2.x - X1.y);   // conj(X1) + i conj(X2) at N - n
}

// The block x kernel: lines of 1024 points (and, by choice, double-precision
// lines of 512).  Resident CTAs to ask the register allocator for: 3 for
// blocks of up to 256 threads; 2 for the 384-thread FP32 blocks of N = 1024
// (80 registers instead of 123, two CTAs per SM instead of one).
template <typename T, int N> struct XlineMinCtas {
  static constexpr int NT = round32(3 * XlineB<T, N>::v * (N / FftPlan<N>::E));
  static constexpr int v = (sizeof(T) == 4 && N >= 1024) ? 2 : min_ctas(NT, 3);
};

template <typename T, int N>
__global__ void __launch_bounds__(round32(3 * XlineB<T, N>::v *(N / FftPlan<N>::E)), XlineMinCtas<T, N>::v)
    k_xline_nl(const __grid_constant__ XlineNLArgs<T> a) {
  using C = typename CT<T>::type;
  using EN = FftEnds<N>;
  constexpr int B = XlineB<T, N>::v;
  constexpr int H = N / 2 + 1;
  constexpr int NCOL = 3 * B;
  constexpr int LD = NCOL + 1;         // odd stride: rows fall in distinct bank groups
  constexpr int E = EN::E;
  constexpr int P = N / E;
  constexpr int NF = NCOL * P;         // FFT threads, position index fastest
  constexpr int NQ = NCOL / 2;         // forward sequences
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *s = reinterpret_cast<C *>(smem_raw);
  __shared__ double red[3 * 32];
  const int NT = blockDim.x;
  const int line0 = blockIdx.x * B;
  const T sc = T(a.s);
  // Inverse transforms.  Column 6j+q of line pair (a = 2j, b = 2j+1) holds
  // (u_a,v_a) (u_b,v_b) (w_a,w_b) (ox_a,oy_a) (ox_b,oy_b) (oz_a,oz_b): each
  // pair is two quantities of the same kind and scale.
  {
    const bool act = threadIdx.x < NF;
    const int p = threadIdx.x % P, col = threadIdx.x / P;
    const int j = col / 6, q = col % 6;
    const int la = line0 + 2 * j, lb = la + 1;
    const C *f1, *f2;
    int l1, l2;
    switch (q) {
      case 0: f1 = a.U; l1 = la; f2 = a.V; l2 = la; break;
      case 1: f1 = a.U; l1 = lb; f2 = a.V; l2 = lb; break;
      case 2: f1 = a.W; l1 = la; f2 = a.W; l2 = lb; break;
      case 3: f1 = a.OX; l1 = la; f2 = a.OY; l2 = la; break;
      case 4: f1 = a.OX; l1 = lb; f2 = a.OY; l2 = lb; break;
      default: f1 = a.OZ; l1 = la; f2 = a.OZ; l2 = lb; break;
    }
    const bool v1 = act && l1 < a.nlines, v2 = act && l2 < a.nlines;
    const long long pin = a.pin ? a.pin : a.nxh;
    const C *r1 = f1 + (long long)l1 * pin, *r2 = f2 + (long long)l2 * pin;
    C v[E];
#pragma unroll
    for (int i = 0; i < E; ++i) {
      const int n = EN::in_row(p, i);
      const int kk = n <= N / 2 ? n : N - n;
      const bool kp = xkeep(a.kxa, kk, N);
      const int sl = xslot(a.nyq, kk, N);
      const C X1 = (v1 && kp) ? r1[sl] : mkc<C>(0, 0);
      const C X2 = (v2 && kp) ? r2[sl] : mkc<C>(0, 0);
      v[i] = pack_pair<C, N>(n, X1, X2);
    }
    fft_regs<C, N, true>(v, s, LD, col, p, act, a.tw);
    if (act) {
#pragma unroll
      for (int i = 0; i < E; ++i) s[EN::out_row(p, i) * LD + col] = v[i];
    }
  }
  __syncthreads();
  // (omega x u) * s at every point; written back as (px_a,py_a) (pz_a,pz_b)
  // (px_b,py_b) in columns 6j, 6j+1, 6j+2; the CFL maxima are taken in T
  // (exact) and widened for the block reduction
  T m0 = 0, m1 = 0, m2 = 0;
  for (int it = threadIdx.x; it < N * (B / 2); it += NT) {
    const int n = it % N, j = it / N;
    C *r = s + n * LD + 6 * j;
    const C c0 = r[0], c1 = r[1], c2 = r[2], c3 = r[3], c4 = r[4], c5 = r[5];
    const T uu[2] = {c0.x, c1.x}, vv[2] = {c0.y, c1.y}, ww[2] = {c2.x, c2.y};
    const T ox[2] = {c3.x, c4.x}, oy[2] = {c3.y, c4.y}, oz[2] = {c5.x, c5.y};
    T px[2], py[2], pz[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      px[h] = (oy[h] * ww[h] - oz[h] * vv[h]) * sc;
      py[h] = (oz[h] * uu[h] - ox[h] * ww[h]) * sc;
      pz[h] = (ox[h] * vv[h] - oy[h] * uu[h]) * sc;
      m0 = fmax(m0, fabs(uu[h]));
      m1 = fmax(m1, fabs(vv[h]));
      m2 = fmax(m2, fabs(ww[h]));
    }
    r[0] = mkc<C>(px[0], py[0]);
    r[1] = mkc<C>(pz[0], pz[1]);
    r[2] = mkc<C>(px[1], py[1]);
  }
  __syncthreads();
  // forward transforms of the NQ product sequences
  {
    const bool act = threadIdx.x < NQ * P;
    const int p = threadIdx.x % P, q = threadIdx.x / P;
    const int col = 6 * (q / 3) + q % 3;
    C v[E];
    if (act) {
#pragma unroll
      for (int i = 0; i < E; ++i) v[i] = s[EN::in_row(p, i) * LD + col];
    }
    __syncthreads();
    fft_regs<C, N, false>(v, s, LD, col, p, act, a.tw);
    if (act) {
#pragma unroll
      for (int i = 0; i < E; ++i) s[EN::out_row(p, i) * LD + col] = v[i];
    }
  }
  __syncthreads();
  // unpack two real transforms per sequence and store
  const long long pout = a.pout ? a.pout : a.nxh;
  for (int it = threadIdx.x; it < NQ * H; it += NT) {
    const int k = it % H, q = it / H;
    const int j = q / 3, c = q % 3;
    const int col = 6 * j + c;
    const C zk = s[k * LD + col], zn = s[((N - k) % N) * LD + col];
    const C X1 = mkc<C>(T(0.5) * (zk.x + zn.x), T(0.5) * (zk.y - zn.y));
    const C X2 = mkc<C>(T(0.5) * (zk.y + zn.y), T(-0.5) * (zk.x - zn.x));
    const int la = line0 + 2 * j, lb = la + 1;
    if (!xkeep(a.kxa, k, N)) continue;
    const int sl = xslot(a.nyq, k, N);
    if (c == 0) {
      if (la < a.nlines) {
        a.NX[(long long)la * pout + sl] = X1;
        a.NY[(long long)la * pout + sl] = X2;
      }
    } else if (c == 1) {
      if (la < a.nlines) a.NZ[(long long)la * pout + sl] = X1;
      if (lb < a.nlines) a.NZ[(long long)lb * pout + sl] = X2;
    } else {
      if (lb < a.nlines) {
        a.NX[(long long)lb * pout + sl] = X1;
        a.NY[(long long)lb * pout + sl] = X2;
      }
    }
  }
  // CFL reduction
  m0 = warp_max(m0);
  m1 = warp_max(m1);
  m2 = warp_max(m2);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    red[wid] = (double)m0;
    red[32 + wid] = (double)m1;
    red[64 + wid] = (double)m2;
  }
  __syncthreads();
  if (wid == 0) {
    const int nw = NT >> 5;
    double x0 = lane < nw ? red[lane] : 0, x1 = lane < nw ? red[32 + lane] : 0,
           x2 = lane < nw ? red[64 + lane] : 0;
    x0 = warp_max(x0);
    x1 = warp_max(x1);
    x2 = warp_max(x2);
    if (lane == 0 && a.st) {
      // B divides ny*nz, so every line of the CTA belongs to one box
      double *um = a.st[line0 / a.lines_per_box].umax;
      atomic_max_nonneg(um + 0, x0 * a.s);
      atomic_max_nonneg(um + 1, x1 * a.s);
      atomic_max_nonneg(um + 2, x2 * a.s);
    }
  }
}

// Warp-granular variant of the fused x pass for double-precision lines of 512
// points (whose fields do not fit a warp's registers): each warp owns one
// line pair from its loads to its stores and synchronises only with
// __syncwarp, so the SM overlaps one warp's memory phases with another's
// transforms (the block-wide barriers of k_xline_nl serialise them).  Columns
// of a warp's tile are the six sequences of k_xline_nl, stored column-major
// with the row / R0 skew; a sequence runs the three-stage plan on all 32
// threads.
template <typename T, int N> struct XlineWarp {
  static constexpr bool on = N == 512 && sizeof(T) == 8;
  static constexpr int wpb = 1;
  using Plan = WarpPlan<512>;
};

// Second half of the warp-granular fused x pass for one line pair (la, lb):
// the inverse transforms are in the warp's tile s (column-major, skewed);
// (omega x u) * s, the three forward transforms, the unpacking into the
// output half lines and the CFL maxima of the pair.
template <typename T, int N>
__device__ __forceinline__ void xline_w_tail(typename CT<T>::type *s, const XlineNLArgs<T> &a, long long la,
                                             long long lb, int lane, long long pout) {
  using C = typename CT<T>::type;
  using PL = typename XlineWarp<T, N>::Plan;
  using EN = FftEndsP<PL>;
  using AD = AddrSkew<PL::R[0]>;
  constexpr int E = PL::E;
  constexpr int H = N / 2 + 1;
  constexpr int LDC = N + N / PL::R[0];
  const T sc = T(a.s);
  __syncwarp();
  // (omega x u) * s, written back as (px_a,py_a) (pz_a,pz_b) (px_b,py_b) in
  // columns 0..2; the CFL maxima are taken in T (exact) and widened at the end
  T m0 = 0, m1 = 0, m2 = 0;
#pragma unroll 4
  for (int n = lane; n < N; n += 32) {
    const C c0 = s[AD::at(n, 0, LDC)], c1 = s[AD::at(n, 1, LDC)], c2 = s[AD::at(n, 2, LDC)];
    const C c3 = s[AD::at(n, 3, LDC)], c4 = s[AD::at(n, 4, LDC)], c5 = s[AD::at(n, 5, LDC)];
    const T uu[2] = {c0.x, c1.x}, vv[2] = {c0.y, c1.y}, ww[2] = {c2.x, c2.y};
    const T ox[2] = {c3.x, c4.x}, oy[2] = {c3.y, c4.y}, oz[2] = {c5.x, c5.y};
    T px[2], py[2], pz[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      px[h] = (oy[h] * ww[h] - oz[h] * vv[h]) * sc;
      py[h] = (oz[h] * uu[h] - ox[h] * ww[h]) * sc;
      pz[h] = (ox[h] * vv[h] - oy[h] * uu[h]) * sc;
      m0 = fmax(m0, fabs(uu[h]));
      m1 = fmax(m1, fabs(vv[h]));
      m2 = fmax(m2, fabs(ww[h]));
    }
    s[AD::at(n, 0, LDC)] = mkc<C>(px[0], py[0]);
    s[AD::at(n, 1, LDC)] = mkc<C>(pz[0], pz[1]);
    s[AD::at(n, 2, LDC)] = mkc<C>(px[1], py[1]);
  }
  __syncwarp();
  // forward transforms of the three product sequences
#pragma unroll 1
  for (int q = 0; q < 3; ++q) {
    C v[E];
#pragma unroll
    for (int i = 0; i < E; ++i) v[i] = s[AD::at(EN::in_row(lane, i), q, LDC)];
    __syncwarp();
    fft_regs_p<C, PL, false, true, AD>(v, s, LDC, q, lane, true, a.tw);
#pragma unroll
    for (int i = 0; i < E; ++i) s[AD::at(EN::out_row(lane, i), q, LDC)] = v[i];
  }
  __syncwarp();
  // unpack two real transforms per sequence and store
  for (int k = lane; k < H; k += 32) {
    if (!xkeep(a.kxa, k, N)) continue;
    const int sl = xslot(a.nyq, k, N);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const C zk = s[AD::at(k, q, LDC)], zn = s[AD::at((N - k) % N, q, LDC)];
      const C X1 = mkc<C>(T(0.5) * (zk.x + zn.x), T(0.5) * (zk.y - zn.y));
      const C X2 = mkc<C>(T(0.5) * (zk.y + zn.y), T(-0.5) * (zk.x - zn.x));
      if (q == 0) {
        a.NX[la * pout + sl] = X1;
        a.NY[la * pout + sl] = X2;
      } else if (q == 1) {
        a.NZ[la * pout + sl] = X1;
        a.NZ[lb * pout + sl] = X2;
      } else {
        a.NX[lb * pout + sl] = X1;
        a.NY[lb * pout + sl] = X2;
      }
    }
  }
  // CFL maxima of this line pair (both lines lie in one box: ny*nz is even)
  m0 = warp_max(m0);
  m1 = warp_max(m1);
  m2 = warp_max(m2);
  if (lane == 0 && a.st) {
    double *um = a.st[la / a.lines_per_box].umax;
    atomic_max_nonneg(um + 0, (double)m0 * a.s);
    atomic_max_nonneg(um + 1, (double)m1 * a.s);
    atomic_max_nonneg(um + 2, (double)m2 * a.s);
  }
}

template <typename T, int N>
__global__ void __launch_bounds__(32 * XlineWarp<T, N>::wpb)
    k_xline_nl_w(const __grid_constant__ XlineNLArgs<T> a) {
  using C = typename CT<T>::type;
  using PL = typename XlineWarp<T, N>::Plan;
  using EN = FftEndsP<PL>;
  using AD = AddrSkew<PL::R[0]>;
  constexpr int E = PL::E;
  constexpr int P = N / E;                // threads per sequence
  static_assert(P == 32, "a sequence on all lanes");
  constexpr int LDC = N + N / PL::R[0];   // column length with the skew
  constexpr int WPB = XlineWarp<T, N>::wpb;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  C *s = reinterpret_cast<C *>(smem_raw) + (size_t)warp * 6 * LDC;
  const long long la = 2 * ((long long)blockIdx.x * WPB + warp), lb = la + 1;
  if (la >= a.nlines) return;
  const C *f1s[6] = {a.U, a.U, a.W, a.OX, a.OX, a.OZ};
  const C *f2s[6] = {a.V, a.V, a.W, a.OY, a.OY, a.OZ};
  const long long l1s[6] = {la, lb, la, la, lb, la};
  const long long l2s[6] = {la, lb, lb, la, lb, lb};
  const int p = lane;   // position in the sequence
  const long long pin = a.pin ? a.pin : a.nxh, pout = a.pout ? a.pout : a.nxh;
  // inverse transforms: round r transforms sequence r; the loads of the next
  // round are issued before this round's transform.  A lane loads
  // only its rows n = p + P i <= N/2 (i < E/2, and i = E/2 at p = 0); row
  // N - n of the Hermitian mirror is row n' = (P - p) + P (E - 1 - i) of lane
  // P - p (lane p = 0: its own row P (E - i)), taken by a shuffle, so every
  // half-line element is read from global memory once.
  static_assert(PL::R[0] == E, "first-stage rows n = p + P i");
  C x1[E], x2[E];
  auto load = [&](const C *g1, const C *g2) {
#pragma unroll
    for (int i = 0; i <= E / 2; ++i) {
      const int n = p + P * i;   // <= N / 2 for i < E / 2 and for p = 0
      const bool kp = (i < E / 2 || p == 0) && xkeep(a.kxa, n, N);
      const int sl = xslot(a.nyq, n, N);
      x1[i] = kp ? g1[sl] : mkc<C>(0, 0);
      x2[i] = kp ? g2[sl] : mkc<C>(0, 0);
    }
  };
  const int mirror = (lane & ~(P - 1)) | ((P - p) & (P - 1));   // lane of the mirror rows
  auto mirror_fill = [&]() {
#pragma unroll
    for (int i = E / 2; i < E; ++i) {
      const int j = E - 1 - i;
      C m1 = mkc<C>(__shfl_sync(0xffffffffu, x1[j].x, mirror), __shfl_sync(0xffffffffu, x1[j].y, mirror));
      C m2 = mkc<C>(__shfl_sync(0xffffffffu, x2[j].x, mirror), __shfl_sync(0xffffffffu, x2[j].y, mirror));
      if (p == 0) {   // rows 0 and N/2 are its own loads; N - P i = P (E - i)
        m1 = i == E / 2 ? x1[i] : x1[E - i];
        m2 = i == E / 2 ? x2[i] : x2[E - i];
      }
      x1[i] = m1;
      x2[i] = m2;
    }
  };
  load(f1s[0] + l1s[0] * pin, f2s[0] + l2s[0] * pin);
#pragma unroll 1
  for (int q = 0; q < 6; ++q) {
    C v[E];
    mirror_fill();
#pragma unroll
    for (int i = 0; i < E; ++i) v[i] = pack_pair<C, N>(EN::in_row(p, i), x1[i], x2[i]);
    if (q + 1 < 6) {
      const int qn = q + 1;
      load(f1s[qn] + l1s[qn] * pin, f2s[qn] + l2s[qn] * pin);
    }
    fft_regs_p<C, PL, true, true, AD>(v, s, LDC, q, p, true, a.tw);
#pragma unroll
    for (int i = 0; i < E; ++i) s[AD::at(EN::out_row(p, i), q, LDC)] = v[i];
  }
  xline_w_tail<T, N>(s, a, la, lb, lane, pout);
}

// ------------------------------------------------ fused x pass, fields in registers
// One complex value, zero where !on; volatile, so that loads stay where they
// are issued, ahead of the transforms that hide them.
__device__ __forceinline__ float2 ld_on(const float2 *p, bool on) {
  float2 x = make_float2(0.f, 0.f);
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\t@q ld.global.v2.f32 {%0, %1}, [%2];\n\t}"
               : "+f"(x.x), "+f"(x.y)
               : "l"(p), "r"((unsigned)on));
  return x;
}
__device__ __forceinline__ double2 ld_on(const double2 *p, bool on) {
  double2 x = make_double2(0.0, 0.0);
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\t@q ld.global.v2.f64 {%0, %1}, [%2];\n\t}"
               : "+d"(x.x), "+d"(x.y)
               : "l"(p), "r"((unsigned)on));
  return x;
}
// The Hermitian sequence of two real lines: put(q, re, im) with the value of
// row p + P q of X1 + i X2, q < E, from the own rows n = p + P i <= N/2 (i <=
// E/2; i = E/2 is lane 0's Nyquist row) of the half lines x1, x2, whose
// imaginary parts at rows 0 and N/2 are zero.  Lane p forms its rows' values
// and their mirrors', which belong to lane P - p.
template <int E, typename C, typename PUT> __device__ __forceinline__ void pack_lines(const C *x1, const C *x2, int p,
                                                                                      int mirror, PUT put) {
  using T = decltype(C{}.x);
#pragma unroll
  for (int i = 0; i < E / 2; ++i) put(i, x1[i].x - x2[i].y, x1[i].y + x2[i].x);
#pragma unroll
  for (int i = 0; i < E / 2; ++i) {
    // lane p sends the mirror of its row i, lane 0 (its own partner) that of row i + 1
    const int j = i + 1;
    T re = x1[i].x + x2[i].y, im = x2[i].x - x1[i].y;
    const T re0 = x1[j].x + x2[j].y, im0 = x2[j].x - x1[j].y;
    re = p == 0 ? re0 : re;
    im = p == 0 ? im0 : im;
    put(E - 1 - i, __shfl_sync(0xffffffffu, re, mirror), __shfl_sync(0xffffffffu, im, mirror));
  }
}

// The exponent field of m >= 0, and 2^e (0 for e = -bias).  By bits in FP32:
// with ldexp the 256-point pass takes 138 us instead of 130 (256^3); in FP64
// ldexp is the faster (324 us against 338).
__device__ __forceinline__ int expo(float m) { return __float_as_int(m) >> 23; }
__device__ __forceinline__ int expo(double m) { return __double2hiint(m) >> 20; }
template <typename T> __device__ __forceinline__ T pow2(int e) {
  if constexpr (sizeof(T) == 4) return __int_as_float((127 + e) << 23);
  else return e == -1023 ? 0 : ldexp(1.0, e);
}
// The exponent e with which 2^e brings the half line x2 to the magnitude of x1
// (largest component of each, over the line's P lanes): they share one complex
// sequence, whose parts are rounded relative to each other; pow2(-e) undoes it.
// Where one of them vanishes, its part of the result is the other's rounding,
// which may be far above the field it belongs to: for a vanishing x2, e is the
// type's bias, whose pow2(-e) is 0; for a vanishing x1, flat is set.
template <int P, int H, typename C> __device__ __forceinline__ int balance(const C *x1, const C *x2, bool &flat) {
  using T = decltype(C{}.x);
  constexpr int bias = sizeof(T) == 4 ? 127 : 1023;
  T m1 = 0, m2 = 0;
#pragma unroll
  for (int i = 0; i <= H; ++i) {
    m1 = fmax(m1, fmax(fabs(x1[i].x), fabs(x1[i].y)));
    m2 = fmax(m2, fmax(fabs(x2[i].x), fabs(x2[i].y)));
  }
#pragma unroll
  for (int o = P / 2; o; o >>= 1) {
    m1 = fmax(m1, __shfl_xor_sync(0xffffffffu, m1, o));
    m2 = fmax(m2, __shfl_xor_sync(0xffffffffu, m2, o));
  }
  flat = m1 == 0;
  return m2 > 0 ? m1 > 0 ? max(1 - bias, min(bias - 1, expo(m1) - expo(m2))) : 0 : bias;
}

// Exchange tile of one line: rows skewed by row / R0, or for the 4 x 4 x ..
// plans of 96 and 192 exchanged by an exclusive or within 16, so that the
// strided writes of a stage and the consecutive reads of the next fall in
// distinct banks for 8- and 16-byte elements (counted for every access of
// every plan).
template <typename PL> struct XTile {
  static constexpr int N = PL::N, R0 = PL::R[0];
  static constexpr int SK = (R0 == 8 || R0 == 16) ? R0 : 4;
  static constexpr bool XOR = N == 96 || N == 192;
  static constexpr int pitch = PL::NST == 1 ? 0 : XOR ? N + (N == 96 ? 8 : 0) : N + N / SK;
  __device__ static __forceinline__ int at(int row, int) { return XOR ? row ^ (row >> 2 & 15) : row + row / SK; }
};
template <typename T, int N> struct XReg {
  using PL = XPlan<T, N>;
  // up to 48 (FP32) or 36 (FP64) held values per thread, a line within a warp
  static constexpr bool on = PL::P <= 32 && PL::E <= (sizeof(T) == 8 ? 12 : 16);
  static constexpr int NT = 128;                      // threads of a full block
  static constexpr size_t tw = ((size_t)vtw_size<PL>() * 2 * sizeof(T) + 15) / 16 * 16;
  static constexpr size_t line = (size_t)XTile<PL>::pitch * 16;
  static constexpr size_t smem(int threads) { return tw + threads / PL::P * line; }
  static constexpr int minb = sizeof(T) == 8 ? (PL::E <= 8 ? 3 : 2) : (PL::E <= 8 ? 5 : PL::E == 12 ? 4 : 3);
};

// Fused x pass: P lanes own one line from its loads to its stores.  Every plan
// gives a lane the rows p + P q at both ends of a transform, so u, v, w and the
// vorticity of a row meet in one lane's registers after the inverse
// transforms, the cross product is formed there and is the forward
// transforms' input; shared memory carries only each transform's exchanges.
// A line's six real lines are three sequences: U + iV and OX + i OY, in single
// precision transformed together as pairs, and W + i 2^e OZ, whose parts are
// brought to one magnitude first (the transform rounds them relative to each
// other; e is the difference of the half lines' exponents, exact both ways).
// Forward, px + i py and pz + i 0 (its transform is the half line itself).
// A lane loads its rows up to N/2 and forms both that row's value and its
// Hermitian mirror's, which goes to the lane that holds row N - n by shuffle.
// Against the block kernel (fields in shared memory, bank conflicts) and the
// warp kernels it replaces, us: 32 boxes of 64^3 FP32 150 -> 73, of 32^3 29 -> 17,
// 128^3 56 -> 25, 256^3 162 -> 131 (FP64 397 -> 326), 512^3 1698 -> 1285.  At 256 in
// FP32 it is balanced: issue 57-60%, FMA pipe 50%, L1 60-64%, 12 warps by registers;
// FP64 is bound by L1 (82-88%), the exchanges.  All loads of a line up front (the
// third sequence's during the pair's transform) brought 179 -> 140 at 256.
template <typename T, int N>
__global__ void __launch_bounds__(XReg<T, N>::NT, XReg<T, N>::minb)
    k_xline_nl_g(const __grid_constant__ XlineNLArgs<T> a) {
  using C = typename CT<T>::type;
  using SH = XReg<T, N>;
  using PL = typename SH::PL;
  using EN = VEnds<PL>;
  using AD = XTile<PL>;
  using V1 = VC<T>;
  constexpr int E = PL::E, P = PL::P, H = E / 2;
  constexpr bool PAIR = sizeof(T) == 4;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V1 *twt = reinterpret_cast<V1 *>(smem_raw);
  pdl_launch();
  vtw_fill<PL, V1>(twt, a.tw, threadIdx.x, blockDim.x);
  __syncthreads();
  pdl_wait();
  const int g = threadIdx.x / P, p = threadIdx.x % P, lane = threadIdx.x & 31;
  unsigned char *tile = smem_raw + SH::tw + (size_t)g * SH::line;
  V1 *s1 = reinterpret_cast<V1 *>(tile);
  const long long pin = a.pin ? a.pin : a.nxh, pout = a.pout ? a.pout : a.nxh;
  // last lines first: what pass B wrote last is still in L2
  const unsigned blk = gridDim.x - 1 - blockIdx.x;
  const long long line = (long long)blk * (blockDim.x / P) + g;
  const bool on = line < a.nlines;
  const int mirror = (lane & ~(P - 1)) | ((P - p) & (P - 1));   // lane of rows N - n
  auto sync = []() { __syncwarp(); };
  // own rows n = p + P i, i <= H (i = H: the Nyquist row of lane 0), bit i of own
  unsigned own = 0;
#pragma unroll
  for (int i = 0; i <= H; ++i)
    if (on && (i < H || p == 0) && xkeep(a.kxa, p + P * i, N)) own |= 1u << i;
  const int nyq = a.nyq ? a.nyq : N / 2;
  auto load = [&](const C *f, C *x) {
    const C *r = f + line * pin;
#pragma unroll
    for (int i = 0; i <= H; ++i) {
      x[i] = ld_on(r + (i == H ? nyq : p + P * i), own >> i & 1);
    }
    if (p == 0) x[0].y = x[H].y = 0;   // a C2R drops these imaginary parts
  };
  auto shfl = [&](T v) { return __shfl_sync(0xffffffffu, v, mirror); };
  auto pack = [&](const C *x1, const C *x2, auto put) { pack_lines<E>(x1, x2, p, mirror, put); };
  T down, keep;   // factors of oz and w (0 where they vanish: a value that is no number stays one)
  V1 w[E];   // (w, 2^e oz) at row p + P q in w[out_i(q)]
  T u_[E], v_[E], ox_[E], oy_[E];
  C xw[H + 1], xo[H + 1];
  if constexpr (PAIR) {
    using V2 = VC<f2>;
    V2 z[E], x[E];
    {
      C x1[H + 1], x2[H + 1], x3[H + 1], x4[H + 1];
      load(a.U, x1);
      load(a.V, x2);
      load(a.OX, x3);
      load(a.OY, x4);
      load(a.W, xw);   // on their way during the pair's transform
      load(a.OZ, xo);
      T re[E], im[E];
      pack(x1, x2, [&](int q, T r, T i) { re[q] = r, im[q] = i; });
      pack(x3, x4, [&](int q, T r, T i) { z[EN::in_i(q)] = V2{mkf2(re[q], r), mkf2(im[q], i)}; });
    }
    vfft<PL, true, AD>(z, x, reinterpret_cast<V2 *>(tile), 0, p, twt, sync);
#pragma unroll
    for (int i = 0; i < E; ++i) u_[i] = f2_lo(x[i].re), v_[i] = f2_lo(x[i].im), ox_[i] = f2_hi(x[i].re), oy_[i] = f2_hi(x[i].im);
  } else {
    load(a.U, xw);
    load(a.V, xo);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      V1 z[E], x[E];
      pack(xw, xo, [&](int q, T r, T i) { z[EN::in_i(q)] = V1{r, i}; });
      load(k == 0 ? a.OX : a.W, xw);   // the next sequence's rows
      load(k == 0 ? a.OY : a.OZ, xo);
      vfft<PL, true, AD>(z, x, s1, 0, p, twt, sync);
      sync();
#pragma unroll
      for (int i = 0; i < E; ++i) (k == 0 ? u_ : ox_)[i] = x[i].re, (k == 0 ? v_ : oy_)[i] = x[i].im;
    }
  }
  {
    bool flat;
    const int d = balance<P, H>(xw, xo, flat);
    const T up = pow2<T>(d);
#pragma unroll
    for (int i = 0; i <= H; ++i) xo[i] = mkc<C>(xo[i].x * up, xo[i].y * up);
    V1 z[E];
    pack(xw, xo, [&](int q, T r, T i) { z[EN::in_i(q)] = V1{r, i}; });
    sync();
    vfft<PL, true, AD>(z, w, s1, 0, p, twt, sync);
    sync();
    down = pow2<T>(-d);
    keep = flat ? T(0) : T(1);
  }
  // (omega x u) s at the lane's rows, and the CFL maxima
  const T sc = T(a.s);
  T m0 = 0, m1 = 0, m2 = 0;
  T px[E], py[E], pz[E];
#pragma unroll
  for (int i = 0; i < E; ++i) {
    const T u = u_[i], v = v_[i], ww = w[i].re * keep, oz = w[i].im * down, ox = ox_[i], oy = oy_[i];
    px[i] = (oy * ww - oz * v) * sc;
    py[i] = (oz * u - ox * ww) * sc;
    pz[i] = (ox * v - oy * u) * sc;
    m0 = fmax(m0, fabs(u));
    m1 = fmax(m1, fabs(v));
    m2 = fmax(m2, fabs(ww));
  }
  // forward; rows k = p + P i <= N/2 of the half lines: of px + i py by
  // X1 = (Z[k] + conj Z[N-k]) / 2, X2 = (Z[k] - conj Z[N-k]) / 2i, of pz its transform
  C *const dx = a.NX + line * pout, *const dy = a.NY + line * pout, *const dz = a.NZ + line * pout;
  auto store = [&](int i, T zr, T zi, T nr, T ni, bool xy, T fr, T fi, bool z) {
    if (!(own >> i & 1)) return;
    const int sl = i == H ? nyq : p + P * i;
    if (xy) {
      dx[sl] = mkc<C>(T(0.5) * (zr + nr), T(0.5) * (zi - ni));
      dy[sl] = mkc<C>(T(0.5) * (zi + ni), T(0.5) * (nr - zr));
    }
    if (z) dz[sl] = mkc<C>(fr, fi);
  };
  if constexpr (PAIR) {
    using V2 = VC<f2>;
    V2 z[E], x[E];
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const int i = EN::out_i(q);
      z[EN::in_i(q)] = V2{mkf2(px[i], pz[i]), mkf2(py[i], T(0))};
    }
    vfft<PL, false, AD>(z, x, reinterpret_cast<V2 *>(tile), 0, p, twt, sync);
#pragma unroll
    for (int i = 0; i <= H; ++i) {
      const V2 zk = x[EN::out_i(i)];
      T nr = f2_lo(zk.re), ni = f2_lo(zk.im);   // i = H: row N/2, its own mirror
      if (i < H) {
        const V2 b = x[EN::out_i(E - 1 - i)], b0 = x[EN::out_i((E - i) % E)];
        nr = shfl(p == 0 ? f2_lo(b0.re) : f2_lo(b.re));
        ni = shfl(p == 0 ? f2_lo(b0.im) : f2_lo(b.im));
      }
      store(i, f2_lo(zk.re), f2_lo(zk.im), nr, ni, true, f2_hi(zk.re), f2_hi(zk.im), true);
    }
  } else {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      V1 z[E], x[E];
#pragma unroll
      for (int q = 0; q < E; ++q) {
        const int i = EN::out_i(q);
        z[EN::in_i(q)] = k == 0 ? V1{px[i], py[i]} : V1{pz[i], T(0)};
      }
      if (k) sync();
      vfft<PL, false, AD>(z, x, s1, 0, p, twt, sync);
#pragma unroll
      for (int i = 0; i <= H; ++i) {
        const V1 zk = x[EN::out_i(i)];
        T nr = zk.re, ni = zk.im;
        if (k == 0 && i < H) {
          const V1 b = x[EN::out_i(E - 1 - i)], b0 = x[EN::out_i((E - i) % E)];
          nr = shfl(p == 0 ? b0.re : b.re);
          ni = shfl(p == 0 ? b0.im : b.im);
        }
        store(i, zk.re, zk.im, nr, ni, k == 0, zk.re, zk.im, k == 1);
      }
    }
  }
  if (on)
    for (int j = p; j < a.npad; j += P) dx[nyq + 1 + j] = dy[nyq + 1 + j] = dz[nyq + 1 + j] = mkc<C>(0, 0);
  // CFL maxima: of the lane's line, then of the warp's lines where they share a box
  if (!a.st) return;
#pragma unroll
  for (int o = P / 2; o; o >>= 1) {
    m0 = fmax(m0, __shfl_xor_sync(0xffffffffu, m0, o));
    m1 = fmax(m1, __shfl_xor_sync(0xffffffffu, m1, o));
    m2 = fmax(m2, __shfl_xor_sync(0xffffffffu, m2, o));
  }
  const int box = (int)((on ? line : (long long)a.nlines - 1) / a.lines_per_box);
  bool lead = p == 0 && on;
  if (P < 32 && __all_sync(0xffffffffu, box == __shfl_sync(0xffffffffu, box, 0))) {
#pragma unroll
    for (int o = 16; o >= P; o >>= 1) {
      m0 = fmax(m0, __shfl_xor_sync(0xffffffffu, m0, o));
      m1 = fmax(m1, __shfl_xor_sync(0xffffffffu, m1, o));
      m2 = fmax(m2, __shfl_xor_sync(0xffffffffu, m2, o));
    }
    lead = lane == 0 && on;
  }
  if (lead) {
    // only a larger value needs the atomic (the stored one never decreases)
    double *um = a.st[box].umax;
    const double x[3] = {(double)m0 * a.s, (double)m1 * a.s, (double)m2 * a.s};
#pragma unroll
    for (int c = 0; c < 3; ++c)
      if (!(x[c] <= __ldcg(um + c))) atomic_max_nonneg(um + c, x[c]);
  }
}

// The fused x pass of 96- (FP32) and 192-point lines of large boxes (the rule
// stands at the launch): k_xline_nl_g with split plans (SplitPlan), so that each transform exchanges once, not twice, through the
// shared memory that bounds it.  A block of 8 lines: R1 lanes a line load,
// form the sequences and run the inverse transforms' first stage; after one
// barrier R0 lanes a line run the second stage, form the products and run the
// forward transforms' first stage; R1 lanes a line finish and store.  The tile
// rows are skewed by row / R of the stage that writes them (16-byte accesses
// of every stage free of bank conflicts at the pitches of SplitPlan).  Against
// k_xline_nl_g, us: 32 boxes of 96^3 FP32 285 -> 253 (L1 87% -> 67-75%, now bound by
// load latency and the block's barriers), 192^3 FP32 77 -> 68, FP64 165 -> 148.
template <typename T, int N> struct XSplit {
  using SP = SplitPlan<N>;
  static constexpr int L = 8, PO = SP::R1, PI = SP::R0, NT = L * (PO > PI ? PO : PI);
  static constexpr int ntw = (SP::R1 - 1) * SP::R0 + (SP::R0 - 1) * SP::R1;
  static constexpr size_t tw = ((size_t)ntw * 2 * sizeof(T) + 15) / 16 * 16;
  static constexpr size_t buf = (size_t)L * SP::pitch * 16;   // a pair of sequences (FP32) or one (FP64)
  static constexpr size_t smem = tw + (sizeof(T) == 4 ? buf + buf / 2 : 3 * buf);
  // 96 FP32: 18 warps by 96 registers (some spills) 258 us, 15 by 128 270, 21 by
  // 80 275 (32 boxes of 96^3); 192 FP32: 16 warps 65 us, 12 71 (192^3)
  static constexpr int minb = sizeof(T) == 8 ? 2 : (N == 96 ? 6 : 4);
};
template <typename T, int N>
__global__ void __launch_bounds__(XSplit<T, N>::NT, XSplit<T, N>::minb)
    k_xline_nl_s(const __grid_constant__ XlineNLArgs<T> a) {
  using C = typename CT<T>::type;
  using SH = XSplit<T, N>;
  using SP = SplitPlan<N>;
  using V1 = VC<T>;
  using VP = VC<typename VecOf<T>::R>;   // the pair (FP32); FP64 transforms its two sequences one by one
  constexpr int R0 = SP::R0, R1 = SP::R1, H = R0 / 2, L = SH::L, PO = SH::PO, PI = SH::PI, NP = sizeof(T) == 4 ? 1 : 2;
  constexpr bool PAIR = NP == 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int ex[L];
  __shared__ bool noW[L];
  V1 *twi = reinterpret_cast<V1 *>(smem_raw), *twf = twi + (R1 - 1) * R0;
  pdl_launch();
  for (int i = threadIdx.x; i < (R1 - 1) * R0; i += SH::NT) twi[i] = VtwOf<V1>::of(__ldg(a.tw + (1 + i / R0) * (i % R0)));
  for (int i = threadIdx.x; i < (R0 - 1) * R1; i += SH::NT) twf[i] = VtwOf<V1>::of(__ldg(a.tw + (1 + i / R1) * (i % R1)));
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const unsigned blk = gridDim.x - 1 - blockIdx.x;   // last lines first, as pass B left them in L2
  const long long line0 = (long long)blk * L;
  const bool outer = threadIdx.x < L * PO, inner = threadIdx.x < L * PI;   // whole warps
  const int lo = threadIdx.x / PO, po = threadIdx.x % PO, li = threadIdx.x / PI, pi = threadIdx.x % PI;
  const bool on = outer && line0 + lo < a.nlines;
  const long long pin = a.pin ? a.pin : a.nxh, pout = a.pout ? a.pout : a.nxh;
  const int mirror = (lane & ~(PO - 1)) | ((PO - po) & (PO - 1));
  const int nyq = a.nyq ? a.nyq : N / 2;
  auto bufp = [&](int k, int line) { return reinterpret_cast<VP *>(smem_raw + SH::tw + k * SH::buf) + line * SP::pitch; };
  auto bufs = [&](int line) { return reinterpret_cast<V1 *>(smem_raw + SH::tw + NP * SH::buf) + line * SP::pitch; };
  auto inv_at = [](int row) { return row + row / R0; };   // written p R0 + r
  auto fwd_at = [](int row) { return row + row / R1; };   // written p R1 + r
  unsigned own = 0;   // bit i: row po + PO i is read and written
#pragma unroll
  for (int i = 0; i <= H; ++i)
    if (on && (i < H || po == 0) && xkeep(a.kxa, po + PO * i, N)) own |= 1u << i;
  if (outer) {
    auto load = [&](const C *f, C *x) {
      const C *r = f + (line0 + lo) * pin;
#pragma unroll
      for (int i = 0; i <= H; ++i) x[i] = ld_on(r + (i == H ? nyq : po + PO * i), own >> i & 1);
      if (po == 0) x[0].y = x[H].y = 0;   // a C2R drops these imaginary parts
    };
    C x1[H + 1], x2[H + 1], x3[H + 1], x4[H + 1], x5[H + 1], x6[H + 1];
    load(a.U, x1);
    load(a.V, x2);
    load(a.OX, x3);
    load(a.OY, x4);
    load(a.W, x5);
    load(a.OZ, x6);
    if constexpr (PAIR) {
      VP z[R0], y[R0];
      T re[R0], im[R0];
      pack_lines<R0>(x1, x2, po, mirror, [&](int q, T r, T i) { re[q] = r, im[q] = i; });
      pack_lines<R0>(x3, x4, po, mirror, [&](int q, T r, T i) { z[q] = VP{mkf2(re[q], r), mkf2(im[q], i)}; });
      vdft<R0, true>(z, y);
#pragma unroll
      for (int r = 0; r < R0; ++r) bufp(0, lo)[inv_at(po * R0 + r)] = y[r];
    } else {
      V1 z[R0], y[R0];
      pack_lines<R0>(x1, x2, po, mirror, [&](int q, T r, T i) { z[q] = V1{r, i}; });
      vdft<R0, true>(z, y);
#pragma unroll
      for (int r = 0; r < R0; ++r) reinterpret_cast<V1 *>(bufp(0, lo))[inv_at(po * R0 + r)] = y[r];
      pack_lines<R0>(x3, x4, po, mirror, [&](int q, T r, T i) { z[q] = V1{r, i}; });
      vdft<R0, true>(z, y);
#pragma unroll
      for (int r = 0; r < R0; ++r) reinterpret_cast<V1 *>(bufp(1, lo))[inv_at(po * R0 + r)] = y[r];
    }
    bool flat;
    const int d = balance<PO, H>(x5, x6, flat);
    if (po == 0) ex[lo] = d, noW[lo] = flat;
    const T up = ldexp(T(1), d);   // ldexp: 251 us where pow2 takes 262 (32 boxes of 96^3)
#pragma unroll
    for (int i = 0; i <= H; ++i) x6[i] = mkc<C>(x6[i].x * up, x6[i].y * up);
    V1 z[R0], y[R0];
    pack_lines<R0>(x5, x6, po, mirror, [&](int q, T r, T i) { z[q] = V1{r, i}; });
    vdft<R0, true>(z, y);
#pragma unroll
    for (int r = 0; r < R0; ++r) bufs(lo)[inv_at(po * R0 + r)] = y[r];
  }
  __syncthreads();
  VP fy[NP][R1];   // first stage of the forward transforms
  T m0 = 0, m1 = 0, m2 = 0;
  if (inner) {
    auto second = [&](auto *b, auto *x) {
      using V = std::remove_pointer_t<decltype(b)>;
      V v[R1];
#pragma unroll
      for (int r = 0; r < R1; ++r) v[r] = b[inv_at(pi + r * R0)];
#pragma unroll
      for (int r = 1; r < R1; ++r) v[r] = vtwmul<true>(v[r], twi[(r - 1) * R0 + pi]);
      vdft<R1, true>(v, x);
    };
    VP x[NP][R1];
    V1 w[R1];
#pragma unroll
    for (int k = 0; k < NP; ++k) second(bufp(k, li), x[k]);
    second(bufs(li), w);
    constexpr int bias = sizeof(T) == 4 ? 127 : 1023;
    const T keep = noW[li] ? T(0) : T(1);
    const T down = ex[li] == bias ? T(0) : ldexp(T(1), -ex[li]), sc = T(a.s);
    VP f[NP][R1];
#pragma unroll
    for (int q = 0; q < R1; ++q) {
      T u, v, ox, oy;
      if constexpr (PAIR) u = f2_lo(x[0][q].re), v = f2_lo(x[0][q].im), ox = f2_hi(x[0][q].re), oy = f2_hi(x[0][q].im);
      else u = x[0][q].re, v = x[0][q].im, ox = x[1][q].re, oy = x[1][q].im;
      const T ww = w[q].re * keep, oz = w[q].im * down;
      const T px = (oy * ww - oz * v) * sc, py = (oz * u - ox * ww) * sc, pz = (ox * v - oy * u) * sc;
      m0 = fmax(m0, fabs(u));
      m1 = fmax(m1, fabs(v));
      m2 = fmax(m2, fabs(ww));
      if constexpr (PAIR) f[0][q] = VP{mkf2(px, pz), mkf2(py, T(0))};
      else f[0][q] = VP{px, py}, f[1][q] = VP{pz, T(0)};
    }
#pragma unroll
    for (int k = 0; k < NP; ++k) vdft<R1, false>(f[k], fy[k]);
  }
  __syncthreads();   // the inverse transforms' tiles are free
  if (inner) {
#pragma unroll
    for (int k = 0; k < NP; ++k)
#pragma unroll
      for (int r = 0; r < R1; ++r) bufp(k, li)[fwd_at(pi * R1 + r)] = fy[k][r];
  }
  __syncthreads();
  if (outer) {
    VP x[NP][R0];
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      VP v[R0];
#pragma unroll
      for (int r = 0; r < R0; ++r) v[r] = bufp(k, lo)[fwd_at(po + r * R1)];
#pragma unroll
      for (int r = 1; r < R0; ++r) v[r] = vtwmul<false>(v[r], twf[(r - 1) * R1 + po]);
      vdft<R0, false>(v, x[k]);
    }
    // rows k = po + PO i <= N/2 of the half lines (as k_xline_nl_g)
    C *const dx = a.NX + (line0 + lo) * pout, *const dy = a.NY + (line0 + lo) * pout, *const dz = a.NZ + (line0 + lo) * pout;
    auto re = [&](int k, int i) {
      if constexpr (PAIR) return k == 0 ? f2_lo(x[0][i].re) : f2_hi(x[0][i].re);
      else return x[k][i].re;
    };
    auto im = [&](int k, int i) {
      if constexpr (PAIR) return k == 0 ? f2_lo(x[0][i].im) : f2_hi(x[0][i].im);
      else return x[k][i].im;
    };
#pragma unroll
    for (int i = 0; i <= H; ++i) {
      const T zr = re(0, i), zi = im(0, i);
      T nr = zr, ni = zi;   // i = H: row N/2, its own mirror
      if (i < H) {
        nr = __shfl_sync(0xffffffffu, po == 0 ? re(0, (R0 - i) % R0) : re(0, R0 - 1 - i), mirror);
        ni = __shfl_sync(0xffffffffu, po == 0 ? im(0, (R0 - i) % R0) : im(0, R0 - 1 - i), mirror);
      }
      if (own >> i & 1) {
        const int sl = i == H ? nyq : po + PO * i;
        dx[sl] = mkc<C>(T(0.5) * (zr + nr), T(0.5) * (zi - ni));
        dy[sl] = mkc<C>(T(0.5) * (zi + ni), T(0.5) * (nr - zr));
        dz[sl] = mkc<C>(re(1, i), im(1, i));
      }
    }
    if (on)
      for (int j = po; j < a.npad; j += PO) dx[nyq + 1 + j] = dy[nyq + 1 + j] = dz[nyq + 1 + j] = mkc<C>(0, 0);
  }
  if (!a.st || !inner) return;
  // CFL maxima (a box has a multiple of 16 lines, so the block's lines share one)
  m0 = warp_max(m0);
  m1 = warp_max(m1);
  m2 = warp_max(m2);
  if (lane == 0) {
    double *um = a.st[line0 / a.lines_per_box].umax;
    const double m[3] = {(double)m0 * a.s, (double)m1 * a.s, (double)m2 * a.s};
#pragma unroll
    for (int c = 0; c < 3; ++c)
      if (!(m[c] <= __ldcg(um + c))) atomic_max_nonneg(um + c, m[c]);
  }
}

// ----------------------------------------------- fused x pass of the transposed term
template <typename T> struct XlineVjpArgs {
  using C = typename CT<T>::type;
  const C *U, *V, *W, *OX, *OY, *OZ, *FX, *FY, *FZ;   // (kx, y, z) rows of `pitch`
  C *A[3], *B[3];                                      // forward x transforms of u x phi and phi x omega
  const C *tw;
  int nlines, pitch;
};
template <typename T, int N> struct XVjp {
  using PL = XPlan<T, N>;
  static constexpr int minb = sizeof(T) == 8 ? 2 : (PL::E <= 8 ? 4 : PL::E == 12 ? 3 : 2);
};

// The x pass of rhs_nonlinear's transpose: C2R of u, omega and phi, the cross
// products u x phi and phi x omega, and their R2C, in the manner of
// k_xline_nl_g.  The products are taken one after the other, so that a lane
// holds two vectors at a time.
// A transform rounds the parts of its sequence relative to the larger one, and
// neither the cotangent's scale is the flow's nor one component's another's: a
// sequence holds two neighbouring lines (a, b) of one field.  The P-lane groups
// of a and b (neighbours in a warp) each transform one of two fields,
// U_a + i U_b and V_a + i V_b, and swap a real line, after which either holds
// both fields of its own line; the other way round forward.  (FX, FY) are the
// second of a pair in FP32; then (W, FZ); (OX, OY) with OZ, alone on its line.
// It replaces nine C2R and six R2C lines of global memory traffic and a
// pointwise kernel, four kernels of 58 us at 96^3 FP32.  With both parts of a
// sequence from one line, and small ones lost in large ones, it took 28.5 us at
// 96^3 FP32 and 12.1 at 64^3 FP64 (from a cold L2); the swaps make it 29.9, 12.8.
template <typename T, int N>
__global__ void __launch_bounds__(XReg<T, N>::NT, XVjp<T, N>::minb)
    k_xline_vjp(const __grid_constant__ XlineVjpArgs<T> a) {
  using C = typename CT<T>::type;
  using SH = XReg<T, N>;
  using PL = typename SH::PL;
  using EN = VEnds<PL>;
  using AD = XTile<PL>;
  using V1 = VC<T>;
  using V2 = VC<f2>;
  constexpr int E = PL::E, P = PL::P, H = E / 2;
  constexpr bool PAIR = sizeof(T) == 4;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V1 *twt = reinterpret_cast<V1 *>(smem_raw);
  pdl_launch();
  vtw_fill<PL, V1>(twt, a.tw, threadIdx.x, blockDim.x);
  __syncthreads();
  pdl_wait();
  const int g = threadIdx.x / P, p = threadIdx.x % P, lane = threadIdx.x & 31;
  const bool odd = g & 1;
  unsigned char *tile = smem_raw + SH::tw + (size_t)g * SH::line;
  V1 *s1 = reinterpret_cast<V1 *>(tile);
  V2 *s2 = reinterpret_cast<V2 *>(tile);
  const unsigned blk = gridDim.x - 1 - blockIdx.x;   // last lines first, as pass B left them in L2
  const long long line = (long long)blk * (blockDim.x / P) + g, la = line - odd;
  const bool on = line < a.nlines;   // of both lines: their number is even
  const int mirror = (lane & ~(P - 1)) | ((P - p) & (P - 1));
  auto sync = []() { __syncwarp(); };
  auto load = [&](const C *f, long long l, C *x) {
    const C *r = f + l * a.pitch + p;
#pragma unroll
    for (int i = 0; i <= H; ++i) x[i] = ld_on(r + P * i, on && (i < H || p == 0));
    if (p == 0) x[0].y = x[H].y = 0;   // a C2R drops these imaginary parts
  };
  // v[i] of the other line's group in exchange for this one's
  auto swap = [&](T *v) {
    if constexpr (P < 32) {
#pragma unroll
      for (int i = 0; i < E; ++i) v[i] = __shfl_xor_sync(0xffffffffu, v[i], P);
    } else {   // the two warps of a pair, through their tiles
      auto both = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + (g >> 1)) : "memory"); };
      T *mine = reinterpret_cast<T *>(tile) + lane;
      const T *other = reinterpret_cast<const T *>(smem_raw + SH::tw + (size_t)(g ^ 1) * SH::line) + lane;
      static_assert(E * 32 * sizeof(T) <= SH::line, "a line's values fit its tile");
      sync();   // the transform's reads of the tile are through
#pragma unroll
      for (int i = 0; i < E; ++i) mine[32 * i] = v[i];
      both();
#pragma unroll
      for (int i = 0; i < E; ++i) v[i] = other[32 * i];
      both();
    }
  };
  // the real lines of both fields on the own line, from lines a (re) and b (im) of the own field
  auto own = [&](T *re, T *im, T *f0, T *f1) {
    T x[E];
#pragma unroll
    for (int i = 0; i < E; ++i) x[i] = odd ? re[i] : im[i];
    swap(x);
#pragma unroll
    for (int i = 0; i < E; ++i) {
      const T r = re[i], m = im[i];
      f0[i] = odd ? x[i] : r;
      f1[i] = odd ? m : x[i];
    }
  };
  // inverse transform of X1 + i X2 into (re, im) at row p + P q in [out_i(q)]
  auto inv1 = [&](const C *x1, const C *x2, T *re, T *im) {
    V1 z[E], x[E];
    pack_lines<E>(x1, x2, p, mirror, [&](int q, T r, T i) { z[EN::in_i(q)] = V1{r, i}; });
    sync();
    vfft<PL, true, AD>(z, x, s1, 0, p, twt, sync);
#pragma unroll
    for (int i = 0; i < E; ++i) re[i] = x[i].re, im[i] = x[i].im;
  };
  auto inv2 = [&](const C *x1, const C *x2, const C *x3, const C *x4, T *r1, T *i1, T *r2, T *i2) {
    if constexpr (PAIR) {
      V2 z[E], x[E];
      T re[E], im[E];
      pack_lines<E>(x1, x2, p, mirror, [&](int q, T r, T i) { re[q] = r, im[q] = i; });
      pack_lines<E>(x3, x4, p, mirror, [&](int q, T r, T i) { z[EN::in_i(q)] = V2{mkf2(re[q], r), mkf2(im[q], i)}; });
      sync();
      vfft<PL, true, AD>(z, x, s2, 0, p, twt, sync);
#pragma unroll
      for (int i = 0; i < E; ++i)
        r1[i] = f2_lo(x[i].re), i1[i] = f2_lo(x[i].im), r2[i] = f2_hi(x[i].re), i2[i] = f2_hi(x[i].im);
    } else {
      inv1(x1, x2, r1, i1);
      inv1(x3, x4, r2, i2);
    }
  };
  // forward transforms of the own line's c0, c1, c2, stored as half lines of d[0..2]:
  // one of c0 and c1 for both lines, c2 + i 0
  auto fwd = [&](T *c0, T *c1, const T *c2, C *const *d) {
    T x1[E];
#pragma unroll
    for (int i = 0; i < E; ++i) x1[i] = odd ? c0[i] : c1[i];
    swap(x1);
#pragma unroll
    for (int i = 0; i < E; ++i) {
      const T r = odd ? x1[i] : c0[i];
      c1[i] = odd ? c1[i] : x1[i];   // line b
      c0[i] = r;                     // line a
    }
    C *const d0 = odd ? d[1] : d[0], *const d2 = d[2];
    auto store = [&](int i, T zr, T zi, T nr, T ni) {
      if (!(on && (i < H || p == 0))) return;
      C *const o = d0 + la * a.pitch + p + P * i;
      o[0] = mkc<C>(T(0.5) * (zr + nr), T(0.5) * (zi - ni));
      o[a.pitch] = mkc<C>(T(0.5) * (zi + ni), T(0.5) * (nr - zr));
    };
    auto store3 = [&](int i, T zr, T zi) {
      if (on && (i < H || p == 0)) d2[line * a.pitch + p + P * i] = mkc<C>(zr, zi);
    };
    if constexpr (PAIR) {
      V2 z[E], x[E];
#pragma unroll
      for (int q = 0; q < E; ++q) {
        const int i = EN::out_i(q);
        z[EN::in_i(q)] = V2{mkf2(c0[i], c2[i]), mkf2(c1[i], T(0))};
      }
      sync();
      vfft<PL, false, AD>(z, x, s2, 0, p, twt, sync);
#pragma unroll
      for (int i = 0; i <= H; ++i) {
        const V2 zk = x[EN::out_i(i)];
        T nr = f2_lo(zk.re), ni = f2_lo(zk.im);   // i = H: row N/2, its own mirror
        if (i < H) {
          const V2 b = x[EN::out_i(E - 1 - i)], b0 = x[EN::out_i((E - i) % E)];
          nr = __shfl_sync(0xffffffffu, p == 0 ? f2_lo(b0.re) : f2_lo(b.re), mirror);
          ni = __shfl_sync(0xffffffffu, p == 0 ? f2_lo(b0.im) : f2_lo(b.im), mirror);
        }
        store(i, f2_lo(zk.re), f2_lo(zk.im), nr, ni);
        store3(i, f2_hi(zk.re), f2_hi(zk.im));
      }
    } else {
      V1 z[E], x[E];
#pragma unroll
      for (int q = 0; q < E; ++q) {
        const int i = EN::out_i(q);
        z[EN::in_i(q)] = V1{c0[i], c1[i]};
      }
      sync();
      vfft<PL, false, AD>(z, x, s1, 0, p, twt, sync);
#pragma unroll
      for (int i = 0; i <= H; ++i) {
        const V1 zk = x[EN::out_i(i)];
        T nr = zk.re, ni = zk.im;
        if (i < H) {
          const V1 b = x[EN::out_i(E - 1 - i)], b0 = x[EN::out_i((E - i) % E)];
          nr = __shfl_sync(0xffffffffu, p == 0 ? b0.re : b.re, mirror);
          ni = __shfl_sync(0xffffffffu, p == 0 ? b0.im : b.im, mirror);
        }
        store(i, zk.re, zk.im, nr, ni);
      }
#pragma unroll
      for (int q = 0; q < E; ++q) z[EN::in_i(q)] = V1{c2[EN::out_i(q)], T(0)};
      sync();
      vfft<PL, false, AD>(z, x, s1, 0, p, twt, sync);
#pragma unroll
      for (int i = 0; i <= H; ++i) store3(i, x[EN::out_i(i)].re, x[EN::out_i(i)].im);
    }
  };
  T u[E], v[E], w[E], fx[E], fy[E], fz[E];
  {
    C x1[H + 1], x2[H + 1], x3[H + 1], x4[H + 1], x5[H + 1], x6[H + 1];
    const C *const q1 = odd ? a.V : a.U, *const q2 = odd ? a.FY : a.FX, *const q3 = odd ? a.FZ : a.W;
    load(q1, la, x1);
    load(q1, la + 1, x2);
    load(q2, la, x3);
    load(q2, la + 1, x4);
    load(q3, la, x5);   // on their way during the first transforms
    load(q3, la + 1, x6);
    inv2(x1, x2, x3, x4, u, v, fx, fy);
    own(u, v, u, v);
    own(fx, fy, fx, fy);
    inv1(x5, x6, w, fz);
    own(w, fz, w, fz);
  }
  C x1[H + 1], x2[H + 1], x3[H + 1], x0[H + 1];
  const C *const q1 = odd ? a.OY : a.OX;
  load(q1, la, x1);
  load(q1, la + 1, x2);
  load(a.OZ, line, x3);
#pragma unroll
  for (int i = 0; i <= H; ++i) x0[i] = mkc<C>(0, 0);
#pragma unroll
  for (int i = 0; i < E; ++i) {   // u x phi
    const T c0 = v[i] * fz[i] - w[i] * fy[i], c1 = w[i] * fx[i] - u[i] * fz[i], c2 = u[i] * fy[i] - v[i] * fx[i];
    u[i] = c0, v[i] = c1, w[i] = c2;
  }
  fwd(u, v, w, a.A);
  T zero[E];
  inv2(x1, x2, x3, x0, u, v, w, zero);   // omega
  own(u, v, u, v);
#pragma unroll
  for (int i = 0; i < E; ++i) {   // phi x omega
    const T c0 = fy[i] * w[i] - fz[i] * v[i], c1 = fz[i] * u[i] - fx[i] * w[i], c2 = fx[i] * v[i] - fy[i] * u[i];
    u[i] = c0, v[i] = c1, w[i] = c2;
  }
  fwd(u, v, w, a.B);
}

// ------------------------------------------------------- plain x-line transforms
template <typename T> struct XlineArgs {
  using C = typename CT<T>::type;
  const void *in[6];
  void *out[6];
  const C *tw;
  int nlines, nxh;
  int pitch;               // row pitch (complex elements) of the half lines; 0: nxh
  int absval;              // with vmax: maxima of |x| (1) or of x (0)
  double scale;            // multiplies the output
  unsigned long long *vmax;   // C2R: take the maximum of each field into vmax[field] (max_key) and store nothing
};

// Doubles in increasing order as unsigned integers, for an atomic maximum
// (0 is below every value); the host inverts it (max_of_key).
__host__ __device__ __forceinline__ unsigned long long max_key_bits(unsigned long long b) {
  return b >> 63 ? ~b : b | 0x8000000000000000ull;
}

// P lanes own a pair of lines (la, lb) as one complex sequence X1 + i X2, in
// registers but for the exchanges (the plans and tiles of k_xline_nl_g; 16
// values a thread in both precisions, 32 at 1024).  8 and 12 points by two lanes:
// with one, a lane walks a whole line and a warp's accesses spread over 64 of them
// (12 x 256 x 256 FP64 C2R 29.7 us against 17.1, rhs_adj 391 / 340; 8 x 512 x 512 FP32
// C2R 56 / 35).
template <int N> struct LPlan : VPlan<N> {};
#define DNSBOX_LPLAN(NN, EE, ...)                                                                                    \
  template <> struct LPlan<NN> {                                                                                     \
    static constexpr int N = NN, E = EE, P = NN / EE;                                                                \
    static constexpr int R[] = {__VA_ARGS__};                                                                        \
    static constexpr int NST = sizeof(R) / sizeof(int);                                                              \
    __host__ __device__ static constexpr int ns(int s) { int q = 1; for (int i = 0; i < s; ++i) q *= R[i]; return q; } \
  };
DNSBOX_LPLAN(8, 4, 2, 4)
DNSBOX_LPLAN(12, 6, 2, 6)
DNSBOX_LPLAN(1024, 32, 16, 16, 4)
#undef DNSBOX_LPLAN
template <typename T, int N> struct XPlain {
  using PL = LPlan<N>;
  static constexpr int NT = 128;
  static constexpr size_t tw = ((size_t)vtw_size<PL>() * 2 * sizeof(T) + 15) / 16 * 16;
  static constexpr size_t line = (size_t)XTile<PL>::pitch * 2 * sizeof(T);
  static constexpr size_t smem(int threads) { return tw + threads / PL::P * line; }
  static constexpr int minb = sizeof(T) == 8 ? (PL::E > 16 ? 2 : 3) : (PL::E > 16 ? 3 : 5);
};

// C2R along x: half lines (nxh complex) -> real lines (N).  blockIdx.y = field.
// Against the row-tile kernels before it the 256^3 FP32 pair of transforms goes
// from 240 to 170 us.
template <typename T, int N>
__global__ void __launch_bounds__(XPlain<T, N>::NT, XPlain<T, N>::minb)
    k_xline_c2r(const __grid_constant__ XlineArgs<T> a) {
  using C = typename CT<T>::type;
  using SH = XPlain<T, N>;
  using PL = typename SH::PL;
  using EN = VEnds<PL>;
  using V = VC<T>;
  constexpr int E = PL::E, P = PL::P, H = E / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V *twt = reinterpret_cast<V *>(smem_raw);
  pdl_launch();
  vtw_fill<PL, V>(twt, a.tw, threadIdx.x, blockDim.x);
  __syncthreads();
  pdl_wait();
  const int g = threadIdx.x / P, p = threadIdx.x % P, lane = threadIdx.x & 31;
  V *s = reinterpret_cast<V *>(smem_raw + SH::tw + (size_t)g * SH::line);
  const long long la = 2 * ((long long)blockIdx.x * (blockDim.x / P) + g);
  const bool va = la < a.nlines, vb = la + 1 < a.nlines;
  const long long pitch = a.pitch ? a.pitch : a.nxh;
  const C *in = reinterpret_cast<const C *>(a.in[blockIdx.y]) + la * pitch;
  C x1[H + 1], x2[H + 1];
#pragma unroll
  for (int i = 0; i <= H; ++i) {
    x1[i] = ld_on(in + p + P * i, va && (i < H || p == 0));
    x2[i] = ld_on(in + pitch + p + P * i, vb && (i < H || p == 0));
  }
  if (p == 0) x1[0].y = x1[H].y = x2[0].y = x2[H].y = 0;   // a C2R drops these imaginary parts
  V z[E], x[E];
  pack_lines<E>(x1, x2, p, (lane & ~(P - 1)) | ((P - p) & (P - 1)), [&](int q, T r, T i) { z[EN::in_i(q)] = V{r, i}; });
  vfft<PL, true, XTile<PL>>(z, x, s, 0, p, twt, []() { __syncwarp(); });
  const T sc = T(a.scale);
  if (a.vmax) {
    T m = -INFINITY;
#pragma unroll
    for (int i = 0; i < E; ++i) {
      const T r = x[i].re * sc, q = x[i].im * sc;
      if (va) m = fmax(m, a.absval ? fabs(r) : r);
      if (vb) m = fmax(m, a.absval ? fabs(q) : q);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) {   // only a larger value needs the atomic
      const unsigned long long key = max_key_bits((unsigned long long)__double_as_longlong((double)m));
      if (key > __ldcg(a.vmax + blockIdx.y)) atomicMax(a.vmax + blockIdx.y, key);
    }
    return;
  }
  T *out = reinterpret_cast<T *>(a.out[blockIdx.y]) + la * N + p;
#pragma unroll
  for (int q = 0; q < E; ++q) {
    const V v = x[EN::out_i(q)];
    if (va) out[P * q] = v.re * sc;
    if (vb) out[N + P * q] = v.im * sc;
  }
}

// R2C along x: real lines -> half lines, two lines per transform.
template <typename T, int N>
__global__ void __launch_bounds__(XPlain<T, N>::NT, XPlain<T, N>::minb)
    k_xline_r2c(const __grid_constant__ XlineArgs<T> a) {
  using C = typename CT<T>::type;
  using SH = XPlain<T, N>;
  using PL = typename SH::PL;
  using EN = VEnds<PL>;
  using V = VC<T>;
  constexpr int E = PL::E, P = PL::P, H = E / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V *twt = reinterpret_cast<V *>(smem_raw);
  pdl_launch();
  vtw_fill<PL, V>(twt, a.tw, threadIdx.x, blockDim.x);
  __syncthreads();
  pdl_wait();
  const int g = threadIdx.x / P, p = threadIdx.x % P, lane = threadIdx.x & 31;
  V *s = reinterpret_cast<V *>(smem_raw + SH::tw + (size_t)g * SH::line);
  const long long la = 2 * ((long long)blockIdx.x * (blockDim.x / P) + g);
  const bool va = la < a.nlines, vb = la + 1 < a.nlines;
  const T *in = reinterpret_cast<const T *>(a.in[blockIdx.y]) + la * N + p;
  V z[E], x[E];
#pragma unroll
  for (int q = 0; q < E; ++q) {
    const T r = va ? in[P * q] : T(0), i = vb ? in[N + P * q] : T(0);
    z[EN::in_i(q)] = V{r, i};
  }
  vfft<PL, false, XTile<PL>>(z, x, s, 0, p, twt, []() { __syncwarp(); });
  const T sc = T(a.scale), hs = T(0.5);
  const long long pitch = a.pitch ? a.pitch : a.nxh;
  C *out = reinterpret_cast<C *>(a.out[blockIdx.y]) + la * pitch;
  const int mirror = (lane & ~(P - 1)) | ((P - p) & (P - 1));
#pragma unroll
  for (int i = 0; i <= H; ++i) {
    const V zk = x[EN::out_i(i)];
    T nr = zk.re, ni = zk.im;   // i = H: row N/2, its own mirror
    if (i < H) {
      const V b = x[EN::out_i(E - 1 - i)], b0 = x[EN::out_i((E - i) % E)];
      nr = __shfl_sync(0xffffffffu, p == 0 ? b0.re : b.re, mirror);
      ni = __shfl_sync(0xffffffffu, p == 0 ? b0.im : b.im, mirror);
    }
    if (i < H || p == 0) {
      if (va) out[p + P * i] = mkc<C>(hs * (zk.re + nr) * sc, hs * (zk.im - ni) * sc);
      if (vb) out[pitch + p + P * i] = mkc<C>(hs * (zk.im + ni) * sc, hs * (nr - zk.re) * sc);
    }
  }
}

// ------------------------------------------------------------- z finish
enum FinishMode : int {
  FIN_RHS = 0,         // out <- N(u)
  FIN_PRED = 1,        // out <- IF (uin + dt N); nold <- N if nold
  FIN_CORR = 2,        // state <- 0.5 (IF state + uin) + 0.5 dt N
  FIN_AB2 = 3,         // state(=uin) <- IF uin + c1 IF N + c2 E2 nold; nold <- N
};

template <typename T> struct FinishArgs {
  using C = typename CT<T>::type;
  const C *n3;             // 3 fields (kx, ky, kz): the nonlinear term after the forward z pass
  const C *uin;            // 3 fields, RHS input (forcing)
  C *out;                  // FIN_RHS / FIN_PRED output (3 fields)
  C *state;                // FIN_CORR state (3 fields)
  C *nold;                 // AB2 history (3 fields)
  const C *force;          // fixed spectral forcing added to N (3 fields) or null
  const StepState *st;     // per-box step state (blockIdx.y)
  const double *nu_box;    // per-box viscosity or null (use nu)
  double *partials;        // per-CTA (E, D) of the new state, or null; gridDim.x pairs per box
  long long nh;            // elements between components (all boxes of one component)
  long long bstride;       // elements between boxes
  int nx, ny, nz, nxh;
  double ax, ay, az;
  double nu, Q, Pin;
  double kcut2;            // largest k.k whose root is at most kCutOff (kcut2_of)
  double cutx, cuty, cutz, sph2;
  int bandlim, spherical, ab2_standard;
  double s;                // scalemodes
  AxisKeep kx, ky, kz;     // pruning: only kept (kz, ky) rows and kept kx modes are visited
  // layout of n3 when it is a padded workspace field: row pitch, elements
  // between components and between boxes; 0: the state's (nxh, nh, bstride)
  int n3_pitch, n3_nyq;    // n3_nyq: slot of the Nyquist column (0: nx / 2)
  long long n3_nh, n3_bstride;
  // a ky slab of a box split over ranks: row ky of this launch is ky0 + ky of
  // an axis of ny_k rows (0, 0: the box's own rows)
  int ky0, ny_k;
};

// The largest double whose square root is at most kcut (both roundings are
// IEEE), so that k.k <= kcut2_of(kcut) decides sqrt(k.k) <= kcut without a
// double-precision root per mode; -1 for a negative cut-off.
inline double kcut2_of(double kcut) {
  if (!(kcut >= 0.0)) return -1.0;
  double t = kcut * kcut;
  while (std::sqrt(t) > kcut) t = std::nextafter(t, 0.0);
  while (std::isfinite(t) && std::sqrt(std::nextafter(t, HUGE_VAL)) <= kcut) t = std::nextafter(t, HUGE_VAL);
  return t;
}

// Spectral finish after the forward z transform (the second half of one
// right-hand side's pass E): per mode the 2/3 mask, the pressure projection,
// band or fixed forcing and the integrating-factor update, one warp per
// (kz, ky) row of kx modes.  n3 holds the z-transformed nonlinear term.  Rows
// run over the kept kz and ky indices (every row when not pruning), by ky, last
// ky first (the order in which pass E1 wrote them: the newest still in L2),
// over the kept kx only (two rows per warp, the second in place of the next 32
// columns, measured 64 against 57 us at 256^3 FP32); the row's E and D sums (fixed lane order) go to
// partials[kz ny + ky] of the box, and the finalize reads the rows a pruned
// launch does not visit as zero.  Each lane batches the global operands of
// two modes before any store.  MODE (a FinishMode) is a template parameter so
// that only the operands of the update in use occupy registers.
// Resident blocks per SM asked of the register allocator: the FP32
// corrector and AB2 finishes (115-120 registers, two blocks) are held to
// three blocks.
template <typename T, int MODE> struct FinishMinB {
  static constexpr int v = (sizeof(T) == 4 && (MODE == 2 || MODE == 3)) ? 3 : 0;
};

template <typename T, int MODE>
__global__ void __launch_bounds__(256, FinishMinB<T, MODE>::v)
    k_finish_rows(const __grid_constant__ FinishArgs<T> a, int nrows) {
  using C = typename CT<T>::type;
  constexpr int CH = 2;
  pdl_launch();
  const int lane = threadIdx.x & 31;
  const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= nrows) return;   // whole warps: no block-level synchronisation below
  // rows by ky, last ky first (the order in which pass E1 wrote them, the
  // newest still in L2), kz within
  const int nkz = a.kz.count();
  const int oy = w / nkz;
  const int ky = a.ky.map(a.ky.count() - 1 - oy), kz = a.kz.map(w - oy * nkz);
  const int box = blockIdx.y;
  const long long rowbase = ((long long)kz * a.ny + ky) * a.nxh + (long long)box * a.bstride;
  const long long n3nh = a.n3_nh ? a.n3_nh : a.nh;
  const long long n3row = ((long long)kz * a.ny + ky) * (a.n3_pitch ? a.n3_pitch : a.nxh) +
                          (long long)box * (a.n3_bstride ? a.n3_bstride : a.bstride);
  const double kyr = k_full(a.ky0 + ky, a.ny_k ? a.ny_k : a.ny, a.ay);
  const double kzr = k_full(kz, a.nz, a.az);
  const bool rowcut = fabs(kyr) >= a.cuty || fabs(kzr) >= a.cutz;
  const bool need_u = a.bandlim || MODE != FIN_RHS;
  // kept kx, ascending per lane as in a full launch (so that the sums agree bit
  // for bit): lane, lane + 32, .. below lim, then in its lane the Nyquist column
  const int lim = a.kx.a ? a.kx.a : a.nxh, end = a.kx.a ? lim + 32 : lim;
  const int nql = a.kx.a ? (a.nx >> 1) & 31 : -1;
  auto column = [&](int s, bool &ok) {   // s = lane + 32 j
    ok = s < lim;
    if (s >= lim && s < lim + 32 && lane == nql) {
      ok = true;
      return a.nx >> 1;
    }
    return s;
  };
  const StepState *st = a.st + box;
  pdl_wait();
  const double nu = a.nu_box ? a.nu_box[box] : a.nu;
  const double dt = st->dt;
  const double fc = a.bandlim ? a.Pin / (2.0 * st->eband) : 0.0;
  double c1 = 0, c2 = 0, tau2 = 0;
  if (MODE == FIN_AB2) {
    const double tn = st->t, tm = st->t_prev;
    if (a.ab2_standard) {
      const double h = tn - tm;
      c1 = dt * (1.0 + dt / (2.0 * h));
      c2 = -dt * dt / (2.0 * h);
    } else {  // dnsbox.f90:150-161
      c1 = 0.5 * (tn + tn + dt - 2.0 * tm);
      c2 = 0.5 * (2.0 * tn - tn - dt - tm);
    }
    tau2 = dt + tn - tm;
  }
  double esum = 0.0, dsum = 0.0;
  for (int s0 = lane; s0 - lane < end; s0 += 32 * CH) {
    C nn[CH][3], uu[CH][3], ss[CH][3], no[CH][3];
    bool ok[CH];
#pragma unroll
    for (int h = 0; h < CH; ++h) {
      const int kx = column(s0 + 32 * h, ok[h]);
      const C *n3 = a.n3 + n3row + xslot(a.n3_nyq, kx, a.nx);
      const long long idx = rowbase + kx;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        nn[h][c] = ok[h] ? n3[c * n3nh] : mkc<C>(0, 0);
        uu[h][c] = ok[h] && need_u ? a.uin[c * a.nh + idx] : mkc<C>(0, 0);
        ss[h][c] = ok[h] && MODE == FIN_CORR ? a.state[c * a.nh + idx] : mkc<C>(0, 0);
        no[h][c] = ok[h] && MODE == FIN_AB2 ? a.nold[c * a.nh + idx] : mkc<C>(0, 0);
      }
    }
#pragma unroll
    for (int h = 0; h < CH; ++h) {
      if (!ok[h]) continue;
      bool unused;
      const int kx = column(s0 + 32 * h, unused);
      const long long idx = rowbase + kx;
      const double kxr = k_half(kx, a.nx, a.ax);
      const double wk = (kxr == 0.0) ? 0.5 : 1.0;   // state.f90:436-440
      const double k2 = kxr * kxr + kyr * kyr + kzr * kzr;
      const bool zero = (kxr == 0.0) && (kyr == 0.0) && (kzr == 0.0);
      const bool cut = (a.spherical && k2 >= a.sph2) || fabs(kxr) >= a.cutx || rowcut || zero;
      C Nc[3];
      if (cut) {
        Nc[0] = Nc[1] = Nc[2] = mkc<C>(0, 0);
      } else {
        // phat = -(i k . n) / (-(k.k))  (rhs.f90:101-106), in T: the masks
        // above and below are decided in FP64 (the same kept set in every
        // precision), the pointwise arithmetic in the state's precision
        const T kr[3] = {T(kxr), T(kyr), T(kzr)}, k2t = T(k2);
        const T knre = kr[0] * nn[h][0].x + kr[1] * nn[h][1].x + kr[2] * nn[h][2].x;
        const T knim = kr[0] * nn[h][0].y + kr[1] * nn[h][1].y + kr[2] * nn[h][2].y;
        const T pre = -knim / k2t, pim = knre / k2t;
        const bool forced = a.bandlim && k2 <= a.kcut2;
        const T fct = T(fc);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          T re = -nn[h][c].x + kr[c] * pim;
          T im = -nn[h][c].y - kr[c] * pre;
          if (forced) {
            re += fct * uu[h][c].x;
            im += fct * uu[h][c].y;
          }
          if (a.force) {
            const C q = a.force[c * a.nh + idx];
            re += q.x;
            im += q.y;
          }
          Nc[c] = mkc<C>(re, im);
        }
      }
      if (MODE == FIN_RHS) {
#pragma unroll
        for (int c = 0; c < 3; ++c) a.out[c * a.nh + idx] = Nc[c];
        continue;
      }
      const T IF = if_exp<T>((a.Q - nu * k2) * dt);
      const T tdt = T(dt);
      if (MODE == FIN_PRED) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const C u = uu[h][c];
          a.out[c * a.nh + idx] = mkc<C>((u.x + tdt * Nc[c].x) * IF, (u.y + tdt * Nc[c].y) * IF);
          if (a.nold) a.nold[c * a.nh + idx] = Nc[c];
        }
        continue;
      }
      C un[3];
      if (MODE == FIN_CORR) {
        const T hf = T(0.5), hdt = T(0.5 * dt);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const C u = ss[h][c], us = uu[h][c];
          un[c] = mkc<C>(hf * (IF * u.x + us.x) + hdt * Nc[c].x, hf * (IF * u.y + us.y) + hdt * Nc[c].y);
          a.state[c * a.nh + idx] = un[c];
        }
      } else {  // FIN_AB2
        const T e1c1 = T(c1) * IF;
        const T e2c2 = T(c2) * if_exp<T>((a.Q - nu * k2) * tau2);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const C u = uu[h][c], o = no[h][c];
          un[c] = mkc<C>(IF * u.x + e1c1 * Nc[c].x + e2c2 * o.x, IF * u.y + e1c1 * Nc[c].y + e2c2 * o.y);
          a.state[c * a.nh + idx] = un[c];
          a.nold[c * a.nh + idx] = Nc[c];
        }
      }
      double e2 = 0;
#pragma unroll
      for (int c = 0; c < 3; ++c) e2 += (double)un[c].x * un[c].x + (double)un[c].y * un[c].y;
      esum += wk * e2;
      dsum += 2.0 * wk * k2 * e2;
    }
  }
  if (a.partials) {
    esum = warp_sum(esum);
    dsum = warp_sum(dsum);
    if (lane == 0) {
      double *pp = a.partials + 2 * ((long long)box * a.nz * a.ny + (long long)kz * a.ny + ky);
      pp[0] = esum;
      pp[1] = dsum;
    }
  }
}


}  // namespace dnsbox
