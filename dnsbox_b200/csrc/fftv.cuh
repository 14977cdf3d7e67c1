// FFT stages on 16-byte elements held in registers: one complex double, or two
// single-precision complex values of the same position of two transforms
// (packed as a pair of real parts and a pair of imaginary parts).
//
// Single precision on sm_100a runs add, mul and fma on pairs of registers
// (.f32x2): the pipe does the same 128 lanes per clock and SM as the scalar
// form, at half the issue slots (measured: 63.9 pair instructions per clock
// against 125.6 scalar ones, and a pair instruction leaves the second slot to
// an integer instruction).  With the real parts of two transforms in one pair
// and the imaginary parts in another, every operation of an FFT is a pair
// operation -- the products with twiddles too, whose (re, im) form needs four
// scalar instructions and whose factors +-i cost no instruction -- and each
// twiddle, address and predicate serves two values.
//
// The algorithm is the Stockham scheme of fft.cuh.
#pragma once

#include "common.cuh"

namespace dnsbox {

// ------------------------------------------------------------- real "vectors"
struct f2 {
  unsigned long long u;
};
__device__ __forceinline__ f2 mkf2(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.u) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float f2_lo(f2 a) { return __uint_as_float((unsigned)a.u); }
__device__ __forceinline__ float f2_hi(f2 a) { return __uint_as_float((unsigned)(a.u >> 32)); }
__device__ __forceinline__ f2 vadd(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.u) : "l"(a.u), "l"(b.u));
  return r;
}
__device__ __forceinline__ f2 vsub(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.u) : "l"(a.u), "l"(b.u));
  return r;
}
__device__ __forceinline__ f2 vmul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.u) : "l"(a.u), "l"(b.u));
  return r;
}
// a b + c
__device__ __forceinline__ f2 vfma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.u) : "l"(a.u), "l"(b.u), "l"(c.u));
  return r;
}
__device__ __forceinline__ f2 vneg(f2 a) { return f2{a.u ^ 0x8000000080000000ull}; }
template <typename T> __device__ __forceinline__ T vadd(T a, T b) { return a + b; }
template <typename T> __device__ __forceinline__ T vsub(T a, T b) { return a - b; }
template <typename T> __device__ __forceinline__ T vmul(T a, T b) { return a * b; }
template <typename T> __device__ __forceinline__ T vfma(T a, T b, T c) { return a * b + c; }
template <typename T> __device__ __forceinline__ T vneg(T a) { return -a; }
// a constant in every part
template <typename R> struct VBc {
  __device__ static __forceinline__ R of(double c) { return R(c); }
};
template <> struct VBc<f2> {
  __device__ static __forceinline__ f2 of(double c) { return mkf2((float)c, (float)c); }
};

// A complex value of R parts (16 bytes for double and for a pair of floats).
template <typename R> struct alignas(2 * sizeof(R)) VC {
  R re, im;
};
// Element type and transforms per thread of a precision.
template <typename T> struct VecOf;
template <> struct VecOf<double> {
  using R = double;
  static constexpr int cols = 1;
};
template <> struct VecOf<float> {
  using R = f2;
  static constexpr int cols = 2;
};

// Two neighbouring single-precision complex values as they lie in memory.
// Converting them to pairs takes three moves for two values, so it is left to
// the first butterfly level, whose sums are scalar instructions that write
// the pairs, and back to the last level (XOp): twice the instructions of one
// level of each, no moves, and no register is waiting for its partner while
// the loads are in flight.
struct Raw2 {
  float4 q;
};
__device__ __forceinline__ VC<f2> vconv(Raw2 a) { return VC<f2>{mkf2(a.q.x, a.q.z), mkf2(a.q.y, a.q.w)}; }
template <typename R> __device__ __forceinline__ VC<R> vconv(VC<R> a) { return a; }

// ----------------------------------------------------------------- butterflies
// Elementary operations with operands of type A and a result of type O:
// a + b, a - b, a + i' b, a - i' b (i' = -i forward, i inverse) and the same
// with b times a real constant.
template <typename O, typename A> struct XOp;
template <typename R> struct XOp<VC<R>, VC<R>> {
  using V = VC<R>;
  static __device__ __forceinline__ V add(V a, V b) { return V{vadd(a.re, b.re), vadd(a.im, b.im)}; }
  static __device__ __forceinline__ V sub(V a, V b) { return V{vsub(a.re, b.re), vsub(a.im, b.im)}; }
  template <bool INV> static __device__ __forceinline__ V addi(V a, V b) {
    return INV ? V{vsub(a.re, b.im), vadd(a.im, b.re)} : V{vadd(a.re, b.im), vsub(a.im, b.re)};
  }
  static __device__ __forceinline__ V fma(V a, double c, V b) {
    const R k = VBc<R>::of(c);
    return V{vfma(b.re, k, a.re), vfma(b.im, k, a.im)};
  }
  template <bool INV> static __device__ __forceinline__ V fmai(V a, double c, V b) {
    const R p = VBc<R>::of(INV ? -c : c), n = VBc<R>::of(INV ? c : -c);
    return V{vfma(b.im, p, a.re), vfma(b.re, n, a.im)};
  }
};
template <> struct XOp<VC<f2>, Raw2> {
  using V = VC<f2>;
  static __device__ __forceinline__ V add(Raw2 a, Raw2 b) {
    return V{mkf2(a.q.x + b.q.x, a.q.z + b.q.z), mkf2(a.q.y + b.q.y, a.q.w + b.q.w)};
  }
  static __device__ __forceinline__ V sub(Raw2 a, Raw2 b) {
    return V{mkf2(a.q.x - b.q.x, a.q.z - b.q.z), mkf2(a.q.y - b.q.y, a.q.w - b.q.w)};
  }
};
template <> struct XOp<Raw2, VC<f2>> {
  using V = VC<f2>;
  static __device__ __forceinline__ Raw2 mk(float a, float b, float c, float d) { return Raw2{make_float4(a, b, c, d)}; }
  static __device__ __forceinline__ Raw2 add(V a, V b) {
    return mk(f2_lo(a.re) + f2_lo(b.re), f2_lo(a.im) + f2_lo(b.im), f2_hi(a.re) + f2_hi(b.re), f2_hi(a.im) + f2_hi(b.im));
  }
  static __device__ __forceinline__ Raw2 sub(V a, V b) {
    return mk(f2_lo(a.re) - f2_lo(b.re), f2_lo(a.im) - f2_lo(b.im), f2_hi(a.re) - f2_hi(b.re), f2_hi(a.im) - f2_hi(b.im));
  }
  template <bool INV> static __device__ __forceinline__ Raw2 addi(V a, V b) {
    if (INV)
      return mk(f2_lo(a.re) - f2_lo(b.im), f2_lo(a.im) + f2_lo(b.re), f2_hi(a.re) - f2_hi(b.im), f2_hi(a.im) + f2_hi(b.re));
    return mk(f2_lo(a.re) + f2_lo(b.im), f2_lo(a.im) - f2_lo(b.re), f2_hi(a.re) + f2_hi(b.im), f2_hi(a.im) - f2_hi(b.re));
  }
  static __device__ __forceinline__ Raw2 fma(V a, double c, V b) {
    const float k = (float)c;
    return mk(fmaf(f2_lo(b.re), k, f2_lo(a.re)), fmaf(f2_lo(b.im), k, f2_lo(a.im)), fmaf(f2_hi(b.re), k, f2_hi(a.re)),
              fmaf(f2_hi(b.im), k, f2_hi(a.im)));
  }
  template <bool INV> static __device__ __forceinline__ Raw2 fmai(V a, double c, V b) {
    const float p = INV ? -(float)c : (float)c;
    return mk(fmaf(f2_lo(b.im), p, f2_lo(a.re)), fmaf(f2_lo(b.re), -p, f2_lo(a.im)), fmaf(f2_hi(b.im), p, f2_hi(a.re)),
              fmaf(f2_hi(b.re), -p, f2_hi(a.im)));
  }
};
template <typename A> struct VOf;
template <typename R> struct VOf<VC<R>> { using type = VC<R>; };
template <> struct VOf<Raw2> { using type = VC<f2>; };

template <bool INV, typename O, typename A> __device__ __forceinline__ void vdft2(const A &a, const A &b, O &x, O &y) {
  const A s = a, t = b;
  x = XOp<O, A>::add(s, t);
  y = XOp<O, A>::sub(s, t);
}

template <bool INV, typename O, typename A>
__device__ __forceinline__ void vdft3(const A &a0, const A &a1, const A &a2, O &x0, O &x1, O &x2) {
  using V = typename VOf<A>::type;
  const V t = XOp<V, A>::add(a1, a2), d = XOp<V, A>::sub(a1, a2), z = vconv(a0);
  const V m = XOp<V, V>::fma(z, -0.5, t);
  x0 = XOp<O, V>::add(z, t);
  x1 = XOp<O, V>::template fmai<INV>(m, 0.86602540378443864676372317075294, d);
  x2 = XOp<O, V>::template fmai<INV>(m, -0.86602540378443864676372317075294, d);
}

template <bool INV, typename O, typename A>
__device__ __forceinline__ void vdft4(const A &a0, const A &a1, const A &a2, const A &a3, O &x0, O &x1, O &x2, O &x3) {
  using V = typename VOf<A>::type;
  const V t0 = XOp<V, A>::add(a0, a2), t1 = XOp<V, A>::sub(a0, a2), t2 = XOp<V, A>::add(a1, a3), d = XOp<V, A>::sub(a1, a3);
  x0 = XOp<O, V>::add(t0, t2);
  x2 = XOp<O, V>::sub(t0, t2);
  x1 = XOp<O, V>::template addi<INV>(t1, d);
  x3 = XOp<O, V>::template addi<!INV>(t1, d);
}

// a (c - i s) forward, a (c + i s) inverse, for constants c, s
template <bool INV, typename V> __device__ __forceinline__ V vrot(V a, double c, double s) {
  using R = decltype(V{}.re);
  const R cc = VBc<R>::of(c), sp = VBc<R>::of(INV ? -s : s), sn = VBc<R>::of(INV ? s : -s);
  V r;
  r.re = vfma(a.im, sp, vmul(a.re, cc));
  r.im = vfma(a.re, sn, vmul(a.im, cc));
  return r;
}

template <bool INV, typename O, typename A> __device__ __forceinline__ void vdft8(const A *v, O *x) {
  using V = typename VOf<A>::type;
  using R = decltype(V{}.re);
  constexpr double r = 0.70710678118654752440084436210485;
  V e[4], o[4];
  vdft4<INV>(v[0], v[2], v[4], v[6], e[0], e[1], e[2], e[3]);
  vdft4<INV>(v[1], v[3], v[5], v[7], o[0], o[1], o[2], o[3]);
  x[0] = XOp<O, V>::add(e[0], o[0]);
  x[4] = XOp<O, V>::sub(e[0], o[0]);
  // o W8^1 = r (o + i' o), o W8^3 = r (i' o - o) with i' = -+ i; W8^2 = i'
  const V w1 = XOp<V, V>::template addi<INV>(o[1], o[1]), w3 = XOp<V, V>::template addi<!INV>(o[3], o[3]);
  x[1] = XOp<O, V>::fma(e[1], r, w1);
  x[5] = XOp<O, V>::fma(e[1], -r, w1);
  x[2] = XOp<O, V>::template addi<INV>(e[2], o[2]);
  x[6] = XOp<O, V>::template addi<!INV>(e[2], o[2]);
  x[3] = XOp<O, V>::fma(e[3], -r, w3);
  x[7] = XOp<O, V>::fma(e[3], r, w3);
}

// 16 points as 4 x 4: X[k1 + 4 k2] = sum_n2 W4^(n2 k2) W16^(n2 k1) sum_n1 a[4 n1 + n2] W4^(n1 k1)
template <bool INV, typename O, typename A> __device__ __forceinline__ void vdft16(const A *v, O *x) {
  using V = typename VOf<A>::type;
  constexpr double c1 = 0.92387953251128675612818318939679, s1 = 0.38268343236508977172845998403040;
  constexpr double r = 0.70710678118654752440084436210485;
  V b[16];   // b[n2 + 4 k1]
#pragma unroll
  for (int n2 = 0; n2 < 4; ++n2)
    vdft4<INV>(v[n2], v[n2 + 4], v[n2 + 8], v[n2 + 12], b[n2], b[n2 + 4], b[n2 + 8], b[n2 + 12]);
  // twiddles W16^(n2 k1)
  b[5] = vrot<INV>(b[5], c1, s1);
  b[9] = vrot<INV>(b[9], r, r);
  b[13] = vrot<INV>(b[13], s1, c1);
  b[6] = vrot<INV>(b[6], r, r);
  b[14] = vrot<INV>(b[14], -r, r);
  b[7] = vrot<INV>(b[7], s1, c1);
  b[11] = vrot<INV>(b[11], -r, r);
  b[15] = vrot<INV>(b[15], -c1, -s1);
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) {
    if (k1 == 2) {   // b[10] carries W16^4 = -+ i: folded into its sums
      const V t0 = XOp<V, V>::template addi<INV>(b[8], b[10]), t1 = XOp<V, V>::template addi<!INV>(b[8], b[10]);
      const V t2 = XOp<V, V>::add(b[9], b[11]), d = XOp<V, V>::sub(b[9], b[11]);
      x[2] = XOp<O, V>::add(t0, t2);
      x[10] = XOp<O, V>::sub(t0, t2);
      x[6] = XOp<O, V>::template addi<INV>(t1, d);
      x[14] = XOp<O, V>::template addi<!INV>(t1, d);
    } else {
      vdft4<INV>(b[4 * k1], b[1 + 4 * k1], b[2 + 4 * k1], b[3 + 4 * k1], x[k1], x[k1 + 4], x[k1 + 8], x[k1 + 12]);
    }
  }
}

// 6 = 2 x 3 and 12 = 3 x 4 points by the prime-factor maps (no twiddles):
// N = N1 N2, n = N2 n1 + N1 n2, k = N2 (1/N2 mod N1) k1 + N1 (1/N1 mod N2) k2 (mod N)
template <bool INV, typename O, typename A> __device__ __forceinline__ void vdft6(const A *v, O *x) {
  using V = typename VOf<A>::type;
  V a[2][3];
#pragma unroll
  for (int n1 = 0; n1 < 2; ++n1)
    vdft3<INV>(v[3 * n1], v[(3 * n1 + 2) % 6], v[(3 * n1 + 4) % 6], a[n1][0], a[n1][1], a[n1][2]);
#pragma unroll
  for (int k2 = 0; k2 < 3; ++k2) vdft2<INV>(a[0][k2], a[1][k2], x[(4 * k2) % 6], x[(3 + 4 * k2) % 6]);
}
template <bool INV, typename O, typename A> __device__ __forceinline__ void vdft12(const A *v, O *x) {
  using V = typename VOf<A>::type;
  V a[3][4];
#pragma unroll
  for (int n1 = 0; n1 < 3; ++n1)
    vdft4<INV>(v[4 * n1], v[(4 * n1 + 3) % 12], v[(4 * n1 + 6) % 12], v[(4 * n1 + 9) % 12], a[n1][0], a[n1][1], a[n1][2],
               a[n1][3]);
#pragma unroll
  for (int k2 = 0; k2 < 4; ++k2)
    vdft3<INV>(a[0][k2], a[1][k2], a[2][k2], x[(9 * k2) % 12], x[(4 + 9 * k2) % 12], x[(8 + 9 * k2) % 12]);
}

// R-point DFT of v into x (distinct arrays)
template <int R, bool INV, typename O, typename A> __device__ __forceinline__ void vdft(const A *v, O *x) {
  if constexpr (R == 2) vdft2<INV>(v[0], v[1], x[0], x[1]);
  else if constexpr (R == 3) vdft3<INV>(v[0], v[1], v[2], x[0], x[1], x[2]);
  else if constexpr (R == 4) vdft4<INV>(v[0], v[1], v[2], v[3], x[0], x[1], x[2], x[3]);
  else if constexpr (R == 6) vdft6<INV>(v, x);
  else if constexpr (R == 8) vdft8<INV>(v, x);
  else if constexpr (R == 12) vdft12<INV>(v, x);
  else if constexpr (R == 16) vdft16<INV>(v, x);
  else static_assert(R == 2, "unsupported radix");
}

// ----------------------------------------------------------------------- plans
// E values per thread, P = N / E threads per transform, radices of the stages
// (the product of the first s is the sub-transform length of stage s).  A
// thread's rows are p, p + P, p + 2 P, ... at both ends of the transform,
// whatever the radices (in_q and out_q give the order in which its registers
// hold them).  12 values as radix 12, 4 x 4 x 6 and 4 x 4 x 12: one or two
// shared-memory exchanges where the radix-2/3/4/8 plans of fft.cuh need two
// or three, in half the registers at 24, 96 and 192.
template <int N> struct VPlan;
#define DNSBOX_VPLAN(NN, EE, ...)                                                                                    \
  template <> struct VPlan<NN> {                                                                                     \
    static constexpr int N = NN, E = EE, P = NN / EE;                                                                \
    static constexpr int R[] = {__VA_ARGS__};                                                                        \
    static constexpr int NST = sizeof(R) / sizeof(int);                                                              \
    __host__ __device__ static constexpr int ns(int s) { int q = 1; for (int i = 0; i < s; ++i) q *= R[i]; return q; } \
  };
DNSBOX_VPLAN(8, 8, 8)
DNSBOX_VPLAN(12, 12, 12)
DNSBOX_VPLAN(16, 4, 4, 4)
DNSBOX_VPLAN(24, 12, 4, 6)
DNSBOX_VPLAN(32, 8, 8, 4)
DNSBOX_VPLAN(48, 12, 12, 4)
DNSBOX_VPLAN(64, 8, 8, 8)
DNSBOX_VPLAN(96, 12, 4, 4, 6)
DNSBOX_VPLAN(128, 16, 16, 8)
DNSBOX_VPLAN(192, 12, 4, 4, 12)
DNSBOX_VPLAN(256, 16, 16, 16)
DNSBOX_VPLAN(512, 16, 16, 8, 4)
DNSBOX_VPLAN(1024, 16, 16, 16, 4)
#undef DNSBOX_VPLAN

// Two-stage plans N = R0 R1 with one butterfly a thread in each stage: R1
// threads of R0 values, rows p + R1 q, then R0 threads of R1 values, rows p +
// R0 q.  The x lines of 96 and 192 points, whose plans of equal shares need two
// exchanges, run their inverse transforms this way and their forward ones the
// other way round.
template <int N> struct SplitPlan {
  static constexpr bool on = false;
};
template <> struct SplitPlan<96> {
  static constexpr bool on = true;
  static constexpr int R0 = 12, R1 = 8, pitch = 108;
};
template <> struct SplitPlan<192> {
  static constexpr bool on = true;
  static constexpr int R0 = 12, R1 = 16, pitch = 220;
};

// Plans of the x lines, at most 32 threads per line (a warp synchronises
// itself): 16 values in single precision, 8 in double precision (three
// sequences of a line are held at once) where the length allows it.
template <typename T, int N> struct XPlan : VPlan<N> {};
#define DNSBOX_XPLAN(TT, NN, EE, ...)                                                                                \
  template <> struct XPlan<TT, NN> {                                                                                 \
    static constexpr int N = NN, E = EE, P = NN / EE;                                                                \
    static constexpr int R[] = {__VA_ARGS__};                                                                        \
    static constexpr int NST = sizeof(R) / sizeof(int);                                                              \
    __host__ __device__ static constexpr int ns(int s) { int q = 1; for (int i = 0; i < s; ++i) q *= R[i]; return q; } \
  };
DNSBOX_XPLAN(double, 128, 8, 8, 4, 4)
DNSBOX_XPLAN(double, 256, 8, 8, 8, 4)
#undef DNSBOX_XPLAN

// Register i of a thread holds row p + P in_q(i) before and p + P out_q(i)
// after the transform; in_i / out_i are the inverse maps.
template <class PL> struct VEnds {
  static constexpr int E = PL::E, R0 = PL::R[0], RL = PL::R[PL::NST - 1];
  __host__ __device__ static constexpr int in_q(int i) { return i / R0 + (i % R0) * (E / R0); }
  __host__ __device__ static constexpr int out_q(int i) { return i / RL + (i % RL) * (E / RL); }
  __host__ __device__ static constexpr int in_i(int q) { return (q % (E / R0)) * R0 + q / (E / R0); }
  __host__ __device__ static constexpr int out_i(int q) { return (q % (E / RL)) * RL + q / (E / RL); }
};

// Per-stage twiddle tables [r - 1][j] in shared memory.
template <class PL, int S> __host__ __device__ constexpr int vtw_off() {
  int o = 0;
  for (int t = 1; t < S; ++t) o += (PL::R[t] - 1) * PL::ns(t);
  return o;
}
template <class PL> __host__ __device__ constexpr int vtw_size() { return vtw_off<PL, PL::NST>(); }

template <typename V> struct VtwOf;
template <> struct VtwOf<VC<double>> {
  __device__ static __forceinline__ VC<double> of(double2 w) { return VC<double>{w.x, w.y}; }
};
template <> struct VtwOf<VC<float>> {
  __device__ static __forceinline__ VC<float> of(float2 w) { return VC<float>{w.x, w.y}; }
};
template <> struct VtwOf<VC<f2>> {
  __device__ static __forceinline__ VC<f2> of(float2 w) { return VC<f2>{mkf2(w.x, w.x), mkf2(w.y, w.y)}; }
};
// Entry i of the tables, from the N-point table exp(-2 pi i k / N).
template <class PL, int S = 1, typename C> __device__ __forceinline__ C vtw_entry(const C *__restrict__ tw, int i) {
  static_assert(S < PL::NST, "a plan of one stage has no twiddles");
  constexpr int NS = PL::ns(S), R = PL::R[S], TS = PL::N / (NS * R);
  if constexpr (S + 1 < PL::NST) {
    if (i >= (R - 1) * NS) return vtw_entry<PL, S + 1>(tw, i - (R - 1) * NS);
  }
  return __ldg(tw + (1 + i / NS) * (i % NS) * TS);
}
// All tables, by all threads of the block.
template <class PL, typename V, typename C>
__device__ __forceinline__ void vtw_fill(V *t, const C *__restrict__ tw, int tid, int nthreads) {
  if constexpr (PL::NST > 1)
    for (int i = tid; i < vtw_size<PL>(); i += nthreads) t[i] = VtwOf<V>::of(vtw_entry<PL>(tw, i));
}

template <bool INV, typename V> __device__ __forceinline__ V vtwmul(V a, V w) {
  using R = decltype(V{}.re);
  const R ni = vneg(w.im);
  V r;   // forward a w, inverse a conj(w)
  r.re = vfma(a.im, INV ? w.im : ni, vmul(a.re, w.re));
  r.im = vfma(a.re, INV ? ni : w.im, vmul(a.im, w.re));
  return r;
}

// a pair with one twiddle for both transforms
template <bool INV> __device__ __forceinline__ VC<f2> vtwmul(VC<f2> a, VC<float> w) {
  return vtwmul<INV>(a, VC<f2>{mkf2(w.re, w.re), mkf2(w.im, w.im)});
}

// ---------------------------------------------------------------------- stages
// Whole transform of the values v (first-stage order) into x (last-stage
// order), exchanged through the tile s; AD::at(row, col) gives an element's
// place.  sync() separates the phases (a block or a warp barrier).  The tile
// may be reused after the caller's next barrier.
template <class PL, bool INV, class AD, int S, typename O, typename V, typename W, typename SYNC>
__device__ __forceinline__ void vfft_stage(O *x, V *s, int col, int p, const W *tw, SYNC sync) {
  constexpr int R = PL::R[S], NS = PL::ns(S), E = PL::E, M = E / R, P = PL::P, NB = PL::N / R;
  constexpr bool last = S + 1 == PL::NST;
  V y[last ? 1 : E];
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const int b = p + m * P;
    V v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = s[AD::at(b + r * NB, col)];
    const int j = b % NS;
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = vtwmul<INV>(v[r], tw[vtw_off<PL, S>() + (r - 1) * NS + j]);
    if constexpr (last) vdft<R, INV>(v, x + m * R);
    else vdft<R, INV>(v, y + m * R);
  }
  if constexpr (!last) {
    sync();
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int b = p + m * P, o = (b / NS) * NS * R + b % NS;
#pragma unroll
      for (int r = 0; r < R; ++r) s[AD::at(o + r * NS, col)] = y[m * R + r];
    }
    sync();
    vfft_stage<PL, INV, AD, S + 1>(x, s, col, p, tw, sync);
  }
}
template <class PL, bool INV, class AD, typename O, typename A, typename V, typename W, typename SYNC>
__device__ __forceinline__ void vfft(const A *v, O *x, V *s, int col, int p, const W *tw, SYNC sync) {
  constexpr int R = PL::R[0], M = PL::E / R, P = PL::P;
  if constexpr (PL::NST == 1) {
    vdft<R, INV>(v, x);
  } else {
    V y[PL::E];
#pragma unroll
    for (int m = 0; m < M; ++m) vdft<R, INV>(v + m * R, y + m * R);
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int r = 0; r < R; ++r) s[AD::at((p + m * P) * R + r, col)] = y[m * R + r];
    sync();
    vfft_stage<PL, INV, AD, 1>(x, s, col, p, tw, sync);
  }
}

}  // namespace dnsbox
