// fft_lane.cuh -- FFT butterflies on groups of transforms, one group per
// 16-byte shared-memory element.
//
// An element CV<T> holds one complex value of W transforms: W = 2 for float
// (two transforms side by side in the two halves of 64-bit registers, added
// and multiplied with the f32x2 instructions), W = 1 for double.  One FP32
// thread therefore carries two transforms through the index arithmetic, the
// twiddle reads and the 16-byte shared-memory accesses of one, and issues
// one instruction for two FP32 operations; the FP64 kernels run the same
// code on single transforms.  (Measured on B200: f32x2 has the FP32 lanes'
// rate, 128 per clock and SM, at half the issue slots, and a negated
// operand written half by half costs no instruction.)
//
// Stages are those of fft_smem.cuh: DIF forward with the twiddles after the
// butterfly, DIT inverse with the conjugate twiddles before it, the slot
// order of ct_radix.
#pragma once
#include "fft_smem.cuh"

#include <type_traits>

namespace fg {

#ifdef FG_HOST_EMU
struct F2 {
  float x, y;
};
inline F2 f2_make(float x, float y) { return F2{x, y}; }
inline float f2_lo(F2 a) { return a.x; }
inline float f2_hi(F2 a) { return a.y; }
inline F2 vadd(F2 a, F2 b) { return F2{a.x + b.x, a.y + b.y}; }
inline F2 vsub(F2 a, F2 b) { return F2{a.x - b.x, a.y - b.y}; }
inline F2 vmul(F2 a, F2 b) { return F2{a.x * b.x, a.y * b.y}; }
inline F2 vfma(F2 a, F2 b, F2 c) { return F2{fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)}; }
inline double fma_rn(double a, double b, double c) { return fma(a, b, c); }
#else
struct F2 {
  unsigned long long b;
};
__device__ __forceinline__ F2 f2_make(float x, float y) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.b) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float f2_lo(F2 a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.b));
  return x;
}
__device__ __forceinline__ float f2_hi(F2 a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.b));
  return y;
}
__device__ __forceinline__ F2 vadd(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.b) : "l"(a.b), "l"(b.b));
  return r;
}
__device__ __forceinline__ F2 vsub(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.b) : "l"(a.b), "l"(b.b));
  return r;
}
__device__ __forceinline__ F2 vmul(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.b) : "l"(a.b), "l"(b.b));
  return r;
}
__device__ __forceinline__ F2 vfma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.b) : "l"(a.b), "l"(b.b), "l"(c.b));
  return r;
}
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
#endif
__device__ __forceinline__ F2 vneg(F2 a) { return f2_make(-f2_lo(a), -f2_hi(a)); }
__device__ __forceinline__ double vadd(double a, double b) { return a + b; }
__device__ __forceinline__ double vsub(double a, double b) { return a - b; }
__device__ __forceinline__ double vmul(double a, double b) { return a * b; }
__device__ __forceinline__ double vfma(double a, double b, double c) { return fma_rn(a, b, c); }
__device__ __forceinline__ double vneg(double a) { return -a; }

template <typename T> struct LaneOf;
template <> struct LaneOf<float> { using V = F2; };
template <> struct LaneOf<double> { using V = double; };
template <typename T> using lane_t = typename LaneOf<T>::V;
// transforms per element
template <typename T> constexpr int kLanes = 16 / (2 * (int)sizeof(T));

// lane l of a value; a value from its lanes (double: the first), the same
// value in every lane
template <int L> __device__ __forceinline__ float vget(F2 a) { return L == 0 ? f2_lo(a) : f2_hi(a); }
template <int L> __device__ __forceinline__ double vget(double a) { return a; }
__device__ __forceinline__ F2 vpack(float a, float b) { return f2_make(a, b); }
__device__ __forceinline__ double vpack(double a, double) { return a; }
__device__ __forceinline__ F2 vall(float a) { return f2_make(a, a); }
__device__ __forceinline__ double vall(double a) { return a; }

template <typename T>
struct CV {
  lane_t<T> re, im;
};

// 16-byte shared-memory (and global) accesses of an element
#ifdef FG_HOST_EMU
template <typename T> inline CV<T> cv_ld(const CV<T>* p) { return *p; }
template <typename T> inline void cv_st(CV<T>* p, const CV<T>& v) { *p = v; }
template <typename T> inline CV<T> cv_stream(const CV<T>* p) { return *p; }
#else
__device__ __forceinline__ CV<float> cv_ld(const CV<float>* p) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  CV<float> r;
  r.re.b = v.x;
  r.im.b = v.y;
  return r;
}
__device__ __forceinline__ CV<double> cv_ld(const CV<double>* p) {
  const double2 v = *reinterpret_cast<const double2*>(p);
  CV<double> r;
  r.re = v.x;
  r.im = v.y;
  return r;
}
__device__ __forceinline__ void cv_st(CV<float>* p, const CV<float>& v) {
  *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(v.re.b, v.im.b);
}
__device__ __forceinline__ void cv_st(CV<double>* p, const CV<double>& v) {
  *reinterpret_cast<double2*>(p) = make_double2(v.re, v.im);
}
// a read-once global element that should not displace cached tables
__device__ __forceinline__ CV<float> cv_stream(const CV<float>* p) {
  CV<float> r;
  asm("ld.global.nc.L1::no_allocate.v2.b64 {%0, %1}, [%2];" : "=l"(r.re.b), "=l"(r.im.b) : "l"(p));
  return r;
}
__device__ __forceinline__ CV<double> cv_stream(const CV<double>* p) {
  CV<double> r;
  asm("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(r.re), "=d"(r.im) : "l"(p));
  return r;
}
#endif

// W neighbouring complex values of a row <-> one element
__device__ __forceinline__ CV<float> cv_of(const float4& v) { return CV<float>{vpack(v.x, v.z), vpack(v.y, v.w)}; }
__device__ __forceinline__ CV<double> cv_of(const double2& v) { return CV<double>{v.x, v.y}; }
__device__ __forceinline__ void cv_row(float4* p, const CV<float>& v) {
  float4 r;
  r.x = vget<0>(v.re);
  r.y = vget<0>(v.im);
  r.z = vget<1>(v.re);
  r.w = vget<1>(v.im);
  *p = r;
}
__device__ __forceinline__ void cv_row(double2* p, const CV<double>& v) { *p = make_double2(v.re, v.im); }
template <typename T> struct RowVec;  // 16 bytes of a spectrum row
template <> struct RowVec<float> { using type = float4; };
template <> struct RowVec<double> { using type = double2; };
template <typename T> using rowvec = typename RowVec<T>::type;

template <typename T> __device__ __forceinline__ CV<T> cvadd(const CV<T>& a, const CV<T>& b) {
  return CV<T>{vadd(a.re, b.re), vadd(a.im, b.im)};
}
template <typename T> __device__ __forceinline__ CV<T> cvsub(const CV<T>& a, const CV<T>& b) {
  return CV<T>{vsub(a.re, b.re), vsub(a.im, b.im)};
}
// times -i (forward) or +i (inverse)
template <typename T, bool INV> __device__ __forceinline__ CV<T> cvmul_mi(const CV<T>& a) {
  return INV ? CV<T>{vneg(a.im), a.re} : CV<T>{a.im, vneg(a.re)};
}
// times the twiddle w in every lane (INV: its conjugate).  The table entry is
// one complex number: using a 32-bit register for both halves of an f32x2
// operand costs no instruction.
template <typename T, bool INV> __device__ __forceinline__ CV<T> cvtw(const CV<T>& a, const cplx<T>& w) {
  const lane_t<T> c = vall(w.x), s = vall(w.y);
  if (INV) return CV<T>{vfma(a.re, c, vmul(a.im, s)), vfma(a.im, c, vneg(vmul(a.re, s)))};
  return CV<T>{vfma(a.re, c, vneg(vmul(a.im, s))), vfma(a.im, c, vmul(a.re, s))};
}

template <typename T, int R, bool INV> struct DftV;

template <typename T, bool INV> struct DftV<T, 2, INV> {
  static __device__ __forceinline__ void run(CV<T>* v) {
    const CV<T> a = v[0], b = v[1];
    v[0] = cvadd(a, b);
    v[1] = cvsub(a, b);
  }
};

template <typename T, bool INV> struct DftV<T, 3, INV> {
  static __device__ __forceinline__ void run(CV<T>* v) {
    const lane_t<T> mh = vall((T)-0.5), s3 = vall((T)0.86602540378443864676);  // sin(2 pi / 3)
    const CV<T> t1 = cvadd(v[1], v[2]), t2 = cvsub(v[1], v[2]);
    const CV<T> m{vfma(t1.re, mh, v[0].re), vfma(t1.im, mh, v[0].im)};
    v[0] = cvadd(v[0], t1);
    // y1 = m -+ i s3 t2, y2 = m +- i s3 t2
    const CV<T> p{vfma(t2.im, s3, m.re), vfma(vneg(t2.re), s3, m.im)}, n{vfma(vneg(t2.im), s3, m.re), vfma(t2.re, s3, m.im)};
    v[1] = INV ? n : p;
    v[2] = INV ? p : n;
  }
};

template <typename T, bool INV> struct DftV<T, 4, INV> {
  static __device__ __forceinline__ void run(CV<T>* v) {
    const CV<T> t0 = cvadd(v[0], v[2]), t1 = cvsub(v[0], v[2]), t2 = cvadd(v[1], v[3]), t3 = cvsub(v[1], v[3]);
    v[0] = cvadd(t0, t2);
    v[2] = cvsub(t0, t2);
    const CV<T> p{vadd(t1.re, t3.im), vsub(t1.im, t3.re)}, n{vsub(t1.re, t3.im), vadd(t1.im, t3.re)};
    v[1] = INV ? n : p;
    v[3] = INV ? p : n;
  }
};

template <typename T, bool INV> struct DftV<T, 1, INV> {
  static __device__ __forceinline__ void run(CV<T>*) {}
};

template <typename T, bool INV> struct DftV<T, 5, INV> {
  static __device__ __forceinline__ void run(CV<T>* v) {
    const lane_t<T> c1 = vall((T)0.30901699437494742410), c2 = vall((T)-0.80901699437494742410);
    const lane_t<T> s1 = vall((T)0.95105651629515357212), s2 = vall((T)0.58778525229247312917);
    const CV<T> t1 = cvadd(v[1], v[4]), t2 = cvadd(v[2], v[3]), t3 = cvsub(v[1], v[4]), t4 = cvsub(v[2], v[3]);
    const CV<T> a1{vfma(t1.re, c1, vfma(t2.re, c2, v[0].re)), vfma(t1.im, c1, vfma(t2.im, c2, v[0].im))};
    const CV<T> a2{vfma(t1.re, c2, vfma(t2.re, c1, v[0].re)), vfma(t1.im, c2, vfma(t2.im, c1, v[0].im))};
    const CV<T> b1{vfma(t3.re, s1, vmul(t4.re, s2)), vfma(t3.im, s1, vmul(t4.im, s2))};
    const CV<T> b2{vfma(t3.re, s2, vneg(vmul(t4.re, s1))), vfma(t3.im, s2, vneg(vmul(t4.im, s1)))};
    v[0] = cvadd(v[0], cvadd(t1, t2));
    // y = a -+ i b
    const CV<T> p1{vadd(a1.re, b1.im), vsub(a1.im, b1.re)}, n1{vsub(a1.re, b1.im), vadd(a1.im, b1.re)};
    const CV<T> p2{vadd(a2.re, b2.im), vsub(a2.im, b2.re)}, n2{vsub(a2.re, b2.im), vadd(a2.im, b2.re)};
    v[1] = INV ? n1 : p1;
    v[4] = INV ? p1 : n1;
    v[2] = INV ? n2 : p2;
    v[3] = INV ? p2 : n2;
  }
};

// 6 = 2 x 3 by the Chinese remainder map: no twiddles.
template <typename T, bool INV> struct DftV<T, 6, INV> {
  static __device__ __forceinline__ void run(CV<T>* v) {
    CV<T> s[3] = {cvadd(v[0], v[3]), cvadd(v[2], v[5]), cvadd(v[4], v[1])};
    CV<T> d[3] = {cvsub(v[0], v[3]), cvsub(v[2], v[5]), cvsub(v[4], v[1])};
    DftV<T, 3, INV>::run(s);
    DftV<T, 3, INV>::run(d);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      v[(4 * k) % 6] = s[k];
      v[(3 + 4 * k) % 6] = d[k];
    }
  }
};

template <typename T, bool INV> struct DftV<T, 8, INV> {
  static __device__ __forceinline__ void run(CV<T>* v) {
    const lane_t<T> h = vall((T)0.70710678118654752440);  // 1/sqrt(2)
    CV<T> a[4], b[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      a[q] = cvadd(v[q], v[q + 4]);
      b[q] = cvsub(v[q], v[q + 4]);
    }
    const lane_t<T> p1 = vadd(b[1].re, b[1].im), m1 = vsub(b[1].im, b[1].re);
    const lane_t<T> p3 = vadd(b[3].re, b[3].im), m3 = vsub(b[3].im, b[3].re);
    // b[q] *= w8^q
    b[1] = INV ? CV<T>{vneg(vmul(m1, h)), vmul(p1, h)} : CV<T>{vmul(p1, h), vmul(m1, h)};
    b[2] = cvmul_mi<T, INV>(b[2]);
    b[3] = INV ? CV<T>{vneg(vmul(p3, h)), vneg(vmul(m3, h))} : CV<T>{vmul(m3, h), vneg(vmul(p3, h))};
    DftV<T, 4, INV>::run(a);
    DftV<T, 4, INV>::run(b);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      v[2 * s] = a[s];
      v[2 * s + 1] = b[s];
    }
  }
};

template <typename T, bool INV> struct DftV<T, 16, INV> {
  // 4 x 4 as Dft<T, 16, INV>
  static __device__ __forceinline__ CV<T> tw(const CV<T>& a, T cr, T ci) {
    const lane_t<T> c = vall(cr), s = vall(ci);
    return CV<T>{vfma(a.re, c, vneg(vmul(a.im, s))), vfma(a.re, s, vmul(a.im, c))};
  }
  static __device__ __forceinline__ void run(CV<T>* v) {
    const T c1 = (T)0.92387953251128675613, s1 = (T)0.38268343236508977173, h = (T)0.70710678118654752440;
    const T sg = INV ? (T)1 : (T)-1;
    CV<T> a[4][4];
#pragma unroll
    for (int q1 = 0; q1 < 4; ++q1) {
#pragma unroll
      for (int q2 = 0; q2 < 4; ++q2) a[q1][q2] = v[q1 + 4 * q2];
      DftV<T, 4, INV>::run(a[q1]);
    }
    a[1][1] = tw(a[1][1], c1, sg * s1);
    a[1][2] = tw(a[1][2], h, sg * h);
    a[1][3] = tw(a[1][3], s1, sg * c1);
    a[2][1] = tw(a[2][1], h, sg * h);
    a[2][2] = cvmul_mi<T, INV>(a[2][2]);
    a[2][3] = tw(a[2][3], -h, sg * h);
    a[3][1] = tw(a[3][1], s1, sg * c1);
    a[3][2] = tw(a[3][2], -h, sg * h);
    a[3][3] = tw(a[3][3], -c1, -sg * s1);
#pragma unroll
    for (int s2 = 0; s2 < 4; ++s2) {
      CV<T> b[4] = {a[0][s2], a[1][s2], a[2][s2], a[3][s2]};
      DftV<T, 4, INV>::run(b);
#pragma unroll
      for (int s1i = 0; s1i < 4; ++s1i) v[s2 + 4 * s1i] = b[s1i];
    }
  }
};

// 9, 10, 12 and 15 as Dft of fft_smem.cuh.
template <typename T, int N1, int N2, bool INV> struct DftVCrt {
  static __device__ __forceinline__ void run(CV<T>* v) {
    constexpr int N = N1 * N2;
    constexpr int c1 = N2 * (N2 % N1 == 1 ? 1 : N1 - 1), c2 = N1 * (N1 % N2 == 1 ? 1 : N1 * 2 % N2 == 1 ? 2 : N1 * 3 % N2 == 1 ? 3 : 4);
    static_assert(c1 % N1 == 1 && c2 % N2 == 1, "");
    CV<T> a[N1][N2];
#pragma unroll
    for (int i = 0; i < N1; ++i) {
#pragma unroll
      for (int j = 0; j < N2; ++j) a[i][j] = v[(N2 * i + N1 * j) % N];
      DftV<T, N2, INV>::run(a[i]);
    }
#pragma unroll
    for (int j = 0; j < N2; ++j) {
      CV<T> b[N1];
#pragma unroll
      for (int i = 0; i < N1; ++i) b[i] = a[i][j];
      DftV<T, N1, INV>::run(b);
#pragma unroll
      for (int i = 0; i < N1; ++i) v[(c1 * i + c2 * j) % N] = b[i];
    }
  }
};
template <typename T, bool INV> struct DftV<T, 10, INV> : DftVCrt<T, 2, 5, INV> {};
template <typename T, bool INV> struct DftV<T, 12, INV> : DftVCrt<T, 3, 4, INV> {};
template <typename T, bool INV> struct DftV<T, 15, INV> : DftVCrt<T, 3, 5, INV> {};
template <typename T, bool INV> struct DftV<T, 9, INV> {
  static __device__ __forceinline__ void run(CV<T>* v) {
    const T sg = INV ? (T)1 : (T)-1;
    const T c[3] = {(T)0.76604444311897803520, (T)0.17364817766693034885, (T)-0.93969262078590838405};
    const T s[3] = {(T)0.64278760968653932632, (T)0.98480775301220805937, (T)0.34202014332566873304};
    CV<T> a[3][3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
#pragma unroll
      for (int r = 0; r < 3; ++r) a[q][r] = v[q + 3 * r];
      DftV<T, 3, INV>::run(a[q]);
    }
    auto tw = [&](const CV<T>& x, int k) { return cvtw<T, false>(x, mk<cplx<T>>(c[k], sg * s[k])); };
    a[1][1] = tw(a[1][1], 0);
    a[1][2] = tw(a[1][2], 1);
    a[2][1] = tw(a[2][1], 1);
    a[2][2] = tw(a[2][2], 2);
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      CV<T> b[3] = {a[0][r], a[1][r], a[2][r]};
      DftV<T, 3, INV>::run(b);
#pragma unroll
      for (int q = 0; q < 3; ++q) v[r + 3 * q] = b[q];
    }
  }
};

// ------------------------------------------------ lengths known at run time
// Two stages n = r1 r2, r1 >= r2, r1 <= 16 and r2 <= 10: every n <= 100 of
// factors 2, 3, 5 and most up to 160.  even: r1 even (the x pass, whose r2 may
// then be the larger one).  False: no such split (125, an x length 150).
__host__ __device__ inline bool lane_radix(int r) {
  return (r >= 2 && r <= 6) || r == 8 || r == 9 || r == 10 || r == 12 || r == 15 || r == 16;
}
inline bool lane_split(int n, bool even, int* r1, int* r2) {
  int best = 0;
  for (int a = 2; a <= 16; ++a) {
    if (n % a != 0 || !lane_radix(a) || (even && a % 2 != 0)) continue;
    const int b = n / a;
    if (b > 10 || (b > 1 && !lane_radix(b)) || (!even && b > a)) continue;
    const int larger = a > b ? a : b;  // the most even split
    if (best == 0 || larger < best) {
      best = larger;
      *r1 = a;
      *r2 = b;
    }
  }
  return best != 0;
}
// f(std::integral_constant<int, r>) for a radix known at run time
template <class F>
__device__ __forceinline__ void first_radix(int r, F&& f) {
  switch (r) {
    case 2: f(std::integral_constant<int, 2>()); break;
    case 3: f(std::integral_constant<int, 3>()); break;
    case 4: f(std::integral_constant<int, 4>()); break;
    case 5: f(std::integral_constant<int, 5>()); break;
    case 6: f(std::integral_constant<int, 6>()); break;
    case 8: f(std::integral_constant<int, 8>()); break;
    case 9: f(std::integral_constant<int, 9>()); break;
    case 10: f(std::integral_constant<int, 10>()); break;
    case 12: f(std::integral_constant<int, 12>()); break;
    case 15: f(std::integral_constant<int, 15>()); break;
    case 16: f(std::integral_constant<int, 16>()); break;
    default: break;
  }
}
template <class F>
__device__ __forceinline__ void second_radix(int r, F&& f) {
  switch (r) {
    case 1: f(std::integral_constant<int, 1>()); break;
    case 2: f(std::integral_constant<int, 2>()); break;
    case 3: f(std::integral_constant<int, 3>()); break;
    case 4: f(std::integral_constant<int, 4>()); break;
    case 5: f(std::integral_constant<int, 5>()); break;
    case 6: f(std::integral_constant<int, 6>()); break;
    case 8: f(std::integral_constant<int, 8>()); break;
    case 9: f(std::integral_constant<int, 9>()); break;
    case 10: f(std::integral_constant<int, 10>()); break;
    default: break;
  }
}
// Quotients by a number known at launch, n d < 2^31: multiplication by
// ceil(2^32 / d).
struct FastDiv {
  unsigned mul;  // 0: d = 1
  int d;
};
inline FastDiv fast_div(int d) { return FastDiv{d == 1 ? 0u : (unsigned)((0x100000000ull + d - 1) / d), d}; }
__device__ __forceinline__ int fdiv(int n, const FastDiv& f) {
  return f.mul == 0 ? n : (int)(((unsigned long long)(unsigned)n * f.mul) >> 32);
}

// Twiddles of a first stage of radix R1 in the order its threads read them,
// tab[s * NB + b] = scale w_n^(b s), b < NB: neighbouring butterflies b read
// neighbouring entries.  tw: exp(-2 pi i k / n), k = 0..n-1.
template <typename T, int N, int R1, int NB>
__device__ __forceinline__ void stage_twiddles(cplx<T>* tab, const cplx<T>* __restrict__ tw, T scale) {
  for (int i = threadIdx.x; i < R1 * NB; i += blockDim.x) {
    const cplx<T> w = tw[((i / NB) * (i % NB)) % N];
    tab[i] = mk<cplx<T>>(scale * w.x, scale * w.y);
  }
}

// Tasks 0 .. COUNT-1 of a stage over threads 0 .. NT-1 (others do nothing).
template <int COUNT, int NT, class F>
__device__ __forceinline__ void lane_tasks(int tid, F&& f) {
  if constexpr (COUNT == NT || COUNT == 2 * NT) {
    if (tid < NT) {
#pragma unroll
      for (int k = 0; k < COUNT / NT; ++k) f(tid + k * NT);
    }
  } else {
#pragma unroll 1
    for (int t = tid < NT ? tid : COUNT; t < COUNT; t += NT) {
      int u = t;
#ifndef FG_HOST_EMU
      asm volatile("" : "+r"(u));  // keeps a task's twiddles from being hoisted out of the loop (spills)
#endif
      f(u);
    }
  }
}

}  // namespace fg
