// Register-resident complex FFTs of compile-time length, natural order in and
// out, with the conventions of fft_reg.cuh:
//
//   cfft<N, S>(x):  x[k] <- sum_n x[n] exp(S 2 pi i n k / N),  N = 8, 16, 24
//   mfft<N, S>(x):  the same in FP32, N = 8, 16, 24, 32, with the roundings of
//                   fft_reg.cuh (below)
//
// Two element types: double2, and cpx, an FP32 complex number in one 64-bit
// register pair.  On cpx one packed instruction (add/sub/mul/fma.rn.f32x2)
// works on the real and the imaginary part together.  The packed instructions
// run at the FP32 pipe's rate (128 lanes per clock and SM, the same as scalar
// ones: measured), so they take half the issue slots, which is what the
// transforms of the collision kernels were short of.  Where a value is needed
// times i, its producer writes the parts in swapped order with two scalar
// adds (the same pipe time as one packed add) and the consumer is an FMA
// with (-1, 1) factors.
//
// In cfft the 8-point kernels have their sqrt(1/2) factors folded into FMAs (52
// operations), N = 16 is two of them and N = 24 the prime-factor
// (Good-Thomas) transform: 3 and 8 have no common factor, so 8 three-point
// and 3 eight-point transforms need no twiddle factors between them (252
// operations against 308 for the mixed-radix 8 x 3 transform of fft_reg.cuh);
// its index maps are compile-time register names.
#pragma once

#include "dgfs_common.cuh"

namespace dgfs {

struct cpx {
  unsigned long long v;  // low half: real part
};

__device__ __forceinline__ cpx cpk(float re, float im) {
  cpx r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(re), "f"(im));
  return r;
}
__device__ __forceinline__ float cre(cpx a) { return __uint_as_float((unsigned)a.v); }
__device__ __forceinline__ float cim(cpx a) { return __uint_as_float((unsigned)(a.v >> 32)); }
// the element type of a precision, from and to its parts and to float2 / double2
template <typename T> struct vec_of;
template <> struct vec_of<float> { using type = cpx; };
template <> struct vec_of<double> { using type = double2; };
template <typename T> using vx = typename vec_of<T>::type;
__device__ __forceinline__ cpx vmk(float re, float im) { return cpk(re, im); }
__device__ __forceinline__ double2 vmk(double re, double im) { return make_double2(re, im); }
__device__ __forceinline__ double cre(double2 a) { return a.x; }
__device__ __forceinline__ double cim(double2 a) { return a.y; }
__device__ __forceinline__ cpx from_c(float2 a) { return cpk(a.x, a.y); }
__device__ __forceinline__ double2 from_c(double2 a) { return a; }
__device__ __forceinline__ float2 to_c(cpx a) { return make_float2(cre(a), cim(a)); }
__device__ __forceinline__ double2 to_c(double2 a) { return a; }

__device__ __forceinline__ cpx vadd(cpx a, cpx b) {
  cpx r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ cpx vsub(cpx a, cpx b) {
  cpx r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ cpx vmul(cpx a, cpx b) {  // part by part
  cpx r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ cpx vfma(cpx a, cpx b, cpx c) {  // a b + c part by part
  cpx r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ double2 vmul(double2 a, double2 b) { return make_double2(a.x * b.x, a.y * b.y); }
__device__ __forceinline__ double2 vfma(double2 a, double2 b, double2 c) {
  return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y));
}
__device__ __forceinline__ double2 vadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 vsub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }

// a + i s h b from bs = b with its parts swapped: (a.x - s h b.y, a.y + s h b.x);
// S = +-1, H = 0 (h = 1) or 1 (h = sin(pi/3))
template <int S, int H> __device__ __forceinline__ cpx add_rot(cpx a, cpx bs) {
  constexpr float h = H ? 0.86602540378443864676f : 1.f;
  return vfma(bs, cpk(-S * h, S * h), a);
}
template <int S, int H> __device__ __forceinline__ double2 add_rot(double2 a, double2 bs) {
  if constexpr (H) return make_double2(fma(bs.x, -S * 0.86602540378443864676, a.x), fma(bs.y, S * 0.86602540378443864676, a.y));
  else if constexpr (S > 0) return make_double2(a.x - bs.x, a.y + bs.y);
  else return make_double2(a.x + bs.x, a.y - bs.y);
}
// a - b with the parts swapped
__device__ __forceinline__ cpx sub_swap(cpx a, cpx b) { return cpk(cim(a) - cim(b), cre(a) - cre(b)); }
__device__ __forceinline__ double2 sub_swap(double2 a, double2 b) { return make_double2(a.y - b.y, a.x - b.x); }
// (1 + i S) a
template <int S> __device__ __forceinline__ cpx mul_1i(cpx a) {
  return S > 0 ? cpk(cre(a) - cim(a), cim(a) + cre(a)) : cpk(cre(a) + cim(a), cim(a) - cre(a));
}
template <int S> __device__ __forceinline__ double2 mul_1i(double2 a) {
  return S > 0 ? make_double2(a.x - a.y, a.y + a.x) : make_double2(a.x + a.y, a.y - a.x);
}
// a + S sqrt(1/2) t
template <int S> __device__ __forceinline__ cpx add_h(cpx a, cpx t) {
  return vfma(t, cpk(S * 0.70710678118654752440f, S * 0.70710678118654752440f), a);
}
template <int S> __device__ __forceinline__ double2 add_h(double2 a, double2 t) {
  return make_double2(fma(t.x, S * 0.70710678118654752440, a.x), fma(t.y, S * 0.70710678118654752440, a.y));
}
// a - b / 2
__device__ __forceinline__ cpx sub_half(cpx a, cpx b) { return vfma(b, cpk(-0.5f, -0.5f), a); }
__device__ __forceinline__ double2 sub_half(double2 a, double2 b) {
  return make_double2(fma(b.x, -0.5, a.x), fma(b.y, -0.5, a.y));
}
// a + i S b
template <int S> __device__ __forceinline__ double2 add_i(double2 a, double2 b) {
  return S > 0 ? make_double2(a.x - b.y, a.y + b.x) : make_double2(a.x + b.y, a.y - b.x);
}
// a (c + i s)
__device__ __forceinline__ double2 mul_w(double2 a, double c, double s) {
  return make_double2(fma(-s, a.y, c * a.x), fma(s, a.x, c * a.y));
}

// cos(2 pi j / 96); sin(2 pi j / 96) = cos96(j - 24)
__host__ __device__ constexpr double cos96(int j) {
  constexpr double c[25] = {
      1.0, 0.99785892323860350673, 0.99144486137381041114, 0.98078528040323044912, 0.96592582628906828674,
      0.94693012949510566425, 0.92387953251128675612, 0.89687274153268830389, 0.86602540378443864676,
      0.83146961230254523707, 0.79335334029123516457, 0.75183980747897739640, 0.70710678118654752440,
      0.65934581510006886842, 0.60876142900872063941, 0.55557023301960222474, 0.5, 0.44228869021900128199,
      0.38268343236508977172, 0.32143946530316158070, 0.25881904510252076234, 0.19509032201612826784,
      0.13052619222005159154, 0.06540312923014306681, 0.0};
  j = j < 0 ? -j : j;
  j %= 96;
  j = j > 48 ? 96 - j : j;
  return j > 24 ? -c[48 - j] : c[j];
}
// SW: the third output with its parts swapped
template <int S, bool SW, typename C> __device__ __forceinline__ void cfft4(C& a, C& b, C& c, C& d) {
  const C s0 = vadd(a, c), d0 = vsub(a, c), s1 = vadd(b, d), d1 = sub_swap(b, d);
  a = vadd(s0, s1);
  if constexpr (SW) c = sub_swap(s0, s1);
  else c = vsub(s0, s1);
  b = add_rot<S, 0>(d0, d1);
  d = add_rot<-S, 0>(d0, d1);
}

// 8 points, outputs x0 .. x7 in place of inputs x0 .. x7
template <int S, typename C>
__device__ __forceinline__ void cfft8(C& x0, C& x1, C& x2, C& x3, C& x4, C& x5, C& x6, C& x7) {
  C e0 = x0, e1 = x2, e2 = x4, e3 = x6, o0 = x1, o1 = x3, o2 = x5, o3 = x7;
  cfft4<S, false>(e0, e1, e2, e3);
  cfft4<S, true>(o0, o1, o2, o3);
  x0 = vadd(e0, o0);
  x4 = vsub(e0, o0);
  const C t1 = mul_1i<S>(o1), t3 = mul_1i<-S>(o3);
  x1 = add_h<1>(e1, t1);
  x5 = add_h<-1>(e1, t1);
  x2 = add_rot<S, 0>(e2, o2);
  x6 = add_rot<-S, 0>(e2, o2);
  x3 = add_h<-1>(e3, t3);
  x7 = add_h<1>(e3, t3);
}

template <int N, int S, typename C> __device__ __forceinline__ void cfft(C (&x)[N]) {
  static_assert(N == 8 || N == 16 || N == 24, "cfft lengths");
  if constexpr (N == 8) {
    cfft8<S>(x[0], x[1], x[2], x[3], x[4], x[5], x[6], x[7]);
  } else if constexpr (N == 24) {
    // n = 8 n1 + 3 n2, k = 16 k1 + 9 k2 (mod 24): W24^{nk} = W3^{n1 k1} W8^{n2 k2}
    sfor<0, 8>([&](auto c) {
      constexpr int n = 3 * decltype(c)::value;
      C &a = x[n % 24], &b = x[(8 + n) % 24], &d = x[(16 + n) % 24];
      const C s = vadd(b, d), ds = sub_swap(b, d), e = sub_half(a, s);
      a = vadd(a, s);
      b = add_rot<S, 1>(e, ds);
      d = add_rot<-S, 1>(e, ds);
    });
    C y[24];
    sfor<0, 3>([&](auto c) {
      constexpr int m = 8 * decltype(c)::value, q = 16 * decltype(c)::value;
      C t[8];
      sfor<0, 8>([&](auto i) { t[decltype(i)::value] = x[(m + 3 * decltype(i)::value) % 24]; });
      cfft8<S>(t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7]);
      sfor<0, 8>([&](auto i) { y[(q + 9 * decltype(i)::value) % 24] = t[decltype(i)::value]; });
    });
#pragma unroll
    for (int i = 0; i < 24; ++i) x[i] = y[i];
  } else {
    C e[N / 2], o[N / 2];
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      e[i] = x[2 * i];
      o[i] = x[2 * i + 1];
    }
    cfft<N / 2, S>(e);
    cfft<N / 2, S>(o);
    sfor<0, N / 2>([&](auto c) {
      constexpr int j = decltype(c)::value;
      if constexpr (8 * j == N) {
        const C t = mul_1i<S>(o[j]);
        x[j] = add_h<1>(e[j], t);
        x[j + N / 2] = add_h<-1>(e[j], t);
      } else if constexpr (8 * j == 3 * N) {
        const C t = mul_1i<-S>(o[j]);
        x[j] = add_h<-1>(e[j], t);
        x[j + N / 2] = add_h<1>(e[j], t);
      } else if constexpr (4 * j == N) {
        x[j] = add_i<S>(e[j], o[j]);
        x[j + N / 2] = add_i<-S>(e[j], o[j]);
      } else {
        const C t = j == 0 ? o[j] : mul_w(o[j], cos96(j * (96 / N)), S * cos96(j * (96 / N) - 24));
        x[j] = vadd(e[j], t);
        x[j + N / 2] = vsub(e[j], t);
      }
    });
  }
}

// ---- FP32 transforms of the VHS collision kernels ------------------------------
//
//   mfft<N, S>(x), N = 8 Q, Q = 1 .. 4: 8 points (4 x 2), one layer of
//   twiddles, Q points
//
// the mixed-radix transform of fft_reg.cuh operation by operation, on packed
// values: every sum, product and fused product is rounded where that
// transform rounds it, so the results are its results bit for bit.  The
// collision kernels take it in FP32 because Q near equilibrium is the small
// difference of gain and loss (1e-6 to 1e-5 of either at a distance of 1e-2) and
// shows the transforms' round-off: with two radix-2 layers of rounded twiddles
// over 8-point kernels the error of Q was 1.26 times as large at N = 32; with
// cfft<24> it is 0.78 times, but at a distance of 1e-2 either change is percents
// of Q.
//
//   mfft_scaled<N, S>(x, m): the same of x[k] m(k), real factors: the products
//   of the first butterflies' leading terms are fused into their sums.

// i S a
template <int S> __device__ __forceinline__ cpx rot_i(cpx a) {
  return S > 0 ? cpk(-cim(a), cre(a)) : cpk(cim(a), -cre(a));
}
// a exp(S 2 pi i m / N)
template <int N, int S, int m> __device__ __forceinline__ cpx mtwiddle(cpx a) {
  constexpr int mm = m % N;
  if constexpr (mm == 0) {
    return a;
  } else if constexpr (2 * mm == N) {
    return cpk(-cre(a), -cim(a));
  } else if constexpr (4 * mm == N) {
    return rot_i<S>(a);
  } else if constexpr (4 * mm == 3 * N) {
    return rot_i<-S>(a);
  } else {
    constexpr float c = (float)cos96(mm * (96 / N)), s = S * (float)cos96(mm * (96 / N) - 24);
    return cpk(fmaf(cre(a), c, -__fmul_rn(cim(a), s)), fmaf(cim(a), c, __fmul_rn(cre(a), s)));
  }
}

// the rest of an 8-point transform whose two 4-point ones are done:
// e = transform of the even, o of the odd inputs (o[2] with its parts swapped)
template <int S> __device__ __forceinline__ void mfft8_join(const cpx (&e)[4], const cpx (&o)[4], cpx (&t)[8]) {
  t[0] = vadd(e[0], o[0]);
  t[4] = vsub(e[0], o[0]);
  const cpx w1 = mtwiddle<8, S, 1>(o[1]), w3 = mtwiddle<8, S, 3>(o[3]);
  t[1] = vadd(e[1], w1);
  t[5] = vsub(e[1], w1);
  t[2] = add_rot<S, 0>(e[2], o[2]);
  t[6] = add_rot<-S, 0>(e[2], o[2]);
  t[3] = vadd(e[3], w3);
  t[7] = vsub(e[3], w3);
}

// outputs of the 8-point transforms t[q] of x[Q r + q], through the twiddles
// and the Q-point transforms
template <int N, int S> __device__ __forceinline__ void mfft_join(cpx (&t)[N / 8][8], cpx (&x)[N]) {
  constexpr int Q = N / 8;
  sfor<0, 8>([&](auto kc) {
    constexpr int k = decltype(kc)::value;
    if constexpr (Q == 1) {
      x[k] = t[0][k];
    } else if constexpr (Q == 2) {
      const cpx b = mtwiddle<N, S, k>(t[1][k]);
      x[k] = vadd(t[0][k], b);
      x[k + 8] = vsub(t[0][k], b);
    } else if constexpr (Q == 3) {
      const cpx a = t[0][k], b = mtwiddle<N, S, k>(t[1][k]), c = mtwiddle<N, S, 2 * k>(t[2][k]);
      const cpx s = vadd(b, c), ds = sub_swap(b, c), e = sub_half(a, s);
      x[k] = vadd(a, s);
      x[k + 8] = add_rot<S, 1>(e, ds);
      x[k + 16] = add_rot<-S, 1>(e, ds);
    } else {
      cpx a = t[0][k], b = mtwiddle<N, S, k>(t[1][k]), c = mtwiddle<N, S, 2 * k>(t[2][k]),
          d = mtwiddle<N, S, 3 * k>(t[3][k]);
      cfft4<S, false>(a, b, c, d);
      x[k] = a;
      x[k + 8] = b;
      x[k + 16] = c;
      x[k + 24] = d;
    }
  });
}

template <int N, int S> __device__ __forceinline__ void mfft(cpx (&x)[N]) {
  constexpr int Q = N / 8;
  static_assert(N % 8 == 0 && Q >= 1 && Q <= 4, "8 Q points");
  cpx t[Q][8];
  sfor<0, Q>([&](auto qc) {
    constexpr int q = decltype(qc)::value;
    cpx e[4] = {x[q], x[q + 2 * Q], x[q + 4 * Q], x[q + 6 * Q]};
    cpx o[4] = {x[q + Q], x[q + 3 * Q], x[q + 5 * Q], x[q + 7 * Q]};
    cfft4<S, false>(e[0], e[1], e[2], e[3]);
    cfft4<S, true>(o[0], o[1], o[2], o[3]);
    mfft8_join<S>(e, o, t[q]);
  });
  mfft_join<N, S>(t, x);
}

// cfft4 of a m0, b m1, c m2, d m3.  Scalar: a packed factor (m, m) costs a move
template <int S, bool SW>
__device__ __forceinline__ void mfft4_scaled(cpx& a, cpx& b, cpx& c, cpx& d, float m0, float m1, float m2, float m3) {
  const float p2x = __fmul_rn(cre(c), m2), p2y = __fmul_rn(cim(c), m2);
  const float p3x = __fmul_rn(cre(d), m3), p3y = __fmul_rn(cim(d), m3);
  const cpx s0 = cpk(fmaf(cre(a), m0, p2x), fmaf(cim(a), m0, p2y));
  const cpx d0 = cpk(fmaf(cre(a), m0, -p2x), fmaf(cim(a), m0, -p2y));
  const cpx s1 = cpk(fmaf(cre(b), m1, p3x), fmaf(cim(b), m1, p3y));
  const cpx d1 = cpk(fmaf(cim(b), m1, -p3y), fmaf(cre(b), m1, -p3x));  // parts swapped
  a = vadd(s0, s1);
  if constexpr (SW) c = sub_swap(s0, s1);
  else c = vsub(s0, s1);
  b = add_rot<S, 0>(d0, d1);
  d = add_rot<-S, 0>(d0, d1);
}

template <int N, int S, typename M> __device__ __forceinline__ void mfft_scaled(cpx (&x)[N], const M& m) {
  constexpr int Q = N / 8;
  static_assert(N % 8 == 0 && Q >= 1 && Q <= 4, "8 Q points");
  cpx t[Q][8];
  sfor<0, Q>([&](auto qc) {
    constexpr int q = decltype(qc)::value;
    cpx e[4] = {x[q], x[q + 2 * Q], x[q + 4 * Q], x[q + 6 * Q]};
    cpx o[4] = {x[q + Q], x[q + 3 * Q], x[q + 5 * Q], x[q + 7 * Q]};
    mfft4_scaled<S, false>(e[0], e[1], e[2], e[3], m(q), m(q + 2 * Q), m(q + 4 * Q), m(q + 6 * Q));
    mfft4_scaled<S, true>(o[0], o[1], o[2], o[3], m(q + Q), m(q + 3 * Q), m(q + 5 * Q), m(q + 7 * Q));
    mfft8_join<S>(e, o, t[q]);
  });
  mfft_join<N, S>(t, x);
}

// ---- the collision kernels' lines in either precision ---------------------------
template <int N, int S> __device__ __forceinline__ void vfft(cpx (&x)[N]) { mfft<N, S>(x); }
template <int N, int S> __device__ __forceinline__ void vfft(double2 (&x)[N]) { cfft<N, S>(x); }
template <int N, int S, typename M> __device__ __forceinline__ void vfft_scaled(cpx (&x)[N], const M& m) {
  mfft_scaled<N, S>(x, m);
}
template <int N, int S, typename M> __device__ __forceinline__ void vfft_scaled(double2 (&x)[N], const M& m) {
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const double f = m(k);
    x[k] = make_double2(x[k].x * f, x[k].y * f);
  }
  cfft<N, S>(x);
}
// a b and a (1 - b) with the roundings of FP32 stated: which of the two products
// of a sum is rounded by itself is the compiler's choice otherwise
__device__ __forceinline__ float2 mul_r(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -__fmul_rn(a.y, b.y)), fmaf(a.y, b.x, __fmul_rn(a.x, b.y)));
}
__device__ __forceinline__ float2 mul_1m(float2 a, float2 b) {
  const float c = 1.f - b.x;
  return make_float2(fmaf(a.y, b.y, __fmul_rn(a.x, c)), fmaf(a.y, c, -__fmul_rn(a.x, b.y)));
}
// a b, the other product of the imaginary part rounded by itself
__device__ __forceinline__ float2 mul_s(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -__fmul_rn(a.y, b.y)), fmaf(a.x, b.y, __fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ double2 mul_r(double2 a, double2 b) { return cmul(a, b); }
__device__ __forceinline__ double2 mul_s(double2 a, double2 b) { return cmul(a, b); }
__device__ __forceinline__ double2 mul_1m(double2 a, double2 b) { return cmul(a, make_double2(1.0 - b.x, -b.y)); }
// Re(a b)
__device__ __forceinline__ float re_mul(float2 a, float2 b) { return fmaf(a.x, b.x, -__fmul_rn(a.y, b.y)); }
__device__ __forceinline__ double re_mul(double2 a, double2 b) { return a.x * b.x - a.y * b.y; }
// s + Re r^2 + Re n^2 (FP32), or s + Re r Im r + Re n Im n: the same of r and n
// made from (1 + i) F (FP64)
__device__ __forceinline__ float add_squares(cpx r, cpx n, float s) {
  const float v = fmaf(cre(r), cre(r), -__fmul_rn(cim(r), cim(r)));
  return __fadd_rn(s, fmaf(-cim(n), cim(n), fmaf(cre(n), cre(n), v)));
}
__device__ __forceinline__ double add_squares(double2 r, double2 n, double s) { return fma(r.x, r.y, fma(n.x, n.y, s)); }

}  // namespace dgfs
