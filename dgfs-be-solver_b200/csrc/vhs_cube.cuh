// Single-CTA fast-spectral VHS kernel (FP32 N <= 24, FP64 N = 16): the whole N^3
// problem of one point lives in one CTA's shared memory, so no transform
// crosses SMs, and the transform count is nearly halved by an exact
// restatement that uses the reality of f.
//
// The reference (frfs/solvers/dgfs/scattering.py:227-286, vhs-gll.mako)
// computes per radial node p and direction q
//     t3 = IFFT(cos a F), t4 = IFFT(sin a F),  S = t3^2 + t4^2 (complex),
// with F = FFT(f)/V and a(l) = fac_p s_q.l, then
//     Q = prefac (Re IFFT(sum_p w1_p FFT(sum_q S)) - f Re IFFT(b2 F)).
// w1_p and b2 depend on |l| only, and the index grid maps -l onto itself up
// to the Nyquist index (l0 holds -N/2 but not +N/2), so both are even on the
// grid: Re IFFT(w FFT(S)) = IFFT(w FFT(Re S)) and only Re S matters.
// Let l' = -l (mod N).  Real f gives F(l') = conj F(l), and
// a(l') = -a(l) - theta(l), theta = fac_p N sum over the axes where l sits on
// the Nyquist index of s_q[axis] (theta = 0 off those planes).  Splitting
// cos a F and sin a F into parts that are even and odd under l -> l'
// (conjugated) gives exactly
//     Re S = Re(R^2) + Re(Nq^2),
//     R  = IFFT(m F),  m = (cos a + cos(a+th) + sin a + sin(a+th)) / 2,
//     Nq = IFFT(n F),  n = (cos a - cos(a+th) + sin a - sin(a+th)) / 2,
// where n vanishes off the three Nyquist planes, so Nq is three 2D
// transforms broadcast along one axis with a (-1)^x sign:
//     Nq(x) = (-1)^x1 T1(x2,x3) + (-1)^x2 T2(x1,x3) + (-1)^x3 T3(x1,x2).
// Off the Nyquist planes m = cos a + sin a: one complex transform per (p, q)
// instead of two.  Per point: 1 + Nrho M + Nrho + 2 full transforms plus
// the 2D ones (reference: 3 Nrho M + 3).
//
// FP64 restates it once more, also exactly: with P = (1 + i) R, Re R^2 =
// Re P Im P (and Re Nq^2 likewise), so it transforms F^ = (1 + i) F and
// accumulates one product per field.  FP32 keeps F^ = F and the squares, and
// the mixed-radix transforms, in a fixed order of roundings (fft_vec.cuh): near
// equilibrium Q is 1e-6 to 1e-2 of the gain, and what is left of it depends on
// that order.
//
// What bounds it: shared memory, the FP32 pipe and the passes' latencies.  Per
// (p, q) the work cube crosses shared memory four times (two exchanges) and
// every complex value takes 13 to 16 operations a pass.  So: a thread owns one
// line (N = 24: 18 warps and 2 for the Nyquist planes, five per scheduler; nine
// warps with two lines per thread left one scheduler with half as many again as
// the others), in FP32 as packed registers (fft_vec.cuh: sums and differences
// in half the issue slots); everything that only its own thread
// touches -- the spectrum line and the sums S_p -- lives in tensor memory,
// which costs neither registers nor shared-memory bandwidth; and no shared
// access of the main threads conflicts.
//
// Layout in shared memory (complex float):
//   sW   work cube: line (k1, k2) at k1 PS + off(k2), off(k) = N k + (k >= N/2).
//        Half a warp of the first pass is 8 planes x {k2, k2 + N/2}, of the
//        second 8 planes x {x3, x3 + 1}, of the third 8 x3 x {x2, x2 + N/2}:
//        16 distinct 8-byte banks each (FP64: 8 lanes, 8 16-byte banks)
//   sT1 [x2][x3], sT2 [x1][x3], sT3 [x2][x1]: the transformed Nyquist planes
//   sN   [k][line] the spectrum on the Nyquist planes; sX their first axis
//   phases of (p, q) and of the next, in two slots
// The main threads are N/8 groups, each owning 8 planes k1: the second pass of
// a group needs only that group's first pass, so groups synchronise among
// themselves.  The third pass releases the cube as soon as its values are in
// registers, so its arithmetic runs beside the next first pass.  NQ more
// threads transform the Nyquist planes and fetch the next phases.  The gain
// spectrum is kept in a global (L2-resident) slice per CTA, [k3][line].
//
// Measured on one B200 (FP32, N = 24, 12 x 16 (p, q), 576 points): 4.54 ms a
// sweep against 5.17 ms for two lines per thread with scalar transforms, with
// the same roundings.  N = 16 (8 x 6): FP64, one point 59 us against 191 us for
// the two-CTA push kernel (its radial nodes spread over the SMs); FP32, 592
// points 0.48 ms against 1.16 ms, but its error is 1.2 times that of the push
// kernel's two transforms per (p, q), so there it is not the default.
#pragma once

#include "fft_vec.cuh"
#include "tcgen05.cuh"
#include "vhs_kernel.cuh"
#include "vhs_variant.h"

namespace dgfs {

template <typename T, int N> struct CubeGeom {
  static constexpr int HN = N / 2, H = HN + 1, NN = N * N, V = NN * N;
  static constexpr int NM = NN;                      // main threads, one line each
  static constexpr int GT = 8 * N;                   // threads per group of 8 planes
  static constexpr int NQ = 3 * N <= 32 ? 32 : 64;   // Nyquist threads, one or two lines each
  static constexpr int NT = NM + NQ;
  static constexpr int PS = NN + (sizeof(T) == 4 ? 2 : 1);  // plane stride of the work cube
  static constexpr int PHS = 3 * N + 4;              // one phase slot
  // FP64 keeps the gain spectrum for k1 <= N/2 (the transform of a real S_p),
  // FP32 all of it: mirrored values differ from transformed ones by round-off
  static constexpr int GK = sizeof(T) == 4 ? N : H, NL = GK * N;  // lines of the gain spectrum
  static constexpr int SL = NL * N;                  // gain spectrum slice (complex)
  // tensor memory columns: per main warp 2 N values of F^, then N of S
  static constexpr int WD = sizeof(T) / 4;           // columns per value
  static constexpr int TW = 3 * N * WD, TUSED = (NM / 32 + 3) / 4 * TW;
  static constexpr int TCOLS = TUSED <= 32 ? 32 : TUSED <= 64 ? 64 : TUSED <= 128 ? 128 : TUSED <= 256 ? 256 : 512;
  static constexpr int OFF_W = 0;
  static constexpr int OFF_T1 = OFF_W + N * PS;
  static constexpr int OFF_T2 = OFF_T1 + NN;
  static constexpr int OFF_T3 = OFF_T2 + NN;
  static constexpr int OFF_N = OFF_T3 + N * (N + 2);
  static constexpr int OFF_X = OFF_N + 3 * NN;
  static constexpr int OFF_PH = OFF_X + 3 * N * (N + 1);
  static constexpr int SMEM = (OFF_PH + 2 * PHS) * 2 * (int)sizeof(T);  // bytes
  __host__ __device__ static constexpr int off(int k) { return N * k + (k >= HN ? 1 : 0); }
  static_assert(N % 8 == 0 && 3 * N <= 2 * NQ && NM % 32 == 0, "thread roles");
  static_assert(OFF_T2 % 2 == 0 && OFF_T3 % 2 == 0 && OFF_PH % 2 == 0 && PHS % 2 == 0, "16-byte sections");
};

// Radial-node chunks per point.  A launch with few points would leave SMs
// idle with one point per CTA, so each point's P radial nodes can be split
// into P work items of one node each: cost ~ waves x (nodes per item x
// (3 M + 3) + kFixed) passes.  kFixed is what an item costs before its first
// node and after its last (its own transform of f, the tables, the slice and
// the point's last pass), fitted from the time per wave of split and of whole
// items: 37 passes at N = 24 (P = 12, M = 16: 155 against 1,140 us a wave; M = 6:
// 104 against 514 us), 47 at N = 16 FP32 (P = 8, M = 6: 39 against 123 us) and 44
// in FP64 (57 against 185 us).  So a split pays up to 7, 3 and 3 waves, which 37
// gives in all three: at N = 24 86 points take 1,086 us split and 87 or more,
// whole, 1,140 us; at N = 16 55 points take 109 us split and 56 or more, whole,
// 123 us (FP64 171 and 185 us).  Only 1 or P chunks: with one node per chunk the
// final sum over the chunks' slices adds the nodes in the same order as the
// unsplit accumulation, so a point's Q does not depend on the launch it is part
// of (bit for bit).  Items are capped at kCubeSlices per CTA of the grid (the
// partial-spectrum scratch), and more points than CTAs are not split.
// Every CTA computes the same value.
__device__ __forceinline__ int cube_chunks(int npts, int G, int P, int M) {
  if (P < 2 || npts > G || (long long)npts * P > (long long)kCubeSlices * G) return 1;
  constexpr double kFixed = 37.0;
  const double per_node = 3.0 * M + 3.0;
  const double whole = (double)((npts + G - 1) / G) * (P * per_node + kFixed);
  const double split = (double)(((long long)npts * P + G - 1) / G) * (per_node + kFixed);
  return split < whole ? P : 1;
}

// Cycles between the starts of the second pass of a scheduler's successive
// warps: staggered, the loads of one warp run beside the arithmetic of
// another and the stores of a third (N = 24, five warps per scheduler: 1 to 4 %
// of a sweep; 60, 100 and 200 cycles measure the
// same; at N = 16, two or three warps, with and without measure the same in
// either precision, so it is left out there).
constexpr unsigned kStagger = 100;

template <typename T, int N, int MINB>
__global__ void __launch_bounds__(CubeGeom<T, N>::NT, MINB) vhs_cube_kernel(const VhsArgs<T> a) {
  using G = CubeGeom<T, N>;
  using C = vx<T>;   // in registers
  using CM = cx<T>;  // in the tables and the scratch
  constexpr int WD = G::WD;
  constexpr bool ROT = sizeof(T) == 8;  // F^ = (1 + i) F, else F
  constexpr int HN = G::HN, NN = G::NN, V = G::V, NM = G::NM, GT = G::GT, NT = G::NT, PS = G::PS, PHS = G::PHS;
  constexpr int B_ALL = 0, B_T = 1, B_G = 2;  // named barriers: CTA, Nyquist tables, groups

  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* const base = reinterpret_cast<C*>(smem_raw);
  C* const sW = base + G::OFF_W;
  C* const sT1 = base + G::OFF_T1;
  C* const sT2 = base + G::OFF_T2;
  C* const sT3 = base + G::OFF_T3;
  C* const sN = base + G::OFF_N;
  C* const sX = base + G::OFF_X;
  CM* const sPh = reinterpret_cast<CM*>(base + G::OFF_PH);
  __shared__ double sRed[5][NT / 32];
  __shared__ double sLam[5];
  __shared__ uint32_t s_tmem;
  __shared__ __align__(8) uint64_t s_read;  // every main warp has read its part of the cube
  __shared__ int s_gave_up;

  const int tid = threadIdx.x;
  const bool is_main = tid < NM;
  const int tq = tid - NM;
  CM* const fcg = a.fc + (size_t)blockIdx.x * G::SL;
  const int npq = a.P * a.M;

  // roles of a main thread: first pass line (k1, k2), second pass line
  // (k1, x3 = r), third pass line (x2 = r, x3 = k1)
  const int grp = tid / GT, gu = tid % GT, k1 = 8 * grp + gu % 8, r = gu / 8, k2 = (r & 1) * HN + (r >> 1);
  // place of line (k1, k2) in the gain spectrum: FP32, where only this thread
  // touches it, by thread, so that a warp's accesses are whole 128-byte lines
  // (N = 24: a point call 157 us, a sweep of 576 points 4.54 ms; by line 198 us
  // and 4.76 ms, the sum of a split point's 12 slices alone 58 us); FP64 by line
  const int gpos = G::GK == N ? tid : k1 * N + k2;
  C* const w1p = sW + k1 * PS + G::off(k2);
  C* const w2p = sW + k1 * PS + r;
  const int x2 = r, x3 = k1, wid = tid / 32;
  C* const w3p = sW + G::off(x2) + x3;

  // second pass, in place
  auto pass2 = [&](auto sgn) {
    constexpr int S = decltype(sgn)::value;
    C x[N];
#pragma unroll
    for (int j = 0; j < N; ++j) x[j] = w2p[G::off(j)];
    vfft<N, S>(x);
#pragma unroll
    for (int j = 0; j < N; ++j) w2p[G::off(j)] = x[j];
  };
  // axis phases e^{i fac_p s_q[ax] l0[k]} of (p, q) and Theta_ax =
  // e^{i fac_p N s_q[ax]} = conj(e^{i fac_p s_q[ax] l0[N/2]})^2.  Nyquist
  // threads carry one or two entries each.
  constexpr int NPH = (3 * N + G::NQ - 1) / G::NQ;
  auto phase_fetch = [&](int pq, CM (&e)[NPH]) {
#pragma unroll
    for (int i = 0; i < NPH; ++i) {
      const int n = tq + i * G::NQ;
      e[i] = n < 3 * N ? a.phase[(size_t)pq * 3 * N + n] : mk<CM>(T(0), T(0));
    }
  };
  auto phase_store = [&](const CM (&e)[NPH], int slot) {
#pragma unroll
    for (int i = 0; i < NPH; ++i) {
      const int n = tq + i * G::NQ;
      CM* dst = sPh + slot * PHS;
      if (n < 3 * N) dst[n] = e[i];
      if (n < 3 * N && n % N == HN) {
        const CM ce = mk<CM>(e[i].x, -e[i].y);
        dst[3 * N + n / N] = mul_r(ce, ce);
      }
    }
  };
  // F^ at (k1, k2, k3) from the work cube; FP32: k3 > N/2 from the conjugate
  // mirror
  auto Fat = [&](int i1, int i2, int i3) -> C {
    if (ROT || i3 <= HN) return sW[i1 * PS + G::off(i2) + i3];
    const C c = sW[(N - i1) % N * PS + G::off((N - i2) % N) + N - i3];
    return vmk(cre(c), -cim(c));
  };
  const int npts = a.pcount ? min(a.npts, *a.pcount) : a.npts;
  // work item = (point, chunk of radial nodes); with KP > 1 each chunk's
  // partial gain spectrum goes to its own scratch slice and the CTA that
  // finishes a point's last chunk (a counter per point) sums the slices and
  // completes the point.  No CTA waits for another.
  // The values that stay fixed over an item live in shared memory (s_kp;
  // s_it = first and end radial node, upt, elem): read where needed, they
  // hold no registers through the (p, q) loop.
  __shared__ int s_last, s_kp, s_ni, s_ga, s_it[4];
  {
    const int kp = a.pdone ? cube_chunks(npts, gridDim.x, a.P, a.M) : 1;
    const int nitems = npts * kp;
    // as few CTAs as the number of waves needs (same makespan): the SMs
    // left over stay free for kernels on other streams (the surrogate's
    // network path runs beside its plain fallback)
    const int waves = (nitems + gridDim.x - 1) / gridDim.x;
    const int gactive = waves > 0 ? (nitems + waves - 1) / waves : 0;
    if ((int)blockIdx.x >= gactive) return;  // uniform over the CTA, before any barrier
    if (tid == 0) {
      mbar_init(&s_read, NM / 32);
      s_gave_up = 0;
      s_kp = kp;
      s_ni = nitems;
      s_ga = gactive;
    }
  }
  if (tid < 32) tmem_alloc(&s_tmem, G::TCOLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // this thread's lane and columns: F^ of line (k1, k2), then S of (x2, x3)
  const uint32_t tmF = s_tmem + ((uint32_t)(tid / 32 % 4 * 32) << 16) + tid / 128 * G::TW, tmS = tmF + 2 * N * WD;
  uint32_t rphase = 0;  // parity of s_read's current phase
  constexpr int SC = N % 16 ? 8 : 16;  // values per step of the last pass
  // F^ of this thread's line
  auto load_line = [&](C (&x)[N]) {
    uint32_t t[2 * N * WD];
    tm_load(tmF, t);
    tm_wait(t);
#pragma unroll
    for (int k = 0; k < N; ++k) x[k] = vmk(tm_get(t, 2 * k, T(0)), tm_get(t, 2 * k + 1, T(0)));
  };

  for (int item = blockIdx.x; item < s_ni; item += s_ga) {
    const int ip = item / s_kp;
    const int pt = a.plist ? a.plist[a.pt0 + ip] : a.pt0 + ip;
    if ((unsigned)pt >= (unsigned)(a.nupts * a.neles)) continue;  // uniform over the CTA
    if (tid == 0) {
      const int ch = item % s_kp;
      s_it[0] = ch * a.P / s_kp;
      s_it[1] = (ch + 1) * a.P / s_kp;
      s_it[2] = pt / a.neles;
      s_it[3] = pt % a.neles;
    }

    // ---- F^ from FFT(f) / V ---------------------------------------------
    if (is_main) {
      const int64_t b0 = soa_ix(pt / a.neles, a.ldim, pt % a.neles, (int64_t)(k1 * N + k2) * N, V, a.soasz);
      C x[N];
#pragma unroll
      for (int k = 0; k < N; ++k) x[k] = vmk(a.f[b0 + (int64_t)k * a.soasz], T(0));
      vfft<N, -1>(x);
#pragma unroll
      for (int k = 0; k < N; ++k) w1p[k] = x[k];
    }
    __syncthreads();
    if (is_main) pass2(std::integral_constant<int, -1>{});
    __syncthreads();
    if (is_main) {
      const T iv = T(1) / T(V);
      C x[N];
#pragma unroll
      for (int i = 0; i < N; ++i) x[i] = w3p[i * PS];
      vfft<N, -1>(x);
#pragma unroll
      for (int i = 0; i < N; ++i) w3p[i * PS] = vmul(ROT ? mul_1i<1>(x[i]) : x[i], vmk(iv, iv));
    }
    __syncthreads();
    if (is_main) {
      uint32_t t[2 * N * WD];
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const C v = Fat(k1, k2, i);
        tm_put(t, 2 * i, cre(v));
        tm_put(t, 2 * i + 1, cim(v));
      }
      tm_store(tmF, t);
      tmem_store_wait();
    } else {
#pragma unroll 1
      for (int t = tq; t < 3 * N * N; t += G::NQ) {
        const int k = t / (3 * N), line = t % (3 * N), which = line / N, j = line % N;
        sN[t] = which == 0 ? Fat(HN, j, k) : which == 1 ? Fat(j, HN, k) : Fat(j, k, HN);
      }
      CM e[NPH];
      phase_fetch(s_it[0] * a.M, e);
      phase_store(e, 0);
    }
    __syncthreads();

    // ---- gain: fC = sum_p w1_p FFT(sum_q Re S_pq) ---------------------------
    // Both kinds of threads run the same sequence of CTA-wide barriers: one
    // per (p, q) and two per p.
    if (is_main) {
      int slot = 0;
#pragma unroll 1
      for (int p = s_it[0]; p < s_it[1]; ++p) {
#pragma unroll 1
        for (int q = 0; q < a.M; ++q) {
          // pass 1: m F^ along k3.  m = Re((E + E t)(1 - i)) / 2 with
          // E = E12 E3[k3] and t the Nyquist factor (1 off the planes): per
          // line A = (E12 + E12 t12) (1 - i) / 2 (A3 on the k3 = N/2 plane),
          // then m = Re(A E3[k3])
          {
            const CM* ph = sPh + slot * PHS;
            const CM E12 = mul_r(ph[k1], ph[N + k2]);
            const CM th1 = ph[3 * N], th2 = ph[3 * N + 1];
            const CM t12 = k1 != HN ? th2 : k2 == HN ? mul_r(th1, th2) : th1;
            const CM Et = k1 == HN || k2 == HN ? mul_r(E12, t12) : E12;
            const CM s0 = cadd(E12, Et), s3 = cadd(E12, mul_s(Et, ph[3 * N + 2]));
            const CM A = mk<CM>(T(0.5) * (s0.x + s0.y), T(0.5) * (s0.y - s0.x));
            const CM A3 = mk<CM>(T(0.5) * (s3.x + s3.y), T(0.5) * (s3.y - s3.x));
            C x[N];
            load_line(x);
            // e3[N - k] = conj e3[k]
            vfft_scaled<N, 1>(x, [&](int k) {
              const CM e = ph[2 * N + (k <= HN ? k : N - k)];
              return re_mul(k == HN ? A3 : A, k <= HN ? e : mk<CM>(e.x, -e.y));
            });
            mbar_wait_bounded(&s_read, rphase ^ 1, a.err, &s_gave_up);  // the previous cube is read
#pragma unroll
            for (int k = 0; k < N; ++k) w1p[k] = x[k];
          }
          slot ^= 1;
          bar_arrive(B_T, NT);        // done with the Nyquist tables of the previous (p, q)
          bar_sync(B_G + grp, GT);    // this group's planes are complete
          if constexpr (NM / 32 > 8) {
            const unsigned t0 = clock();
            while (clock() - t0 < (unsigned)(wid >> 2) * kStagger) {
            }
          }
          pass2(std::integral_constant<int, 1>{});
          bar_sync(B_ALL, NT);        // the cube and the Nyquist tables are complete
          // pass 3: lines (x2, x3) along k1; S += Re R^2 + Re Nq^2 with
          // Nq = s1 T1(x2, x3) + s2 T2(x1, x3) + s3 T3(x1, x2), s = (-1)^x
          C x[N];
#pragma unroll
          for (int i = 0; i < N; ++i) x[i] = w3p[i * PS];
          __syncwarp();
          if (tid % 32 == 0) mbar_arrive(&s_read);  // this warp's part of the cube may be overwritten
          rphase ^= 1;
          uint32_t t[N * WD];
          tmem_store_wait();
          tm_load(tmS, t);
          vfft<N, 1>(x);
          const T s2 = (x2 & 1) ? T(-1) : T(1), s3 = (x3 & 1) ? T(-1) : T(1);
          const C t1 = sT1[x2 * N + x3], t1n = vmul(t1, vmk(T(-1), T(-1))), c2 = vmk(s2, s2), c3 = vmk(s3, s3);
          tm_wait(t);
#pragma unroll
          for (int i = 0; i < N; ++i) {
            const C n = vfma(sT3[x2 * (N + 1) + i], c3, vfma(sT2[i * N + x3], c2, (i & 1) ? t1n : t1));
            tm_put(t, i, add_squares(x[i], n, q == 0 ? T(0) : tm_get(t, i, T(0))));
          }
          tm_store(tmS, t);
        }
        // FFT(S_p): lines of the third pass along x1 from the accumulators,
        // each thread to the entries it read last, then planes k1 < GK
        {
          C x[N];
          tmem_store_wait();
          uint32_t t[N * WD];
          tm_load(tmS, t);
          tm_wait(t);
#pragma unroll
          for (int i = 0; i < N; ++i) x[i] = vmk(tm_get(t, i, T(0)), T(0));
          vfft<N, -1>(x);
#pragma unroll
          for (int i = 0; i < G::GK; ++i) w3p[i * PS] = x[i];
        }
        bar_sync(B_ALL, NT);
        if (k1 < G::GK) pass2(std::integral_constant<int, -1>{});
        bar_sync(B_ALL, NT);
        if (k1 < G::GK) {
          // line (k1, k2) along x3.  All loads of the accumulated line are
          // issued before its first store (the slices could alias w1 as far
          // as the compiler knows)
          const T* w1 = a.w1t + (size_t)p * V + k1 * N + k2;
          CM* const fca = (s_kp == 1 ? fcg : a.fcp + (size_t)item * G::SL) + gpos;
          C x[N];
#pragma unroll
          for (int k = 0; k < N; ++k) x[k] = w1p[k];
          vfft<N, -1>(x);
#pragma unroll
          for (int k = 0; k < N; ++k) {
            const T w = __ldg(w1 + k * NN);
            x[k] = vmul(x[k], vmk(w, w));
          }
          if (p > s_it[0]) {
#pragma unroll
            for (int k = 0; k < N; ++k) x[k] = vadd(from_c(fca[k * G::NL]), x[k]);
          }
#pragma unroll
          for (int k = 0; k < N; ++k) fca[k * G::NL] = to_c(x[k]);
        }
      }
    } else {
      int slot = 0;
#pragma unroll 1
      for (int p = s_it[0]; p < s_it[1]; ++p) {
#pragma unroll 1
        for (int q = 0; q < a.M; ++q) {
          const int pq = p * a.M + q;
          CM phn[NPH];
          if (pq + 1 < npq) phase_fetch(pq + 1, phn);
          // n F^ on the Nyquist planes: plane 1 (k1 = N/2) lines over k3,
          // plane 2 (k2 = N/2, k1 != N/2) lines over k3, plane 3 (k3 = N/2,
          // k1, k2 != N/2) lines over k2.  On a line only the phase of the
          // running axis changes, so n = Re(D (1 - i)) / 2 with D = E (1 - t)
          // becomes n = Re(A e[k]) with one coefficient A per line (A3 where
          // k meets the Nyquist index of the running axis).
#pragma unroll 1
          for (int line = tq; line < 3 * N; line += G::NQ) {
            const int which = line / N, j = line % N;
            const bool p3 = which == 2;
            const CM* ph = sPh + slot * PHS;
            const CM th1 = ph[3 * N], th2 = ph[3 * N + 1], th3 = ph[3 * N + 2];
            const CM Eb = mul_r(ph[which == 0 ? HN : j], ph[which == 0 ? N + j : p3 ? 2 * N + HN : N + HN]);
            const CM tb = p3 ? th3 : which == 1 ? th2 : j == HN ? mul_r(th1, th2) : th1;
            const CM tb3 = mul_r(tb, th3);
            CM B = mul_1m(Eb, tb);
            CM B3 = p3 ? mk<CM>(T(0), T(0)) : mul_1m(Eb, tb3);
            if (which != 0 && j == HN) B = B3 = mk<CM>(T(0), T(0));
            const CM A = mk<CM>(T(0.5) * (B.x + B.y), T(0.5) * (B.y - B.x));
            const CM A3 = mk<CM>(T(0.5) * (B3.x + B3.y), T(0.5) * (B3.y - B3.x));
            const CM* ev = ph + (p3 ? N : 2 * N);
            C x[N];
#pragma unroll
            for (int k = 0; k < N; ++k) x[k] = sN[k * 3 * N + line];
            vfft_scaled<N, 1>(x, [&](int k) { return re_mul(k == HN ? A3 : A, ev[k]); });
#pragma unroll
            for (int k = 0; k < N; ++k) sX[line * (N + 1) + k] = x[k];
          }
          if (pq + 1 < npq) phase_store(phn, slot ^ 1);
          slot ^= 1;
          bar_sync(B_T, NT);  // every first axis is done, and no main thread reads the old tables
#pragma unroll 1
          for (int line = tq; line < 3 * N; line += G::NQ) {
            const int which = line / N, j = line % N;
            C x[N];
#pragma unroll
            for (int i = 0; i < N; ++i) x[i] = sX[(which * N + i) * (N + 1) + j];
            vfft<N, 1>(x);
            // element i of the column: T1[i][j], T2[i][j], T3[j][i]
            C* const d = which == 0 ? sT1 + j : which == 1 ? sT2 + j : sT3 + j * (N + 1);
            const int de = which == 2 ? 1 : N;
#pragma unroll
            for (int i = 0; i < N; ++i) d[i * de] = x[i];
          }
          bar_sync(B_ALL, NT);
        }
        bar_sync(B_ALL, NT);
        bar_sync(B_ALL, NT);
      }
    }

    if (s_kp > 1) {
      // publish this chunk's slice; the point's last chunk goes on
      __threadfence();
      __syncthreads();
      if (tid == 0) s_last = atomicAdd(a.pdone + item / s_kp, 1) == s_kp - 1;
      __syncthreads();
      if (!s_last) continue;  // uniform over the CTA
      __threadfence();
    }

    // ---- Q = prefac (Re IFFT(fC) - f Re IFFT(b2 F)) ----------------------------
    // Two transforms: fC, summed from FP32 transforms, carries round-off, and
    // packing it with b2 F into one transform would leak that round-off into
    // the loss term as a constant times f (a momentum error proportional to
    // rho u).  Of the transform of b2 F^ (in FP64 (1 + i) times the real collision
    // frequency) the real part is kept where S was.
    if (is_main) {
      const T* b2 = a.b2t + k1 * N + k2;
      C x[N];
      load_line(x);
      vfft_scaled<N, 1>(x, [&](int k) { return __ldg(b2 + k * NN); });
#pragma unroll
      for (int k = 0; k < N; ++k) w1p[k] = x[k];
    }
    __syncthreads();
    if (is_main) pass2(std::integral_constant<int, 1>{});
    __syncthreads();
    if (is_main) {
      C x[N];
#pragma unroll
      for (int i = 0; i < N; ++i) x[i] = w3p[i * PS];
      vfft<N, 1>(x);
      uint32_t t[N * WD];
#pragma unroll
      for (int i = 0; i < N; ++i) tm_put(t, i, cre(x[i]));
      tm_store(tmS, t);
      tmem_store_wait();
    }
    __syncthreads();
    // QG = Re IFFT(fC); the chunks' slices are summed in a fixed order (L2
    // reads: other CTAs wrote them).  FP64: planes k1 > N/2 are the
    // conjugate mirror of k1 < N/2.
    if (is_main) {
      const bool mir = k1 >= G::GK;
      const int kp = s_kp, i0 = item - item % kp;
      const CM* src = (kp == 1 ? fcg : a.fcp + (size_t)i0 * G::SL) + (mir ? (N - k1) * N + (N - k2) % N : gpos);
      C x[N];
#pragma unroll
      for (int k = 0; k < N; ++k) x[k] = from_c(__ldcg(src + k * G::NL));
#pragma unroll 1
      for (int c = 1; c < kp; ++c) {
        src += G::SL;
#pragma unroll
        for (int k = 0; k < N; ++k) x[k] = vadd(x[k], from_c(__ldcg(src + k * G::NL)));
      }
      if (mir) {
        // x[k] <- conj x[-k]
        sfor<1, HN>([&](auto kc) {
          constexpr int k = decltype(kc)::value;
          const C t = x[k];
          x[k] = vmk(cre(x[N - k]), -cim(x[N - k]));
          x[N - k] = vmk(cre(t), -cim(t));
        });
        x[0] = vmk(cre(x[0]), -cim(x[0]));
        x[HN] = vmk(cre(x[HN]), -cim(x[HN]));
      }
      vfft<N, 1>(x);
#pragma unroll
      for (int k = 0; k < N; ++k) w1p[k] = x[k];
    }
    __syncthreads();
    if (is_main) pass2(std::integral_constant<int, 1>{});
    __syncthreads();
    double mom[5] = {0, 0, 0, 0, 0};
    // bank entry of v = i N^2 + x2 N + x3 is b0 + i st: v enters the AoSoA index
    // linearly
    const int64_t b0 = soa_ix(s_it[2], a.ldim, s_it[3], x2 * N + x3, V, a.soasz), st = (int64_t)NN * a.soasz;
    if (is_main) {
      C x[N];
#pragma unroll
      for (int i = 0; i < N; ++i) x[i] = w3p[i * PS];
      vfft<N, 1>(x);
      sfor<0, N / SC>([&](auto cc) {
        constexpr int c = decltype(cc)::value;
        uint32_t t[SC * WD];
        tm_load(tmS + SC * c * WD, t);
        // f first, every load of the step issued before its first store of Q
        // (which may alias f as far as the compiler knows)
        T fl[SC];
#pragma unroll
        for (int h = 0; h < SC; ++h) fl[h] = a.f[b0 + (SC * c + h) * st];
        tm_wait(t);
#pragma unroll
        for (int h = 0; h < SC; ++h) {
          const int i = SC * c + h;
          const T qq = a.prefac * (cre(x[i]) - fl[h] * tm_get(t, h, T(0)));
          if (!a.project) a.Q[b0 + i * st] = qq;
          tm_put(t, h, qq);
        }
        if (a.project) {
#pragma unroll
          for (int h = 0; h < SC; ++h) {
            const int v = (SC * c + h) * NN + x2 * N + x3;
            const double c0 = a.cvec[v], c1 = a.cvec[V + v], c2 = a.cvec[2 * V + v];
            const double d = (double)tm_get(t, h, T(0));
            mom[0] += d;
            mom[1] += d * c0;
            mom[2] += d * c1;
            mom[3] += d * c2;
            mom[4] += d * (c0 * c0 + c1 * c1 + c2 * c2);
          }
          tm_store(tmS + SC * c * WD, t);
        }
      });
      tmem_store_wait();
    }
    if (a.project) {  // uniform: every thread takes part in the reduction
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        double s = mom[k];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if ((tid & 31) == 0) sRed[k][tid >> 5] = s;
      }
      __syncthreads();
      if (tid < 5) {
        double s = 0;
        for (int w = 0; w < NT / 32; ++w) s += sRed[tid][w];
        sRed[tid][0] = s;
      }
      __syncthreads();
      if (tid < 5) {
        double l = 0;
        for (int j = 0; j < 5; ++j) l += a.ginv[tid * 5 + j] * sRed[j][0];
        sLam[tid] = l;
      }
      __syncthreads();
      if (is_main) {
        sfor<0, N / SC>([&](auto cc) {
          constexpr int c = decltype(cc)::value;
          uint32_t t[SC * WD];
          tm_load(tmS + SC * c * WD, t);
          tm_wait(t);
#pragma unroll
          for (int h = 0; h < SC; ++h) {
            const int v = (SC * c + h) * NN + x2 * N + x3;
            const double c0 = a.cvec[v], c1 = a.cvec[V + v], c2 = a.cvec[2 * V + v];
            a.Q[b0 + (SC * c + h) * st] =
                (T)((double)tm_get(t, h, T(0)) - (sLam[0] + sLam[1] * c0 + sLam[2] * c1 + sLam[3] * c2 +
                                                         sLam[4] * (c0 * c0 + c1 * c1 + c2 * c2)));
          }
        });
      }
    }
    if (s_kp > 1 && tid == 0) a.pdone[item / s_kp] = 0;  // every chunk has counted: ready for the next launch
    __syncthreads();  // the work cube and fC are reused by the next point
  }
  __syncthreads();
  if (tid < 32) tmem_dealloc(s_tmem, G::TCOLS);
}

}  // namespace dgfs
