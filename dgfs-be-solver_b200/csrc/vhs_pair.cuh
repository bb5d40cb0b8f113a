// Two-CTA fast-spectral VHS kernel for grids that do not fit one SM's
// shared memory: FP32 at N = 32 and FP64 at N = 24.
//
// The same exact restatement of the reference's operator as the single-CTA
// kernel (vhs_cube.cuh: one complex transform IFFT(m F^) per (p, q), F^ =
// (1 + i) F in FP64 and F in FP32, the Nyquist-plane term Nq as three 2D
// transforms, Re S = Re R^2 + Re Nq^2, fC = sum_p w1_p FFT(S_p), Q = prefac
// (Re IFFT(fC) - f Re IFFT(b2 F)); frfs/solvers/dgfs/scattering.py:227-286 and
// vhs-gll.mako:103-266), for a thread-block cluster of two CTAs per solution
// point, persistent over the bank.
//
// Data distribution (rank r of the pair, MH = N/2, Q = N/4):
//   k-slab   CTA r owns MH planes k1, closed under k1 -> -k1 mod N, in slots
//            (pair_kmap): K_0 = {0..Q-1, MH, N-Q+1..N-1}, K_1 = {Q..MH-1,
//            MH+1..N-Q}; in FP64 slots below Q (and slot Q of K_0, k1 = MH) hold the
//            k1 <= N/2 the gain spectrum is kept for (S_p is real), in FP32 it is
//            kept on all lines for k3 <= N/2;
//   x-slab   CTA r owns x2 in X_r = [MH r, MH r + MH).
// A 3D inverse transform runs along k3 on the lines (k1 in K_r, k2), along
// k2 on the lines (k1 in K_r, x3), then along k1 on the lines (x2 in X_r,
// x3).  Between the second and third passes each CTA hands the half of its
// k-slab that the other owns in x (MH complex values per line) to the other
// through a staging buffer in the pair's global scratch (L2 resident):
// coalesced stores, one cluster barrier (release/acquire at cluster scope),
// coalesced L2 loads straight into the third pass's registers.  Measured per
// (p, q), this moves a CTA's half slab about three times faster than remote
// shared-memory stores (st.async into the peer's work cube, an earlier form
// of this kernel).  The staging buffers alternate between consecutive
// exchanges, so the barrier of one exchange also tells a CTA that the peer
// has finished reading the buffer it is about to refill.  Forward transforms
// (FFT(S_p)) run the passes in the opposite order with the same exchange.
//
// What bounds it: as in the single-CTA kernel, shared memory, the pipe of the
// precision and the passes' latencies.  A thread owns one line of every pass
// (MH N main threads); its spectrum line F^ and its sums S_p live in tensor
// memory (read per (p, q) from L2 and from shared memory before); for N = 32
// a warp is one plane k1, so the first two passes need no barrier at all
// between them (N = 24: groups of 4 planes, 3 warps).  The third pass releases
// the work cube as soon as its values are in registers.  NQ more threads
// transform the Nyquist planes (one line each).  In FP64 the Nyquist products,
// which need only the CTA's own tables, are added while the halves travel; FP32
// adds them after the third pass, in the order of roundings of fft_vec.cuh.
// Measured on one B200: FP32 N = 32 (16 x 24 (p, q)), 2,592 points: 114.3 ms a
// sweep against 140.5 ms for two lines per thread with scalar transforms, with
// the same roundings (120.6 ms with the Nyquist lines on main threads);
// FP64 N = 24, 576 points: 10.5 ms against 15.05 ms (11.8 ms; 10.98 ms with the
// Nyquist products after the third pass).  Handing over by one thread's
// cluster-scope mbarrier arrivals after a CTA barrier, instead of the cluster
// barrier, was 7 to 8 % slower in either.
//
// Shared memory (complex): W [MH][N][N + 1], the Nyquist planes T1 [x2 in
// X_r][x3], T2 [x1][x3], T3 [x2 in X_r][x1], F^ on them [k][line] and their
// first axis [line][k], two phase slots.
#pragma once

#include "fft_vec.cuh"
#include "tcgen05.cuh"
#include "vhs_push.cuh"
#include "vhs_variant.h"

namespace dgfs {

// OWN: the Nyquist lines have threads of their own; otherwise the first 3 N
// main threads take them beside their own lines (fewer warps, more registers
// per thread).
template <typename T, int N_, bool OWN> struct PairGeom {
  static constexpr int N = N_, H = N / 2 + 1, NY = N / 2, NN = N * N, V = N * N * N;
  static constexpr int MH = N / 2;           // k1 (x2) values per CTA
  static constexpr int Q = N / 4;
  static constexpr int LP = N + 1;           // padded line stride
  static constexpr int NM = MH * N;          // main threads, one line each
  static constexpr int NQ = (3 * N + 31) / 32 * 32;  // threads with a Nyquist line (whole warps)
  static constexpr int NT = NM + (OWN ? NQ : 0);
  static constexpr int GT = N == 32 ? 32 : 4 * N;    // threads whose planes a second pass needs
  static constexpr int PHS = 3 * N + 4;
  static constexpr int WD = sizeof(T) / 4;
  // tensor memory columns: per main warp 2 N values of F^, then N of S
  static constexpr int TW = 3 * N * WD, TUSED = (NM / 32 + 3) / 4 * TW;
  static constexpr int TCOLS = TUSED <= 256 ? 256 : 512;
  static constexpr int OFF_W = 0;                        // [MH][N][LP]
  static constexpr int OFF_T1 = OFF_W + MH * N * LP;     // [MH][N]
  static constexpr int OFF_T2 = OFF_T1 + MH * N;         // [N][N]
  static constexpr int OFF_T3 = OFF_T2 + NN;             // [MH][LP]
  static constexpr int OFF_N = OFF_T3 + MH * LP;         // [N][3 N]
  static constexpr int OFF_X = OFF_N + 3 * NN;           // [3 N][LP]
  static constexpr int OFF_PH = OFF_X + 3 * N * LP;      // [2][PHS]
  static constexpr int SMEM = (OFF_PH + 2 * PHS) * 2 * (int)sizeof(T);  // bytes
  static constexpr int SLICE = H * NN;                   // F in the scratch, [k3][k1][k2]
  // gain spectrum of a CTA: FP64 the lines k1 <= N/2, FP32 every line for
  // k3 <= N/2; the rest is the conjugate mirror
  static constexpr int GL = sizeof(T) == 4 ? NM : (Q + 1) * N;  // lines
  static constexpr int GK = sizeof(T) == 4 ? H : N;             // entries of a line
  static constexpr int GSL = GL * GK;                           // [k3][line]
  static constexpr int XSLAB = MH * MH * N;              // entries per staging buffer [slot][j][x3]
  // scratch per pair: F, the gain spectra of both CTAs (which double as the
  // exchange buffer of the forward transform of f), [2 CTAs][2] staging
  static constexpr int SCRATCH = SLICE + 2 * GSL + 4 * XSLAB;
  static_assert(N % 8 == 0 && NM % 32 == 0 && NM % GT == 0 && GT % 32 == 0, "thread roles");
  static_assert(2 * GSL >= SLICE, "exchange buffer");
};

template <int N> __device__ __forceinline__ int pair_owner(int k1) {
  constexpr int Q = N / 4, MH = N / 2;
  return (k1 < Q || k1 == MH || k1 > N - Q) ? 0 : 1;
}
template <int N> __device__ __forceinline__ int pair_kinv(int k1) {
  constexpr int Q = N / 4, MH = N / 2;
  return k1 < Q ? k1 : k1 == MH ? Q : k1 > N - Q ? k1 - N + MH : k1 < MH ? k1 - Q : k1 - Q - 1;
}
template <int N> __device__ __forceinline__ int pair_kmap(int r, int l) {
  constexpr int Q = N / 4, MH = N / 2;
  return r == 0 ? (l < Q ? l : l == Q ? MH : l + N - MH) : (l < Q ? l + Q : l + Q + 1);
}

__device__ __forceinline__ void cl_sync() {
  cl_arrive();
  cl_wait();
}

template <typename T, int NV, bool OWN>
__global__ void __launch_bounds__(PairGeom<T, NV, OWN>::NT, 1) vhs_pair_kernel(const VhsArgs<T> a) {
  using G = PairGeom<T, NV, OWN>;
  using C = vx<T>;   // in registers
  using CM = cx<T>;  // in the tables and the scratch
  constexpr int N = G::N, NY = G::NY, NN = G::NN, V = G::V, LP = G::LP, NM = G::NM, MH = G::MH, Q = G::Q;
  constexpr int NT = G::NT, GT = G::GT, PHS = G::PHS, WD = G::WD;
  constexpr bool ROT = sizeof(T) == 8;  // F^ = (1 + i) F, else F
  constexpr int B_T = 1, B_N = 2, B_G = 3;  // named barriers: old and new Nyquist tables, groups

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
  __shared__ double sMom[5];
  __shared__ uint32_t s_tmem;
  __shared__ __align__(8) uint64_t s_read;  // every main warp has read its part of the work cube
  __shared__ int s_gave_up;

  cg::cluster_group cluster = cg::this_cluster();
  const int r = (int)cluster.block_rank();
  const int tid = threadIdx.x;
  const bool is_main = tid < NM;
  const int tq = OWN ? tid - NM : tid;  // Nyquist line
  const bool nyq_warp = tq >= 0 && tq < G::NQ;
  const int cid = blockIdx.x / 2, ncl = gridDim.x / 2;
  CM* const Fg = a.fc + (size_t)cid * G::SCRATCH;
  CM* const Xf = Fg + G::SLICE;            // exchange buffer of the forward transform of f
  CM* const fC = Xf + r * G::GSL;          // this CTA's gain spectrum
  CM* const Xs = Xf + 2 * G::GSL;          // staging: [rank][buffer][slot][j][x3]
  const int npq = a.P * a.M;
  // a main thread's line in every pass: hi = plane slot (or x2 - MH r in the
  // third pass), lo = k2 or x3
  const int lo = tid % N, hi = tid / N, wid = tid / 32;
  const int k1 = pair_kmap<N>(r, hi), x2 = MH * r + hi;
  C* const w1p = sW + tid * LP;                // line (slot, k2) along k3
  C* const w2p = sW + hi * N * LP + lo;        // line (slot, x3) along k2: stride LP
  C* const w3p = sW + x2 * LP + lo;            // line (x2, x3) along the slots: stride N LP
  const bool gain_line = !ROT || hi < Q || (hi == Q && r == 0);  // FP64: k1 <= N/2
  uint32_t peer = (uint32_t)(r ^ 1);
  int xb = 0;  // staging buffer of the next exchange
  auto xmine = [&]() { return Xs + (size_t)(r * 2 + xb) * G::XSLAB + lo; };
  auto xpeer = [&]() { return (const CM*)(Xs + (size_t)((r ^ 1) * 2 + xb) * G::XSLAB + lo); };

  if (tid == 0) {
    mbar_init(&s_read, NM / 32);
    s_gave_up = 0;
  }
  if (tid < 32) tmem_alloc(&s_tmem, G::TCOLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // this thread's lane and columns: F^ of line (k1, k2), then S of (x2, x3)
  const uint32_t tmF = s_tmem + ((uint32_t)(wid % 4 * 32) << 16) + wid / 4 * G::TW, tmS = tmF + 2 * N * WD;
  uint32_t rphase = 0;  // parity of s_read's current phase
  auto load_line = [&](C (&x)[N]) {
    uint32_t t[2 * N * WD];
    tm_load(tmF, t);
    tm_wait(t);
#pragma unroll
    for (int k = 0; k < N; ++k) x[k] = vmk(tm_get(t, 2 * k, T(0)), tm_get(t, 2 * k + 1, T(0)));
  };
  // the planes of this thread's group are complete in the work cube
  auto group_sync = [&]() {
    if constexpr (GT == 32) __syncwarp();
    else bar_sync(B_G + tid / GT, GT);
  };
  // second pass of an inverse transform: of the N outputs (index x2) the MH
  // with x2 in X_r stay in the work cube, the others go to this CTA's staging
  // buffer [slot][x2 - MH (1 - r)][x3] for the peer
  auto pass2_out = [&]() {
    C x[N];
#pragma unroll
    for (int j = 0; j < N; ++j) x[j] = w2p[j * LP];
    vfft<N, +1>(x);
    CM* const xs = xmine() + hi * MH * N;
#pragma unroll
    for (int j = 0; j < MH; ++j) {
      w2p[(MH * r + j) * LP] = r ? x[MH + j] : x[j];
      __stcg(xs + j * N, to_c(r ? x[j] : x[MH + j]));
    }
  };
  // third-pass line along k1: the planes of this CTA from its work cube, the
  // others from the peer's staging buffer
  auto load3 = [&](C (&x)[N]) {
    const CM* const xp = xpeer() + hi * N;
#pragma unroll
    for (int k = 0; k < N; ++k)
      x[k] = pair_owner<N>(k) == r ? w3p[pair_kinv<N>(k) * N * LP] : from_c(__ldcg(xp + pair_kinv<N>(k) * MH * N));
    xb ^= 1;
  };
  constexpr int NPH = (3 * N + G::NQ - 1) / G::NQ;
  static_assert(NPH == 1, "one phase entry per Nyquist thread");
  auto phase_fetch = [&](int pq) -> CM {
    return nyq_warp && tq < 3 * N ? a.phase[(size_t)pq * 3 * N + tq] : mk<CM>(T(0), T(0));
  };
  auto phase_store = [&](CM e, int slot) {
    if (nyq_warp && tq < 3 * N) {
      CM* dst = sPh + slot * PHS;
      dst[tq] = e;
      if (tq % N == NY) {
        const CM ce = mk<CM>(e.x, -e.y);
        dst[3 * N + tq / N] = mul_r(ce, ce);
      }
    }
  };

  const int which = tq / N, jn = tq % N;
  const bool p3 = which == 2;
  auto nyq_first = [&](int slot) {
    // n F^ on the Nyquist planes (vhs_cube.cuh): plane 1 (k1 = N/2)
    // lines over k3, plane 2 (k2 = N/2) lines over k3, plane 3
    // (k3 = N/2) lines over k2; one coefficient per line
    if (tq < 3 * N) {
      const CM* ph = sPh + slot * PHS;
      const CM th1 = ph[3 * N], th2 = ph[3 * N + 1], th3 = ph[3 * N + 2];
      const CM Eb = mul_r(ph[which == 0 ? NY : jn], ph[which == 0 ? N + jn : p3 ? 2 * N + NY : N + NY]);
      const CM tb = p3 ? th3 : which == 1 ? th2 : jn == NY ? mul_r(th1, th2) : th1;
      const CM tb3 = mul_r(tb, th3);
      CM B = mul_1m(Eb, tb);
      CM B3 = p3 ? mk<CM>(T(0), T(0)) : mul_1m(Eb, tb3);
      if (which != 0 && jn == NY) B = B3 = mk<CM>(T(0), T(0));
      const CM A = mk<CM>(T(0.5) * (B.x + B.y), T(0.5) * (B.y - B.x));
      const CM A3 = mk<CM>(T(0.5) * (B3.x + B3.y), T(0.5) * (B3.y - B3.x));
      const CM* ev = ph + (p3 ? N : 2 * N);
      C x[N];
#pragma unroll
      for (int k = 0; k < N; ++k) x[k] = sN[k * 3 * N + tq];
      vfft_scaled<N, 1>(x, [&](int k) { return re_mul(k == NY ? A3 : A, ev[k]); });
#pragma unroll
      for (int k = 0; k < N; ++k) sX[tq * LP + k] = x[k];
    }
  };
  auto nyq_second = [&]() {
    // second axes: columns x3 of planes 1 and 2, the columns x2 of
    // plane 3 that this CTA's third pass reads
    if (tq < 2 * N || (p3 && jn / MH == r)) {
      C x[N];
#pragma unroll
      for (int i = 0; i < N; ++i) x[i] = sX[(which * N + i) * LP + jn];
      vfft<N, 1>(x);
      if (which == 0) {  // rows x2 of this CTA's half
#pragma unroll
        for (int i = 0; i < MH; ++i) sT1[i * N + jn] = r ? x[MH + i] : x[i];
      } else {
        C* const d = p3 ? sT3 + (jn % MH) * LP : sT2 + jn;
        const int de = p3 ? 1 : N;
#pragma unroll
        for (int i = 0; i < N; ++i) d[i * de] = x[i];
      }
    }
  };

  const int npts = a.pcount ? min(a.npts, *a.pcount) : a.npts;
#pragma unroll 1
  for (int ip = cid; ip < npts; ip += ncl) {
    const int pt = a.plist ? a.plist[a.pt0 + ip] : a.pt0 + ip;
    // listed ids come from device memory: both CTAs read the same entry and
    // skip together, so the cluster barriers stay paired
    if ((unsigned)pt >= (unsigned)(a.nupts * a.neles)) continue;
    const int upt = pt / a.neles, elem = pt % a.neles;

    // ---- F = FFT(f) / V into the scratch, k3 <= N/2 ------------------------
    // lines (x1 = MH r + hi, x2 = lo) along x3, then (x1, k3) along x2, then
    // through the scratch to lines (k2, k3) along x1
    if (is_main) {
      const int64_t b0 = soa_ix(upt, a.ldim, elem, (int64_t)((MH * r + hi) * N + lo) * N, V, a.soasz);
      C x[N];
#pragma unroll
      for (int k = 0; k < N; ++k) x[k] = vmk(a.f[b0 + (int64_t)k * a.soasz], T(0));
      vfft<N, -1>(x);
#pragma unroll
      for (int k = 0; k <= NY; ++k) w1p[k] = x[k];
    }
    __syncthreads();
#pragma unroll 1
    for (int t = tid; t < MH * G::H; t += NT) {
      const int x1l = t / G::H, k3 = t % G::H;
      C x[N];
#pragma unroll
      for (int j = 0; j < N; ++j) x[j] = sW[(x1l * N + j) * LP + k3];
      vfft<N, -1>(x);
#pragma unroll
      for (int j = 0; j < N; ++j) Xf[(k3 * N + MH * r + x1l) * N + j] = to_c(x[j]);
    }
    cl_sync();  // the exchange buffer is complete (cluster-scope release/acquire)
#pragma unroll 1
    for (int t = tid; t < MH * G::H; t += NT) {
      const int k2 = MH * r + t / G::H, k3 = t % G::H;
      const T iv = T(1) / T(V);
      C x[N];
#pragma unroll
      for (int i = 0; i < N; ++i) x[i] = from_c(__ldcg(Xf + (k3 * N + i) * N + k2));
      vfft<N, -1>(x);
#pragma unroll
      for (int i = 0; i < N; ++i) Fg[(k3 * N + i) * N + k2] = to_c(vmul(x[i], vmk(iv, iv)));
    }
    cl_sync();  // F complete in the scratch; the exchange buffer may be reused
    // F^ at (k1, k2, k3) from the half spectrum (written by both CTAs:
    // read through L2)
    auto Fat = [&](int i1, int i2, int i3) -> C {
      const bool mir = i3 > NY;
      const CM c = __ldcg(Fg + (mir ? ((N - i3) * N + (N - i1) % N) * N + (N - i2) % N : (i3 * N + i1) * N + i2));
      const C v = vmk(c.x, mir ? -c.y : c.y);
      return ROT ? mul_1i<1>(v) : v;
    };
    if (is_main) {
      uint32_t t[2 * N * WD];
#pragma unroll
      for (int k = 0; k < N; ++k) {
        const C v = Fat(k1, lo, k);
        tm_put(t, 2 * k, cre(v));
        tm_put(t, 2 * k + 1, cim(v));
      }
      tm_store(tmF, t);
      tmem_store_wait();
    }
    if (nyq_warp) {
#pragma unroll 1
      for (int t = tq; t < 3 * NN; t += G::NQ) {
        const int k = t / (3 * N), line = t % (3 * N), which = line / N, j = line % N;
        sN[t] = which == 0 ? Fat(NY, j, k) : which == 1 ? Fat(j, NY, k) : Fat(j, k, NY);
      }
      phase_store(phase_fetch(0), 0);
    }
    __syncthreads();

    // ---- gain: fC = sum_p w1_p FFT(sum_q Re S_pq) ---------------------------
    // Both kinds of threads run the same sequence of cluster barriers: one per
    // (p, q) and one per p, and one CTA barrier per p.
    if (is_main) {
      int slot = 0;
#pragma unroll 1
      for (int p = 0; p < a.P; ++p) {
#pragma unroll 1
        for (int q = 0; q < a.M; ++q) {
          CM phn = mk<CM>(T(0), T(0));
          if (!OWN && nyq_warp) {
            const int pq = p * a.M + q;
            if (pq + 1 < npq) phn = phase_fetch(pq + 1);
            nyq_first(slot);
            phase_store(phn, slot ^ 1);
          }
          // pass 1: m F^ along k3 (vhs_cube.cuh)
          {
            const CM* ph = sPh + slot * PHS;
            const CM E12 = mul_r(ph[k1], ph[N + lo]);
            const CM th1 = ph[3 * N], th2 = ph[3 * N + 1];
            const CM t12 = k1 != NY ? th2 : lo == NY ? mul_r(th1, th2) : th1;
            const CM Et = k1 == NY || lo == NY ? mul_r(E12, t12) : E12;
            const CM s0 = cadd(E12, Et), s3 = cadd(E12, mul_s(Et, ph[3 * N + 2]));
            const CM A = mk<CM>(T(0.5) * (s0.x + s0.y), T(0.5) * (s0.y - s0.x));
            const CM A3 = mk<CM>(T(0.5) * (s3.x + s3.y), T(0.5) * (s3.y - s3.x));
            C x[N];
            load_line(x);
            // e3[N - k] = conj e3[k]
            vfft_scaled<N, 1>(x, [&](int k) {
              const CM e = ph[2 * N + (k <= NY ? k : N - k)];
              return re_mul(k == NY ? A3 : A, k <= NY ? e : mk<CM>(e.x, -e.y));
            });
            mbar_wait_bounded(&s_read, rphase ^ 1, a.err, &s_gave_up);  // the previous cube is read
#pragma unroll
            for (int k = 0; k < N; ++k) w1p[k] = x[k];
          }
          slot ^= 1;
          // done with the Nyquist tables of the previous (p, q)
          if (!OWN && nyq_warp) {
            bar_sync(B_T, NT);
            nyq_second();
          } else {
            bar_arrive(B_T, NT);
          }
          group_sync();
          pass2_out();
          cl_arrive();
          // S += Re R^2 + Re Nq^2 on this thread's third-pass line, Nq = s1 T1(x2,
          // x3) + s2 T2(x1, x3) + s3 T3(x1, x2) with s = (-1)^x.  FP64 adds
          // Re Nq^2 while the halves travel; FP32 both at once after the third
          // pass, in the order in which they are rounded
          bar_sync(B_N, NT);    // the Nyquist tables are complete
          constexpr int SC = 8;  // values per step
          const T s2 = (x2 & 1) ? T(-1) : T(1), s3 = (lo & 1) ? T(-1) : T(1);
          const C t1 = sT1[tid], t1n = vmul(t1, vmk(T(-1), T(-1))), c2 = vmk(s2, s2), c3 = vmk(s3, s3);
          auto nyq_at = [&](int i) {
            return vfma(sT3[hi * LP + i], c3, vfma(sT2[i * N + lo], c2, (i & 1) ? t1n : t1));
          };
          // S <- f(i, S) over the line
          auto update = [&](auto&& f) {
            tmem_store_wait();
            sfor<0, N / SC>([&](auto cc) {
              constexpr int c = decltype(cc)::value;
              uint32_t t[SC * WD];
              tm_load(tmS + SC * c * WD, t);
              tm_wait(t);
#pragma unroll
              for (int h = 0; h < SC; ++h) tm_put(t, h, f(SC * c + h, tm_get(t, h, T(0))));
              tm_store(tmS + SC * c * WD, t);
            });
          };
          if constexpr (ROT) {
            update([&](int i, T s) {
              const C n = nyq_at(i);
              return fma(cre(n), cim(n), q == 0 ? T(0) : s);
            });
          }
          cl_wait();            // both halves staged
          // pass 3: lines (x2, x3) along k1
          C x[N];
          load3(x);
          __syncwarp();
          if (tid % 32 == 0) mbar_arrive(&s_read);  // this warp's part of the cube may be overwritten
          rphase ^= 1;
          vfft<N, 1>(x);
          if constexpr (ROT) update([&](int i, T s) { return fma(cre(x[i]), cim(x[i]), s); });
          else update([&](int i, T s) { return add_squares(x[i], nyq_at(i), q == 0 ? T(0) : s); });
        }

        // fC += w1_p FFT(S_p) on the gain lines: lines (x2, x3) along x1
        // from S (each thread to the entries it read last), the exchange to
        // k-slabs, lines (k1, x3) along x2, lines (k1, k2) along x3
        {
          C x[N];
          uint32_t t[N * WD];
          tmem_store_wait();
          tm_load(tmS, t);
          tm_wait(t);
#pragma unroll
          for (int i = 0; i < N; ++i) x[i] = vmk(tm_get(t, i, T(0)), T(0));
          vfft<N, -1>(x);
          CM* const xs = xmine() + hi * N;
#pragma unroll
          for (int k = 0; k < (ROT ? NY + 1 : N); ++k) {
            if (pair_owner<N>(k) == r) w3p[pair_kinv<N>(k) * N * LP] = x[k];
            else __stcg(xs + pair_kinv<N>(k) * MH * N, to_c(x[k]));
          }
        }
        cl_sync();  // both halves staged
        if (gain_line) {
          const CM* const xp = xpeer() + hi * MH * N;
          C x[N];
#pragma unroll
          for (int j = 0; j < N; ++j) x[j] = j / MH == r ? w2p[j * LP] : from_c(__ldcg(xp + (j % MH) * N));
          vfft<N, -1>(x);
#pragma unroll
          for (int j = 0; j < N; ++j) w2p[j * LP] = x[j];
        }
        xb ^= 1;
        __syncthreads();
        if (gain_line) {
          const T* w1 = a.w1t + (size_t)p * V + k1 * N + lo;
          CM* const fca = fC + tid;
          C x[N];
#pragma unroll
          for (int k = 0; k < N; ++k) x[k] = w1p[k];
          vfft<N, -1>(x);
          // read-modify-write in steps of 8: the loads of a step issued
          // together, fewer live registers than the whole line
#pragma unroll
          for (int k0 = 0; k0 < G::GK; k0 += 8) {
            C acc[8];
            if (p > 0) {
#pragma unroll
              for (int k = 0; k < 8 && k0 + k < G::GK; ++k) acc[k] = from_c(fca[(k0 + k) * G::GL]);
            }
#pragma unroll
            for (int k = 0; k < 8 && k0 + k < G::GK; ++k) {
              const T w = __ldg(w1 + (k0 + k) * NN);
              const C v = vmul(x[k0 + k], vmk(w, w));
              fca[(k0 + k) * G::GL] = to_c(p > 0 ? vadd(acc[k], v) : v);
            }
          }
        }
      }
    } else {
      int slot = 0;
#pragma unroll 1
      for (int p = 0; p < a.P; ++p) {
#pragma unroll 1
        for (int q = 0; q < a.M; ++q) {
          const int pq = p * a.M + q;
          const CM phn = pq + 1 < npq ? phase_fetch(pq + 1) : mk<CM>(T(0), T(0));
          nyq_first(slot);
          phase_store(phn, slot ^ 1);
          slot ^= 1;
          bar_sync(B_T, NT);  // every first axis is done, and no main thread reads the old tables
          nyq_second();
          bar_arrive(B_N, NT);
          cl_sync();
        }
        cl_sync();
        __syncthreads();
      }
    }
    __syncthreads();

    // ---- Q = prefac (Re IFFT(fC) - f Re IFFT(b2 F)) ----------------------------
    // Two inverse transforms: of b2 F^ (its real part, the collision
    // frequency, kept where S was), then of the gain spectrum.  The staging
    // buffer's index is a main thread's business; every thread takes the
    // barriers.
    double lam[5] = {0, 0, 0, 0, 0}, mom[5] = {0, 0, 0, 0, 0};
    // bank entries v = i N^2 + x2 N + x3 are b0 + i st
    const int64_t b0 = soa_ix(upt, a.ldim, elem, (int64_t)x2 * N + lo, V, a.soasz), st = (int64_t)NN * a.soasz;
#pragma unroll 1
    for (int t = 0; t < 2; ++t) {
      if (is_main) {
        C x[N];
        if (t == 0) {
          const T* b2 = a.b2t + k1 * N + lo;
          load_line(x);
#pragma unroll
          for (int k = 0; k < N; ++k) {
            const T b = __ldg(b2 + k * NN);
            x[k] = vmul(x[k], vmk(b, b));
          }
        } else {
          const CM* const src = fC + tid;
          const CM* const srm = fC + pair_kinv<N>((N - k1) % N) * N + (N - lo) % N;  // the mirrored line
#pragma unroll
          for (int k = 0; k < N; ++k) {
            const bool mir = ROT ? !gain_line : k > NY;
            const CM c = mir ? srm[(N - k) % N * G::GL] : src[k * G::GL];
            x[k] = vmk(c.x, mir ? -c.y : c.y);
          }
        }
        vfft<N, 1>(x);
#pragma unroll
        for (int k = 0; k < N; ++k) w1p[k] = x[k];
        group_sync();
        pass2_out();
      }
      cl_sync();
      if (is_main) {
        C x[N];
        load3(x);
        vfft<N, 1>(x);
        constexpr int SC = 8;
        sfor<0, N / SC>([&](auto cc) {
          constexpr int c = decltype(cc)::value;
          uint32_t w[SC * WD];
          if (t == 0) {
#pragma unroll
            for (int h = 0; h < SC; ++h) tm_put(w, h, cre(x[SC * c + h]));
          } else {
            tm_load(tmS + SC * c * WD, w);
            T fl[SC];
#pragma unroll
            for (int h = 0; h < SC; ++h) fl[h] = a.f[b0 + (SC * c + h) * st];
            tm_wait(w);
#pragma unroll
            for (int h = 0; h < SC; ++h) {
              const int i = SC * c + h;
              const T qq = a.prefac * (cre(x[i]) - fl[h] * tm_get(w, h, T(0)));
              tm_put(w, h, qq);
              if (!a.project) a.Q[b0 + i * st] = qq;
            }
            if (a.project) {
#pragma unroll
              for (int h = 0; h < SC; ++h) {
                const int v = (SC * c + h) * NN + x2 * N + lo;
                const double c0 = a.cvec[v], c1 = a.cvec[V + v], c2 = a.cvec[2 * V + v];
                const double d = (double)tm_get(w, h, T(0));
                mom[0] += d;
                mom[1] += d * c0;
                mom[2] += d * c1;
                mom[3] += d * c2;
                mom[4] += d * (c0 * c0 + c1 * c1 + c2 * c2);
              }
            }
          }
          tm_store(tmS + SC * c * WD, w);
        });
        tmem_store_wait();
      }
      __syncthreads();
    }

    // the optional FP64 projection onto zero mass, momentum and energy over
    // both halves
    if (a.project) {
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
        sMom[tid] = s;
      }
      cl_sync();  // both halves' moments in place
      double mt[5];
#pragma unroll
      for (int k = 0; k < 5; ++k) mt[k] = sMom[k] + cluster.map_shared_rank(sMom, (int)peer)[k];
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        double s = 0;
#pragma unroll
        for (int j = 0; j < 5; ++j) s += a.ginv[k * 5 + j] * mt[j];
        lam[k] = s;
      }
      if (is_main) {
        constexpr int SC = 8;
        sfor<0, N / SC>([&](auto cc) {
          constexpr int c = decltype(cc)::value;
          uint32_t w[SC * WD];
          tm_load(tmS + SC * c * WD, w);
          tm_wait(w);
#pragma unroll
          for (int h = 0; h < SC; ++h) {
            const int v = (SC * c + h) * NN + x2 * N + lo;
            const double c0 = a.cvec[v], c1 = a.cvec[V + v], c2 = a.cvec[2 * V + v];
            a.Q[b0 + (SC * c + h) * st] =
                (T)((double)tm_get(w, h, T(0)) -
                    (lam[0] + lam[1] * c0 + lam[2] * c1 + lam[3] * c2 + lam[4] * (c0 * c0 + c1 * c1 + c2 * c2)));
          }
        });
      }
    }
    // the next point rewrites the scratch and the moments: both CTAs done
    cl_sync();
  }
  if (tid < 32) tmem_dealloc(s_tmem, G::TCOLS);
  cl_sync();  // no CTA leaves while the peer may still address its memory
}

}  // namespace dgfs
