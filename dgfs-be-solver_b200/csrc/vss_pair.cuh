// Two-CTA binary-mixture VSS kernel (FP32, N = 24).
//
// The operator of vss_push.cuh (one collision pair (p, q) of frfs's DGFSBi
// VSS model, frfs/solvers/dgfsbi/scattering.py:227-315 with the kernels of
// dgfsbi/kernels/scattering/vss-gll.mako), with the point's data in the
// shared memory of a two-CTA cluster instead of an 8-CTA exchange:
//
//   F = FFT(f_p) / V, G = FFT(f_q) / V (half spectra k3 <= N/2 in the
//   pair's L2 scratch; k3 > N/2 from the conjugate mirror, f being real)
//   for every radial node x and direction y:
//     g = IFFT(e^{+i kq a} F), h = IFFT(e^{-i kp a} G)
//     QGhat += b_xy FFT(g h)
//   Q_pq = prefac (Re IFFT(QGhat) - f_p Re IFFT(c G))
//
// Data distribution (rank r of the pair): CTA r owns the k1 values K_r of
// the two-CTA VHS kernel (vhs_pair.cuh) and the x2 half X_r = [MH r,
// MH r + MH).  An inverse transform runs along k3 on the lines (k1 in K_r,
// k2), along k2 on the lines (k1 in K_r, x3), hands the other CTA the half
// of every line it owns in x2 (a staging buffer in the L2 scratch, one
// cluster barrier), and runs along k1 on the lines (x2 in X_r, x3).  The
// forward transform of g h runs the other way: along x1, the hand-over of
// the k1 the other CTA owns, along x2, along x3.
//
// 576 threads: 288 take the g field's lines and 288 the h field's (one line
// each per pass, packed FP32 transforms, fft_vec.cuh); the forward transform
// of g h uses the first 288, beside which the h threads already run the first
// two passes of the next direction.  Each thread's spectrum line and, for the
// first 288, the gain spectrum QGhat of line (k1, k2) live in tensor memory; a
// second pass waits for its group of 4 planes only.  What bounds it is the
// chain of six passes and two cluster barriers per direction.  Measured on one
// B200 (N = 24, 12 x 32 directions, four ordered pairs, 144 points): 25.3 ms
// against 32.7 ms with the spectra read from L2, QGhat in shared memory, scalar
// transforms and every pass behind a CTA barrier.  Handing over by one thread's
// cluster-scope mbarrier arrivals, with the two fields' chains decoupled,
// measured 25.1 ms and was not kept.
// Shared memory (complex float): Wg, Wh [MH][N][N+1], the h field after its
// third pass [x1][line], two phase slots [2 fields][3][N]: 173 KB.
#pragma once

#include "vhs_pair.cuh"
#include "vss_push.cuh"

namespace dgfs {

template <int N_> struct VssPairGeom {
  static constexpr int N = N_, H = N / 2 + 1, NY = N / 2, NN = N * N, V = N * N * N;
  static constexpr int MH = N / 2, LP = N + 1;
  static constexpr int NL = MH * N;                  // lines of a pass and field
  static constexpr int NT = 2 * NL;                  // threads: a g line and an h line each
  static constexpr int GT = 4 * N;                   // threads of a group of 4 planes
  static constexpr int WSZ = MH * N * LP;            // cx per work cube
  static constexpr int OFF_WG = 0, OFF_WH = WSZ, OFF_SH = 2 * WSZ;
  static constexpr int OFF_PH = OFF_SH + N * NL;     // [2 slots][2 fields][3][N]
  static constexpr int SMEM_CX = OFF_PH + 2 * 6 * N;
  static constexpr int SLICE = H * NN;               // half spectrum in the scratch
  static constexpr int XSLAB = MH * MH * N;          // staging buffer [k1l][j][x3]
  // scratch per pair: F, G, staging of the inverse transforms [2 CTAs][2
  // alternating][2 fields] and of the forward one [2 CTAs][2]
  static constexpr int SCRATCH = 2 * SLICE + 12 * XSLAB;
  static constexpr int TW = 4 * N;                   // tensor memory columns per warp: line, QGhat
  static constexpr int TCOLS = 512;
  static_assert(NT % 32 == 0 && NL % 32 == 0 && GT % 32 == 0 && NL % GT == 0 && NT <= 1024, "thread layout");
  static_assert((NT / 32 + 3) / 4 * TW <= TCOLS, "tensor memory");
};

template <int N>
__global__ void __launch_bounds__(VssPairGeom<N>::NT, 1) vss_pair_kernel(const VssArgs<float> a) {
  using G = VssPairGeom<N>;
  using C = cpx;
  using CM = float2;
  constexpr int H = G::H, NY = G::NY, NN = G::NN, V = G::V, LP = G::LP, MH = G::MH, NL = G::NL, GT = G::GT;

  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* const base = reinterpret_cast<C*>(smem_raw);
  CM* const sPh = reinterpret_cast<CM*>(base + G::OFF_PH);
  __shared__ uint32_t s_tmem;

  cg::cluster_group cluster = cg::this_cluster();
  const int r = (int)cluster.block_rank();
  const int tid = threadIdx.x, wid = tid / 32;
  // field of this thread (0: g from F, 1: h from G) and its line in a pass:
  // hi = L / N (k1l, or x2l in the third pass), lo = L % N (k2, x3)
  const int fld = tid / NL, L = tid % NL, hi = L / N, lo = L % N;
  const int k1 = pair_kmap<N>(r, hi), x2 = MH * r + hi;
  C* const sW = base + (fld ? G::OFF_WH : G::OFF_WG);
  C* const w1p = sW + L * LP;               // line (k1l, k2) along k3
  C* const w2p = sW + hi * N * LP + lo;     // line (k1l, x3) along k2
  C* const w3p = sW + x2 * LP + lo;         // line (x2, x3) along k1l: stride N LP
  C* const sH = base + G::OFF_SH + L;       // h of line L: stride NL
  const int cid = blockIdx.x / 2, ncl = gridDim.x / 2;
  CM* const Fg = a.fc + (size_t)cid * G::SCRATCH;
  CM* const Gg = Fg + G::SLICE;
  CM* const Xi = Gg + G::SLICE + fld * G::XSLAB + lo;  // inverse staging [rank][parity][field][k1l][j][x3]
  CM* const Xf = Gg + G::SLICE + 8 * G::XSLAB + lo;    // forward staging [rank][parity][k1l][x2l][x3]
  const int npq = a.P * a.M;
  // a spectrum value at (k1, k2, k3) from a half spectrum in the scratch
  auto at = [&](const CM* S, int i1, int i2, int i3) -> C {
    if (i3 <= NY) return from_c(__ldcg(S + (i3 * N + i1) * N + i2));
    const CM c = __ldcg(S + ((N - i3) * N + (N - i1) % N) * N + (N - i2) % N);
    return vmk(c.x, -c.y);
  };
  auto group_sync = [&]() { bar_sync(1 + tid / GT, GT); };

  if (tid < 32) tmem_alloc(&s_tmem, G::TCOLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmF = s_tmem + ((uint32_t)(wid % 4 * 32) << 16) + wid / 4 * G::TW, tmQ = tmF + 2 * N;

  // first pass of an inverse transform is in the work cube: the second pass
  // (lines (k1l, x3) along k2) of exchange `par`; outputs with x2 in X_r stay
  // in the cube, the others go to the staging buffer
  auto pass2_out = [&](int par) {
    group_sync();
    C x[N];
#pragma unroll
    for (int j = 0; j < N; ++j) x[j] = w2p[j * LP];
    cfft<N, 1>(x);
    CM* const xs = Xi + (r * 2 + par) * 2 * G::XSLAB + hi * MH * N;
#pragma unroll
    for (int j = 0; j < MH; ++j) {
      w2p[(MH * r + j) * LP] = r ? x[MH + j] : x[j];
      __stcg(xs + j * N, to_c(r ? x[j] : x[MH + j]));
    }
  };
  // passes 1 and 2 of direction pq's field
  auto inverse12 = [&](int pq) {
    const CM* ph = sPh + (pq & 1) * 6 * N + fld * 3 * N;
    const CM e12 = cmul(ph[k1], ph[N + lo]);
    uint32_t t[2 * N];
    tm_load(tmF, t);
    tm_wait(t);
    C x[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const CM e = cmul(e12, ph[2 * N + k]);
      const float re = tm_get(t, 2 * k, 0.f), im = tm_get(t, 2 * k + 1, 0.f);
      x[k] = vmk(re * e.x - im * e.y, re * e.y + im * e.x);
    }
    cfft<N, 1>(x);
#pragma unroll
    for (int k = 0; k < N; ++k) w1p[k] = x[k];
    pass2_out(pq & 1);
  };
  // third-pass line along k1: this CTA's planes from the cube, the others
  // from the peer's staging buffer
  auto load3 = [&](C (&x)[N], int par) {
    const CM* const xp = Xi + ((r ^ 1) * 2 + par) * 2 * G::XSLAB + hi * N;
#pragma unroll
    for (int k = 0; k < N; ++k)
      x[k] = pair_owner<N>(k) == r ? w3p[pair_kinv<N>(k) * N * LP] : from_c(__ldcg(xp + pair_kinv<N>(k) * MH * N));
  };

#pragma unroll 1
  for (int ip = cid; ip < a.npts; ip += ncl) {
    const int pt = a.pt0 + ip;
    const int upt = pt / a.neles, elem = pt % a.neles;

    // ---- F = FFT(f_p) / V (field 0) and G = FFT(f_q) / V (field 1) -------
    // lines (x1 = MH r + hi, x2 = lo) along x3, then (x1l, k3) along x2,
    // through the scratch, then (k2, k3) along x1
    {
      const float* f = fld ? a.fq : a.fp;
      const int64_t b0 = soa_ix(upt, a.ldim, elem, (int64_t)((MH * r + hi) * N + lo) * N, V, a.soasz);
      C x[N];
#pragma unroll
      for (int k = 0; k < N; ++k) x[k] = vmk(f[b0 + (int64_t)k * a.soasz], 0.f);
      cfft<N, -1>(x);
#pragma unroll
      for (int k = 0; k <= NY; ++k) w1p[k] = x[k];
    }
    __syncthreads();
    // exchange buffer [k3][x1][k2] of each field: the half spectrum slot
    // itself (written by both CTAs, each its x1 half)
    CM* const S = fld ? Gg : Fg;
#pragma unroll 1
    for (int t = L; t < MH * H; t += NL) {
      const int x1l = t / H, k3 = t % H;
      C x[N];
#pragma unroll
      for (int j = 0; j < N; ++j) x[j] = sW[(x1l * N + j) * LP + k3];
      cfft<N, -1>(x);
#pragma unroll
      for (int j = 0; j < N; ++j) __stcg(S + (k3 * N + MH * r + x1l) * N + j, to_c(x[j]));
    }
    cl_sync();  // every x1 of both fields in the scratch
    // lines (k2 in this CTA's half, k3) along x1, into registers, then
    // back in place once both CTAs have read (a second barrier)
    C y[N];
    const bool fwd3 = L < MH * H;
    const int k2f = MH * r + (fwd3 ? L / H : 0), k3f = fwd3 ? L % H : 0;
    if (fwd3) {
#pragma unroll
      for (int i = 0; i < N; ++i) y[i] = from_c(__ldcg(S + (k3f * N + i) * N + k2f));
      cfft<N, -1>(y);
    }
    cl_sync();  // both CTAs hold their lines of the exchange buffer
    if (fwd3) {
      const float iv = 1.f / (float)V;
#pragma unroll
      for (int i = 0; i < N; ++i) __stcg(S + (k3f * N + i) * N + k2f, to_c(vmul(y[i], vmk(iv, iv))));
    }
    if (tid < 6 * N) sPh[tid] = a.phase[tid];
    cl_sync();  // F and G complete in the scratch
    {
      uint32_t t[2 * N];
#pragma unroll
      for (int k = 0; k < N; ++k) {
        const C v = at(S, k1, lo, k);
        tm_put(t, 2 * k, cre(v));
        tm_put(t, 2 * k + 1, cim(v));
      }
      tm_store(tmF, t);
      tmem_store_wait();
    }
    __syncthreads();

    // Per direction two cluster barriers: #1 hands over the inverse
    // transforms, #2 the forward one.  The h threads wait for #2 only after
    // the first two passes of the next direction.
    inverse12(0);
#pragma unroll 1
    for (int pq = 0; pq < npq; ++pq) {
      const CM phn = (tid < 6 * N && pq + 1 < npq) ? a.phase[(size_t)(pq + 1) * 6 * N + tid] : make_float2(0.f, 0.f);
      if (fld && pq > 0) cl_wait();  // #2 of the previous direction
      cl_sync();                     // #1: both halves staged
      // ---- pass 3: g or h on the line (x2 = MH r + hi, x3 = lo) --------------
      C x[N];
      load3(x, pq & 1);
      cfft<N, 1>(x);
      if (fld) {
#pragma unroll
        for (int i = 0; i < N; ++i) sH[i * NL] = x[i];
      }
      if (tid < 6 * N && pq + 1 < npq) sPh[((pq + 1) & 1) * 6 * N + tid] = phn;
      __syncthreads();  // h and the next phases in place
      // ---- g h, forward along x1; the k1 the peer owns go to its buffer ------
      if (!fld) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const C h = sH[i * NL];
          x[i] = vmk(cre(x[i]) * cre(h) - cim(x[i]) * cim(h), cre(x[i]) * cim(h) + cim(x[i]) * cre(h));
        }
        cfft<N, -1>(x);
        CM* const xs = Xf + (r * 2 + (pq & 1)) * G::XSLAB + hi * N;
#pragma unroll
        for (int k = 0; k < N; ++k) {
          if (pair_owner<N>(k) == r) w3p[pair_kinv<N>(k) * N * LP] = x[k];
          else __stcg(xs + pair_kinv<N>(k) * MH * N, to_c(x[k]));
        }
      }
      cl_arrive();  // #2
      if (fld) {
        if (pq + 1 < npq) inverse12(pq + 1);
        continue;
      }
      cl_wait();
      // ---- forward along x2 on the lines (k1l, x3) ----------------------------
      const CM* const xp = Xf + ((r ^ 1) * 2 + (pq & 1)) * G::XSLAB + hi * MH * N;
#pragma unroll
      for (int j = 0; j < N; ++j) x[j] = j / MH == r ? w2p[j * LP] : from_c(__ldcg(xp + (j % MH) * N));
      cfft<N, -1>(x);
#pragma unroll
      for (int j = 0; j < N; ++j) w2p[j * LP] = x[j];
      group_sync();
      // ---- forward along x3 on the lines (k1l, k2); QGhat += b FFT(g h) ------
#pragma unroll
      for (int k = 0; k < N; ++k) x[k] = w1p[k];
      cfft<N, -1>(x);
      const CM* bb = a.bt + (size_t)pq * V + k1 * N + lo;
      tmem_store_wait();
      sfor<0, N / 8>([&](auto cc) {
        constexpr int c = decltype(cc)::value;
        uint32_t t[16];
        CM b[8];
        tm_load(tmQ + 16 * c, t);
#pragma unroll
        for (int i = 0; i < 8; ++i) b[i] = __ldg(bb + (8 * c + i) * NN);
        tm_wait(t);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const C v = x[8 * c + i];
          const float q0 = pq == 0 ? 0.f : tm_get(t, 2 * i, 0.f), q1 = pq == 0 ? 0.f : tm_get(t, 2 * i + 1, 0.f);
          tm_put(t, 2 * i, q0 + b[i].x * cre(v) - b[i].y * cim(v));
          tm_put(t, 2 * i + 1, q1 + b[i].x * cim(v) + b[i].y * cre(v));
        }
        tm_store(tmQ + 16 * c, t);
      });
      if (pq + 1 < npq) inverse12(pq + 1);
    }
    if (fld) cl_wait();  // #2 of the last direction

    // ---- QG = IFFT(QGhat) (field 0), fL = IFFT(c G) (field 1) ---------------
    {
      uint32_t t[2 * N];
      tmem_store_wait();
      tm_load(fld ? tmF : tmQ, t);
      tm_wait(t);
      C x[N];
#pragma unroll
      for (int k = 0; k < N; ++k) {
        const float re = tm_get(t, 2 * k, 0.f), im = tm_get(t, 2 * k + 1, 0.f);
        if (fld) {
          const CM c = __ldg(a.c + (k1 * N + lo) * N + k);
          x[k] = vmk(re * c.x - im * c.y, re * c.y + im * c.x);
        } else {
          x[k] = vmk(re, im);
        }
      }
      cfft<N, 1>(x);
#pragma unroll
      for (int k = 0; k < N; ++k) w1p[k] = x[k];
      pass2_out(npq & 1);
      cl_sync();
      load3(x, npq & 1);
      cfft<N, 1>(x);
      if (fld) {
#pragma unroll
        for (int i = 0; i < N; ++i) sH[i * NL] = x[i];
      }
      __syncthreads();
      if (!fld) {
        // x2 = MH r + hi, x3 = lo: bank entries v = x1 N^2 + x2 N + x3
        const int64_t b0 = soa_ix(upt, a.ldim, elem, (int64_t)x2 * N + lo, V, a.soasz);
        const int64_t st = (int64_t)NN * a.soasz;
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const float qv = a.prefac * (cre(x[i]) - a.fp[b0 + i * st] * cre(sH[i * NL]));
          a.Q[b0 + i * st] = a.accumulate ? a.Q[b0 + i * st] + qv : qv;
        }
      }
    }
    // the next point rewrites the scratch and the work cubes: both CTAs done
    cl_sync();
  }
  if (tid < 32) tmem_dealloc(s_tmem, G::TCOLS);
  cl_sync();  // no CTA leaves while the peer may still address its memory
}

}  // namespace dgfs
