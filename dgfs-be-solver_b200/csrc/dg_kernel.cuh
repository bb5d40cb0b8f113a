// FR-DG advection residual over all discrete velocities.
//
// Banks are frfs's AoSoA(32) layout: value (row i, velocity v, element e) at
// i*ldim + ((e/32)*V + v)*32 + e%32, so the 32 elements of one block at one
// velocity form one coalesced 128-byte row.  A CTA of 256 threads takes one
// 32-element block (lane = element) and a chunk of 8*VPT velocities (warp w
// takes v = chunk + 8*it + w): consecutive warps read consecutive rows.  The
// element operators travel in the kernel parameters (constant bank) and every
// loop over them is unrolled, so matrix entries are FMA operands, not loads.
// The residual stages the block's element geometry (metric terms, 1/|J|,
// scaled normals, partner offsets) in shared memory once per CTA, one row of
// GS values per lane read with 16-byte loads, and reuses it for every
// velocity of the chunk.
//
//   dg_interp_kernel    uf = M0 u at the flux points (frfs/solvers/dgfs/
//                        elements.py:55-59, 'disu')
//   dg_bcsum_kernel     diffuse-wall sums over velocities in FP64
//                        (kernels/bcs/dgfs-wall-diffuse-update.mako:14-36)
//   dg_residual_kernel  R = -(1/|J|)[(M1 - M3 M2) F~ + M3 F^] with the upwind
//                        common flux at every flux point (interfaces,
//                        boundaries and faces shared with another partition),
//                        fused with the Runge-Kutta combination
//                        out = a A + b B + g (R + C)
//                        (elements.py:49-118, intcflux.mako, bccflux.mako,
//                        mpicflux.mako, rusanov.mako:46-50, negdivconf.mako,
//                        axnpby.mako)
//   dg_pack_kernel      face values at the flux points on partition faces
//                        into a send buffer (the 'pack' kernel of frfs's MPI
//                        interfaces, inters.py:61-112)
#pragma once

#include "dgfs_common.cuh"

namespace dgfs {

enum DgBcKind {
  BC_WALL_DIFFUSE = 0,
  BC_INLET = 1,
  BC_OUTLET = 2,
  BC_VANISH = 3,
  BC_WALL_SPECULAR = 4,
  BC_WALL_DIFFUSE_CYL = 5
};

template <typename T, int U, int F, int D> struct DgOps {
  T m0[F][U];
  T m132[U][D * U];
  T m3[U][F];
};

// The same operators on a tensor-product element of n x n points (upt j n + i:
// i along xi, j along eta; faces bottom, right, top, left with n flux points
// each, in ascending order), as 1D factors:
//   M0    traces l[0], l[1] at -1 and +1 along the axis across a face
//   M1    the derivative d along either axis
//   M3    lift = la (along the face) x lc[end] (across it)
// dgfs_dg_create finds them in the matrices it is given and uses them only if
// they reproduce every entry (dg_factor).
template <typename T, int n> struct DgFac {
  T l[2][n];
  T d[n][n];
  T la[n][n];
  T lc[2][n];
};

template <typename T> struct DgArgs {
  int V, neles, v0, nv;
  int64_t ldim_u;          // leading dimension of solution banks
  int64_t ldim_f;          // leading dimension of the flux-point scratch
  const T* u;              // solution bank [U][V][E] (AoSoA 32)
  T* uf;                   // flux-point values [F][V][E] (AoSoA 32)
  T* out;                  // residual / RK output bank
  const T* A;              // optional terms of out = a A + b B + g (R + C)
  const T* B;
  const T* Cq;
  T alpha, beta, gamma;
  // geometry (SoA over elements)
  const T* smats;          // [D][U][D][E]
  const T* rcpdjac;        // [U][E]
  const T* nrm;            // [F][D][E] unit outward normals
  const T* mag;            // [F][E]    |S^T n|
  const int* part;         // [F][E]    fpt_r*E + e_r, or -(b+1) for boundary b
  const T* cvx;            // [V] velocity grid
  const T* cvy;
  const T* cvz;
  // boundaries
  const int* bkind;        // [nb]
  const int* bgroup;       // [nb]
  const T* guw;            // [ngroups][3]
  const T* gfw;            // [ngroups][V]
  const int* grefl;        // [ngroups][V]
  const T* bwall;          // [nb][4] wall Ux, Uy, Uz, T per boundary point (cylinder wall)
  const double* bcvals;    // [nb][2]
  int nb;                  // boundary flux points
  // per element block: geometry rows [nblk][32][GS] and partner offsets
  // [nblk][32][PS] (>= 0: flux-bank offset of the partner at v = 0;
  // -1-b: boundary point b < nb; -1-(nb+h): row h of the halo)
  const T* geoblk;
  const int64_t* pblk;
  const T* halo;           // [nhalo][V] partner face values from other partitions
  int* err;                // set to 1 when a bounded wait of the tensor-core residual ran out
};

// Shared-memory row of one element (T values): metric terms S[k][i][kk]
// (k-major, D*D per solution point), 1/|J| (padded to a 16-byte multiple),
// |S^T n| n at the flux points [F][D]; GS pads the row so that the 16-byte
// loads of 8 consecutive lanes fall in distinct bank quads.  Partner offsets
// [F] int64 per lane, padded to PS likewise.
template <typename T, int U, int F, int D> struct DgGeo {
  static constexpr int VW = 16 / (int)sizeof(T);
  static constexpr int OS = 0, NS = U * D * D;
  static constexpr int OR = NS, NR = ((U + VW - 1) / VW) * VW;
  static constexpr int ON = OR + NR, NN = F * D;
  static constexpr int G = ON + NN;
  static constexpr int GS = sizeof(T) == 4 ? G + ((4 - G % 8) + 8) % 8 : G + ((2 - G % 4) + 4) % 4;
  static constexpr int PS = F + ((2 - F % 4) + 4) % 4;
  static_assert(NS % VW == 0 && NN % VW == 0, "16-byte sections");
};

template <typename T, int U> struct DgMassOps {
  T m12[U][U];
};

__device__ __forceinline__ int64_t aos32(int64_t row, int64_t ldim, int64_t e, int64_t v, int64_t V) {
  return row * ldim + ((e >> 5) * V + v) * 32 + (e & 31);
}

// Programmatic dependent launch.  The interp and boundary-sum kernels wait
// for their predecessor in the stream to complete (a no-op when they were
// not launched as dependents), then let their own dependent start: a
// dependent that starts early therefore finds everything before them
// complete and may read the banks (u and the Runge-Kutta terms) before its
// own wait; it reads their outputs (face values, boundary sums) only after
// that wait.  The residual never triggers early: whatever follows it starts
// after it has completed.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename T, int U, int F, int D, int VPT>
__global__ void __launch_bounds__(256) dg_interp_kernel(const DgArgs<T> a, const DgOps<T, U, F, D> op) {
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t e = (int64_t)blockIdx.x * 32 + lane;
  if (e >= a.neles) return;
  const int vend = a.v0 + a.nv;
  const int vbeg = a.v0 + (int)blockIdx.y * (8 * VPT) + w;
#pragma unroll 1
  for (int it = 0; it < VPT; ++it) {
    const int v = vbeg + 8 * it;
    if (v >= vend) break;
    const int64_t o = ((int64_t)blockIdx.x * a.V + v) * 32 + lane;
    T u[U];
    const T* up = a.u + o;
#pragma unroll
    for (int i = 0; i < U; ++i, up += a.ldim_u) u[i] = __ldg(up);
    T* fp = a.uf + o;
#pragma unroll
    for (int f = 0; f < F; ++f, fp += a.ldim_f) {
      T s = T(0);
#pragma unroll
      for (int i = 0; i < U; ++i) s = fma(op.m0[f][i], u[i], s);
      *fp = s;
    }
  }
}

// out = M12 u at the solution points of velocities [v0, v0 + nv): the
// 'invmass' kernel of DGFSElements (frfs/solvers/dgfs/elements.py:161-164),
// M12 = V^T V with V the orthonormal basis at the solution points.
template <typename T, int U>
__global__ void __launch_bounds__(256) dg_invmass_kernel(const DgArgs<T> a, const DgMassOps<T, U> op) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = (int)(t & 31);
  const int64_t w = t >> 5;
  const int v = a.v0 + (int)(w % a.nv);
  const int64_t e = (w / a.nv) * 32 + lane;
  if (e >= a.neles) return;
  T u[U];
#pragma unroll
  for (int i = 0; i < U; ++i) u[i] = a.u[aos32(i, a.ldim_u, e, v, a.V)];
#pragma unroll
  for (int r = 0; r < U; ++r) {
    T s = T(0);
#pragma unroll
    for (int i = 0; i < U; ++i) s = fma(op.m12[r][i], u[i], s);
    a.out[aos32(r, a.ldim_u, e, v, a.V)] = s;
  }
}

// Diffuse-wall sums, pass 1: block (chunk, group) reduces 32 boundary flux
// points over one chunk of the velocity range in FP64 (8 velocity lanes per
// point) and writes partials[chunk][b] = (sum_{c.n>=0} (c-Uw).n f cw,
// sum_{c.n<0} (c-Uw).n fw cw).
template <typename T, int D>
__global__ void __launch_bounds__(256) dg_bcsum_kernel(const DgArgs<T> a, const int* __restrict__ bfpt,
                                                      const int* __restrict__ bele, int nb, double cw,
                                                      int chunk, double* __restrict__ partials) {
  __shared__ double s0[8][32], s1[8][32];
  pdl_wait();
  pdl_trigger();
  const int bl = threadIdx.x & 31, vg = threadIdx.x >> 5;
  const int b = blockIdx.y * 32 + bl;
  const int vbeg = a.v0 + blockIdx.x * chunk;
  const int vend = min(a.v0 + a.nv, vbeg + chunk);
  double acc0 = 0.0, acc1 = 0.0;
  const int kind = b < nb ? a.bkind[b] : -1;
  if (kind == BC_WALL_DIFFUSE || kind == BC_WALL_DIFFUSE_CYL) {
    const int j = bfpt[b], e = bele[b], g = a.bgroup[b];
    const bool cyl = kind == BC_WALL_DIFFUSE_CYL;
    double n[D], uw[3], tw = 1.0;
#pragma unroll
    for (int d = 0; d < D; ++d) n[d] = (double)a.nrm[((int64_t)j * D + d) * a.neles + e];
#pragma unroll
    for (int d = 0; d < 3; ++d) uw[d] = cyl ? (double)a.bwall[b * 4 + d] : (double)a.guw[g * 3 + d];
    if (cyl) tw = (double)a.bwall[b * 4 + 3];
    for (int v = vbeg + vg; v < vend; v += 8) {
      const double dc[3] = {(double)a.cvx[v] - uw[0], (double)a.cvy[v] - uw[1], (double)a.cvz[v] - uw[2]};
      const double dx = dc[0], dy = dc[1], dz = dc[2];
      double fac = 0.0;
#pragma unroll
      for (int d = 0; d < D; ++d) fac += dc[d] * n[d];
      if (fac >= 0.0) {
        acc0 += fac * (double)a.uf[aos32(j, a.ldim_f, e, v, a.V)] * cw;
      } else {
        // the cylinder wall's Maxwellian exp(-|c - U|^2 / T), unnormalised
        // like the reference's (the ratio of the two sums normalises it;
        // bcs/dgfs-wall-diffuse-cyl-update.mako)
        const double fw = cyl ? exp(-(dx * dx + dy * dy + dz * dz) / tw) : (double)a.gfw[(int64_t)g * a.V + v];
        acc1 += fac * fw * cw;
      }
    }
  }
  s0[vg][bl] = acc0;
  s1[vg][bl] = acc1;
  __syncthreads();
  if (vg == 0 && b < nb) {
    double r0 = 0.0, r1 = 0.0;
    for (int k = 0; k < 8; ++k) {
      r0 += s0[k][bl];
      r1 += s1[k][bl];
    }
    partials[((int64_t)blockIdx.x * nb + b) * 2] = r0;
    partials[((int64_t)blockIdx.x * nb + b) * 2 + 1] = r1;
  }
}

// Pass 2: one warp per boundary point sums the chunks into bcvals in a
// fixed order (lane-strided partial sums, then a fixed butterfly), so the
// result is the same on every run.
__global__ void __launch_bounds__(256) dg_bcsum_finish_kernel(const int* __restrict__ bkind, int nb, int nchunks,
                                                             const double* __restrict__ partials,
                                                             double* __restrict__ bcvals, int reset) {
  pdl_wait();
  pdl_trigger();
  const int b = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (b >= nb || (bkind[b] != BC_WALL_DIFFUSE && bkind[b] != BC_WALL_DIFFUSE_CYL)) return;  // uniform per warp
  double r0 = 0.0, r1 = 0.0;
  for (int c = lane; c < nchunks; c += 32) {
    r0 += partials[((int64_t)c * nb + b) * 2];
    r1 += partials[((int64_t)c * nb + b) * 2 + 1];
  }
  for (int o = 16; o > 0; o >>= 1) {
    r0 += __shfl_xor_sync(0xffffffffu, r0, o);
    r1 += __shfl_xor_sync(0xffffffffu, r1, o);
  }
  if (lane == 0) {
    if (reset) {
      bcvals[2 * b] = r0;
      bcvals[2 * b + 1] = r1;
    } else {
      bcvals[2 * b] += r0;
      bcvals[2 * b + 1] += r1;
    }
  }
}

template <typename T> struct Vec16;
template <> struct Vec16<float> { using type = float4; };
template <> struct Vec16<double> { using type = double2; };

// n 16-byte loads from shared memory into r[0 .. n*VW)
template <typename T, int N> __device__ __forceinline__ void lds16(const T* src, T* r) {
  using V4 = typename Vec16<T>::type;
  constexpr int VW = 16 / (int)sizeof(T);
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const V4 q = reinterpret_cast<const V4*>(src)[j];
    if constexpr (VW == 4) {
      r[4 * j] = q.x; r[4 * j + 1] = q.y; r[4 * j + 2] = q.z; r[4 * j + 3] = q.w;
    } else {
      r[2 * j] = q.x; r[2 * j + 1] = q.y;
    }
  }
}

// Ghost value of boundary point b at velocity v (bccflux.mako with the
// bcs/*.mako kinds) into *val, or true where it is the interior face value;
// nmv = |S^T n| n, whose sign tests equal the unit normal's.
template <typename T, int D>
__device__ __forceinline__ bool dg_ghost(const DgArgs<T>& a, int b, int v, int64_t e, int f, const T* c, const T* nmv,
                                         T* val) {
  const int kind = a.bkind[b], g = a.bgroup[b];
  if (kind == BC_WALL_DIFFUSE || kind == BC_INLET) {
    T fac = (c[0] - a.guw[g * 3]) * nmv[0];
#pragma unroll
    for (int d = 1; d < D; ++d) fac = fma(c[d] - a.guw[g * 3 + d], nmv[d], fac);
    if (!(fac < T(0))) return true;
    const T fw = a.gfw[(int64_t)g * a.V + v];
    *val = kind == BC_INLET ? fw : fw * (T)(-a.bcvals[2 * b] / a.bcvals[2 * b + 1]);
    return false;
  }
  if (kind == BC_WALL_DIFFUSE_CYL) {
    // bcs/dgfs-wall-diffuse-cyl.mako: wall state of this boundary point
    const T* w = a.bwall + (int64_t)b * 4;
    const T dc[3] = {c[0] - w[0], c[1] - w[1], c[2] - w[2]};
    T fac = dc[0] * nmv[0];
#pragma unroll
    for (int d = 1; d < D; ++d) fac = fma(dc[d], nmv[d], fac);
    if (!(fac < T(0))) return true;
    const T mx = exp(-(dc[0] * dc[0] + dc[1] * dc[1] + dc[2] * dc[2]) / w[3]);
    *val = mx * (T)(-a.bcvals[2 * b] / a.bcvals[2 * b + 1]);
    return false;
  }
  if (kind == BC_VANISH) {
    T nc = nmv[0] * c[0];
#pragma unroll
    for (int d = 1; d < D; ++d) nc = fma(nmv[d], c[d], nc);
    *val = T(0);
    return !(nc < T(0));
  }
  if (kind == BC_WALL_SPECULAR) {
    *val = a.uf[aos32(f, a.ldim_f, e, a.grefl[(int64_t)g * a.V + v], a.V)];
    return false;
  }
  return true;  // outlet
}

// Launch shapes (the autotuner's choice, dgfs_dg_select): VPT velocities per
// warp and CTA chunk; PF = 1 loads the Runge-Kutta terms A, B, C of an
// iteration together with u, before the flux work, as one combination
// K = a A + b B + g C (U more registers); MB CTAs of 256 per SM the
// register budget is compiled for (FP32 p <= 2 needs 80 registers at
// PF = 0, FP32 p = 3 and FP64 p <= 2 128, FP64 p = 3 160).
template <typename T, int U, int F, int D, int VPT, int PF, int MB>
__global__ void __launch_bounds__(256, MB)
    dg_residual_kernel(const DgArgs<T> a, const DgOps<T, U, F, D> op) {
  using G = DgGeo<T, U, F, D>;
  __shared__ __align__(16) T sg[32 * G::GS];
  __shared__ __align__(16) int64_t sp[32 * G::PS];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  {
    const T* gs = a.geoblk + (size_t)blockIdx.x * 32 * G::GS;
    for (int i = threadIdx.x; i < 32 * G::GS; i += 256) sg[i] = gs[i];
    const int64_t* ps = a.pblk + (size_t)blockIdx.x * 32 * G::PS;
    for (int i = threadIdx.x; i < 32 * G::PS; i += 256) sp[i] = ps[i];
  }
  __syncthreads();
  const int64_t e = (int64_t)blockIdx.x * 32 + lane;
  if (e >= a.neles) return;
  const T* gl = sg + lane * G::GS;
  const int64_t* pl = sp + lane * G::PS;
  const int vend = a.v0 + a.nv;
  const int vbeg = a.v0 + (int)blockIdx.y * (8 * VPT) + w;

#pragma unroll 1
  for (int it = 0; it < VPT; ++it) {
    const int v = vbeg + 8 * it;
    if (v >= vend) break;
    const int64_t o = ((int64_t)blockIdx.x * a.V + v) * 32 + lane;

    // every bank value of this (v, e) first, so the loads overlap
    T u[U];
    {
      const T* up = a.u + o;
#pragma unroll
      for (int i = 0; i < U; ++i, up += a.ldim_u) u[i] = __ldg(up);
    }
    T K[PF ? U : 1];
    if constexpr (PF != 0) {
#pragma unroll
      for (int r = 0; r < U; ++r) {
        const int64_t ro = o + (int64_t)r * a.ldim_u;
        T k = a.Cq ? a.gamma * __ldg(a.Cq + ro) : T(0);
        if (a.A) k = fma(a.alpha, __ldg(a.A + ro), k);
        if (a.B) k = fma(a.beta, __ldg(a.B + ro), k);
        K[r] = k;
      }
    }
    // the face values come from the interp kernel: wait for it (returns at
    // once after the first iteration)
    pdl_wait();
    T urv[F];
#pragma unroll
    for (int f = 0; f < F; f += 2) {
      const longlong2 pb = reinterpret_cast<const longlong2*>(pl)[f / 2];
      urv[f] = pb.x >= 0 ? a.uf[pb.x + (int64_t)v * 32] : T(0);
      if (f + 1 < F) urv[f + 1] = pb.y >= 0 ? a.uf[pb.y + (int64_t)v * 32] : T(0);
    }
    const T c[3] = {__ldg(a.cvx + v), __ldg(a.cvy + v), __ldg(a.cvz + v)};

    // R = (M1 - M3 M2) F~ + M3 F^, accumulated term by term so that only
    // the U partial sums and u stay live
    T R[U];
#pragma unroll
    for (int r = 0; r < U; ++r) R[r] = T(0);

    // common normal fluxes |S^T n| F^ at this element's flux points
    {
      T nm[G::NN];
#pragma unroll
      for (int f = 0; f < F; ++f) {
        // scaled normals fetched where first used (16 bytes at a time)
        if ((f * D) % G::VW == 0) lds16<T, 1>(gl + G::ON + f * D, nm + f * D);
        T ul = T(0);
#pragma unroll
        for (int i = 0; i < U; ++i) ul = fma(op.m0[f][i], u[i], ul);
        const T* nmv = nm + f * D;
        T nc = nmv[0] * c[0];
#pragma unroll
        for (int d = 1; d < D; ++d) nc = fma(nmv[d], c[d], nc);
        T ur = urv[f];
        const int64_t pb = pl[f];
        if (pb < 0) {
          const int b = (int)(-pb - 1);
          if (b >= a.nb) ur = a.halo[(int64_t)(b - a.nb) * a.V + v];
          else if (dg_ghost<T, D>(a, b, v, e, f, c, nmv, &ur)) ur = ul;
        }
        // upwind flux (rusanov.mako:46-50) with the scaled normal
        const T fh = T(0.5) * nc * (ul + ur) + T(0.5) * fabs(nc) * (ul - ur);
#pragma unroll
        for (int r = 0; r < U; ++r) R[r] = fma(op.m3[r][f], fh, R[r]);
      }
    }

    // transformed flux at the solution points F~_(i,k) = (sum_kk S_ik,kk c_kk) u_k
    {
      T sm[G::NS];
#pragma unroll
      for (int k = 0; k < U; ++k)
#pragma unroll
        for (int i = 0; i < D; ++i) {
          if (((k * D + i) * D) % G::VW == 0) lds16<T, 1>(gl + G::OS + (k * D + i) * D, sm + (k * D + i) * D);
          T s = T(0);
#pragma unroll
          for (int kk = 0; kk < D; ++kk) s = fma(sm[(k * D + i) * D + kk], c[kk], s);
          const T ft = s * u[k];
#pragma unroll
          for (int r = 0; r < U; ++r) R[r] = fma(op.m132[r][i * U + k], ft, R[r]);
        }
    }

    T rj[G::NR];
    lds16<T, G::NR / G::VW>(gl + G::OR, rj);
    if constexpr (PF != 0) {
      T* op_ = a.out + o;
#pragma unroll
      for (int r = 0; r < U; ++r, op_ += a.ldim_u) *op_ = fma(a.gamma, -rj[r] * R[r], K[r]);
    } else {
      const T* ap = a.A ? a.A + o : nullptr;
      const T* bp = a.B ? a.B + o : nullptr;
      const T* cp = a.Cq ? a.Cq + o : nullptr;
      T* op_ = a.out + o;
#pragma unroll
      for (int r = 0; r < U; ++r) {
        const T Rr = -rj[r] * R[r];
        T res = a.gamma * (cp ? Rr + __ldg(cp) : Rr);
        if (ap) res = fma(a.alpha, __ldg(ap), res);
        if (bp) res = fma(a.beta, __ldg(bp), res);
        *op_ = res;
        op_ += a.ldim_u;
        if (ap) ap += a.ldim_u;
        if (bp) bp += a.ldim_u;
        if (cp) cp += a.ldim_u;
      }
    }
  }
}

// uf = M0 u from the 1D traces: n terms per flux point instead of n^2
template <typename T, int n, int VPT>
__global__ void __launch_bounds__(256) dg_interp_fac_kernel(const DgArgs<T> a, const DgFac<T, n> op) {
  constexpr int U = n * n;
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t e = (int64_t)blockIdx.x * 32 + lane;
  if (e >= a.neles) return;
  const int vend = a.v0 + a.nv;
  const int vbeg = a.v0 + (int)blockIdx.y * (8 * VPT) + w;
#pragma unroll 1
  for (int it = 0; it < VPT; ++it) {
    const int v = vbeg + 8 * it;
    if (v >= vend) break;
    const int64_t o = ((int64_t)blockIdx.x * a.V + v) * 32 + lane;
    T u[U];
    const T* up = a.u + o;
#pragma unroll
    for (int i = 0; i < U; ++i, up += a.ldim_u) u[i] = __ldg(up);
    T* fp = a.uf + o;
#pragma unroll
    for (int face = 0; face < 4; ++face) {
      const int end = face == 1 || face == 2;
      const bool xi = face & 1;  // the face is across the xi axis
#pragma unroll
      for (int t = 0; t < n; ++t, fp += a.ldim_f) {
        T s = op.l[end][0] * u[xi ? t * n : t];
#pragma unroll
        for (int i = 1; i < n; ++i) s = fma(op.l[end][i], u[xi ? t * n + i : i * n + t], s);
        *fp = s;
      }
    }
  }
}

// The residual on 1D factors.  Same work mapping, shapes and epilogue as
// dg_residual_kernel, which needs U (F + D U) + F U multiply-adds per velocity
// and element with every matrix entry a constant of its own (p = 3: 1,024 and
// 4 KB); the factors need 4 n^2 (traces) + 2 n^3 (derivative) + 4 n^2 (traces
// of the transformed flux) + 8 n^2 (lift) (p = 3: 384, 48 constants), so the
// loads bound the kernel instead of the instructions.  Boundary and halo flux
// points are evaluated in a loop over the lane's own ones before the flux work
// (its code once, not once per flux point); interior warps skip it.  PF: the
// Runge-Kutta terms are loaded ahead and kept as they are, so that the small
// ones are added first, as without PF (added up ahead they would cost one
// rounding at the size of f more: error of a stage 4.0e-8 instead of 3.2e-8).
// B is loaded at the end: in the steppers it is u, whose lines L1 still holds.
// C is loaded with u where the registers allow (EARLY: FP32 p <= 2, FP64 p = 1),
// else after the xi half; FP64 p = 2, 91 elements, N = 24: 179 us early, 167 late.
template <typename T, int n, int VPT, int PF, int MB>
__global__ void __launch_bounds__(256, MB) dg_residual_fac_kernel(const DgArgs<T> a, const DgFac<T, n> op) {
  constexpr int U = n * n, F = 4 * n, D = 2;
  constexpr bool EARLY = U * sizeof(T) <= 36;
  using G = DgGeo<T, U, F, D>;
  __shared__ __align__(16) T sg[32 * G::GS];
  __shared__ __align__(16) int64_t sp[32 * G::PS];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  {
    const T* gs = a.geoblk + (size_t)blockIdx.x * 32 * G::GS;
    for (int i = threadIdx.x; i < 32 * G::GS; i += 256) sg[i] = gs[i];
    const int64_t* ps = a.pblk + (size_t)blockIdx.x * 32 * G::PS;
    for (int i = threadIdx.x; i < 32 * G::PS; i += 256) sp[i] = ps[i];
  }
  __syncthreads();
  const int64_t e = (int64_t)blockIdx.x * 32 + lane;
  if (e >= a.neles) return;
  const T* gl = sg + lane * G::GS;
  const int64_t* pl = sp + lane * G::PS;
  const int vend = a.v0 + a.nv;
  const int vbeg = a.v0 + (int)blockIdx.y * (8 * VPT) + w;
  unsigned bmask = 0;  // flux points whose partner is not an element of this part
#pragma unroll
  for (int f = 0; f < F; ++f) bmask |= pl[f] < 0 ? 1u << f : 0u;

#pragma unroll 1
  for (int it = 0; it < VPT; ++it) {
    const int v = vbeg + 8 * it;
    if (v >= vend) break;
    const int64_t o = ((int64_t)blockIdx.x * a.V + v) * 32 + lane;

    // every bank value of this (v, e) first, so the loads overlap
    T u[U];
    {
      const T* up = a.u + o;
#pragma unroll
      for (int i = 0; i < U; ++i, up += a.ldim_u) u[i] = __ldg(up);
    }
    T xa[PF ? U : 1], cq[PF ? U : 1];
    if constexpr (PF != 0) {
#pragma unroll
      for (int r = 0; r < U; ++r) xa[r] = a.A ? __ldg(a.A + o + (int64_t)r * a.ldim_u) : T(0);
    }
    if constexpr (PF != 0 && EARLY) {
#pragma unroll
      for (int r = 0; r < U; ++r) cq[r] = a.Cq ? __ldg(a.Cq + o + (int64_t)r * a.ldim_u) : T(0);
    }
    // the face values come from the interp kernel: wait for it (returns at
    // once after the first iteration)
    pdl_wait();
    T urv[F];
#pragma unroll
    for (int f = 0; f < F; f += 2) {
      const longlong2 pb = reinterpret_cast<const longlong2*>(pl)[f / 2];
      urv[f] = pb.x >= 0 ? a.uf[pb.x + (int64_t)v * 32] : T(0);
      urv[f + 1] = pb.y >= 0 ? a.uf[pb.y + (int64_t)v * 32] : T(0);
    }
    const T c[3] = {__ldg(a.cvx + v), __ldg(a.cvy + v), __ldg(a.cvz + v)};
    unsigned omask = 0;  // boundary points whose ghost value is the interior one
    if (bmask) {
      for (unsigned m = bmask; m; m &= m - 1) {
        const int f = __ffs(m) - 1, b = (int)(-pl[f] - 1);
        T val = T(0);
        if (b >= a.nb) {
          val = a.halo[(int64_t)(b - a.nb) * a.V + v];
        } else {
          const T nmv[D] = {gl[G::ON + f * D], gl[G::ON + f * D + 1]};
          if (dg_ghost<T, D>(a, b, v, e, f, c, nmv, &val)) omask |= 1u << f;
        }
#pragma unroll
        for (int g = 0; g < F; ++g) urv[g] = g == f ? val : urv[g];
      }
    }

    // transformed flux at the solution points F~_(i,k) = (sum_kk S_ik,kk c_kk) u_k
    T fx[U], fe[U];
    if constexpr (G::VW == 4) {
#pragma unroll
      for (int k = 0; k < U; ++k) {
        T sm[4];
        lds16<T, 1>(gl + G::OS + 4 * k, sm);
        fx[k] = fma(sm[1], c[1], sm[0] * c[0]) * u[k];
        fe[k] = fma(sm[3], c[1], sm[2] * c[0]) * u[k];
      }
    } else {
#pragma unroll
      for (int k = 0; k < U; ++k) {
        T sm[4];
        lds16<T, 2>(gl + G::OS + 4 * k, sm);
        fx[k] = fma(sm[1], c[1], sm[0] * c[0]) * u[k];
        fe[k] = fma(sm[3], c[1], sm[2] * c[0]) * u[k];
      }
    }
    // common normal flux |S^T n| F^ at flux point f (rusanov.mako:46-50 with
    // the scaled normal), ul the interior trace
    auto common = [&](int f, T ul) -> T {
      const T nc = fma(gl[G::ON + f * D + 1], c[1], gl[G::ON + f * D] * c[0]);
      const T ur = omask >> f & 1 ? ul : urv[f];
      return T(0.5) * nc * (ul + ur) + T(0.5) * fabs(nc) * (ul - ur);
    };
    T R[U];
    // along xi (faces 3 and 1), then along eta (faces 0 and 2): the derivative
    // and the lift of the jump between common and interior normal flux
    {
      T j0[n], j1[n];
#pragma unroll
      for (int t = 0; t < n; ++t) {
        T ul0 = op.l[0][0] * u[t * n], ul1 = op.l[1][0] * u[t * n];
        T g0 = op.l[0][0] * fx[t * n], g1 = op.l[1][0] * fx[t * n];
#pragma unroll
        for (int i = 1; i < n; ++i) {
          ul0 = fma(op.l[0][i], u[t * n + i], ul0);
          ul1 = fma(op.l[1][i], u[t * n + i], ul1);
          g0 = fma(op.l[0][i], fx[t * n + i], g0);
          g1 = fma(op.l[1][i], fx[t * n + i], g1);
        }
        j0[t] = common(3 * n + t, ul0) + g0;
        j1[t] = common(n + t, ul1) - g1;
      }
#pragma unroll
      for (int j = 0; j < n; ++j) {
        T h0 = op.la[j][0] * j0[0], h1 = op.la[j][0] * j1[0];
#pragma unroll
        for (int t = 1; t < n; ++t) {
          h0 = fma(op.la[j][t], j0[t], h0);
          h1 = fma(op.la[j][t], j1[t], h1);
        }
#pragma unroll
        for (int i = 0; i < n; ++i) {
          T s = fma(op.lc[1][i], h1, op.lc[0][i] * h0);
#pragma unroll
          for (int k = 0; k < n; ++k) s = fma(op.d[i][k], fx[j * n + k], s);
          R[j * n + i] = s;
        }
      }
    }
    if constexpr (PF != 0 && !EARLY) {
#pragma unroll
      for (int r = 0; r < U; ++r) cq[r] = a.Cq ? __ldg(a.Cq + o + (int64_t)r * a.ldim_u) : T(0);
    }
    {
      T j0[n], j1[n];
#pragma unroll
      for (int t = 0; t < n; ++t) {
        T ul0 = op.l[0][0] * u[t], ul1 = op.l[1][0] * u[t];
        T g0 = op.l[0][0] * fe[t], g1 = op.l[1][0] * fe[t];
#pragma unroll
        for (int i = 1; i < n; ++i) {
          ul0 = fma(op.l[0][i], u[i * n + t], ul0);
          ul1 = fma(op.l[1][i], u[i * n + t], ul1);
          g0 = fma(op.l[0][i], fe[i * n + t], g0);
          g1 = fma(op.l[1][i], fe[i * n + t], g1);
        }
        j0[t] = common(t, ul0) + g0;
        j1[t] = common(2 * n + t, ul1) - g1;
      }
#pragma unroll
      for (int i = 0; i < n; ++i) {
        T h0 = op.la[i][0] * j0[0], h1 = op.la[i][0] * j1[0];
#pragma unroll
        for (int t = 1; t < n; ++t) {
          h0 = fma(op.la[i][t], j0[t], h0);
          h1 = fma(op.la[i][t], j1[t], h1);
        }
#pragma unroll
        for (int j = 0; j < n; ++j) {
          T s = fma(op.lc[1][j], h1, fma(op.lc[0][j], h0, R[j * n + i]));
#pragma unroll
          for (int k = 0; k < n; ++k) s = fma(op.d[j][k], fe[k * n + i], s);
          R[j * n + i] = s;
        }
      }
    }

    const T* const rj = gl + G::OR;
    // out = alpha A + beta B + gamma (R + C), the small terms added first
    if constexpr (PF != 0) {
      const T* bp = a.B ? a.B + o : nullptr;
      T* op_ = a.out + o;
#pragma unroll
      for (int r = 0; r < U; ++r) {
        T res = a.gamma * (-rj[r] * R[r] + cq[r]);
        if (a.A) res = fma(a.alpha, xa[r], res);
        if (bp) res = fma(a.beta, __ldg(bp + (int64_t)r * a.ldim_u), res);
        op_[(int64_t)r * a.ldim_u] = res;
      }
    } else {
      const T* ap = a.A ? a.A + o : nullptr;
      const T* bp = a.B ? a.B + o : nullptr;
      const T* cp = a.Cq ? a.Cq + o : nullptr;
      T* op_ = a.out + o;
#pragma unroll
      for (int r = 0; r < U; ++r) {
        const T Rr = -rj[r] * R[r];
        T res = a.gamma * (cp ? Rr + __ldg(cp) : Rr);
        if (ap) res = fma(a.alpha, __ldg(ap), res);
        if (bp) res = fma(a.beta, __ldg(bp), res);
        *op_ = res;
        op_ += a.ldim_u;
        if (ap) ap += a.ldim_u;
        if (bp) bp += a.ldim_u;
        if (cp) cp += a.ldim_u;
      }
    }
  }
}

// send[s][v] = uf[sfpt[s]][v][sele[s]] for every velocity: the face values a
// neighbouring partition needs, one row per shared flux point.
template <typename T>
__global__ void __launch_bounds__(256) dg_pack_kernel(const T* __restrict__ uf, int64_t ldim_f, int V,
                                                     const int* __restrict__ sfpt, const int* __restrict__ sele,
                                                     int nsend, T* __restrict__ send) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)nsend * V) return;
  const int s = (int)(t / V), v = (int)(t % V);
  send[t] = uf[aos32(sfpt[s], ldim_f, sele[s], v, V)];
}

}  // namespace dgfs
