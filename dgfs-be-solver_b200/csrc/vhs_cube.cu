// Launch shapes of the single-CTA VHS kernel (vhs_cube.cuh).
#include "vhs_cube.cuh"

namespace dgfs {

template <typename T, int N, int MINB> static cudaError_t launch_cube(const VhsArgs<T>& a, int nctas, cudaStream_t s) {
  using G = CubeGeom<T, N>;
  vhs_cube_kernel<T, N, MINB><<<nctas, G::NT, G::SMEM, s>>>(a);
  return cudaGetLastError();
}

template <typename T, int N, int MINB> static VhsVariant make_cube() {
  using G = CubeGeom<T, N>;
  VhsVariant v{};
  v.prec = 8 * (int)sizeof(T);
  v.N = N;
  v.C = 1;
  v.push = 2;
  v.minb = MINB;
  v.threads = G::NT;
  v.smem = G::SMEM;
  v.scratch_cx = v.slice_cx = G::SL;
  v.fn = (const void*)vhs_cube_kernel<T, N, MINB>;
  if constexpr (sizeof(T) == 8) v.launch64 = launch_cube<T, N, MINB>;
  else v.launch32 = launch_cube<T, N, MINB>;
  return v;
}

VhsVariant cube_variant(int prec, int N) {
  if (prec == 64) return make_cube<double, 16, 1>();
  if (N == 8) return make_cube<float, 8, 4>();
  if (N == 16) return make_cube<float, 16, 2>();
  return make_cube<float, 24, 1>();
}

}  // namespace dgfs
