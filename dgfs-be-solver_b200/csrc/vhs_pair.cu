// Launch shapes of the two-CTA VHS kernel (vhs_pair.cuh).
#include "vhs_pair.cuh"

namespace dgfs {

template <typename T, int N, bool OWN> static cudaError_t launch_pair(const VhsArgs<T>& a, int nclusters, cudaStream_t s) {
  using G = PairGeom<T, N, OWN>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nclusters * 2, 1, 1);
  cfg.blockDim = dim3(G::NT, 1, 1);
  cfg.dynamicSmemBytes = G::SMEM;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, vhs_pair_kernel<T, N, OWN>, a);
}

template <typename T, int N, bool OWN> static VhsVariant make_pair() {
  using G = PairGeom<T, N, OWN>;
  VhsVariant v{};
  v.prec = 8 * (int)sizeof(T);
  v.N = N;
  v.C = 2;
  v.db = OWN ? 1 : 0;
  v.push = 3;
  v.minb = 1;
  v.threads = G::NT;
  v.smem = G::SMEM;
  v.scratch_cx = G::SCRATCH;
  v.fn = (const void*)vhs_pair_kernel<T, N, OWN>;
  if constexpr (sizeof(T) == 8) v.launch64 = launch_pair<double, N, OWN>;
  else v.launch32 = launch_pair<float, N, OWN>;
  return v;
}

VhsVariant pair_variant(int prec, bool own) {
  if (prec == 64) return own ? make_pair<double, 24, true>() : make_pair<double, 24, false>();
  return own ? make_pair<float, 32, true>() : make_pair<float, 32, false>();
}

}  // namespace dgfs
