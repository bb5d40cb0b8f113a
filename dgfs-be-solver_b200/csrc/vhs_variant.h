// A compiled launch shape of the VHS operator, as vhs.cu lists them; each
// kernel family builds its shapes in its own translation unit.
#pragma once

#include <stddef.h>

#include <cuda_runtime.h>

namespace dgfs {

template <typename T> struct VhsArgs;

struct VhsVariant {
  int prec, N, C, db, minb, threads, push;
  size_t smem;
  size_t scratch_cx;  // two-CTA kernel: complex scratch per cluster
  size_t slice_cx;    // single-CTA kernel: complex entries of one gain-spectrum slice
  const void* fn;
  cudaError_t (*launch32)(const VhsArgs<float>&, int, cudaStream_t);
  cudaError_t (*launch64)(const VhsArgs<double>&, int, cudaStream_t);
};

// partial-spectrum slices per CTA of the single-CTA kernel: a launch on few
// points splits them into one work item per radial node, at most so many per
// CTA of the grid
constexpr int kCubeSlices = 24;

// single-CTA kernel (kind 2 in dgfs_vhs_variant_kind): FP32 N = 8, 16, 24 and
// FP64 N = 16
VhsVariant cube_variant(int prec, int N);
// two-CTA kernel (kind 3): FP32 N = 32 and FP64 N = 24; own: Nyquist lines on
// threads of their own
VhsVariant pair_variant(int prec, bool own);

}  // namespace dgfs
