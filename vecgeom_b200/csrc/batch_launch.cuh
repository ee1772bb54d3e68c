// batch_launch.cuh -- launches of the FP64 batch kernels of one shape; each group of
// shapes is instantiated in a file of its own (batch_*.cu).
//
// Compiled with -fmad=false (see the Makefile): no a*b+c is contracted into an
// FMA, so each result rounds exactly as the reference Scalar build compiled
// with -ffp-contract=off.
#pragma once
#include <algorithm>

#include "batch.cuh"
#include "dispatch.h"
#include "geometry.h"
#include "refine.cuh"

namespace vgb {

// Launches a batch kernel so that its set-up overlaps the end of the batch kernel before
// it in the stream (batch_kernel_begin).
template <class... K, class... A>
void launch_overlapped(void (*k)(K...), dim3 grid, size_t smem, cudaStream_t s, const A &...a) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = dim3(kBatchBlock);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, k, a...);
}

inline int grid_for(int64_t n) {
  // enough CTAs to fill 148 SMs x 8 resident 256-thread CTAs; grid-stride beyond
  const int64_t want = (n + kBatchBlock - 1) / kBatchBlock;
  const int64_t cap = 148 * 8 * 4;
  return (int)(want < 1 ? 1 : (want > cap ? cap : want));
}

// The regrouped walks (polycone and polyhedron distances) refill a warp's lanes
// from the warp's own stream of points, so they keep lanes busier when each warp
// owns more points: a quarter of the grid above (measured: polyhedron
// DistanceToIn/Out 7.0 k/5.7 k -> 7.9 k/7.4 k Mpoints/s, polycone DistanceToIn
// 5.8 k -> 6.2 k, and polycone DistanceToOut regrouped 7.6 k, against 6.8 k on
// one lane), while the other kernels run fastest with the full grid.
constexpr int kWalkGridCap = 148 * 8;

template <class Ops, class P>
vgb_status BatchLaunch<Ops, P>::batch(const P &prm, const DXform &X, int op, BatchIO io,
                                      cudaStream_t s, int32_t rec_len, int precision) {
  // FP32+refine: DistanceToIn of the shapes with a float selector (refine.cuh);
  // every other (shape, op) computes in FP64 in both forms
  if constexpr (!std::is_void<typename RefineDti<Ops>::type>::value) {
    if (precision == VGB_PREC_FP32_REFINE && op == VGB_OP_DISTANCE_TO_IN) {
      const int64_t tiles = (io.n + kRefineTile - 1) / kRefineTile;
      const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(tiles, 148 * 8));
      k_refine_dti<typename RefineDti<Ops>::type, Ops, P><<<grid, kRefineBlock, 0, s>>>(prm, X, io);
      count_launch();
      cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) return cuda_error(e, "vgb_batch: kernel launch");
      return VGB_OK;
    }
  }
  io.stage = (Stageable<P>::value && rec_len > 0 && rec_len <= kStageMaxDoubles) ? rec_len : 0;
  const size_t smem = (size_t)io.stage * sizeof(double);
  const int grid = grid_for(io.n);
  switch (op) {
#define VGB_OP_CASE(OPC)                                                      \
  case OPC:                                                                   \
    launch_overlapped(k_batch<Ops, P, OPC>,                                   \
                      RegroupedWalk<Ops, OPC>::value ? std::min(grid, kWalkGridCap) : grid, smem, \
                      s, prm, X, io);                                         \
    break;
    VGB_OP_CASE(VGB_OP_CONTAINS)
    VGB_OP_CASE(VGB_OP_INSIDE)
    VGB_OP_CASE(VGB_OP_DISTANCE_TO_IN)
    VGB_OP_CASE(VGB_OP_DISTANCE_TO_OUT)
    VGB_OP_CASE(VGB_OP_SAFETY_TO_IN)
    VGB_OP_CASE(VGB_OP_SAFETY_TO_OUT)
    VGB_OP_CASE(VGB_OP_DISTANCE_TO_IN_MINIMIZE)
    VGB_OP_CASE(VGB_OP_SAFETY_TO_IN_MINIMIZE)
    VGB_OP_CASE(VGB_OP_SAFETY_TO_OUT_MINIMIZE)
    VGB_OP_CASE(VGB_OP_DISTANCE_TO_OUT_NODE)
    VGB_OP_CASE(VGB_OP_PLACED_DISTANCE_TO_OUT)
#undef VGB_OP_CASE
  default:
    return set_error(VGB_EINVAL, "vgb_batch: unknown op %d", op);
  }
  count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_error(e, "vgb_batch: kernel launch");
  return VGB_OK;
}

// Whether an output of a fused call shares memory with one of the inputs it reads.
inline bool fused_in_place(const FusedIO &io) {
  const double *in[] = {io.x, io.y, io.z, io.dx, io.dy, io.dz, io.step};
  const bool dirs = io.ops & ((1u << VGB_OP_DISTANCE_TO_IN) | (1u << VGB_OP_DISTANCE_TO_OUT));
  for (int op = 0; op < 6; ++op) {
    if (!((io.ops >> op) & 1u)) continue;
    const uintptr_t size = op == VGB_OP_CONTAINS ? 1 : op == VGB_OP_INSIDE ? 4 : 8;
    const uintptr_t o = reinterpret_cast<uintptr_t>(io.out[op]), oe = o + size * io.n;
    for (int k = 0; k < (dirs ? 7 : 3); ++k) {
      const uintptr_t i = reinterpret_cast<uintptr_t>(in[k]);
      if (o < i + 8 * io.n && i < oe) return true;
    }
  }
  return false;
}

template <class Ops, class P>
vgb_status BatchLaunch<Ops, P>::fused(const P &prm, const DXform &X, const FusedIO &io,
                                      cudaStream_t s, int32_t rec_len) {
  bool rows = false;
  if constexpr (SplitFused<P>::value) {
    // the rows of a call read the inputs independently of each other's stores, so a call
    // that writes an output over one of its inputs takes the kernel whose threads read a
    // point's inputs before they store
    rows = !fused_in_place(io);
    if (rows) {
      const int groups = (io.ops & kPointOps ? 1 : 0) +
                         (io.ops & (1u << VGB_OP_DISTANCE_TO_IN) ? 1 : 0) +
                         (io.ops & (1u << VGB_OP_DISTANCE_TO_OUT) ? 1 : 0);
      const int32_t stage =
          (Stageable<P>::value && rec_len > 0 && rec_len <= kStageMaxDoubles) ? rec_len : 0;
      const dim3 grid(std::min(grid_for(io.n), kWalkGridCap), groups);
      launch_overlapped(k_fused_split<Ops, P>, grid, (size_t)stage * sizeof(double), s, prm, X, io,
                        stage);
    }
  }
  if (!rows) launch_overlapped(k_fused<Ops, P>, dim3(grid_for(io.n)), 0, s, prm, X, io);
  count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_error(e, "vgb_batch_fused: kernel launch");
  return VGB_OK;
}

}  // namespace vgb
