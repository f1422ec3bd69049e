// mix_kernels.cuh -- launch interface of the ensemble's polyhedron kernels
// (mix_kernels.cu; the geometry and narrow phases are in mix_device.cuh).
//
// Per step, before the sphere step k_ens_step:
//   k_mix_geom        world-frame vertex offsets and face planes of every
//                     polyhedron from its orientation (FP64)
//   k_mix_poly_step   one to four warps per polyhedron that take its tests in turn:
//                     sphere neighbours a slot per lane (the pair's force and
//                     torque on the sphere left in the slot for the sphere
//                     step), polyhedron neighbours and near triangles one at a
//                     time with a warp sharing the separating-axis queries; then
//                     one warp sums in slot order and integrates (translation,
//                     Euler's equations in the body frame, quaternion)
// and per re-sort, after the sphere list:
//   k_mix_plist       the 64-slot neighbour list of every polyhedron, its
//                     tangential histories carried by partner pid
//   k_mix_twins       per sphere slot holding a polyhedron, the polyhedron's
//                     slot that holds the sphere
#pragma once

#include "ens_kernels.cuh"
#include "mix_device.cuh"

namespace blaze {

// Warps that take a polyhedron (an SM holds 16 warps of 128 registers): four up
// to two waves of blocks, two up to five waves, else one.  More warps shorten a rock's chain of tests
// and take other rocks' places.  Time of k_mix_poly_step in us with 4, 2 and 1
// warps a rock:
//   drum, 1,000 rocks among 20,000 balls   40.1  39.9  48.4
//   drum, 4,000 among 24,000               56.5  52.0  65.3
//   settled box of 4,000                   37.1  37.8  41.6   loose 34.5 26.1 19.5
//   settled box of 8,000                   58.2  44.8  50.3   loose 56.4 42.3 29.1
//   settled box of 16,000                 101.0  77.8  55.0   loose 95.1 73.2 44.2
// and a whole step with 4 and 2, alone: 200 rocks among 4,000 balls 44.5 and
// 50.1, 1,000 among 20,000 70.7 and 73.9; with 2 and 1, 5,000 among 100,000 in the
// drum 128 and 138.
inline int mix_warps(int npoly) {
  return npoly <= 2 * 148 * 4 ? 4 : (npoly <= 5 * 148 * 8 ? 2 : 1);
}

// Staged polyhedra -> the state right after blaze_ens_set_state (memory
// order = the caller's order): pos4.w = -bounding radius, angv4.w = id,
// orientation, memory position, path and both list copies cleared.
void mix_launch_mark(const EnsBufs& b, int cur, const MixBufs& m, const int* caller_index,
                     const float4* quat, cudaStream_t st);
void mix_launch_geom(const MixBufs& m, const RoundLink& round, cudaStream_t st);
void mix_launch_plist(const EnsGeom& g, const EnsBufs& b, const MixBufs& m,
                      const uint32_t* start, StepCtl* ctl,
                      const int* gate, cudaStream_t st);
// After k_mix_plist: per sphere slot holding a polyhedron, the polyhedron's
// slot that holds the sphere.
void mix_launch_twins(const EnsBufs& b, const MixBufs& m, int n, StepCtl* ctl, const int* gate,
                      cudaStream_t st);
void mix_launch_poly_step(const EnsGeom& g, const EnsBufs& b, const MixBufs& m, int cur,
                          StepCtl* ctl, StepLink link, const EnsCapture* cap, cudaStream_t st);

}  // namespace blaze
