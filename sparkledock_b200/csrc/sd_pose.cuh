// Exact FP64 pose transforms shared by the scoring kernels.  Compiled with -fmad=false so each
// multiply and add rounds separately, in the order of the reference:
//   receptor  r = r0; for j: if mask: r += mode_j * ext_j        prepare_gso_tasks.cc:465-482
//   ligand    l = l0; for j: if mask: l += mode_j * ext_j        :487-504
//             l = q (0,l) conj(q)/|q|^2  (rotate)                :277-338
//             l += t                                             :518-526
#pragma once
#include "sd_internal.h"

namespace sd {

// quaternion inverse exactly as rotate() forms it (prepare_gso_tasks.cc:288-298)
__device__ __forceinline__ void quat_inverse(const double* q, double* qi) {
  double w = q[0], x = q[1], y = q[2], z = q[3];
  double n2 = w * w + x * x + y * y + z * z;
  qi[0] = q[0] / n2;
  qi[1] = -q[1] / n2;
  qi[2] = -q[2] / n2;
  qi[3] = -q[3] / n2;
}

// rotate one point (prepare_gso_tasks.cc:301-329), same expression order
__device__ __forceinline__ void quat_rotate(const double* q, const double* qi, double& px, double& py, double& pz) {
  double c0 = 0, c1 = px, c2 = py, c3 = pz;
  double d0 = (q[0] * c0 - q[1] * c1 - q[2] * c2 - q[3] * c3);
  double d1 = (q[0] * c1 + q[1] * c0 + q[2] * c3 - q[3] * c2);
  double d2 = (q[0] * c2 - q[1] * c3 + q[2] * c0 + q[3] * c1);
  double d3 = (q[0] * c3 + q[1] * c2 - q[2] * c1 + q[3] * c0);
  px = (d0 * qi[1] + d1 * qi[0] + d2 * qi[3] - d3 * qi[2]);
  py = (d0 * qi[2] - d1 * qi[3] + d2 * qi[0] + d3 * qi[1]);
  pz = (d0 * qi[3] + d1 * qi[2] - d2 * qi[1] + d3 * qi[0]);
}

// one atom plus its masked mode displacements, each multiply and add rounded: coordinates [3][n] and
// modes [nm][3][n] in slot order, so a warp's consecutive slots read full lines
__device__ __forceinline__ void anm_exact(const double* xyz, const double* modes, const int* mask, int n, int nm,
                                          const double* ext, int slot, double& x, double& y, double& z) {
  const size_t st = n;
  const double* p = xyz + slot;
  x = p[0];
  y = p[st];
  z = p[2 * st];
  if (mask[slot] != 1) return;
  const double* M = modes + slot;
#pragma unroll 2
  for (int m = 0; m < nm; ++m, M += 3 * st) {
    const double e = ext[m];
    x += M[0] * e;
    y += M[st] * e;
    z += M[2 * st] * e;
  }
}

// the same of kP poses (extents from pose[p] + e0) with one read of the modes
template <int kP>
__device__ __forceinline__ void anm_exact(const double* xyz, const double* modes, const int* mask, int n, int nm,
                                          const double* const (&pose)[kP], int e0, int slot, double (&r)[kP][3]) {
  const size_t st = n;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double v = xyz[slot + d * st];
#pragma unroll
    for (int p = 0; p < kP; ++p) r[p][d] = v;
  }
  if (mask[slot] != 1) return;
  const double* M = modes + slot;
#pragma unroll 2
  for (int m = 0; m < nm; ++m, M += 3 * st) {
    const double mx = M[0], my = M[st], mz = M[2 * st];
#pragma unroll
    for (int p = 0; p < kP; ++p) {
      const double e = pose[p][e0 + m];
      r[p][0] += mx * e;
      r[p][1] += my * e;
      r[p][2] += mz * e;
    }
  }
}

// a displaced ligand atom rotated and translated into the pose
__device__ __forceinline__ void ligand_place(const double* pose, double& x, double& y, double& z) {
  double q[4] = {pose[3], pose[4], pose[5], pose[6]}, qi[4];
  quat_inverse(q, qi);
  quat_rotate(q, qi, x, y, z);
  x += pose[0];
  y += pose[1];
  z += pose[2];
}

// receptor atom in tile slot `slot`, extents e_rec = pose + 7
__device__ __forceinline__ void receptor_exact(const DevComplex& C, int nslots, int slot, const double* pose,
                                               double& x, double& y, double& z) {
  anm_exact(C.r_xyz, C.r_modes, C.r_mask, nslots, C.nmr, pose + 7, slot, x, y, z);
}

// ligand atom in chunk slot s
__device__ __forceinline__ void ligand_exact(const DevComplex& C, int s, const double* pose, const double* q,
                                             const double* qi, double& x, double& y, double& z) {
  anm_exact(C.l_xyz, C.l_modes, C.l_mask, C.nlchunks * SD_TILE, C.nml, pose + 7 + C.nmr, s, x, y, z);
  quat_rotate(q, qi, x, y, z);
  x += pose[0];
  y += pose[1];
  z += pose[2];
}

// the same displacement for kP poses (extents estride doubles apart) with fused multiply-adds (half
// the FP64 instructions) and one read of the modes, for coordinates that are then rounded to FP32:
// the difference is of the order of an FP64 rounding
template <int kP>
__device__ __forceinline__ void anm_fused(const double* xyz, const double* modes, const int* mask, int n, int nm,
                                          const double* ext, int estride, int slot, double (&r)[kP][3]) {
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double v = xyz[slot + d * n];
#pragma unroll
    for (int p = 0; p < kP; ++p) r[p][d] = v;
  }
  if (mask[slot] != 1) return;
  int o = slot;
#pragma unroll 5
  for (int m = 0; m < nm; ++m, o += 3 * n) {
    const double M0 = modes[o], M1 = modes[o + n], M2 = modes[o + 2 * n];
#pragma unroll
    for (int p = 0; p < kP; ++p) {
      const double e = ext[p * estride + m];
      r[p][0] = fma(M0, e, r[p][0]);
      r[p][1] = fma(M1, e, r[p][1]);
      r[p][2] = fma(M2, e, r[p][2]);
    }
  }
}

// half extent of a group's box on an axis, wider by what the box test may lose in FP32 (three roundings of
// 2^-24 of the largest coordinate: centre, extent and difference); -inf stays for an empty group (lo > hi)
__device__ __forceinline__ float half_extent(float lo, float hi) {
  return fmaf(5e-7f, fmaxf(fabsf(lo), fabsf(hi)), 0.5f * (hi - lo));
}

__device__ __forceinline__ int nslots_of(const DevComplex& C) { return C.ntiles * SD_TILE; }

}  // namespace sd
