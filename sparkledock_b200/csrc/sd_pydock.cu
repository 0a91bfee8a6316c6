// pyDock-style electrostatics + Lennard-Jones energy and its adjoint (project-defined; the
// reference has no such scoring function).  Specification, also restated by the oracle
// (oracle/sd_oracle.c, or_pydock_*):
//   x = |r_i - l_j|^2
//   elec_ij = 332.0636/4 * q_i q_j / (x + 1)           distance-dependent dielectric 4r, soft core
//   lj_ij   = 4 eps_ij (s^6 - s^3),  s = sig_ij^2 / (x + 0.5 sig_ij^2)
//             eps_ij = sqrt(eps_a eps_b), sig_ij = (sig_a + sig_b)/2 (20-type table)
//   S(x; on, off) = CHARMM switch (off - x)^2 (off + 2x - 3 on) / (off - on)^3 on on < x < off
//   E = sum_{x < 225} elec S(x;196,225) + 0.1 sum_{x < 64} lj S(x;49,64);   score = -E
// Gradient with respect to the pose: translation (3), left tangent rotation w with
// q <- exp(w/2) q (3), receptor and ligand ANM extents:
//   dE/dt = sum_j F_j, dE/dw = sum_j (l_j - t) x F_j, dE/de_lig_m = sum_j mask_j (R M_mj).F_j,
//   dE/de_rec_m = sum_i mask_i M_mi.G_i, with F_j = dE/dl_j, G_i = dE/dr_i (pair forces).
//
// Kernel: one CTA (8 warps) per pose at a time, persistent over a work list; receptor tiles of
// 32 (one lane per atom) culled against the ligand sphere and against spatial ligand chunks, and
// each tile's candidate ligand atoms against the bounding boxes of its four groups of 8 atoms.  A
// step evaluates 8 receptor atoms x 4 candidates of one group, one pair per lane.  GRAD adds
// per-lane receptor force accumulators (summed over the four rows at the end of a group, projected
// onto the receptor modes at the end of each tile) and per-ligand-atom force accumulators in shared
// memory (a row's three components reduced together in four shuffles, one shared atomic), projected
// onto t, w and the ligand modes at the end of the pose.
#include <cuda_runtime.h>

#include "sd_internal.h"
#include "sd_pose.cuh"

namespace sd {

namespace {

constexpr int kPdWarps = 8;
constexpr double kKe = 332.0636 / 4.0;

// a ligand atom in shared memory (position relative to t, charge): one 16-byte load in FP32
template <class T>
struct alignas(16) LigAtom {
  T x, y, z, q;
};
// the LJ pair parameters of two types, read together
template <class T>
struct alignas(2 * sizeof(T)) LjPair {
  T eps, sig2;
};

// the switch with its constant 1 / (off2 - on2)^3 passed in (both widths are fixed)
template <class T>
__device__ __forceinline__ void pd_switch(T x, T on2, T off2, T rden, T& s, T& ds) {
  if (x <= on2) {
    s = T(1);
    ds = T(0);
    return;
  }
  if (x >= off2) {
    s = T(0);
    ds = T(0);
    return;
  }
  const T a = off2 - x;
  s = a * a * (off2 + T(2) * x - T(3) * on2) * rden;
  ds = T(6) * a * (on2 - x) * rden;
}

// pair energy and dE/dx for x < 225; two divisions per pair (1 / (x + 1) and, inside 8 A,
// 1 / (x + sig2 / 2)), every other quotient a product with them
template <class T>
__device__ __forceinline__ T pd_pair(T x, T qq, T eps, T sig2, T& dedx) {
  T s, ds;
  const T inv = T(1) / (x + T(1));
  const T el = qq * inv;
  pd_switch<T>(x, T(196), T(225), T(1) / T(24389), s, ds);  // (225 - 196)^3
  T e = el * s;
  T de = -el * inv * s + el * ds;
  if (x < T(64)) {
    const T rden = T(1) / (x + T(0.5) * sig2);
    const T sv = sig2 * rden;
    const T s2 = sv * sv, s3 = s2 * sv, s6 = s3 * s3;
    const T lj = T(4) * eps * (s6 - s3);
    const T dsv = -sv * rden;
    const T dlj = T(4) * eps * (T(6) * s3 * s2 - T(3) * s2) * dsv;  // d(s^6 - s^3)/ds = 6 s^5 - 3 s^2
    pd_switch<T>(x, T(49), T(64), T(1) / T(3375), s, ds);  // (64 - 49)^3
    e += T(0.1) * (lj * s);
    de += T(0.1) * (dlj * s + lj * ds);
  }
  dedx = de;
  return e;
}

constexpr int kRows = SD_TILE / SD_GROUP;  // groups of a tile; candidates of a step (one row of 8 lanes each)
constexpr int kPdList = 128;               // candidates of a group between two drains of the lists

// a warp's tile
template <class T>
struct PdWarp {
  LigAtom<T> rec[SD_TILE];           // receptor atoms (position relative to t, charge)
  float4 box[2 * kRows];             // centre and half extent of each group's bounding box
  int lj[SD_TILE];
  unsigned short list[kRows][kPdList];  // each group's candidates: ligand slots
  unsigned short pend[64];           // pending candidate ligand slots of the tile
};

template <class T>
__device__ __forceinline__ T warp_sum(T v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

}  // namespace

// out_grad: nullable [n][6 + nmr + nml] (GRAD), energies go to C.scoring as score (-E) and to
// L.energy_out (E) when set.  kSpill: the per-pose arrays live in this CTA's slice of the global
// scratch L.spill instead of shared memory (ligands too large for it).  Four CTAs per SM (64
// registers a thread) wherever the accumulators allow it: the pair terms are latency chains.
template <class T, bool GRAD, bool kSpill>
__global__ void __launch_bounds__(kPdWarps * 32, GRAD && sizeof(T) == 8 ? 2 : 4) pydock_kernel(ScoreLaunch L, double* out_grad) {
  extern __shared__ __align__(16) unsigned char smem_dyn[];
  PdWarp<T>& W = reinterpret_cast<PdWarp<T>*>(smem_dyn)[threadIdx.x >> 5];
  unsigned char* const smem =
      kSpill ? L.spill + (size_t)blockIdx.x * L.spill_stride : smem_dyn + kPdWarps * sizeof(PdWarp<T>);
  __shared__ double sh_pose[7 + 2 * SD_MAX_MODES];
  __shared__ double sh_q[4], sh_qi[4];
  __shared__ LjPair<T> sh_lj[SD_LJ_TYPES * SD_LJ_TYPES];
  __shared__ double sh_red[kPdWarps][32];
  __shared__ float sh_rot[9];
  __shared__ float sh_bound[2];
  __shared__ int sh_item, sh_ntile, sh_next;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt_mask = (1u << lane) - 1u;
  const int atom = lane & (SD_GROUP - 1), crow = lane / SD_GROUP;  // a step's atom and candidate row
  for (int k = tid; k < SD_LJ_TYPES * SD_LJ_TYPES; k += blockDim.x) {
    const int a = k / SD_LJ_TYPES, b = k % SD_LJ_TYPES;
    sh_lj[k].eps = (T)sqrt(L.lj_eps[a] * L.lj_eps[b]);
    const double sg = 0.5 * (L.lj_sigma[a] + L.lj_sigma[b]);
    sh_lj[k].sig2 = (T)(sg * sg);
  }
  StepCtl* ctl = L.ctl;
  const int parity = ctl->parity;
  const int count = ctl->count[parity];
  const int* work = L.work[parity];
  unsigned long long n_done = 0;

  for (;;) {
    __syncthreads();
    if (tid == 0) sh_item = atomicAdd(&ctl->grab[parity], 1);
    __syncthreads();
    const int item = sh_item;
    if (item >= count) break;
    const int w = work[item];
    const int ci = wi_complex(w), p = wi_local(w);
    const DevComplex& C = L.cplx[ci];
    const int nslots = nslots_of(C), pl = C.pl, nlc = C.nlchunks, nls = nlc * SD_TILE;
    const double* pose_g = C.pos + (size_t)p * pl;
    if (tid < pl) sh_pose[tid] = pose_g[tid];
    __syncthreads();
    if (tid == 0) {
      for (int k = 0; k < 4; ++k) sh_q[k] = sh_pose[3 + k];
      quat_inverse(sh_q, sh_qi);
      float dR = 0.f, dL = 0.f;
      for (int m = 0; m < C.nmr; ++m) dR += fabsf((float)sh_pose[7 + m]) * C.mnorm_r[m];
      for (int m = 0; m < C.nml; ++m) dL += fabsf((float)sh_pose[7 + C.nmr + m]) * C.mnorm_l[m];
      sh_bound[0] = dR * 1.0001f + 1e-4f;
      sh_bound[1] = dL * 1.0001f + 1e-4f;
      const double n = sqrt(sh_q[0] * sh_q[0] + sh_q[1] * sh_q[1] + sh_q[2] * sh_q[2] + sh_q[3] * sh_q[3]);
      const float w0 = (float)(sh_q[0] / n), x = (float)(sh_q[1] / n), y = (float)(sh_q[2] / n),
                  z = (float)(sh_q[3] / n);
      sh_rot[0] = 1 - 2 * (y * y + z * z);
      sh_rot[1] = 2 * (x * y - w0 * z);
      sh_rot[2] = 2 * (x * z + w0 * y);
      sh_rot[3] = 2 * (x * y + w0 * z);
      sh_rot[4] = 1 - 2 * (x * x + z * z);
      sh_rot[5] = 2 * (y * z - w0 * x);
      sh_rot[6] = 2 * (x * z - w0 * y);
      sh_rot[7] = 2 * (y * z + w0 * x);
      sh_rot[8] = 1 - 2 * (x * x + y * y);
      sh_ntile = 0;
      sh_next = 0;
      double rx = C.lig_ref[0], ry = C.lig_ref[1], rz = C.lig_ref[2];
      quat_rotate(sh_q, sh_qi, rx, ry, rz);
      double* ref = C.ref + (size_t)p * 3;
      ref[0] = rx + sh_pose[0];
      ref[1] = ry + sh_pose[1];
      ref[2] = rz + sh_pose[2];
    }
    __syncthreads();
    const double tx = sh_pose[0], ty = sh_pose[1], tz = sh_pose[2];
    const float dR = sh_bound[0], dL = sh_bound[1];
    // per-pose arrays: ligand atoms [nls + 1] (LigAtom<T>; the last a far atom, the padding), GRAD: fx,
    // fy, fz [nls + 1] (T), chunk spheres [nlc] (float4), llj [nls + 1], near tiles [ntiles] as found,
    // in order of distance, and their distances
    LigAtom<T>* la = reinterpret_cast<LigAtom<T>*>(smem);
    T* fx = reinterpret_cast<T*>(la + nls + 1);  // GRAD only: [3][nls + 4]
    const int fstride = nls + 4;
    float4* chS = reinterpret_cast<float4*>(fx + (GRAD ? 3 * fstride : 0));
    int* llj = reinterpret_cast<int*>(chS + nlc);
    int* tlist = llj + nls + 1;
    int* tord = tlist + C.ntiles;
    float* tdist = reinterpret_cast<float*>(tord + C.ntiles);
    if (tid == 0) {
      la[nls] = LigAtom<T>{(T)3e18, (T)3e18, (T)3e18, T(0)};
      llj[nls] = 0;
    }
    if (GRAD)
      for (int s = tid; s < 3 * fstride; s += blockDim.x) fx[s] = T(0);
    for (int s = tid; s < nls; s += blockDim.x) {
      if (C.l_perm[s] >= 0) {
        double x, y, z;
        ligand_exact(C, s, sh_pose, sh_q, sh_qi, x, y, z);
        la[s] = LigAtom<T>{(T)(x - tx), (T)(y - ty), (T)(z - tz), (T)(kKe * (double)C.l_q[s])};
        llj[s] = C.l_lj[s] * SD_LJ_TYPES;
      } else {
        la[s] = LigAtom<T>{(T)1e18, (T)1e18, (T)1e18, T(0)};
        llj[s] = 0;
      }
    }
    for (int c = tid; c < nlc; c += blockDim.x) {
      const float4 cc = C.l_chunk[c];
      const float X = sh_rot[0] * cc.x + sh_rot[1] * cc.y + sh_rot[2] * cc.z;
      const float Y = sh_rot[3] * cc.x + sh_rot[4] * cc.y + sh_rot[5] * cc.z;
      const float Z = sh_rot[6] * cc.x + sh_rot[7] * cc.y + sh_rot[8] * cc.z;
      chS[c] = make_float4(X, Y, Z, cc.w + dL);
    }
    const float lig_reach = C.lig_radius + dL;
    for (int k = tid; k < C.ntiles; k += blockDim.x) {
      const float4 tile = C.r_tile[k];
      const float cx = (float)((double)tile.x - tx), cy = (float)((double)tile.y - ty),
                  cz = (float)((double)tile.z - tz);
      const float reach = 15.0f + dR + SD_CULL_MARGIN + tile.w + lig_reach;
      const float dd = cx * cx + cy * cy + cz * cz;
      if (dd <= reach * reach) {
        const int at = atomicAdd(&sh_ntile, 1);
        tlist[at] = k;
        tdist[at] = dd;
      }
    }
    __syncthreads();
    const int ntile = sh_ntile;
    // the tiles closest to the ligand centre (t) have the most pairs: taken first, the warps finish a
    // pose together
    const bool sorted = ntile <= 512;
    if (sorted) {
      for (int t = tid; t < ntile; t += blockDim.x) {
        const float d = tdist[t];
        int rank = 0;
        for (int u = 0; u < ntile; ++u) {
          const float e = tdist[u];
          rank += (e < d || (e == d && u < t)) ? 1 : 0;
        }
        tord[rank] = tlist[t];
      }
      __syncthreads();
    }
    const int* tl = sorted ? tord : tlist;
    double es = 0.0;  // energy: FP64 per-lane sum of the pair terms
    T grec[SD_MAX_MODES];
    for (int m = 0; m < SD_MAX_MODES; ++m) grec[m] = T(0);

    for (;;) {
      int ti = 0;
      if (lane == 0) ti = atomicAdd(&sh_next, 1);
      ti = __shfl_sync(0xffffffffu, ti, 0);
      if (ti >= ntile) break;
      const int k = tl[ti];
      const float4 tile = C.r_tile[k];
      const float cx = (float)((double)tile.x - tx), cy = (float)((double)tile.y - ty),
                  cz = (float)((double)tile.z - tz);
      const float reach = 15.0f + dR + SD_CULL_MARGIN + tile.w;
      const float reach2 = reach * reach;
      const int slot = k * SD_TILE + lane;
      const bool active = C.r_orig[slot] >= 0;
      LigAtom<T> own{(T)1e18, (T)1e18, (T)1e18, T(0)};
      if (active) {
        double x, y, z;
        receptor_exact(C, nslots, slot, sh_pose, x, y, z);
        own = LigAtom<T>{(T)(x - tx), (T)(y - ty), (T)(z - tz), (T)C.r_q[slot]};
      }
      __syncwarp();
      W.rec[lane] = own;
      W.lj[lane] = active ? C.r_lj[slot] : 0;
      {
        // bounding box of each group of 8 lanes (an empty group's half extent is -inf: no candidate)
        float lo[3] = {(float)own.x, (float)own.y, (float)own.z}, hi[3] = {lo[0], lo[1], lo[2]};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          if (!active) {
            lo[d] = 3e38f;
            hi[d] = -3e38f;
          }
#pragma unroll
          for (int o = 1; o < SD_GROUP; o <<= 1) {
            lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
            hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
          }
        }
        if (atom == 0) {
          W.box[2 * crow] = make_float4(0.5f * (lo[0] + hi[0]), 0.5f * (lo[1] + hi[1]), 0.5f * (lo[2] + hi[2]), 0.f);
          W.box[2 * crow + 1] =
              make_float4(0.5f * (hi[0] - lo[0]), 0.5f * (hi[1] - lo[1]), 0.5f * (hi[2] - lo[2]), 0.f);
        }
      }
      __syncwarp();
      T gx = T(0), gy = T(0), gz = T(0);  // dE/dr of this lane's atom of the tile
      int ncand = 0, cb = 0;
      unsigned cm = 0;
      bool more = true;
      do {
        // fill each group's list until the ligand is exhausted or a list may overflow
        unsigned cnt[kRows];
#pragma unroll
        for (int g = 0; g < kRows; ++g) cnt[g] = 0;
        unsigned longest = 0;
        do {
          // collect candidates until a round is full or the ligand is exhausted
          while (ncand < 32) {
            if (cm == 0) {
              if (cb >= nlc) break;
              const int c = cb + lane;
              bool cnear = false;
              if (c < nlc) {
                const float4 ch = chS[c];
                const float ex = ch.x - cx, ey = ch.y - cy, ez = ch.z - cz, r = reach + ch.w;
                cnear = ex * ex + ey * ey + ez * ez <= r * r;
              }
              cm = __ballot_sync(0xffffffffu, cnear);
              cb += 32;
              continue;
            }
            const int sb = (cb - 32 + __ffs(cm) - 1) * SD_TILE;
            cm &= cm - 1;
            const LigAtom<T> ca = la[sb + lane];
            const float ax = (float)ca.x - cx, ay = (float)ca.y - cy, az = (float)ca.z - cz;
            const bool cand = ax * ax + ay * ay + az * az <= reach2;
            const unsigned am = __ballot_sync(0xffffffffu, cand);
            if (cand) W.pend[ncand + __popc(am & lt_mask)] = (unsigned short)(sb + lane);
            ncand += __popc(am);
          }
          __syncwarp();
          const int nb = min(ncand, 32);
          const int s = lane < nb ? W.pend[lane] : nls;
          const LigAtom<T> c = la[s];
          const float x = (float)c.x, y = (float)c.y, z = (float)c.z;
#pragma unroll
          for (int g = 0; g < kRows; ++g) {
            const float4 bc = W.box[2 * g], bh = W.box[2 * g + 1];
            const float ex = fmaxf(fabsf(x - bc.x) - bh.x, 0.f), ey = fmaxf(fabsf(y - bc.y) - bh.y, 0.f),
                        ez = fmaxf(fabsf(z - bc.z) - bh.z, 0.f);
            const bool in = fmaf(ez, ez, fmaf(ey, ey, ex * ex)) <= 225.1f;
            const unsigned am = __ballot_sync(0xffffffffu, in);
            if (in) W.list[g][cnt[g] + __popc(am & lt_mask)] = (unsigned short)s;
            cnt[g] += __popc(am);
            longest = max(longest, cnt[g]);
          }
          // keep the candidates beyond the first 32
          const int rest = ncand - nb;
          int carry = 0;
          if (lane < rest) carry = W.pend[32 + lane];
          __syncwarp();
          if (lane < rest) W.pend[lane] = (unsigned short)carry;
          ncand = rest;
          __syncwarp();
          more = ncand > 0 || cm != 0 || cb < nlc;
        } while (more && longest <= kPdList - 32 - kRows);
        // each list is padded with the far atom to whole steps
#pragma unroll
        for (int g = 0; g < kRows; ++g)
          if (lane < kRows) W.list[g][cnt[g] + lane] = (unsigned short)nls;
        __syncwarp();
        unsigned counts = cnt[0] | cnt[1] << 8 | cnt[2] << 16 | cnt[3] << 24;
        for (int g = 0; g < kRows; ++g, counts >>= 8) {
          const LigAtom<T> r = W.rec[g * SD_GROUP + atom];
          const LjPair<T>* ljrow = sh_lj + W.lj[g * SD_GROUP + atom];
          const unsigned short* list = W.list[g] + crow;
          const int n = (int)(counts & 255u);
          T hx = T(0), hy = T(0), hz = T(0);  // dE/dr of this lane's pairs
          for (int c = 0; c < n; c += kRows) {
            const int s = list[c];
            const LigAtom<T> a = la[s];
            const T dx = r.x - a.x, dy = r.y - a.y, dz = r.z - a.z;
            const T x = dx * dx + dy * dy + dz * dz;
            T f0 = T(0), f1 = T(0), f2 = T(0);
            if (x < T(225)) {
              T dedx;
              // the table is symmetric (products and sums of the two types' parameters), so it is read as
              // [ligand type][receptor type]: the lanes of one candidate read entries of one row
              const LjPair<T> lj = ljrow[llj[s]];
              const T e = pd_pair<T>(x, r.q * a.q, lj.eps, lj.sig2, dedx);
              es += (double)e;
              if (GRAD) {
                const T g2 = T(2) * dedx;
                f0 = g2 * dx;
                f1 = g2 * dy;
                f2 = g2 * dz;
                hx += f0;
                hy += f1;
                hz += f2;
              }
            }
            if (GRAD) {
              // the row's forces on its candidate: lanes 0, 2 and 4 of the row end with x, y and z
              const bool h4 = (lane & 4) != 0, h2 = (lane & 2) != 0;
              const T k0 = (h4 ? f2 : f0) + __shfl_xor_sync(0xffffffffu, h4 ? f0 : f2, 4);
              const T k1 = (h4 ? T(0) : f1) + __shfl_xor_sync(0xffffffffu, h4 ? f1 : T(0), 4);
              T v = (h2 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, h2 ? k0 : k1, 2);
              v += __shfl_xor_sync(0xffffffffu, v, 1);
              if ((lane & 1) == 0 && atom < 6) atomicAdd(&fx[(atom >> 1) * fstride + s], -v);
            }
          }
          if (GRAD) {
            // sum over the rows; the lanes of the group's own row keep it
            hx += __shfl_xor_sync(0xffffffffu, hx, 8);
            hy += __shfl_xor_sync(0xffffffffu, hy, 8);
            hz += __shfl_xor_sync(0xffffffffu, hz, 8);
            hx += __shfl_xor_sync(0xffffffffu, hx, 16);
            hy += __shfl_xor_sync(0xffffffffu, hy, 16);
            hz += __shfl_xor_sync(0xffffffffu, hz, 16);
            if (crow == g) {
              gx += hx;
              gy += hy;
              gz += hz;
            }
          }
        }
        __syncwarp();
      } while (more);
      if (GRAD && active && C.r_mask[slot] == 1) {
        for (int m = 0; m < C.nmr; ++m) {
          const double* M = C.r_modes + (size_t)m * 3 * nslots + slot;
          grec[m] += (T)M[0] * gx + (T)M[nslots] * gy + (T)M[2 * (size_t)nslots] * gz;
        }
      }
    }
    __syncthreads();
    // pose results: energy (and gradient) reduced in FP64 over the block
    double acc[1 + 6 + 2 * SD_MAX_MODES];
    const int ng = GRAD ? 6 + C.nmr + C.nml : 0;
    acc[0] = es;
    if (GRAD) {
      for (int k = 1; k <= ng; ++k) acc[k] = 0.0;
      for (int m = 0; m < C.nmr; ++m) acc[1 + 6 + m] = (double)grec[m];
      // ligand side: F_j projected on t, w, ligand modes
      double Rm[9];
      {
        // rotation of rotate() for the (possibly non-unit) quaternion, in FP64
        const double* q = sh_q;
        const double n2 = q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3];
        const double w0 = q[0], x = q[1], y = q[2], z = q[3];
        Rm[0] = (w0 * w0 + x * x - y * y - z * z) / n2;
        Rm[1] = 2 * (x * y - w0 * z) / n2;
        Rm[2] = 2 * (x * z + w0 * y) / n2;
        Rm[3] = 2 * (x * y + w0 * z) / n2;
        Rm[4] = (w0 * w0 - x * x + y * y - z * z) / n2;
        Rm[5] = 2 * (y * z - w0 * x) / n2;
        Rm[6] = 2 * (x * z - w0 * y) / n2;
        Rm[7] = 2 * (y * z + w0 * x) / n2;
        Rm[8] = (w0 * w0 - x * x - y * y + z * z) / n2;
      }
      for (int s = tid; s < nls; s += blockDim.x) {
        if (C.l_perm[s] < 0) continue;
        const double Fx = (double)fx[s], Fy = (double)fx[fstride + s], Fz = (double)fx[2 * fstride + s];
        const double px = (double)la[s].x, py = (double)la[s].y, pz = (double)la[s].z;  // l_j - t
        acc[1] += Fx;
        acc[2] += Fy;
        acc[3] += Fz;
        acc[4] += py * Fz - pz * Fy;
        acc[5] += pz * Fx - px * Fz;
        acc[6] += px * Fy - py * Fx;
        if (C.l_mask[s] == 1)
          for (int m = 0; m < C.nml; ++m) {
            const double* M = C.l_modes + (size_t)m * 3 * nls + s;
            const double M0 = M[0], M1 = M[nls], M2 = M[2 * (size_t)nls];
            const double RMx = Rm[0] * M0 + Rm[1] * M1 + Rm[2] * M2;
            const double RMy = Rm[3] * M0 + Rm[4] * M1 + Rm[5] * M2;
            const double RMz = Rm[6] * M0 + Rm[7] * M1 + Rm[8] * M2;
            acc[1 + 6 + C.nmr + m] += RMx * Fx + RMy * Fy + RMz * Fz;
          }
      }
    }
    for (int k = 0; k <= ng; ++k) {
      const double v = warp_sum<double>(acc[k]);
      if (lane == 0) sh_red[warp][k] = v;
    }
    __syncthreads();
    if (tid <= ng) {
      double v = 0.0;
      for (int i = 0; i < kPdWarps; ++i) v += sh_red[i][tid];
      if (tid == 0) {
        C.scoring[p] = -v;
        if (L.energy_out) L.energy_out[p] = v;
        ++n_done;
      } else if (GRAD && out_grad) {
        out_grad[(size_t)p * ng + (tid - 1)] = v;
      }
    }
  }
  if (tid == 0 && n_done) atomicAdd(&ctl->stats[ST_SCORED], n_done);
}

// bytes of a CTA's per-pose arrays, and of its warps' buffers in front of them (always shared memory)
size_t pydock_smem_bytes(int precision, bool grad, int max_nl, int max_nr) {
  const size_t nlc = (size_t)(max_nl + SD_TILE - 1) / SD_TILE, nls = nlc * SD_TILE;
  const size_t ts = precision == SD_PREC_MIXED ? 4 : 8;
  return ts * (4 * (nls + 1) + (grad ? 3 * (nls + 4) : 0)) + 16 * nlc + 4 * (nls + 1) +
         12 * ((max_nr + SD_TILE - 1) / SD_TILE) + 16;
}
size_t pydock_warp_bytes(int precision) {
  return kPdWarps * (precision == SD_PREC_MIXED ? sizeof(PdWarp<float>) : sizeof(PdWarp<double>));
}

const void* pydock_kernel_ptr(int precision, bool grad, bool spill) {
  if (precision == SD_PREC_MIXED) {
    if (spill) return grad ? (const void*)pydock_kernel<float, true, true> : (const void*)pydock_kernel<float, false, true>;
    return grad ? (const void*)pydock_kernel<float, true, false> : (const void*)pydock_kernel<float, false, false>;
  }
  if (spill) return grad ? (const void*)pydock_kernel<double, true, true> : (const void*)pydock_kernel<double, false, true>;
  return grad ? (const void*)pydock_kernel<double, true, false> : (const void*)pydock_kernel<double, false, false>;
}

int pydock_launch(const ScoreLaunch& L, int precision, bool grad, double* out_grad, int grid, size_t smem,
                  cudaStream_t st, bool spill) {
  ScoreLaunch l = L;
  void* args[] = {(void*)&l, (void*)&out_grad};
  if (cudaLaunchKernel(pydock_kernel_ptr(precision, grad, spill), dim3(grid), dim3(kPdWarps * 32), args,
                       smem, st) != cudaSuccess)
    return SD_ERR_CUDA;
  return cudaGetLastError() == cudaSuccess ? SD_OK : SD_ERR_CUDA;
}

int pydock_threads() { return kPdWarps * 32; }

}  // namespace sd
