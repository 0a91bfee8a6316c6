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
// Kernel: one CTA (4 to 24 warps, PdShape) per pose at a time, persistent over a work list; receptor tiles
// of 32 (one lane per atom) culled against the ligand sphere and against spatial ligand chunks, and
// each tile's candidate ligand atoms against the bounding boxes of its four groups of 8 atoms (45 %
// of a group's listed pairs are inside the cutoff, 21 % of a tile's).  A step evaluates 8 receptor
// atoms x 8 candidates of one group, two atoms per lane (FP32 in packed instructions).  GRAD adds
// per-lane receptor force accumulators (summed over the rows at the end of a group, projected onto
// the receptor modes at the end of each tile) and per-ligand-atom force accumulators in shared
// memory (a row's three components reduced together in three shuffles, one shared atomic), projected
// onto t, w and the ligand modes at the end of the pose.
//
// What bounds it: instruction issue (0.7 of the slots) and, with forces, the latency of the shuffles
// and shared atomics; memory traffic is small.  Measured on 3002 / 1274 atoms, 4,096 poses, the whole
// call, against the earlier kernel (one candidate of a tile over all its lanes, 15 shuffles and 3
// atomics for two candidates): FP32 gradients 5.94 -> 3.65 ms, FP32 energies 3.68 -> 1.89 ms; 2,000 FP64
// energies 2.17 -> 1.33 ms, FP64 gradients 4.70 -> 2.43 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "sd_internal.h"
#include "sd_packed.cuh"
#include "sd_pose.cuh"

namespace sd {

namespace {

// Warps of a CTA and CTAs per SM of each shape.  PD_ORDINARY: 8 warps, as many CTAs as fit; FP32 gradients 12,
// two CTAs (their ligand forces take 24 bytes an atom).  PD_MID and PD_SMALL: FP32 gradients of smaller
// molecules (pydock_grad_shape).  PD_FEW: at most one pose per SM, so one CTA with all the warps that the
// registers allow, for a pose's time
__host__ __device__ constexpr int pd_warps(bool fp64, bool grad, int shape) {
  return shape == PD_FEW ? (grad && fp64 ? 16 : 24) : shape == PD_MID ? 8 : shape == PD_SMALL ? 4 : grad && !fp64 ? 12 : 8;
}
__host__ __device__ constexpr int pd_ctas(bool grad, int shape) {
  return shape == PD_FEW ? 1 : shape == PD_MID ? 3 : shape == PD_SMALL ? 6 : grad ? 2 : 4;
}
constexpr double kKe = 332.0636 / 4.0;

// an atom in shared memory (position relative to t, the ligand's negated, charge): one 16-byte load in FP32
template <class T>
struct alignas(16) LigAtom {
  T x, y, z, q;
};
// the LJ pair parameters of two types, read together
template <class T>
struct alignas(2 * sizeof(T)) LjPair {
  T eps, sig2;
};

// two values of T, one per receptor atom of a lane; FP32 in packed instructions
template <class T>
struct V2 {
  T a, b;
  __device__ __forceinline__ V2() {}
  __device__ __forceinline__ V2(T x, T y) : a(x), b(y) {}
  __device__ __forceinline__ explicit V2(T x) : a(x), b(x) {}
  __device__ __forceinline__ T first() const { return a; }
  __device__ __forceinline__ T second() const { return b; }
};
template <class T>
__device__ __forceinline__ V2<T> operator+(V2<T> x, V2<T> y) { return V2<T>(x.a + y.a, x.b + y.b); }
template <class T>
__device__ __forceinline__ V2<T> operator-(V2<T> x, V2<T> y) { return V2<T>(x.a - y.a, x.b - y.b); }
template <class T>
__device__ __forceinline__ V2<T> operator*(V2<T> x, V2<T> y) { return V2<T>(x.a * y.a, x.b * y.b); }
template <>
struct V2<float> {
  float2x v;
  __device__ __forceinline__ V2() {}
  __device__ __forceinline__ V2(float x, float y) : v(pack2(x, y)) {}
  __device__ __forceinline__ explicit V2(float x) : v(pack2(x, x)) {}
  __device__ __forceinline__ float first() const { float x, y; unpack2(v, x, y); return x; }
  __device__ __forceinline__ float second() const { float x, y; unpack2(v, x, y); return y; }
};
__device__ __forceinline__ V2<float> operator+(V2<float> x, V2<float> y) { x.v = add2(x.v, y.v); return x; }
// -0 read at run time: x y + (-0) is the product rounded once, and cannot be contracted with an addition
// that follows (a packed multiply followed by a packed add was, measured, whatever -fmad says)
__constant__ float c_minus_zero[2] = {-0.f, -0.f};
__device__ __forceinline__ V2<float> operator*(V2<float> x, V2<float> y) {
  x.v = fma2(x.v, y.v, pack2(c_minus_zero[0], c_minus_zero[1]));
  return x;
}
// x - y as x + (-1) y: the product is exact, so the difference is rounded once
__device__ __forceinline__ V2<float> operator-(V2<float> x, V2<float> y) { x.v = fma2(y.v, pack2(-1.f, -1.f), x.v); return x; }

// the switch at x with its constant 1 / (off2 - on2)^3 passed in, from its polynomial's value v and slope dv
template <class T>
__device__ __forceinline__ void pd_switch(T x, T on2, T off2, T v, T dv, T& s, T& ds) {
  const bool in = x > on2 && x < off2;
  s = in ? v : (x <= on2 ? T(1) : T(0));
  ds = in ? dv : T(0);
}

// the LJ term of a pair inside 8 A added to its energy and dE/dx
template <class T>
__device__ __forceinline__ void pd_lj(T x, const LjPair<T>* pl, T& e, T& de) {
  if (x < T(64)) {
    const LjPair<T> p = *pl;
    const T rden = T(1) / (x + T(0.5) * p.sig2);
    const T sv = p.sig2 * rden;
    const T s2 = sv * sv, s3 = s2 * sv, s6 = s3 * s3;
    const T v = T(4) * p.eps * (s6 - s3);
    const T dsv = -sv * rden;
    const T dv = T(4) * p.eps * (T(6) * s3 * s2 - T(3) * s2) * dsv;  // d(s^6 - s^3)/ds = 6 s^5 - 3 s^2
    const T a = T(64) - x, c = T(1) / T(3375);                       // (64 - 49)^3
    T s, ds;
    pd_switch<T>(x, T(49), T(64), a * a * (T(64) + T(2) * x - T(147)) * c, T(6) * a * (T(49) - x) * c, s, ds);
    e += T(0.1) * (v * s);
    de += T(0.1) * (dv * s + v * ds);
  }
}

// energies e and dE/dx of two pairs at squared distances x (both 0 from 225 on, where the switch is);
// two divisions per pair (1 / (x + 1) and, inside 8 A, 1 / (x + sig2 / 2)), every other quotient a
// product with them.  The LJ terms stand behind a branch of the whole warp: neighbours in a list are
// neighbours in space, so many steps have no pair inside 8 A
template <class T>
__device__ __forceinline__ void pd_pairs(V2<T> x, V2<T> qq, const LjPair<T>* l0, const LjPair<T>* l1, T (&e)[2],
                                         V2<T>& dedx) {
  const V2<T> y = x + V2<T>(T(1));
  const V2<T> inv(T(1) / y.first(), T(1) / y.second());
  // (the cutoff holds for charges that are not finite too: 0 of the switch times them would not be 0)
  const V2<T> el0 = qq * inv, el(x.first() < T(225) ? el0.first() : T(0), x.second() < T(225) ? el0.second() : T(0));
  const V2<T> a = V2<T>(T(225)) - x, c(T(1) / T(24389));  // (225 - 196)^3
  const V2<T> v = a * a * (V2<T>(T(225)) + V2<T>(T(2)) * x - V2<T>(T(588))) * c;
  const V2<T> dv = V2<T>(T(6)) * a * (V2<T>(T(196)) - x) * c;
  const T x0 = x.first(), x1 = x.second();
  T s[2], ds[2];
  pd_switch<T>(x0, T(196), T(225), v.first(), dv.first(), s[0], ds[0]);
  pd_switch<T>(x1, T(196), T(225), v.second(), dv.second(), s[1], ds[1]);
  const V2<T> S(s[0], s[1]), E = el * S;
  const V2<T> D = el * V2<T>(ds[0], ds[1]) - el * inv * S;
  e[0] = E.first();
  e[1] = E.second();
  dedx = D;
  if (__any_sync(0xffffffffu, x0 < T(64) || x1 < T(64))) {
    T d0 = D.first(), d1 = D.second();
    pd_lj<T>(x0, l0, e[0], d0);
    pd_lj<T>(x1, l1, e[1], d1);
    dedx = V2<T>(d0, d1);
  }
}

// The force on a ligand atom, summed by all warps.  FP32: a 64-bit fixed-point number in units of
// 1 / scale (a power of two that the host derives from the largest possible pair force, so the sum
// cannot overflow), as two 32-bit words added by integer shared atomics, which the hardware has (an FP32
// shared atomic is a compare-and-swap loop).  The sum is exact, so it does not depend on the order.  A
// value that is not finite (a charge or parameter was not) sets *bad.  FP64 keeps its own type: fixed
// point would be coarser than it.
template <class T>
struct Force {
  T v;
  static constexpr int kWords = 1;
};
template <>
struct Force<float> {
  unsigned v;
  static constexpr int kWords = 2;
};
__device__ __forceinline__ void add_force(Force<float>* f, int words, int i, float v, float scale, int* bad) {
  const float q = v * scale;
  if (!(fabsf(q) < 9.0e18f)) *bad = 1;
  const long long n = __float2ll_rn(q);
  const unsigned lo = (unsigned)n;
  const unsigned old = atomicAdd(&f[i].v, lo);
  const unsigned hi = (unsigned)(n >> 32) + (old + lo < lo ? 1u : 0u);
  if (hi) atomicAdd(&f[words + i].v, hi);
}
__device__ __forceinline__ double force_of(const Force<float>* f, int words, int i, float scale) {
  const long long n = (long long)((unsigned long long)f[words + i].v << 32 | f[i].v);
  return (double)n / (double)scale;
}
__device__ __forceinline__ void add_force(Force<double>* f, int, int i, double v, float, int*) {
  atomicAdd(&f[i].v, v);
}
__device__ __forceinline__ double force_of(const Force<double>* f, int, int i, float) { return f[i].v; }

constexpr int kGroups = SD_TILE / SD_GROUP;
constexpr int kRow = SD_GROUP / 2;         // lanes of a row: one candidate, two atoms of the group per lane
constexpr int kRows = 32 / kRow;           // candidates of a step
constexpr int kPdList = 128;               // candidates of a group between two drains of the lists
constexpr int kOrderMax = 512;             // near tiles that are ordered by distance

// a warp's tile
template <class T>
struct PdWarp {
  LigAtom<T> rec[SD_TILE];           // receptor atoms (position relative to t, charge)
  float4 box[2 * kGroups];           // centre and half extent of each group's bounding box
  int lj[SD_TILE];
  unsigned short list[kGroups][kPdList];  // each group's candidates: ligand slots
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
// registers a thread) without forces: the pair terms are latency chains.
template <class T, bool GRAD, bool kSpill, int kShape>
__global__ void __launch_bounds__(pd_warps(sizeof(T) == 8, GRAD, kShape) * 32, pd_ctas(GRAD, kShape))
pydock_kernel(ScoreLaunch L, double* out_grad) {
  constexpr int kWarps = pd_warps(sizeof(T) == 8, GRAD, kShape);
  extern __shared__ __align__(16) unsigned char smem_dyn[];
  PdWarp<T>& W = reinterpret_cast<PdWarp<T>*>(smem_dyn)[threadIdx.x >> 5];
  unsigned char* const smem =
      kSpill ? L.spill + (size_t)blockIdx.x * L.spill_stride : smem_dyn + kWarps * sizeof(PdWarp<T>);
  __shared__ double sh_pose[7 + 2 * SD_MAX_MODES];
  __shared__ double sh_q[4], sh_qi[4];
  __shared__ LjPair<T> sh_lj[SD_LJ_TYPES * SD_LJ_TYPES];
  __shared__ double sh_red[kWarps][32];
  __shared__ float sh_rot[9];
  __shared__ float sh_bound[2];
  __shared__ int sh_item, sh_ntile, sh_next, sh_bad;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt_mask = (1u << lane) - 1u;
  const int atom = lane & (kRow - 1), crow = lane / kRow;  // a step's first atom (the other: + kRow) and row
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
      sh_bad = 0;
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
    // per-pose arrays: ligand atoms [nls + 1] (the last a far atom, the padding), GRAD: their forces
    // [words][3][nls + 4], chunk spheres [nlc], near tiles [ntiles] as found, the same in order of distance
    // and their distances (each [kOrderMax] at most: more are not ordered), LJ types [nls + 1]
    LigAtom<T>* la = reinterpret_cast<LigAtom<T>*>(smem);
    Force<T>* fx = reinterpret_cast<Force<T>*>(la + nls + 1);  // GRAD only
    const int fstride = nls + 4;
    float4* chS = reinterpret_cast<float4*>(fx + (GRAD ? Force<T>::kWords * 3 * fstride : 0));
    int* tlist = reinterpret_cast<int*>(chS + nlc);
    int* tord = tlist + C.ntiles;
    float* tdist = reinterpret_cast<float*>(tord + min(C.ntiles, kOrderMax));
    unsigned char* llj = reinterpret_cast<unsigned char*>(tdist + min(C.ntiles, kOrderMax));
    if (tid == 0) {
      la[nls] = LigAtom<T>{(T)1e17, (T)1e17, (T)1e17, T(0)};
      llj[nls] = 0;
    }
    if (GRAD)
      for (int s = tid; s < Force<T>::kWords * 3 * fstride; s += blockDim.x) fx[s].v = 0;
    for (int s = tid; s < nls; s += blockDim.x) {
      if (C.l_perm[s] >= 0) {
        double x, y, z;
        ligand_exact(C, s, sh_pose, sh_q, sh_qi, x, y, z);
        la[s] = LigAtom<T>{-(T)(x - tx), -(T)(y - ty), -(T)(z - tz), (T)(kKe * (double)C.l_q[s])};
        llj[s] = (unsigned char)C.l_lj[s];
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
        if (at < kOrderMax) tdist[at] = dd;
      }
    }
    __syncthreads();
    const int ntile = sh_ntile;
    // the tiles closest to the ligand centre (t) have the most pairs: taken first, the warps finish a
    // pose together
    const bool sorted = ntile <= kOrderMax;
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
        if (lane % SD_GROUP == 0) {
          W.box[2 * (lane / SD_GROUP)] =
              make_float4(0.5f * (lo[0] + hi[0]), 0.5f * (lo[1] + hi[1]), 0.5f * (lo[2] + hi[2]), 0.f);
          W.box[2 * (lane / SD_GROUP) + 1] =
              make_float4(half_extent(lo[0], hi[0]), half_extent(lo[1], hi[1]), half_extent(lo[2], hi[2]), 0.f);
        }
      }
      __syncwarp();
      T gx = T(0), gy = T(0), gz = T(0);  // dE/dr of this lane's atom of the tile
      int ncand = 0, cb = 0;
      unsigned cm = 0;
      bool more = true;
      do {
        // fill each group's list until the ligand is exhausted or a list may overflow
        unsigned cnt[kGroups];
#pragma unroll
        for (int g = 0; g < kGroups; ++g) cnt[g] = 0;
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
            const float ax = (float)ca.x + cx, ay = (float)ca.y + cy, az = (float)ca.z + cz;
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
          for (int g = 0; g < kGroups; ++g) {
            const float4 bc = W.box[2 * g], bh = W.box[2 * g + 1];
            const float ex = fmaxf(fabsf(x + bc.x) - bh.x, 0.f), ey = fmaxf(fabsf(y + bc.y) - bh.y, 0.f),
                        ez = fmaxf(fabsf(z + bc.z) - bh.z, 0.f);
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
        for (int g = 0; g < kGroups; ++g)
          if (lane < kRows) W.list[g][cnt[g] + lane] = (unsigned short)nls;
        __syncwarp();
        unsigned counts = cnt[0] | cnt[1] << 8 | cnt[2] << 16 | cnt[3] << 24;
        for (int g = 0; g < kGroups; ++g, counts >>= 8) {
          if ((counts & 255u) == 0) continue;
          const LigAtom<T> ra = W.rec[g * SD_GROUP + atom], rb = W.rec[g * SD_GROUP + atom + kRow];
          const V2<T> rx(ra.x, rb.x), ry(ra.y, rb.y), rz(ra.z, rb.z), rq(ra.q, rb.q);
          // the LJ table is symmetric (products and sums of the two types' parameters), so it is read as
          // [ligand type][receptor type]: the lanes of one candidate read entries of one row
          const LjPair<T>* lja = sh_lj + W.lj[g * SD_GROUP + atom];
          const LjPair<T>* ljb = sh_lj + W.lj[g * SD_GROUP + atom + kRow];
          const unsigned short* list = W.list[g] + crow;
          const int n = (int)(counts & 255u);
          V2<T> hx(T(0)), hy(T(0)), hz(T(0));  // dE/dr of this lane's pairs
          for (int c = 0; c < n; c += kRows) {
            const int s = list[c];
            const LigAtom<T> l = la[s];
            const int lj = llj[s] * SD_LJ_TYPES;
            const V2<T> dx = rx + V2<T>(l.x), dy = ry + V2<T>(l.y), dz = rz + V2<T>(l.z);
            const V2<T> x = dx * dx + dy * dy + dz * dz;
            T e[2];
            V2<T> dedx;
            pd_pairs<T>(x, rq * V2<T>(l.q), lja + lj, ljb + lj, e, dedx);
            es += (double)e[0];
            es += (double)e[1];
            if (GRAD) {
              const V2<T> g2 = V2<T>(T(2)) * dedx;
              const V2<T> fx2 = g2 * dx, fy2 = g2 * dy, fz2 = g2 * dz;
              hx = hx + fx2;
              hy = hy + fy2;
              hz = hz + fz2;
              // the row's forces on its candidate: lanes 0, 1 and 2 of the row end with x, y and z
              const T f0 = fx2.first() + fx2.second(), f1 = fy2.first() + fy2.second(), f2 = fz2.first() + fz2.second();
              const bool h2 = (lane & 2) != 0, h1 = (lane & 1) != 0;
              const T k0 = (h2 ? f2 : f0) + __shfl_xor_sync(0xffffffffu, h2 ? f0 : f2, 2);
              const T k1 = (h2 ? T(0) : f1) + __shfl_xor_sync(0xffffffffu, h2 ? f1 : T(0), 2);
              const T v = (h1 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, h1 ? k0 : k1, 1);
              if (atom < 3) add_force(fx, 3 * fstride, atom * fstride + s, -v, L.force_scale, &sh_bad);
            }
          }
          if (GRAD) {
            // sum over the rows; the lanes of the group's own atoms keep it
            T a[6] = {hx.first(), hy.first(), hz.first(), hx.second(), hy.second(), hz.second()};
#pragma unroll
            for (int k = 0; k < 6; ++k)
#pragma unroll
              for (int o = kRow; o < 32; o <<= 1) a[k] += __shfl_xor_sync(0xffffffffu, a[k], o);
            if (lane / SD_GROUP == g) {
              const bool second = (lane & kRow) != 0;
              gx += second ? a[3] : a[0];
              gy += second ? a[4] : a[1];
              gz += second ? a[5] : a[2];
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
      for (int k = 1; k <= ng; ++k) acc[k] = sh_bad ? nan("") : 0.0;
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
        const double Fx = force_of(fx, 3 * fstride, s, L.force_scale),
                     Fy = force_of(fx, 3 * fstride, fstride + s, L.force_scale),
                     Fz = force_of(fx, 3 * fstride, 2 * fstride + s, L.force_scale);
        const double px = -(double)la[s].x, py = -(double)la[s].y, pz = -(double)la[s].z;  // l_j - t
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
      for (int i = 0; i < kWarps; ++i) v += sh_red[i][tid];
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
  const size_t nt = (size_t)(max_nr + SD_TILE - 1) / SD_TILE;
  const size_t ts = precision == SD_PREC_MIXED ? 4 : 8;
  // forces: 24 bytes an atom in both types
  return ts * 4 * (nls + 1) + (grad ? 24 * (nls + 4) : 0) + 16 * nlc + (nls + 1) +
         4 * nt + 8 * std::min<size_t>(nt, kOrderMax) + 16;
}
size_t pydock_warp_bytes(int precision, bool grad, int shape) {
  const bool fp64 = precision != SD_PREC_MIXED;
  return pd_warps(fp64, grad, shape) * (fp64 ? sizeof(PdWarp<double>) : sizeof(PdWarp<float>));
}

// The scale of FP32 ligand forces: pair forces are at most 0.7 kKe q q' (electrostatics) plus 1.6 eps
// (3072 / sig^2 + 26) (LJ: |6 s^5 - 3 s^2| <= 192, s^2 <= 4, within 8 A; over the type pairs that occur: bit a of
// rec_types, bit b of lig_types), times the receptor's atoms.  0 where the unit would be coarser than 2^-30
// (charges of 100 and more on both sides, or a sigma below 0.01 A) or no bound exists: FP64 gradients then.
float pydock_force_scale(double max_q_rec, double max_q_lig, const double* eps, const double* sigma,
                         unsigned rec_types, unsigned lig_types, int max_nr) {
  double lj = 0;
  for (int a = 0; a < SD_LJ_TYPES; ++a)
    for (int b = 0; b < SD_LJ_TYPES; ++b) {
      if (!(rec_types >> a & 1u) || !(lig_types >> b & 1u)) continue;
      const double e = std::sqrt(eps[a] * eps[b]), sg = 0.5 * (sigma[a] + sigma[b]);
      const double v = 1.6 * e * ((sg != 0 ? 3072.0 / (sg * sg) : 0.0) + 26.0);
      if (!std::isfinite(v)) return 0.f;
      lj = std::max(lj, v);
    }
  const double f = (0.7 * kKe * max_q_rec * max_q_lig + lj) * std::max(8, max_nr);
  if (!(f <= 0x1p31)) return 0.f;
  const int k = (int)std::floor(61.0 - std::log2(std::max(f, 1e-9)));
  return std::ldexp(1.0f, std::min(100, k));
}

// The shape of a gradient call of many poses: FP32 takes the one with the most warps resident on an SM beside the
// arrays of a complex of this size (7 KiB of a CTA are its static arrays, 1 KiB the system's), the smallest
// CTAs among equals, as a warp without a tile only waits.  4,096 poses, ms with 4 x 6, 8 x 3 and 12 x 2 warps x
// CTAs: 200/100 atoms 0.42, 0.59, 0.76; 757/481 1.29, 1.35, 1.75; 1500/700 2.1, 1.88, 2.28; 3002/1274 5.4, 3.50,
// 3.65; 3002/1766 9.8, 5.8, 4.72; 3002/2100 11.8, 6.9, 8.3; 3002/2500 24, 13.2, 9.7.  (12 warps for all sizes were
// slower than the earlier kernel for the smallest: 0.76 against 0.69 ms.)
// Where all poses are resident in that shape at once, the warps of a pose count: then the fewest rounds over the
// warps that have a part of it.  (757/481: 300 poses 0.34 ms in 4 x 6, 0.23 in 8 x 3, 0.27 in 12 x 2.)
// Where shared memory holds one CTA only, two with their arrays in global scratch (PD_SCRATCH) have more warps: 2,000
// poses of 757/2500 atoms 3.85 -> 3.18 ms in FP32, 5.0 -> 3.3 ms in FP64, 50/3503 4.4 -> 2.4 ms in FP64.
int pydock_grad_shape(int precision, int nl, int nr, int poses, int smem_sm, int nsm) {
  const size_t need = pydock_smem_bytes(precision, true, nl, nr);
  int ctas[4] = {}, best = PD_ORDINARY;
  for (int shape : {PD_ORDINARY, PD_MID, PD_SMALL}) {
    if (precision != SD_PREC_MIXED && shape != PD_ORDINARY) continue;
    const size_t cta = need + pydock_warp_bytes(precision, true, shape) + (precision == SD_PREC_MIXED ? 8192 : 10240);
    ctas[shape] = std::min((int)(smem_sm / cta), pd_ctas(true, shape));
    const int warps = pd_warps(precision != SD_PREC_MIXED, true, shape);
    if (ctas[shape] * warps >= ctas[best] * pd_warps(precision != SD_PREC_MIXED, true, best)) best = shape;
  }
  if (ctas[PD_ORDINARY] == 0 || (ctas[best] == 1 && poses > nsm)) return PD_SCRATCH;
  if (precision != SD_PREC_MIXED || poses > ctas[best] * nsm) return best;
  // (tiles, or chunks of the ligand, whose atoms are placed and whose forces are projected by all warps)
  const int parts = (std::max(nr, nl) + SD_TILE - 1) / SD_TILE;
  double least = 1e300;
  for (int shape : {PD_SMALL, PD_MID, PD_ORDINARY}) {
    if (ctas[shape] == 0) continue;
    const int rounds = (poses + ctas[shape] * nsm - 1) / (ctas[shape] * nsm);
    const double time = (double)rounds / std::min(pd_warps(false, true, shape), parts);
    if (time < least) {
      least = time;
      best = shape;
    }
  }
  return best;
}

template <class T, bool GRAD>
static const void* kernel_of(bool spill, int shape) {
  if (spill) return (const void*)pydock_kernel<T, GRAD, true, PD_ORDINARY>;
  if constexpr (GRAD && sizeof(T) == 4) {
    if (shape == PD_MID) return (const void*)pydock_kernel<T, GRAD, false, PD_MID>;
    if (shape == PD_SMALL) return (const void*)pydock_kernel<T, GRAD, false, PD_SMALL>;
  }
  return shape == PD_FEW ? (const void*)pydock_kernel<T, GRAD, false, PD_FEW>
                         : (const void*)pydock_kernel<T, GRAD, false, PD_ORDINARY>;
}

// (the spill instantiation has the ordinary shape: another is ignored with it)
const void* pydock_kernel_ptr(int precision, bool grad, bool spill, int shape) {
  if (precision == SD_PREC_MIXED)
    return grad ? kernel_of<float, true>(spill, shape) : kernel_of<float, false>(spill, shape);
  return grad ? kernel_of<double, true>(spill, shape) : kernel_of<double, false>(spill, shape);
}

int pydock_launch(const ScoreLaunch& L, int precision, bool grad, double* out_grad, int grid, size_t smem,
                  cudaStream_t st, bool spill, int shape) {
  ScoreLaunch l = L;
  void* args[] = {(void*)&l, (void*)&out_grad};
  if (cudaLaunchKernel(pydock_kernel_ptr(precision, grad, spill, shape), dim3(grid),
                       dim3(pydock_threads(precision, grad, spill ? PD_ORDINARY : shape)), args, smem, st) != cudaSuccess)
    return SD_ERR_CUDA;
  return cudaGetLastError() == cudaSuccess ? SD_OK : SD_ERR_CUDA;
}

int pydock_threads(int precision, bool grad, int shape) {
  return pd_warps(precision != SD_PREC_MIXED, grad, shape) * 32;
}

}  // namespace sd
