// DFIRE pair scoring of glowworm poses on sm_100a.
//
// Replaces the reference's pose kernels + DFIRE tile kernel + energy reduce
// (prepare_gso_task.cu:268-494, :1820-2286, :2377-2433) and follows the CPU semantics of
// cdfire_calculate_dfire (prepare_gso_tasks.cc:1522-1615):
//   E = sum_i ( sum_j [d2_ij <= 225] table[tR_i][tL_j][dist_to_bins[(int)(2 sqrt(d2)-1)]-1] )
//   score = -(0.0157 E - 4.7)
//
// Persistent kernels, one or two poses per CTA at a time, dynamic work grabbing:
//  * FP64_REF (here): every pair in FP64, each receptor atom's partial v_i summed in ascending j and
//    the pose energy over the v_i in ascending i, as the reference;
//  * FP64 (sd_score_fp64.cuh): the same sums, so the same bits, over the pairs that culling leaves;
//  * MIXED (sd_score_mixed.cuh): the same table values in another order of summation.
// FP64 and MIXED take distances from FP32 coordinates centred on the pose translation: an exact
// per-pair bin unless the distance lies within a proven error bound of a bin or cutoff edge, in which
// case the pair is decided in FP64 from the exact transforms.
#include <cuda_runtime.h>

#include <algorithm>

#include "sd_internal.h"
#include "sd_packed.cuh"
#include "sd_pose.cuh"

namespace sd {

__constant__ double c_T[32];   // exact FP64 key thresholds: key(d2) = #{m>=1 : T[m] <= d2}

void set_key_thresholds(const double* t) {
  double T[32];
  for (int m = 0; m < 32; ++m) T[m] = m < 30 ? t[m] : 1e300;
  cudaMemcpyToSymbol(c_T, T, sizeof T);
}

// dist_to_bins[key] - 1 (interface.h:30-35) for key 0..29; key 29 (d2 == 225) gives 20, which
// with the flat index reads the next ligand type's bin 0 exactly as the reference does.
__constant__ int c_binlut[32] = {0,  0,  0,  1,  2,  3,  4,  5,  6,  7,  8,  9,  10, 11, 12, 13,
                                 13, 14, 14, 15, 15, 16, 16, 17, 17, 18, 18, 19, 19, 20, 20, 20};

struct LigD {
  double x, y, z;
  int col;
  int pad;
};

__device__ __forceinline__ int exact_key(double d2, const double* T) {
  float f = sqrtf((float)d2) * 2.0f - 1.0f;
  int k = (int)f;
  k = k < 0 ? 0 : (k > 29 ? 29 : k);
  if (k < 29 && d2 >= T[k + 1]) ++k;
  else if (k > 0 && d2 < T[k]) --k;
  return k;
}

// SD_PREC_FP64_REF: all Nr*Nl pairs in FP64, one lane per receptor atom, ligand atoms in order.  16
// warps per CTA: the per-pose shared memory (receptor accumulators, ligand atoms) allows two CTAs per
// SM, so the warps per CTA set the SM's residency.  kSpill: the per-pose arrays live in this CTA's slice
// of the global scratch L.spill instead (complexes too large for shared memory); the arithmetic is the
// same.
constexpr int kRefThreads = 512;

template <bool kSpill>
__global__ void __launch_bounds__(kRefThreads) dfire_score_ref_kernel(ScoreLaunch L) {
  extern __shared__ __align__(16) unsigned char smem_dyn[];
  unsigned char* const smem = kSpill ? L.spill + (size_t)blockIdx.x * L.spill_stride : smem_dyn;
  __shared__ double sh_pose[7 + 2 * SD_MAX_MODES];
  __shared__ double sh_q[4], sh_qi[4];
  __shared__ double sh_T[32];
  __shared__ int sh_lut[32];
  __shared__ int sh_item, sh_next;
  __shared__ unsigned long long sh_z, sh_cut, sh_pairs, sh_evals;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < 32) {
    sh_T[tid] = c_T[tid];
    sh_lut[tid] = c_binlut[tid];
  }
  if (tid == 0) {
    sh_z = 0;
    sh_cut = 0;
    sh_pairs = 0;
    sh_evals = 0;
  }
  unsigned long long n_pairs = 0, n_evals = 0;  // per thread
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
    const int nl = C.nl, nr = C.nr, nslots = nslots_of(C), pl = C.pl;
    const double* pose_g = C.pos + (size_t)p * pl;
    if (tid < pl) sh_pose[tid] = pose_g[tid];
    __syncthreads();
    if (tid == 0) {
      sh_q[0] = sh_pose[3];
      sh_q[1] = sh_pose[4];
      sh_q[2] = sh_pose[5];
      sh_q[3] = sh_pose[6];
      quat_inverse(sh_q, sh_qi);
      sh_next = 0;
    }
    __syncthreads();
    // ---- ligand of this pose into shared memory ----
    const double tx = sh_pose[0], ty = sh_pose[1], tz = sh_pose[2];
    LigD* ligD = reinterpret_cast<LigD*>(smem);
    double* vacc = reinterpret_cast<double*>(ligD + nl);
    for (int s = tid; s < C.nlchunks * SD_TILE; s += blockDim.x) {
      const int j = C.l_perm[s];
      if (j < 0) continue;
      double x, y, z;
      ligand_exact(C, s, sh_pose, sh_q, sh_qi, x, y, z);
      ligD[j] = LigD{x, y, z, C.l_col[s], 0};
    }
    for (int i = tid; i < nr; i += blockDim.x) vacc[i] = 0.0;
    if (tid == 0) {
      // ligand reference point (prepare_gso_tasks.cc:460, :513, :524-526)
      double x = C.lig_ref[0], y = C.lig_ref[1], z = C.lig_ref[2];
      quat_rotate(sh_q, sh_qi, x, y, z);
      double* ref = C.ref + (size_t)p * 3;
      ref[0] = x + tx;
      ref[1] = y + ty;
      ref[2] = z + tz;
    }
    __syncthreads();
    for (;;) {
      int k = 0;
      if (lane == 0) k = atomicAdd(&sh_next, 1);
      k = __shfl_sync(0xffffffffu, k, 0);
      if (k >= C.ntiles) break;
      const int slot = k * SD_TILE + lane;
      const int orig = C.r_orig[slot];
      if (orig < 0) continue;  // padding of the last tile
      double rx, ry, rz;
      receptor_exact(C, nslots, slot, sh_pose, rx, ry, rz);
      const int row = C.r_row[slot];
      double v = 0.0;  // FP64 partial of receptor atom `orig`
      for (int j = 0; j < nl; ++j) {
        const LigD l = ligD[j];
        const double ddx = rx - l.x, ddy = ry - l.y, ddz = rz - l.z;
        const double d2 = ddx * ddx + ddy * ddy + ddz * ddz;
        if (d2 <= SD_CUTOFF2) {
          int key;
          if (d2 == 0.0) {
            key = 0;
            atomicAdd(&sh_z, 1ull);
          } else {
            key = exact_key(d2, sh_T);
            if (key == 29) atomicAdd(&sh_cut, 1ull);
          }
          v += L.table64[row + l.col + sh_lut[key]];
          ++n_pairs;
        }
      }
      n_evals += nl;
      vacc[orig] = v;
    }
    __syncthreads();
    // reference order: E += v_i for i ascending (zero partials skipped)
    double E = 0.0;
    if (warp == 0) {
      for (int base = 0; base < nr; base += 32) {
        const double vv = base + lane < nr ? vacc[base + lane] : 0.0;
        unsigned m = __ballot_sync(0xffffffffu, vv != 0.0);
        while (m) {
          const int b = __ffs(m) - 1;
          m &= m - 1;
          E += __shfl_sync(0xffffffffu, vv, b);
        }
      }
    }
    if (tid == 0) {
      const double score = ((E)*0.0157 - 4.7) * -1;
      C.scoring[p] = score;
      if (L.energy_out) L.energy_out[p] = E;
      ++n_done;
    }
  }
  if (n_pairs) atomicAdd(&sh_pairs, n_pairs);
  if (n_evals) atomicAdd(&sh_evals, n_evals);
  __syncthreads();
  if (tid == 0) {
    if (sh_pairs) atomicAdd(&ctl->stats[ST_PAIRS], sh_pairs);
    if (sh_evals) atomicAdd(&ctl->stats[ST_EVALS], sh_evals);
    if (n_done) atomicAdd(&ctl->stats[ST_SCORED], n_done);
    if (sh_z) atomicAdd(&ctl->stats[ST_D2ZERO], sh_z);
    if (sh_cut) atomicAdd(&ctl->stats[ST_D2CUT], sh_cut);
  }
}

}  // namespace sd

#include "sd_score_mixed.cuh"
#include "sd_score_fp64.cuh"

namespace sd {

// compiled variants of the mixed DFIRE kernel (kernel, warps per CTA, minimum resident CTAs per
// SM); the host autotuner times them on the context's own poses and keeps the fastest
struct MixedVariant {
  const void* fn;
  int warps;
  int min_blocks;
};
#define SD_MIXED(W, B) { (const void*)dfire_score_mixed_kernel<W, B, false, false>, W, B }
#define SD_MIXED_WIDE(W, B) { (const void*)dfire_score_mixed_kernel<W, B, false, true>, W, B }
// 24 or 28 warps per SM in all of them (80 or 72 registers a thread).  Fewer and larger CTAs hold fewer
// copies of the ligand in shared memory and leave L1 more room for gathers in flight; smaller ones
// lose less at the end of a batch.  Measured (M poses/s for 12x2, 14x2, 8x3, 6x4): 757/481 atoms 7.4,
// 7.2, 9.5, 9.7; 3002/1274 2.97, 3.01, 2.36, 2.78; 6032/1766 1.90, 1.50, 1.77, 1.41; 17307/1125 2.50,
// 2.58, 2.04, 2.31.  Variant 0 is the default before the autotuner has run.  The variants give
// bit-identical energies (same per-tile work and summation order), so the tuner's choice never changes
// a result.
static const MixedVariant kMixedVariants[] = {
    SD_MIXED(12, 2), SD_MIXED(14, 2), SD_MIXED(8, 3), SD_MIXED(6, 4),
};
static const MixedVariant kMixedWide[] = {
    SD_MIXED_WIDE(12, 2), SD_MIXED_WIDE(14, 2), SD_MIXED_WIDE(8, 3), SD_MIXED_WIDE(6, 4),
};
// stateless calls with at most one pose per SM: one CTA per SM with as many warps as fit, for a pose's
// time (100 poses of 2000 / 1000 atoms, the whole call: 138 us with 12 warps, 124 us with 24)
static const MixedVariant kMixedFew = SD_MIXED(24, 1), kMixedFewWide = SD_MIXED_WIDE(24, 1);
// the spill instantiation of the mixed kernel: variant 0's shape (the per-tile work, and so every
// energy, is the same in every variant)
static const MixedVariant kMixedSpill = {(const void*)dfire_score_mixed_kernel<12, 2, true, true>, 12, 2};

// shapes of the culled FP64 kernel, the smallest CTAs first (fp64_shape)
static const MixedVariant kFp64Shapes[] = {
    {(const void*)dfire_score_fp64_kernel<4, 6, false>, 4, 6},
    {(const void*)dfire_score_fp64_kernel<6, 4, false>, 6, 4},
    {(const void*)dfire_score_fp64_kernel<8, 3, false>, 8, 3},
    {(const void*)dfire_score_fp64_kernel<12, 2, false>, 12, 2},
    {(const void*)dfire_score_fp64_kernel<24, 1, false>, 24, 1},
    {(const void*)dfire_score_fp64_kernel<16, 1, false>, 16, 1},
    {(const void*)dfire_score_fp64_kernel<8, 1, false>, 8, 1},
};
static const MixedVariant kFp64Spill = {(const void*)dfire_score_fp64_kernel<12, 2, true>, 12, 2};
constexpr int kNumFp64Shapes = sizeof(kFp64Shapes) / sizeof(kFp64Shapes[0]);

constexpr int kNumMixedVariants = sizeof(kMixedVariants) / sizeof(kMixedVariants[0]);
static_assert(sizeof(kMixedWide) == sizeof(kMixedVariants), "wide forms of all variants");
static_assert(kNumMixedVariants <= SD_MAX_VARIANTS, "variant table");

static const MixedVariant& mixed_variant(int v) {
  const bool wide = (v & SD_WIDE) != 0;
  v &= ~SD_WIDE;
  if (v == SD_FEW) return wide ? kMixedFewWide : kMixedFew;
  if (v >= kNumMixedVariants) v = 0;
  return wide ? kMixedWide[v] : kMixedVariants[v];
}

// whether tiles may meet more than kNear pairs near an edge: their share of the pairs grows with the ligand's
// radius (1.8e-4 at 64 A, and a tile in an overlapping pose meets 12,800 pairs at most, so 2 of them; compact
// ligands have 24 A at 1,274 atoms and 60 A at 20,000)
bool wide_ligand(float radius) { return !(radius <= 64.f); }

// bytes of the scorer's per-warp buffers, in dynamic shared memory in front of the per-pose arrays
// (alone there in the spill instantiation)
size_t score_warp_bytes(int precision, int scoring, int variant, bool spill) {
  if (scoring == SD_SCORING_PYDOCK) return pydock_warp_bytes(precision, false, !spill && variant == SD_FEW ? PD_FEW : PD_ORDINARY);
  if (precision == SD_PREC_FP64_REF) return 0;
  if (precision == SD_PREC_FP64) return sizeof(OrdBufs) * (spill ? kFp64Spill : kFp64Shapes[variant]).warps;
  return sizeof(WarpBufs) * (spill ? kMixedSpill.warps : mixed_variant(variant).warps);
}

// bytes of a CTA's per-pose arrays; poses: of the mixed DFIRE scorer's batch (the others take one)
size_t score_smem_bytes(int precision, int scoring, int max_nr, int max_nl, int poses) {
  if (scoring == SD_SCORING_PYDOCK) return pydock_smem_bytes(precision, false, max_nl, max_nr);
  if (precision == SD_PREC_MIXED) {
    const size_t nlc = (size_t)(max_nl + SD_TILE - 1) / SD_TILE;
    const size_t ntiles = (size_t)(max_nr + SD_TILE - 1) / SD_TILE;
    return poses * (8 * ((ntiles + 1) & ~(size_t)1) + 16 * (nlc * SD_TILE + 1 + nlc)) + 4 * (3 * ntiles + nlc);
  }
  if (precision == SD_PREC_FP64) {
    const size_t nls = (size_t)(max_nl + SD_TILE - 1) / SD_TILE * SD_TILE;
    return (size_t)8 * ((max_nr + 1) & ~1) + 16 * (nls + 1) + (size_t)12 * ((max_nr + SD_TILE - 1) / SD_TILE);
  }
  return (size_t)32 * max_nl + (size_t)8 * max_nr;
}

// The culled FP64 kernel's shape for these sizes and at most `poses` poses (1 KiB of each CTA is the system's, 1 KiB
// covers the static arrays); the last one when none fits (the caller then spills).  Small CTAs lose least where
// warps wait for each other at a pose's end, so the first whose CTAs are all resident is taken (the v_i of a large
// receptor fill the shared memory).  Where it has all poses resident at once, a pose's time counts: the fewest
// rounds over the warps that have a tile, among equals the fewest rounds, then the most registers.  Measured, M poses/s of
// large calls with 4x6, 6x4, 8x3, 12x2, 16x1, 8x1 (* its CTAs are not all resident): 757/481 5.66, 5.60, 5.25,
// 4.00, 2.58, 2.57; 1000/800 3.16*, 3.46, 3.42, 2.79, 1.82, 1.72; 1700/600 3.26*, 3.61, 3.74, 3.16, 2.08, 1.94;
// 2516/1061 -, 1.82*, 2.04, 2.06, 1.42, 1.09; 3002/1274 -, -, 1.40*, 1.72, 1.26, 0.89; 12000/300 16x1 2.39, 8x1 2.16;
// 21500/500 16x1 1.69 (spilled), 8x1 1.28.  Microseconds of 16 and 200 poses of 3002/1274: 12x2 199, 250; 16x1 174,
// 275; 8x1 235, 387; of 200/100: 12x2 62, 70; 16x1 54, 80; 8x1 53, 78.  24x1 has 80 registers a thread against 128
// of 16x1 and is slower but for large ligands, which all threads place and list: 6 poses with 24x1 and 16x1 of
// 3000/1274 174, 152; 700/4700 249, 238; 1500/2500 235, 202; 3000/2500 227, 241; 6000/4700 472, 497.
int fp64_shape(int max_nr, int max_nl, int smem_sm, int poses, int nsm) {
  const int ntiles = (max_nr + SD_TILE - 1) / SD_TILE;  // a warp without a tile only waits
  auto fits = [&](int v) {
    if (kFp64Shapes[v].warps == 24 && (max_nl <= 2048 || max_nr <= 1024)) return false;  // see above
    const size_t cta = score_smem_bytes(SD_PREC_FP64, SD_SCORING_DFIRE, max_nr, max_nl, 1) +
                       score_warp_bytes(SD_PREC_FP64, SD_SCORING_DFIRE, v, false) + 2048;
    return cta * kFp64Shapes[v].min_blocks <= (size_t)smem_sm;
  };
  int best = 0;
  while (best < kNumFp64Shapes - 1 && !fits(best)) ++best;
  if (poses > kFp64Shapes[best].min_blocks * nsm) return best;
  int rounds = 0, eff = 0;
  for (int v = best; v < kNumFp64Shapes; ++v) {
    if (!fits(v)) continue;
    const int slots = kFp64Shapes[v].min_blocks * nsm;
    const int r = std::max(1, (poses + slots - 1 - slots / 16) / slots);  // a few more share the first round
    const int e = std::min(kFp64Shapes[v].warps, ntiles);
    if (eff == 0 || r * eff < rounds * e || (r * eff == rounds * e && r <= rounds)) {
      rounds = r;
      eff = e;
      best = v;
    }
  }
  return best;
}
int mixed_variant_count() { return kNumMixedVariants; }
int mixed_variant_warps(int v) { return mixed_variant(v).warps; }
int mixed_variant_min_blocks(int v) { return mixed_variant(v).min_blocks; }

int score_threads_of(int precision, int scoring, int variant, bool spill) {
  if (scoring == SD_SCORING_PYDOCK) return pydock_threads(precision, false, !spill && variant == SD_FEW ? PD_FEW : PD_ORDINARY);
  if (precision == SD_PREC_FP64_REF) return kRefThreads;
  if (precision == SD_PREC_FP64) return (spill ? kFp64Spill : kFp64Shapes[variant]).warps * 32;
  return (spill ? kMixedSpill : mixed_variant(variant)).warps * 32;
}

const void* score_kernel_ptr(int precision, int scoring, int variant, bool spill) {
  if (scoring == SD_SCORING_PYDOCK) return pydock_kernel_ptr(precision, false, spill, variant == SD_FEW ? PD_FEW : PD_ORDINARY);
  switch (precision) {
    case SD_PREC_FP64_REF:
      return spill ? (const void*)dfire_score_ref_kernel<true> : (const void*)dfire_score_ref_kernel<false>;
    case SD_PREC_FP64: return (spill ? kFp64Spill : kFp64Shapes[variant]).fn;
    default: return (spill ? kMixedSpill : mixed_variant(variant)).fn;
  }
}

int score_launch(const ScoreLaunch& L, int precision, int scoring, int grid, size_t smem, cudaStream_t st, int variant,
                 bool spill) {
  if (scoring == SD_SCORING_PYDOCK)
    return pydock_launch(L, precision, false, nullptr, grid, smem, st, spill, variant == SD_FEW ? PD_FEW : PD_ORDINARY);
  ScoreLaunch l = L;
  void* args[] = {(void*)&l};
  if (cudaLaunchKernel(score_kernel_ptr(precision, scoring, variant, spill), dim3(grid),
                       dim3(score_threads_of(precision, scoring, variant, spill)), args, smem, st) != cudaSuccess)
    return SD_ERR_CUDA;
  return cudaGetLastError() == cudaSuccess ? SD_OK : SD_ERR_CUDA;
}

// ---- per-pair bins of one pose (parity/debug), thread per pair, by the steps of the precision's scorer: FP32
// terms and the exact transforms where they do not settle a pair, or the exact transforms alone (FP64_REF) ----
// C: the complex with pos at the pose and ref at three doubles that the prologue may write
__global__ void dfire_bins_kernel(DevComplex C, int precision, int* bins, int* fallback) {
  __shared__ PoseBufs Q;
  if (threadIdx.x < 32) pose_prologue(C, 0, Q, threadIdx.x);
  __syncthreads();
  const int nl = C.nl, nslots = nslots_of(C), nls = C.nlchunks * SD_TILE;
  const long long total = (long long)nslots * nl;
  const float cut2 = 225.0f + Q.B, inner = settled_half(Q.B);
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int slot = (int)(idx / nl), j = (int)(idx % nl);
    const int orig = C.r_orig[slot];
    if (orig < 0) continue;
    int bin = -1;
    bool settled = false;
    if (precision != SD_PREC_FP64_REF) {
      double r[1][3], l[1][3];
      anm_fused<1>(C.r_xyz, C.r_modes, C.r_mask, nslots, C.nmr, &Q.pose[7], 0, slot, r);
      anm_fused<1>(C.l_xyz, C.l_modes, C.l_mask, nls, C.nml, &Q.pose[7 + C.nmr], 0, C.l_slot[j], l);
      const float x = (float)(r[0][0] - Q.pose[0]), y = (float)(r[0][1] - Q.pose[1]), z = (float)(r[0][2] - Q.pose[2]);
      const double* R = Q.rot;
      const float4 lig = make_float4(-(float)fma(R[0], l[0][0], fma(R[1], l[0][1], R[2] * l[0][2])),
                                     -(float)fma(R[3], l[0][0], fma(R[4], l[0][1], R[5] * l[0][2])),
                                     -(float)fma(R[6], l[0][0], fma(R[7], l[0][1], R[8] * l[0][2])), 0.f);
      float d2[2], mid[2];
      int b[2];
      pair_terms(pack2(x, x), pack2(y, y), pack2(z, z), lig, d2, mid, b);
      settled = inner > 0.f && !(d2[0] <= cut2 && fabsf(mid[0]) >= inner);
      if (settled && d2[0] <= cut2) bin = b[0] - kMagicBits;
    }
    if (!settled) {
      if (precision != SD_PREC_FP64_REF) atomicAdd(fallback, 1);
      double rx, ry, rz, lx, ly, lz;
      receptor_exact(C, nslots, slot, Q.pose, rx, ry, rz);
      ligand_exact(C, C.l_slot[j], Q.pose, Q.q, Q.qi, lx, ly, lz);
      const double ddx = rx - lx, ddy = ry - ly, ddz = rz - lz;
      const double e2 = ddx * ddx + ddy * ddy + ddz * ddz;
      if (e2 <= SD_CUTOFF2) bin = c_binlut[e2 == 0.0 ? 0 : exact_key(e2, c_T)];
    }
    bins[(size_t)orig * nl + j] = bin;
  }
}

int bins_launch(const DevComplex& C, int precision, int* d_bins, int* d_fallback, cudaStream_t st) {
  dfire_bins_kernel<<<148 * 8, 256, 0, st>>>(C, precision, d_bins, d_fallback);
  return cudaGetLastError() == cudaSuccess ? SD_OK : SD_ERR_CUDA;
}

}  // namespace sd
