// Mixed-precision DFIRE scoring (included by sd_score.cu: shares its constant-memory key
// thresholds and exact_key).
//
// Same contract as the FP64 kernels: the energy of cdfire_calculate_dfire
// (prepare_gso_tasks.cc:1522-1615) with every bin identical to the FP64 reference bin, FP64 sums
// of FP64 table values, but in a free order, which the kernel uses:
//  * persistent CTAs take poses from the device work list, two at a time while there are plenty
//    (consecutive items are glowworms of one swarm, so they meet the same receptor tiles): one read
//    of a tile's or chunk's modes serves both.  Per pose the ligand is transformed (FP64, rounded to
//    FP32 centred on the pose translation t, stored negated) for the spatial chunks of 32 atoms that
//    some receptor tile within reach can reach, and the near receptor tiles are ordered largest-first
//    (closest to a ligand centroid) so warps finish a batch together;
//  * a warp takes a receptor tile (one lane per atom, FP64 ANM transform rounded to FP32), rejects
//    ligand chunks by bounding spheres and ligand atoms by the tile's sphere, and tests the survivors,
//    32 at a time, against the bounding boxes of the tile's four groups of 8 atoms (boxes of the
//    transformed atoms).  Each group has its own candidate list: the groups are small enough that 45 %
//    of the pairs of a group and its candidates are inside the cutoff (21 % for a whole tile and its
//    candidates), so every pair is evaluated where it stands, without a pre-filter or compaction;
//  * a step evaluates 8 atoms x 8 candidates, two atoms per lane in packed FP32 (pair_terms): d^2, d by
//    an approximate square root, the bin coordinate and its distance from the nearest edge.  A pair
//    inside the cutoff and further from an edge than the proven FP32 error has its FP64 bin, and its
//    value is gathered (through L2 only) and added by the next step, so that it is in flight while the
//    next step is evaluated.  A bit per step notes a pair near an edge; such pairs are found again after
//    the group's loop and decided in FP64 from the exact transforms (counted as fallbacks).  Each lane sums its values in FP64 (Kahan
//    sums of an FP32-rounded table were measured to miss 1e-5 at 60k pairs per pose);
//  * fixed summation order: a tile's lane sums are reduced by warp shuffles when the tile is done and
//    stored in a per-pose shared slot of that tile; at the end one warp per pose adds the slots in a
//    fixed order.  What happens inside a tile depends only on the pose and the tile, never on which
//    warp took it, when, or beside which other pose, and no compiled variant changes it, so a pose's
//    energy is the same bits in every run, every variant and every entry point.
//
// What bounds it: each gather is one sector from L2, and an SM receives about one per clock (random
// 8-byte gathers alone measured 2.9e11/s on 148 SMs at 1965 MHz).  On 3002 / 1274 atoms (57 k pairs
// in the cutoff per pose) it runs at 1.7e11 pairs/s, 0.58 of that; the modes' reads add a quarter to
// the sectors (half of that before two poses shared them), and L1 must hold the gathers in flight, so
// the shared memory a CTA takes costs speed too.  Measured on 8,000 to 20,000 poses, poses/s, against
// the earlier kernel (FP16 pre-filter of tile x candidate pairs, a ring of in-cutoff pairs, one pose
// per CTA): 3002/1274 2.34 M -> 3.01 M, 17307/1125 2.02 M -> 2.58 M, 6032/1766 1.34 M -> 1.90 M,
// 757/481 6.9 M -> 9.7 M.
#pragma once

namespace sd {
namespace {

constexpr int kGroup = SD_GROUP;      // receptor atoms of a group (one row of 8 lanes)
constexpr int kGroups = SD_TILE / kGroup;
constexpr int kRow = 8;               // candidates of a step: 8 rows of 4 lanes, two atoms of the group per lane
constexpr int kPoses = 2;             // poses of a batch: they share the reads of modes and tiles
constexpr int kList = 160;            // candidates of a group between two drains of the lists
constexpr int kNear = 16;             // pairs of a tile decided in FP64 side by side (more: decide_near)
static_assert(kList / kRow <= 32, "a bit per step");
static_assert(kGroups * kList * 2 >= 64 * 4, "decide_near collects up to 63 pairs in the lists");
constexpr float kMagic = 12582912.0f; // 1.5 * 2^23: adding it rounds to an integer in the low bits
constexpr int kMagicBits = 0x4B400000;

// one pose of a CTA's batch
struct __align__(16) PoseBufs {
  double pose[7 + 2 * SD_MAX_MODES + 1];
  double q[4], qi[4];
  double rot[9 + 1];
  float rotf[9];
  float gc[3];                       // ligand centroid, rotated (centred on t)
  float dR, dL, B;                   // bounds: receptor and ligand ANM displacement, FP32 error of d^2
  float pad;
};

struct __align__(16) WarpBufs {
  float4 rec[kPoses][SD_TILE];       // receptor atom of each lane centred on t, row bits
  float4 box[2 * kGroups];           // centre and half extent of each group's bounding box
  unsigned short list[kGroups][kList];  // each group's candidates: ligand slots
  unsigned near[kNear];              // pairs to decide in FP64: ligand slot * 32 + receptor lane
  unsigned short pend[64];           // pending candidate ligand slots of the tile (below SD_MAX_LIG)
};

// The table value of one pair decided in FP64 from the exact transforms (0 outside the cutoff); counts
// the pair in cnt[0], d^2 == 0 in cnt[1], d^2 == 225 in cnt[2] and a pair inside the cutoff in cnt[3].
// Not inlined: it is rare (about ten pairs of a pose), and inlined its registers slowed the pair loop.
__device__ __noinline__ double decide_pair(const DevComplex& C, const double* pose, const double* q, const double* qi,
                                           const double* T, const double* table, int slot, int s,
                                           unsigned long long* cnt) {
  double rx, ry, rz, lx, ly, lz;
  receptor_exact(C, nslots_of(C), slot, pose, rx, ry, rz);
  ligand_exact(C, s, pose, q, qi, lx, ly, lz);
  const double dx = rx - lx, dy = ry - ly, dz = rz - lz;
  const double e2 = dx * dx + dy * dy + dz * dz;
  atomicAdd(&cnt[0], 1ull);
  if (!(e2 <= SD_CUTOFF2)) return 0.0;
  atomicAdd(&cnt[3], 1ull);
  int key = 0;
  if (e2 == 0.0) {
    atomicAdd(&cnt[1], 1ull);
  } else {
    key = exact_key(e2, T);
    if (key == 29) atomicAdd(&cnt[2], 1ull);
  }
  return table[C.r_row[slot] + C.l_col[s] + c_binlut[key]];
}

__device__ __forceinline__ float sqrt_approx(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Two pairs of a lane (two receptor atoms, one candidate l, coordinates negated): FP32 d^2, the
// distance of the bin coordinate from the middle of its bin (0.5: on an edge) and the bin plus kMagicBits.
// Bin coordinate of distance d: min(2d - 3, d + 5) (bins of 0.5 A below 8 A, of 1 A above; below 2 A all
// bin 0), here less 0.5 so that rounding to the nearest integer is the floor, and no more than 20, so
// that a pair well outside the cutoff (19.5) is not near an edge.
__device__ __forceinline__ void pair_terms(float2x rx, float2x ry, float2x rz, const float4& l, float (&d2)[2],
                                           float (&mid)[2], int (&bin)[2]) {
  const float2x ex = add2(rx, pack2(l.x, l.x)), ey = add2(ry, pack2(l.y, l.y)), ez = add2(rz, pack2(l.z, l.z));
  unpack2(fma2(ez, ez, fma2(ey, ey, mul2(ex, ex))), d2[0], d2[1]);
  const float2x d = pack2(sqrt_approx(d2[0]), sqrt_approx(d2[1]));
  float a0, a1, b0, b1;
  unpack2(fma2(d, pack2(2.0f, 2.0f), pack2(-3.5f, -3.5f)), a0, a1);
  unpack2(add2(d, pack2(4.5f, 4.5f)), b0, b1);
  const float2x f = pack2(fminf(fminf(a0, b0), 20.0f), fminf(fminf(a1, b1), 20.0f));
  const float2x fi = add2(f, pack2(kMagic, kMagic));
  unpack2(add2(f, fma2(fi, pack2(-1.0f, -1.0f), pack2(kMagic, kMagic))), mid[0], mid[1]);
  unpack2(fi, a0, a1);
  bin[0] = max(__float_as_int(a0), kMagicBits);
  bin[1] = max(__float_as_int(a1), kMagicBits);
}

// prologue of pose p by one warp: quaternion inverse (one division per lane, bit-identical to
// quat_inverse), rotation matrix, ANM displacement bounds, reference point
__device__ __forceinline__ void pose_prologue(const DevComplex& C, int p, PoseBufs& Q, int lane) {
  if (lane < C.pl) Q.pose[lane] = C.pos[(size_t)p * C.pl + lane];
  __syncwarp();
  const double w0 = Q.pose[3], x = Q.pose[4], y = Q.pose[5], z = Q.pose[6];
  const double n2 = w0 * w0 + x * x + y * y + z * z;
  if (lane < 4) {
    const double qv = Q.pose[3 + lane];
    Q.q[lane] = qv;
    Q.qi[lane] = (lane == 0 ? qv : -qv) / n2;
  }
  {
    // rotation matrix of the (possibly not normalised) quaternion, one element per lane
    double rv = 0.0;
    switch (lane) {
      case 0: rv = w0 * w0 + x * x - y * y - z * z; break;
      case 1: rv = 2 * (x * y - w0 * z); break;
      case 2: rv = 2 * (x * z + w0 * y); break;
      case 3: rv = 2 * (x * y + w0 * z); break;
      case 4: rv = w0 * w0 - x * x + y * y - z * z; break;
      case 5: rv = 2 * (y * z - w0 * x); break;
      case 6: rv = 2 * (x * z - w0 * y); break;
      case 7: rv = 2 * (y * z + w0 * x); break;
      case 8: rv = w0 * w0 - x * x - y * y + z * z; break;
      default: break;
    }
    rv /= n2;
    if (lane < 9) {
      Q.rot[lane] = rv;
      Q.rotf[lane] = (float)rv;
    }
  }
  float tR = lane < C.nmr ? fabsf((float)Q.pose[7 + lane]) * C.mnorm_r[lane] : 0.f;
  float tL = lane < C.nml ? fabsf((float)Q.pose[7 + C.nmr + lane]) * C.mnorm_l[lane] : 0.f;
  for (int o = 16; o > 0; o >>= 1) {
    tR += __shfl_xor_sync(0xffffffffu, tR, o);
    tL += __shfl_xor_sync(0xffffffffu, tL, o);
  }
  __syncwarp();
  if (lane < 3)
    Q.gc[lane] = Q.rotf[3 * lane] * C.lig_ctr[0] + Q.rotf[3 * lane + 1] * C.lig_ctr[1] +
                 Q.rotf[3 * lane + 2] * C.lig_ctr[2];
  if (lane == 0) {
    const float dR = tR * 1.0001f + 1e-4f, dL = tL * 1.0001f + 1e-4f;
    Q.dR = dR;
    Q.dL = dL;
    // bound of |FP32 d2 - FP64 d2| for pairs within 15.1 A (coordinates centred on t)
    const float RL = C.lig_radius + dL;
    const float u32 = 5.9604645e-8f;
    Q.B = 2.0f * (2.02f * u32 * (26.2f * (2.0f * RL + 15.1f) + 228.0f) + 3.0f * u32 * 228.0f) + 1e-6f;
    // ligand reference point (prepare_gso_tasks.cc:460, :513, :524-526)
    double rx = C.lig_ref[0], ry = C.lig_ref[1], rz = C.lig_ref[2];
    quat_rotate(Q.q, Q.qi, rx, ry, rz);
    double* ref = C.ref + (size_t)p * 3;
    ref[0] = rx + Q.pose[0];
    ref[1] = ry + Q.pose[1];
    ref[2] = rz + Q.pose[2];
  }
}

// bounding box of each group of 8 lanes of a tile (own: the lane's atom; an empty group's half extent is
// -inf, so no point is near it)
__device__ __forceinline__ void group_boxes(const float4& own, bool active, int lane, float4* box) {
  float lo[3] = {own.x, own.y, own.z}, hi[3] = {own.x, own.y, own.z};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (!active) {
      lo[d] = 3e38f;
      hi[d] = -3e38f;
    }
#pragma unroll
    for (int o = 1; o < kGroup; o <<= 1) {
      lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
      hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
    }
  }
  if ((lane & (kGroup - 1)) == 0) {
    box[2 * (lane / kGroup)] = make_float4(0.5f * (lo[0] + hi[0]), 0.5f * (lo[1] + hi[1]), 0.5f * (lo[2] + hi[2]), 0.f);
    box[2 * (lane / kGroup) + 1] =
        make_float4(half_extent(lo[0], hi[0]), half_extent(lo[1], hi[1]), half_extent(lo[2], hi[2]), 0.f);
  }
}

// squared distance of a point (negated) from group g's box
__device__ __forceinline__ float box_distance2(const float4* box, int g, const float4& l) {
  const float4 bc = box[2 * g], bh = box[2 * g + 1];
  const float ex = fmaxf(fabsf(l.x + bc.x) - bh.x, 0.f), ey = fmaxf(fabsf(l.y + bc.y) - bh.y, 0.f),
              ez = fmaxf(fabsf(l.z + bc.z) - bh.z, 0.f);
  return fmaf(ez, ez, fmaf(ey, ey, ex * ex));
}

// half a bin less the bin coordinate's error: |d_fp32 - d| <= B / 30 inside the cutoff (B bounds d^2
// there, its leading term is 2 d |error of the difference vector|), times the slope 2, plus FP32
// roundings (square root 2^-22, coordinate up to 20).  Not above 0 (atoms 5e5 A and more from t, up to a bound
// that is infinite): no pair is settled in FP32, where a coordinate need not be finite and the far atoms that
// fill the lists up are no longer far
__device__ __forceinline__ float settled_half(float B) { return 0.5f - (B * 0.0673f + 2e-5f); }

// The near pairs of a tile that has more than kNear of them, found again (one lane per receptor atom, the tile's
// candidates in turn) and decided 32 side by side; buf: the warp's lists, which are done with by then.  600
// poses of 3002 / 1274 atoms, the ligand moved away from its origin by 500, 4,000 and 16,000 A: 0.49, 0.79 and
// 1.02 ms; 6.0, 50 and 92 ms with every pair of such tiles in FP64
__device__ __noinline__ double decide_near(const DevComplex& C, const PoseBufs& Q, const float4* lig, const float4* chS,
                                           const float4* rec, unsigned* buf, int k, const double* T,
                                           const double* table, unsigned long long* cnt) {
  const int lane = threadIdx.x & 31;
  const float4 tile = C.r_tile[k], own = rec[lane];
  const float cx = (float)((double)tile.x - Q.pose[0]), cy = (float)((double)tile.y - Q.pose[1]),
              cz = (float)((double)tile.z - Q.pose[2]);
  const float reach = 15.0f + Q.dR + SD_CULL_MARGIN + tile.w;
  const float cut2 = 225.0f + Q.B, inner = settled_half(Q.B);
  const float2x rx = pack2(own.x, own.x), ry = pack2(own.y, own.y), rz = pack2(own.z, own.z);
  double v = 0.0;
  int n = 0;
  auto decide = [&]() {
    __syncwarp();
    if (lane < n)
      v += decide_pair(C, Q.pose, Q.q, Q.qi, T, table, k * SD_TILE + (int)(buf[lane] & 31), (int)(buf[lane] >> 5), cnt);
    __syncwarp();
  };
  for (int cb = 0; cb < C.nlchunks; cb += 32) {
    bool cnear = false;
    if (cb + lane < C.nlchunks) {
      const float4 ch = chS[cb + lane];
      const float ex = ch.x - cx, ey = ch.y - cy, ez = ch.z - cz, r = reach + ch.w;
      cnear = ex * ex + ey * ey + ez * ez <= r * r;
    }
    for (unsigned cm = __ballot_sync(0xffffffffu, cnear); cm; cm &= cm - 1) {
      const int sb = (cb + __ffs(cm) - 1) * SD_TILE;
      const float4 la = lig[sb + lane];
      const float ax = la.x + cx, ay = la.y + cy, az = la.z + cz;
      const bool cand = fmaf(az, az, fmaf(ay, ay, ax * ax)) <= reach * reach;
      for (unsigned am = __ballot_sync(0xffffffffu, cand); am; am &= am - 1) {
        const int s = sb + __ffs(am) - 1;
        float d2[2], mid[2];
        int bin[2];
        pair_terms(rx, ry, rz, lig[s], d2, mid, bin);
        const bool near = d2[0] <= cut2 && fabsf(mid[0]) >= inner;
        const unsigned nm = __ballot_sync(0xffffffffu, near);
        if (near) buf[n + __popc(nm & ((1u << lane) - 1u))] = (unsigned)s * 32u + (unsigned)lane;
        n += __popc(nm);
        if (n >= 32) {
          decide();
          n -= 32;
          const unsigned rest = lane < n ? buf[32 + lane] : 0u;
          __syncwarp();
          if (lane < n) buf[lane] = rest;
        }
      }
    }
  }
  decide();
  return v;
}

}  // namespace

// Variants differ only in warps per CTA and resident CTAs per SM: a tile is always processed by
// one warp in the same way, so they give identical energies.  kSpill: the per-pose arrays (tile
// sums, transformed ligand, chunk spheres, tile lists) live in this CTA's slice of the global
// scratch L.spill, for complexes too large for shared memory; the arithmetic is the same.  kWide: for
// ligands that reach far (wide_ligand), with decide_near, which costs the pair loop registers: 8,000 poses of
// 3002 / 1274 atoms 2.89 -> 2.93 ms, 3,000 of 17307 / 1125 1.39 -> 1.41 ms
template <int kWarps, int kMinBlocks, bool kSpill, bool kWide>
__global__ void __launch_bounds__(kWarps * 32, kMinBlocks) dfire_score_mixed_kernel(ScoreLaunch L) {
  constexpr int kSortMax = 512;        // near tiles ordered largest-first up to this many
  extern __shared__ __align__(16) unsigned char smem_dyn[];
  WarpBufs* const wb = reinterpret_cast<WarpBufs*>(smem_dyn);
  unsigned char* const smem =
      kSpill ? L.spill + (size_t)blockIdx.x * L.spill_stride : smem_dyn + kWarps * sizeof(WarpBufs);
  __shared__ PoseBufs sh_p[kPoses];
  __shared__ double sh_T[32];
  __shared__ int sh_item, sh_ntile, sh_next;
  __shared__ unsigned long long sh_cnt[5];  // fallback, d2 == 0, d2 == 225, pairs, evaluations

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < 32) sh_T[tid] = c_T[tid];
  if (tid < 5) sh_cnt[tid] = 0;
  StepCtl* ctl = L.ctl;
  const int parity = ctl->parity;
  const int count = ctl->count[parity];
  const int* work = L.work[parity];
  unsigned n_done = 0;
  const unsigned lt_mask = (1u << lane) - 1u;
  WarpBufs& W = wb[warp];
  // the first n_pairs * 2 items are taken two at a time, the last ones (two rounds of the grid) one
  // at a time, so that the CTAs finish together
  const int n_pairs = L.poses_per_cta > 1 ? max(0, (count - 2 * (int)gridDim.x) / 2) : 0;

  for (;;) {
    __syncthreads();
    if (tid == 0) sh_item = atomicAdd(&ctl->grab[parity], 1);
    __syncthreads();
    int item = sh_item < n_pairs ? 2 * sh_item : sh_item + n_pairs;
    const int item_end = sh_item < n_pairs ? item + 2 : item + 1;
    if (item >= count) break;
    while (item < item_end) {
      const int ci = wi_complex(work[item]);
      const int np = item + 1 < item_end && wi_complex(work[item + 1]) == ci ? 2 : 1;  // poses of this batch
      const int first = wi_local(work[item]), second = wi_local(work[item + np - 1]);
      item += np;
      const DevComplex& C = L.cplx[ci];
      const int nslots = nslots_of(C), nlc = C.nlchunks;
      if (warp < np) {
        pose_prologue(C, warp == 0 ? first : second, sh_p[warp], lane);
        if (warp == 0 && lane == 0) {
          sh_ntile = 0;
          sh_next = 0;
        }
      }
      __syncthreads();
      const int nls = nlc * SD_TILE, ntiles = C.ntiles, tstride = (ntiles + 1) & ~1;
      double* tsum = reinterpret_cast<double*>(smem);  // [np][tstride] FP64 energy of each tile of each pose
      // [np][nls + 1] ligand atoms centred on t and negated, col bits; [nls] a far atom, the padding
      float4* ligS = reinterpret_cast<float4*>(tsum + np * tstride);
      float4* chS = ligS + np * (nls + 1);             // [np][nlc] centre + radius
      int* tlist = reinterpret_cast<int*>(chS + np * nlc);  // [ntiles] tiles within reach: tile * 4 + poses (bits)
      int* tord = tlist + ntiles;                      // [ntiles] the same, largest first
      float* tdist = reinterpret_cast<float*>(tord + ntiles);  // [ntiles]
      int* cneed = reinterpret_cast<int*>(tdist + ntiles);     // [nlc] chunk within reach of a near tile
      for (int c = tid; c < nlc; c += blockDim.x) {
        const float4 cc = C.l_chunk[c];
        for (int p = 0; p < np; ++p) {
          const float* R = sh_p[p].rotf;
          const float X = R[0] * cc.x + R[1] * cc.y + R[2] * cc.z;
          const float Y = R[3] * cc.x + R[4] * cc.y + R[5] * cc.z;
          const float Z = R[6] * cc.x + R[7] * cc.y + R[8] * cc.z;
          chS[p * nlc + c] = make_float4(X, Y, Z, cc.w + sh_p[p].dL);
        }
        cneed[c] = 0;
      }
      if (tid < np) ligS[tid * (nls + 1) + nls] = make_float4(3e18f, 3e18f, 3e18f, 0.f);
      for (int k = tid; k < np * tstride; k += blockDim.x) tsum[k] = 0.0;
      for (int k = tid; k < ntiles; k += blockDim.x) {
        const float4 tile = C.r_tile[k];
        int bits = 0;
        float dmin = 3.0e38f;
        for (int p = 0; p < np; ++p) {
          const PoseBufs& Q = sh_p[p];
          const float cx = (float)((double)tile.x - Q.pose[0]), cy = (float)((double)tile.y - Q.pose[1]),
                      cz = (float)((double)tile.z - Q.pose[2]);
          const float reach = 15.0f + Q.dR + SD_CULL_MARGIN + tile.w + (C.lig_radius + Q.dL);
          if (cx * cx + cy * cy + cz * cz <= reach * reach) {
            bits |= 1 << p;
            // distance from the ligand centroid: the closest tiles have the most pairs; a NaN
            // (non-finite quaternion) leaves 3e38, so the ranking below stays a strict total order
            const float ex = cx - Q.gc[0], ey = cy - Q.gc[1], ez = cz - Q.gc[2];
            dmin = fminf(dmin, ex * ex + ey * ey + ez * ez);
          }
        }
        if (bits) {
          const int at = atomicAdd(&sh_ntile, 1);
          tlist[at] = k * 4 + bits;
          tdist[at] = dmin;
        }
      }
      __syncthreads();
      const int ntile = sh_ntile;
      const bool sorted = ntile <= kSortMax;
      // which ligand chunks any near tile can reach (the same test as the per-tile one below, with
      // 0.01 A to spare, so a chunk that is not needed is never read)
      for (int t = warp; t < ntile; t += kWarps) {
        const int kb = tlist[t];
        const float4 tile = C.r_tile[kb >> 2];
        for (int p = 0; p < np; ++p) {
          if (!(kb >> p & 1)) continue;
          const PoseBufs& Q = sh_p[p];
          const float cx = (float)((double)tile.x - Q.pose[0]), cy = (float)((double)tile.y - Q.pose[1]),
                      cz = (float)((double)tile.z - Q.pose[2]);
          const float rt = 15.0f + Q.dR + SD_CULL_MARGIN + tile.w;
          for (int c = lane; c < nlc; c += 32) {
            const float4 ch = chS[p * nlc + c];
            const float ex = ch.x - cx, ey = ch.y - cy, ez = ch.z - cz, r = rt + ch.w + 0.01f;
            if (ex * ex + ey * ey + ez * ez <= r * r) cneed[c] = 1;
          }
        }
      }
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
      }
      __syncthreads();
      // the ligand of each pose (both from one read of its modes)
      for (int s = tid; s < nls; s += kWarps * 32) {
        if (!cneed[s >> 5]) continue;
        if (C.l_perm[s] >= 0) {
          double l[kPoses][3];
          anm_fused<kPoses>(C.l_xyz, C.l_modes, C.l_mask, nls, C.nml, &sh_p[0].pose[7 + C.nmr],
                            (int)(sizeof(PoseBufs) / sizeof(double)), s, l);
          const float col = __int_as_float(C.l_col[s]);
#pragma unroll
          for (int p = 0; p < kPoses; ++p) {
            if (p >= np) break;
            const double* R = sh_p[p].rot;
            ligS[p * (nls + 1) + s] = make_float4(-(float)fma(R[0], l[p][0], fma(R[1], l[p][1], R[2] * l[p][2])),
                                                  -(float)fma(R[3], l[p][0], fma(R[4], l[p][1], R[5] * l[p][2])),
                                                  -(float)fma(R[6], l[p][0], fma(R[7], l[p][1], R[8] * l[p][2])), col);
          }
        } else {
          for (int p = 0; p < np; ++p) ligS[p * (nls + 1) + s] = make_float4(1e18f, 1e18f, 1e18f, __int_as_float(0));
        }
      }
      __syncthreads();
      const int* tl = sorted ? tord : tlist;
      double acc = 0.0;           // per-lane FP64 sum of table values
      double pv[2] = {0.0, 0.0};  // values gathered by the previous step, added by the next
      const double* table = L.table64;
      unsigned pose_pairs = 0, pose_evals = 0;  // of this warp's tiles (pairs per lane)

      for (;;) {
        int ti = 0;
        if (lane == 0) ti = atomicAdd(&sh_next, 1);
        ti = __shfl_sync(0xffffffffu, ti, 0);
        if (ti >= ntile) break;
        const int kb = tl[ti], k = kb >> 2;
        const int slot = k * SD_TILE + lane;
        const bool active = C.r_orig[slot] >= 0;
        const unsigned act_mask = __ballot_sync(0xffffffffu, active);
        {
          // the tile's atoms in each pose, from one read of their modes
          const int row = active ? C.r_row[slot] - kMagicBits : 0;
          double r[kPoses][3];
          anm_fused<kPoses>(C.r_xyz, C.r_modes, C.r_mask, nslots, C.nmr, &sh_p[0].pose[7],
                            (int)(sizeof(PoseBufs) / sizeof(double)), slot, r);
#pragma unroll
          for (int p = 0; p < kPoses; ++p) {
            const double* t = sh_p[p].pose;
            W.rec[p][lane] = active ? make_float4((float)(r[p][0] - t[0]), (float)(r[p][1] - t[1]),
                                                  (float)(r[p][2] - t[2]), __int_as_float(row))
                                    : make_float4(1e18f, 1e18f, 1e18f, 0.f);
          }
        }
        for (int p = 0; p < np; ++p) {
          if (!(kb >> p & 1)) continue;
          const PoseBufs& Q = sh_p[p];
          const float4 tile = C.r_tile[k];
          const float cx = (float)((double)tile.x - Q.pose[0]), cy = (float)((double)tile.y - Q.pose[1]),
                      cz = (float)((double)tile.z - Q.pose[2]);
          const float reach = 15.0f + Q.dR + SD_CULL_MARGIN + tile.w;
          const float reach2 = reach * reach;
          const float cut2 = 225.0f + Q.B;
          const float box_cut = 225.1f + Q.B;
          const float inner = settled_half(Q.B);
          const float4* const lig = ligS + p * (nls + 1);
          const float4* const rec = W.rec[p];
          __syncwarp();
          group_boxes(rec[lane], active, lane, W.box);
          __syncwarp();

          unsigned nnear = 0, npairs = 0, nevals = 0;
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
                    const float4 ch = chS[p * nlc + c];
                    const float ex = ch.x - cx, ey = ch.y - cy, ez = ch.z - cz, r = reach + ch.w;
                    cnear = ex * ex + ey * ey + ez * ez <= r * r;  // same expression as the cneed test
                  }
                  cm = __ballot_sync(0xffffffffu, cnear);
                  cb += 32;
                  continue;
                }
                const int sb = (cb - 32 + __ffs(cm) - 1) * SD_TILE;
                cm &= cm - 1;
                const float4 la = lig[sb + lane];
                const float ax = la.x + cx, ay = la.y + cy, az = la.z + cz;
                const bool cand = fmaf(az, az, fmaf(ay, ay, ax * ax)) <= reach2;
                const unsigned am = __ballot_sync(0xffffffffu, cand);
                if (cand) W.pend[ncand + __popc(am & lt_mask)] = (unsigned short)(sb + lane);
                ncand += __popc(am);
              }
              __syncwarp();
              const int nb = min(ncand, 32);
              const int s = lane < nb ? W.pend[lane] : nls;
              const float4 l4 = lig[s];
#pragma unroll
              for (int g = 0; g < kGroups; ++g) {
                const bool in = box_distance2(W.box, g, l4) <= box_cut;
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
            } while (more && longest <= kList - 32 - kRow);
            // each list is padded with the far atom to whole steps
#pragma unroll
            for (int g = 0; g < kGroups; ++g) {
              if (lane < kRow) W.list[g][cnt[g] + lane] = (unsigned short)nls;
              nevals += cnt[g] * __popc((act_mask >> (g * kGroup)) & 255u);
            }
            __syncwarp();
            unsigned counts = cnt[0] | cnt[1] << 8 | cnt[2] << 16 | cnt[3] << 24;
            for (int g = 0; g < kGroups; ++g, counts >>= 8) {
              const float4 r0 = rec[g * kGroup + (lane & 3)], r1 = rec[g * kGroup + (lane & 3) + 4];
              const float2x rx = pack2(r0.x, r1.x), ry = pack2(r0.y, r1.y), rz = pack2(r0.z, r1.z);
              const double* row0 = table + __float_as_int(r0.w);
              const double* row1 = table + __float_as_int(r1.w);
              const unsigned short* list = W.list[g] + lane / 4;
              const int n = (int)(counts & 255u);
              unsigned near_steps = 0;  // steps of this list with a pair of this lane near an edge, the first highest
              for (int c = 0; c < n; c += kRow) {
                const float4 l = lig[list[c]];
                float d2[2], mid[2];
                int bin[2];
                pair_terms(rx, ry, rz, l, d2, mid, bin);
                near_steps += near_steps + (fmaxf(fabsf(mid[0]), fabsf(mid[1])) >= inner ? 1u : 0u);
                const double* at[2] = {row0 + (__float_as_int(l.w) + bin[0]), row1 + (__float_as_int(l.w) + bin[1])};
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  acc += pv[h];
                  // a pair inside the cutoff and away from a bin's edge: its value, through L2 only (each
                  // is used once, and cached in L1 it would evict the atom and mode lines that the next
                  // tiles read again)
                  asm("{\n\t.reg .pred p;\n\t.reg .f32 m;\n\t"
                      "abs.f32 m, %4;\n\t"
                      "setp.le.f32 p, %2, %3;\n\t"
                      "setp.lt.and.f32 p, m, %5, p;\n\t"
                      "mov.f64 %0, 0d0000000000000000;\n\t"
                      "@p ld.global.cg.f64 %0, [%6];\n\t"
                      "@p add.u32 %1, %1, 1;\n\t}"
                      : "=&d"(pv[h]), "+r"(npairs)
                      : "f"(d2[h]), "f"(cut2), "f"(mid[h]), "f"(inner), "l"(at[h]));
                }
              }
              near_steps = __reduce_or_sync(0xffffffffu, near_steps);
              const int last = (n - 1) / kRow;  // below 32: kList / kRow steps at most
              while (near_steps) {
                // a step with such a pair (about twelve of a pose): find the pairs again
                const int b = 31 - __clz(near_steps);
                near_steps ^= 1u << b;
                const int s = list[(last - b) * kRow];
                const float4 l = lig[s];
                float d2[2], mid[2];
                int bin[2];
                pair_terms(rx, ry, rz, l, d2, mid, bin);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  const bool near = d2[h] <= cut2 && fabsf(mid[h]) >= inner;
                  const unsigned nm = __ballot_sync(0xffffffffu, near);
                  const unsigned place = nnear + __popc(nm & lt_mask);
                  if (near && place < kNear)
                    W.near[place] = (unsigned)s * 32u + (unsigned)(g * kGroup + (lane & 3) + 4 * h);
                  nnear += __popc(nm);
                }
              }
            }
            __syncwarp();
          } while (more);
          __syncwarp();
          if (kWide && nnear > kNear && inner > 0.f) {
            acc += decide_near(C, Q, lig, chS + p * nlc, rec, (unsigned*)W.list, k, sh_T, table, sh_cnt);
          } else if (nnear <= kNear && inner > 0.f) {
            for (int i = lane; i < (int)nnear; i += 32) {
              const unsigned e = W.near[i];
              acc += decide_pair(C, Q.pose, Q.q, Q.qi, sh_T, table, k * SD_TILE + (int)(e & 31), (int)(e >> 5), sh_cnt);
            }
          } else {
            // coordinates so large that FP32 settles nothing (without kWide also too many pairs): the whole tile in FP64
            npairs = 0;
            acc = 0.0;
            pv[0] = pv[1] = 0.0;
            if (active)
              for (int s = 0; s < nls; ++s)
                if (C.l_perm[s] >= 0) acc += decide_pair(C, Q.pose, Q.q, Q.qi, sh_T, table, slot, s, sh_cnt);
          }
          __syncwarp();
          // the tile's energy: the last step's gathers, then the lane sums in a fixed shuffle order,
          // into the tile's slot
          acc += pv[0];
          acc += pv[1];
          pv[0] = pv[1] = 0.0;
          double v = acc;
          for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
          if (lane == 0) tsum[p * tstride + k] = v;
          pose_pairs += npairs;
          pose_evals += nevals;
          acc = 0.0;
        }
      }
      // counters, then the pose energy: warp 0 adds the tile slots in a fixed order
      const unsigned wp = __reduce_add_sync(0xffffffffu, pose_pairs);
      if (lane == 0) {
        if (wp) atomicAdd(&sh_cnt[3], (unsigned long long)wp);
        if (pose_evals) atomicAdd(&sh_cnt[4], (unsigned long long)pose_evals);
      }
      __syncthreads();
      if (warp < np) {
        double v = 0.0;
        for (int k = lane; k < ntiles; k += 32) v += tsum[warp * tstride + k];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) {
          const int p = warp == 0 ? first : second;
          C.scoring[p] = ((v)*0.0157 - 4.7) * -1;
          if (L.energy_out) L.energy_out[p] = v;
        }
      }
      n_done += np;
      if (item < item_end) __syncthreads();
    }
  }
  __syncthreads();
  if (tid == 0) {
    if (n_done) atomicAdd(&ctl->stats[ST_SCORED], (unsigned long long)n_done);
    if (sh_cnt[0]) atomicAdd(&ctl->stats[ST_FALLBACK], sh_cnt[0]);
    if (sh_cnt[1]) atomicAdd(&ctl->stats[ST_D2ZERO], sh_cnt[1]);
    if (sh_cnt[2]) atomicAdd(&ctl->stats[ST_D2CUT], sh_cnt[2]);
    if (sh_cnt[3]) atomicAdd(&ctl->stats[ST_PAIRS], sh_cnt[3]);
    if (sh_cnt[4]) atomicAdd(&ctl->stats[ST_EVALS], sh_cnt[4]);
  }
}

}  // namespace sd
