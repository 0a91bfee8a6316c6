// Culled FP64 DFIRE scoring (SD_PREC_FP64; included by sd_score.cu after sd_score_mixed.cuh, whose
// pair_terms, groups and FP64 pair decision it shares).
//
// The energy of cdfire_calculate_dfire (prepare_gso_tasks.cc:1522-1615) bit for bit: every bin is the
// FP64 reference bin, each receptor atom's partial v_i adds the FP64 table values of its pairs in
// ascending ligand index j, and the pose energy adds the v_i in ascending receptor index i (pairs
// outside the cutoff and atoms without pairs add +0.0, which never changes a sum).  Only where the
// value of a pair comes from is different: a bin proven by the FP32 distance and its error bound needs
// no FP64 distance; the pairs near an edge (about ten of a pose) are decided from the exact transforms.
//  * one CTA per pose; the ligand stays in original order, so candidates are listed in ascending j;
//  * a warp takes a receptor tile, lists the candidates of each of its four groups of 8 atoms by the
//    groups' bounding boxes (as the mixed scorer), and goes through the four lists together, 8
//    candidates of each at a time: 8 atoms x 8 candidates per step, two atoms per lane; the values are
//    written to the warp's shared matrix, and then every lane adds its own atom's values in order.
//
// What bounds it: as the mixed scorer, the gathers and the issue slots (L1 data path 78 % busy, 0.6 of
// the issue slots on 3002 / 1274 atoms), and besides the sum over the v_i at the end of a pose, a chain
// of dependent FP64 additions that one warp does (the zeros are taken out first: 17307 / 1125 atoms ran
// 1.8 times as fast with that).  Measured, M poses/s, against the earlier kernel (FP64 distance of every
// pair of a tile and its candidates, one lane per receptor atom): 757/481 1.80 -> 5.62, 2516/1061 0.93
// -> 1.97, 3002/1274 0.84 -> 1.73, 6032/1766 0.34 -> 0.85, 17307/1125 0.43 -> 1.08.
#pragma once

namespace sd {
namespace {

constexpr int kOrdList = 128;                   // candidates of a group between two drains
constexpr int kOrdGroup = kGroup * kRow + 8;    // doubles of a group's values (padded: no bank conflicts)

struct __align__(16) OrdBufs {
  double val[kGroups * kOrdGroup];   // [group][candidate][atom & 3][atom >> 2] values of a round
  float4 rec[SD_TILE];               // receptor atom of each lane centred on t, row bits
  float4 box[2 * kGroups];
  unsigned short list[kGroups][kOrdList + kRow];  // each group's candidates: ligand indices, ascending
  unsigned short pend[64];           // pending candidates of the tile
};

}  // namespace

template <int kWarps, int kMinBlocks, bool kSpill>
__global__ void __launch_bounds__(kWarps * 32, kMinBlocks) dfire_score_fp64_kernel(ScoreLaunch L) {
  constexpr int kSortMax = 512;
  extern __shared__ __align__(16) unsigned char smem_dyn[];
  OrdBufs* const wb = reinterpret_cast<OrdBufs*>(smem_dyn);
  unsigned char* const smem =
      kSpill ? L.spill + (size_t)blockIdx.x * L.spill_stride : smem_dyn + kWarps * sizeof(OrdBufs);
  __shared__ PoseBufs Q;
  __shared__ double sh_T[32];
  __shared__ int sh_item, sh_ntile, sh_next, sh_moved[2][kWarps];
  __shared__ unsigned long long sh_cnt[5];  // decided in FP64, d2 == 0, d2 == 225, pairs, evaluations

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < 32) sh_T[tid] = c_T[tid];
  if (tid < 5) sh_cnt[tid] = 0;
  StepCtl* ctl = L.ctl;
  const int parity = ctl->parity;
  const int count = ctl->count[parity];
  const int* work = L.work[parity];
  unsigned n_done = 0;
  const unsigned lt_mask = (1u << lane) - 1u;
  OrdBufs& W = wb[warp];
  const double* table = L.table64;

  for (;;) {
    __syncthreads();
    if (tid == 0) sh_item = atomicAdd(&ctl->grab[parity], 1);
    __syncthreads();
    const int item = sh_item;
    if (item >= count) break;
    const int p = wi_local(work[item]);
    const DevComplex& C = L.cplx[wi_complex(work[item])];
    const int nslots = nslots_of(C), nls = C.nlchunks * SD_TILE, nr = C.nr, ntiles = C.ntiles;
    double* vacc = reinterpret_cast<double*>(smem);  // [nr] v_i, original order
    float4* lig = reinterpret_cast<float4*>(vacc + ((nr + 1) & ~1));  // [nls + 1] original order, negated, col bits
    int* tlist = reinterpret_cast<int*>(lig + nls + 1);      // [ntiles] tiles within reach
    int* tord = tlist + ntiles;                              // [ntiles] the same, closest first
    float* tdist = reinterpret_cast<float*>(tord + ntiles);  // [ntiles]
    if (warp == 0) {
      pose_prologue(C, p, Q, lane);
      if (lane == 0) {
        sh_ntile = 0;
        sh_next = 0;
      }
    }
    for (int i = tid; i < nr; i += blockDim.x) vacc[i] = 0.0;
    __syncthreads();
    for (int k = tid; k < ntiles; k += blockDim.x) {
      const float4 tile = C.r_tile[k];
      const float cx = (float)((double)tile.x - Q.pose[0]), cy = (float)((double)tile.y - Q.pose[1]),
                  cz = (float)((double)tile.z - Q.pose[2]);
      const float reach = 15.0f + Q.dR + SD_CULL_MARGIN + tile.w + (C.lig_radius + Q.dL);
      if (cx * cx + cy * cy + cz * cz <= reach * reach) {
        const int at = atomicAdd(&sh_ntile, 1);
        const float ex = cx - Q.gc[0], ey = cy - Q.gc[1], ez = cz - Q.gc[2];
        tlist[at] = k;
        tdist[at] = fminf(3.0e38f, ex * ex + ey * ey + ez * ez);  // a NaN ranks last
      }
    }
    for (int s = tid; s <= nls; s += blockDim.x) {
      const int j = s < nls ? C.l_perm[s] : -1;
      if (j >= 0) {
        double l[1][3];
        anm_fused<1>(C.l_xyz, C.l_modes, C.l_mask, nls, C.nml, &Q.pose[7 + C.nmr], 0, s, l);
        const double* R = Q.rot;
        lig[j] = make_float4(-(float)fma(R[0], l[0][0], fma(R[1], l[0][1], R[2] * l[0][2])),
                             -(float)fma(R[3], l[0][0], fma(R[4], l[0][1], R[5] * l[0][2])),
                             -(float)fma(R[6], l[0][0], fma(R[7], l[0][1], R[8] * l[0][2])),
                             __int_as_float(C.l_col[s]));
      }
      if (s >= C.nl) lig[s] = make_float4(3e18f, 3e18f, 3e18f, 0.f);  // the padding
    }
    __syncthreads();
    const int ntile = sh_ntile;
    const bool sorted = ntile <= kSortMax;
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
    const double tx = Q.pose[0], ty = Q.pose[1], tz = Q.pose[2];
    const float cut2 = 225.0f + Q.B, box_cut = 225.1f + Q.B, inner = settled_half(Q.B);
    const bool settled = inner > 0.f;  // else every listed pair is decided in FP64
    unsigned pose_pairs = 0, pose_evals = 0;

    for (;;) {
      int ti = 0;
      if (lane == 0) ti = atomicAdd(&sh_next, 1);
      ti = __shfl_sync(0xffffffffu, ti, 0);
      if (ti >= ntile) break;
      const int k = tl[ti], slot = k * SD_TILE + lane;
      const float4 tile = C.r_tile[k];
      const float cx = (float)((double)tile.x - tx), cy = (float)((double)tile.y - ty),
                  cz = (float)((double)tile.z - tz);
      const float reach = 15.0f + Q.dR + SD_CULL_MARGIN + tile.w, reach2 = reach * reach;
      const int orig = C.r_orig[slot];
      const bool active = orig >= 0;
      const unsigned act_mask = __ballot_sync(0xffffffffu, active);
      float4 own = make_float4(1e18f, 1e18f, 1e18f, 0.f);
      if (active) {
        double r[1][3];
        anm_fused<1>(C.r_xyz, C.r_modes, C.r_mask, nslots, C.nmr, &Q.pose[7], 0, slot, r);
        own = make_float4((float)(r[0][0] - tx), (float)(r[0][1] - ty), (float)(r[0][2] - tz),
                          __int_as_float(C.r_row[slot] - kMagicBits));
      }
      __syncwarp();
      W.rec[lane] = own;
      group_boxes(own, active, lane, W.box);
      __syncwarp();
      double v = 0.0;  // FP64 partial of receptor atom `orig`
      int ncand = 0, cb = 0;
      bool more = true;
      do {
        // fill each group's list, in ascending j, until the ligand is exhausted or a list may overflow
        unsigned cnt[kGroups];
#pragma unroll
        for (int g = 0; g < kGroups; ++g) cnt[g] = 0;
        unsigned longest = 0;
        do {
          while (ncand < 32 && cb < nls) {
            const float4 la = lig[cb + lane];
            const float ax = la.x + cx, ay = la.y + cy, az = la.z + cz;
            const bool cand = fmaf(az, az, fmaf(ay, ay, ax * ax)) <= reach2;
            const unsigned am = __ballot_sync(0xffffffffu, cand);
            if (cand) W.pend[ncand + __popc(am & lt_mask)] = (unsigned short)(cb + lane);
            ncand += __popc(am);
            cb += 32;
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
          more = ncand > 0 || cb < nls;
        } while (more && longest <= kOrdList - 32);
        // each list is padded with the far atom to whole steps
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
          if (lane < kRow) W.list[g][cnt[g] + lane] = (unsigned short)nls;
          pose_evals += lane == 0 ? cnt[g] * __popc((act_mask >> (g * kGroup)) & 255u) : 0;
        }
        __syncwarp();
        const unsigned counts = cnt[0] | cnt[1] << 8 | cnt[2] << 16 | cnt[3] << 24;
        for (int c = 0; c < (int)longest; c += kRow) {
          // 8 candidates of every group that has as many: their values into the matrix
          double pv[2] = {0.0, 0.0};
          int pg = -1;  // group of the values in flight
          for (int g = 0; g < kGroups; ++g) {
            if (c >= (int)((counts >> (8 * g)) & 255u)) continue;
            const float4 r0 = W.rec[g * kGroup + (lane & 3)], r1 = W.rec[g * kGroup + (lane & 3) + 4];
            const int j = W.list[g][c + lane / 4];
            const float4 l = lig[j];
            float d2[2], mid[2];
            int bin[2];
            pair_terms(pack2(r0.x, r1.x), pack2(r0.y, r1.y), pack2(r0.z, r1.z), l, d2, mid, bin);
            double val[2];
            const bool ok0 = d2[0] <= cut2, ok1 = d2[1] <= cut2;
            const bool near0 = (ok0 && fabsf(mid[0]) >= inner) || !settled,
                       near1 = (ok1 && fabsf(mid[1]) >= inner) || !settled;
            const int i0 = __float_as_int(r0.w) + __float_as_int(l.w) + bin[0],
                      i1 = __float_as_int(r1.w) + __float_as_int(l.w) + bin[1];
            val[0] = ok0 && !near0 ? __ldcg(table + i0) : 0.0;
            val[1] = ok1 && !near1 ? __ldcg(table + i1) : 0.0;
            pose_pairs += (ok0 && !near0) + (ok1 && !near1);
            if (__any_sync(0xffffffffu, near0 || near1)) {
              // (not the padding of the lists: unsettled, it is listed and near)
              if (near0 && j < C.nl)
                val[0] = decide_pair(C, Q.pose, Q.q, Q.qi, sh_T, table, k * SD_TILE + g * kGroup + (lane & 3),
                                     C.l_slot[j], sh_cnt);
              if (near1 && j < C.nl)
                val[1] = decide_pair(C, Q.pose, Q.q, Q.qi, sh_T, table, k * SD_TILE + g * kGroup + (lane & 3) + 4,
                                     C.l_slot[j], sh_cnt);
            }
            if (pg >= 0) *reinterpret_cast<double2*>(&W.val[pg * kOrdGroup + 2 * lane]) = make_double2(pv[0], pv[1]);
            pv[0] = val[0];
            pv[1] = val[1];
            pg = g;
          }
          *reinterpret_cast<double2*>(&W.val[pg * kOrdGroup + 2 * lane]) = make_double2(pv[0], pv[1]);
          __syncwarp();
          // this lane's atom: its values in order
          if (c < (int)((counts >> (8 * (lane / kGroup))) & 255u)) {
            const double* m = &W.val[(lane / kGroup) * kOrdGroup + 2 * (lane & 3) + ((lane >> 2) & 1)];
#pragma unroll
            for (int q = 0; q < kRow; ++q) v += m[8 * q];
          }
          __syncwarp();
        }
      } while (more);
      if (active) vacc[orig] = v;
    }
    const unsigned wp = __reduce_add_sync(0xffffffffu, pose_pairs);
    if (lane == 0) {
      if (wp) atomicAdd(&sh_cnt[3], (unsigned long long)wp);
      if (pose_evals) atomicAdd(&sh_cnt[4], (unsigned long long)pose_evals);
    }
    __syncthreads();
    // reference order: E += v_i for i ascending.  The non-zero v_i (adding +0.0 changes nothing) are first
    // moved together in place, one block of 32 per warp and round: a round writes only where this or an
    // earlier round has read
    int nv = 0;
    for (int base = 0, round = 0; base < nr; base += kWarps * 32, ++round) {
      const int i = base + warp * 32 + lane;
      const double x = i < nr ? vacc[i] : 0.0;
      const unsigned m = __ballot_sync(0xffffffffu, x != 0.0);
      if (lane == 0) sh_moved[round & 1][warp] = __popc(m);
      __syncthreads();
      int before = 0, total = 0;
      for (int w = 0; w < kWarps; ++w) {
        const int n = sh_moved[round & 1][w];
        before += w < warp ? n : 0;
        total += n;
      }
      if (x != 0.0) vacc[nv + before + __popc(m & lt_mask)] = x;
      nv += total;
    }
    __syncthreads();
    if (warp == 0) {
      double E = 0.0;
      int i = 0;
      for (; i + 16 <= nv; i += 16) {
        double x[16];
#pragma unroll
        for (int b = 0; b < 16; ++b) x[b] = vacc[i + b];
#pragma unroll
        for (int b = 0; b < 16; ++b) E += x[b];
      }
      for (; i < nv; ++i) E += vacc[i];
      if (lane == 0) {
        C.scoring[p] = ((E)*0.0157 - 4.7) * -1;
        if (L.energy_out) L.energy_out[p] = E;
      }
    }
    ++n_done;
  }
  __syncthreads();
  if (tid == 0) {
    if (sh_cnt[1]) atomicAdd(&ctl->stats[ST_D2ZERO], sh_cnt[1]);
    if (sh_cnt[2]) atomicAdd(&ctl->stats[ST_D2CUT], sh_cnt[2]);
    if (sh_cnt[3]) atomicAdd(&ctl->stats[ST_PAIRS], sh_cnt[3]);
    if (sh_cnt[4]) atomicAdd(&ctl->stats[ST_EVALS], sh_cnt[4]);
    if (n_done) atomicAdd(&ctl->stats[ST_SCORED], (unsigned long long)n_done);
  }
}

}  // namespace sd
