// GSO update of all swarms: luciferin, neighbours, probabilistic selection, movement and
// vision range.  One CTA per swarm, FP64 with no contraction: a warp per glowworm for swarms of up to
// SD_WARP_G, a thread per glowworm above.
//
// Semantics: cal_gso_tasks_cpu passes 1-3 after scoring (prepare_gso_tasks.cc:558-559,
// :600-707, :716-814) with compute_probability_moving_from_neighbors (:1463-1488),
// select_random_neighbor (:1424-1459), slerp (:1370-1421) and move_extent (:1352-1368).
// Replaces the reference GPU kernels generate_energy_v2 / cal_move_neighbors /
// move_position_v2 (prepare_gso_task.cu:2377-2433, :791-897, :1059-1136).
//
// The update is synchronous (every glowworm selects from pre-move state): luciferin and
// reference points of the swarm are staged in shared memory, and a barrier separates the
// reads of the chosen neighbours' positions from the writes of the moved positions.  The
// neighbour list is never stored: its length, probability total and the cumulative choice
// are recomputed in two ordered scans over the swarm, which gives the same floating-point
// sums as the reference's list.  Moved glowworms are appended to the next work list; the
// last CTA to finish advances the step (parity, draw cursors, counters) so that the whole
// step can be replayed from a CUDA graph.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "sd_crmath.h"
#include "sd_internal.h"

namespace sd {

__device__ __forceinline__ void move_extent_dev(double* self, const double* other, int n_ext, double step) {
  double delta[SD_MAX_MODES];
  double n = 0;
  for (int i = 0; i < n_ext; ++i) {
    delta[i] = other[i] - self[i];
    n += delta[i] * delta[i];
  }
  n = sqrt(n);
  if (n >= 1e-8) {
    for (int i = 0; i < n_ext; ++i) {
      delta[i] *= step / n;
      self[i] += delta[i];
    }
  }
}

__device__ __forceinline__ void slerp_dev(double* self, double* other, double step) {
  double sn = 0, on = 0;
  for (int i = 0; i < 4; ++i) {
    sn += (self[i] * self[i]);
    on += (other[i] * other[i]);
  }
  sn = sqrt(sn);
  on = sqrt(on);
  for (int i = 0; i < 4; ++i) {
    self[i] /= sn;
    other[i] /= on;
  }
  double q_dot = 0;
  for (int i = 0; i < 4; ++i) q_dot += self[i] * other[i];
  if (q_dot < 0) {
    q_dot = q_dot * -1;
    for (int i = 0; i < 4; ++i) self[i] = -self[i];
  }
  if (q_dot > 0.9995) {
    for (int i = 0; i < 4; ++i) self[i] = self[i] + step * (other[i] - self[i]);
    double rn = 0;
    for (int i = 0; i < 4; ++i) rn += (self[i] * self[i]);
    rn = sqrt(rn);
    for (int i = 0; i < 4; ++i) self[i] /= rn;
  } else {
    q_dot = (q_dot < 1) ? q_dot : 1;
    q_dot = (q_dot > -1) ? q_dot : -1;
    const double omega = sd_acos_cr(q_dot);
    const double so = sd_sin_cr(omega);
    const double tmp0 = (sd_sin_cr((1.0 - step) * omega) / so);
    const double tmp1 = (sd_sin_cr(step * omega) / so);
    for (int i = 0; i < 4; ++i) self[i] = tmp0 * self[i] + tmp1 * other[i];
  }
}

// Neighbours of glowworm g (luciferin shL[G] and reference points shR[G][3] of its swarm in shared
// memory; vision range vr) in ascending n (prepare_gso_tasks.cc:615-640), their probability total
// (:1476-1484) and the first whose cumulative probability reaches the draw *u (:1441-1450).
// Returns the choice (g itself without neighbours) and the count in nn; counts the draws <= 0 with
// neighbours (the reference reads neighbors[-1]; the first is taken) and the cumulative shortfalls
// (the last is taken).
__device__ __forceinline__ int choose_neighbour(const double* shL, const double* shR, int G, int g, double Lg,
                                                double vr, const double* u_ptr, int& nn,
                                                unsigned long long* uzero, unsigned long long* shortfall) {
  const double cx = shR[g * 3], cy = shR[g * 3 + 1], cz = shR[g * 3 + 2];
  const double sq = vr * vr;
  double total = 0;
  nn = 0;
  for (int n = 0; n < G; ++n) {
    const double Ln = shL[n];
    if (n != g && Lg < Ln) {
      const double dx = cx - shR[n * 3], dy = cy - shR[n * 3 + 1], dz = cz - shR[n * 3 + 2];
      double distance = 0;
      distance += dx * dx;
      distance += dy * dy;
      distance += dz * dz;
      if (distance < sq) {
        ++nn;
        total += Ln - Lg;
      }
    }
  }
  if (nn == 0) return g;
  const double u = *u_ptr;
  double sum = 0.0;
  int picked = -1, last = -1;
  if (!(sum < u)) atomicAdd(uzero, 1ull);
  for (int n = 0; n < G && picked < 0; ++n) {
    const double Ln = shL[n];
    if (n != g && Lg < Ln) {
      const double dx = cx - shR[n * 3], dy = cy - shR[n * 3 + 1], dz = cz - shR[n * 3 + 2];
      double distance = 0;
      distance += dx * dx;
      distance += dy * dy;
      distance += dz * dz;
      if (distance < sq) {
        last = n;
        if (!(sum < u)) {
          picked = n;  // only reached when u <= 0
        } else {
          sum += (Ln - Lg) / total;
          if (!(sum < u)) picked = n;
        }
      }
    }
  }
  if (picked < 0) {
    picked = last;
    atomicAdd(shortfall, 1ull);
  }
  return picked;
}

// Movement of one glowworm towards the chosen neighbour's pose mv (prepare_gso_tasks.cc:772-794):
// translation by step_t along the direction, slerp of the quaternion, receptor and ligand extents.
__device__ __forceinline__ void move_towards(double* cur, double* mv, int nmr, int nml, const GsoParamsDev& P) {
  double delta[3], n = 0;
  for (int d = 0; d < 3; ++d) {
    delta[d] = mv[d] - cur[d];
    n += (delta[d] * delta[d]);
  }
  n = sqrt(n);
  if (n >= 1e-8) {
    for (int d = 0; d < 3; ++d) {
      delta[d] *= (P.step_t / n);
      cur[d] += delta[d];
    }
  }
  slerp_dev(cur + 3, mv + 3, P.step_r);
  move_extent_dev(cur + 7, mv + 7, nmr, P.step_nm);
  move_extent_dev(cur + 7 + nmr, mv + 7 + nmr, nml, P.step_nm);
}

// the last CTA of a step: work list of the next step, counters, and the draws one column further for
// every complex
__device__ __forceinline__ void advance_step(const GsoLaunch& L, int parity, int tid) {
  __threadfence();
  if (tid == 0) {
    StepCtl* ctl = L.ctl;
    ctl->count[parity] = 0;
    ctl->grab[parity] = 0;
    ctl->grab[parity ^ 1] = 0;
    ctl->parity = parity ^ 1;
    ctl->done_blocks = 0;
    ctl->step += 1;
    ctl->stats[ST_STEPS] += 1;
    __threadfence();
  }
  if (tid < L.ncplx) L.cplx[tid].draw_cursor += 1;
}

// ---- a warp per selection, four lanes per movement ----
// The thread-per-glowworm update below is one long chain per thread: two scans over the swarm and five
// double-double series.  Here a warp finds a glowworm's neighbours by ballots and only walks through
// them (the sums keep their order); then four lanes move a glowworm, the three displacements side by
// side and the series of a slerp in two turns (cosine and sine, then three sines).  Measured per launch
// against the kernel below: 4 swarms x 50 glowworms 69 -> 22 us, 402 x 200 130 -> 124 us, 1,245 x 200
// 329 -> 323 us, 40 x 512 179 -> 138 us.

// move_extent of n components from place i0 of a pose, and the moved components into out
__device__ __forceinline__ void move_part(const double* own, const double* other, double* out, int i0, int n,
                                          double step) {
  double len = 0;
  for (int i = 0; i < n; ++i) {
    const double delta = other[i0 + i] - own[i0 + i];
    len += delta * delta;
  }
  len = sqrt(len);
  const bool far = len >= 1e-8;
  const double f = far ? step / len : 0.0;
  for (int i = 0; i < n; ++i) {
    const double o = own[i0 + i];
    double delta = other[i0 + i] - o;
    delta *= f;
    out[i0 + i] = far ? o + delta : o;
  }
}

// slerp_dev by the four lanes of a row (`part` 0 .. 3, all with the same quaternions); every lane of the
// warp calls it, and those without a glowworm (live false) get no meaningful result
__device__ __forceinline__ void slerp_row(double (&q)[4], double (&o)[4], int part, double step) {
  double sn = 0, on = 0;
  for (int i = 0; i < 4; ++i) {
    sn += (q[i] * q[i]);
    on += (o[i] * o[i]);
  }
  sn = sqrt(sn);
  on = sqrt(on);
  for (int i = 0; i < 4; ++i) {
    q[i] /= sn;
    o[i] /= on;
  }
  double dot = 0;
  for (int i = 0; i < 4; ++i) dot += q[i] * o[i];
  if (dot < 0) {
    dot = dot * -1;
    for (int i = 0; i < 4; ++i) q[i] = -q[i];
  }
  const bool linear = dot > 0.9995;
  if (!__all_sync(0xffffffffu, linear)) {
    double x = (dot < 1) ? dot : 1;
    x = (x > -1) ? x : -1;
    // acos as sd_acos_cr for an argument in [0, 1]: the cosine series in even lanes, the sine in odd ones
    double omega = acos(x);
    const sdcr::dd y = {omega, 0.0};
    const sdcr::Terms& t = sdcr::terms();
    sdcr::dd r = sdcr::series(y, (part & 1) ? t.sin_t : t.cos_t);
    if (part & 1) r = sdcr::dd_mul(y, r);
    const double c_hi = __shfl_sync(0xffffffffu, r.hi, 0, 4), c_lo = __shfl_sync(0xffffffffu, r.lo, 0, 4);
    const double s_hi = __shfl_sync(0xffffffffu, r.hi, 1, 4);
    if (x < 1.0 && !(omega < 1e-8)) {
      const sdcr::dd y1 = sdcr::two_sum(omega, ((c_hi - x) + c_lo) / s_hi);
      omega = y1.hi + y1.lo;
    }
    const double v = sd_sin_cr(part == 0 ? omega : (part == 1 ? (1.0 - step) * omega : step * omega));
    const double so = __shfl_sync(0xffffffffu, v, 0, 4);
    const double tmp0 = (__shfl_sync(0xffffffffu, v, 1, 4) / so), tmp1 = (__shfl_sync(0xffffffffu, v, 2, 4) / so);
    if (!linear)
      for (int i = 0; i < 4; ++i) q[i] = tmp0 * q[i] + tmp1 * o[i];
  }
  if (linear) {
    for (int i = 0; i < 4; ++i) q[i] = q[i] + step * (o[i] - q[i]);
    double rn = 0;
    for (int i = 0; i < 4; ++i) rn += (q[i] * q[i]);
    rn = sqrt(rn);
    for (int i = 0; i < 4; ++i) q[i] /= rn;
  }
}

__global__ void __launch_bounds__(1024) gso_warp_kernel(GsoLaunch L) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int sh_base, sh_last;
  __shared__ unsigned long long sh_uzero, sh_short;
  __shared__ int sh_wcount[SD_WARP_G / 32], sh_woff[SD_WARP_G / 32];
  const int sw_packed = L.swarm_map[blockIdx.x];
  const int ci = wi_complex(sw_packed), s = wi_local(sw_packed);
  DevComplex& C = L.cplx[ci];
  const int G = C.G, pl = C.pl, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  double* shL = reinterpret_cast<double*>(smem);  // [G] luciferin
  double* shR = shL + G;                          // [G][3] reference points
  double* shP = shR + 3 * G;                      // [G][pl] poses after the move
  int* shS = reinterpret_cast<int*>(shP + (size_t)G * pl);  // [G] selection
  StepCtl* ctl = L.ctl;
  const int parity = ctl->parity;
  const GsoParamsDev P = L.p;
  const size_t k0 = (size_t)s * G;
  if (tid == 0) {
    sh_uzero = 0;
    sh_short = 0;
  }
  // luciferin (prepare_gso_tasks.cc:558)
  for (int g = tid; g < G; g += blockDim.x) {
    const size_t k = k0 + g;
    const double Lg = (1.0 - P.rho) * C.luciferin[k] + P.gamma * C.scoring[k];
    C.luciferin[k] = Lg;
    C.step[k] += 1;
    shL[g] = Lg;
  }
  for (int i = tid; i < 3 * G; i += blockDim.x) shR[i] = C.ref[k0 * 3 + i];
  __syncthreads();
  const double* draws = C.draws + (size_t)s * C.draw_steps * G + (size_t)C.draw_cursor * G;
  for (int g = warp; g < G; g += nwarps) {
    const size_t k = k0 + g;
    const double Lg = shL[g], vr = C.vision[k], u = draws[g];
    const double cx = shR[g * 3], cy = shR[g * 3 + 1], cz = shR[g * 3 + 2], sq = vr * vr;
    // neighbours in ascending n (prepare_gso_tasks.cc:615-640); their probability total (:1476-1484)
    double total = 0;
    int nn = 0;
    unsigned mask = 0;  // lane w: neighbours among glowworms 32 w .. 32 w + 31
    for (int base = 0; base < G; base += 32) {
      const int n = base + lane;
      bool nb = false;
      double gain = 0;
      if (n < G && n != g) {
        const double Ln = shL[n];
        if (Lg < Ln) {
          const double dx = cx - shR[n * 3], dy = cy - shR[n * 3 + 1], dz = cz - shR[n * 3 + 2];
          double distance = 0;
          distance += dx * dx;
          distance += dy * dy;
          distance += dz * dz;
          nb = distance < sq;
          gain = Ln - Lg;
        }
      }
      const unsigned m = __ballot_sync(0xffffffffu, nb);
      if (lane == (base >> 5)) mask = m;
      nn += __popc(m);
      for (unsigned r = m; r; r &= r - 1) total += __shfl_sync(0xffffffffu, gain, __ffs(r) - 1);
    }
    // the first whose cumulative probability reaches the draw (:1441-1450); u <= 0: the first; a
    // shortfall: the last
    int sel = g;
    if (nn > 0) {
      double sum = 0.0;
      int picked = -1, last = -1;
      if (!(sum < u)) {
        if (lane == 0) atomicAdd(&sh_uzero, 1ull);
      }
      for (int base = 0; base < G && picked < 0; base += 32) {
        const unsigned m = __shfl_sync(0xffffffffu, mask, base >> 5);
        const double share = (m >> lane) & 1u ? (shL[base + lane] - Lg) / total : 0.0;
        for (unsigned r = m; r && picked < 0; r &= r - 1) {
          const int b = __ffs(r) - 1;
          last = base + b;
          if (!(sum < u)) {
            picked = last;  // only reached when u <= 0
          } else {
            sum += __shfl_sync(0xffffffffu, share, b);
            if (!(sum < u)) picked = last;
          }
        }
      }
      if (picked < 0) {
        picked = last;
        if (lane == 0) atomicAdd(&sh_short, 1ull);
      }
      sel = picked;
    }
    if (lane == 0) {
      shS[g] = sel;
      C.moved[k] = sel != g ? 1 : 0;
      C.nnei[k] = nn;
      C.select[k] = sel;
      // vision range (:806-808)
      double v = vr + P.beta * (P.max_neighbors - nn);
      if (v < 0.0) v = 0;
      if (v > P.max_vision) v = P.max_vision;
      C.vision[k] = v;
    }
  }
  __syncthreads();
  // movement (:772-794) from the pre-move poses in global memory, which nothing writes before the barrier
  for (int g0 = warp * 8; g0 < G; g0 += nwarps * 8) {
    const int g = g0 + (lane >> 2), part = lane & 3;
    const bool moved = g < G && shS[g] != g;
    if (!__any_sync(0xffffffffu, moved)) continue;
    const double* own = C.pos + (k0 + (moved ? g : 0)) * pl;
    const double* other = C.pos + (k0 + (moved ? shS[g] : 0)) * pl;
    double* out = shP + (size_t)(moved ? g : 0) * pl;
    double q[4], o[4];
    for (int i = 0; i < 4; ++i) {
      q[i] = own[3 + i];
      o[i] = other[3 + i];
    }
    if (moved && part < 3)
      move_part(own, other, out, part == 0 ? 0 : (part == 1 ? 7 : 7 + C.nmr), part == 0 ? 3 : (part == 1 ? C.nmr : C.nml),
                part == 0 ? P.step_t : P.step_nm);
    __syncwarp();
    slerp_row(q, o, part, P.step_r);
    if (moved && part == 3)
      for (int i = 0; i < 4; ++i) out[3 + i] = q[i];
  }
  __syncthreads();  // all reads of pre-move positions are done
  for (int g = warp; g < G; g += nwarps)
    if (shS[g] != g && lane < pl) C.pos[(k0 + g) * pl + lane] = shP[(size_t)g * pl + lane];
  // next work list: moved glowworms, in glowworm order within the swarm
  for (int g0 = warp * 32; g0 < G; g0 += blockDim.x) {
    const bool moved = g0 + lane < G && shS[g0 + lane] != g0 + lane;
    const unsigned bal = __ballot_sync(0xffffffffu, moved);
    if (lane == 0) sh_wcount[g0 >> 5] = __popc(bal);
  }
  __syncthreads();
  if (tid == 0) {
    int acc = 0;
    for (int w = 0; w < (G + 31) / 32; ++w) {
      sh_woff[w] = acc;
      acc += sh_wcount[w];
    }
    sh_base = acc ? atomicAdd(&ctl->count[parity ^ 1], acc) : 0;
  }
  __syncthreads();
  for (int g0 = warp * 32; g0 < G; g0 += blockDim.x) {
    const bool moved = g0 + lane < G && shS[g0 + lane] != g0 + lane;
    const unsigned bal = __ballot_sync(0xffffffffu, moved);
    if (moved)
      L.work[parity ^ 1][sh_base + sh_woff[g0 >> 5] + __popc(bal & ((1u << lane) - 1u))] = wi_pack(ci, (int)k0 + g0 + lane);
  }
  // last block advances the step
  __syncthreads();
  if (tid == 0) {
    if (sh_uzero) atomicAdd(&ctl->stats[ST_UZERO], sh_uzero);
    if (sh_short) atomicAdd(&ctl->stats[ST_SHORT], sh_short);
    __threadfence();
    const int done = atomicAdd(&ctl->done_blocks, 1);
    sh_last = done == L.nswarms_total - 1;
  }
  __syncthreads();
  if (sh_last) advance_step(L, parity, tid);
}

__global__ void __launch_bounds__(SD_MAX_G) gso_kernel(GsoLaunch L) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int sh_base, sh_last;
  __shared__ unsigned long long sh_uzero, sh_short;
  const int sw_packed = L.swarm_map[blockIdx.x];
  const int ci = wi_complex(sw_packed), s = wi_local(sw_packed);
  DevComplex& C = L.cplx[ci];
  const int G = C.G, pl = C.pl, g = threadIdx.x;
  const bool live = g < G;
  double* shL = reinterpret_cast<double*>(smem);  // [G]
  double* shR = shL + G;                          // [G][3]
  StepCtl* ctl = L.ctl;
  const int parity = ctl->parity;
  const GsoParamsDev P = L.p;
  if (g == 0) {
    sh_uzero = 0;
    sh_short = 0;
  }
  const size_t k = (size_t)s * G + g;
  // luciferin (prepare_gso_tasks.cc:558)
  double Lg = 0.0;
  if (live) {
    Lg = (1.0 - P.rho) * C.luciferin[k] + P.gamma * C.scoring[k];
    C.luciferin[k] = Lg;
    C.step[k] += 1;
    shL[g] = Lg;
    shR[g * 3] = C.ref[k * 3];
    shR[g * 3 + 1] = C.ref[k * 3 + 1];
    shR[g * 3 + 2] = C.ref[k * 3 + 2];
  }
  __syncthreads();
  int sel = g, nn = 0;
  if (live)
    sel = choose_neighbour(shL, shR, G, g, Lg, C.vision[k],
                           C.draws + (size_t)s * C.draw_steps * G + (size_t)C.draw_cursor * G + g, nn, &sh_uzero,
                           &sh_short);
  // copy of the chosen neighbour's pre-move position (:689-693)
  double mv[7 + 2 * SD_MAX_MODES], cur[7 + 2 * SD_MAX_MODES];
  if (live) {
    const double* src = C.pos + ((size_t)s * G + sel) * pl;
    const double* own = C.pos + k * pl;
    for (int i = 0; i < pl; ++i) {
      mv[i] = src[i];
      cur[i] = own[i];
    }
  }
  __syncthreads();  // all reads of pre-move positions are done
  bool moved = false;
  if (live) {
    moved = sel != g;
    C.moved[k] = moved ? 1 : 0;
    C.nnei[k] = nn;
    C.select[k] = sel;
    if (moved) {
      move_towards(cur, mv, C.nmr, C.nml, P);
      double* own = C.pos + k * pl;
      for (int i = 0; i < pl; ++i) own[i] = cur[i];
    }
    // vision range (:806-808)
    double vr = C.vision[k] + P.beta * (P.max_neighbors - nn);
    if (vr < 0.0) vr = 0;
    if (vr > P.max_vision) vr = P.max_vision;
    C.vision[k] = vr;
  }
  // next work list: moved glowworms, in glowworm order within the swarm
  const unsigned bal = __ballot_sync(0xffffffffu, moved);
  __shared__ int sh_wcount[SD_MAX_G / 32], sh_woff[SD_MAX_G / 32];
  const int lane = g & 31, wid = g >> 5, nw = blockDim.x >> 5;
  if (lane == 0) sh_wcount[wid] = __popc(bal);
  __syncthreads();
  if (g == 0) {
    int acc = 0;
    for (int w = 0; w < nw; ++w) {
      sh_woff[w] = acc;
      acc += sh_wcount[w];
    }
    sh_base = acc ? atomicAdd(&ctl->count[parity ^ 1], acc) : 0;
  }
  __syncthreads();
  if (moved) {
    const int pos_in = sh_base + sh_woff[wid] + __popc(bal & ((1u << lane) - 1u));
    L.work[parity ^ 1][pos_in] = wi_pack(ci, (int)k);
  }
  // last block advances the step
  __syncthreads();
  if (g == 0) {
    if (sh_uzero) atomicAdd(&ctl->stats[ST_UZERO], sh_uzero);
    if (sh_short) atomicAdd(&ctl->stats[ST_SHORT], sh_short);
    __threadfence();
    const int done = atomicAdd(&ctl->done_blocks, 1);
    sh_last = done == L.nswarms_total - 1;
  }
  __syncthreads();
  if (sh_last) advance_step(L, parity, g);
}

// Swarms of more than SD_MAX_G glowworms (more than one CTA's threads): the same update with each
// thread taking glowworms tid, tid + blockDim.x, ...  A thread can no longer hold the chosen
// neighbours' pre-move poses of all its glowworms across a barrier, so every pose is first copied to
// L.pos_prev (one row of SD_POSE_LEN(10, 10) doubles per glowworm of the context) and the moves read
// the copies.  Moved glowworms are appended to the next work list one CTA-wide chunk at a time.
__global__ void __launch_bounds__(SD_MAX_G) gso_kernel_large(GsoLaunch L) {
  constexpr int kRow = SD_POSE_LEN(SD_MAX_MODES, SD_MAX_MODES);
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int sh_base, sh_last;
  __shared__ unsigned long long sh_uzero, sh_short;
  __shared__ int sh_wcount[SD_MAX_G / 32], sh_woff[SD_MAX_G / 32];
  const int sw_packed = L.swarm_map[blockIdx.x];
  const int ci = wi_complex(sw_packed), s = wi_local(sw_packed);
  DevComplex& C = L.cplx[ci];
  const int G = C.G, pl = C.pl, tid = threadIdx.x, B = blockDim.x;
  double* shL = reinterpret_cast<double*>(smem);  // [G]
  double* shR = shL + G;                          // [G][3]
  StepCtl* ctl = L.ctl;
  const int parity = ctl->parity;
  const GsoParamsDev P = L.p;
  double* prev = L.pos_prev + ((size_t)C.gbase + (size_t)s * G) * kRow;
  if (tid == 0) {
    sh_uzero = 0;
    sh_short = 0;
  }
  // luciferin (prepare_gso_tasks.cc:558), staging, pre-move copies
  for (int g = tid; g < G; g += B) {
    const size_t k = (size_t)s * G + g;
    const double Lg = (1.0 - P.rho) * C.luciferin[k] + P.gamma * C.scoring[k];
    C.luciferin[k] = Lg;
    C.step[k] += 1;
    shL[g] = Lg;
    shR[g * 3] = C.ref[k * 3];
    shR[g * 3 + 1] = C.ref[k * 3 + 1];
    shR[g * 3 + 2] = C.ref[k * 3 + 2];
    for (int i = 0; i < pl; ++i) prev[(size_t)g * kRow + i] = C.pos[k * pl + i];
  }
  __syncthreads();
  unsigned moved_bits = 0;  // bit c: glowworm c * B + tid moved
  for (int g = tid, c = 0; g < G; g += B, ++c) {
    const size_t k = (size_t)s * G + g;
    int nn = 0;
    const int sel = choose_neighbour(shL, shR, G, g, shL[g], C.vision[k],
                                     C.draws + (size_t)s * C.draw_steps * G + (size_t)C.draw_cursor * G + g, nn,
                                     &sh_uzero, &sh_short);
    const bool moved = sel != g;
    C.moved[k] = moved ? 1 : 0;
    C.nnei[k] = nn;
    C.select[k] = sel;
    if (moved) {
      double mv[kRow], cur[kRow];
      for (int i = 0; i < pl; ++i) {
        mv[i] = prev[(size_t)sel * kRow + i];
        cur[i] = prev[(size_t)g * kRow + i];
      }
      move_towards(cur, mv, C.nmr, C.nml, P);
      for (int i = 0; i < pl; ++i) C.pos[k * pl + i] = cur[i];
      moved_bits |= 1u << c;
    }
    // vision range (:806-808)
    double vr = C.vision[k] + P.beta * (P.max_neighbors - nn);
    if (vr < 0.0) vr = 0;
    if (vr > P.max_vision) vr = P.max_vision;
    C.vision[k] = vr;
  }
  // next work list, chunk by chunk, in glowworm order within a chunk
  const int lane = tid & 31, wid = tid >> 5, nw = B >> 5;
  for (int c = 0; c * B < G; ++c) {
    const bool moved = (moved_bits >> c) & 1u;
    const unsigned bal = __ballot_sync(0xffffffffu, moved);
    if (lane == 0) sh_wcount[wid] = __popc(bal);
    __syncthreads();
    if (tid == 0) {
      int acc = 0;
      for (int w = 0; w < nw; ++w) {
        sh_woff[w] = acc;
        acc += sh_wcount[w];
      }
      sh_base = acc ? atomicAdd(&ctl->count[parity ^ 1], acc) : 0;
    }
    __syncthreads();
    if (moved) {
      const int pos_in = sh_base + sh_woff[wid] + __popc(bal & ((1u << lane) - 1u));
      L.work[parity ^ 1][pos_in] = wi_pack(ci, s * G + c * B + tid);
    }
    __syncthreads();
  }
  // last block advances the step
  if (tid == 0) {
    if (sh_uzero) atomicAdd(&ctl->stats[ST_UZERO], sh_uzero);
    if (sh_short) atomicAdd(&ctl->stats[ST_SHORT], sh_short);
    __threadfence();
    const int done = atomicAdd(&ctl->done_blocks, 1);
    sh_last = done == L.nswarms_total - 1;
  }
  __syncthreads();
  if (sh_last) advance_step(L, parity, tid);
}

// shared memory of gso_warp_kernel: luciferin, reference points, moved poses and selections of one swarm
static size_t gso_warp_smem(int max_g) { return (size_t)max_g * (8 * (4 + SD_POSE_LEN(SD_MAX_MODES, SD_MAX_MODES)) + 4); }

// once per context that has such swarms, before any capture
int gso_prepare_warp() {
  return cudaFuncSetAttribute((const void*)gso_warp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)gso_warp_smem(SD_WARP_G)) == cudaSuccess
             ? SD_OK
             : SD_ERR_CUDA;
}

// max_g up to SD_WARP_G.  32 warps a CTA while every swarm has an SM, 16 beyond.  A step with 8, 16 and 32 warps
// (the scorer of 20/20 atoms included): 20 swarms x 200 glowworms 208, 163, 146 us; 148 x 200 671, 622, 605;
// 200 x 200 863, 821, 830; 402 x 200 1602, 1601, 1602; but 300 x 512 3722, 3242, 3050
int gso_launch_warp(const GsoLaunch& L, int max_g, int nsm, cudaStream_t st) {
  const int threads = 32 * std::min(max_g, L.nswarms_total <= nsm ? 32 : 16);
  gso_warp_kernel<<<L.nswarms_total, threads, gso_warp_smem(max_g), st>>>(L);
  return cudaGetLastError() == cudaSuccess ? SD_OK : SD_ERR_CUDA;
}

int gso_launch(const GsoLaunch& L, int threads, cudaStream_t st) {
  // shared: luciferin + reference points of the swarm's glowworms
  const size_t smem = (size_t)SD_MAX_G * 4 * sizeof(double);
  gso_kernel<<<L.nswarms_total, threads, smem, st>>>(L);
  return cudaGetLastError() == cudaSuccess ? SD_OK : SD_ERR_CUDA;
}

// once per context that has such swarms, before any capture: the large kernel's shared memory
int gso_prepare_large() {
  return cudaFuncSetAttribute((const void*)gso_kernel_large, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)((size_t)SD_MAX_GLOWWORMS * 4 * sizeof(double))) == cudaSuccess
             ? SD_OK
             : SD_ERR_CUDA;
}

int gso_launch_large(const GsoLaunch& L, int max_g, cudaStream_t st) {
  // shared: luciferin + reference points of the swarm's glowworms
  const size_t smem = (size_t)max_g * 4 * sizeof(double);
  gso_kernel_large<<<L.nswarms_total, SD_MAX_G, smem, st>>>(L);
  return cudaGetLastError() == cudaSuccess ? SD_OK : SD_ERR_CUDA;
}

// the slerp's correctly rounded functions evaluated on the device (parity checking): fn 0 acos,
// fn 1 sin
__global__ void crmath_eval_kernel(int fn, const double* x, long long n, double* out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = fn == 0 ? sd_acos_cr(x[i]) : sd_sin_cr(x[i]);
}

}  // namespace sd

extern "C" int sd_crmath_eval(int device, int fn, const double* x, long long n, double* out) {
  if ((fn != 0 && fn != 1) || n < 0 || (n > 0 && (!x || !out))) return sd::fail(SD_ERR_ARG, "sd_crmath_eval: bad arguments");
  if (n == 0) return SD_OK;
  if (cudaSetDevice(device) != cudaSuccess) return sd::fail(SD_ERR_CUDA, "sd_crmath_eval: bad device");
  double* d = nullptr;
  if (cudaMalloc(&d, (size_t)n * 2 * sizeof(double)) != cudaSuccess) {
    cudaGetLastError();
    return sd::fail(SD_ERR_OOM, "sd_crmath_eval: cudaMalloc failed");
  }
  cudaError_t e = cudaMemcpy(d, x, (size_t)n * sizeof(double), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    sd::crmath_eval_kernel<<<148 * 8, 256>>>(fn, d, n, d + n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d + n, (size_t)n * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? SD_OK : sd::fail(SD_ERR_CUDA, std::string("sd_crmath_eval: ") + cudaGetErrorString(e));
}
