// Internal declarations shared by the host runtime and the kernels.
#pragma once
#include <cstddef>
#include <cstdint>
#include <string>
#include <vector>

#include <nvtx3/nvToolsExt.h>

#include "../../include/sparkle_b200.h"

#if defined(__CUDACC__)
#include <cuda_runtime.h>
#endif

#define SD_TABLE_SIZE (SD_DFIRE_TYPES * SD_DFIRE_TYPES * SD_DFIRE_BINS)
#define SD_ROW (SD_DFIRE_TYPES * SD_DFIRE_BINS)  /* 3360 */
#define SD_CUTOFF2 225.0
#define SD_MAX_COMPLEX 32
#define SD_TILE 32              /* receptor atoms per tile (one warp lane each) */
#define SD_GROUP 8              /* consecutive atoms of a tile that are compact by themselves */
#define SD_MAX_LIG 65504        /* ligand atoms: the mixed scorer's 16-bit ligand slot indices */
#define SD_MAX_REC (1 << 22)    /* receptor atoms */
#define SD_MAX_G 1024           /* glowworms per swarm with one thread each (one CTA per swarm) */
#define SD_WARP_G 512           /* glowworms per swarm with one warp each: their moved poses in shared memory */
#define SD_MAX_GLOWWORMS 6144   /* glowworms per swarm: luciferin + reference points in shared memory */
#define SD_CULL_MARGIN 0.05f    /* A, covers FP32 rounding of the conservative culling tests */
#define SD_MAX_VARIANTS 16      /* compiled variants of the mixed DFIRE kernel (autotuner) */
#define SD_FEW SD_MAX_VARIANTS  /* the kernels' variant for at most one pose per SM (not tuned) */
#define SD_WIDE 32              /* added to a variant of the mixed DFIRE kernel: its form for far-reaching ligands */
#define SD_NOALLOC_MAX_POSES 65536           /* poses per sd_score_poses_noalloc call */
#define SD_NOALLOC_SCRATCH_BYTES (288 * 1024) /* its file-scope device scratch array */

namespace sd {

// a named NVTX range over a scope: the entry points show up by name on a profiler's timeline
// (no cost when no profiler is attached)
struct NvtxRange {
  explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(const NvtxRange&) = delete;
  NvtxRange& operator=(const NvtxRange&) = delete;
};

// thread-local error message; returns code
int fail(int code, const std::string& msg);
void mvee_center(const double* p, int n, double tol, double* center);

// accessors of sd_structure (sd_structure.cc)
int structure_atoms(const sd_structure* s, std::vector<double>& xyz, std::vector<std::string>& names,
                    std::vector<int>& residue_first);
const std::vector<double>& structure_raw_xyz(const sd_structure* s);
const std::vector<std::string>& structure_residue_names(const sd_structure* s);
const std::vector<int>& structure_residue_first(const sd_structure* s);
const double* structure_translation(const sd_structure* s);

}  // namespace sd

#if defined(__CUDACC__)
namespace sd {

// ---- device-side view of one complex (lives in device memory, read by every kernel) ----
struct DevComplex {
  int nr, nl, nmr, nml, S, G, pl;
  int ntiles;           // receptor tiles of SD_TILE slots
  int gbase, sbase;     // first global glowworm / swarm index of this complex
  // receptor in tile order (slot = tile*32 + lane); padded slots far away, with r_orig = -1
  const int* r_orig;
  const int* r_slot;       // [nr] original receptor index -> slot
  const double* r_xyz;     // [3][nslots]
  const double* r_modes;   // [nmr][3][nslots]
  const int* r_mask;       // [nslots]
  const int* r_row;        // [nslots] DFIRE row base tR*3360
  const float4* r_tile;    // [ntiles] centre (rest frame) + radius
  const float* r_q;        // [nslots] charge (pyDock)
  const int* r_lj;         // [nslots] LJ type (pyDock)
  // ligand in spatial chunks of 32 (slot = chunk*32 + lane; padded slots far away, with l_perm = -1)
  int nlchunks;
  const int* l_perm;       // [nlchunks*32] slot -> original ligand index, or -1
  const int* l_slot;       // [nl] original ligand index -> slot
  const float4* l_chunk;   // [nlchunks] centre (ligand frame) + radius
  const double* l_xyz;     // [3][nlchunks*32]
  const double* l_modes;   // [nml][3][nlchunks*32]
  const int* l_mask;
  const int* l_col;        // [nlchunks*32] tL*20
  const float* l_q;        // [nlchunks*32] charge, LJ type (pyDock)
  const int* l_lj;
  float lig_ctr[3];        // ligand centroid (ligand frame)
  float mnorm_r[SD_MAX_MODES], mnorm_l[SD_MAX_MODES];  // max per-atom mode norm (rounded up)
  float lig_radius;        // max |l0_j| (rounded up)
  double lig_ref[3];
  // GSO state [S][G]
  double* pos;
  double* scoring;
  double* luciferin;
  double* vision;
  int* step;
  int* moved;
  int* nnei;
  int* select;
  double* ref;             // [S][G][3]
  const double* draws;     // [S][draw_steps][G]
  int draw_steps;
  int draw_cursor;         // advanced by the GSO kernel (device copy authoritative)
};

struct StepCtl {
  int count[2];            // items in work list [parity]
  int grab[2];             // next item to grab in list [parity]
  int parity;
  int done_blocks;         // GSO blocks finished in this step
  int step;
  int pad;
  unsigned long long stats[12];  // mirrors sd_stats order
};

enum { ST_SCORED = 0, ST_STEPS, ST_FALLBACK, ST_D2ZERO, ST_D2CUT, ST_UZERO, ST_SHORT, ST_TIMEOUT, ST_PAIRS, ST_EVALS };

struct GsoParamsDev {
  double rho, gamma, beta, max_vision, step_t, step_r, step_nm;
  int max_neighbors;
};

// work item: complex index in the top 8 bits, local glowworm index below
__host__ __device__ inline int wi_pack(int c, int local) { return (c << 24) | local; }
__host__ __device__ inline int wi_complex(int w) { return (int)((unsigned)w >> 24); }
__host__ __device__ inline int wi_local(int w) { return w & 0xFFFFFF; }

struct ScoreLaunch {
  const DevComplex* cplx;
  StepCtl* ctl;
  const int* work[2];
  const double* table64;   // [SD_TABLE_SIZE + 32] zero padded
  const double* lj_eps;    // [20] pyDock
  const double* lj_sigma;
  float force_scale;       // pyDock gradients in FP32: units of the ligand forces' fixed point
  int poses_per_cta;       // mixed DFIRE: 2 when two poses' arrays fit, else 1
  double* energy_out;      // nullable [local glowworm] raw energies (stateless scoring)
  // per-CTA global scratch that replaces the dynamic shared memory of the spill instantiations
  // (complexes whose per-pose arrays do not fit in shared memory); null otherwise
  unsigned char* spill;
  size_t spill_stride;     // bytes per CTA
};

struct GsoLaunch {
  DevComplex* cplx;
  StepCtl* ctl;
  int* work[2];
  const int* swarm_map;    // [total swarms] packed (complex, local swarm)
  int nswarms_total;
  int ncplx;               // <= 32 (the last CTA's first warp advances their draw cursors)
  GsoParamsDev p;
  double* pos_prev;        // swarms over SD_MAX_G glowworms: pre-move pose copies [glowworms][27]
};

// kernel launchers (sd_score.cu, sd_gso.cu)
// spill: the instantiation that keeps its per-pose arrays in L.spill instead of shared memory
int score_launch(const ScoreLaunch& L, int precision, int scoring, int grid, size_t smem, cudaStream_t st, int variant,
                 bool spill);
size_t score_smem_bytes(int precision, int scoring, int max_nr, int max_nl, int poses);
size_t score_warp_bytes(int precision, int scoring, int variant, bool spill);
int score_threads_of(int precision, int scoring, int variant, bool spill);
int fp64_shape(int max_nr, int max_nl, int smem_sm, int poses, int nsm);
const void* score_kernel_ptr(int precision, int scoring, int variant, bool spill);
int mixed_variant_count();
bool wide_ligand(float radius);
int mixed_variant_warps(int v);
int mixed_variant_min_blocks(int v);
int gso_launch(const GsoLaunch& L, int threads, cudaStream_t st);
int gso_launch_large(const GsoLaunch& L, int max_g, cudaStream_t st);
int gso_launch_warp(const GsoLaunch& L, int max_g, int nsm, cudaStream_t st);
int gso_prepare_large();
int gso_prepare_warp();
int bins_launch(const DevComplex& C, int precision, int* d_bins, int* d_fallback, cudaStream_t st);
size_t pydock_smem_bytes(int precision, bool grad, int max_nl, int max_nr);
// shapes of the pyDock kernel (sd_pydock.cu); PD_SCRATCH: the ordinary one with its arrays in global scratch
enum PdShape { PD_ORDINARY = 0, PD_FEW, PD_MID, PD_SMALL, PD_SCRATCH };
size_t pydock_warp_bytes(int precision, bool grad, int shape);
int pydock_grad_shape(int precision, int nl, int nr, int poses, int smem_sm, int nsm);
float pydock_force_scale(double max_q_rec, double max_q_lig, const double* eps, const double* sigma,
                         unsigned rec_types, unsigned lig_types, int max_nr);
const void* pydock_kernel_ptr(int precision, bool grad, bool spill, int shape);
int pydock_launch(const ScoreLaunch& L, int precision, bool grad, double* out_grad, int grid, size_t smem,
                  cudaStream_t st, bool spill, int shape);
int pydock_threads(int precision, bool grad, int shape);
int init_state_launch(const DevComplex& C, double luciferin, double vision, cudaStream_t st);
int worklist_launch(const DevComplex* cplx, const int* swarm_map, int nswarms, StepCtl* ctl, int* work,
                    cudaStream_t st);
int stateless_prepare_launch(StepCtl* ctl, DevComplex* cplx, const DevComplex& desc, int* work, int ci, int n,
                             cudaStream_t st);
int check_finite_launch(const double* v, size_t n, int* bad, cudaStream_t st);
void set_key_thresholds(const double* t64);
size_t cluster_smem_bytes(int G);
int materialise_launch(const DevComplex* d_cplx, int ci, const int* d_poses, int n, int nr, int nl, double* d_rec,
                       double* d_lig, cudaStream_t st);
int cluster_launch(const DevComplex* d_cplx, int ci, int s0, int ns, int G, const int* d_rb, int nbr,
                   const int* d_lb_idx, int nbl, double* d_bb, int* d_ncl, int* d_rep, int* d_len, int* d_member,
                   cudaStream_t st);

}  // namespace sd
#endif  // __CUDACC__
