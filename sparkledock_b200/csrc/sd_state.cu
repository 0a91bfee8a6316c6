// Small kernels of the host runtime: a complex's starting state, the work list of the next GSO step,
// the bookkeeping of a stateless call, and the check of uploaded poses.  They replace host loops over
// the state with uploads and downloads of whole arrays (a work list used to be built from every
// complex's flags on the host, at each call that set one complex's state), and the read-back, three
// uploads and synchronisation in front of each stateless call.
#include <cuda_runtime.h>

#include "sd_internal.h"

namespace sd {

// the reference's SoA initialisation (prepare_gso_tasks.cc:386-400)
__global__ void init_state_kernel(DevComplex C, double luciferin, double vision) {
  const int n = C.S * C.G;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    C.luciferin[k] = luciferin;
    C.vision[k] = vision;
    C.scoring[k] = 0.0;
    C.step[k] = 0;
    C.moved[k] = 0;
    C.nnei[k] = 0;
    C.select[k] = k % C.G;
    for (int d = 0; d < 3; ++d) C.ref[3 * (size_t)k + d] = 0.0;
  }
}

// poses to rescore (moved, or not scored yet), one CTA per swarm, appended to work list 0
__global__ void __launch_bounds__(256) worklist_kernel(const DevComplex* cplx, const int* swarm_map, StepCtl* ctl,
                                                       int* work) {
  __shared__ int sh_count[8], sh_base;
  const int sw = swarm_map[blockIdx.x], ci = wi_complex(sw);
  const DevComplex& C = cplx[ci];
  const int G = C.G, k0 = wi_local(sw) * G, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int g0 = 0; g0 < G; g0 += 256) {
    const int k = k0 + g0 + tid;
    const bool in = g0 + tid < G && (C.moved[k] || C.step[k] == 0);
    const unsigned m = __ballot_sync(0xffffffffu, in);
    if (lane == 0) sh_count[warp] = __popc(m);
    __syncthreads();
    if (tid == 0) {
      int n = 0;
      for (int w = 0; w < 8; ++w) {
        const int c = sh_count[w];
        sh_count[w] = n;
        n += c;
      }
      sh_base = n ? atomicAdd(&ctl->count[0], n) : 0;
    }
    __syncthreads();
    if (in) work[sh_base + sh_count[warp] + __popc(m & ((1u << lane) - 1u))] = wi_pack(ci, k);
    __syncthreads();
  }
}

// a stateless call on n poses of complex ci: its descriptor, work list and counters
__global__ void stateless_prepare_kernel(StepCtl* ctl, DevComplex* cplx, DevComplex desc, int* work, int ci, int n) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  if (tid == 0) {
    ctl->count[0] = n;
    ctl->count[1] = 0;
    ctl->grab[0] = ctl->grab[1] = 0;
    ctl->parity = 0;
    cplx[ci] = desc;
  }
  for (int i = tid; i < n; i += gridDim.x * blockDim.x) work[i] = wi_pack(ci, i);
}

// *bad = 1 if one of the n values is not finite
__global__ void check_finite_kernel(const double* v, size_t n, int* bad) {
  bool b = false;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    b |= !isfinite(v[i]);
  if (b) *bad = 1;
}

static int launched() { return cudaGetLastError() == cudaSuccess ? SD_OK : SD_ERR_CUDA; }

int init_state_launch(const DevComplex& C, double luciferin, double vision, cudaStream_t st) {
  init_state_kernel<<<148 * 4, 256, 0, st>>>(C, luciferin, vision);
  return launched();
}

int worklist_launch(const DevComplex* cplx, const int* swarm_map, int nswarms, StepCtl* ctl, int* work,
                    cudaStream_t st) {
  worklist_kernel<<<nswarms, 256, 0, st>>>(cplx, swarm_map, ctl, work);
  return launched();
}

int stateless_prepare_launch(StepCtl* ctl, DevComplex* cplx, const DevComplex& desc, int* work, int ci, int n,
                             cudaStream_t st) {
  const int blocks = n < 256 * 592 ? (n + 255) / 256 : 592;
  stateless_prepare_kernel<<<blocks, 256, 0, st>>>(ctl, cplx, desc, work, ci, n);
  return launched();
}

int check_finite_launch(const double* v, size_t n, int* bad, cudaStream_t st) {
  check_finite_kernel<<<148 * 8, 256, 0, st>>>(v, n, bad);
  return launched();
}

}  // namespace sd
