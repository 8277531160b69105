// k_noalloc.cu -- the diagonal GW self-energy without any device allocation.
//
// Who needs this: Fortran/C hosts that own all device memory themselves -- a code that carves
// every buffer out of one preallocated pool, runs under a hard device-memory budget, or drives
// a hot loop (e.g. the evGW cycle) in which the library must not allocate behind its back.
// Such callers cannot let the library call cudaMalloc, so they cannot use the context-based
// entry points (whose workspace is allocated on first use).  This entry point takes only
// caller-owned device buffers and a stream and allocates nothing.
//
// Its only scratch (the per-chunk partial sums of the pole sweep) is the file-scope array
// below: QK_NOALLOC_SCRATCH_DOUBLES doubles (3 MiB), resident on every GPU that loads the
// library until the process exits.  Limits that follow from it: nBas <= 1024 orbitals, and
// at most 128 excitation chunks (chosen internally).
//
// Set-up: every call looks up the array's device address with cudaGetSymbolAddress on the
// device that is current at the call (a host-side lookup that allocates nothing), so the address
// stays right after cudaDeviceReset or a context change.  All calls share the one array and it
// keeps the last call's contents, so calls whose kernels overlap on the GPU (different streams
// or host threads on one device) race with each other; serialise them.
#include "qk_internal.cuh"
#include "qk_poles.cuh"

#define QK_NOALLOC_MAX_N 1024
#define QK_NOALLOC_MAX_CHUNKS 128
#define QK_NOALLOC_SCRATCH_DOUBLES (3 * QK_NOALLOC_MAX_CHUNKS * QK_NOALLOC_MAX_N)

static __device__ __align__(256) double qk_noalloc_scratch[QK_NOALLOC_SCRATCH_DOUBLES];

namespace {

// the pole sums of RGW_self_energy_diag.f90:44-84, a CTA per (tile of 8 orbitals, m chunk)
__global__ void __launch_bounds__(qk_poles::WARPS * 32, 2)
    k_sigma_partial_noalloc(int N, int nC, int nO, int nR, int nS, int nchunks, int mper, double eta,
                            const double* __restrict__ e, const double* __restrict__ Om,
                            const double* __restrict__ rho, double* __restrict__ part) {
  using namespace qk_poles;
  __shared__ Tile T;
  const int pend = N - nR;
  const int base = nC + blockIdx.x * PT;
  const int np = min(PT, pend - base);
  if (threadIdx.x < np) {
    T.p[threadIdx.x] = base + threadIdx.x;
    T.w[threadIdx.x] = e[base + threadIdx.x];
  }
  __syncthreads();
  Range g;
  g.N = N;
  g.nO = nO;
  g.q0 = nC;
  g.q1 = pend;
  g.m0 = blockIdx.y * mper;
  g.m1 = min(nS, g.m0 + mper);
  tile_sums<KIND_ETA>(T, np, g, e, Om, rho, eta, 0.0, part + (size_t)blockIdx.y * N,
                      (size_t)nchunks * N);
}

__global__ void k_sigma_final_noalloc(int N, int nC, int nO, int nR, int nchunks,
                                      const double* __restrict__ part, double* __restrict__ Sig,
                                      double* __restrict__ Z, double* __restrict__ EcGM) {
  __shared__ double red[32];
  const double gm = qk_poles::final_sums(N, nC, nO, nR, nchunks, part, Sig, Z);
  const double tot = qk_block_sum(gm, red);
  if (threadIdx.x == 0) *EcGM = -2.0 * tot;
}

// device address of the scratch array on the current device (the host-side symbol is only a
// stand-in); resolved on every call, since a reset or a new context may move the module
int scratch_for_current_device(double** out) {
  void* ptr = nullptr;
  if (cudaGetSymbolAddress(&ptr, qk_noalloc_scratch) != cudaSuccess || !ptr) return QK_ERR_CUDA;
  *out = (double*)ptr;
  return QK_OK;
}

}  // namespace

extern "C" int qk_RGW_self_energy_diag_noalloc_dev(double eta, int nBas, int nOrb, int nC, int nO,
                                                   int nV, int nR, int nS, const double* d_e,
                                                   const double* d_Om, const double* d_rho,
                                                   double* d_EcGM, double* d_Sig, double* d_Z,
                                                   void* stream) {
  const int N = nBas;
  const int no = nO - nC, nv = N - nO - nR;
  if (N <= 0 || nC < 0 || nR < 0 || no <= 0 || nv <= 0 || (long long)no * nv != nS)
    return QK_ERR_ARG;
  // QuAcK's counts: nV = nBas - nO (frozen virtuals included), nO <= nOrb <= nBas
  if (nV != N - nO || nOrb < nO || nOrb > N) return QK_ERR_ARG;
  if (N > QK_NOALLOC_MAX_N) return QK_ERR_ARG;  // beyond the static scratch (nBas <= 1024)
  if (!d_e || !d_Om || !d_rho || !d_EcGM || !d_Sig || !d_Z) return QK_ERR_ARG;
  double* part = nullptr;
  int st = scratch_for_current_device(&part);
  if (st != QK_OK) return st;
  // one 32-lane group of m a chunk, more above 128 chunks (the scratch array's size); every
  // partial sum that the reduction reads is written by the sweep
  const int nact = N - nR - nC;
  const int ptiles = (nact + qk_poles::PT - 1) / qk_poles::PT;
  const int groups = (nS + 31) / 32;
  const int mper = 32 * ((groups + QK_NOALLOC_MAX_CHUNKS - 1) / QK_NOALLOC_MAX_CHUNKS);
  const int nchunks = (nS + mper - 1) / mper;
  cudaStream_t s = (cudaStream_t)stream;
  // launch statuses are taken from the launches themselves, so an earlier error left by the
  // caller's own work is neither reported as this call's nor cleared
  {
    int a0 = N, a1 = nC, a2 = nO, a3 = nR, a4 = nS, a5 = nchunks, a6 = mper;
    double a7 = eta;
    const double *p8 = d_e, *p9 = d_Om, *p10 = d_rho;
    double* p11 = part;
    void* args[] = {&a0, &a1, &a2, &a3, &a4, &a5, &a6, &a7, &p8, &p9, &p10, &p11};
    if (cudaLaunchKernel((const void*)k_sigma_partial_noalloc, dim3(ptiles, nchunks),
                         dim3(qk_poles::WARPS * 32), args, 0, s) != cudaSuccess)
      return QK_ERR_CUDA;
  }
  {
    int a0 = N, a1 = nC, a2 = nO, a3 = nR, a4 = nchunks;
    const double* p5 = part;
    double *p6 = d_Sig, *p7 = d_Z, *p8 = d_EcGM;
    void* args[] = {&a0, &a1, &a2, &a3, &a4, &p5, &p6, &p7, &p8};
    if (cudaLaunchKernel((const void*)k_sigma_final_noalloc, dim3(1), dim3(1024), args, 0, s) !=
        cudaSuccess)
      return QK_ERR_CUDA;
  }
  if (cudaStreamSynchronize(s) != cudaSuccess) return QK_ERR_CUDA;
  return QK_OK;
}
