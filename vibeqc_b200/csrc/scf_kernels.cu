// SCF-stage kernels over a batch of equally sized molecules.
//
// sp2_update: one step of second-order spectral projection (Niklasson,
// Phys. Rev. B 66, 155115 (2002)) for every molecule of a chunk, given
// X and X2 = X X.  It serves the purification whose X X is a sliced int8
// product (ozaki_gemm.cu); the FP64 purification, which updates the density by
// default, is one launch of its own (sp2_purify.cu).  Each CTA recomputes tr X
// and tr X^2 of its molecule, chooses X^2 or 2X - X^2 (whichever moves tr X
// toward n_occ) and writes its slice of the next iterate to a separate buffer.
// A molecule whose idempotency error |tr X - tr X^2| fell below tol is copied
// unchanged and flagged, so a fixed number of steps can run without host
// synchronisation.  Purification replaces the per-iteration batched eigensolver
// of the reference's device SCF loop (src/scf/cuda/df_scf_library.cpp,
// cusolverDnXsyevBatched).
//
// scf_change, scf_record: convergence test and bookkeeping of an iteration.
#include "vqc_df.h"
#include "vqc_kernels.cuh"
#include "vqc_plan.hpp"

namespace vqc {

__device__ __forceinline__ double block_sum(double v, double* red) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x < 32) {
    s = threadIdx.x < (blockDim.x + 31) / 32 ? red[threadIdx.x] : 0.0;
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if (threadIdx.x == 0) red[0] = s;
  }
  __syncthreads();
  return red[0];
}

__global__ void __launch_bounds__(256) sp2_update_kernel(const double* __restrict__ x,
                                                         const double* __restrict__ x2,
                                                         double* __restrict__ xout, int n,
                                                         double nocc, double tol,
                                                         int* __restrict__ done) {
  __shared__ double red[32];
  const int m = blockIdx.y;
  const size_t base = (size_t)m * n * n;
  const size_t nn = (size_t)n * n;
  double t1 = 0.0, t2 = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    t1 += x[base + (size_t)i * n + i];
    t2 += x2[base + (size_t)i * n + i];
  }
  // inputs are never written by this kernel, so every CTA of a molecule sees
  // the same traces and takes the same branch
  const double tr = block_sum(t1, red);
  const double tr2 = block_sum(t2, red);
  const bool converged = done[m] != 0 || fabs(tr - tr2) < tol;
  const bool square = fabs(tr2 - nocc) < fabs(2.0 * tr - tr2 - nocc);
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < nn;
       idx += (size_t)gridDim.x * blockDim.x) {
    const double a = x[base + idx], b = x2[base + idx];
    xout[base + idx] = converged ? a : (square ? b : 2.0 * a - b);
  }
  if (converged && blockIdx.x == 0 && threadIdx.x == 0) done[m] = 1;
}

// ---------------------------------------------------------------------------
// Convergence test and bookkeeping of one SCF iteration for every molecule of
// a chunk: the rms density change, the reference's criteria, the state of the
// molecules that are still active copied to the results, and the new density
// and factor taken over.  Two launches in place of about forty elementwise
// ones, which cost a small molecule's iteration more host time than its
// kernels take: one water molecule 14.7 -> 11.9 ms, 2428 -> 1979 launches.
// ---------------------------------------------------------------------------

constexpr int kRecSlices = 32;

struct RecordSpin {
  const double *d_new, *c_new, *f;
  double *d, *c, *d_final, *c_final, *f_final;
};

struct RecordParams {
  RecordSpin spin[2];
  int nspin, n, ncol, slices, iteration, may_converge;
  double e_tol, d_tol, c_tol, loose_tol, e_round;
  const double *energy, *cmax, *e_old_in;
  const int* active_in;
  double *e_old_out, *final_e, *final_de, *final_drms, *partial;
  int* active_out;
  long long* iters;
  int* converged;
  int* flags;  // [0] a molecule is active; [1] an active one's residual is above loose_tol
};

__global__ void __launch_bounds__(256) scf_change_kernel(RecordParams p) {
  __shared__ double red[32];
  const size_t nn = (size_t)p.n * p.n, base = (size_t)blockIdx.y * nn;
  double s = 0.0;
  for (int sp = 0; sp < p.nspin; ++sp)
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < nn; i += (size_t)gridDim.x * 256) {
      const double v = p.spin[sp].d_new[base + i] - p.spin[sp].d[base + i];
      s = fma(v, v, s);
    }
  s = block_sum(s, red);
  if (threadIdx.x == 0) p.partial[blockIdx.y * kRecSlices + blockIdx.x] = s;
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < 2) p.flags[threadIdx.x] = 0;
}

__global__ void __launch_bounds__(256) scf_record_kernel(RecordParams p) {
  const int m = blockIdx.y;
  const size_t nn = (size_t)p.n * p.n, nc = (size_t)p.n * p.ncol;
  double sum = 0.0;  // the same order in every CTA: they decide alike
  for (int g = 0; g < p.slices; ++g) sum += p.partial[m * kRecSlices + g];
  const double drms = sqrt(sum / ((double)p.nspin * (double)nn));
  const double e = p.energy[m], eo = p.e_old_in[m];
  double de = fabs(e - eo);
  if (isnan(de)) de = INFINITY;
  const double eo_abs = isnan(eo) ? 0.0 : fabs(eo);
  const double guard = p.e_round * fmax(fmax(fabs(e), eo_abs), 1.0);
  const bool was = p.active_in[m] != 0;
  const bool done = p.may_converge && de < p.e_tol + guard && drms < p.d_tol && p.cmax[m] <= p.c_tol;
  const bool stays = was && !done;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (was) {
      p.final_e[m] = e;
      p.final_de[m] = de;
      p.final_drms[m] = drms;
      p.iters[m] = p.iteration;
      if (done) p.converged[m] = 1;
      if (!(p.cmax[m] <= p.loose_tol)) atomicOr(p.flags + 1, 1);
    }
    if (stays) atomicOr(p.flags, 1);
    p.active_out[m] = stays ? 1 : 0;
    p.e_old_out[m] = e;
  }
  if (!was) return;
  const size_t start = (size_t)blockIdx.x * 256 + threadIdx.x, step = (size_t)gridDim.x * 256;
  for (int sp = 0; sp < p.nspin; ++sp) {
    const RecordSpin& s = p.spin[sp];
    for (size_t i = start; i < nn; i += step) {
      const size_t k = m * nn + i;
      s.d_final[k] = s.d[k];
      s.f_final[k] = s.f[k];
      if (stays) s.d[k] = s.d_new[k];
    }
    for (size_t i = start; i < nc; i += step) {
      const size_t k = m * nc + i;
      s.c_final[k] = s.c[k];
      if (stays) s.c[k] = s.c_new[k];
    }
  }
}

}  // namespace vqc

extern "C" int vqc_sp2_update(const double* x, const double* x2, double* xout, int32_t nmol,
                              int32_t n, double nocc, double tol, int32_t* done, void* stream) {
  using namespace vqc;
  if (!x || !x2 || !xout || !done || nmol <= 0 || n <= 0)
    return fail(VQC_STATUS_INVALID_ARGUMENT, "sp2_update: bad argument");
  const size_t nn = (size_t)n * n;
  int ctas = (int)((nn + 255 * 8 - 1) / (256 * 8));  // ~8 elements per thread
  ctas = ctas < 1 ? 1 : (ctas > 64 ? 64 : ctas);
  dim3 grid(ctas, nmol);
  sp2_update_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(x, x2, xout, n, nocc, tol, done);
  count_launch();
  return cuda_status(cudaGetLastError(), "sp2_update");
}

extern "C" int vqc_scf_record(const vqc_scf_record_args* a, void* stream) {
  using namespace vqc;
  if (!a || a->struct_size < sizeof(vqc_scf_record_args) || a->nmol <= 0 || a->nmol > 65535 || a->n <= 0 ||
      a->ncol < 0 || a->nspin < 1 || a->nspin > 2 || !a->energy || !a->cmax || !a->e_old_in ||
      !a->active_in || !a->e_old_out || !a->active_out || !a->final_e || !a->final_de ||
      !a->final_drms || !a->partial || !a->iters || !a->converged || !a->flags)
    return fail(VQC_STATUS_INVALID_ARGUMENT, "scf_record: bad argument");
  RecordParams p{};
  for (int s = 0; s < a->nspin; ++s) {
    p.spin[s] = RecordSpin{a->d_new[s], a->c_new[s], a->f[s], a->d[s], a->c[s],
                           a->d_final[s], a->c_final[s], a->f_final[s]};
    if (!a->d_new[s] || !a->f[s] || !a->d[s] || !a->d_final[s] || !a->f_final[s] ||
        (a->ncol > 0 && (!a->c_new[s] || !a->c[s] || !a->c_final[s])))
      return fail(VQC_STATUS_INVALID_ARGUMENT, "scf_record: null matrix");
  }
  p.nspin = a->nspin;
  p.n = a->n;
  p.ncol = a->ncol;
  p.iteration = a->iteration;
  p.may_converge = a->may_converge;
  p.e_tol = a->energy_tolerance;
  p.d_tol = a->density_tolerance;
  p.c_tol = a->commutator_tolerance;
  p.loose_tol = a->loose_tolerance;
  p.e_round = a->energy_roundoff;
  p.energy = a->energy;
  p.cmax = a->cmax;
  p.e_old_in = a->e_old_in;
  p.active_in = a->active_in;
  p.e_old_out = a->e_old_out;
  p.active_out = a->active_out;
  p.final_e = a->final_e;
  p.final_de = a->final_de;
  p.final_drms = a->final_drms;
  p.partial = a->partial;
  p.iters = reinterpret_cast<long long*>(a->iters);
  p.converged = a->converged;
  p.flags = a->flags;
  const size_t nn = (size_t)a->n * a->n;
  const size_t want = (nn + 2047) / 2048;  // eight elements a thread
  p.slices = (int)(want > (size_t)kRecSlices ? kRecSlices : want);
  cudaStream_t st = (cudaStream_t)stream;
  scf_change_kernel<<<dim3(p.slices, a->nmol), 256, 0, st>>>(p);
  scf_record_kernel<<<dim3(p.slices, a->nmol), 256, 0, st>>>(p);
  count_launch();
  count_launch();
  return cuda_status(cudaGetLastError(), "scf_record");
}
