// Launch-side definitions shared by the kernel translation units and the
// plan/C-ABI layer.
#pragma once

#include "vqc_internal.cuh"

namespace vqc {

// per (angular-momentum class, molecule) work entry
struct ClassMol {
  int mol;
  int pair_begin;   // first pair of this molecule in the class pair list
  int aux_begin;    // first aux shell with the class aux l in this molecule
  int naux;         // number of such aux shells
  int ntriples;     // work items (pairs x aux shells, or pairs)
  int chunk_begin;  // first CTA of this entry
};

struct ClassLaunch {
  int la, lb, lc;
  int nab;    // 3-centre: largest primitive count of the class's orbital pairs
  int lanes;  // 1-electron values: lanes per shell pair
  const int2* pairs;
  const ClassMol* cms;
  int ncm;
  int nblocks;
};

struct KernelArgs {
  DevBasis orb, aux;
  const double* xyz;
  const double* charge;
  const DevMol* mols;
  double* out;
  double* out2;
  double* out3;
  const double* w1;  // derivative weights (Abar / Mbar / densities)
  const double* w2;
  double* grad;
};

__host__ __device__ constexpr int round32(int n) { return (n + 31) / 32 * 32; }
__host__ __device__ constexpr int out_count(int l, bool sph) { return sph ? 2 * l + 1 : (l + 1) * (l + 2) / 2; }

// triples per CTA of the 3-centre value kernel: <= 256 threads and a shared
// staging block of at most 40 KB
__host__ __device__ constexpr int slots3c(int la, int lb, int lc, bool sph) {
  return (256 / ncart(lc)) < (5120 / (ncart(lc) * out_count(la, sph) * out_count(lb, sph)))
             ? (256 / ncart(lc))
             : (5120 / (ncart(lc) * out_count(la, sph) * out_count(lb, sph)));
}

// Resident CTAs per SM requested from the compiler for the 3-centre kernels:
// the low-l classes (the most frequent and the most contracted) are latency-
// bound on FP64 dependencies at one or two CTAs, so they are compiled to fit
// more (fewer registers, a few hundred bytes of spills); the high-l classes
// keep their registers.  Measured on 48 clusters: values 127 -> 79 ms,
// derivatives 171 -> 128 ms per step.  The two lowest sums take more still:
// (ss|s) values 0.129 -> 0.125, (ps|s) 0.184 -> 0.165 ms for 8 x (H2O)9.
__host__ __device__ constexpr int min_ctas3c(int la, int lb, int lc) {
  return la + lb + lc <= 1 ? 4 : (la + lb + lc <= 3 ? 3 : (la + lb + lc <= 5 ? 2 : 1));
}
__host__ __device__ constexpr int min_ctas_grad3c(int la, int lb, int lc) {
  return la + lb + lc <= 0 ? 4 : (la + lb + lc <= 1 ? 3 : (la + lb + lc <= 5 ? 2 : 1));
}
// Resident CTAs per SM requested for the root-parallel 3-centre kernels:
// enough for about 512 threads per SM (at most 128 registers a thread), and
// for 1024 and 768 in the lowest classes, whose state fits 64 and 80 registers
// with little spilled ((ps|p) values 0.506 -> 0.344 ms for 8 x (H2O)9, (ss|p)
// derivatives 0.382 -> 0.346 ms for 12 x (H2O)6).
__host__ __device__ constexpr int min_ctas_rp(int threads, int ltot) {
  const int want = ltot <= 1 ? 1024 : (ltot <= 2 ? 768 : 512);
  return threads >= want ? 1 : (want / threads > 8 ? 8 : want / threads);
}

template <int LA, int LB, int LC, bool SPH>
struct Int3cCfg {
  static constexpr int NOA = out_count(LA, SPH), NOB = out_count(LB, SPH), NOC = out_count(LC, SPH);
  static constexpr int SLOTS = slots3c(LA, LB, LC, SPH);
  static constexpr int THREADS = SLOTS * ncart(LC);
};

__host__ __device__ constexpr int slots2c(int lc) { return 256 / ncart(lc); }

template <int LA, int LC, bool SPH>
struct Int2cCfg {
  static constexpr int NOA = out_count(LA, SPH), NOC = out_count(LC, SPH);
  static constexpr int SLOTS = slots2c(LC);
  static constexpr int THREADS = SLOTS * ncart(LC);
};

// ---------------------------------------------------------------------------
// Primitive pairs of a 3-centre CTA.  A CTA's triples run over the aux shells
// of a few orbital shell pairs, so every thread of a pair needs the same
// Gaussian products: the CTA forms each once, in shared memory, instead of an
// exponential, a division and a dozen products per thread and primitive pair
// (most of which kPrimPairCut then drops).  Entries are listed pair by pair
// with a fixed stride (the largest primitive count of the class's pairs) and
// worked through in windows of kPairTab, so any contraction fits.  The kernels
// stay bound by latency (FP64 pipe 12-40 % active): 8 x (H2O)9 values 5.86 ->
// 4.67 ms with this table, the paired Rys coefficients and more resident warps
// for the lowest classes together, 12 x (H2O)6 derivatives 5.72 -> 5.18 ms.
// ---------------------------------------------------------------------------

constexpr int kPairTab = 256;  // entries per window: 16 KB, ten 5 x 5 pairs
struct PrimPair {
  double p, hip;      // exponent sum a + b, 0.5 / (a + b)
  double k;           // 2 pi^(5/2) K_ab c_a c_b / (a + b); 0: below kPrimPairCut
  double x, y, z;     // Gaussian-product centre
  double a2, b2;      // 2 a, 2 b
};
using PairTable = PrimPair[kPairTab];

// Runs body(e0, e1) over the entries [e0, e1) of this thread's pair (index
// ``mine`` with nab primitive pairs among the CTA's npairs pairs, which start
// at pairs[0]; nab = 0: none), window by window.  Every thread of the CTA must
// call it; shared memory is synchronised before the first body and after the
// last one.
template <class Body>
__device__ __forceinline__ void for_prim_pairs(PairTable& tab, const DevBasis& orb,
                                               const double* __restrict__ xyz,
                                               const int2* __restrict__ pairs, int npairs, int stride,
                                               int mine, int nab, Body&& body) {
  const int total = npairs * stride;
  for (int w0 = 0; w0 < total; w0 += kPairTab) {
    const int w1 = min(total, w0 + kPairTab);
    for (int e = w0 + threadIdx.x; e < w1; e += blockDim.x) {
      const int q = e / stride, i = e - q * stride;
      const int2 pr = pairs[q];
      const int nb = orb.nprim[pr.y];
      if (i >= orb.nprim[pr.x] * nb) continue;  // padding, read by no thread
      const int ia = orb.prim_off[pr.x] + i / nb, ib = orb.prim_off[pr.y] + i % nb;
      const double a = orb.exps[ia], b = orb.exps[ib];
      const double* A = xyz + 3 * orb.atom[pr.x];
      const double* B = xyz + 3 * orb.atom[pr.y];
      const double d[3] = {A[0] - B[0], A[1] - B[1], A[2] - B[2]};
      const double p = a + b, ip = 1.0 / p;
      const double kab = exp(-a * b * ip * (d[0] * d[0] + d[1] * d[1] + d[2] * d[2])) *
                         orb.coefs[ia] * orb.coefs[ib];
      PrimPair& t = tab[e - w0];
      t.p = p;
      t.hip = 0.5 * ip;
      t.k = fabs(kab) < kPrimPairCut ? 0.0 : 2.0 * kPi * kPi * sqrt(kPi) * ip * kab;
      t.x = (a * A[0] + b * B[0]) * ip;
      t.y = (a * A[1] + b * B[1]) * ip;
      t.z = (a * A[2] + b * B[2]) * ip;
      t.a2 = 2.0 * a;
      t.b2 = 2.0 * b;
    }
    __syncthreads();
    const int e0 = max(w0, mine * stride), e1 = min(w1, mine * stride + nab);
    if (e0 < e1) body(tab + (e0 - w0), tab + (e1 - w0));
    __syncthreads();
  }
}

// What a thread needs of its triple beside the primitive pairs, loaded while
// the CTA forms those: the orbital pair's centres, the aux shell's and its
// first primitive (the only one of uncontracted sets).
struct Triple {
  int nab, nc, pc0;
  double A[3], ab[3], C[3], g0, c0;
  __device__ __forceinline__ Triple() : nab(0), nc(0), pc0(0), g0(1.0), c0(0.0) {
    A[0] = A[1] = A[2] = ab[0] = ab[1] = ab[2] = C[0] = C[1] = C[2] = 0.0;
  }
  __device__ __forceinline__ void load(const DevBasis& orb, const DevBasis& aux,
                                       const double* __restrict__ xyz, int2 pr, int sc) {
    nab = orb.nprim[pr.x] * orb.nprim[pr.y];
    pc0 = aux.prim_off[sc];
    nc = aux.nprim[sc];
    const double* a = xyz + 3 * orb.atom[pr.x];
    const double* b = xyz + 3 * orb.atom[pr.y];
    const double* c = xyz + 3 * aux.atom[sc];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      A[d] = a[d];
      ab[d] = a[d] - b[d];
      C[d] = c[d];
    }
    g0 = aux.exps[pc0];
    c0 = aux.coefs[pc0];
  }
};

// Class-molecule entry of a CTA: the last whose chunk_begin is not above the
// block index.  A warp looks at 32 evenly spaced entries of the remaining range
// per load, so n entries take log32(n) dependent loads, which every CTA waits
// for: one up to 32 molecules, three up to 32768 (a bisection takes 5 and 15).
// Every lane of a full warp must call it.
__device__ __forceinline__ int find_cm(const ClassMol* __restrict__ cms, int ncm, int block) {
  const int lane = threadIdx.x & 31;
  int lo = 0, n = ncm;  // the entry lies in [lo, lo + n), and cms[lo] is not above
  for (;;) {
    const int step = (n + 31) / 32, i = lane * step;
    const bool below = i < n && cms[lo + i].chunk_begin <= block;
    const int skip = (__popc(__ballot_sync(0xffffffffu, below)) - 1) * step;
    lo += skip;
    if (step == 1) return lo;
    n = min(step, n - skip);
  }
}

// One-electron kernels: k1eLanes lanes per shell pair.  With one thread per
// pair a class of contracted pairs was a few hundred warps, each a serial
// chain over primitive pairs times nuclei (5 % of the resident-warp limit,
// FP64 pipe 4 % active).  The lanes split the nuclei; with fewer nuclei than
// lanes, the primitive pairs as well.  (ss) derivatives of 12 x (H2O)6 0.290 ->
// 0.068 ms, (ps) 0.245 -> 0.082; (ss) values of 8 x (H2O)9 0.151 -> 0.056.
// A CTA takes k1ePairs pairs of one molecule.  A CTA of 128 pairs spread over
// eight launched ones left most of these empty for small molecules: values of
// 16384 waters 6.4 -> 2.2 ms, derivatives 9.6 -> 3.7, of 32768 H2 0.58 -> 0.14
// and 1.31 -> 0.40.
constexpr int k1eLanes = 8;
constexpr int k1ePairs = 128 / k1eLanes;
// Where the pairs alone fill the GPU, lanes beyond the nuclei only add loads,
// shuffles and the transforms' idle ones: values then take two lanes a pair
// (512 x Ar6 STO-3G 0.281 -> 0.143 ms, one lane 0.214; 16384 waters 2.2 -> 1.2).  The chunks a class must have grow with the nuclei, whose
// loop is the tail: eight and two lanes 0.082 / 0.088 for 32 x (H2O)4 (832 (ss)
// chunks), 0.126 / 0.119 for 64 (1664), 0.339 / 0.325 for 32 x (H2O)9 (4032),
// 0.318 / 0.382 for 8 x (H2O)16 (3168).  Derivatives stay ahead with eight.
constexpr int k1eFewLanes = 2;
inline int lanes_1e(int nblocks, int atoms_per_molecule) {
  return nblocks >= 1024 && nblocks / 170 >= atoms_per_molecule ? k1eFewLanes : k1eLanes;
}

template <int LANES>
struct Lanes1e {
  int lane, c0, dc, k0, dk;
  __device__ __forceinline__ explicit Lanes1e(int natom) {
    lane = threadIdx.x % LANES;
    dc = 1;
    while (dc < LANES && dc < natom) dc *= 2;
    dk = LANES / dc;
    c0 = lane % dc;
    k0 = lane / dc;
  }
};

bool dispatch_int3c(const ClassLaunch& cl, const KernelArgs& k, bool sph, cudaStream_t st);
bool dispatch_int2c(const ClassLaunch& cl, const KernelArgs& k, bool sph, cudaStream_t st);
bool dispatch_int1e(const ClassLaunch& cl, const KernelArgs& k, bool sph, cudaStream_t st);
bool dispatch_grad3c(const ClassLaunch& cl, const KernelArgs& k, bool sph, cudaStream_t st);
bool dispatch_grad2c(const ClassLaunch& cl, const KernelArgs& k, bool sph, cudaStream_t st);
bool dispatch_grad1e(const ClassLaunch& cl, const KernelArgs& k, bool sph, cudaStream_t st);

}  // namespace vqc
