// Whole SP2 purification (Niklasson, Phys. Rev. B 66, 155115 (2002)) of a batch
// of equally sized symmetric FP64 matrices in one launch: Gershgorin bounds,
// the map of the spectrum into [0, 1], every X <- X^2 or 2X - X^2 step until
// |tr X - tr X^2| < tol and kPolish steps more, and the projector out.
//
// X stays exactly symmetric, so a step forms only the tiles on or above the
// diagonal (half the flops of a plain product) and mirrors them, and
// tr X^2 = |X|_F^2 is known as soon as X is written: the branch of a step is
// decided before its product, the update is the product's epilogue, and no
// pass over X remains beside the tile loads.  Products run on the FP64 tensor
// pipe (mma.m8n8k4, the same FP64 FMA rate as the scalar pipe at a quarter of
// its operand reads).
//
// Two forms, chosen by choose() below:
//   sp2_small_kernel  one CTA per molecule, X double-buffered in shared memory;
//     steps are separated by one __syncthreads.  Bound by one SM's FP64 rate
//     and, for the smallest, by the step's latency chain.
//   sp2_group_kernel  a group of co-resident CTAs per molecule (cooperative
//     launch) over X in L2; steps are separated by a barrier of the group in
//     global memory (bounded wait).  Bound by the FP64 rate for many large
//     molecules, by barrier and load latency for few.
//
// Measured on B200 against a batched DGEMM and an update kernel per step in
// 8-step graphs with a host read of the flags after each: 14 x N = 312
// 2.72 -> 1.72 ms a purification, 1 x N = 1000 4.7 -> 2.8; the purifications of
// one water molecule's SCF (N = 24, 14 of them) 2.55 -> 0.61 ms of GPU time and
// five host reads fewer each.
#include "vqc_df.h"
#include "vqc_kernels.cuh"
#include "vqc_plan.hpp"

namespace vqc {
namespace sp2 {

__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

__device__ __forceinline__ double warp_sum(double v) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}
__device__ __forceinline__ double warp_min(double v) {
  for (int off = 16; off > 0; off >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
  for (int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}

// Once |tr X - tr X^2| < tol, kPolish more steps, X^2 and then 2X - X^2: they
// square the distance of every eigenvalue from 0 and from 1, so the projector
// is idempotent to rounding instead of to whatever below tol the last step
// happened to reach (the distance from eigenvectors scattered over 1e-14 to
// 5e-13 with it), for 4 % of the steps.
constexpr int kPolish = 2;

// the smaller of |tr X^2 - n_occ| and |tr(2X - X^2) - n_occ| picks the step
__device__ __forceinline__ bool take_square(double tr, double tr2, double nocc) {
  return fabs(tr2 - nocc) < fabs(2.0 * tr - tr2 - nocc);
}

// row tile and column tile (>= row tile) of upper-triangle tile t of nt x nt
__device__ __forceinline__ void tile_of(int t, int nt, int& rt, int& ct) {
  rt = 0;
  while (t >= nt - rt) {
    t -= nt - rt;
    ++rt;
  }
  ct = rt + t;
}

// Gershgorin interval of one row by a warp
__device__ __forceinline__ void row_bounds(const double* __restrict__ f, int n, int i, int lane,
                                           double& lo, double& hi) {
  double s = 0.0;
  for (int j = lane; j < n; j += 32) s += fabs(f[(size_t)i * n + j]);
  s = warp_sum(s);
  const double d = f[(size_t)i * n + i], radius = s - fabs(d);
  lo = fmin(lo, d - radius);
  hi = fmax(hi, d + radius);
}

__device__ __forceinline__ double mapped(const double* __restrict__ f, int n, int i, int j,
                                         double emin, double emax) {
  const double v = 0.5 * (f[(size_t)i * n + j] + f[(size_t)j * n + i]);
  return ((i == j ? emax : 0.0) - v) / (emax - emin);
}

// ---------------------------------------------------------------------------
// one CTA per molecule, X in shared memory
// ---------------------------------------------------------------------------

constexpr int kSmallThreads = 512;
constexpr int kSmallWarps = kSmallThreads / 32;

// rows padded to a multiple of 8 (zeros), row stride = rows + 4: 4 or 12
// modulo 16 doubles, so the 4 x 4 fragment of a half-warp covers all 16
// eight-byte banks
__host__ __device__ inline int small_rows(int n) { return (n + 7) & ~7; }
__host__ __device__ inline size_t small_smem(int n) {
  return sizeof(double) * (2 * (size_t)small_rows(n) * (small_rows(n) + 4) + 4 * kSmallWarps);
}
constexpr int kSmallMaxN = 112;  // two buffers of 112 x 116 doubles: 208 KB

__global__ void __launch_bounds__(kSmallThreads)
    sp2_small_kernel(const double* __restrict__ fo, int n, double nocc, double tol, int max_steps,
                     double* __restrict__ out) {
  extern __shared__ double sm[];
  const int np = small_rows(n), ld = np + 4;
  const int bufs = np * ld;
  double* red = sm + 2 * (size_t)np * ld;  // [parity][2][warps]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const double* f = fo + (size_t)blockIdx.x * n * n;
  double lo = INFINITY, hi = -INFINITY;
  for (int i = warp; i < n; i += kSmallWarps) row_bounds(f, n, i, lane, lo, hi);
  if (lane == 0) {
    red[warp] = lo;
    red[kSmallWarps + warp] = hi;
  }
  for (int i = tid; i < 2 * np * ld; i += kSmallThreads) sm[i] = 0.0;
  __syncthreads();
  for (int w = 0; w < kSmallWarps; ++w) {
    lo = fmin(lo, red[w]);
    hi = fmax(hi, red[kSmallWarps + w]);
  }
  double tr = 0.0, fro = 0.0;
  for (int i = warp; i < n; i += kSmallWarps)
    for (int j = lane; j < n; j += 32) {
      const double v = mapped(f, n, i, j, lo, hi);
      sm[i * ld + j] = v;
      fro = fma(v, v, fro);
      if (i == j) tr += v;
    }
  const int nt = (np + 15) / 16, ntiles = nt * (nt + 1) / 2;
  const int fr = lane >> 2, fc = lane & 3;
  int cur = 0, polish = 0;
  for (int step = 0;; ++step) {
    tr = warp_sum(tr);
    fro = warp_sum(fro);
    double* rp = red + 2 * kSmallWarps * ((step + 1) & 1);
    if (lane == 0) {
      rp[warp] = tr;
      rp[kSmallWarps + warp] = fro;
    }
    __syncthreads();
    tr = fro = 0.0;
    for (int w = 0; w < kSmallWarps; ++w) {  // the same order in every thread
      tr += rp[w];
      fro += rp[kSmallWarps + w];
    }
    if (polish || fabs(tr - fro) < tol) ++polish;
    if (polish > kPolish || (!polish && step >= max_steps)) break;
    const bool square = polish ? polish == 1 : take_square(tr, fro, nocc);
    const double* x = sm + cur * bufs;
    double* xn = sm + (cur ^ 1) * bufs;
    tr = fro = 0.0;
    for (int t = warp; t < ntiles; t += kSmallWarps) {
      int rt, ct;
      tile_of(t, nt, rt, ct);
      const int r0 = rt * 16, c0 = ct * 16;
      // the second 8-row half of the last tile may not exist: read the first again
      const double* a0 = x + (r0 + fr) * ld + fc;
      const double* a1 = r0 + 8 < np ? a0 + 8 * ld : a0;
      const double* b0 = x + (c0 + fr) * ld + fc;
      const double* b1 = c0 + 8 < np ? b0 + 8 * ld : b0;
      double acc[2][2][2] = {};
#pragma unroll 4
      for (int k = 0; k < np; k += 4) {
        const double u0 = a0[k], u1 = a1[k], v0 = b0[k], v1 = b1[k];
        dmma(acc[0][0], u0, v0);
        dmma(acc[0][1], u0, v1);
        dmma(acc[1][0], u1, v0);
        dmma(acc[1][1], u1, v1);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int r = r0 + 8 * i + fr, c = c0 + 8 * j + 2 * fc + e;
            if (r > c || c >= n) continue;
            const double s = acc[i][j][e];
            const double v = square ? s : 2.0 * x[r * ld + c] - s;
            xn[r * ld + c] = v;
            xn[c * ld + r] = v;
            fro = fma(r == c ? v : 2.0 * v, v, fro);
            if (r == c) tr += v;
          }
    }
    cur ^= 1;
  }
  double* o = out + (size_t)blockIdx.x * n * n;
  for (int i = warp; i < n; i += kSmallWarps)
    for (int j = lane; j < n; j += 32) o[(size_t)i * n + j] = sm[cur * bufs + i * ld + j];
}

// ---------------------------------------------------------------------------
// a group of CTAs per molecule, X in L2
// ---------------------------------------------------------------------------

constexpr int kKB = 32;          // K columns per pipeline stage
constexpr int kLdS = kKB + 4;    // stage row stride (4 modulo 16 doubles)
constexpr int kStages = 3;
constexpr unsigned long long kWaitNs = 2000000000ull;

struct GroupParams {
  const double* fo;
  double* out;
  double* x;        // [group][2][n][ld]
  double* part;     // [group][2][2][G]
  unsigned* count;  // [group] barrier arrivals, zeroed before the launch
  int* error;
  int nmol, n, ld, ngroups, G, max_steps;
  double nocc, tol;
};

template <int BM>
struct GroupCfg {
  // warps in a 2 x (BM / 16) grid, each BM/2 x 16
  static constexpr int WARPS = BM / 8, THREADS = 32 * WARPS, MI = BM / 16, NI = 2;
  static constexpr int STAGE = 2 * BM * kLdS;  // doubles: row panel, column panel
  static constexpr int SMEM = kStages * STAGE * 8;
  static constexpr int CTAS = BM == 32 ? 4 : 2;
};

__device__ __forceinline__ void cp16(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes)
               : "memory");
}

// Barrier of the group's CTAs: generation g ends when all have arrived g
// times.  The launch is cooperative, so every CTA is resident and the wait
// ends; it is bounded all the same.  False: expired (every thread sees it).
__device__ bool group_barrier(unsigned* count, unsigned target, int* error, int* flag) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(count, 1u);
    unsigned seen;
    unsigned long long t0 = 0;
    int ok = 1, polls = 0;
    for (;;) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(count) : "memory");
      if (seen >= target) break;
      if ((++polls & 1023) == 0) {
        unsigned long long now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        if (t0 == 0) t0 = now;
        if (now - t0 > kWaitNs) {
          atomicExch(error, 31);
          ok = 0;
          break;
        }
      }
    }
    __threadfence();
    *flag = ok;
  }
  __syncthreads();
  return *flag != 0;
}

template <int BM>
__global__ void __launch_bounds__(GroupCfg<BM>::THREADS, GroupCfg<BM>::CTAS)
    sp2_group_kernel(GroupParams p) {
  using C = GroupCfg<BM>;
  extern __shared__ __align__(16) double sm[];
  __shared__ double red[2][C::WARPS];
  __shared__ int flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int fr = lane >> 2, fc = lane & 3;
  const int group = blockIdx.x / p.G, rank = blockIdx.x % p.G;
  const int n = p.n, ld = p.ld, G = p.G;
  const size_t xsize = (size_t)n * ld;
  double* xbase = p.x + group * 2 * xsize;  // two iterates
  double* part = p.part + (size_t)group * 4 * G;
  unsigned* count = p.count + group;
  unsigned arrived = 0;
  const int nt = (n + BM - 1) / BM, ntiles = nt * (nt + 1) / 2;
  const int nk = (ld + kKB - 1) / kKB;
  const int wr = (warp & 1) * (BM / 2), wc = (warp >> 1) * 16;
  int parity = 0;

  // CTA sums of two values into this rank's slot of the group
  auto publish = [&](double a, double b) {
    a = warp_sum(a);
    b = warp_sum(b);
    __syncthreads();
    if (lane == 0) {
      red[0][warp] = a;
      red[1][warp] = b;
    }
    __syncthreads();
    if (tid == 0) {
      double u = 0.0, v = 0.0;
      for (int w = 0; w < C::WARPS; ++w) {
        u += red[0][w];
        v += red[1][w];
      }
      __stcg(part + (size_t)parity * 2 * G + rank, u);
      __stcg(part + (size_t)parity * 2 * G + G + rank, v);
    }
  };
  // totals over the group's slots, by every warp in the same order
  auto totals = [&](double& a, double& b) {
    a = b = 0.0;
    for (int g = lane; g < G; g += 32) {
      a += __ldcg(part + (size_t)parity * 2 * G + g);
      b += __ldcg(part + (size_t)parity * 2 * G + G + g);
    }
    a = warp_sum(a);
    b = warp_sum(b);
    parity ^= 1;
  };

  for (int mol = group; mol < p.nmol; mol += p.ngroups) {
    const double* f = p.fo + (size_t)mol * n * n;
    double lo = INFINITY, hi = -INFINITY;
    for (int i = rank * C::WARPS + warp; i < n; i += G * C::WARPS) row_bounds(f, n, i, lane, lo, hi);
    __syncthreads();
    if (lane == 0) {
      red[0][warp] = lo;
      red[1][warp] = hi;
    }
    __syncthreads();
    if (tid == 0) {
      for (int w = 0; w < C::WARPS; ++w) {
        lo = fmin(lo, red[0][w]);
        hi = fmax(hi, red[1][w]);
      }
      __stcg(part + (size_t)parity * 2 * G + rank, lo);
      __stcg(part + (size_t)parity * 2 * G + G + rank, hi);
    }
    arrived += G;
    if (!group_barrier(count, arrived, p.error, &flag)) return;
    lo = INFINITY;
    hi = -INFINITY;
    for (int g = lane; g < G; g += 32) {
      lo = fmin(lo, __ldcg(part + (size_t)parity * 2 * G + g));
      hi = fmax(hi, __ldcg(part + (size_t)parity * 2 * G + G + g));
    }
    lo = warp_min(lo);
    hi = warp_max(hi);
    parity ^= 1;
    double tr = 0.0, fro = 0.0;
    for (int i = rank * C::WARPS + warp; i < n; i += G * C::WARPS)
      for (int j = lane; j < ld; j += 32) {
        const double v = j < n ? mapped(f, n, i, j, lo, hi) : 0.0;
        __stcg(xbase + (size_t)i * ld + j, v);
        if (j >= n) __stcg(xbase + xsize + (size_t)i * ld + j, 0.0);  // padding columns stay zero
        fro = fma(v, v, fro);
        if (i == j) tr += v;
      }
    int cur = 0, polish = 0;
    for (int step = 0;; ++step) {
      publish(tr, fro);
      arrived += G;
      if (!group_barrier(count, arrived, p.error, &flag)) return;
      totals(tr, fro);
      if (polish || fabs(tr - fro) < p.tol) ++polish;
      if (polish > kPolish || (!polish && step >= p.max_steps)) break;
      const bool square = polish ? polish == 1 : take_square(tr, fro, p.nocc);
      const double* x = xbase + cur * xsize;
      double* xn = xbase + (cur ^ 1) * xsize;
      tr = fro = 0.0;
      for (int t = rank; t < ntiles; t += G) {
        int rt, ct;
        tile_of(t, nt, rt, ct);
        const int r0 = rt * BM, c0 = ct * BM;
        const bool diag = rt == ct;  // one panel serves both sides
        auto load = [&](int kb) {
          const uint32_t s = (uint32_t)__cvta_generic_to_shared(sm + (kb % kStages) * C::STAGE);
          const int rows = diag ? BM : 2 * BM;
          for (int q = tid; q < rows * (kKB / 2); q += C::THREADS) {
            const int r = q / (kKB / 2), k = (q % (kKB / 2)) * 2;
            const int gr = r < BM ? r0 + r : c0 + r - BM, gk = kb * kKB + k;
            const bool in = gr < n && gk < ld;  // outside: zeros, nothing is read
            cp16(s + (r * kLdS + k) * 8, x + (in ? (size_t)gr * ld + gk : 0), in ? 16 : 0);
          }
        };
        double acc[C::MI][C::NI][2] = {};
#pragma unroll
        for (int kb = 0; kb < kStages - 1; ++kb) {
          if (kb < nk) load(kb);
          asm volatile("cp.async.commit_group;" ::: "memory");
        }
        // the diagonal tile's warps below its diagonal have nothing to add
        const bool idle = diag && wr >= wc + 16;
        for (int kb = 0; kb < nk; ++kb) {
          asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
          __syncthreads();  // stage kb is complete; the stage read in kb - 1 is free
          if (kb + kStages - 1 < nk) load(kb + kStages - 1);
          asm volatile("cp.async.commit_group;" ::: "memory");
          if (idle) continue;
          const double* s = sm + (kb % kStages) * C::STAGE;
          const double* a = s + (wr + fr) * kLdS + fc;
          const double* b = s + ((diag ? 0 : BM) + wc + fr) * kLdS + fc;
#pragma unroll
          for (int k = 0; k < kKB; k += 4) {
            double u[C::MI], v[C::NI];
#pragma unroll
            for (int i = 0; i < C::MI; ++i) u[i] = a[i * 8 * kLdS + k];
#pragma unroll
            for (int j = 0; j < C::NI; ++j) v[j] = b[j * 8 * kLdS + k];
#pragma unroll
            for (int i = 0; i < C::MI; ++i)
#pragma unroll
              for (int j = 0; j < C::NI; ++j) dmma(acc[i][j], u[i], v[j]);
          }
        }
        __syncthreads();  // the next tile's loads reuse the stages
#pragma unroll
        for (int i = 0; i < C::MI; ++i)
#pragma unroll
          for (int j = 0; j < C::NI; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int r = r0 + wr + 8 * i + fr, c = c0 + wc + 8 * j + 2 * fc + e;
              if (r > c || c >= n) continue;
              const double s = acc[i][j][e];
              const double v = square ? s : 2.0 * __ldcg(x + (size_t)r * ld + c) - s;
              __stcg(xn + (size_t)r * ld + c, v);
              if (r != c) __stcg(xn + (size_t)c * ld + r, v);
              fro = fma(r == c ? v : 2.0 * v, v, fro);
              if (r == c) tr += v;
            }
      }
      cur ^= 1;
    }
    double* o = p.out + (size_t)mol * n * n;
    for (int i = rank * C::WARPS + warp; i < n; i += G * C::WARPS)
      for (int j = lane; j < n; j += 32) o[(size_t)i * n + j] = __ldcg(xbase + cur * xsize + (size_t)i * ld + j);
    // the next molecule rewrites the iterates: its first write comes after the
    // bounds barrier, which every CTA reaches only after this copy
  }
}

// Nothing or everything occupied: zero or the identity, whatever the spectrum.
// The steps cannot reach the identity where a Gershgorin bound is an
// eigenvalue (it is mapped to 0 and stays there), as for one function or a
// diagonal matrix.  Non-finite elements stay visible.
__global__ void __launch_bounds__(256)
    sp2_trivial_kernel(const double* __restrict__ fo, size_t total, int n, double diagonal,
                       double* __restrict__ out) {
  for (size_t e = (size_t)blockIdx.x * 256 + threadIdx.x; e < total; e += (size_t)gridDim.x * 256) {
    const size_t nn = (size_t)n * n, base = e / nn * nn;
    const int i = (int)((e - base) / n), j = (int)((e - base) % n);
    const double sum = fo[e] + fo[base + (size_t)j * n + i];
    out[e] = (i == j ? diagonal : 0.0) + 0.0 * sum;
  }
}

struct Choice {
  int path;  // 1: one CTA per molecule; 2, 3: groups with 32- and 64-row tiles
  int ngroups, G;
};

// Groups of G CTAs for nmol molecules in r rounds, minimising the step time
// r * (barrier + tiles per CTA * tile time): a tile of BM rows costs BM^2 n
// FMAs at one SM's 64 a cycle, shared by the CTAs resident on it.  The cycles
// of a barrier (4000) and of filling a tile's pipeline (1500) and the factor
// on the FMAs (1.4) are round numbers that rank plans: of 32- and 64-row tiles
// the pick was the faster, or within 1 %, at 51 of 52 pairs of N = 120-2000
// and 1-128 molecules (32 x N = 312: 3.08 against 2.91 ms).
static Choice plan_groups(int nmol, int n, int bm, int resident, int sms, double& cost) {
  const int nt = (n + bm - 1) / bm, tiles = nt * (nt + 1) / 2;
  Choice best{bm == 32 ? 2 : 3, 0, 0};
  cost = 1e300;
  const int r0 = (nmol + resident - 1) / resident;
  for (int r = r0; r < r0 + 64; ++r) {
    const int groups = (nmol + r - 1) / r;
    int g = resident / groups;
    g = g > tiles ? tiles : g;
    const int per = (tiles + g - 1) / g;
    g = (tiles + per - 1) / per;  // no CTA without a tile in the last pass
    const int share = (groups * g + sms - 1) / sms;
    const double c = r * (4000.0 + (double)per * (1500.0 + (double)share * bm * bm * n / 64.0 * 1.4));
    if (c < cost) {
      cost = c;
      best.ngroups = groups;
      best.G = g;
    }
    if (groups == 1) break;
  }
  return best;
}

static cudaError_t choose(int nmol, int n, int path, Choice& ch) {
  int dev = 0, sms = 0;
  cudaError_t e;
  if ((e = cudaGetDevice(&dev))) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev))) return e;
  // Measured us a purification, one CTA against 32-row groups: N = 24 57 / 176,
  // N = 64 115 / 237, N = 72 (128 molecules) 158 / 542, N = 96 279 / 291-309,
  // 128 x N = 96 294 / 599; N = 112 347-368 / 316-356 for up to 8 molecules but
  // 366 / 427 for 32 and 383 / 1029 for 128, as one SM per molecule stays
  // cheaper once the molecules alone fill a good part of the GPU.
  if (path == 0 && (n <= 96 || (n <= kSmallMaxN && nmol >= 24))) path = 1;
  if (path == 1) {
    ch = Choice{1, nmol, 1};
    return cudaSuccess;
  }
  double c32 = 0, c64 = 0;
  Choice a{}, b{};
  for (int bm : {32, 64}) {
    const void* fn = bm == 32 ? (const void*)sp2_group_kernel<32> : (const void*)sp2_group_kernel<64>;
    const int smem = bm == 32 ? GroupCfg<32>::SMEM : GroupCfg<64>::SMEM;
    if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem))) return e;
    int per_sm = 0;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
             &per_sm, fn, bm == 32 ? GroupCfg<32>::THREADS : GroupCfg<64>::THREADS, smem)))
      return e;
    if (per_sm < 1) return cudaErrorLaunchOutOfResources;
    if (bm == 32) a = plan_groups(nmol, n, bm, per_sm * sms, sms, c32);
    else b = plan_groups(nmol, n, bm, per_sm * sms, sms, c64);
  }
  if (!a.G || !b.G) return cudaErrorInvalidConfiguration;
  ch = path == 2 ? a : (path == 3 ? b : (c64 < c32 ? b : a));
  return cudaSuccess;
}

static size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }
static int group_ld(int n) { return (n + 7) & ~7; }

static size_t workspace(const Choice& ch, int n) {
  if (ch.path == 1) return 0;
  return align256(sizeof(unsigned) * ch.ngroups) + align256(sizeof(double) * 4 * ch.ngroups * ch.G) +
         align256(sizeof(double) * 2 * ch.ngroups * (size_t)n * group_ld(n));
}

}  // namespace sp2
}  // namespace vqc

using namespace vqc;

extern "C" {

int vqc_sp2_purify_workspace(int32_t nmol, int32_t n, int32_t path, uint64_t* bytes) {
  if (!bytes || nmol <= 0 || n <= 0 || path < 0 || path > 3 || (path == 1 && n > sp2::kSmallMaxN))
    return fail(VQC_STATUS_INVALID_ARGUMENT, "sp2_purify_workspace: bad argument");
  sp2::Choice ch{};
  cudaError_t e = sp2::choose(nmol, n, path, ch);
  if (e != cudaSuccess) return cuda_status(e, "sp2_purify_workspace");
  *bytes = sp2::workspace(ch, n);
  return VQC_STATUS_SUCCESS;
}

int vqc_sp2_purify(const double* fo, int32_t nmol, int32_t n, double nocc, double tol,
                   int32_t max_steps, int32_t path, double* out, void* work, uint64_t work_bytes,
                   int32_t* error, void* stream) {
  if (!fo || !out || !error || nmol <= 0 || n <= 0 || max_steps < 0 || path < 0 || path > 3 ||
      (path == 1 && n > sp2::kSmallMaxN))
    return fail(VQC_STATUS_INVALID_ARGUMENT, "sp2_purify: bad argument");
  cudaStream_t st = (cudaStream_t)stream;
  if (nocc <= 0.0 || nocc >= n) {
    const size_t total = (size_t)nmol * n * n, ctas = (total + 255) / 256;
    sp2::sp2_trivial_kernel<<<(int)(ctas > 16 * 148 ? 16 * 148 : ctas), 256, 0, st>>>(
        fo, total, n, nocc <= 0.0 ? 0.0 : 1.0, out);
    count_launch();
    return cuda_status(cudaGetLastError(), "sp2_purify");
  }
  sp2::Choice ch{};
  cudaError_t e = sp2::choose(nmol, n, path, ch);
  if (e != cudaSuccess) return cuda_status(e, "sp2_purify");
  if (ch.path == 1) {
    const int smem = (int)sp2::small_smem(n);
    if ((e = cudaFuncSetAttribute(sp2::sp2_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sp2::small_smem(sp2::kSmallMaxN))))
      return cuda_status(e, "sp2_purify");
    sp2::sp2_small_kernel<<<nmol, sp2::kSmallThreads, smem, st>>>(fo, n, nocc, tol, max_steps, out);
    count_launch();
    return cuda_status(cudaGetLastError(), "sp2_purify");
  }
  if (!work || work_bytes < sp2::workspace(ch, n) || ((uintptr_t)work & 255))
    return fail(VQC_STATUS_INVALID_ARGUMENT, "sp2_purify: workspace too small or not 256-byte aligned");
  char* w = static_cast<char*>(work);
  sp2::GroupParams p{};
  p.fo = fo;
  p.out = out;
  p.count = reinterpret_cast<unsigned*>(w);
  const size_t cbytes = sp2::align256(sizeof(unsigned) * ch.ngroups);
  w += cbytes;
  p.part = reinterpret_cast<double*>(w);
  w += sp2::align256(sizeof(double) * 4 * ch.ngroups * ch.G);
  p.x = reinterpret_cast<double*>(w);
  p.error = error;
  p.nmol = nmol;
  p.n = n;
  p.ld = sp2::group_ld(n);
  p.ngroups = ch.ngroups;
  p.G = ch.G;
  p.max_steps = max_steps;
  p.nocc = nocc;
  p.tol = tol;
  if ((e = cudaMemsetAsync(p.count, 0, cbytes, st))) return cuda_status(e, "sp2_purify");
  void* args[] = {&p};
  const bool small_tiles = ch.path == 2;
  e = cudaLaunchCooperativeKernel(
      small_tiles ? (const void*)sp2::sp2_group_kernel<32> : (const void*)sp2::sp2_group_kernel<64>,
      dim3(ch.ngroups * ch.G), dim3(small_tiles ? sp2::GroupCfg<32>::THREADS : sp2::GroupCfg<64>::THREADS),
      args, small_tiles ? sp2::GroupCfg<32>::SMEM : sp2::GroupCfg<64>::SMEM, st);
  count_launch();
  return cuda_status(e, "sp2_purify");
}

}  // extern "C"
