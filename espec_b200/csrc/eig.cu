// eig.cu -- batched initial-state eigensolver on 2D grids (eSPec's LANCZSG,
// lanczsc.f:56-120, with LNZ lnz.f:76-119 and REORT reort.f:65-80), FP64.
//
// One CTA per problem (one potential), or a cluster of two where that leaves no SM
// without a problem: for each of nstates target states, explicitly restarted
// Lanczos -- m Lanczos steps with full classical
// Gram-Schmidt reorthogonalisation from the current vector, the lowest Ritz
// pair of the m x m tridiagonal matrix, restart from that Ritz vector --
// until the true residual |H v - theta v| (one more H*v) is at most tol.  The
// states already found are locked: projected out of every restart vector and
// kept in the reorthogonalisation set (without that, the reference's K-th
// Ritz vector can settle on a higher state; espec.f:896-903 restricts
// LANCZSG to the ground state).
// DSTEVX('V','I') is replaced by multisection on the Sturm count (one warp,
// 33 points per round) and inverse iteration for the Ritz vector.  Every
// application of H is counted: the count is the cost metric of the solver.
// Cold start: the reference's LCG vectors (rans.f:38-39, NSEED = 1, first N
// draws discarded, lanczsc.f:56-62); warm start: any given vectors.
#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>
#include <vector>

#include "espec_gpu.h"
#include "espec_internal.h"

namespace espec {
namespace {

// 16 warps of up to 128 registers: a thread keeps 16 to 32 loads in flight
constexpr int kEigThreads = 512;
// CTA sums run over kEigChains accumulation chains (chain u: points u, u +
// kEigChains, ...), each thread two of them, chains added in warps of 32
constexpr int kEigChains = 1024;
// points of a current vector kept in shared memory (beside 31 KB of static arrays)
constexpr int kEigMaxSmemN = 24 * 1024;
// points from which two CTAs share a problem: six restarts of two states, 16 problems, ms
// with one CTA and with two: 1024 points 4.9 and 5.3, 1440 5.7 and 5.9, 2025 7.7 and 7.2,
// 2048 6.0 and 6.0, 2304 7.4 and 6.6, 4096 9.5 and 7.7, 16384 33 and 21
constexpr int kEigMinSplitN = 2048;
constexpr int kEigMaxM = 40;      // NREORT = 40 in lanczsc.f:55
constexpr int kEigMaxStates = 16;  // locked states held in the reorthogonalisation

struct EigArgs {
  int nx, ny, n;
  double shm[2], sht30;
  const double* vpot;   // [nprob][n]
  const double* start;  // [nprob][nstates][n]
  double* L;            // [nprob][m][n]
  double* work;         // [nprob][n]: H vi - bt v_prev of an iteration
  double* vec;          // [nprob][nstates][n]
  double* eval;         // [nprob][nstates]
  double* resid;        // [nprob][nstates]
  int* matvecs;         // [nprob][nstates]
  int nstates, m, maxrest;
  double tol;
};

// H_FD x (au2di.f:57-225) at point k of an nx x ny grid, x scaled by d
__device__ __forceinline__ double hx(const EigArgs& a, const double* V, const double* x, int k,
                                     double d) {
  const int i = k % a.nx, j = k / a.nx;
  double s = (a.sht30 + V[k]) * (x[k] * d);
  const double h0 = a.shm[0], h1 = a.shm[1];
  if (i >= 2) s += h0 * (x[k - 2] * d);
  if (i >= 1) s += -16.0 * h0 * (x[k - 1] * d);
  if (i + 1 < a.nx) s += -16.0 * h0 * (x[k + 1] * d);
  if (i + 2 < a.nx) s += h0 * (x[k + 2] * d);
  const int sy = a.nx;
  if (j >= 2) s += h1 * (x[k - 2 * sy] * d);
  if (j >= 1) s += -16.0 * h1 * (x[k - sy] * d);
  if (j + 1 < a.ny) s += -16.0 * h1 * (x[k + sy] * d);
  if (j + 2 < a.ny) s += h1 * (x[k + 2 * sy] * d);
  return s;
}

// A problem's share of this CTA: with CS = 2 the chains are split between the two
// CTAs of a cluster (rank 0: chains 0..511), so a thread has one, and values that
// the other CTA needs are stored in its shared memory as well.  Every sum keeps
// the order it has in one CTA: the results do not depend on CS.
template <int CS>
struct Share {
  static constexpr int kStep = CS * kEigThreads;  // from point to point of a thread
  int rank, first;
  __device__ __forceinline__ Share()
      : rank(CS == 1 ? 0 : (int)(blockIdx.x & 1)), first((int)threadIdx.x + rank * kEigThreads) {}
  // chain (of the thread's two, CS = 1) of its i-th point
  static __device__ __forceinline__ int chain(int i) { return CS == 1 ? i & 1 : 0; }
  __device__ __forceinline__ void sync() const {
    if (CS == 1) {
      __syncthreads();
    } else {
      asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
      asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    }
  }
  // vectors in global memory: with one CTA by way of L1, which holds those of a small
  // grid; with two past it, since the other CTA writes to them
  __device__ __forceinline__ double load(const double* p) const {
    return CS == 1 ? *p : __ldcg(p);
  }
  // *p = v here and in the other CTA (p in shared memory)
  __device__ __forceinline__ void put(double* p, double v) const {
    *p = v;
    if (CS == 2) {
      uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank ^ 1));
      asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(r), "d"(v) : "memory");
    }
  }
};

// sum of all chains: the thread's chain sums x0 (and x1, CS = 1).  Two buffers
// [2][kEigChains / 32] in turn: a CTA may store its part of the next sum in its
// partner while that one still reads this sum, but not of the sum after it, since the
// partner has arrived at the next sum's barrier by then.
template <int CS>
__device__ __forceinline__ double chain_sum(const Share<CS>& sh, double x0, double x1,
                                            double* bufs, int& turn) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* ws = bufs + turn * (kEigChains / 32);
  turn ^= 1;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    x0 += __shfl_xor_sync(0xffffffffu, x0, o);
    if (CS == 1) x1 += __shfl_xor_sync(0xffffffffu, x1, o);
  }
  if (lane == 0) {
    sh.put(ws + warp + sh.rank * (kEigThreads / 32), x0);
    if (CS == 1) ws[warp + kEigThreads / 32] = x1;
  }
  sh.sync();
  double s = 0.0;
  for (int w = 0; w < kEigChains / 32; ++w) s += ws[w];
  __syncthreads();
  return s;
}

// red[q] = <x, Y_q>, q < nl + nlock, with Y_q = L_q (q < nl) or lock_(q-nl).
// Each product is two accumulation chains per lane (points lane + 64 i and
// lane + 32 + 64 i); a warp takes one chain set of one vector at a time, so
// that even the first iterations of a restart keep every warp loading, with
// kDotLoads loads of the vector in flight per lane (with two, one CTA drew
// about 20 GB/s).  part: [2 (kEigMaxM + kEigMaxStates)][32] in shared memory.
constexpr int kDotLoads = 32, kTailLoads = 8;
template <int CS>
__device__ __forceinline__ void warp_dots(const Share<CS>& sh, const double* x, const double* L,
                                          int nl, const double* lock, int nlock, int n,
                                          double* part, double* red) {
  constexpr int NW = kEigThreads / 32;  // even: a vector's two chain sets stay in one CTA
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nv = nl + nlock;
  if (CS == 1 && n < kEigMinSplitN) {
    // a small grid: both chains of a vector in one warp, no exchange (three restarts of
    // two states, with it and the loads by way of L1: 35 points 1.58 -> 1.01 ms, 256 1.32
    // -> 1.07, 1024 1.70 -> 1.53, 2025 2.53 -> 2.29)
    for (int q = warp; q < nv; q += NW) {
      const double* y = q < nl ? L + (long)q * n : lock + (long)(q - nl) * n;
      double s[2] = {0.0, 0.0};
      for (int k = lane; k < n; k += 32 * kTailLoads) {
        double v[kTailLoads], u[kTailLoads];
#pragma unroll
        for (int j = 0; j < kTailLoads; ++j) {
          const bool in = k + 32 * j < n;
          v[j] = in ? sh.load(y + k + 32 * j) : 0.0;
          u[j] = in ? x[k + 32 * j] : 0.0;
        }
#pragma unroll
        for (int j = 0; j < kTailLoads; ++j)
          if (k + 32 * j < n) s[j & 1] += u[j] * v[j];
      }
      double d = s[0] + s[1];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
      if (lane == 0) red[q] = d;
    }
    __syncthreads();
    return;
  }
  for (int task = warp + sh.rank * NW; task < 2 * nv; task += CS * NW) {
    const int q = task >> 1;
    const double* y = q < nl ? L + (long)q * n : lock + (long)(q - nl) * n;
    double s = 0.0;
    int k = lane + 32 * (task & 1);
    for (; k + 64 * (kDotLoads - 1) < n; k += 64 * kDotLoads) {
      double v[kDotLoads];
#pragma unroll
      for (int j = 0; j < kDotLoads; ++j) v[j] = sh.load(y + k + 64 * j);
#pragma unroll
      for (int j = 0; j < kDotLoads; ++j) s += x[k + 64 * j] * v[j];
    }
    for (; k < n; k += 64 * kTailLoads) {
      double v[kTailLoads], u[kTailLoads];
#pragma unroll
      for (int j = 0; j < kTailLoads; ++j) {
        const bool in = k + 64 * j < n;
        v[j] = in ? sh.load(y + k + 64 * j) : 0.0;
        u[j] = in ? x[k + 64 * j] : 0.0;
      }
#pragma unroll
      for (int j = 0; j < kTailLoads; ++j)
        if (k + 64 * j < n) s += u[j] * v[j];
    }
    part[task * 32 + lane] = s;
  }
  __syncthreads();
  for (int q = warp; q < nv; q += NW) {
    if (CS == 2 && (2 * q / NW & 1) != sh.rank) continue;
    double s = part[2 * q * 32 + lane] + part[(2 * q + 1) * 32 + lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) sh.put(red + q, s);
  }
  sh.sync();
}

// w[i] = init(k_i) - sum_j lock_j(k_i) a_j - sum_q L_q(k_i) b_q (or plus),
// for the thread's points, P at a time and 16 / P vectors so that their loads overlap;
// put(k, chain, w) takes each, in order.  Four; two on one CTA's grids of up to two points
// per thread, where loads for points that do not exist cost as much as the others (three
// states, 40 vectors, two restarts, ms with four and two: 256 points 1.50 and 1.42, 600 2.04 and
// 1.87, 1024 2.32 and 2.18, but 1296 2.77 and 2.79)
template <int P, int CS, class Init, class Put>
__device__ __forceinline__ void combine_points(const Share<CS>& sh, const double* lock,
                                               const double* ca, int nlock, const double* L,
                                               const double* cb, int nl, int n, bool plus,
                                               Init init, Put put) {
  for (int k0 = sh.first; k0 < n; k0 += P * sh.kStep) {
    double w[P];
    int kk[P];
#pragma unroll
    for (int i = 0; i < P; ++i) {
      kk[i] = min(k0 + i * sh.kStep, n - 1);
      w[i] = init(kk[i]);
    }
    for (int j = 0; j < nlock; ++j) {
      const double c = ca[j];
#pragma unroll
      for (int i = 0; i < P; ++i) w[i] -= c * sh.load(lock + (long)j * n + kk[i]);
    }
    if (plus) {
#pragma unroll 16 / P
      for (int q = 0; q < nl; ++q) {
        const double c = cb[q];
#pragma unroll
        for (int i = 0; i < P; ++i) w[i] += c * sh.load(L + (long)q * n + kk[i]);
      }
    } else {
#pragma unroll 16 / P
      for (int q = 0; q < nl; ++q) {
        const double c = cb[q];
#pragma unroll
        for (int i = 0; i < P; ++i) w[i] -= c * sh.load(L + (long)q * n + kk[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < P; ++i)
      if (k0 + i * sh.kStep < n) put(k0 + i * sh.kStep, sh.chain(i), w[i]);
  }
}
template <int CS, class Init, class Put>
__device__ __forceinline__ void combine(const Share<CS>& sh, const double* lock, const double* ca,
                                        int nlock, const double* L, const double* cb, int nl,
                                        int n, bool plus, Init init, Put put) {
  if (CS == 1 && n <= 2 * sh.kStep)
    combine_points<2>(sh, lock, ca, nlock, L, cb, nl, n, plus, init, put);
  else
    combine_points<4>(sh, lock, ca, nlock, L, cb, nl, n, plus, init, put);
}

// number of eigenvalues of the tridiagonal (d, e) below x (Sturm count)
__device__ __forceinline__ int sturm(int m, const double* d, const double* e2, double x) {
  int c = 0;
  double q = d[0] - x;
  if (q < 0) ++c;
  for (int i = 1; i < m; ++i) {
    if (q == 0.0) q = 1e-300;
    q = d[i] - x - e2[i - 1] / q;
    if (q < 0) ++c;
  }
  return c;
}

// Solves (T - th I) y = b in place (b in y), T symmetric tridiagonal with
// diagonal al and off-diagonal bt: Gaussian elimination of the subdiagonal
// with a row interchange whenever the subdiagonal entry is the larger pivot
// (the interchange fills a second superdiagonal), then back substitution.
__host__ __device__ inline void tri_solve_pivoted(int m, const double* al, const double* bt,
                                                  double th, double* y) {
  double d[kEigMaxM], du[kEigMaxM], du2[kEigMaxM];
  for (int i = 0; i < m; ++i) {
    d[i] = al[i] - th;
    du[i] = i + 1 < m ? bt[i] : 0.0;
    du2[i] = 0.0;
  }
  for (int i = 0; i + 1 < m; ++i) {
    const double sub = bt[i];  // row i+1, column i
    if (fabs(d[i]) >= fabs(sub)) {
      if (d[i] == 0.0) d[i] = 1e-300;
      const double f = sub / d[i];
      d[i + 1] -= f * du[i];
      y[i + 1] -= f * y[i];
    } else {
      const double f = d[i] / sub;
      const double di1 = d[i + 1], dui1 = du[i + 1];
      d[i] = sub;
      d[i + 1] = du[i] - f * di1;
      du[i] = di1;
      du2[i] = dui1;
      du[i + 1] = -f * dui1;
      const double yi = y[i];
      y[i] = y[i + 1];
      y[i + 1] = yi - f * y[i + 1];
    }
  }
  if (d[m - 1] == 0.0) d[m - 1] = 1e-300;
  for (int i = m - 1; i >= 0; --i) {
    double s = y[i];
    if (i + 1 < m) s -= du[i] * y[i + 1];
    if (i + 2 < m) s -= du2[i] * y[i + 2];
    y[i] = s / d[i];
  }
}

}  // namespace

// SM: the current vector in shared memory (grids up to kEigMaxSmemN points), all
// of it in each CTA of a cluster; otherwise it is the work array in global memory
template <bool SM, int CS>
__global__ void __launch_bounds__(kEigThreads, 1) eig_kernel(EigArgs a) {
  static_assert(SM || CS == 1, "a cluster exchanges the current vector through shared memory");
  constexpr int NV = kEigMaxM + kEigMaxStates;
  extern __shared__ double eig_dyn[];
  __shared__ double part[2 * NV * 32];
  __shared__ double ws[2 * (kEigChains / 32)];
  __shared__ double red[NV];
  __shared__ double s_al[kEigMaxM], s_bt[kEigMaxM], s_e2[kEigMaxM], s_y[kEigMaxM];
  __shared__ double s_theta;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int p = blockIdx.x / CS, n = a.n, m = a.m;
  const Share<CS> sh;
  int turn = 0;  // chain_sum's buffer
  const int k1 = sh.first, step = sh.kStep;
  const double* V = a.vpot + (long)p * n;
  double* L = a.L + (long)p * m * n;
  double* work = a.work + (long)p * n;
  double* F = SM ? eig_dyn : work;  // the current vector

  for (int K = 0; K < a.nstates; ++K) {
    const double* st = a.start + ((long)p * a.nstates + K) * n;
    double* v = a.vec + ((long)p * a.nstates + K) * n;
    for (int k = t; k < n; k += kEigThreads) F[k] = st[k];
    sh.sync();  // and the state before is in a.vec
    int count = 0;
    double res = 0.0;
    const double* lock = a.vec + (long)p * a.nstates * n;  // states 0..K-1
    for (int rs = 0; rs < a.maxrest; ++rs) {
      // ---- project the locked states out of the current vector
      if (K > 0) {
        warp_dots(sh, F, nullptr, 0, lock, K, n, part, red);
        combine(sh, lock, red, K, nullptr, nullptr, 0, n, false, [&](int k) { return F[k]; },
                [&](int k, int, double w) { F[k] = w; });
        __syncthreads();
      }
      // ---- m Lanczos steps (lnz.f:76-119)
      double nn[2] = {0.0, 0.0};
      for (int k = k1, i = 0; k < n; k += step, ++i) {
        if (sh.chain(i)) nn[1] += F[k] * F[k];
        else nn[0] += F[k] * F[k];
      }
      double bt0 = sqrt(chain_sum(sh, nn[0], nn[1], ws, turn));
      for (int it = 0; it < m; ++it) {
        double* Li = L + (long)it * n;
        const double* Lp = it ? L + (long)(it - 1) * n : nullptr;
#pragma unroll 4
        for (int k = k1; k < n; k += step) {
          const double vi = F[k] / bt0;
          Li[k] = vi;
          if (SM) sh.put(F + k, vi);
        }
        sh.sync();
        // w = H vi - bt0 v_prev into work, al = <vi, w> (lnz.f:96-107)
        const double* x = SM ? F : Li;
        nn[0] = nn[1] = 0.0;
#pragma unroll 2
        for (int k0 = k1; k0 < n; k0 += kEigChains) {
#pragma unroll
          for (int c = 0; c < 2 / CS; ++c) {
            const int k = k0 + c * kEigThreads;
            if (k < n) {
              const double vp = it ? Lp[k] : 0.0;
              const double w = hx(a, V, x, k, 1.0) - bt0 * vp;
              work[k] = w;
              nn[c] += x[k] * w;
            }
          }
        }
        const double al = chain_sum(sh, nn[0], nn[1], ws, turn);
        if (t == 0) s_al[it] = al;
        ++count;
        // work = w - al vi, then classical Gram-Schmidt against the locked
        // states and L_0..L_it (reort.f:65-80: all dot products, then all
        // updates): one pass for the dots, one for the updates and the norm
#pragma unroll 4
        for (int k = k1; k < n; k += step) {
          const double w = work[k] - al * x[k];
          if (SM) sh.put(F + k, w);
          else F[k] = w;
        }
        sh.sync();
        warp_dots(sh, F, L, it + 1, lock, K, n, part, red);
        nn[0] = nn[1] = 0.0;
        combine(sh, lock, red + it + 1, K, L, red, it + 1, n, false, [&](int k) { return F[k]; },
                [&](int k, int c, double w) {
                  F[k] = w;
                  nn[c] += w * w;
                });
        bt0 = sqrt(chain_sum(sh, nn[0], nn[1], ws, turn));
        if (t == 0) s_bt[it] = bt0;
      }
      __syncthreads();
      // ---- lowest Ritz pair of T (DSTEVX('V','I',...,IL,IU))
      if (warp == 0) {
        if (lane == 0) {
          for (int i = 0; i + 1 < m; ++i) s_e2[i] = s_bt[i] * s_bt[i];
        }
        __syncwarp();
        double lo = 1e300, hi = -1e300;
        for (int i = 0; i < m; ++i) {  // Gershgorin interval
          const double r = (i > 0 ? fabs(s_bt[i - 1]) : 0.0) + (i + 1 < m ? fabs(s_bt[i]) : 0.0);
          lo = fmin(lo, s_al[i] - r);
          hi = fmax(hi, s_al[i] + r);
        }
        const double span = hi - lo;
        lo -= 1e-12 * span + 1e-300;
        hi += 1e-12 * span + 1e-300;
        // multisection: the K-th eigenvalue lies where the count passes K
        for (int round = 0; round < 16; ++round) {
          const double x = lo + (hi - lo) * (lane + 1) / 33.0;
          const int c = sturm(m, s_al, s_e2, x);
          const unsigned below = __ballot_sync(0xffffffffu, c <= 0);  // points below all
          const int nb = __popc(below);  // counts grow with x: the first nb points
          const double nlo = nb > 0 ? lo + (hi - lo) * nb / 33.0 : lo;
          const double nhi = nb < 32 ? lo + (hi - lo) * (nb + 1) / 33.0 : hi;
          lo = nlo;
          hi = nhi;
          if (hi - lo <= 4e-16 * fmax(fabs(lo), fabs(hi))) break;
        }
        if (lane == 0) {
          const double th = 0.5 * (lo + hi);
          s_theta = th;
          // inverse iteration on T - th I from a vector of ones, three
          // sweeps, each a tridiagonal solve with row interchanges
          double y[kEigMaxM];
          for (int i = 0; i < m; ++i) y[i] = 1.0;
          for (int sweep = 0; sweep < 3; ++sweep) {
            tri_solve_pivoted(m, s_al, s_bt, th, y);
            double nrm = 0.0;
            for (int i = 0; i < m; ++i) nrm += y[i] * y[i];
            nrm = sqrt(nrm);
            for (int i = 0; i < m; ++i) y[i] /= nrm;
          }
          for (int i = 0; i < m; ++i) s_y[i] = y[i];
        }
      }
      __syncthreads();
      // ---- the new vector L y, normalised (lanczsc.f:99-113, FATN = ECNORM)
      nn[0] = nn[1] = 0.0;
      combine(sh, nullptr, nullptr, 0, L, s_y, m, n, true, [](int) { return 0.0; },
              [&](int k, int c, double w) {
                F[k] = w;
                nn[c] += w * w;
              });
      const double inv = 1.0 / sqrt(chain_sum(sh, nn[0], nn[1], ws, turn));
      for (int k = k1; k < n; k += step) {
        if (SM) sh.put(F + k, F[k] * inv);
        else F[k] *= inv;
      }
      sh.sync();
      // ---- true residual |H v - theta v|
      const double th = s_theta;
      nn[0] = nn[1] = 0.0;
      for (int k = k1, i = 0; k < n; k += step, ++i) {
        const double r = hx(a, V, F, k, 1.0) - th * F[k];
        if (sh.chain(i)) nn[1] += r * r;
        else nn[0] += r * r;
      }
      ++count;
      res = sqrt(chain_sum(sh, nn[0], nn[1], ws, turn));
      if (res <= a.tol) break;
    }
    for (int k = k1; k < n; k += step) v[k] = F[k];
    if (t == 0 && sh.rank == 0) {
      const long o = (long)p * a.nstates + K;
      a.eval[o] = s_theta;
      a.resid[o] = res;
      a.matvecs[o] = count;
    }
    __syncthreads();
  }
}

// LCG of rans.f:38-39 (NSEED = MOD(NSEED*1029 + 221591, 2^20), RAN = NSEED/2^20)
// jumped ahead: value number idx (1-based) of the sequence from seed 1
__global__ void lcg_kernel(double* out, long count, long first) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const unsigned long long M = 1ull << 20;
  // affine map f(x) = A x + C; f^j by binary powering
  unsigned long long A = 1, C = 0, bA = 1029, bC = 221591;
  unsigned long long e = (unsigned long long)(first + i);
  while (e) {
    if (e & 1) {  // (A, C) <- (bA, bC) o (A, C)
      C = (bA * C + bC) % M;
      A = (bA * A) % M;
    }
    bC = (bA * bC + bC) % M;
    bA = (bA * bA) % M;
    e >>= 1;
  }
  const unsigned long long x = (A * 1ull + C) % M;
  out[i] = (double)x / (double)M;
}

}  // namespace espec

using namespace espec;

#define EIG_CK(call)                                         \
  do {                                                       \
    cudaError_t e_ = (call);                                 \
    if (e_ != cudaSuccess) return set_cuda_error(#call, e_); \
  } while (0)

// 2D coupled Morse family (potfuncs.f:104-108 Morse terms plus a bilinear
// coupling): V = De1 (1 - e^{-a1 (x-re1)})^2 + De2 (1 - e^{-a2 (y-re2)})^2
// + lam (x-re1)(y-re2), params [nprob][5] = (De1, a1, De2, a2, lam)
__global__ void morse2d_kernel(const double* params, int nprob, int nx, int ny, double x0,
                               double hxs, double y0, double hys, double re1, double re2,
                               double* vpot) {
  const long n = (long)nx * ny;
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= n * nprob) return;
  const long p = gid / n, k = gid % n;
  const int i = (int)(k % nx), j = (int)(k / nx);
  const double x = x0 + i * hxs, y = y0 + j * hys;
  const double* q = params + p * 5;
  const double ex = 1.0 - exp(-q[1] * (x - re1)), ey = 1.0 - exp(-q[3] * (y - re2));
  vpot[gid] = q[0] * ex * ex + q[2] * ey * ey + q[4] * (x - re1) * (y - re2);
}

extern "C" int espec_eig_morse2d(int nprob, const double* params, const int* np, double xi,
                                 double xf, double yi, double yf, double re1, double re2,
                                 double* vpot, void* stream) {
  if (nprob <= 0 || !params || !np || !vpot || np[0] < 2 || np[1] < 2)
    return set_error(ESPEC_EINVAL, "bad argument");
  const long tot = (long)np[0] * np[1] * nprob;
  morse2d_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      params, nprob, np[0], np[1], xi, (xf - xi) / (np[0] - 1), yi, (yf - yi) / (np[1] - 1), re1,
      re2, vpot);
  EIG_CK(cudaGetLastError());
  return ESPEC_OK;
}

extern "C" int espec_eig_lcg_start(double* d_out, int n, int nstates, void* stream) {
  // lanczsc.f:56-62: N draws discarded, then N draws per state
  if (!d_out || n <= 0 || nstates <= 0) return set_error(ESPEC_EINVAL, "bad argument");
  const long count = (long)n * nstates;
  lcg_kernel<<<(unsigned)((count + 255) / 256), 256, 0, (cudaStream_t)stream>>>(d_out, count,
                                                                               (long)n + 1);
  EIG_CK(cudaGetLastError());
  return ESPEC_OK;
}

extern "C" int espec_eig_solve_dev(int nprob, const int* np, const double* shm,
                                   const double* vpot, const double* start, int nstates, int m,
                                   double tol, int maxrest, double* vec, double* eval,
                                   double* resid, int* matvecs, double* work_L, double* work_v,
                                   void* stream) {
  if (nprob <= 0 || !np || !shm || !vpot || !start || !vec || !eval || !resid || !matvecs ||
      !work_L || !work_v)
    return set_error(ESPEC_EINVAL, "null argument");
  if (m < 2 || m > kEigMaxM) return set_error(ESPEC_EINVAL, "Lanczos length must be 2..48");
  if (nstates < 1 || nstates > kEigMaxStates) return set_error(ESPEC_EINVAL, "nstates must be 1..16");
  if (np[0] < 1 || np[1] < 1) return set_error(ESPEC_EINVAL, "bad grid");
  EigArgs a{};
  a.nx = np[0];
  a.ny = np[1];
  a.n = np[0] * np[1];
  a.shm[0] = shm[0];
  a.shm[1] = shm[1];
  a.sht30 = 30.0 * (shm[0] + shm[1]);
  a.vpot = vpot;
  a.start = start;
  a.L = work_L;
  a.work = work_v;
  a.vec = vec;
  a.eval = eval;
  a.resid = resid;
  a.matvecs = matvecs;
  a.nstates = nstates;
  a.m = m;
  a.maxrest = maxrest;
  a.tol = tol;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t smem = sizeof(double) * (size_t)a.n, most = sizeof(double) * kEigMaxSmemN;
  int dev = 0, nsm = 0;
  EIG_CK(cudaGetDevice(&dev));
  EIG_CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  if (a.n > kEigMaxSmemN) {
    eig_kernel<false, 1><<<nprob, kEigThreads, 0, st>>>(a);
  } else if (2 * nprob <= nsm && a.n >= kEigMinSplitN) {
    static DeviceFlags attr;
    EIG_CK(set_max_smem_once(attr, eig_kernel<true, 2>, most));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2 * (unsigned)nprob);
    cfg.blockDim = dim3(kEigThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute la{};
    la.id = cudaLaunchAttributeClusterDimension;
    la.val.clusterDim.x = 2;
    la.val.clusterDim.y = la.val.clusterDim.z = 1;
    cfg.attrs = &la;
    cfg.numAttrs = 1;
    EIG_CK(cudaLaunchKernelEx(&cfg, eig_kernel<true, 2>, a));
  } else {
    static DeviceFlags attr;
    EIG_CK(set_max_smem_once(attr, eig_kernel<true, 1>, most));
    eig_kernel<true, 1><<<nprob, kEigThreads, smem, st>>>(a);
  }
  EIG_CK(cudaGetLastError());
  return ESPEC_OK;
}
