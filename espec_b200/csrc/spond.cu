// spond.cu -- split-operator propagation (PSPOFFT / PSPOFFTAUX, pspofft.f,
// spofft.f:64-200) on one 2D or 3D grid, FP64 or mixed (FP32 data, FP64
// tables), and the plan behind espec_spond_* (include/espec_gpu.h).
//
// A run is one cooperative kernel (spond.cuh, nd_kernel) of at most one CTA per
// SM; its passes are separated by grid barriers with a bounded wait.  Passes
// per step, the V half-steps of consecutive steps merged (g = h^2):
//   2D: x pass [inverse x, C(t), x-space phase, forward x]; y pass [forward y,
//       kinetic phase, inverse y]
//   3D: x pass; y pass [forward y]; z pass [forward z, kinetic, inverse z];
//       y pass [inverse y]; or, where an xy plane fits in shared memory, one
//       pass [inverse y, x pass, forward y] over whole planes and the z pass
// Lines are transformed in the registers of 4 to 32 lanes (LineFft); between
// the passes a line stays in the transform's storage order, and only the
// kinetic pass needs the frequencies, via its table (freq_at).  The fftshift
// swaps of spofft.f:120-133/178-191 cancel and are not done; the 1/N of the
// reference's B factor is folded into the kinetic table.
#include <cuda/atomic>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <utility>
#include <vector>

#include "cplx.cuh"
#include "espec_gpu.h"
#include "espec_internal.h"
#include "cplx_io.cuh"
#include "spond.cuh"

namespace espec {
using namespace nd;
namespace {

// SOD tables: vc = CST V, ab = CST VABC or the mask, w = conj(psi0)
__global__ void sod_setup_nd_kernel(long n, const double* vpot, const double* vabc, int kabs,
                                    double cst, const double2* psi0, double* vc, double* ab,
                                    double2* w) {
  const long x = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= n) return;
  vc[x] = cst * vpot[x];
  ab[x] = kabs == 1 ? cst * vabc[x] : (kabs == 2 ? vabc[x] : 0.0);
  w[x] = make_double2(psi0[x].x, -psi0[x].y);
}

// EFFT4 (eigenergfft.f:58-100) and the norm of a natural-order state psi
// given its forward transform khat in the passes' storage order:
// sum V |psi|^2 + (1/N) sum TC |khat|^2 and sum |psi|^2, per-CTA partials
__global__ void nd_energy_kernel(const double2* psi, const double* vpot, const cpx<double>* khat,
                                 const double* tcp, long n, double rn, double2* part) {
  __shared__ double2 red[256];
  double e = 0.0, nr = 0.0;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long)gridDim.x * blockDim.x) {
    const double2 p = psi[i];
    const double a2 = p.x * p.x + p.y * p.y;
    const cpx<double> k = khat[i];
    e += vpot[i] * a2 + rn * tcp[i] * (k.x * k.x + k.y * k.y);
    nr += a2;
  }
  red[threadIdx.x] = make_double2(e, nr);
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      red[threadIdx.x].x += red[threadIdx.x + o].x;
      red[threadIdx.x].y += red[threadIdx.x + o].y;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

// C(t) of each step: the partial sums of the CTAs, a warp per step; NaN where
// a grid barrier of the run gave up
__global__ void csum_kernel(const double2* cpart, int nparts, int nsteps, int first,
                            double2* c_out, const int* err) {
  const int lane = threadIdx.x & 31;
  const int s = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5) + first;
  if (s > nsteps) return;
  double sr = 0.0, si = 0.0;
  for (int i = lane; i < nparts; i += 32) {
    const double2 p = cpart[(long)s * nparts + i];
    sr += p.x;
    si += p.y;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sr += __shfl_xor_sync(kFull, sr, o);
    si += __shfl_xor_sync(kFull, si, o);
  }
  if (*err) sr = si = nan("");
  if (lane == 0) c_out[s] = make_double2(sr, si);
}

// after the energies' transform: (energy, norm) from the CTAs' sums, one warp, and whether
// a wait of the transform or of the last run gave up (bar: arrivals and flags, the run's
// first).  The transform's arrivals and flag go back to zero for the next one.
__global__ void nd_energy_sum_kernel(const double2* part, int nparts, unsigned long long* bar,
                                     double2* out) {
  const int lane = threadIdx.x & 31;
  double e = 0.0, nr = 0.0;
  for (int i = lane; i < nparts; i += 32) {
    e += part[i].x;
    nr += part[i].y;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    e += __shfl_xor_sync(kFull, e, o);
    nr += __shfl_xor_sync(kFull, nr, o);
  }
  if (lane == 0) {
    out[0] = make_double2(e, nr);
    out[1] = make_double2(*(const int*)(bar + 3), *(const int*)(bar + 1));
    bar[2] = bar[3] = 0;
  }
}

// Frequency (FFT order) at place s of an axis's transform.  Positions p of the
// line transform hold frequency brev_P(p / 32) + P brev_32(p % 32), N = 32 P; a
// pass that stores its registers writes position (t << LE) | e at place e L + t
// (coalesced), a fused plane is stored by position.
__host__ __device__ inline int freq_at(int s, int ln, bool by_pos) {
  const int le = ln == 9 ? 4 : 3, lt = ln - le;
  const int p = by_pos ? s : ((s & ((1 << lt) - 1)) << le) | (s >> lt);
  return brev_bits(p >> 5, ln - 5) + (brev_bits(p & 31, 5) << (ln - 5));
}
struct NdLayout {
  int ln[3];
  bool by_pos[3];
};
// index into the reference's FFT-order table of the frequency stored at i,
// mirrored to its FFT sign (fft3d.f: ISN = +1 is exp(+2 pi i jk/n))
__device__ __forceinline__ long tc_index(const NdLayout& l, long i) {
  long idx = 0;
  int shift = 0;
  for (int ax = 0; ax < 3 && l.ln[ax] > 0; ++ax) {
    const int n = 1 << l.ln[ax];
    const int s = (int)(i >> shift) & (n - 1);
    idx += (long)((n - freq_at(s, l.ln[ax], l.by_pos[ax])) & (n - 1)) << shift;
    shift += l.ln[ax];
  }
  return idx;
}
// TC of FFT-order index idx: the sum of the axis tables t (x, y, z one after the
// other), or with `defect` the only TC(1..NP1) that dkeft.f:80-137 fills
__device__ __forceinline__ double tc_value(const NdLayout& l, const double* t, bool defect,
                                           long idx) {
  const long nx = 1L << l.ln[0], ny = 1L << l.ln[1];
  if (defect) return idx < nx ? t[idx] : 0.0;
  double s = t[idx & (nx - 1)] + t[nx + ((idx >> l.ln[0]) & (ny - 1))];
  if (l.ln[2] > 0) s += t[nx + ny + (idx >> (l.ln[0] + l.ln[1]))];
  return s;
}
__device__ __forceinline__ void put_k(cpx<double>* o, double th, double n) {
  double s, c;
  sincos(th, &s, &c);
  *o = mk(c / n, -s / n);
}
__device__ __forceinline__ void put_k(PhF* o, double th, double n) { *o = make_phf(-th, 1.0 / n); }

// kinetic factors in storage order: e^{-i CST1 TC}/N (and cos, sin for the
// reference-defect form), or CST TC/N for second-order differences
template <typename R>
__global__ void nd_kinetic_kernel(NdLayout l, long n, const double* t, bool defect, bool sod,
                                  double cst, typename Ph<R>::type* K, double* kq) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double th = cst * tc_value(l, t, defect, tc_index(l, i));
  if (sod) {  // CST TC B (sodfft.f:100-104,119)
    if constexpr (sizeof(R) == 8) K[i] = mk(th / n, 0.0);
    return;
  }
  put_k(K + i, th, (double)n);
  if (kq) {
    double s, c;
    sincos(th, &s, &c);
    kq[i] = c;
    kq[n + i] = s;
  }
}
__global__ void nd_tc_kernel(NdLayout l, long n, const double* t, bool defect, double* tcp) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) tcp[i] = tc_value(l, t, defect, tc_index(l, i));
}

// x-space tables (spofft.f:120-133, 162-191): h = e^{-i cst2 V} (x e^{cst2
// VABC} for .VOPTIC), g = h^2 (x mask), hm = h mask, w = conj(psi0) hm
__device__ __forceinline__ void put_ph(cpx<double>* o, double phi, double a) {
  double s, c;
  sincos(phi, &s, &c);
  *o = mk(c * a, s * a);
}
__device__ __forceinline__ void put_ph(PhF* o, double phi, double a) { *o = make_phf(phi, a); }

template <typename R>
__global__ void nd_setup_kernel(long n, const double* vpot, const double* vabc, int absorb,
                                double cst2, const double2* psi0, typename Ph<R>::type* g,
                                typename Ph<R>::type* h, typename Ph<R>::type* hm, double2* w) {
  const long x = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= n) return;
  const double th = cst2 * vpot[x];
  double hmag = 1.0, mask = 1.0;
  if (absorb == ESPEC_ABS_VOPTIC) hmag = exp(cst2 * vabc[x]);
  if (absorb == ESPEC_ABS_SMOOTHW) mask = vabc[x];
  double s1, c1, s2, c2;
  sincos(th, &s1, &c1);
  sincos(2.0 * th, &s2, &c2);
  (void)s2;
  (void)c2;
  put_ph(g + x, -2.0 * th, hmag * hmag * mask);
  put_ph(h + x, -th, hmag);
  put_ph(hm + x, -th, hmag * mask);
  const double hr = c1 * hmag * mask, hi = -s1 * hmag * mask;
  const double2 p = psi0[x];
  w[x] = make_double2(p.x * hr + p.y * hi, p.x * hi - p.y * hr);
}

}  // namespace
}  // namespace espec

// ---------------------------------------------------------------------------
// plan
// ---------------------------------------------------------------------------
using namespace espec;

struct espec_spond_plan {
  int ndim = 2, np[3] = {1, 1, 1};
  long n = 0;
  double sh[3] = {1, 1, 1}, sm[3] = {1, 1, 1};
  double dt_fs = 0.0;
  int precision = ESPEC_FP64, absorb = 0, quirks = 0, method = ESPEC_SPO;
  double2* d_prev = nullptr;  // SOD: psi(t - dt), natural order
  double* d_sod = nullptr;    // SOD: vc, ab (n each)
  bool loaded = false;
  void* d_psi = nullptr;      // cpx<R> state
  double2* d_psi0 = nullptr;
  double2* d_out = nullptr;
  double* d_vpot = nullptr;
  double* d_vabc = nullptr;
  void* d_tab = nullptr;      // g, h, hm, w, K (cpx<R>)
  double* d_kq = nullptr;     // quirk cos/sin tables
  double2* d_cpart = nullptr;
  double2* d_c = nullptr;
  void* d_tw[3] = {nullptr, nullptr, nullptr};
  int c_cap = -1;
  int nsm = 0;
  double* d_tax = nullptr;         // DIGT axis tables (or the defect's TC(1..NP1))
  bool k_ready = false;            // the kinetic table is built (it depends on the plan alone)
  // grid barrier arrivals and error flag of the propagation, then of the energies' transform
  unsigned long long* d_bar = nullptr;
  bool has_state = false;          // d_out holds the state of the last run
  // energy diagnostics (FP64 in both forms)
  cpx<double>* d_khat = nullptr;
  double* d_tcp = nullptr;         // TC in the passes' storage order
  RotD* d_tw64[3] = {nullptr, nullptr, nullptr};
  double2* d_epart = nullptr;
  HostStage stage;                 // host transfers: (re | im) blocks, contiguous
};

namespace {

bool line_ok(int n) { return n == 32 || n == 64 || n == 128 || n == 256 || n == 512; }

const double kDigtTwoPi = 6.283185307;  // dkeft.f:38

void digt_axis_host(int n, double sh, double sm, double* t) { espec::digt_1d(n, sh, sm, t); }

// kinetic table TC in the reference's FFT order (x fastest): the outer sum of
// the axis tables, or with ESPEC_Q_DIGT_ND the 2D/3D loops of dkeft.f:80-137
// as they are written (only TC(1..NP1) is filled)
void digt_nd(const espec_spond_plan* p, std::vector<double>& tc) {
  const int nx = p->np[0], ny = p->np[1], nz = p->ndim > 2 ? p->np[2] : 1;
  tc.assign((size_t)p->n, 0.0);
  if (p->quirks & ESPEC_Q_DIGT_ND) {
    double dp[3];
    for (int a = 0; a < p->ndim; ++a) dp[a] = kDigtTwoPi / (p->np[a] * p->sh[a]);
    if (p->ndim == 2) {
      double p1 = 0, p2 = 0;
      for (int j = 0; j < ny / 2; ++j) {
        for (int i = 0; i < nx / 2; ++i) {
          tc[i] = p1 * p1 / (2 * p->sm[0]) + p2 * p2 / (2 * p->sm[1]);
          p1 = p1 + dp[0];
        }
        p2 = p2 + dp[1];
      }
      p1 = -(p1 + dp[0]);
      p2 = -(p2 + dp[1]);
      for (int j = ny / 2; j < ny; ++j) {
        for (int i = nx / 2; i < nx; ++i) {
          tc[i] = p1 * p1 / (2 * p->sm[0]) + p2 * p2 / (2 * p->sm[1]);
          p1 = p1 + dp[0];
        }
        p2 = p2 + dp[1];
      }
    } else {
      double p1 = 0, p2 = 0, p3 = 0;
      for (int k = 0; k < nz / 2; ++k) {
        for (int j = 0; j < ny / 2; ++j) {
          for (int i = 0; i < nx / 2; ++i) {
            tc[i] = p1 * p1 / (2 * p->sm[0]) + p2 * p2 / (2 * p->sm[1]) +
                    p3 * p3 / (2 * p->sm[2]);
            p1 = p1 + dp[0];
          }
          p2 = p2 + dp[1];
        }
        p3 = p3 + dp[2];
      }
      p1 = -(p1 + dp[0]);
      p2 = -(p2 + dp[1]);
      p3 = -(p3 + dp[2]);
      for (int k = nz / 2; k < nz; ++k) {
        for (int j = ny / 2; j < ny; ++j) {
          for (int i = nx / 2; i < nx; ++i) {
            tc[i] = p1 * p1 / (2 * p->sm[0]) + p2 * p2 / (2 * p->sm[1]) +
                    p3 * p3 / (2 * p->sm[2]);
            p1 = p1 + dp[0];
          }
          p2 = p2 + dp[1];
        }
        p3 = p3 + dp[2];
      }
    }
    return;
  }
  std::vector<double> t[3];
  for (int a = 0; a < p->ndim; ++a) {
    t[a].resize(p->np[a]);
    digt_axis_host(p->np[a], p->sh[a], p->sm[a], t[a].data());
  }
  for (int k = 0; k < nz; ++k)
    for (int j = 0; j < ny; ++j)
      for (int i = 0; i < nx; ++i)
        tc[i + (size_t)nx * (j + (size_t)ny * k)] =
            t[0][i] + t[1][j] + (p->ndim > 2 ? t[2][k] : 0.0);
}

#define ND_CK(call)                                          \
  do {                                                       \
    cudaError_t e_ = (call);                                 \
    if (e_ != cudaSuccess) return set_cuda_error(#call, e_); \
  } while (0)

// how a grid's passes are cut
struct NdConfig {
  int threads = 256, grid = 1, lc = 3, fused = 0, kstage = 0;
  size_t smem = 0;
  NdLayout layout{};
};

template <typename R>
size_t packed_bytes(int ln) {
  const size_t b = sizeof(typename Rot<R>::type);
  switch (ln) {
    case 5: return b * LineFft<R, 5>::count() * LineFft<R, 5>::L;
    case 6: return b * LineFft<R, 6>::count() * LineFft<R, 6>::L;
    case 7: return b * LineFft<R, 7>::count() * LineFft<R, 7>::L;
    case 8: return b * LineFft<R, 8>::count() * LineFft<R, 8>::L;
    default: return b * LineFft<R, 9>::count() * LineFft<R, 9>::L;
  }
}

// Threads: 512 where a thread's points, twiddles and preloaded factors fit 128
// registers, else 256 (FP64 lines of 256 and 512 points, FP32 of 512).
// Fused xy planes: where a plane and the copies of its rows' inputs fit in
// shared memory and there are planes for most SMs, or for half of them and a plane
// is one line per group of lanes -- the y passes then cost no memory traffic and no
// grid barrier, but a plane runs on one SM.  Us per step, fused and separate: 128^3
// mixed 57 and 64, 64 x 64 x 256 44 and 49, 64 x 32 x 128 15.1 and 17.8, 32 x 64 x 64
// 14.1 and 14.7; 64^3 18.7 and 16.9, 128 x 64 x 64 mixed 23.0 and 19.7, 64 x 64 x 32 18.2
// and 14.2.  Not with z lines of 512 points, whose CTAs have 256 threads: 32 x 32 x 512
// 45.1 and 38.5 (SOD 69.7 and 51.7), 128 x 32 x 512 120 and 114, 64 x 64 x 512 113 and 114
// (SOD 174 and 169).
// Tiles of the column passes: 8 adjacent columns (128 bytes in FP64), fewer
// where that would leave SMs without a tile.  CTAs: the fewest that keep the
// largest share, at most one per SM.
template <typename R>
NdConfig nd_config(const espec_spond_plan* p) {
  NdConfig c;
  int mx = 0;
  for (int ax = 0; ax < p->ndim; ++ax) {
    int l = 5;
    while ((1 << l) < p->np[ax]) ++l;
    c.layout.ln[ax] = l;
    mx = l > mx ? l : mx;
  }
  const int* ln = c.layout.ln;
  c.threads = mx <= kMaxLn512<R> ? 512 : 256;
  const size_t plane = sizeof(cpx<R>) * (size_t)p->np[0] * p->np[1];
  size_t tw = 0;
  for (int ax = 0; ax < p->ndim; ++ax) tw += packed_bytes<R>(ln[ax]);
  const bool planes = (p->np[2] >= 128 && p->np[2] < 512) ||
                      (p->np[2] >= 64 && p->np[2] < 128 && p->np[0] * p->np[1] <= 2048);
  c.fused = p->ndim == 3 && planes && tw + plane + 65536 <= kNdMaxSmem;
  for (int ax = 0; ax < 2; ++ax) c.layout.by_pos[ax] = c.fused;
  auto threads_of = [&](int ax) { return ln[ax] == 9 ? 5 : ln[ax] - 3; };  // log2, per line
  auto tiles = [&](int lc) {
    long t = p->n >> (ln[p->ndim - 1] + lc);
    if (p->ndim == 3 && !c.fused) t = std::min(t, p->n >> (ln[1] + lc));
    return t;
  };
  int lmin = 5 - threads_of(p->ndim - 1);  // a tile's group is whole warps
  if (p->ndim == 3 && !c.fused) lmin = std::max(lmin, 5 - threads_of(1));
  lmin = std::max(lmin, 1);
  while (c.lc > lmin && tiles(c.lc) < 96) --c.lc;
  const long rows = c.fused ? p->np[2] : (p->n >> ln[0]) >> (5 - threads_of(0));
  long want = std::max(rows, tiles(c.lc));
  if (want > p->nsm) {
    const long per = (want + p->nsm - 1) / p->nsm;
    want = (want + per - 1) / per;
  }
  c.grid = (int)want;
  // a grid that gives 8 warps of a CTA no second line (of the plane, or of the z
  // tiles) keeps 256 threads
  if (c.fused) {
    const long gt = 1L << (threads_of(2) + c.lc);
    if ((long)p->np[0] << threads_of(1) <= 256 && (long)p->np[1] << threads_of(0) <= 256 &&
        tiles(c.lc) * gt <= 256L * c.grid)
      c.threads = 256;  // 64 x 32 x 128: SOD 23.2 -> 18.4 us a step, SPO 18.9 -> 15.2
  } else if ((p->n >> ln[0]) / (32 >> threads_of(0)) <= 8L * c.grid) {
    c.threads = 256;
  }
  const int e = mx == 9 ? 16 : 8;
  size_t ex = sizeof(cpx<R>) * (size_t)c.threads * e * 9 / 8;
  if (c.fused) ex = std::max(ex, plane + (size_t)c.threads / 32 * 4096);
  // the kinetic pass copies tiles ahead where a group has more than one (with
  // one there is nothing to overlap), their rows are whole 16-byte pieces, the
  // buffers fit and a line has 8 points per thread
  const int ka = p->ndim - 1, gt = 1 << (threads_of(ka) + c.lc), groups = c.threads / gt;
  const size_t tile = (sizeof(cpx<R>) + sizeof(typename Ph<R>::type)) * (size_t)p->np[ka] << c.lc;
  const size_t kst = sizeof(cpx<R>) * (size_t)c.threads * 9 + 2 * groups * tile;
  if (ln[ka] <= 8 && c.lc >= 2 && !(p->quirks & ESPEC_Q_SPO_INPLACE) &&
      tiles(c.lc) > (long)c.grid * groups && tw + kst <= kNdMaxSmem) {
    c.kstage = 1;
    ex = std::max(ex, kst);
  }
  c.smem = tw + ex;
  return c;
}

// DIGT's axis tables x, y, z, or with ESPEC_Q_DIGT_ND the TC(1..NP1) it fills
int upload_axis_tables(espec_spond_plan* p, cudaStream_t st) {
  std::vector<double> t;
  if (p->quirks & ESPEC_Q_DIGT_ND) {
    digt_nd(p, t);
    t.resize(p->np[0]);
  } else {
    size_t o = 0;
    for (int ax = 0; ax < p->ndim; ++ax) {
      t.resize(o + p->np[ax]);
      digt_axis_host(p->np[ax], p->sh[ax], p->sm[ax], t.data() + o);
      o += p->np[ax];
    }
  }
  ND_CK(cudaMemcpyAsync(p->d_tax, t.data(), 8 * t.size(), cudaMemcpyHostToDevice, st));
  ND_CK(cudaStreamSynchronize(st));  // the host vector goes out of scope
  return ESPEC_OK;
}

// table block: g, h, hm (PhT) | w (double2) | K (PhT), n entries each
template <typename R>
struct NdTabs {
  using PhT = typename Ph<R>::type;
  PhT *g, *h, *hm, *K;
  double2* w;
  static size_t bytes(long n) { return (size_t)n * (4 * sizeof(PhT) + sizeof(double2)); }
  NdTabs(void* base, long n) {
    char* b = (char*)base;
    w = (double2*)b;
    g = (PhT*)(b + 16 * (size_t)n);
    h = g + n;
    hm = h + n;
    K = hm + n;
  }
};

inline int sod_kabs(const espec_spond_plan* p) {
  if (p->absorb == ESPEC_ABS_VOPTIC) return 1;
  if (p->absorb == ESPEC_ABS_SMOOTHW && !(p->quirks & ESPEC_Q_SOD_SMOOTHW)) return 2;
  return 0;  // sodfft.f:108 compares 7 characters with '.SMOOTHW': never true
}

template <typename R>
int build_tables(espec_spond_plan* p, cudaStream_t st) {
  const long n = p->n;
  NdTabs<R> tb(p->d_tab, n);
  const double cst1 = p->dt_fs / ESPEC_SHFS, cst2 = p->dt_fs / (2.0 * ESPEC_SHFS);
  const bool sod = p->method == ESPEC_SOD;
  const double cst_sod = 2.0 * p->dt_fs / ESPEC_SHFS;  // psodfft.f:81
  if (sod) {
    sod_setup_nd_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
        n, p->d_vpot, p->d_vabc, sod_kabs(p), cst_sod, p->d_psi0, p->d_sod, p->d_sod + n, tb.w);
  } else {
    nd_setup_kernel<R><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
        n, p->d_vpot, p->d_vabc, p->absorb, cst2, p->d_psi0, tb.g, tb.h, tb.hm, tb.w);
  }
  ND_CK(cudaGetLastError());
  if (!p->k_ready) {
    const NdConfig cf = nd_config<R>(p);
    const bool defect = (p->quirks & ESPEC_Q_DIGT_ND) != 0;
    const int rc = upload_axis_tables(p, st);
    if (rc) return rc;
    nd_kinetic_kernel<R><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
        cf.layout, n, p->d_tax, defect, sod, sod ? cst_sod : cst1, tb.K, p->d_kq);
    ND_CK(cudaGetLastError());
    for (int ax = 0; ax < p->ndim; ++ax) {
      const int nl = p->np[ax];
      tw_table_kernel<R><<<(nl + 255) / 256, 256, 0, st>>>((typename Rot<R>::type*)p->d_tw[ax], nl);
      ND_CK(cudaGetLastError());
    }
    p->k_ready = true;
  }
  // a caller may reuse its arrays, and load on another stream next
  ND_CK(cudaStreamSynchronize(st));
  return ESPEC_OK;
}

template <typename R>
NdArgs<R> nd_args(const espec_spond_plan* p, const NdConfig& c) {
  NdArgs<R> a{};
  for (int ax = 0; ax < 3; ++ax) a.ln[ax] = c.layout.ln[ax];
  a.ndim = p->ndim;
  a.n = p->n;
  a.fused = c.fused;
  a.lc = c.lc;
  a.kstage = c.kstage;
  a.psi0 = p->d_psi0;
  a.bar = p->d_bar;
  a.spin_limit = grid_wait_limit();
  return a;
}

template <typename R>
int nd_launch(espec_spond_plan* p, const NdConfig& c, NdArgs<R>& a, cudaStream_t st) {
  a.err = (int*)(a.bar + 1);
  // the arrival count, and the error flag unless the run continues from a state that
  // an earlier one may have spoiled; those of the energies' transform are left at zero
  // by nd_energy_sum_kernel
  const size_t word = sizeof(unsigned long long);
  if (a.op != kOpForward) ND_CK(cudaMemsetAsync(a.bar, 0, a.from_start ? 2 * word : word, st));
  if (grid_short_start()) ND_CK(cudaMemsetAsync(a.bar, 0xFF, word, st));
  cudaError_t e;
  if constexpr (sizeof(R) == 8)
    e = c.threads == 256 ? nd_launch_f64_256(a, c.grid, c.smem, st)
                         : nd_launch_f64_512(a, c.grid, c.smem, st);
  else
    e = c.threads == 256 ? nd_launch_f32_256(a, c.grid, c.smem, st)
                         : nd_launch_f32_512(a, c.grid, c.smem, st);
  ND_CK(e);
  return ESPEC_OK;
}

template <typename R>
int run_steps(espec_spond_plan* p, int nsteps, bool from_start, cudaStream_t st) {
  const NdConfig c = nd_config<R>(p);
  NdArgs<R> a = nd_args<R>(p, c);
  const long n = p->n;
  NdTabs<R> tb(p->d_tab, n);
  a.op = kOpSpo;
  a.nsteps = nsteps;
  a.from_start = from_start;
  a.psi = (cpx<R>*)p->d_psi;
  a.psi_out = p->d_out;
  a.psi_start = from_start ? p->d_psi0 : p->d_out;
  a.g = tb.g;
  a.h = tb.h;
  a.hm = tb.hm;
  a.w = tb.w;
  a.K = tb.K;
  a.kq_c = p->d_kq;
  a.kq_s = p->d_kq ? p->d_kq + n : nullptr;
  a.kq_scale = 1.0 / (double)n;
  a.cpart = p->d_cpart;
  for (int ax = 0; ax < p->ndim; ++ax) a.tw[ax] = (const typename Rot<R>::type*)p->d_tw[ax];
  if (nsteps == 0)  // psi(TF) = psi(0)
    ND_CK(cudaMemcpyAsync(p->d_out, p->d_psi0, 16 * n, cudaMemcpyDeviceToDevice, st));
  return nd_launch<R>(p, c, a, st);
}

// second-order differences on the grid (psodfft.f:77-206): start-up of two
// half steps from psi0 (psodfft.f:120-152), then leapfrog steps; the newest
// state ends in d_out, the one before in d_prev
int run_sod(espec_spond_plan* p, int nsteps, bool from_start, cudaStream_t st) {
  const NdConfig c = nd_config<double>(p);
  NdArgs<double> a = nd_args<double>(p, c);
  const long n = p->n;
  NdTabs<double> tb(p->d_tab, n);
  a.op = kOpSod;
  a.nsteps = nsteps;
  a.from_start = from_start;
  a.psi = (cpx<double>*)p->d_psi;  // transform scratch
  a.psi_start = from_start ? p->d_psi0 : p->d_out;
  a.cur = p->d_out;
  a.prev = p->d_prev;
  a.w = tb.w;
  a.K = tb.K;
  a.vc = p->d_sod;
  a.ab = p->d_sod + n;
  a.kabs = sod_kabs(p);
  a.cpart = p->d_cpart;
  for (int ax = 0; ax < p->ndim; ++ax) a.tw[ax] = (const RotD*)p->d_tw[ax];
  if (from_start && nsteps == 0) {
    ND_CK(cudaMemcpyAsync(p->d_out, p->d_psi0, 16 * n, cudaMemcpyDeviceToDevice, st));
    ND_CK(cudaMemcpyAsync(p->d_prev, p->d_psi0, 16 * n, cudaMemcpyDeviceToDevice, st));
  }
  const int rc = nd_launch<double>(p, c, a, st);
  if (rc) return rc;
  if (from_start && nsteps == 1)  // the start-up's half-step state is no psi(t - dt)
    ND_CK(cudaMemcpyAsync(p->d_prev, p->d_psi0, 16 * n, cudaMemcpyDeviceToDevice, st));
  // update u writes d_prev for even u, d_out for odd u
  const int updates = nsteps + (from_start && nsteps > 0 ? 1 : 0);
  if (updates % 2 == 1) std::swap(p->d_out, p->d_prev);
  return ESPEC_OK;
}

}  // namespace

namespace espec {
// the N-D kinetic table (TC) in the reference's FFT order, for the drop-ins
void digt_nd_table(int ndim, const int* np, const double* sh, const double* sm, int quirks,
                   double* tc) {
  espec_spond_plan q;
  q.ndim = ndim;
  q.n = 1;
  for (int a = 0; a < ndim; ++a) {
    q.np[a] = np[a];
    q.sh[a] = sh[a];
    q.sm[a] = sm[a];
    q.n *= np[a];
  }
  q.quirks = quirks;
  std::vector<double> t;
  digt_nd(&q, t);
  for (long i = 0; i < q.n; ++i) tc[i] = t[i];
}
}  // namespace espec

extern "C" int espec_spond_create_method(espec_spond_plan** out, int method, int ndim,
                                         const int* np, const double* sh, const double* sm,
                                         double dt_fs, int precision, int absorb, int quirks) {
  if (!out || !np || !sh || !sm) return set_error(ESPEC_EINVAL, "null argument");
  if (method != ESPEC_SPO && method != ESPEC_SOD)
    return set_error(ESPEC_EINVAL, "method must be ESPEC_SPO or ESPEC_SOD");
  if (method == ESPEC_SOD && precision != ESPEC_FP64)
    return set_error(ESPEC_EINVAL, "the SOD propagator runs in FP64");
  const int allowed = method == ESPEC_SOD ? (ESPEC_Q_SOD_SMOOTHW | ESPEC_Q_DIGT_ND)
                                          : (ESPEC_Q_SPO_INPLACE | ESPEC_Q_DIGT_ND);
  if (quirks & ~allowed) return set_error(ESPEC_EINVAL, "quirk not applicable to this method");
  if (ndim != 2 && ndim != 3) return set_error(ESPEC_EINVAL, "ndim must be 2 or 3");
  for (int a = 0; a < ndim; ++a)
    if (!line_ok(np[a]))
      return set_error(ESPEC_EINVAL, "axis sizes must be 32, 64, 128, 256 or 512");
  if (precision != ESPEC_FP64 && precision != ESPEC_MIXED)
    return set_error(ESPEC_EINVAL, "precision must be ESPEC_FP64 or ESPEC_MIXED");
  if (absorb < ESPEC_ABS_NONE || absorb > ESPEC_ABS_SMOOTHW)
    return set_error(ESPEC_EINVAL, "unknown absorber type");
  if ((quirks & ESPEC_Q_SPO_INPLACE) && precision != ESPEC_FP64)
    return set_error(ESPEC_EINVAL, "the reference-defect mode exists for FP64 only");
  auto* p = new espec_spond_plan;
  p->method = method;
  p->ndim = ndim;
  p->n = 1;
  for (int a = 0; a < ndim; ++a) {
    p->np[a] = np[a];
    p->sh[a] = sh[a];
    p->sm[a] = sm[a];
    p->n *= np[a];
  }
  p->dt_fs = dt_fs;
  p->precision = precision;
  p->absorb = absorb;
  p->quirks = quirks;
  int dev = 0;
  cudaError_t de = cudaGetDevice(&dev);
  if (de == cudaSuccess) de = cudaDeviceGetAttribute(&p->nsm, cudaDevAttrMultiProcessorCount, dev);
  if (de != cudaSuccess) {
    delete p;
    return set_cuda_error("device query", de);
  }
  const size_t n = (size_t)p->n;
  const size_t cb = precision == ESPEC_FP64 ? 16 : 8;
  int rc = 0;
  auto fail = [&](int code) {
    void* b[] = {p->d_psi,   p->d_psi0,  p->d_out,   p->d_vpot,  p->d_vabc, p->d_tab,
                 p->d_kq,    p->d_cpart, p->d_c,     p->d_tw[0], p->d_tw[1], p->d_tw[2],
                 p->d_prev,  p->d_sod,   p->d_tax,   p->d_bar};
    for (void* x : b)
      if (x) cudaFree(x);
    delete p;
    return code;
  };
  if ((rc = ck(cudaMalloc(&p->d_psi, cb * n), "cudaMalloc"))) return fail(rc);
  if ((rc = ck(cudaMalloc(&p->d_psi0, 16 * n), "cudaMalloc"))) return fail(rc);
  if ((rc = ck(cudaMalloc(&p->d_out, 16 * n), "cudaMalloc"))) return fail(rc);
  if ((rc = ck(cudaMalloc(&p->d_vpot, 8 * n), "cudaMalloc"))) return fail(rc);
  if ((rc = ck(cudaMalloc(&p->d_vabc, 8 * n), "cudaMalloc"))) return fail(rc);
  const size_t tbytes = precision == ESPEC_FP64 ? NdTabs<double>::bytes((long)n)
                                                : NdTabs<float>::bytes((long)n);
  if ((rc = ck(cudaMalloc(&p->d_tab, tbytes), "cudaMalloc"))) return fail(rc);
  if (quirks & ESPEC_Q_SPO_INPLACE)
    if ((rc = ck(cudaMalloc(&p->d_kq, 16 * n), "cudaMalloc"))) return fail(rc);
  if (method == ESPEC_SOD) {
    if ((rc = ck(cudaMalloc(&p->d_prev, 16 * n), "cudaMalloc"))) return fail(rc);
    if ((rc = ck(cudaMalloc(&p->d_sod, 16 * n), "cudaMalloc"))) return fail(rc);
  }
  size_t tax = 0;
  for (int ax = 0; ax < ndim; ++ax) tax += np[ax];
  if ((rc = ck(cudaMalloc(&p->d_tax, 8 * tax), "cudaMalloc"))) return fail(rc);
  if ((rc = ck(cudaMalloc(&p->d_bar, 4 * sizeof(unsigned long long)), "cudaMalloc"))) return fail(rc);
  if ((rc = ck(cudaMemset(p->d_bar, 0, 4 * sizeof(unsigned long long)), "cudaMemset")))
    return fail(rc);
  for (int ax = 0; ax < ndim; ++ax)
    if ((rc = ck(cudaMalloc(&p->d_tw[ax], sizeof(RotD) * np[ax]), "cudaMalloc"))) return fail(rc);
  *out = p;
  return ESPEC_OK;
}

extern "C" int espec_spond_create(espec_spond_plan** out, int ndim, const int* np,
                                  const double* sh, const double* sm, double dt_fs,
                                  int precision, int absorb, int quirks) {
  return espec_spond_create_method(out, ESPEC_SPO, ndim, np, sh, sm, dt_fs, precision, absorb,
                                   quirks);
}

static const char* const kTimedOut = "a grid barrier of the split-operator kernel timed out";

// results in host memory: complete, or the last run's wait gave up
static int nd_finish(espec_spond_plan* p, cudaStream_t st) {
  int err = 0;
  ND_CK(cudaMemcpyAsync(&err, p->d_bar + 1, sizeof(int), cudaMemcpyDeviceToHost, st));
  ND_CK(cudaStreamSynchronize(st));
  p->stage.flush();
  return err ? set_error(ESPEC_ECUDA, kTimedOut) : ESPEC_OK;
}

extern "C" int espec_spond_previous(espec_spond_plan* p, double* psi_re, double* psi_im,
                                    int where, void* stream) {
  if (!p || p->method != ESPEC_SOD || !p->has_state)
    return set_error(ESPEC_EINVAL, "previous state exists for run SOD plans only");
  if (where & ESPEC_MEM_INTERLEAVED) return set_error(ESPEC_EINVAL, kPreviousParts);
  cudaStream_t st = (cudaStream_t)stream;
  p->stage.drop();
  const int rc = get_complex(p->stage, p->d_prev, psi_re, psi_im, (size_t)p->n, where, st);
  if (rc) return rc;
  if (where == ESPEC_MEM_HOST) return nd_finish(p, st);
  return ESPEC_OK;
}

extern "C" int espec_spond_load(espec_spond_plan* p, const double* vpot, const double* vabc,
                                const double* psi_re, const double* psi_im, int where,
                                void* stream) {
  if (!p || !vpot || !psi_re) return set_error(ESPEC_EINVAL, "null argument");
  if (p->absorb != ESPEC_ABS_NONE && !vabc) return set_error(ESPEC_EINVAL, "absorber table missing");
  cudaStream_t st = (cudaStream_t)stream;
  const size_t n = (size_t)p->n;
  const bool pairs = (where & ESPEC_MEM_INTERLEAVED) != 0;
  where &= ~ESPEC_MEM_INTERLEAVED;
  const cudaMemcpyKind kind =
      where == ESPEC_MEM_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
  ND_CK(cudaMemcpyAsync(p->d_vpot, vpot, 8 * n, kind, st));
  if (p->absorb != ESPEC_ABS_NONE) ND_CK(cudaMemcpyAsync(p->d_vabc, vabc, 8 * n, kind, st));
  const int rp = pairs ? put_pairs(p->d_psi0, psi_re, n, where, st)
                       : put_complex(p->stage, p->d_psi0, psi_re, psi_im, n, where, st);
  if (rp) return rp;
  const int rc = p->precision == ESPEC_FP64 ? build_tables<double>(p, st)
                                            : build_tables<float>(p, st);
  if (rc) return rc;
  p->has_state = false;
  p->loaded = true;
  return ESPEC_OK;
}

static int nd_grid(const espec_spond_plan* p) {
  return p->precision == ESPEC_FP64 ? nd_config<double>(p).grid : nd_config<float>(p).grid;
}

extern "C" int espec_spond_run(espec_spond_plan* p, int nsteps, void* stream) {
  if (!p || nsteps < 0) return set_error(ESPEC_EINVAL, "bad plan or step count");
  if (!p->loaded) return set_error(ESPEC_EINVAL, "espec_spond_load has not been called");
  cudaStream_t st = (cudaStream_t)stream;
  if (p->c_cap != nsteps) {
    if (p->d_c) cudaFree(p->d_c);
    if (p->d_cpart) cudaFree(p->d_cpart);
    p->d_c = nullptr;
    p->d_cpart = nullptr;
    ND_CK(cudaMalloc(&p->d_c, sizeof(double2) * ((size_t)nsteps + 1)));
    ND_CK(cudaMalloc(&p->d_cpart, sizeof(double2) * ((size_t)nsteps + 1) * nd_grid(p)));
    p->c_cap = nsteps;
  }
  const int rc = p->method == ESPEC_SOD
                     ? run_sod(p, nsteps, true, st)
                     : (p->precision == ESPEC_FP64 ? run_steps<double>(p, nsteps, true, st)
                                                   : run_steps<float>(p, nsteps, true, st));
  if (rc) return rc;
  csum_kernel<<<(nsteps + 1 + 7) / 8, 256, 0, st>>>(p->d_cpart, nd_grid(p), nsteps, 0, p->d_c,
                                                     (const int*)(p->d_bar + 1));
  ND_CK(cudaGetLastError());
  p->has_state = true;
  return ESPEC_OK;
}

extern "C" int espec_spond_continue(espec_spond_plan* p, int nsteps, void* stream) {
  if (!p || nsteps < 0) return set_error(ESPEC_EINVAL, "bad plan or step count");
  if (!p->has_state) return set_error(ESPEC_EINVAL, "continue needs a previous run");
  cudaStream_t st = (cudaStream_t)stream;
  if (p->c_cap != nsteps) {
    if (p->d_c) cudaFree(p->d_c);
    if (p->d_cpart) cudaFree(p->d_cpart);
    p->d_c = nullptr;
    p->d_cpart = nullptr;
    ND_CK(cudaMalloc(&p->d_c, sizeof(double2) * ((size_t)nsteps + 1)));
    ND_CK(cudaMalloc(&p->d_cpart, sizeof(double2) * ((size_t)nsteps + 1) * nd_grid(p)));
    p->c_cap = nsteps;
  }
  if (nsteps == 0) return ESPEC_OK;
  const int rc = p->method == ESPEC_SOD
                     ? run_sod(p, nsteps, false, st)
                     : (p->precision == ESPEC_FP64 ? run_steps<double>(p, nsteps, false, st)
                                                   : run_steps<float>(p, nsteps, false, st));
  if (rc) return rc;
  csum_kernel<<<(nsteps + 7) / 8, 256, 0, st>>>(p->d_cpart, nd_grid(p), nsteps, 1, p->d_c,
                                                 (const int*)(p->d_bar + 1));
  ND_CK(cudaGetLastError());
  return ESPEC_OK;
}

extern "C" int espec_spond_energies(espec_spond_plan* p, double* e, double* norm, void* stream) {
  if (!p || !e || !norm) return set_error(ESPEC_EINVAL, "null argument");
  if (!p->loaded) return set_error(ESPEC_EINVAL, "espec_spond_load has not been called");
  cudaStream_t st = (cudaStream_t)stream;
  const long n = p->n;
  const int nb = 256;
  if (!p->d_khat) {
    ND_CK(cudaMalloc(&p->d_khat, sizeof(cpx<double>) * n));
    ND_CK(cudaMalloc(&p->d_tcp, 8 * n));
    ND_CK(cudaMalloc(&p->d_epart, sizeof(double2) * (nb + 2)));
    for (int ax = 0; ax < p->ndim; ++ax) {
      ND_CK(cudaMalloc(&p->d_tw64[ax], sizeof(RotD) * p->np[ax]));
      tw_table_kernel<double><<<(p->np[ax] + 255) / 256, 256, 0, st>>>(p->d_tw64[ax], p->np[ax]);
      ND_CK(cudaGetLastError());
    }
    const int rc = upload_axis_tables(p, st);
    if (rc) return rc;
    // TC in the storage order of the FP64 transform
    nd_tc_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
        nd_config<double>(p).layout, n, p->d_tax, (p->quirks & ESPEC_Q_DIGT_ND) != 0, p->d_tcp);
    ND_CK(cudaGetLastError());
    ND_CK(cudaStreamSynchronize(st));  // later calls may come on other streams
  }
  const NdConfig c = nd_config<double>(p);
  NdArgs<double> a = nd_args<double>(p, c);
  a.op = kOpForward;
  a.bar = p->d_bar + 2;
  a.psi = p->d_khat;
  a.psi_start = p->has_state ? p->d_out : p->d_psi0;
  for (int ax = 0; ax < p->ndim; ++ax) a.tw[ax] = p->d_tw64[ax];
  const int rl = nd_launch<double>(p, c, a, st);
  if (rl) return rl;
  nd_energy_kernel<<<nb, 256, 0, st>>>(a.psi_start, p->d_vpot, p->d_khat, p->d_tcp, n,
                                       1.0 / (double)n, p->d_epart);
  // the sums go straight into page-locked memory where the plan has some
  p->stage.drop();
  double2* hd = (double2*)p->stage.small(2 * sizeof(double2));
  p->stage.drop();
  nd_energy_sum_kernel<<<1, 32, 0, st>>>(p->d_epart, nb, p->d_bar, hd ? hd : p->d_epart + nb);
  ND_CK(cudaGetLastError());
  double2 h[2];
  if (!hd) {
    ND_CK(cudaMemcpyAsync(h, p->d_epart + nb, sizeof h, cudaMemcpyDeviceToHost, st));
    hd = h;
  }
  ND_CK(cudaStreamSynchronize(st));
  if (hd[1].x != 0.0 || (p->has_state && hd[1].y != 0.0))
    return set_error(ESPEC_ECUDA, kTimedOut);
  *e = hd[0].x;
  *norm = hd[0].y;
  return ESPEC_OK;
}

extern "C" int espec_spond_results(espec_spond_plan* p, double* c_re, double* c_im,
                                   double* psi_re, double* psi_im, int where, void* stream) {
  if (!p || p->c_cap < 0) return set_error(ESPEC_EINVAL, "no results: run the plan first");
  cudaStream_t st = (cudaStream_t)stream;
  const size_t nc = (size_t)p->c_cap + 1, n = (size_t)p->n;
  const bool pairs = (where & ESPEC_MEM_INTERLEAVED) != 0;
  where &= ~ESPEC_MEM_INTERLEAVED;
  p->stage.drop();
  int rc = pairs ? get_pairs(p->d_c, c_re, nc, where, st)
                 : get_complex(p->stage, p->d_c, c_re, c_im, nc, where, st);
  if (rc == ESPEC_OK)
    rc = pairs ? get_pairs(p->d_out, psi_re, n, where, st)
               : get_complex(p->stage, p->d_out, psi_re, psi_im, n, where, st);
  if (rc) return rc;
  if (where == ESPEC_MEM_HOST) return nd_finish(p, st);
  return ESPEC_OK;
}

extern "C" void espec_spond_destroy(espec_spond_plan* p) {
  if (!p) return;
  void* b[] = {p->d_psi,    p->d_psi0,  p->d_out,   p->d_vpot,  p->d_vabc,   p->d_tab,
               p->d_kq,     p->d_cpart, p->d_c,     p->d_tw[0], p->d_tw[1],  p->d_tw[2],
               p->d_khat,   p->d_tcp,   p->d_epart, p->d_tw64[0], p->d_tw64[1], p->d_tw64[2],
               p->d_prev,   p->d_sod,   p->d_tax,    p->d_bar};
  for (void* x : b)
    if (x) cudaFree(x);
  p->stage.release();
  delete p;
}
