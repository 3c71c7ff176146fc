// spectrum.cu -- the spectrum stage of eSPec on the GPU, FP64, batched over
// packets: total correlation assembly (espec.f:1545-1576), lifetime
// broadening HWHM (hwhm.f:59-77), window and half swap of SPECTRUMTD
// (spectrumtd.f:58-81), applied as the inverse DFT of FFTNT (cfft.f:6-106)
// reads its input; the DFT as radix-2 Stockham passes (natural order in and
// out) taken four at a time in registers, whole transforms in shared memory up
// to 2^13 points.
// Also the Fortran drop-ins hwhm_ and spectrumtd_ (with the printed table).
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

#include "espec_gpu.h"
#include "espec_internal.h"

namespace espec {
namespace {

constexpr double kHwhmScale = 1.5192676;           // hwhm.f:60-61
constexpr double kEnc = 1.519829846003e-1;         // spectrumtd.f:58
constexpr double kFate = 27.2113834;               // eV per hartree (spectrumtd.f)
constexpr double kTwoPi = 6.283185307179586476925287;

struct PrepArgs {
  int npk, mf;
  long ldc;               // stride of C(t) samples per packet (assemble) / of input (2^mf)
  const double2* in;      // C(t) samples (assemble) or the time signal
  int assemble;
  double dtf, tf;
  int hwhm;               // apply HWHM
  double dem, ta;         // -DE*1.5192676, TAL*1.5192676
  int window;             // 1: .SG
  double taux;            // TMAX^2 / ln(1/WP)^2
  const double2* factor;  // HWHM and window factor of each time, or null (neither)
  double2* out;           // [npk][2^mf]
};

// HWHM (hwhm.f:63-73) and window (spectrumtd.f:62-68) of time j as one complex
// factor: every packet has the same times, so the sine, cosine and exponentials
// are taken once per call and not once per packet (a third of the prep time)
__device__ __forceinline__ double2 time_factor(const PrepArgs& a, long j) {
  const double t = -a.tf + (double)j * a.dtf;
  double sn = 0.0, cs = 1.0, f = 1.0;
  if (a.hwhm) {
    sincos(a.dem * t, &sn, &cs);
    f = exp(-fabs(t) * a.ta);
  }
  if (a.window) f *= exp(-(t * t) / a.taux);
  return make_double2(cs * f, sn * f);
}

// element i of the transform's input for packet p: the half swap of
// spectrumtd.f:73-80 puts time j = i + N/2 (mod N) there; assembled
// (espec.f:1549-1563: C(-t) = C(t)* mirrored onto 2 MC points, MC = N/2) or
// read, times the factor of its time
__device__ __forceinline__ double2 prep_value(const PrepArgs& a, long p, long i) {
  const long N = 1L << a.mf, mc = N / 2;
  const long j = i < mc ? i + mc : i - mc;  // N = 1: 0
  double2 z;
  if (a.assemble && N > 1) {
    const double2* c = a.in + p * a.ldc;
    if (j > mc) {
      z = __ldg(c + (j - mc));
    } else {
      z = __ldg(c + (j == 0 ? mc - 1 : mc - j));
      z.y = -z.y;
    }
  } else {
    z = __ldg(a.in + p * a.ldc + j);
  }
  if (a.factor) {
    const double2 f = __ldg(a.factor + j);
    z = make_double2(f.x * z.x - f.y * z.y, f.x * z.y + f.y * z.x);
  }
  return z;
}

// twiddles w_k = exp(+i twopi k / N), k < N/2 (the backward sign of FFTNT), those
// of each earlier pass s gathered where its threads read them (2^s values from
// 2^s - 1 on), and, when asked for, the factor of every time
struct Twiddles {
  const double2* w;     // w_k, k < N/2: the last pass's values
  const double2* pass;  // the earlier passes' values, or null (no room): w by stride
};
__global__ void spec_table_kernel(PrepArgs a, double2* tw, double2* pass, double2* factor,
                                  double twopi_over_n) {
  const long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long N = 1L << a.mf;
  if (k < N / 2) {
    double s, c;
    sincos(twopi_over_n * (double)k, &s, &c);
    tw[k] = make_double2(c, s);
    if (pass)  // k = q 2^(mf-1-s) is value q of pass s
      for (int s2 = a.mf - 2; s2 >= 0 && (k & ((1L << (a.mf - 1 - s2)) - 1)) == 0; --s2)
        pass[(1L << s2) - 1 + (k >> (a.mf - 1 - s2))] = make_double2(c, s);
  }
  if (factor && k < N) factor[k] = time_factor(a, k);
}

// HWHM and window alone, natural order (hwhm_)
__global__ void spec_hwhm_kernel(PrepArgs a) {
  const long j = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= (1L << a.mf)) return;
  const double2 z = a.in[j], f = time_factor(a, j);
  a.out[j] = make_double2(f.x * z.x - f.y * z.y, f.x * z.y + f.y * z.x);
}

// LOGR consecutive radix-2 Stockham passes s, s+1, ... on the 2^LOGR points
// that meet in them, in registers.  Pass s takes elements j and j + N/2 to
// ((j >> s) << (s + 1)) | k and that + 2^s (k = j mod 2^s), so the points
// j0 + q N / 2^LOGR (j0 < N / 2^LOGR) stay together through LOGR passes: a
// block of the array per output bit found so far, halved by every pass, the
// block's bits reversed extending k.  On return element r belongs at
// (j0 - k) 2^LOGR + k + 2^s brev(r).  The twiddles are the table's for each
// pass, so that FFTNT's single-precision 2 pi enters as it does in the
// reference's radix-2 form.
__host__ __device__ constexpr int brev_c(int v, int bits) {
  int r = 0;
  for (int i = 0; i < bits; ++i) r |= ((v >> i) & 1) << (bits - 1 - i);
  return r;
}
template <int LOGR>
__device__ __forceinline__ void passes(double2* v, const Twiddles& tw, long k, int s, int mf) {
  constexpr int R = 1 << LOGR;
#pragma unroll
  for (int p = 0; p < LOGR; ++p) {
    const int half = R >> (p + 1);
#pragma unroll
    for (int blk = 0; blk < (1 << p); ++blk) {
      const long q0 = k + ((long)brev_c(blk, p) << s);
      const double2 w = __ldg(tw.pass && s + p < mf - 1 ? tw.pass + ((1L << (s + p)) - 1 + q0)
                                                        : tw.w + (q0 << (mf - 1 - s - p)));
#pragma unroll
      for (int q = 0; q < half; ++q) {
        double2& x = v[blk * 2 * half + q];
        double2& y = v[blk * 2 * half + q + half];
        const double2 b = make_double2(y.x * w.x - y.y * w.y, y.x * w.y + y.y * w.x);
        y = make_double2(x.x - b.x, x.y - b.y);
        x = make_double2(x.x + b.x, x.y + b.y);
      }
    }
  }
}

// Transforms of 2^mf points, 4 <= mf <= kOneMax, whole in shared memory: 8
// points per thread, the passes taken three at a time in registers (REM of them,
// the remainder, first), one exchange through shared memory between the groups; the
// input is prepared as it is read and the last group writes the result.
// Small transforms share a CTA.  The exchange adds one element in 8, which
// keeps the stride-8 writes of the first groups on distinct banks.
// HBM then carries the samples once and the spectrum once; with one kernel per
// radix-2 pass every pass moved the whole batch (1024 x 4096 points: 12 passes
// of 134 MB and a prep pass, 295 us).  What is left is latency: 32 warps per SM
// take 64 us; with 16 points per thread and four passes at a time, one exchange
// less but 16 warps, it was 70 us.
constexpr int kOneMax = 13;
constexpr int kOneLog = 3, kOneP = 1 << kOneLog;  // points per thread
constexpr int kOneThreads = 512;
__host__ __device__ __forceinline__ constexpr int padded(int i) { return i + (i >> kOneLog); }

template <int REM, int T>
__global__ void __launch_bounds__(T, 1024 / T) spec_one_kernel(PrepArgs a, Twiddles tw,
                                                                      double scale) {
  extern __shared__ double2 spec_sm[];
  const int mf = a.mf, n = 1 << mf, tp = n >> kOneLog;  // threads of a packet
  const int g = threadIdx.x / tp, t = threadIdx.x % tp;
  const long p = (long)blockIdx.x * (T / tp) + g;
  const bool on = p < a.npk;
  double2* sm = spec_sm + (size_t)g * padded(n);
  double2 v[kOneP];
  constexpr int R = 1 << REM, B = kOneP / R;  // B groups of 2^REM points, k = 0
#pragma unroll
  for (int i = 0; i < B; ++i) {
    const int j0 = t + i * tp;
#pragma unroll
    for (int q = 0; q < R; ++q)
      v[i * R + q] = on ? prep_value(a, p, j0 + q * (n / R)) : make_double2(0.0, 0.0);
  }
#pragma unroll
  for (int i = 0; i < B; ++i) {
    passes<REM>(v + i * R, tw, 0, 0, mf);
    const int j0 = t + i * tp;
#pragma unroll
    for (int r = 0; r < R; ++r) sm[padded(j0 * R + brev_c(r, REM))] = v[i * R + r];
  }
  __syncthreads();
  for (int s = REM; s < mf; s += kOneLog) {
    const int k = t & ((1 << s) - 1);
#pragma unroll
    for (int q = 0; q < kOneP; ++q) v[q] = sm[padded(t + q * tp)];
    passes<kOneLog>(v, tw, k, s, mf);
    const int o = (t - k) * kOneP + k;
    if (s + kOneLog < mf) {
      __syncthreads();
#pragma unroll
      for (int r = 0; r < kOneP; ++r) sm[padded(o + (brev_c(r, kOneLog) << s))] = v[r];
      __syncthreads();
    } else if (on) {
      double2* out = a.out + p * n;
#pragma unroll
      for (int r = 0; r < kOneP; ++r)
        out[o + (brev_c(r, kOneLog) << s)] = make_double2(v[r].x * scale, v[r].y * scale);
    }
  }
}

// LOGR radix-2 passes of every packet from one buffer to the other (x null:
// from the prepared input), for transforms of 1-3 passes and those above
// kOneMax; one thread per group of 2^LOGR points
template <int LOGR>
__global__ void __launch_bounds__(256) spec_pass_kernel(PrepArgs a, const double2* x, double2* y,
                                                        Twiddles tw, int s, double scale) {
  constexpr int R = 1 << LOGR;
  const int mf = a.mf;
  const long N = 1L << mf, M = N >> LOGR;
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= M * a.npk) return;
  const long p = gid >> (mf - LOGR), j0 = gid & (M - 1), k = j0 & ((1L << s) - 1);
  double2 v[R];
#pragma unroll
  for (int q = 0; q < R; ++q)
    v[q] = x ? x[p * N + j0 + q * M] : prep_value(a, p, j0 + q * M);
  passes<LOGR>(v, tw, k, s, mf);
  double2* yp = y + p * N + ((j0 - k) << LOGR) + k;
#pragma unroll
  for (int r = 0; r < R; ++r)
    yp[(long)brev_c(r, LOGR) << s] = make_double2(v[r].x * scale, v[r].y * scale);
}

template <int REM, int T>
cudaError_t launch_one(const PrepArgs& a, const Twiddles& tw, double scale, cudaStream_t st) {
  static DeviceFlags attr;
  const size_t smem = sizeof(double2) * padded(kOneP * T);
  cudaError_t e = set_max_smem_once(attr, spec_one_kernel<REM, T>, smem);
  if (e != cudaSuccess) return e;
  const int per = T >> (a.mf - kOneLog);  // packets per CTA
  spec_one_kernel<REM, T><<<(a.npk + per - 1) / per, T, smem, st>>>(a, tw, scale);
  return cudaGetLastError();
}

cudaError_t launch_pass(int logr, const PrepArgs& a, const double2* x, double2* y,
                        const Twiddles& tw, int s, double scale, cudaStream_t st) {
  const long th = ((1L << a.mf) >> logr) * a.npk;
  const unsigned nb = (unsigned)((th + 255) / 256);
  switch (logr) {
    case 1: spec_pass_kernel<1><<<nb, 256, 0, st>>>(a, x, y, tw, s, scale); break;
    case 2: spec_pass_kernel<2><<<nb, 256, 0, st>>>(a, x, y, tw, s, scale); break;
    case 3: spec_pass_kernel<3><<<nb, 256, 0, st>>>(a, x, y, tw, s, scale); break;
    default: spec_pass_kernel<4><<<nb, 256, 0, st>>>(a, x, y, tw, s, scale); break;
  }
  return cudaGetLastError();
}

// the transform's input into out: for samples that lie in the spectrum's memory, which
// every other form writes to while it still reads samples
__global__ void spec_prep_kernel(PrepArgs a) {
  const long N = 1L << a.mf, mc = N / 2;
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= N * a.npk) return;
  const long p = gid >> a.mf, i = gid & (N - 1);
  double2 z = prep_value(a, p, i);
  if (a.hwhm || a.window) {
    const double2 f = time_factor(a, i < mc ? i + mc : i - mc);
    z = make_double2(f.x * z.x - f.y * z.y, f.x * z.y + f.y * z.x);
  }
  a.out[gid] = z;
}

// mf = 0: the prepared sample is the spectrum (FFTNT returns at N = 1)
__global__ void spec_copy_kernel(PrepArgs a) {
  const long p = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p < a.npk) a.out[p] = prep_value(a, p, 0);
}

}  // namespace
}  // namespace espec

using namespace espec;

#define SPEC_CK(call)                                        \
  do {                                                       \
    cudaError_t e_ = (call);                                 \
    if (e_ != cudaSuccess) return set_cuda_error(#call, e_); \
  } while (0)

// Device-side pipeline: in (device) -> spec (device, [npk][2^mf]); work is a
// device scratch of npk*2^mf double2 plus 2^(mf-1) twiddles.
extern "C" int espec_spectrum_dev(int npk, int mf, const void* in, long ld, int assemble,
                                  double dtf, double tf, double tal, double de, int window,
                                  double wp, int quirks, void* spec, void* work, void* stream) {
  if (npk <= 0 || mf < 0 || mf > 26 || !in || !spec || (mf > 0 && !work))
    return set_error(ESPEC_EINVAL, "bad spectrum arguments");
  if (window == 1 && !(wp > 0.0 && wp < 1.0))
    return set_error(ESPEC_EINVAL, "the .SG window needs 0 < WP < 1");
  cudaStream_t st = (cudaStream_t)stream;
  const long N = 1L << mf;
  PrepArgs a{};
  a.npk = npk;
  a.mf = mf;
  a.ldc = ld;
  a.in = (const double2*)in;
  a.assemble = assemble;
  a.dtf = dtf;
  a.tf = tf;
  a.hwhm = tal >= 0.0;
  a.dem = -de * kHwhmScale;
  a.ta = tal * kHwhmScale;
  a.window = window == 1;
  if (a.window) {
    const double tmax = N * dtf;
    const double l = std::log(1.0 / wp);
    a.taux = tmax * tmax / (l * l);
  }
  a.out = (double2*)spec;
  const bool scaled = a.hwhm || a.window;
  if (mf == 0) {  // FFTNT returns at N = 1 (cfft.f:39)
    // work may be null here: the one time's factor goes through spec
    if (scaled) {
      PrepArgs b = a;
      b.factor = nullptr;
      for (int p = 0; p < npk; ++p) {
        b.in = a.in + p * ld;
        b.out = a.out + p;
        spec_hwhm_kernel<<<1, 1, 0, st>>>(b);
      }
    } else {
      spec_copy_kernel<<<(npk + 255) / 256, 256, 0, st>>>(a);
    }
    SPEC_CK(cudaGetLastError());
    return ESPEC_OK;
  }
  // cfft.f:35 declares TWOPI with a default-real literal: single precision
  const double twopi = (quirks & ESPEC_Q_FFTNT_SP) ? (double)(float)kTwoPi : kTwoPi;
  const long tot = N * npk;
  double2* wk = (double2*)work;
  double2* tw = wk + tot;
  const double rn = 1.0 / N;  // cfft.f:102-105
  // samples in spec's memory: prepared into work, then an odd number of groups of
  // passes from work to spec and back
  const double2* in_end = a.in + (npk - 1) * ld + (assemble ? N / 2 : N);
  if (a.in < a.out + tot && a.out < in_end) {
    PrepArgs b = a;
    b.out = wk;
    spec_prep_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(b);
    SPEC_CK(cudaGetLastError());
    spec_table_kernel<<<(unsigned)((N + 255) / 256), 256, 0, st>>>(a, tw, nullptr, nullptr,
                                                                   twopi / N);
    SPEC_CK(cudaGetLastError());
    const Twiddles tws{tw, nullptr};
    double2 *from = wk, *to = a.out;
    for (int s = 0, left = (mf + 3) / 4 | 1; s < mf; --left) {
      const int lr = (mf - s + left - 1) / left;
      SPEC_CK(launch_pass(lr, a, from, to, tws, s, s + lr == mf ? rn : 1.0, st));
      std::swap(from, to);
      s += lr;
    }
    return ESPEC_OK;
  }
  // groups of up to four passes, the short one first; the groups ping-pong
  // between work and spec and end in spec.  The time factors sit in the
  // buffer that the first group does not write.
  const int ngroups = (mf + 3) / 4;
  const bool one = mf >= 4 && mf <= kOneMax;
  double2* dst = one || ngroups % 2 == 1 ? a.out : wk;
  double2* factor = scaled ? (dst == a.out ? wk : a.out) : nullptr;
  a.factor = factor;
  // a whole-transform call leaves work's signal part free: the factors, then the
  // earlier passes' twiddles
  double2* pass = nullptr;
  if (one && (factor == nullptr || npk >= 2)) pass = factor == wk ? wk + N : wk;
  spec_table_kernel<<<(unsigned)((N + 255) / 256), 256, 0, st>>>(a, tw, pass, factor, twopi / N);
  SPEC_CK(cudaGetLastError());
  const Twiddles tws{tw, pass};
  if (one) {
    cudaError_t e;
    if (mf == kOneMax) {
      e = launch_one<1, 2 * kOneThreads>(a, tws, rn, st);
    } else {
      switch (mf % kOneLog) {
        case 0: e = launch_one<kOneLog, kOneThreads>(a, tws, rn, st); break;
        case 1: e = launch_one<1, kOneThreads>(a, tws, rn, st); break;
        default: e = launch_one<2, kOneThreads>(a, tws, rn, st); break;
      }
    }
    SPEC_CK(e);
    return ESPEC_OK;
  }
  const double2* src = nullptr;
  for (int s = 0; s < mf;) {
    const int lr = s == 0 && mf % 4 ? mf % 4 : 4;
    SPEC_CK(launch_pass(lr, a, src, dst, tws, s, s + lr == mf ? rn : 1.0, st));
    src = dst;
    dst = dst == a.out ? wk : a.out;
    s += lr;
  }
  return ESPEC_OK;
}

extern "C" size_t espec_spectrum_work_bytes(int npk, int mf) {
  return sizeof(double2) * (((size_t)npk << mf) + ((size_t)1 << (mf > 0 ? mf - 1 : 0)));
}

// ---------------------------------------------------------------------------
// Fortran drop-ins
// ---------------------------------------------------------------------------
namespace {

// host arrays U, V of 2^M points through the device pipeline
int run_host(int mf, double dtf, double tf, double tal, double de, int window, double wp,
             int quirks, double* u, double* v) {
  const size_t N = (size_t)1 << mf;
  double2 *d_in = nullptr, *d_spec = nullptr, *d_work = nullptr;
  int rc = 0;
  auto cleanup = [&]() {
    if (d_in) cudaFree(d_in);
    if (d_spec) cudaFree(d_spec);
    if (d_work) cudaFree(d_work);
  };
  if ((rc = ck(cudaMalloc(&d_in, N * 16), "cudaMalloc")) ||
      (rc = ck(cudaMalloc(&d_spec, N * 16), "cudaMalloc")) ||
      (rc = ck(cudaMalloc(&d_work, espec_spectrum_work_bytes(1, mf)), "cudaMalloc"))) {
    cleanup();
    return rc;
  }
  if ((rc = ck(cudaMemcpy2D(d_in, 16, u, 8, 8, N, cudaMemcpyHostToDevice), "H2D")) ||
      (rc = ck(cudaMemcpy2D((char*)d_in + 8, 16, v, 8, 8, N, cudaMemcpyHostToDevice), "H2D")) ||
      (rc = espec_spectrum_dev(1, mf, d_in, (long)N, 0, dtf, tf, tal, de, window, wp, quirks,
                               d_spec, d_work, nullptr)) ||
      (rc = ck(cudaMemcpy2D(u, 8, d_spec, 16, 8, N, cudaMemcpyDeviceToHost), "D2H")) ||
      (rc = ck(cudaMemcpy2D(v, 8, (char*)d_spec + 8, 16, 8, N, cudaMemcpyDeviceToHost), "D2H"))) {
    cleanup();
    return rc;
  }
  cleanup();
  return ESPEC_OK;
}

std::string fmt_f12_7(double x) {
  char buf[64];
  std::snprintf(buf, sizeof buf, "%.7f", x);
  std::string s(buf);
  if (s.size() > 12) {
    if (s.compare(0, 2, "0.") == 0) s.erase(0, 1);
    else if (s.compare(0, 3, "-0.") == 0) s.erase(1, 1);
  }
  if (s.size() > 12) return std::string(12, '*');
  return std::string(12 - s.size(), ' ') + s;
}

}  // namespace

// HWHM (hwhm.f:1-80): TAL is scaled in place as the reference does
extern "C" void hwhm_(const int* m, const double* dt, const double* tf, double* tal,
                      const double* de, double* u, double* v) {
  if (*m < 0 || *m > 26) {
    std::fprintf(stderr, "espec_gpu HWHM: M out of range\n");
    return;
  }
  // only the lifetime/shift factors: no window, no transform
  const size_t N = (size_t)1 << *m;
  double2 *d_in = nullptr, *d_out = nullptr;
  if (cudaMalloc(&d_in, N * 16) != cudaSuccess || cudaMalloc(&d_out, N * 16) != cudaSuccess) {
    std::fprintf(stderr, "espec_gpu HWHM: device allocation failed\n");
    if (d_in) cudaFree(d_in);
    return;
  }
  PrepArgs a{};
  a.npk = 1;
  a.mf = *m;
  a.ldc = (long)N;
  a.in = d_in;
  a.dtf = *dt;
  a.tf = *tf;
  a.hwhm = 1;
  a.dem = -*de * kHwhmScale;
  a.ta = *tal * kHwhmScale;
  a.out = d_out;
  cudaMemcpy2D(d_in, 16, u, 8, 8, N, cudaMemcpyHostToDevice);
  cudaMemcpy2D((char*)d_in + 8, 16, v, 8, 8, N, cudaMemcpyHostToDevice);
  spec_hwhm_kernel<<<(unsigned)((N + 255) / 256), 256>>>(a);
  cudaError_t e = cudaGetLastError();
  cudaMemcpy2D(u, 8, d_out, 16, 8, N, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess)
    e = cudaMemcpy2D(v, 8, (char*)d_out + 8, 16, 8, N, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) std::fprintf(stderr, "espec_gpu HWHM: %s\n", cudaGetErrorString(e));
  cudaFree(d_in);
  cudaFree(d_out);
  *tal = *tal * kHwhmScale;  // hwhm.f:61
}

// SPECTRUMTD (spectrumtd.f:1-116): window, swap, backward FFTNT on the GPU,
// then the printed spectrum table; DE < 0 is set to 0 in the caller's
// variable as the reference does
extern "C" void spectrumtd_(const char* tpwind, const int* m, const double* dt, const double* tf,
                            const double* wp, double* de, double* u, double* v,
                            size_t tpwind_len) {
  const int mf = *m;
  if (*de < 0.0) *de = 0.0;
  auto is = [&](const char* pat) {
    const size_t k = std::strlen(pat);
    return tpwind && tpwind_len >= k && std::memcmp(tpwind, pat, k) == 0;
  };
  int window = -1;
  if (is(".SG")) window = 1;
  else if (is(".NONE") || is(".NULL")) window = 0;
  if (window < 0) {  // spectrumtd.f:70-72 (the reference then stops)
    std::fputs("<<<>>> Windowing function error <<<>>>\n", stdout);
    std::fflush(stdout);
    return;
  }
  if (mf < 0 || mf > 26 ||
      run_host(mf, *dt, *tf, -1.0, 0.0, window, *wp, ESPEC_Q_FFTNT_SP, u, v) != ESPEC_OK) {
    std::fprintf(stderr, "espec_gpu SPECTRUMTD: %s\n", espec_last_error());
    return;
  }
  const std::string out = espec::spectrum_table(mf, *dt, *de, u, v);
  std::fwrite(out.data(), 1, out.size(), stdout);
  std::fflush(stdout);
}

namespace espec {
// spectrumtd.f:84-97 (list-directed head, FORMAT 1011 and 1021): the energy
// axis from -N/2 ENC, the FFTNT output from its second half on
std::string spectrum_table(int mf, double dt, double de, const double* u, const double* v) {
  const size_t N = (size_t)1 << mf;
  double enc = 1.0 / (N * dt) * kEnc;
  enc = enc * kFate;
  double en = -(double)N / 2.0 * enc;
  std::string out = " \n Spectrum:\n =========\n";
  out += "     *E (eV)*           *W*           *FFTr*          *FFTi*\n";
  auto row = [&](size_t i) {
    out += " " + fmt_f12_7(en + de) + "    " + fmt_f12_7(u[i]) + "    " + fmt_f12_7(u[i]) +
           "    " + fmt_f12_7(v[i]) + "\n";
    en = en + enc;
  };
  for (size_t i = N / 2; i < N; ++i) row(i);
  for (size_t i = 0; i < N / 2; ++i) row(i);
  return out;
}
}  // namespace espec
