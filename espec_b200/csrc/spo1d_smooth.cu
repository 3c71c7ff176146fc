// spo1d_smooth.cu -- the split-operator time loop for packet sizes outside the
// register plans of spo1d.cuh whose prime factors are at most 13 (FP64): eSPec's
// FFT (fft3d.f, Singleton's mixed-radix transform) takes any N, and its decks use
// grids such as 200, 250, 300 or 560 points.
//
// One CTA per packet, the packet in shared memory once: the forward transform is
// an in-place decimation in frequency (the output stays in digit-reversed order,
// which the kinetic table follows), the inverse its exact mirror.  A butterfly
// reads and writes the same places, so a pass over the packet needs one barrier
// and no second buffer; the first stage is fused across the step (inverse first
// stage, C(t), x-space phase, forward first stage in registers) and so is the last
// (forward, kinetic phase, inverse): 2 (S - 1) passes per step for S stages, S
// the least for radices up to 16 (1000 = 10 10 10, 560 = 8 7 10: 4 passes).
//
// What bounds it: for a packet per SM the chain of passes, each a shared-memory
// round trip, a butterfly and a barrier (N = 1000: 3.4 us per step); with many,
// the load/store unit, 16 wavefronts per 128 points and pass plus the tables
// from L1 and L2 (2048 packets of 1000 points: 74 G gridpt*steps/s).  The
// Stockham form of spo1d_any.cu, with 2 S' + 2 passes for S' stages of radix 2 to
// 5 and strided twiddles, took 13.4 us per step for one packet and ran at 36 G.
// Twiddles and the kinetic table are laid out by butterfly (adjacent threads,
// adjacent values): read by stride from e^{2 pi i e / N} they doubled the time.
#include <cuda_runtime.h>

#include <algorithm>

#include "espec_internal.h"
#include "spo1d_launch.cuh"
#include "spo1d_smooth.cuh"

namespace espec {
namespace {

// cos and sin of 2 pi j / R
template <int R>
ESPEC_HD double root_c(int j);
template <int R>
ESPEC_HD double root_s(int j);
template <>
ESPEC_HD double root_c<3>(int j) {
  switch (j) {
    case 1: return -0.5;
    case 2: return -0.5;
    default: return 1.0;
  }
}
template <>
ESPEC_HD double root_s<3>(int j) {
  switch (j) {
    case 1: return 0.8660254037844386;
    case 2: return -0.8660254037844386;
    default: return 0.0;
  }
}
template <>
ESPEC_HD double root_c<5>(int j) {
  switch (j) {
    case 1: return 0.30901699437494745;
    case 2: return -0.8090169943749475;
    case 3: return -0.8090169943749475;
    case 4: return 0.30901699437494745;
    default: return 1.0;
  }
}
template <>
ESPEC_HD double root_s<5>(int j) {
  switch (j) {
    case 1: return 0.9510565162951535;
    case 2: return 0.5877852522924731;
    case 3: return -0.5877852522924731;
    case 4: return -0.9510565162951535;
    default: return 0.0;
  }
}
template <>
ESPEC_HD double root_c<7>(int j) {
  switch (j) {
    case 1: return 0.6234898018587335;
    case 2: return -0.2225209339563144;
    case 3: return -0.9009688679024191;
    case 4: return -0.9009688679024191;
    case 5: return -0.2225209339563144;
    case 6: return 0.6234898018587335;
    default: return 1.0;
  }
}
template <>
ESPEC_HD double root_s<7>(int j) {
  switch (j) {
    case 1: return 0.7818314824680298;
    case 2: return 0.9749279121818236;
    case 3: return 0.4338837391175581;
    case 4: return -0.4338837391175581;
    case 5: return -0.9749279121818236;
    case 6: return -0.7818314824680298;
    default: return 0.0;
  }
}
template <>
ESPEC_HD double root_c<8>(int j) {
  switch (j) {
    case 1: return 0.7071067811865476;
    case 2: return 0.0;
    case 3: return -0.7071067811865476;
    case 4: return -1.0;
    case 5: return -0.7071067811865476;
    case 6: return 0.0;
    case 7: return 0.7071067811865476;
    default: return 1.0;
  }
}
template <>
ESPEC_HD double root_s<8>(int j) {
  switch (j) {
    case 1: return 0.7071067811865476;
    case 2: return 1.0;
    case 3: return 0.7071067811865476;
    case 4: return 0.0;
    case 5: return -0.7071067811865476;
    case 6: return -1.0;
    case 7: return -0.7071067811865476;
    default: return 0.0;
  }
}
template <>
ESPEC_HD double root_c<9>(int j) {
  switch (j) {
    case 1: return 0.766044443118978;
    case 2: return 0.17364817766693036;
    case 3: return -0.5;
    case 4: return -0.9396926207859084;
    case 5: return -0.9396926207859084;
    case 6: return -0.5;
    case 7: return 0.17364817766693036;
    case 8: return 0.766044443118978;
    default: return 1.0;
  }
}
template <>
ESPEC_HD double root_s<9>(int j) {
  switch (j) {
    case 1: return 0.6427876096865394;
    case 2: return 0.984807753012208;
    case 3: return 0.8660254037844386;
    case 4: return 0.3420201433256687;
    case 5: return -0.3420201433256687;
    case 6: return -0.8660254037844386;
    case 7: return -0.984807753012208;
    case 8: return -0.6427876096865394;
    default: return 0.0;
  }
}
template <>
ESPEC_HD double root_c<11>(int j) {
  switch (j) {
    case 1: return 0.8412535328311812;
    case 2: return 0.41541501300188644;
    case 3: return -0.14231483827328514;
    case 4: return -0.6548607339452851;
    case 5: return -0.9594929736144974;
    case 6: return -0.9594929736144974;
    case 7: return -0.6548607339452851;
    case 8: return -0.14231483827328514;
    case 9: return 0.41541501300188644;
    case 10: return 0.8412535328311812;
    default: return 1.0;
  }
}
template <>
ESPEC_HD double root_s<11>(int j) {
  switch (j) {
    case 1: return 0.5406408174555976;
    case 2: return 0.9096319953545183;
    case 3: return 0.9898214418809327;
    case 4: return 0.7557495743542583;
    case 5: return 0.28173255684142967;
    case 6: return -0.28173255684142967;
    case 7: return -0.7557495743542583;
    case 8: return -0.9898214418809327;
    case 9: return -0.9096319953545183;
    case 10: return -0.5406408174555976;
    default: return 0.0;
  }
}
template <>
ESPEC_HD double root_c<13>(int j) {
  switch (j) {
    case 1: return 0.8854560256532099;
    case 2: return 0.5680647467311558;
    case 3: return 0.12053668025532305;
    case 4: return -0.3546048870425356;
    case 5: return -0.7485107481711011;
    case 6: return -0.970941817426052;
    case 7: return -0.970941817426052;
    case 8: return -0.7485107481711011;
    case 9: return -0.3546048870425356;
    case 10: return 0.12053668025532305;
    case 11: return 0.5680647467311558;
    case 12: return 0.8854560256532099;
    default: return 1.0;
  }
}
template <>
ESPEC_HD double root_s<13>(int j) {
  switch (j) {
    case 1: return 0.46472317204376856;
    case 2: return 0.8229838658936564;
    case 3: return 0.992708874098054;
    case 4: return 0.9350162426854148;
    case 5: return 0.6631226582407952;
    case 6: return 0.23931566428755777;
    case 7: return -0.23931566428755777;
    case 8: return -0.6631226582407952;
    case 9: return -0.9350162426854148;
    case 10: return -0.992708874098054;
    case 11: return -0.8229838658936564;
    case 12: return -0.46472317204376856;
    default: return 0.0;
  }
}
template <>
ESPEC_HD double root_c<16>(int j) {
  switch (j) {
    case 1: return 0.9238795325112867;
    case 2: return 0.7071067811865476;
    case 3: return 0.3826834323650898;
    case 4: return 0.0;
    case 5: return -0.3826834323650898;
    case 6: return -0.7071067811865476;
    case 7: return -0.9238795325112867;
    case 8: return -1.0;
    case 9: return -0.9238795325112867;
    case 10: return -0.7071067811865476;
    case 11: return -0.3826834323650898;
    case 12: return 0.0;
    case 13: return 0.3826834323650898;
    case 14: return 0.7071067811865476;
    case 15: return 0.9238795325112867;
    default: return 1.0;
  }
}
template <>
ESPEC_HD double root_s<16>(int j) {
  switch (j) {
    case 1: return 0.3826834323650898;
    case 2: return 0.7071067811865476;
    case 3: return 0.9238795325112867;
    case 4: return 1.0;
    case 5: return 0.9238795325112867;
    case 6: return 0.7071067811865476;
    case 7: return 0.3826834323650898;
    case 8: return 0.0;
    case 9: return -0.3826834323650898;
    case 10: return -0.7071067811865476;
    case 11: return -0.9238795325112867;
    case 12: return -1.0;
    case 13: return -0.9238795325112867;
    case 14: return -0.7071067811865476;
    case 15: return -0.3826834323650898;
    default: return 0.0;
  }
}

__device__ __forceinline__ cpx<double> twid(cpx<double> x, double c, double s, bool inv) {
  const double w = inv ? -s : s;
  return mk(fma(x.x, c, -x.y * w), fma(x.x, w, x.y * c));
}

// R-point DFT in registers, natural order, e^{+2 pi i qk/R} (INV: conjugate)
template <int R, bool INV>
struct Dft;

// odd primes: sums and differences of the pairs q, R - q
template <int R, bool INV>
struct Dft {
  static __device__ __forceinline__ void run(cpx<double>* x) {
    constexpr int H = (R - 1) / 2;
    cpx<double> a[H], b[H];
#pragma unroll
    for (int q = 1; q <= H; ++q) {
      a[q - 1] = x[q] + x[R - q];
      b[q - 1] = x[q] - x[R - q];
    }
    const cpx<double> x0 = x[0];
#pragma unroll
    for (int q = 0; q < H; ++q) x[0] = x[0] + a[q];
#pragma unroll
    for (int k = 1; k <= H; ++k) {
      cpx<double> c = x0, s = mk(0.0, 0.0);
#pragma unroll
      for (int q = 1; q <= H; ++q) {
        const double wc = root_c<R>((q * k) % R), ws = root_s<R>((q * k) % R);
        c = mk(fma(wc, a[q - 1].x, c.x), fma(wc, a[q - 1].y, c.y));
        s = q == 1 ? mk(ws * b[0].x, ws * b[0].y)
                   : mk(fma(ws, b[q - 1].x, s.x), fma(ws, b[q - 1].y, s.y));
      }
      const cpx<double> i = INV ? mul_mi(s) : mul_i(s);
      x[k] = c + i;
      x[R - k] = c - i;
    }
  }
};
template <bool INV>
struct Dft<2, INV> {
  static __device__ __forceinline__ void run(cpx<double>* x) {
    const cpx<double> a = x[0], b = x[1];
    x[0] = a + b;
    x[1] = a - b;
  }
};
template <bool INV>
struct Dft<4, INV> {
  static __device__ __forceinline__ void run(cpx<double>* x) {
    const cpx<double> a = x[0] + x[2], b = x[0] - x[2], c = x[1] + x[3];
    const cpx<double> d = INV ? mul_mi(x[1] - x[3]) : mul_i(x[1] - x[3]);
    x[0] = a + c;
    x[2] = a - c;
    x[1] = b + d;
    x[3] = b - d;
  }
};
// A B points, A and B coprime: an A x B DFT without twiddles (Good and Thomas)
template <int A, int B, bool INV>
__device__ __forceinline__ void dft_coprime(cpx<double>* x) {
  constexpr int R = A * B;
  cpx<double> y[R];
#pragma unroll
  for (int b = 0; b < B; ++b) {
    cpx<double> t[A];
#pragma unroll
    for (int a = 0; a < A; ++a) t[a] = x[(B * a + A * b) % R];
    Dft<A, INV>::run(t);
#pragma unroll
    for (int a = 0; a < A; ++a) y[a * B + b] = t[a];
  }
#pragma unroll
  for (int a = 0; a < A; ++a) Dft<B, INV>::run(y + a * B);
#pragma unroll
  for (int k = 0; k < R; ++k) x[k] = y[(k % A) * B + k % B];
}
// A B points with the twiddles W_R^(b ka) between the two steps
template <int A, int B, bool INV>
__device__ __forceinline__ void dft_twiddled(cpx<double>* x) {
  constexpr int R = A * B;
  cpx<double> y[R];
#pragma unroll
  for (int b = 0; b < B; ++b) {
    cpx<double> t[A];
#pragma unroll
    for (int a = 0; a < A; ++a) t[a] = x[a * B + b];
    Dft<A, INV>::run(t);
#pragma unroll
    for (int a = 0; a < A; ++a) {
      const int e = a * b;
      if (e == 0) y[a * B + b] = t[a];
      else if (4 * e == R) y[a * B + b] = INV ? mul_mi(t[a]) : mul_i(t[a]);
      else y[a * B + b] = twid(t[a], root_c<R>(e), root_s<R>(e), INV);
    }
  }
#pragma unroll
  for (int a = 0; a < A; ++a) Dft<B, INV>::run(y + a * B);
#pragma unroll
  for (int k = 0; k < R; ++k) x[k] = y[(k % A) * B + k / A];
}
#define ESPEC_DFT(R, FN, A, B)                                                              \
  template <bool INV>                                                                       \
  struct Dft<R, INV> {                                                                      \
    static __device__ __forceinline__ void run(cpx<double>* x) { FN<A, B, INV>(x); }        \
  };
ESPEC_DFT(6, dft_coprime, 2, 3)
ESPEC_DFT(8, dft_twiddled, 2, 4)
ESPEC_DFT(9, dft_twiddled, 3, 3)
ESPEC_DFT(10, dft_coprime, 2, 5)
ESPEC_DFT(12, dft_coprime, 3, 4)
ESPEC_DFT(14, dft_coprime, 2, 7)
ESPEC_DFT(15, dft_coprime, 3, 5)
ESPEC_DFT(16, dft_twiddled, 4, 4)
#undef ESPEC_DFT

struct Ctx {
  cpx<double>* sm;
  const double2* __restrict__ tw;  // the stages' twiddles (smooth_twiddles)
  int n, t, T;
};

// A stage's places.  Element i of the transform sits at (i / r) p + i % r with r
// the last radix and p the odd one of r, r + 1: the last stage's butterflies then
// meet distinct banks, and every other stage keeps a constant stride.
struct Places {
  int m, step, block;  // butterflies of a block; places from point to point, from block to block
  unsigned inv, inv_last;
  int last, pitch;
  __device__ __forceinline__ Places(const SmoothPlan& pl, int s)
      : m(pl.m[s]), inv(pl.inv[s]), inv_last(pl.inv_last), last(pl.r[pl.ns - 1]), pitch(pl.pitch) {
    step = pl.step[s];
    block = step * pl.r[s];
  }
  // butterfly b: its j within the block, and the place of its first point
  __device__ __forceinline__ int first(int b, int& j) const {
    const int blk = __umulhi((unsigned)b, inv);
    j = b - blk * m;
    return blk * block + at(j);
  }
  __device__ __forceinline__ int at(int j) const {
    const int d = __umulhi((unsigned)j, inv_last);
    return d * pitch + (j - d * last);
  }
};

// forward stage in place: the R-point DFT over stride m, then W_M^(j k)
template <int R>
__device__ __forceinline__ void pass_forward(const Ctx& c, const Places& p, int tw_off) {
  for (int b = c.t; b < c.n / R; b += c.T) {
    int j;
    cpx<double>* x = c.sm + p.first(b, j);
    const double2* w = c.tw + tw_off + j;
    cpx<double> v[R];
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = x[q * p.step];
    Dft<R, false>::run(v);
    x[0] = v[0];
#pragma unroll
    for (int k = 1; k < R; ++k) {
      const double2 wk = __ldg(w + (k - 1) * p.m);
      x[k * p.step] = twid(v[k], wk.x, wk.y, false);
    }
  }
}
template <int R>
__device__ __forceinline__ void pass_inverse(const Ctx& c, const Places& p, int tw_off) {
  for (int b = c.t; b < c.n / R; b += c.T) {
    int j;
    cpx<double>* x = c.sm + p.first(b, j);
    const double2* w = c.tw + tw_off + j;
    cpx<double> v[R];
    v[0] = x[0];
#pragma unroll
    for (int k = 1; k < R; ++k) {
      const double2 wk = __ldg(w + (k - 1) * p.m);
      v[k] = twid(x[k * p.step], wk.x, wk.y, true);
    }
    Dft<R, true>::run(v);
#pragma unroll
    for (int q = 0; q < R; ++q) x[q * p.step] = v[q];
  }
}
// last stage both ways around the kinetic phase; the table of its points runs
// over the butterflies first (smooth_final_freq)
template <int R>
__device__ __forceinline__ void pass_kinetic(const Ctx& c, const SpoArgs<double>& a, int base,
                                             int pitch, bool quirk) {
  const int nb = c.n / R;
  for (int b = c.t; b < nb; b += c.T) {
    cpx<double>* x = c.sm + b * pitch;
    cpx<double> v[R];
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = x[q];
    Dft<R, false>::run(v);
    if (quirk) {  // spofft.f:148-154 as written: V(I) uses the updated U(I)
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const double kc = a.kq_c[base + q * nb + b], ks = a.kq_s[base + q * nb + b];
        const double un = kc * v[q].x + ks * v[q].y;
        const double vn = kc * v[q].y - ks * un;
        v[q] = mk(un * a.kq_scale, vn * a.kq_scale);
      }
    } else {
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = Tab<double>::apply(a.tab.k[base + q * nb + b], v[q]);
    }
    Dft<R, true>::run(v);
#pragma unroll
    for (int q = 0; q < R; ++q) x[q] = v[q];
  }
}
// first stage across the step: its inverse (not at the start), C(t) and the
// x-space phase ph, its forward (not at the end); start: from `src`, |psi|^2 in
// place of C(t); end: psi(TF) to out
enum { kStart = 0, kStep = 1, kEnd = 2 };
template <int R>
__device__ __forceinline__ void pass_x(const Ctx& c, const Places& p, const cpx<double>* ph,
                                       const cpx<double>* wt, const double2* src, double2* out,
                                       int mode, double& cr, double& ci) {
  const int m = c.n / R;
  for (int j = c.t; j < m; j += c.T) {
    cpx<double>* x = c.sm + p.at(j);
    cpx<double> v[R];
    if (mode == kStart) {
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const double2 y = src[j + q * m];
        v[q] = mk(y.x, y.y);
        cr += y.x * y.x + y.y * y.y;
      }
    } else {
      v[0] = x[0];
#pragma unroll
      for (int k = 1; k < R; ++k) {
        const double2 wk = __ldg(c.tw + j + (k - 1) * m);
        v[k] = twid(x[k * p.step], wk.x, wk.y, true);
      }
      Dft<R, true>::run(v);
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const cpx<double> w = wt[j + q * m];
        cr = fma(w.x, v[q].x, fma(-w.y, v[q].y, cr));
        ci = fma(w.x, v[q].y, fma(w.y, v[q].x, ci));
      }
    }
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = Tab<double>::apply(ph[j + q * m], v[q]);
    if (mode == kEnd) {
      if (out) {
#pragma unroll
        for (int q = 0; q < R; ++q) out[j + q * m] = make_double2(v[q].x, v[q].y);
      }
    } else {
      Dft<R, false>::run(v);
      x[0] = v[0];
#pragma unroll
      for (int k = 1; k < R; ++k) {
        const double2 wk = __ldg(c.tw + j + (k - 1) * m);
        x[k * p.step] = twid(v[k], wk.x, wk.y, false);
      }
    }
  }
}

#define ESPEC_RADIX(r, CALL)      \
  switch (r) {                    \
    case 2: CALL(2); break;       \
    case 3: CALL(3); break;       \
    case 4: CALL(4); break;       \
    case 5: CALL(5); break;       \
    case 6: CALL(6); break;       \
    case 7: CALL(7); break;       \
    case 8: CALL(8); break;       \
    case 9: CALL(9); break;       \
    case 10: CALL(10); break;     \
    case 11: CALL(11); break;     \
    case 12: CALL(12); break;     \
    case 13: CALL(13); break;     \
    case 14: CALL(14); break;     \
    case 15: CALL(15); break;     \
    default: CALL(16); break;     \
  }

__global__ void __launch_bounds__(kSmoothMaxThreads) spo_smooth_kernel(SpoArgs<double> a,
                                                                       SmoothPlan pl,
                                                                       const double2* tw,
                                                                       int quirk) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double2 red[kSmoothMaxThreads / 32];
  Ctx c;
  c.sm = reinterpret_cast<cpx<double>*>(smem_raw);
  c.tw = tw;
  c.n = pl.n;
  c.t = threadIdx.x;
  c.T = blockDim.x;
  const int lane = c.t & 31, warp = c.t >> 5, nw = c.T >> 5, last = pl.ns - 1;
  const SpoPacket pk = a.pk[blockIdx.x];
  const int base = pk.off;
  double2* cout = a.c_out + pk.c_off;
  const double2* src = (a.psi_start ? a.psi_start : a.psi0) + base;
  double2* out = a.psi_out ? a.psi_out + base : nullptr;
  bool finite = true;
  // the packet's C(t) sample: warp sums before a barrier, thread 0 after it
  auto put_sum = [&](double cr, double ci) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      cr += __shfl_xor_sync(0xffffffffu, cr, o);
      ci += __shfl_xor_sync(0xffffffffu, ci, o);
    }
    if (lane == 0) red[warp] = make_double2(cr, ci);
  };
  auto take_sum = [&](int step) {
    if (c.t == 0) {
      double sx = 0.0, sy = 0.0;
      for (int i = 0; i < nw; ++i) {
        sx += red[i].x;
        sy += red[i].y;
      }
      if (step > 0) finite = finite && isfinite(sx) && isfinite(sy);
      cout[step] = make_double2(sx, sy);
    }
  };
  const Places p0(pl, 0);
  auto x_pass = [&](int mode, const cpx<double>* ph) {
    double cr = 0.0, ci = 0.0;
#define ESPEC_CALL(R) pass_x<R>(c, p0, ph + base, a.tab.w + base, src, out, mode, cr, ci)
    ESPEC_RADIX(pl.r[0], ESPEC_CALL)
#undef ESPEC_CALL
    put_sum(cr, ci);
    __syncthreads();
  };
  if (a.nsteps == 0) {
    double c0 = 0.0;
    for (int x = c.t; x < c.n; x += c.T) {
      const double2 p = src[x];
      c0 += p.x * p.x + p.y * p.y;
      if (out) out[x] = p;
    }
    put_sum(c0, 0.0);
    __syncthreads();
    if (!a.psi_start) take_sum(0);
    return;
  }
  x_pass(kStart, a.tab.h);
  if (!a.psi_start) take_sum(0);
  for (int step = 1; step <= a.nsteps; ++step) {
    for (int s = 1; s < last; ++s) {
      const Places ps(pl, s);
#define ESPEC_CALL(R) pass_forward<R>(c, ps, pl.tw_off[s])
      ESPEC_RADIX(pl.r[s], ESPEC_CALL)
#undef ESPEC_CALL
      __syncthreads();
    }
#define ESPEC_CALL(R) pass_kinetic<R>(c, a, base, pl.pitch, quirk != 0)
    ESPEC_RADIX(pl.r[last], ESPEC_CALL)
#undef ESPEC_CALL
    __syncthreads();
    for (int s = last - 1; s >= 1; --s) {
      const Places ps(pl, s);
#define ESPEC_CALL(R) pass_inverse<R>(c, ps, pl.tw_off[s])
      ESPEC_RADIX(pl.r[s], ESPEC_CALL)
#undef ESPEC_CALL
      __syncthreads();
    }
    const bool end = step == a.nsteps;
    x_pass(end ? kEnd : kStep, end ? a.tab.hm : a.tab.g);
    take_sum(step);
  }
  if (c.t == 0 && !finite && a.nonfinite) atomicAdd(a.nonfinite, 1);
}

// the fewest radices of at most kSmoothMaxRadix with product n (0: none), then
// the smallest largest radix, by trying every divisor
int best_radices(int n, int depth, int max_r, int* r) {
  if (n == 1) return 0;
  if (depth == 0) return -1;
  for (int d = std::min(n, max_r); d >= 2; --d) {
    if (n % d) continue;
    const int k = best_radices(n / d, depth - 1, d, r + 1);
    if (k >= 0) {
      r[0] = d;
      return k + 1;
    }
  }
  return -1;
}

}  // namespace

// Fewest stages first (each costs two passes per step), then the smallest
// largest radix (registers, and threads per packet); at least two stages.  An odd
// radix goes last, where butterflies are contiguous: its stride meets distinct
// banks; the largest of the others first.
bool smooth_plan(int n, SmoothPlan& pl) {
  if (n < 4 || n % 2) return false;
  int m = n;
  for (int p : {2, 3, 5, 7, 11, 13})
    while (m % p == 0) m /= p;
  if (m != 1) return false;
  int best[kSmoothMaxStages], ns = 0;
  for (int depth = 2; depth <= kSmoothMaxStages && ns == 0; ++depth)
    for (int mr = 2; mr <= kSmoothMaxRadix && ns == 0; ++mr) {
      int r[kSmoothMaxStages];
      const int k = best_radices(n, depth, mr, r);
      if (k >= 2) {
        ns = k;
        std::copy(r, r + k, best);
      }
    }
  if (ns == 0) return false;
  std::sort(best, best + ns, [](int x, int y) { return x > y; });
  for (int s = ns - 1; s >= 0; --s)
    if (best[s] % 2) {
      std::rotate(best + s, best + s + 1, best + ns);
      break;
    }
  pl.n = n;
  pl.ns = ns;
  const int last = best[ns - 1];
  pl.pitch = last | 1;
  auto recip = [](int d) { return (unsigned)(((1ull << 32) + d - 1) / d); };  // d >= 2
  pl.inv_last = recip(last);
  m = n;
  int most = 0, off = 0;
  for (int s = 0; s < ns; ++s) {
    pl.r[s] = best[s];
    m /= best[s];
    pl.m[s] = m;
    pl.inv[s] = m > 1 ? recip(m) : 0u;
    pl.step[s] = s + 1 < ns ? m / last * pl.pitch : 1;
    pl.tw_off[s] = off;
    if (s + 1 < ns) off += (best[s] - 1) * m;
    most = std::max(most, n / best[s]);
  }
  pl.ntw = off;
  pl.threads = std::min(kSmoothMaxThreads, (most + 31) / 32 * 32);
  return true;
}

// place q nb + b of the kinetic table: point q of butterfly b of the last stage
// (nb butterflies), position b r + q of the forward transform
void smooth_final_freq(const SmoothPlan& pl, int* kap) {
  const int r = pl.r[pl.ns - 1], nb = pl.n / r;
  for (int j = 0; j < pl.n; ++j) {
    int f = 0, mult = 1, rem = j;
    for (int s = 0; s < pl.ns; ++s) {
      f += rem / pl.m[s] * mult;
      rem %= pl.m[s];
      mult *= pl.r[s];
    }
    kap[j % r * nb + j / r] = f;
  }
}

// w[e] = e^{2 pi i e / n} gathered per stage: W_M^(j k) at (k - 1) m + j, so that
// the threads of a pass read adjacent values
void smooth_twiddles(const SmoothPlan& pl, const double2* w, double2* tw) {
  for (int s = 0; s + 1 < pl.ns; ++s) {
    const int m = pl.m[s], nm = pl.n / (m * pl.r[s]);
    for (int k = 1; k < pl.r[s]; ++k)
      for (int j = 0; j < m; ++j) tw[pl.tw_off[s] + (k - 1) * m + j] = w[k * j * nm];
  }
}

size_t smooth_smem_bytes(const SmoothPlan& pl) {
  return sizeof(cpx<double>) * (size_t)(pl.n / pl.r[pl.ns - 1]) * pl.pitch;
}

cudaError_t spo_smooth_launch(const SpoArgs<double>& a, const SmoothPlan& pl, const double2* tw,
                              bool quirk, int nblocks, cudaStream_t st) {
  static DeviceFlags f;
  const size_t smem = smooth_smem_bytes(pl);
  if (smem > kMaxSmem - 1024) return cudaErrorInvalidConfiguration;
  cudaError_t e = set_max_smem_once(f, spo_smooth_kernel, kMaxSmem - 1024);
  if (e != cudaSuccess) return e;
  spo_smooth_kernel<<<nblocks, pl.threads, smem, st>>>(a, pl, tw, quirk ? 1 : 0);
  return cudaGetLastError();
}

}  // namespace espec
