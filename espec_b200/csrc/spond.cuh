// spond.cuh -- the passes of the 2D/3D split operator and second-order
// differences (spond.cu): line transforms, x, y and z passes, and the
// cooperative kernel that runs a whole propagation; instantiated per element
// type and CTA size in spond_inst_*.cu.
//
#pragma once
#include <cuda/atomic>
#include <cuda_runtime.h>

#include <type_traits>

#include "cplx.cuh"
#include "espec_gpu.h"
#include "espec_internal.h"

namespace espec {
namespace nd {

constexpr unsigned kFull = 0xffffffffu;
// dynamic shared memory of a CTA: 227 KB less the kernels' static part
constexpr size_t kNdMaxSmem = 227 * 1024 - 2048;

__host__ __device__ __forceinline__ constexpr int brev_bits(int v, int bits) {
  int r = 0;
  for (int i = 0; i < bits; ++i) r |= ((v >> i) & 1) << (bits - 1 - i);
  return r;
}
// Fixed rotations: FP64 as (cos, sin) applied by a complex product; FP32 as
// three lifting shears (RotF), whose rounding is unbiased -- a rounded
// (cos, sin) pair has |w| != 1 and a fixed-angle product loses or gains norm
// systematically, step after step.
template <typename R>
struct Rot;
template <>
struct Rot<double> {
  using type = RotD;
  static __device__ __forceinline__ RotD make(double k_over_n) {  // exp(-2 pi i k/n)
    RotD r;
    sincospi(-2.0 * k_over_n, &r.s, &r.c);
    return r;
  }
};
template <>
struct Rot<float> {
  using type = RotF;
  static __device__ __forceinline__ RotF make(double k_over_n) {
    return make_rotf(-6.283185307179586476925287 * k_over_n);
  }
};
template <typename R>
__device__ __forceinline__ typename Rot<R>::type twid(int k, int n) {
  return Rot<R>::make((double)k / (double)n);
}

// x-space and kinetic factors: FP64 complex, or FP32 lifting rotation with a
// magnitude (the sign of a removed pi folded into it)
struct PhF {
  float t, s, ag;
};
template <typename R>
struct Ph;
template <>
struct Ph<double> {
  using type = cpx<double>;
};
template <>
struct Ph<float> {
  using type = PhF;
};
__host__ __device__ __forceinline__ cpx<double> apply_ph(cpx<double> p, cpx<double> v) {
  return mk(v.x * p.x - v.y * p.y, v.x * p.y + v.y * p.x);
}
__host__ __device__ __forceinline__ cpx<float> apply_ph(PhF p, cpx<float> v) {
  float x = v.x * p.ag, y = v.y * p.ag;
  x = fmaf(-p.t, y, x);
  y = fmaf(p.s, x, y);
  x = fmaf(-p.t, y, x);
  return mk(x, y);
}
// e^{i phi} times a, as stored factors
__host__ __device__ inline PhF make_phf(double phi, double a) {
  const RotF r = make_rotf(phi);
  PhF o;
  o.t = r.t;
  o.s = r.s;
  o.ag = (float)(r.g * a);
  return o;
}

// Line transform of N = 2^LN points (32 <= N <= 512), E points per thread, the
// line's L = N/E threads exchanging through shared memory.  The arithmetic is
// the four-step form N = 32 P: radix-2 decimation in frequency over the P-point
// index (twiddles W_P), the twiddle W_N^(l k1), then radix-2 decimation in
// frequency over the 32-point index l -- one level per bit of the position
// 32 j + l, from the top, in place.  A thread takes LE levels at a time: group
// k holds LE bits of the position (the low end of the group at bit lo(k)) and
// the thread number the other bits, so both partners of a butterfly are in one
// thread.  (One warp per line with the lower five levels by __shfl_xor, the
// form before, evaluated both branches of every butterfly in both lanes and
// moved each word five times: 80 instructions per point against about 45.)
// The inverse is the exact mirror with conjugate twiddles (unnormalised).
template <typename R, int LN>
struct LineFft {
  static constexpr int N = 1 << LN, LE = LN == 9 ? 4 : 3, E = 1 << LE, LT = LN - LE, L = 1 << LT;
  static constexpr int NG = (LN + LE - 1) / LE;  // groups: 5 = 3+2, 6 = 3+3, 7 = 3+3+1, ...
  using T = typename Rot<R>::type;
  static __host__ __device__ constexpr int lo(int k) {
    return LN - LE * (k + 1) > 0 ? LN - LE * (k + 1) : 0;
  }
  static __host__ __device__ constexpr int hi(int k) { return LN - LE * k; }
  // position of element e of thread t in group k
  static __device__ __forceinline__ int pos(int k, int t, int e) {
    const int l = lo(k);
    return ((t >> l) << (l + LE)) | (e << l) | (t & ((1 << l) - 1));
  }
  // twiddle index of the level at bit b at position p: W_2h^(q), q the bits
  // below b of the P-point or the 32-point index
  static __device__ __forceinline__ int tw_index(int b, int p) {
    return b >= 5 ? ((p >> 5) & ((1 << (b - 5)) - 1)) * (N >> (b - 4))
                  : (p & ((1 << b) - 1)) * (N >> (b + 1));
  }
  // the distinct twiddles of the level at bit b of group k, by the bits of e
  // below b that enter its index: nq of them, number red(e); W^0 at compile
  // time is none (the rotation by it is exact in both forms)
  static __host__ __device__ constexpr int sh(int k, int b) {
    return b >= 5 && lo(k) < 5 ? 5 - lo(k) : 0;
  }
  static __host__ __device__ constexpr int nq(int k, int b) { return 1 << (b - lo(k) - sh(k, b)); }
  static __host__ __device__ constexpr bool trivial(int k, int b, int r) {
    return r == 0 && (b >= 5 || lo(k) == 0);
  }
  static __host__ __device__ constexpr int k1_of(int e) {
    return brev_bits((e << lo(0)) >> 5, LN - 5);
  }
  static __host__ __device__ constexpr int count() {  // twiddles of a thread
    int n = 0;
    for (int k = 0; k < NG; ++k)
      for (int b = lo(k); b < hi(k); ++b)
        for (int r = 0; r < nq(k, b); ++r) n += !trivial(k, b, r);
    for (int e = 0; e < E; ++e) n += k1_of(e) != 0;
    return n;
  }
  T wl[NG][E];  // group k, level b, number r: at nq(k, b) + r
  T wb[E];      // W_N^(l k1) of the first group's elements
  int t;

  template <class F>
  __device__ __forceinline__ void each(F f) {
    int i = 0;
#pragma unroll
    for (int k = 0; k < NG; ++k)
#pragma unroll
      for (int b = hi(k) - 1; b >= lo(k); --b)
#pragma unroll
        for (int r = 0; r < nq(k, b); ++r)
          if (!trivial(k, b, r)) f(i++, wl[k][nq(k, b) + r], tw_index(b, pos(k, t, r << sh(k, b))));
#pragma unroll
    for (int e = 0; e < E; ++e)
      if (k1_of(e)) f(i++, wb[e], (pos(0, t, e) & 31) * k1_of(e));
  }
  // every twiddle is W_N^k, k < N, of the line's table (built once per plan in
  // FP64, tw_table_kernel); a CTA keeps them by twiddle and thread, which reads
  // without bank conflicts where W_N^(t k1) by stride k1 does not
  static __device__ __forceinline__ void pack(const T* tab, T* dst) {
    if (threadIdx.x < L) {
      LineFft f;
      f.t = threadIdx.x;
      f.each([&](int i, T&, int index) { dst[i * L + threadIdx.x] = tab[index]; });
    }
  }
  __device__ __forceinline__ void init(const T* packed, int thread) {
    t = thread;
    each([&](int i, T& w, int) { w = packed[i * L + thread]; });
  }
  template <bool INV>
  __device__ __forceinline__ void level(cpx<R>* v, int k, int b) const {
    const int h = 1 << (b - lo(k));
#pragma unroll
    for (int e = 0; e < E; ++e) {
      if (e & h) continue;
      const int r = (e & (h - 1)) >> sh(k, b), n = nq(k, b);
      if (!INV) {
        const cpx<R> x = v[e], y = v[e + h];
        v[e] = x + y;
        v[e + h] = trivial(k, b, r) ? x - y : rot<false>(wl[k][n + r], x - y);
      } else {
        const cpx<R> x = v[e];
        const cpx<R> y = trivial(k, b, r) ? v[e + h] : rot<true>(wl[k][n + r], v[e + h]);
        v[e] = x + y;
        v[e + h] = x - y;
      }
    }
  }
  template <bool INV>
  __device__ __forceinline__ void twiddle(cpx<R>* v) const {
#pragma unroll
    for (int e = 0; e < E; ++e)
      if (k1_of(e)) v[e] = rot<INV>(wb[e], v[e]);
  }
  // from the first group's layout to the last's; at(p): the exchange slot of
  // position p, sync(): a barrier of the line's threads.  A thread writes only
  // the positions it read last, so each exchange needs one barrier, and so
  // does a transform that follows another on the same exchange space.
  template <class At, class Sync>
  __device__ __forceinline__ void forward(cpx<R>* v, At at, Sync sync) const {
#pragma unroll
    for (int k = 0; k < NG; ++k) {
      if (k > 0) {
#pragma unroll
        for (int e = 0; e < E; ++e) *at(pos(k - 1, t, e)) = v[e];
        sync();
#pragma unroll
        for (int e = 0; e < E; ++e) v[e] = *at(pos(k, t, e));
      }
#pragma unroll
      for (int b = hi(k) - 1; b >= lo(k); --b) {
        if (k == 0 && b == 4) twiddle<false>(v);
        level<false>(v, k, b);
      }
      if (k == 0 && lo(k) == 5) twiddle<false>(v);
    }
  }
  template <class At, class Sync>
  __device__ __forceinline__ void inverse(cpx<R>* v, At at, Sync sync) const {
#pragma unroll
    for (int k = NG - 1; k >= 0; --k) {
      if (k < NG - 1) {
#pragma unroll
        for (int e = 0; e < E; ++e) *at(pos(k + 1, t, e)) = v[e];
        sync();
#pragma unroll
        for (int e = 0; e < E; ++e) v[e] = *at(pos(k, t, e));
      }
      if (k == 0 && lo(k) == 5) twiddle<true>(v);
#pragma unroll
      for (int b = lo(k); b < hi(k); ++b) {
        level<true>(v, k, b);
        if (k == 0 && b == 4) twiddle<true>(v);
      }
    }
  }
};

// what the passes of a step read; copied to shared memory by every CTA
template <typename R>
struct NdArgs {
  int ln[3], ndim;        // log2 of the axis lengths (0 for an absent z)
  long n;
  cpx<R>* psi;            // state between the passes, storage order (NdLayout)
  const double2* psi0;    // psi(0), natural order
  const double2* psi_start;  // the natural-order state a run starts from
  double2* psi_out;       // psi(TF), natural order
  using PhT = typename Ph<R>::type;
  const PhT* g;           // x-space factors, natural order
  const PhT* h;
  const PhT* hm;
  const double2* w;       // conj(psi0) hm, for C(t) (FP64 in both forms)
  const PhT* K;           // kinetic factors in storage order
  const double* kq_c;     // reference-defect form: cos / sin(CST1 TC), storage order
  const double* kq_s;
  double kq_scale;
  double2* cpart;         // C(t) partial sums [step][CTA]
  const typename Rot<R>::type* tw[3];  // W_n^k tables of the x, y, z line lengths
  // second-order differences (psodfft.f / sodfft.f:64-126): dst <- old - i f
  // (vc src + T src) [+ f ab src, or times the mask], natural order
  double2 *cur, *prev;
  const double* vc;   // CST V
  const double* ab;   // CST VABC (.VOPTIC) or the .SMOOTHW mask
  int kabs;           // 0 none, 1 complex potential, 2 mask
  // the run
  int op;             // kOpSpo, kOpSod, kOpForward
  int nsteps, from_start;
  int fused;          // 3D: xy planes whole in shared memory
  int lc;             // log2 of the adjacent columns of a tile
  int kstage;         // the kinetic pass copies its tiles ahead (kin_staged)
  unsigned long long* bar;  // grid barrier arrivals of the launch (zeroed before it)
  int* err;                 // set when a barrier wait gave up
  long spin_limit;
};
enum { kOpSpo = 0, kOpSod = 1, kOpForward = 2 };

// W_n^k = exp(-2 pi i k / n), k < n, in the form the line transforms apply
template <typename R>
__global__ void tw_table_kernel(typename Rot<R>::type* tab, int n) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) tab[k] = twid<R>(k, n);
}

// one row update of the second-order-differences form
struct SodRow {
  const double2 *src, *old;
  double2* dst;
  double f;
};

// x-space work of a row between its inverse and its forward transform.  kFirst:
// h psi of a natural-order state, |psi|^2; kMid / kLast: C(t) and the phase g
// or hm; kFwd0: a natural-order state; kUpd / kUpdFwd: the leapfrog update
enum { kFirst = 0, kMid = 1, kLast = 2, kFwd0 = 3, kUpd = 4, kUpdFwd = 5 };
__host__ __device__ constexpr bool row_inverse(int mode) { return mode != kFirst && mode != kFwd0; }
__host__ __device__ constexpr bool row_forward(int mode) { return mode != kLast && mode != kUpd; }

// asynchronous copies into shared memory
template <int BYTES>
__device__ __forceinline__ void copy_async(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int PENDING>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

// what row_points reads of a row's points; loaded before the inverse transform so
// that the two overlap: into registers where they allow it (8 points per thread,
// 256 threads), or (ST) the 16-byte values into the lane's places of shared memory
template <typename R, int E, int MODE, int T, bool ST = false>
struct RowIn {
  static constexpr bool kStaged = ST && E == 8 && row_inverse(MODE);
  static constexpr bool kEarlyP = E == 8 && row_inverse(MODE) && T == 256 && !kStaged;
  static constexpr bool kEarlyQ = kEarlyP || (kStaged && (T == 256 || sizeof(R) == 4));
  double2 p[E], q[E];
  typename Ph<R>::type ph[E];
  double2* st;  // kStaged: [E][32]
  __device__ __forceinline__ const double2* source(const NdArgs<R>& a, const SodRow& o) const {
    return MODE == kMid || MODE == kLast ? a.w : o.src;
  }
  __device__ __forceinline__ void load_p(const NdArgs<R>& a, const SodRow& o, int e, int x) {
    if (MODE == kFirst || MODE == kFwd0) p[e] = a.psi_start[x];
    else if (MODE == kMid || MODE == kLast) p[e] = __ldg(a.w + x);
    else p[e] = o.src[x];
  }
  __device__ __forceinline__ void load_q(const NdArgs<R>& a, const SodRow& o, int e, int x) {
    if (MODE == kFirst) ph[e] = a.h[x];
    else if (MODE == kMid) ph[e] = a.g[x];
    else if (MODE == kLast) ph[e] = a.hm[x];
    else if (MODE == kUpd || MODE == kUpdFwd) q[e] = o.old[x];
  }
  __device__ __forceinline__ void early(const NdArgs<R>& a, const SodRow& o, int x0, int step) {
    if (kStaged) {
      const double2* src = source(a, o);
#pragma unroll
      for (int e = 0; e < E; ++e)
        copy_async<16>(st + 32 * e + (threadIdx.x & 31), src + x0 + e * step);
      copy_commit();
    }
    if (kEarlyP) {
#pragma unroll
      for (int e = 0; e < E; ++e) load_p(a, o, e, x0 + e * step);
    }
    if (kEarlyQ) {
#pragma unroll
      for (int e = 0; e < E; ++e) load_q(a, o, e, x0 + e * step);
    }
  }
};

template <typename R, int LN, int MODE, int T, bool ST>
__device__ __forceinline__ void row_points(const NdArgs<R>& a, const SodRow& o, cpx<R>* v,
                                           RowIn<R, LineFft<R, LN>::E, MODE, T, ST>& in,
                                           const LineFft<R, LN>& fft, int base, double& cr,
                                           double& ci) {
  constexpr int E = LineFft<R, LN>::E, L = LineFft<R, LN>::L;
  if (in.kStaged) copy_wait<0>();  // a lane reads its own copies only
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int x = base + e * L + fft.t;
    // 128 registers: the loads of half a row's points at a time
    if (T == 512 && e == E / 2) asm volatile("" ::: "memory");
    if (in.kStaged) in.p[e] = in.st[32 * e + (threadIdx.x & 31)];
    else if (!in.kEarlyP) in.load_p(a, o, e, x);
    if (!in.kEarlyQ) in.load_q(a, o, e, x);
    const double2 p = in.p[e];
    if (MODE == kFirst) {
      cr += p.x * p.x + p.y * p.y;  // C(0) = <psi0|psi0> (not used when resuming)
      v[e] = apply_ph(in.ph[e], mk((R)p.x, (R)p.y));
    } else if (MODE == kFwd0) {
      if (a.op == kOpSod) cr += p.x * p.x + p.y * p.y;
      v[e] = mk((R)p.x, (R)p.y);
    } else if (MODE == kMid || MODE == kLast) {
      cr += p.x * (double)v[e].x - p.y * (double)v[e].y;
      ci += p.x * (double)v[e].y + p.y * (double)v[e].x;
      v[e] = apply_ph(in.ph[e], v[e]);
      if (MODE == kLast) a.psi_out[x] = make_double2((double)v[e].x, (double)v[e].y);
    } else {
      // T src by the inverse of the transformed copy, then the leapfrog update
      const double2 sj = p, dj = in.q[e];
      const double vc = a.vc[x];
      const double hx = fma(vc, sj.x, (double)v[e].x), hy = fma(vc, sj.y, (double)v[e].y);
      double ox = fma(o.f, hy, dj.x), oy = fma(-o.f, hx, dj.y);
      if (a.kabs == 1) {
        const double abf = o.f * a.ab[x];
        ox = fma(abf, sj.x, ox);
        oy = fma(abf, sj.y, oy);
      } else if (a.kabs == 2) {
        ox *= a.ab[x];
        oy *= a.ab[x];
      }
      o.dst[x] = make_double2(ox, oy);
      const double2 wj = a.w[x];  // conj(psi0)
      cr += wj.x * ox - wj.y * oy;
      ci += wj.x * oy + wj.y * ox;
      v[e] = mk((R)ox, (R)oy);
    }
  }
}

__device__ __forceinline__ void bar_group(int id, int threads) {
  if (threads <= 32) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// places of a line's exchange: skewed for tiles of columns (one element in 8
// added), and for whole rows a swizzle of the low bits -- the low 3 of 16-byte,
// 4 of 8-byte elements, one line of banks -- by the bits above (a Gray code, so
// that both the stride-8 and the stride-16 patterns of the groups and any
// aligned run of columns meet distinct banks)
__device__ __forceinline__ int skew(int p) { return p + (p >> 3); }
template <typename R>
__device__ __forceinline__ int slot_of(int p) {
  if (sizeof(R) == 8) return p ^ (((p >> 3) ^ (p >> 4)) & 7);
  const int h = p >> 4;
  return p ^ ((h ^ (h << 1)) & 15);
}

// x pass: the rows of the grid, 32/L of them per warp; psi holds a row's
// transform in storage order (coalesced for the last group's registers)
template <typename R, int LN, int MODE, int T>
__device__ __noinline__ double2 rows_phase(const NdArgs<R>& a, const SodRow& o,
                                           const typename Rot<R>::type* tab, cpx<R>* sm) {
  using F = LineFft<R, LN>;
  constexpr int N = F::N, E = F::E, L = F::L, LW = 32 / L;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = blockDim.x >> 5, sub = lane / L;
  cpx<R>* ex = sm + (warp * LW + sub) * (N + N / 8);
  F fft;
  fft.init(tab, lane % L);
  auto at = [&](int p) { return ex + slot_of<R>(p); };
  auto sync = [&]() { __syncwarp(); };
  double cr = 0.0, ci = 0.0;
  const int items = (int)(a.n >> LN) / LW, step = gridDim.x * nw;
  for (int it = blockIdx.x + gridDim.x * warp; it < items; it += step) {
    const int base = (it * LW + sub) << LN;
    cpx<R> v[E];
    RowIn<R, E, MODE, T> in;
    if (row_inverse(MODE)) {
#pragma unroll
      for (int e = 0; e < E; ++e) v[e] = a.psi[base + e * L + fft.t];
      in.early(a, o, base + fft.t, L);
      fft.inverse(v, at, sync);
    }
    row_points<R, LN, MODE, T, false>(a, o, v, in, fft, base, cr, ci);
    if (row_forward(MODE)) {
      fft.forward(v, at, sync);
#pragma unroll
      for (int e = 0; e < E; ++e) a.psi[base + e * L + fft.t] = v[e];
    }
    __syncwarp();
  }
  return make_double2(cr, ci);
}

enum { kFwd = 0, kInv = 1, kKin = 2 };

// y or z pass: tiles of 2^lc adjacent x columns of one line set, a group of
// 2^lc L threads per tile (consecutive threads: consecutive columns, so the
// line's points go straight between global memory and registers)
template <typename R, int LN, int MODE, int T>
__device__ __noinline__ void cols_phase(const NdArgs<R>& a, int axis,
                                        const typename Rot<R>::type* tab, cpx<R>* sm) {
  using F = LineFft<R, LN>;
  constexpr int N = F::N, E = F::E, L = F::L;
  const int lc = a.lc, gt = L << lc;  // threads of a group
  const int group = threadIdx.x / gt, ng = blockDim.x / gt;
  const int c = threadIdx.x & ((1 << lc) - 1);
  cpx<R>* ex = sm + ((group * (N + N / 8)) << lc) + c;
  F fft;
  fft.init(tab, (threadIdx.x >> lc) & (L - 1));
  auto at = [&](int p) { return ex + (skew(p) << lc); };
  auto sync = [&]() { bar_group(1 + group, gt); };
  const int ltx = a.ln[0] - lc;  // log2 of the tiles along x
  const int stride = axis == 1 ? 1 << a.ln[0] : 1 << (a.ln[0] + a.ln[1]);  // n <= 2^27
  const int lset = axis == 1 ? a.ln[0] + a.ln[1] : a.ln[0];  // log2 of a line set's pitch
  const int items = (int)(a.n >> (LN + lc));
  for (int it = blockIdx.x + gridDim.x * group; it < items; it += gridDim.x * ng) {
    const int base = ((it >> ltx) << lset) + ((it & ((1 << ltx) - 1)) << lc) + c;
    cpx<R> v[E];
    typename Ph<R>::type kf[E];
    constexpr bool kEarly = MODE == kKin && E == 8 && T == 256;  // as RowIn
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = a.psi[base + (e * L + fft.t) * stride];
    if (kEarly && !a.kq_c) {
#pragma unroll
      for (int e = 0; e < E; ++e) kf[e] = a.K[base + (e * L + fft.t) * stride];
    }
    if (MODE != kInv) fft.forward(v, at, sync);
    if (MODE == kKin) {
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int f = base + (e * L + fft.t) * stride;
        if (a.kq_c) {
          // spofft.f:148-154 as written: V(I) uses the already updated U(I)
          const double kc = a.kq_c[f], ks = a.kq_s[f];
          const double un = kc * (double)v[e].x + ks * (double)v[e].y;
          const double vn = kc * (double)v[e].y - ks * un;
          v[e] = mk((R)(un * a.kq_scale), (R)(vn * a.kq_scale));
        } else {
          v[e] = apply_ph(kEarly ? kf[e] : a.K[f], v[e]);
        }
      }
    }
    if (MODE != kFwd) {
      fft.inverse(v, at, sync);
    }
#pragma unroll
    for (int e = 0; e < E; ++e) a.psi[base + (e * L + fft.t) * stride] = v[e];
    sync();
  }
}

// the kinetic pass with each group's next tile (state and factors) copied into
// shared memory while the current one is transformed: two buffers per group
// behind the exchange space.  Without the copies all warps load, transform and
// store in step and neither the memory nor the FP units stay busy: with them
// (and those of plane_rows) a 128^3 mixed step takes 57 us instead of 80
template <typename R, int LN, int T>
__device__ __noinline__ void kin_staged(const NdArgs<R>& a, int axis,
                                        const typename Rot<R>::type* tab, cpx<R>* sm) {
  using F = LineFft<R, LN>;
  using PhT = typename Ph<R>::type;
  constexpr int N = F::N, E = F::E, L = F::L;
  const int lc = a.lc, gt = L << lc, tid = threadIdx.x & (gt - 1);
  const int group = threadIdx.x / gt, ng = T / gt;
  const int c = threadIdx.x & ((1 << lc) - 1);
  cpx<R>* ex = sm + ((group * (N + N / 8)) << lc) + c;
  const int tile = (N << lc) * (int)(sizeof(cpx<R>) + sizeof(PhT));
  unsigned char* buf = reinterpret_cast<unsigned char*>(sm + T / L * (N + N / 8)) + 2 * group * tile;
  F fft;
  fft.init(tab, (threadIdx.x >> lc) & (L - 1));
  auto at = [&](int p) { return ex + (skew(p) << lc); };
  auto sync = [&]() { bar_group(1 + group, gt); };
  const int ltx = a.ln[0] - lc;
  const int stride = axis == 1 ? 1 << a.ln[0] : 1 << (a.ln[0] + a.ln[1]);
  const int lset = axis == 1 ? a.ln[0] + a.ln[1] : a.ln[0];
  const int items = (int)(a.n >> (LN + lc)), step = gridDim.x * ng;
  auto first = [&](int it) { return ((it >> ltx) << lset) + ((it & ((1 << ltx) - 1)) << lc); };
  auto fetch = [&](int it, int s) {
    unsigned char* d = buf + s * tile;
    const int b0 = first(it);
    const int pc = (int)(sizeof(cpx<R>) << lc) / 16, kc = (int)(sizeof(PhT) << lc) / 16;
    for (int i = tid; i < N * pc; i += gt) {
      const int r = i / pc;
      copy_async<16>(d + 16 * i, reinterpret_cast<const char*>(a.psi + b0 + r * stride) +
                                     16 * (i - r * pc));
    }
    d += (N << lc) * sizeof(cpx<R>);
    for (int i = tid; i < N * kc; i += gt) {
      const int r = i / kc;
      copy_async<16>(d + 16 * i, reinterpret_cast<const char*>(a.K + b0 + r * stride) +
                                     16 * (i - r * kc));
    }
  };
  int it = blockIdx.x + gridDim.x * group, s = 0;
  if (it < items) fetch(it, 0);
  copy_commit();
  for (; it < items; it += step, s ^= 1) {
    if (it + step < items) fetch(it + step, s ^ 1);
    copy_commit();
    copy_wait<1>();
    sync();
    const cpx<R>* x = reinterpret_cast<const cpx<R>*>(buf + s * tile) + c;
    const PhT* kf = reinterpret_cast<const PhT*>(buf + s * tile + (N << lc) * sizeof(cpx<R>)) + c;
    cpx<R> v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = x[(e * L + fft.t) << lc];
    fft.forward(v, at, sync);
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = apply_ph(kf[(e * L + fft.t) << lc], v[e]);
    fft.inverse(v, at, sync);
    const int base = first(it) + c;
#pragma unroll
    for (int e = 0; e < E; ++e) a.psi[base + (e * L + fft.t) * stride] = v[e];
    sync();
  }
}

// the columns of a plane in shared memory, in place (positions along y), the
// exchange through the lines' own places
template <typename R, int LN, bool INV, int THREADS>
__device__ __noinline__ void plane_cols(const NdArgs<R>& a, const typename Rot<R>::type* tab,
                                        cpx<R>* sm) {
  using F = LineFft<R, LN>;
  constexpr int E = F::E, L = F::L;
  // columns of a group: 128 bytes of them, within the CTA's threads
  constexpr int C = sizeof(R) == 4 && 16 * L <= THREADS ? 16 : 8, GT = C * L;
  const int nx = 1 << a.ln[0];
  const int group = threadIdx.x / GT, ng = blockDim.x / GT;
  F fft;
  fft.init(tab, (threadIdx.x / C) % L);
  auto sync = [&]() { bar_group(1 + group, GT); };
  for (int xt = group; xt < nx / C; xt += ng) {
    cpx<R>* col = sm + slot_of<R>(xt * C + threadIdx.x % C);
    auto at = [&](int p) { return col + p * nx; };
    cpx<R> v[E];
    constexpr int k0 = INV ? F::NG - 1 : 0, k1 = INV ? 0 : F::NG - 1;
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = *at(F::pos(k0, fft.t, e));
    if (INV) fft.inverse(v, at, sync);
    else fft.forward(v, at, sync);
#pragma unroll
    for (int e = 0; e < E; ++e) *at(F::pos(k1, fft.t, e)) = v[e];
  }
}

// the rows of a plane in shared memory, in place; behind the plane, 4 KB per warp
// for the rows' 16-byte inputs
template <typename R, int LN, int MODE, int T>
__device__ __noinline__ double2 plane_rows(const NdArgs<R>& a, const SodRow& o,
                                           const typename Rot<R>::type* tab, cpx<R>* sm,
                                           int plane) {
  using F = LineFft<R, LN>;
  constexpr int N = F::N, E = F::E, L = F::L, LW = 32 / L;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int ny = 1 << a.ln[1];
  F fft;
  fft.init(tab, lane % L);
  auto sync = [&]() { __syncwarp(); };
  double cr = 0.0, ci = 0.0;
  for (int y = warp * LW + lane / L; y < ny; y += nw * LW) {
    cpx<R>* row = sm + y * N;
    auto at = [&](int p) { return row + slot_of<R>(p); };
    const int base = ((plane << a.ln[1]) + y) << LN;
    cpx<R> v[E];
    RowIn<R, E, MODE, T, true> in;
    in.st = reinterpret_cast<double2*>(sm + (N << a.ln[1])) + warp * (32 * 8);
    if (row_inverse(MODE)) {
      in.early(a, o, base + fft.t, F::L);
#pragma unroll
      for (int e = 0; e < E; ++e) v[e] = *at(F::pos(F::NG - 1, fft.t, e));
      fft.inverse(v, at, sync);
    }
    row_points<R, LN, MODE, T, true>(a, o, v, in, fft, base, cr, ci);
    if (row_forward(MODE)) {
      fft.forward(v, at, sync);
#pragma unroll
      for (int e = 0; e < E; ++e) *at(F::pos(F::NG - 1, fft.t, e)) = v[e];
    }
  }
  return make_double2(cr, ci);
}

// runs f<LN>() for the line length 2^ln; MAXLN bounds the instantiations
template <int MAXLN, class F>
__device__ __forceinline__ void for_len(int ln, F f) {
  switch (ln) {
    case 5: f(std::integral_constant<int, 5>{}); break;
    case 6: f(std::integral_constant<int, 6>{}); break;
    case 7: f(std::integral_constant<int, 7>{}); break;
    case 8: if constexpr (MAXLN >= 8) f(std::integral_constant<int, 8>{}); break;
    default: if constexpr (MAXLN >= 9) f(std::integral_constant<int, 9>{}); break;
  }
}

// x pass of the whole grid, or with `fused` the x and y transforms of whole xy
// planes (y inverse, the x pass, y forward) in shared memory
template <typename R, int T, int MAXLN, int MODE>
__device__ __forceinline__ double2 x_phase(const NdArgs<R>& a, const SodRow& o,
                                           const typename Rot<R>::type* const* tab, cpx<R>* sm) {
  double2 c = make_double2(0.0, 0.0);
  if (!a.fused) {
    for_len<MAXLN>(a.ln[0], [&](auto ln) {
      c = rows_phase<R, decltype(ln)::value, MODE, T>(a, o, tab[0], sm);
    });
    return c;
  }
  const int lx = a.ln[0], lp = lx + a.ln[1];
  for (int z = blockIdx.x; z < (1 << a.ln[2]); z += gridDim.x) {
    cpx<R>* g = a.psi + ((long)z << lp);
    auto slot = [&](int i) {
    return sm + ((i >> lx) << lx) + slot_of<R>(i & ((1 << lx) - 1));
  };
    if (row_inverse(MODE)) {
#pragma unroll 8
      for (int i = threadIdx.x; i < (1 << lp); i += blockDim.x)
        copy_async<sizeof(cpx<R>)>(slot(i), g + i);
      copy_commit();
      copy_wait<0>();
      __syncthreads();
      for_len<MAXLN>(a.ln[1], [&](auto ln) {
        plane_cols<R, decltype(ln)::value, true, T>(a, tab[1], sm);
      });
      __syncthreads();
    }
    for_len<MAXLN>(lx, [&](auto ln) {
      const double2 d = plane_rows<R, decltype(ln)::value, MODE, T>(a, o, tab[0], sm, z);
      c.x += d.x;
      c.y += d.y;
    });
    if (row_forward(MODE)) {
      __syncthreads();
      for_len<MAXLN>(a.ln[1], [&](auto ln) {
        plane_cols<R, decltype(ln)::value, false, T>(a, tab[1], sm);
      });
      __syncthreads();
#pragma unroll 8
      for (int i = threadIdx.x; i < (1 << lp); i += blockDim.x) g[i] = *slot(i);
    }
    __syncthreads();
  }
  return c;
}

template <typename R, int T, int MAXLN, int MODE>
__device__ __forceinline__ void axis_phase(const NdArgs<R>& a, int axis,
                                           const typename Rot<R>::type* const* tab, cpx<R>* sm) {
  for_len<MAXLN>(a.ln[axis], [&](auto ln) {
    if constexpr (MODE == kKin && decltype(ln)::value <= 8) {
      if (a.kstage) {
        kin_staged<R, decltype(ln)::value, T>(a, axis, tab[axis], sm);
        return;
      }
    }
    cols_phase<R, decltype(ln)::value, MODE, T>(a, axis, tab[axis], sm);
  });
}

// End of a pass: with step >= 0 the CTA's C(t) partial sum of that step, then
// (unless it is the last pass) a grid barrier.  Thread 0's arrival is a
// release ordered after the CTA's writes by bar.sync; every arrival continues
// the release sequence of the earlier ones, so the acquire load that sees the
// last one synchronises with all.  false: a wait gave up.
template <typename R>
__device__ __forceinline__ bool end_pass(const NdArgs<R>& a, double2 c, int step, bool last,
                                         unsigned& passed, double2* s_c, int* s_ok) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (step >= 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      c.x += __shfl_xor_sync(kFull, c.x, o);
      c.y += __shfl_xor_sync(kFull, c.y, o);
    }
    if (lane == 0) s_c[warp] = c;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    *s_ok = 1;
    if (!last && gridDim.x > 1) {
      asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(a.bar), "l"(1ull) : "memory");
      const unsigned long long target = (unsigned long long)(passed + 1u) * gridDim.x;
      cuda::atomic_ref<unsigned long long, cuda::thread_scope_device> cnt(*a.bar);
      cuda::atomic_ref<int, cuda::thread_scope_device> err(*a.err);
      long spins = 0;
      while (cnt.load(cuda::memory_order_acquire) < target) {
        if (++spins > a.spin_limit || err.load(cuda::memory_order_relaxed) != 0) {
          err.store(1, cuda::memory_order_relaxed);
          *s_ok = 0;
          break;
        }
        if (spins > 4096) __nanosleep(32);
      }
    }
  } else if (warp == 1 && step >= 0) {  // beside the wait: no other CTA reads the sum
    double2 t = lane < (int)(blockDim.x >> 5) ? s_c[lane] : make_double2(0.0, 0.0);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      t.x += __shfl_xor_sync(kFull, t.x, o);
      t.y += __shfl_xor_sync(kFull, t.y, o);
    }
    if (lane == 0) a.cpart[(long)step * gridDim.x + blockIdx.x] = t;
  }
  ++passed;
  __syncthreads();
  return *s_ok != 0;
}

// A whole run in one cooperative launch: the passes of every step separated by
// grid barriers.  The state (1 MB for 256 x 256 FP64) stays in L2, and a pass
// of a small grid is a chain of latencies: one launch per pass cost 9 us each
// (launch, table loads and one warp per SM), a pass here about a third.
template <typename R, int T, int MAXLN>
__global__ void __launch_bounds__(T, 1) nd_kernel(const NdArgs<R> ga) {
  extern __shared__ __align__(16) unsigned char nd_raw[];
  __shared__ NdArgs<R> a;
  __shared__ double2 s_c[T / 32];
  __shared__ int s_ok;
  using Tw = typename Rot<R>::type;
  if (threadIdx.x == 0) a = ga;
  // the axes' twiddles, then the exchange space
  Tw* tab[3];
  Tw* next = reinterpret_cast<Tw*>(nd_raw);
  for (int ax = 0; ax < ga.ndim; ++ax) {
    tab[ax] = next;
    for_len<MAXLN>(ga.ln[ax], [&](auto ln) {
      using F = LineFft<R, decltype(ln)::value>;
      F::pack(ga.tw[ax], next);
      next += F::count() * F::L;
    });
  }
  if (ga.ndim < 3) tab[2] = tab[1];
  cpx<R>* sm = reinterpret_cast<cpx<R>*>(next);
  __syncthreads();
  unsigned passed = 0;
  const double2 zero = make_double2(0.0, 0.0);
  auto fence = [&](double2 c, int step, bool last) {
    return end_pass<R>(a, c, step, last, passed, s_c, &s_ok);
  };
  // the passes between two x passes
  auto kin = [&]() -> bool {
    if (a.ndim == 2) {
      axis_phase<R, T, MAXLN, kKin>(a, 1, tab, sm);
      return fence(zero, -1, false);
    }
    if (!a.fused) {
      axis_phase<R, T, MAXLN, kFwd>(a, 1, tab, sm);
      if (!fence(zero, -1, false)) return false;
    }
    axis_phase<R, T, MAXLN, kKin>(a, 2, tab, sm);
    if (!fence(zero, -1, false)) return false;
    if (!a.fused) {
      axis_phase<R, T, MAXLN, kInv>(a, 1, tab, sm);
      return fence(zero, -1, false);
    }
    return true;
  };
  SodRow o{};
  if (a.op == kOpSpo) {
    double2 c = x_phase<R, T, MAXLN, kFirst>(a, o, tab, sm);
    if (!fence(c, 0, a.nsteps == 0)) return;
    for (int s = 1; s <= a.nsteps; ++s) {
      if (!kin()) return;
      const bool end = s == a.nsteps;
      c = end ? x_phase<R, T, MAXLN, kLast>(a, o, tab, sm) : x_phase<R, T, MAXLN, kMid>(a, o, tab, sm);
      if (!fence(c, s, end)) return;
    }
  } else if (a.op == kOpForward) {
    x_phase<R, T, MAXLN, kFwd0>(a, o, tab, sm);
    if (!a.fused) {
      if (!fence(zero, -1, false)) return;
      axis_phase<R, T, MAXLN, kFwd>(a, 1, tab, sm);
    }
    if (a.ndim == 3) {
      if (!fence(zero, -1, false)) return;
      axis_phase<R, T, MAXLN, kFwd>(a, 2, tab, sm);
    }
  } else if constexpr (sizeof(R) == 8) {  // SOD plans are FP64
    // every update's new state is the next one's source: its row is
    // transformed in the same pass.  The start-up (psodfft.f:120-152) is two
    // half steps from psi0 and then psi(t - dt) = psi0.
    const int updates = a.nsteps + (a.from_start && a.nsteps > 0 ? 1 : 0);
    double2* buf[2] = {a.prev, a.cur};
    double2 c = x_phase<R, T, MAXLN, kFwd0>(a, o, tab, sm);
    if (!fence(c, a.from_start ? 0 : -1, updates == 0)) return;
    for (int u = 0; u < updates; ++u) {
      if (!kin()) return;
      o.src = u == 0 ? a.psi_start : buf[(u & 1) ^ 1];
      o.dst = buf[u & 1];
      o.old = a.from_start && u < 3 ? a.psi0 : o.dst;
      o.f = a.from_start && u < 2 ? 0.5 : 1.0;
      const bool end = u + 1 == updates;
      c = end ? x_phase<R, T, MAXLN, kUpd>(a, o, tab, sm) : x_phase<R, T, MAXLN, kUpdFwd>(a, o, tab, sm);
      // updates 0 and 1 both lead to step 1; the sample is the second's
      const int step = a.from_start ? (u == 0 ? -1 : u) : u + 1;
      if (!fence(c, step, end)) return;
    }
  }
}

// one cooperative launch over `grid` CTAs with smem bytes of dynamic shared memory
template <typename R, int T, int MAXLN>
cudaError_t nd_kernel_launch(const NdArgs<R>& a, int grid, size_t smem, cudaStream_t st) {
  static DeviceFlags attr;
  const cudaError_t e = set_max_smem_once(attr, nd_kernel<R, T, MAXLN>, kNdMaxSmem);
  if (e != cudaSuccess) return e;
  NdArgs<R> b = a;
  void* args[] = {&b};
  return cudaLaunchCooperativeKernel((const void*)nd_kernel<R, T, MAXLN>, dim3(grid), dim3(T), args,
                                     smem, st);
}

// longest line (log2) of the 512-thread form
template <typename R>
constexpr int kMaxLn512 = sizeof(R) == 8 ? 7 : 8;

cudaError_t nd_launch_f64_256(const NdArgs<double>& a, int grid, size_t smem, cudaStream_t st);
cudaError_t nd_launch_f64_512(const NdArgs<double>& a, int grid, size_t smem, cudaStream_t st);
cudaError_t nd_launch_f32_256(const NdArgs<float>& a, int grid, size_t smem, cudaStream_t st);
cudaError_t nd_launch_f32_512(const NdArgs<float>& a, int grid, size_t smem, cudaStream_t st);

}  // namespace nd
}  // namespace espec
