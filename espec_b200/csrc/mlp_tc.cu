// mlp_tc.cu -- the warm-start network's products on the 5th-generation tensor
// cores, and the element-wise kernels of its BF16 training step.
//
// The network (5 potential parameters -> 3 x 256 GELU -> coefficients of the
// four lowest eigenvectors) keeps FP32 master weights and trains with BF16
// copies of weights, activations and back-propagated gradients as GEMM
// operands; every product accumulates in FP32.
//
// GEMM: C[M,N] (f32) = alpha op(A) op(B) + beta C, A and B bfloat16.  One CTA owns a
// 128 x BN output tile whose FP32 accumulator lives in tensor memory (TMEM lane =
// tile row, column = tile column).  K advances in stages of 64 through a ring of
// shared-memory buffers: one thread fetches the A and B tiles by TMA
// (gemm_bf16_tma), or 256 threads copy them where TMA's alignment rules do not hold
// (gemm_bf16_tc); one thread issues four tcgen05.mma (M = 128, N = BN, K = 16,
// kind::f16 with BF16 inputs) per stage and commits them to the buffer's mbarrier.
// BN is the largest of 256, 128, 64 that gives every SM a tile more than half full,
// else 32 (launch_any): the network's products have few tiles, and what bounds them is
// the chain of stages.
// The epilogue reads the accumulator with tcgen05.ld (a warp: 32 TMEM lanes, 32
// columns) and turns it in shared memory so that rows are written 128 bytes at a
// time, adding the bias and the activation (or its derivative) on the way.  Every
// mbarrier wait is bounded: on timeout the kernel records it in a device status
// word, skips the epilogue and still releases its TMEM.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "chain.cuh"
#include "espec_gpu.h"
#include "espec_internal.h"

namespace espec {
namespace {

constexpr int kBM = 128;         // tile rows = TMEM lanes
constexpr int kBK = 64;          // k per stage: four MMAs of k = 16
constexpr int kTcThreads = 256;  // staging and epilogue: warp w reads TMEM lanes 32 (w % 4) ...
constexpr int kTcBlock = kTcThreads + 32;  // and one warp that issues the MMAs
constexpr long kWaitLimit = 1L << 22;

__device__ int g_tc_status;  // non-zero: a bounded wait gave up (sticky until read)

struct TcGemm {
  int M, N, K;
  float alpha, beta;
  const uint16_t* A;
  int lda, ta;
  const uint16_t* B;
  int ldb, tb;
  float* C;
  int ldc;
  int a_vec, b_vec;  // 16-byte loads allowed: ld % 8 == 0 and a 16-byte aligned base
  // epilogue kBias: C = acc + bias (row), h = bf16(act ? gelu(C) : C);
  // kGeluBack: C = acc gelu'(z), h = bf16(C)
  const float* bias;
  const float* z;
  uint16_t* h;
  int act;
};
enum { kPlain = 0, kBias = 1, kGeluBack = 2 };

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// shared-memory matrix descriptor of a K-major, no-swizzle operand: start
// address, leading byte offset (between the two 8-element k chunks of one
// MMA), stride byte offset (between 8-row groups), descriptor version 1
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) |
         ((uint64_t)(sbo >> 4) << 32) | (1ull << 46);
}

// instruction descriptor: FP32 accumulator, BF16 A and B, A / B K-major (0)
// or MN-major (1) at bits 15 / 16, N >> 3 at bit 17, M >> 4 at bit 24
template <int BN>
__host__ __device__ constexpr uint32_t idesc_bf16(uint32_t a_mn, uint32_t b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (a_mn << 15) | (b_mn << 16) |
         ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
}

__device__ __forceinline__ uint32_t pack2(uint16_t lo, uint16_t hi) {
  return (uint32_t)lo | ((uint32_t)hi << 16);
}

// Operand tile of R rows (M or N) x 64 k as 8 x 8 core matrices of 16-byte rows:
//  * kcontig source (element (row, k) at X[row ld + k]): K-major core matrices,
//    16-byte row = 8 consecutive k of one row; 128 bytes between row groups (the
//    stride byte offset), 16 R + 16 between k groups (the leading byte offset);
//  * otherwise (element at X[k ld + row]): MN-major core matrices, 16-byte row = 8
//    consecutive rows at one k; 144 bytes between row groups, 18 R between k
//    groups.
// Either way a 16-byte row is 16 contiguous source bytes, one copy when vec
// (aligned; the part beyond nrows or K is zero-filled), else element by element.
// Consecutive threads take consecutive 16-byte pieces of the source, whole 128-byte
// lines per eight threads; the odd group strides put those pieces on distinct banks.
// A thread's pieces keep their places from stage to stage: their addresses and
// sizes are formed once and then advance by a constant.
template <int R>
__host__ __device__ constexpr uint32_t lead_bytes(bool kcontig) {
  return kcontig ? R * 16 + 16 : R * 18;
}
__host__ __device__ constexpr uint32_t stride_bytes(bool kcontig) { return kcontig ? 128 : 144; }
template <int R>
constexpr int kTileBytes = R * 18 * (kBK / 8);
template <int R>
struct Stager {
  static constexpr int kIter = (R * (kBK / 8) + kTcThreads - 1) / kTcThreads;  // pieces per thread
  const uint16_t* src[kIter];
  int cnt[kIter];  // elements that exist: along k (kcontig: at stage 0), else along the rows
  int k[kIter];    // first k of the piece, stage 0
  long step;       // elements from stage to stage
  bool kcontig, vec;
  int K;
  static __device__ __forceinline__ bool live(int i) {
    return R * (kBK / 8) % kTcThreads == 0 || (int)threadIdx.x + i * kTcThreads < R * (kBK / 8);
  }
  static __device__ __forceinline__ int place(int i, bool kcontig) {
    const int it = threadIdx.x + i * kTcThreads;
    const int row = it >> 3, g = it % (R / 8), kk = it / (R / 8);
    return kcontig ? (it & 7) * (int)lead_bytes<R>(true) + (row >> 3) * 128 + (row & 7) * 16
                   : (kk >> 3) * (int)lead_bytes<R>(false) + g * 144 + (kk & 7) * 16;
  }
  __device__ __forceinline__ void init(const uint16_t* X, int ld, bool kc, bool v, int row0,
                                       int nrows, int K_) {
    kcontig = kc;
    vec = v;
    K = K_;
    step = kc ? kBK : (long)kBK * ld;
#pragma unroll
    for (int i = 0; i < kIter; ++i) {
      const int it = threadIdx.x + i * kTcThreads;
      if (kc) {
        const int row = row0 + (it >> 3);
        k[i] = 8 * (it & 7);
        cnt[i] = row < nrows ? 8 : 0;
        src[i] = X + (cnt[i] ? (long)row * ld + k[i] : 0);
      } else {
        const int m = row0 + 8 * (it % (R / 8));
        k[i] = it / (R / 8);
        cnt[i] = min(max(nrows - m, 0), 8);
        src[i] = X + (cnt[i] ? (long)k[i] * ld + m : 0);
      }
    }
  }
  // stage kt into dst
  __device__ __forceinline__ void stage(uint8_t* dst, int kt) const {
#pragma unroll
    for (int i = 0; i < kIter; ++i) {
      if (!live(i)) continue;
      const int left = K - kt * kBK - k[i];  // values of k from the piece's first on
      const int n = kcontig ? (cnt[i] ? min(max(left, 0), 8) : 0) : (left > 0 ? cnt[i] : 0);
      // an empty piece reads nothing: any valid address (src's first element)
      const uint16_t* p = n > 0 ? src[i] + kt * step : src[i];
      uint8_t* d = dst + place(i, kcontig);
      if (vec) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(d)), "l"(p),
                     "r"(2 * n)
                     : "memory");
      } else {
        uint16_t e[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) e[j] = j < n ? p[j] : (uint16_t)0;
        *reinterpret_cast<uint4*>(d) = make_uint4(pack2(e[0], e[1]), pack2(e[2], e[3]),
                                                  pack2(e[4], e[5]), pack2(e[6], e[7]));
      }
    }
  }
};

// bounded wait for the completion of the mbarrier phase with this parity
__device__ __forceinline__ bool wait_phase(uint64_t* bar, uint32_t parity,
                                           long limit = kWaitLimit) {
  const uint32_t a = smem_u32(bar);
  for (long i = 0; i < limit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
    if (i > 64) __nanosleep(64);
  }
  atomicExch(&g_tc_status, 1);
  return false;
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

__device__ __forceinline__ uint16_t bf16_bits(float v) {
  return __bfloat16_as_ushort(__float2bfloat16_rn(v));
}

// GELU(z) = z Phi(z), Phi the standard normal distribution function
__device__ __forceinline__ float gelu(float z) {
  return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f));
}
__device__ __forceinline__ float gelu_grad(float z) {
  return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) +
         z * 0.39894228040143268f * expf(-0.5f * z * z);
}

constexpr int kCopyRing = 4;  // stage buffers
template <int BN>
constexpr size_t tc_smem_bytes() {
  return 1024 + kCopyRing * (size_t)(kTileBytes<kBM> + kTileBytes<BN>) + 192;
}

// What follows the MMAs of a tile: wait for the last commit, write the tile, give
// the tensor memory back.  Warp 8 issued the MMAs; `turn` space: the stage buffers.
template <int BN, int EPI>
__device__ __forceinline__ void finish_tile(const TcGemm& g, uint32_t tmem, uint8_t* base,
                                            uint64_t* last, uint32_t parity, bool some, bool ok,
                                            int m0, int n0) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool mma_warp = warp == kTcThreads / 32;
  __syncwarp();
  // warp w: rows 32 (w % 4) of the tile, columns from 32 (w / 4) on, 64 apart
  const int row0 = m0 + (warp & 3) * 32, col0 = (warp >> 2) * 32;
  // the first columns' pre-activations, on their way while the last MMAs run
  float zf[EPI == kGeluBack ? 32 : 1];
  if (EPI == kGeluBack) {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      zf[i] = !mma_warp && col0 < BN && row0 + i < g.M && n0 + col0 + lane < g.N
                  ? g.z[(long)(row0 + i) * g.ldc + n0 + col0 + lane]
                  : 0.0f;
  }
  // The last commit covers every MMA before it.  Where the MMA thread gave up at an
  // earlier stage nobody makes that commit, and all threads stay here for the whole
  // limit: the wait for the boxes and MMAs still in flight.
  // (With tiles by TMA, warps 1 to 7 have followed no phase and may take an earlier one
  // for the last: it is the barrier they wait at, which the MMA thread reaches after its
  // own wait, and the fence has to follow it.)
  if (some) ok = wait_phase(last, parity) && ok;
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  ok = __syncthreads_and(ok) != 0;
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  if (ok && !mma_warp) {
    // 32 columns at a time: each warp's 32 x 32 piece through shared memory
    float* turn = reinterpret_cast<float*>(base) + warp * (32 * 33);
#pragma unroll 1
    for (int c0 = col0; c0 < BN; c0 += 64) {
      uint32_t r[32];
      if (some) {
        tmem_ld32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0, r);
      } else {  // empty sum
#pragma unroll
        for (int j = 0; j < 32; ++j) r[j] = 0u;
      }
#pragma unroll
      for (int j = 0; j < 32; ++j) turn[lane * 33 + j] = __uint_as_float(r[j]);
      __syncwarp();
      const int n = n0 + c0 + lane;
      const float bias = EPI == kBias && n < g.N ? g.bias[n] : 0.0f;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const int row = row0 + i;
        if (row < g.M && n < g.N) {
          const long o = (long)row * g.ldc + n;
          float v = turn[i * 33 + lane];
          if (EPI == kPlain) {
            v = g.alpha * v;
            if (g.beta != 0.0f) v = some ? fmaf(g.beta, g.C[o], v) : g.beta * g.C[o];
            else if (!some) v = 0.0f;
          } else if (EPI == kBias) {
            v = v + bias;
            if (g.h) g.h[o] = bf16_bits(g.act ? gelu(v) : v);
          } else {
            v = v * gelu_grad(c0 == col0 ? zf[i] : g.z[o]);
            g.h[o] = bf16_bits(v);
          }
          g.C[o] = v;
        }
      }
      __syncwarp();
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (mma_warp)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(BN));
}

template <int BN, int EPI>
__global__ void __launch_bounds__(kTcBlock) gemm_bf16_tc(TcGemm g) {
  static_assert(BN == 32 || BN == 64 || BN == 128 || BN == 256,
                "TMEM columns: a power of two from 32, N tile of one MMA");
  constexpr int kA = kTileBytes<kBM>, kB = kTileBytes<BN>, kRing = kCopyRing;
  static_assert(kRing * kA >= kTcThreads * 33 * 4, "the epilogue turns tiles in the stage buffers");
  chain_start();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sA = base;
  uint8_t* sB = base + kRing * kA;
  uint64_t* full = (uint64_t*)(base + kRing * (kA + kB));  // a buffer's copies have landed
  uint64_t* done = full + kRing;                           // its MMAs have read it
  uint32_t* tmem_slot = (uint32_t*)(done + kRing);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.y * kBM, n0 = blockIdx.x * BN;
  const bool a_kc = !g.ta, b_kc = g.tb != 0, mma_warp = warp == kTcThreads / 32;
  const int nk = (g.K + kBK - 1) / kBK;

  if (threadIdx.x == 0) {
    for (int b = 0; b < kRing; ++b) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(full + b)),
                   "r"(kTcThreads));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(done + b)));
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (mma_warp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  chain_wait();
  bool ok = true;
  if (!mma_warp) {
    Stager<kBM> ta;
    Stager<BN> tb;
    ta.init(g.A, g.lda, a_kc, g.a_vec, m0, g.M, g.K);
    tb.init(g.B, g.ldb, b_kc, g.b_vec, n0, g.N, g.K);
    for (int kt = 0; kt < nk; ++kt) {
      const int b = kt % kRing;
      if (kt >= kRing && !(ok = wait_phase(done + b, (kt / kRing - 1) & 1))) break;
      ta.stage(sA + b * kA, kt);
      tb.stage(sB + b * kB, kt);
      asm volatile("cp.async.wait_all;\n" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.shared::cta.b64 t, [%0];\n\t}\n" ::"r"(
                       smem_u32(full + b))
                   : "memory");
    }
  } else if (lane == 0) {
    const uint32_t idesc = idesc_bf16<BN>(a_kc ? 0u : 1u, b_kc ? 0u : 1u);
    const uint32_t a_lead = lead_bytes<kBM>(a_kc), b_lead = lead_bytes<BN>(b_kc);
    for (int kt = 0; kt < nk; ++kt) {
      const int b = kt % kRing;
      if (!(ok = wait_phase(full + b, (kt / kRing) & 1))) break;
      const uint32_t a0 = smem_u32(sA + b * kA), b0 = smem_u32(sB + b * kB);
#pragma unroll
      for (int j = 0; j < kBK / 16; ++j) {
        const uint64_t da = smem_desc(a0 + j * 2 * a_lead, a_lead, stride_bytes(a_kc));
        const uint64_t db = smem_desc(b0 + j * 2 * b_lead, b_lead, stride_bytes(b_kc));
        const uint32_t acc = (kt > 0 || j > 0) ? 1u : 0u;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
            "l"(da), "l"(db), "r"(idesc), "r"(acc));
      }
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
              smem_u32(done + b))
          : "memory");
    }
  }
  finish_tile<BN, EPI>(g, tmem, base, done + (nk - 1) % kRing, ((nk - 1) / kRing) & 1, nk > 0, ok,
                       m0, n0);
}

// The same product with tiles brought by TMA, for operands whose base and rows are
// 16-byte aligned.  What bounds the network's products is the chain of stages of
// one CTA (16 tiles of 128 x 32 at 256 x 256), and copies by 256 threads, which
// wait, form addresses, issue 16-byte pieces and arrive at every stage, drew 25 GB/s
// per SM.  Here one thread asks for boxes of 64 k and the ring of stages stays in
// flight.  The MMAs, their order and the sums are those of gemm_bf16_tc.
// Against an asynchronous ring filled by the threads (us, before -> now):
// 256 x 256 x 256 7.7 -> 5.6 (4.9 as part of a chain, chain.cuh), 256 x 256 x 1024 16.6 -> 9.7, 256 x 256 x 4096
// 51 -> 25, 2048 x 4096 x 256 35 -> 23, 1024 x 1024 x 1024 32 -> 18.
//
// Tiles in shared memory, op(X) of R rows x 64 k:
//  * K-major source: one box, R rows of 64 k (128 bytes, 128-byte swizzle); 1024
//    bytes between groups of 8 rows;
//  * MN-major source: R / 64 boxes of 64 k rows of 64 row values each (128-byte
//    swizzle); 8 KB between boxes, 1024 bytes between groups of 8 k; for R = 32 one
//    box of 64-byte rows (64-byte swizzle), 512 bytes between groups of 8 k.
template <int R>
constexpr int kBoxBytes = R * kBK * 2;
template <int BN, int RING>
constexpr size_t tma_smem_bytes() {
  return 1024 + RING * (size_t)(kBoxBytes<kBM> + kBoxBytes<BN>) + 192;
}

// descriptor of the 16 k from 16 j on of the tile at addr
template <int R>
__device__ __forceinline__ uint64_t box_desc(uint32_t addr, bool kcontig, int j) {
  const uint32_t at = addr + (kcontig ? 32 : (R == 32 ? 1024 : 2048)) * j;
  const uint32_t lead = 64 * kBK * 2, stride = !kcontig && R == 32 ? 512 : 1024;
  const uint64_t swizzle = !kcontig && R == 32 ? 4 : 2;
  return (uint64_t)((at & 0x3FFFFu) >> 4) | ((uint64_t)(lead >> 4) << 16) |
         ((uint64_t)(stride >> 4) << 32) | (1ull << 46) | (swizzle << 61);
}

// the map's box from (x, y) on; x is a multiple of 32 values, so the copy starts on
// a 16-byte boundary
__device__ __forceinline__ void tma_box(void* dst, const CUtensorMap* map, int x, int y,
                                        uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3}], [%4];\n" ::"r"(smem_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

template <int R>
__device__ __forceinline__ void tma_tile(uint8_t* dst, const CUtensorMap* map, bool kcontig, int k0,
                                         int row0, uint64_t* bar) {
  if (kcontig) {
    tma_box(dst, map, k0, row0, bar);
  } else {
#pragma unroll
    for (int r = 0; r < R; r += 64) tma_box(dst + r * kBK * 2, map, row0 + r, k0, bar);
  }
}

template <int BN, int EPI, int RING>
__global__ void __launch_bounds__(kTcBlock)
    gemm_bf16_tma(const TcGemm g, const __grid_constant__ CUtensorMap map_a,
                  const __grid_constant__ CUtensorMap map_b) {
  constexpr int kA = kBoxBytes<kBM>, kB = kBoxBytes<BN>, kRing = RING;
  static_assert(kRing * kA >= kTcThreads * 33 * 4, "the epilogue turns tiles in the stage buffers");
  chain_start();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sA = base;
  uint8_t* sB = base + kRing * kA;
  uint64_t* full = (uint64_t*)(base + kRing * (kA + kB));  // a buffer's boxes have landed
  uint64_t* done = full + kRing;                                 // its MMAs have read it
  uint32_t* tmem_slot = (uint32_t*)(done + kRing);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.y * kBM, n0 = blockIdx.x * BN;
  const bool a_kc = !g.ta, b_kc = g.tb != 0, mma_warp = warp == kTcThreads / 32;
  const int nk = (g.K + kBK - 1) / kBK;

  if (threadIdx.x == 0) {
    for (int b = 0; b < kRing; ++b) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(full + b)));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(done + b)));
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (mma_warp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  chain_wait();
  bool ok = true;
  if (threadIdx.x == 0) {
    int kt = 0;
    for (; kt < nk; ++kt) {
      const int b = kt % kRing;
      if (kt >= kRing && !(ok = wait_phase(done + b, (kt / kRing - 1) & 1))) break;
      asm volatile(
          "{\n\t.reg .b64 t;\n\t"
          "mbarrier.arrive.expect_tx.shared::cta.b64 t, [%0], %1;\n\t}\n" ::"r"(smem_u32(full + b)),
          "r"(kA + kB)
          : "memory");
      tma_tile<kBM>(sA + b * kA, &map_a, a_kc, kt * kBK, m0, full + b);
      tma_tile<BN>(sB + b * kB, &map_b, b_kc, kt * kBK, n0, full + b);
    }
    // after a wait that gave up: the boxes still on their way
    if (!ok)
      for (int j = kt > kRing ? kt - kRing : 0; j < kt; ++j)
        wait_phase(full + j % kRing, (j / kRing) & 1);
  } else if (mma_warp && lane == 0) {
    const uint32_t idesc = idesc_bf16<BN>(a_kc ? 0u : 1u, b_kc ? 0u : 1u);
    for (int kt = 0; kt < nk; ++kt) {
      const int b = kt % kRing;
      if (!(ok = wait_phase(full + b, (kt / kRing) & 1))) break;
      const uint32_t a0 = smem_u32(sA + b * kA), b0 = smem_u32(sB + b * kB);
#pragma unroll
      for (int j = 0; j < kBK / 16; ++j) {
        const uint64_t da = box_desc<kBM>(a0, a_kc, j), db = box_desc<BN>(b0, b_kc, j);
        const uint32_t acc = (kt > 0 || j > 0) ? 1u : 0u;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
            "l"(da), "l"(db), "r"(idesc), "r"(acc));
      }
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
              smem_u32(done + b))
          : "memory");
    }
  }
  finish_tile<BN, EPI>(g, tmem, base, done + (nk - 1) % kRing, ((nk - 1) / kRing) & 1, nk > 0,
                           ok, m0, n0);
}

// z += b (row broadcast); h = bf16(gelu(z)) when act, else bf16(z) (h optional)
__global__ void bias_gelu_kernel(float* z, const float* b, int rows, int cols, int act,
                                 uint16_t* h) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long)rows * cols) return;
  const float v = z[i] + b[i % cols];
  z[i] = v;
  if (h) h[i] = bf16_bits(act ? gelu(v) : v);
}

// dh <- dh gelu'(z); dzb = bf16(dh)
__global__ void gelu_back_kernel(float* dh, const float* z, long count, uint16_t* dzb) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const float d = dh[i] * gelu_grad(z[i]);
  dh[i] = d;
  dzb[i] = bf16_bits(d);
}

template <bool CHAIN>
__global__ void to_bf16_kernel(const float* x, uint16_t* y, long count) {
  if (CHAIN) {
    chain_start();
    chain_wait();
  }
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) y[i] = bf16_bits(x[i]);
}

// Adam on the FP32 master weights, (lr, 1 - b1^t, 1 - b2^t) from device memory,
// and the BF16 copy the products use
__global__ void adam_bf16_kernel(float* w, const float* g, float* m1, float* m2, long count,
                                 const float* hyper, float b1, float b2, float eps, uint16_t* wb) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const float lr = hyper[0], c1 = hyper[1], c2 = hyper[2];
  const float gi = g[i];
  const float a = b1 * m1[i] + (1.0f - b1) * gi;
  const float b = b2 * m2[i] + (1.0f - b2) * gi * gi;
  m1[i] = a;
  m2[i] = b;
  const float nw = w[i] - lr * (a / c1) / (sqrtf(b / c2) + eps);
  w[i] = nw;
  if (wb) wb[i] = bf16_bits(nw);
}

inline unsigned nblk(long count) { return (unsigned)((count + 255) / 256); }

// tensor map of op(X), `rows` x K, as it lies (tma_tile's boxes)
bool operand_map(CUtensorMap* map, const uint16_t* X, int ld, bool kcontig, int rows, int K,
                 int tile_rows) {
  using Encode = decltype(&cuTensorMapEncodeTiled);
  static const Encode encode = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q{};
    const cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000,
                                                           cudaEnableDefault, &q);
    return e == cudaSuccess && q == cudaDriverEntryPointSuccess ? (Encode)fn : (Encode) nullptr;
  }();
  if (!encode) return false;
  const cuuint64_t dim[2] = {(cuuint64_t)(kcontig ? K : rows), (cuuint64_t)(kcontig ? rows : K)};
  const cuuint64_t stride[1] = {2 * (cuuint64_t)ld};
  const cuuint32_t box[2] = {(cuuint32_t)(kcontig ? kBK : std::min(tile_rows, 64)),
                             (cuuint32_t)(kcontig ? tile_rows : kBK)};
  const cuuint32_t one[2] = {1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<uint16_t*>(X), dim, stride,
                box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                box[0] == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN, int EPI, int RING>
int launch_tma(const TcGemm& g, const CUtensorMap& ma, const CUtensorMap& mb, cudaStream_t st) {
  static DeviceFlags attr;
  constexpr size_t smem = tma_smem_bytes<BN, RING>();
  const cudaError_t a = set_max_smem_once(attr, gemm_bf16_tma<BN, EPI, RING>, smem);
  if (a != cudaSuccess) return set_cuda_error("cudaFuncSetAttribute", a);
  const dim3 grid((g.N + BN - 1) / BN, (g.M + kBM - 1) / kBM);
  const cudaError_t e =
      launch_chained(gemm_bf16_tma<BN, EPI, RING>, grid, kTcBlock, smem, st, g, ma, mb);
  if (e != cudaSuccess) return set_cuda_error("tensor-core GEMM launch", e);
  return ESPEC_OK;
}

// TMA wherever a tensor map can describe the operands (base and rows at multiples of
// 16 bytes): it was the faster form at every size measured (gemm_bf16_tma).  The
// ring: 8 stages of a narrow tile where K has more than 4 (an L2 round trip is several
// stages long), else 4, which lets two CTAs share an SM.
template <int BN, int EPI>
int launch_tc(const TcGemm& g, cudaStream_t st) {
  if (g.K > 0 && g.a_vec && g.b_vec) {
    CUtensorMap ma, mb;
    if (operand_map(&ma, g.A, g.lda, !g.ta, g.M, g.K, kBM) &&
        operand_map(&mb, g.B, g.ldb, g.tb != 0, g.N, g.K, BN)) {
      if (BN <= 64 && g.K > 4 * kBK) return launch_tma<BN, EPI, BN <= 64 ? 8 : 4>(g, ma, mb, st);
      return launch_tma<BN, EPI, 4>(g, ma, mb, st);
    }
  }
  static DeviceFlags attr;
  constexpr size_t smem = tc_smem_bytes<BN>();
  const cudaError_t a = set_max_smem_once(attr, gemm_bf16_tc<BN, EPI>, smem);
  if (a != cudaSuccess) return set_cuda_error("cudaFuncSetAttribute", a);
  const dim3 grid((g.N + BN - 1) / BN, (g.M + kBM - 1) / kBM);
  const cudaError_t e = launch_chained(gemm_bf16_tc<BN, EPI>, grid, kTcBlock, smem, st, g);
  if (e != cudaSuccess) return set_cuda_error("tensor-core GEMM launch", e);
  return ESPEC_OK;
}

// the widest tiles that still give every SM one, of whose columns more than half exist:
// else the next narrower tile does the same work with half the MMA, copies and shared
// memory.  us per product with the tile of 256 columns and now: 20000 x 16 x 256 20.6 ->
// 8.9, 65536 x 64 x 256 40.8 -> 13.1, 65536 x 128 x 256 41.5 -> 28.4, 262144 x 100 x 64
// 163 -> 112; 20000 x 160 x 256 keeps it, 20.8.
template <int EPI>
int launch_any(const TcGemm& g, cudaStream_t st) {
  auto tiles = [&](int bn) {
    return (long)((g.N + bn - 1) / bn) * ((g.M + kBM - 1) / kBM);
  };
  if (g.N > 128 && tiles(256) >= 148) return launch_tc<256, EPI>(g, st);
  if (g.N > 64 && tiles(128) >= 148) return launch_tc<128, EPI>(g, st);
  if (g.N > 32 && tiles(64) >= 148) return launch_tc<64, EPI>(g, st);
  return launch_tc<32, EPI>(g, st);
}

inline int vec_ok(const void* p, int ld) { return ld % 8 == 0 && ((uintptr_t)p & 15) == 0; }

}  // namespace
}  // namespace espec

using namespace espec;

#define TC_CK()                                                                \
  do {                                                                         \
    cudaError_t e_ = cudaGetLastError();                                       \
    if (e_ != cudaSuccess) return set_cuda_error("mlp bf16 kernel launch", e_); \
  } while (0)

extern "C" int espec_gemm_bf16(int M, int N, int K, float alpha, const void* A, int lda, int ta,
                               const void* B, int ldb, int tb, float beta, float* C, int ldc,
                               void* stream) {
  if (M <= 0 || N <= 0 || K < 0 || !C || (K > 0 && (!A || !B)))
    return set_error(ESPEC_EINVAL, "bad GEMM");
  if (lda < (ta ? M : K) || ldb < (tb ? K : N) || ldc < N)
    return set_error(ESPEC_EINVAL, "leading dimension smaller than the row length");
  TcGemm g{M, N, K, alpha, beta, (const uint16_t*)A, lda, ta ? 1 : 0, (const uint16_t*)B, ldb,
           tb ? 1 : 0, C, ldc, vec_ok(A, lda), vec_ok(B, ldb)};
  return launch_any<kPlain>(g, (cudaStream_t)stream);
}

extern "C" int espec_mlp_layer(int rows, int fin, int fout, const void* x, const void* w,
                               const float* b, int act, float* z, void* h, void* stream) {
  if (rows <= 0 || fin <= 0 || fout <= 0 || !x || !w || !b || !z)
    return set_error(ESPEC_EINVAL, "bad network layer");
  TcGemm g{rows, fout, fin, 1.0f, 0.0f, (const uint16_t*)x, fin, 0, (const uint16_t*)w, fout, 0,
           z, fout, vec_ok(x, fin), vec_ok(w, fout)};
  g.bias = b;
  g.h = (uint16_t*)h;
  g.act = act;
  return launch_any<kBias>(g, (cudaStream_t)stream);
}

extern "C" int espec_mlp_layer_back(int rows, int fin, int fout, const void* dz, const void* w,
                                    const float* z_in, float* dz_in, void* dz_in_bf16,
                                    void* stream) {
  if (rows <= 0 || fin <= 0 || fout <= 0 || !dz || !w || !z_in || !dz_in || !dz_in_bf16)
    return set_error(ESPEC_EINVAL, "bad network layer");
  TcGemm g{rows, fin, fout, 1.0f, 0.0f, (const uint16_t*)dz, fout, 0, (const uint16_t*)w, fout, 1,
           dz_in, fin, vec_ok(dz, fout), vec_ok(w, fout)};
  g.z = z_in;
  g.h = (uint16_t*)dz_in_bf16;
  return launch_any<kGeluBack>(g, (cudaStream_t)stream);
}

namespace espec {
namespace {
// One thread waits, with the GEMM's bounded wait, on an mbarrier that nothing
// arrives on and no copy or MMA is attached to: the wait must give up after
// `polls` polls and set the status word.  The barrier is invalidated before
// the CTA exits.
__global__ void mbar_timeout_probe(long polls, int* gave_up) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&bar)));
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    const bool ok = wait_phase(&bar, 0u, polls);
    *gave_up = ok ? 0 : 1;
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];\n" ::"r"(smem_u32(&bar)) : "memory");
  }
}
}  // namespace
}  // namespace espec

extern "C" int espec_selftest_mbar_wait(long polls, int* gave_up) {
  if (polls < 1 || !gave_up) return set_error(ESPEC_EINVAL, "polls must be positive");
  int* d = nullptr;
  cudaError_t e = cudaMalloc(&d, sizeof(int));
  if (e != cudaSuccess) return set_cuda_error("cudaMalloc", e);
  mbar_timeout_probe<<<1, 32>>>(polls, d);
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpy(gave_up, d, sizeof(int), cudaMemcpyDeviceToHost);
  cudaFree(d);
  if (e != cudaSuccess) return set_cuda_error("mbarrier wait self-test", e);
  return ESPEC_OK;
}

extern "C" int espec_gemm_bf16_status(int* timed_out) {
  if (!timed_out) return set_error(ESPEC_EINVAL, "null argument");
  int v = 0, zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_tc_status, sizeof(int));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_tc_status, &zero, sizeof(int));
  if (e != cudaSuccess) return set_cuda_error("tensor-core GEMM status", e);
  *timed_out = v;
  return ESPEC_OK;
}

extern "C" int espec_mlp_bias_gelu(float* z, const float* b, int rows, int cols, int act,
                                   void* h_bf16, void* stream) {
  bias_gelu_kernel<<<nblk((long)rows * cols), 256, 0, (cudaStream_t)stream>>>(
      z, b, rows, cols, act, (uint16_t*)h_bf16);
  TC_CK();
  return ESPEC_OK;
}

extern "C" int espec_mlp_gelu_back(float* dh, const float* z, long count, void* dz_bf16,
                                   void* stream) {
  gelu_back_kernel<<<nblk(count), 256, 0, (cudaStream_t)stream>>>(dh, z, count,
                                                                   (uint16_t*)dz_bf16);
  TC_CK();
  return ESPEC_OK;
}

extern "C" int espec_to_bf16(const float* x, void* y, long count, void* stream) {
  const cudaError_t e = launch_either(to_bf16_kernel<true>, to_bf16_kernel<false>, nblk(count), 256,
                                      (cudaStream_t)stream, x, (uint16_t*)y, count);
  if (e != cudaSuccess) return set_cuda_error("mlp bf16 kernel launch", e);
  return ESPEC_OK;
}

extern "C" int espec_mlp_adam_bf16(float* w, const float* g, float* m1, float* m2, long count,
                                   const float* hyper, float b1, float b2, float eps, void* w_bf16,
                                   void* stream) {
  adam_bf16_kernel<<<nblk(count), 256, 0, (cudaStream_t)stream>>>(w, g, m1, m2, count, hyper, b1,
                                                                  b2, eps, (uint16_t*)w_bf16);
  TC_CK();
  return ESPEC_OK;
}

extern "C" int espec_mlp_forward(int nlayers, const int* width, int rows, const void* x,
                                 const void* const* w, const float* const* b, float* const* z,
                                 void* const* h, void* stream) {
  if (nlayers < 1 || !width || !w || !b || !z || (nlayers > 1 && !h))
    return set_error(ESPEC_EINVAL, "bad network");
  const void* in = x;
  for (int i = 0; i < nlayers; ++i) {
    void* out = i + 1 < nlayers ? h[i] : nullptr;
    const int rc = espec_mlp_layer(rows, width[i], width[i + 1], in, w[i], b[i], i + 1 < nlayers,
                                   z[i], out, stream);
    if (rc) return rc;
    in = out;
  }
  return ESPEC_OK;
}

extern "C" int espec_mlp_backward(int nlayers, const int* width, int rows, const void* const* hs,
                                  const float* const* z, const void* const* w, const float* dy,
                                  float* const* dw, float* const* db, void* work, void* stream) {
  if (nlayers < 1 || rows < 1 || !width || !hs || !z || !w || !dy || !dw || !db || !work)
    return set_error(ESPEC_EINVAL, "bad network");
  size_t wmax = 0;
  for (int i = 1; i <= nlayers; ++i) wmax = width[i] > (int)wmax ? (size_t)width[i] : wmax;
  // the current layer's dz (FP32, two in turn) and its BF16 copies
  const size_t n = (size_t)rows * wmax;
  float* dz[2] = {(float*)work, (float*)work + n};
  uint16_t* d16[2] = {(uint16_t*)(dz[1] + n), (uint16_t*)(dz[1] + n) + n};
  const float* d = dy;
  int cur = 0;
  int rc = espec_to_bf16(dy, d16[0], (long)rows * width[nlayers], stream);
  for (int i = nlayers - 1; i >= 0 && rc == ESPEC_OK; --i) {
    const int fi = width[i], fo = width[i + 1];
    rc = espec_gemm_bf16(fi, fo, rows, 1.0f, hs[i], fi, 1, d16[cur], fo, 0, 0.0f, dw[i], fo, stream);
    if (rc == ESPEC_OK) rc = espec_mlp_colsum(d, rows, fo, db[i], stream);
    if (rc == ESPEC_OK && i > 0) {
      rc = espec_mlp_layer_back(rows, fi, fo, d16[cur], w[i], z[i - 1], dz[cur ^ 1], d16[cur ^ 1],
                                stream);
      cur ^= 1;
      d = dz[cur];
    }
  }
  return rc;
}
