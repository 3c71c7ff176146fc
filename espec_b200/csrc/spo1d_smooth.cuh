// spo1d_smooth.cuh -- 1D packets of even sizes whose prime factors are at most
// 13 (spo1d_smooth.cu): the radix plan of the in-place transform and the launch.
#pragma once
#include <cuda_runtime.h>

#include "spo1d.cuh"

namespace espec {

constexpr int kSmoothMaxStages = 8;
constexpr int kSmoothMaxRadix = 16;
constexpr int kSmoothMaxThreads = 512;

struct SmoothPlan {
  int n, ns, threads;          // size, stages (at least 2), threads of a packet's CTA
  int r[kSmoothMaxStages];     // radix of each stage (product n)
  int m[kSmoothMaxStages];     // n / (r[0] .. r[s]): stride of stage s's butterflies
  unsigned inv[kSmoothMaxStages];  // ceil(2^32 / m[s]): b / m[s] = (b inv) >> 32
  int step[kSmoothMaxStages];      // shared-memory places between the points of a butterfly
  int tw_off[kSmoothMaxStages];    // first twiddle of each stage
  int ntw;                         // twiddles in all
  int pitch;                       // places of a last-stage butterfly (odd)
  unsigned inv_last;               // ceil(2^32 / last radix)
};

// the plan of size n; false where n has a prime factor above 13
bool smooth_plan(int n, SmoothPlan& pl);
// frequency (FFT order) of each place of the kinetic table
void smooth_final_freq(const SmoothPlan& pl, int* kap);
// the stages' twiddles (pl.ntw) from w[e] = e^{2 pi i e / n}
void smooth_twiddles(const SmoothPlan& pl, const double2* w, double2* tw);
// tw: the stages' twiddles
cudaError_t spo_smooth_launch(const SpoArgs<double>& a, const SmoothPlan& pl, const double2* tw,
                              bool quirk, int nblocks, cudaStream_t st);

}  // namespace espec
