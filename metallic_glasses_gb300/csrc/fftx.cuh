// fftx.cuh -- the Green's-function solve in 64-bit fixed point (fftx.cu).
#pragma once
#include <cuda_runtime.h>

#include "fixp.cuh"

namespace stz {

struct Sched;
struct FFTPlan;
struct SolveArgs;

// One radix pass over lines of n: m = n / R butterflies a line, ns the product
// of the radices before; quotients by m and ns as multiply-highs.
struct FxStage {
  int R, m, ns, step;
  unsigned mq, nsq;  // ceil(2^32 / m), ceil(2^32 / ns); 0 for a divisor of 1
};
struct FxSched {
  int n = 1, nst = 0;
  FxStage st[10];
};
FxSched fx_sched(const Sched& s);

// Elements of a line of n in shared memory (padded against bank conflicts).
__host__ __device__ constexpr int fx_ld(int n) { return (n + (n >> 3)) | 1; }

// The longest lines along axis 2 that the fixed-point passes take (the other axes
// end at 1024). A dense line's values lie the lower above the integers' unit the
// longer it is, while an FP64 transform's error hardly grows: random eigenstrain
// is off by 0.60e-15 of the stress at 16x1296 (FP64 passes 1.08e-15), 0.93e-15 at
// 2x2x1728 (0.83e-15), 1.3e-15 at 2x2x3072 (0.84e-15), 2.5e-15 at 16x6144 (1.09e-15).
constexpr int kFxLongest = 1296;
// True when an FP64 solve of lines of n2 runs in fixed point: the lines are short
// enough and the medium's constants fit Green's pass.
bool fftx_fits(int n2, double lambda, double mu);
// The passes up to the spectrum before the last one (along axis 2), which is
// the stress's divided by 2 mu; fftx_factor is what a C2R pass multiplies its
// sums by (2 mu / N).
void fftx_spectrum(const FFTPlan& p, const SolveArgs& a, cudaStream_t st, int64_t* launches);
double fftx_factor(const FFTPlan& p, double mu);
// The C2R pass of a kOutSig64 solve.
void fftx_c2r(const FFTPlan& p, const SolveArgs& a, cudaStream_t st, int64_t* launches);
// Raises the passes' shared-memory limits on the current device: of all kernels,
// or of those that a plan with its present tiles launches.
void fftx_init(const FFTPlan* plan = nullptr);

}  // namespace stz
