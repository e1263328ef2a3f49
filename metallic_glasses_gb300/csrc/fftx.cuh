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

// True when the medium's constants fit the fixed-point Green's pass.
bool fftx_fits(double lambda, double mu);
// The passes up to the spectrum before the last one (along axis 2), which is
// the stress's divided by 2 mu; fftx_factor is what a C2R pass multiplies its
// sums by (2 mu / N).
void fftx_spectrum(const FFTPlan& p, const SolveArgs& a, cudaStream_t st, int64_t* launches);
double fftx_factor(const FFTPlan& p, double mu);
// The C2R pass of a kOutSig64 solve.
void fftx_c2r(const FFTPlan& p, const SolveArgs& a, cudaStream_t st, int64_t* launches);
// Raises the passes' shared-memory limits on the current device.
void fftx_init();

}  // namespace stz
