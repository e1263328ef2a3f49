// fixp.cuh -- 64-bit fixed-point arithmetic for the FP64 forms.
//
// GB300 issues FP64 at 1.7 lanes per clock and SM (measured: 19 SM clocks per
// warp instruction) and a 32 x 32 -> 64 bit integer multiply-add at 32 lanes
// (one clock). A sum of products and an exponential whose operands are held
// as 64-bit fixed point therefore cost a fraction of the same sum in FP64, and
// with the scales chosen below they are more exact on average. What is cut of a
// rate's argument (in powers of two) is the products of low halves, 2^-50 at
// most for each of six in 3D (2^-50.3 together on average, in the mean square)
// and 2^-47 for each of two in 2D (2^-48), where FP64 rounds an argument of size
// 32 to 64 by 2^-48 at every operation; a single sum may come out further off.
//
// Host and device compile the same functions, so the tests check them on the
// CPU against higher precision.
#pragma once
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define FX_HD __host__ __device__ __forceinline__
#else
#define FX_HD inline
#endif

namespace stz {

// a b + c with a 64-bit result, as one multiply-add. Written out: from the C
// expression the compiler forms a general 64 x 64 product when one operand is a
// kernel parameter (five instructions), and of a chain of mad.wide it makes a
// tree of products and separate 64-bit additions (16 more instructions per
// rate, 102 in place of 87); the pair with a carry stays one multiply-add.
FX_HD int64_t fx_wide(int32_t a, int32_t b, int64_t c) {
#ifdef __CUDA_ARCH__
  uint32_t lo, hi;
  asm("mad.lo.cc.s32 %0, %2, %3, %4;\n\tmadc.hi.s32 %1, %2, %3, %5;"
      : "=&r"(lo), "=r"(hi)
      : "r"(a), "r"(b), "r"((uint32_t)c), "r"((uint32_t)((uint64_t)c >> 32)));
  return (int64_t)((uint64_t)hi << 32 | lo);
#else
  return (int64_t)a * b + c;
#endif
}
FX_HD int64_t fx_wide_u(uint32_t a, uint32_t b, int64_t c) {
#ifdef __CUDA_ARCH__
  int64_t r;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
#else
  return (int64_t)((uint64_t)a * b + (uint64_t)c);
#endif
}

// A signed 64-bit value in two signed halves, v = h 2^32 + l with
// -2^31 <= l < 2^31, so that products of halves are signed 32 x 32 bit.
struct Fx {
  int32_t h, l;
};
FX_HD Fx fx_split(int64_t v) {
  Fx r;
  r.l = (int32_t)(uint32_t)(uint64_t)v;
  r.h = (int32_t)((v + 0x80000000ll) >> 32);
  return r;
}

// Sum of products x y of such values, kept as hh 2^64 + mid 2^32: three
// multiply-adds per product (the l l product, below 2^62 of 2^64 hh, is
// dropped). Values of magnitude up to 2^61 and 2^60 leave room for five
// products in mid.
struct FxAcc {
  int64_t hh, mid;
};
FX_HD void fx_mad(FxAcc& a, Fx x, Fx y) {
  a.hh = fx_wide(x.h, y.h, a.hh);
  a.mid = fx_wide(x.h, y.l, a.mid);
  a.mid = fx_wide(x.l, y.h, a.mid);
}
// hh 2^S + mid 2^(S - 32), rounded down (0 < S < 32)
template <int S>
FX_HD int64_t fx_value(const FxAcc& a) {
  return (int64_t)((uint64_t)a.hh << S) + (a.mid >> (32 - S));
}

FX_HD uint64_t fx_bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t b;
  std::memcpy(&b, &x, 8);
  return b;
#endif
}
FX_HD double fx_double(uint64_t b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double x;
  std::memcpy(&x, &b, 8);
  return x;
#endif
}
// x 2^s rounded toward zero, on the integer pipe. *ok is cleared when the
// magnitude is 2^(63 - top) or more (infinities and NaN among them).
template <int top>
FX_HD int64_t fx_from_f64(double x, int s, bool* ok) {
  const uint64_t b = fx_bits(x);
  const int e = (int)(b >> 52) & 0x7ff;
  // m 2^10 of the 53-bit significand m; the value is m 2^(e - 1075)
  const uint64_t m = ((b << 10) & 0x3ffffffffffffc00ull) | (e ? 0x4000000000000000ull : 0ull);
  const int r = 1085 - s - e;  // right shift; at least `top` below the limit
  if (r < top) *ok = false;
  const int64_t v = (int64_t)(m >> (r > 63 ? 63 : (r < 0 ? 0 : r)));
  const int64_t sg = (int64_t)b >> 63;
  return (v ^ sg) - sg;
}

// ------------------------------------------------------------- 2^y
// Y = (y + 1022) 2^53 for 1 <= y + 1022 < 2046. With k = floor(y), j the next
// 11 bits of y and g in [-2^-12, 2^-12) the distance of the rest from the
// middle of its cell,
//   2^y = 2^k T_j (1 + x (1 + e)),  T_j = 2^((j + 1/2) / 2048),  x = g ln 2,
//   e = x/2 + x^2/6 (+ 3 a^2 x / 96 for x^3/24, its best linear fit on
//   |x| <= a = 2^-12 ln 2, error below 2^-56),
// the product T_j ln 2 taken from the table beside T_j. Since the cell's middle
// is tabulated, T_j (1 + x (1 + e)) stays in [1, 2) and needs no normalising.
// The scales make every sum a multiply-add: T_j ln 2 g comes out in the units
// of T_j, and the corrections' high words are taken without a shift.
struct alignas(16) FxExp {
  int64_t t;       // T_j 2^62
  int32_t ph, pl;  // T_j ln 2 2^51 = ph 2^32 + pl
};
constexpr int kFxExpCells = 2048;
constexpr int32_t kFxE1 = 1488522239;  // ln 2 (1 + a^2/16) 2^31
constexpr int32_t kFxE2 = 167930;      // (ln 2)^2 / 6 2^21

FX_HD int fx_exp_cell(uint64_t Y) { return (int)(Y >> 42) & (kFxExpCells - 1); }
// the high word of a product, and rounded to nearest
FX_HD int32_t fx_high(int32_t a, int32_t b) { return (int32_t)(fx_wide(a, b, 0) >> 32); }
FX_HD int32_t fx_high_round(int32_t a, int32_t b) { return (int32_t)(fx_wide(a, b, 1ll << 31) >> 32); }
// 2^(y - k) 2^62 (to 2^-53.6 of it, rms 2^-55.6), plus half a unit of a
// double's last place with ROUND
template <bool ROUND>
FX_HD int64_t fx_exp2_mant(uint64_t Y, const FxExp& q) {
  const int64_t G = (int64_t)((Y << 22) ^ 0x8000000000000000ull);  // g 2^75
  const int32_t gh = (int32_t)(G >> 32);
  const uint32_t gl = (uint32_t)G;
  const int32_t e = (int32_t)(fx_wide(gh, kFxE1 + fx_high(gh, kFxE2), 1 << 30) >> 31);  // e 2^44
  // X = T_j ln 2 g 2^62; its carry-in rounds, and takes the rounding's 512
  const int64_t mid = fx_wide_u((uint32_t)q.ph, gl, fx_wide(q.pl, gh, (1ll << 31) + (ROUND ? 512ll << 32 : 0)));
  const int64_t X = fx_wide(q.ph, gh, mid >> 32);
  return q.t + fx_wide(fx_high_round((int32_t)(X >> 20), e), 256, X);  // x e 2^54
}
// 2^y as a double, rounded to nearest (within 0.85 ulp over 3 10^6 random
// arguments and cell edges against a 113-bit exponential; rms 0.310 ulp, of
// which 0.289 is the rounding itself).
FX_HD uint64_t fx_exp2_bits(uint64_t Y, const FxExp& q) {
  return ((uint64_t)fx_exp2_mant<true>(Y, q) >> 10) + (Y & 0xffe0000000000000ull) / 2;
}
FX_HD int fx_clz(uint64_t v) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)v);
#else
  return v ? __builtin_clzll(v) : 64;
#endif
}
// v >> d, 0 for d of 64 and more
FX_HD uint64_t fx_shr(uint64_t v, int d) {
#ifdef __CUDA_ARCH__
  uint64_t r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(d));  // the count is clamped
  return r;
#else
  return d > 63 ? 0 : v >> d;
#endif
}
// The sum of N <= 4 exponentials as a double: the significands aligned to the
// largest exponent and added as integers (each cut 2^-60 of the largest below),
// one rounding at the end.
template <int N>
FX_HD uint64_t fx_exp2_sum_bits(const uint64_t* Y, const FxExp* q) {
  if (N == 1) return fx_exp2_bits(Y[0], q[0]);
  int k[N], km = 0;
#pragma unroll
  for (int i = 0; i < N; i++) {
    k[i] = (int)(Y[i] >> 53);
    km = k[i] > km ? k[i] : km;
  }
  uint64_t M = 0;
#pragma unroll
  for (int i = 0; i < N; i++) {
    M += fx_shr((uint64_t)fx_exp2_mant<false>(Y[i], q[i]), km - k[i] + 2);
  }
  const int z = fx_clz(M) - 1;  // 0 .. 2
  return (((M << z) + 512) >> 10) + ((uint64_t)(uint32_t)(km + 2 - z) << 52);
}

// The table, from the square roots 2^(2^-i), i = 1 .. 12, as 126-bit fixed
// point (integer arithmetic only: the same bits on every host; fixp.cpp).
void fx_exp_table(FxExp* t);

// Constants of the fixed-point rates of one FP64 context. In 3D the rate
// argument in log2 units, y = log2(vt) - dF log2(e)/kT + sum_c W_c M_mc, with
// W = (s_xx - s_zz, s_yy - s_zz, s_yz, s_xz, s_xy) and M the modes times V0
// 1e-18 J log2(e) / (2 kT) (shears doubled), is held
// as (y + 1022) 2^53 = 2^5 (hh 2^64 + mid 2^32) / 2^64 of an FxAcc.
// Scales: with L = ceil(log2(max_m sum_c |M_mc|)) stresses carry 2^(51 + L) and
// modes 2^(61 - L), so stresses (the field's, the uniform one and their sum) below
// 2^(8 - L) GPa (8 GPa at 455 K and 1 nm^3) move y by at most 512; with LB = ceil(log2(log2(e)/kT)) barriers carry
// 2^(51 + LB), the constant 2^(61 - LB). A site beyond these limits (or not
// finite) sends its block through the FP64 chain.
struct RateFx {
  int on;             // 0: the context's constants do not fit, every block takes the FP64 chain
  int sw, sq;         // binary scales of the stresses and the barriers
  Fx nb;              // -log2(e)/kT
  int64_t c_hh, c_mid;  // log2(vt) + 1022
  uint64_t neg;       // Y above this: a positive rate argument (a negative barrier)
  uint64_t mark;      // Y above this: a barrier below 0.33 eV (the avalanche's marks)
  const FxExp* tab;   // device table
  Fx m[20][5];
  int32_t mt[20];     // the modes' traces (rounding, some 1e-17), which s_zz multiplies
  // 2D model (see R2Fx in kmc.cu): the work scale V0 1e-18 J log2(e) / (2 kT)
  // of the stress coordinates and log2(e) x 2^61; the powers ft^(m + 2) of the
  // crystal-like types' factors x 2^62; the decay of the temporary softening
  // underflows beyond this time
  Fx w2, l2e;
  Fx ftp[3][20];
  double decayed;
  // ... and its stored operands, kept with Q0, deps and prev_deps
  uint64_t* cq;       // [MODES][N] log2(vt) + 1022 - Q0 log2(e)/kT, x 2^53; 0: a value of the
                      // (mode, site) does not fit
  Fx *dx, *dxy;       // [MODES][N] deps xx and xy, x 2^60 (the modes are traceless)
  Fx *ux, *uxy;       // [MODES][N] deps xx and xy over the mode's norm, x 2^60 (softening only)
  Fx* pn;             // [2][N] (xx - yy) and 2 xy of the last increment over its norm, x 2^60
  int grid;           // resident blocks of the rate kernel (at most nblk split)
  int split;          // parts that a block's modes are split into (rate_fx_split)
};
constexpr int kFxRateShift = 5;
// the smallest and largest Y of a site before its stress terms
constexpr uint64_t kFxY0Min = (uint64_t)514 << 53, kFxY0Max = (uint64_t)1533 << 53;

// exp(-2 pi i k / n), k = 0 .. count-1, as split fixed point (x 2^62): the
// halves of the real part, then of the imaginary part (fixp.cpp).
struct alignas(16) FxTwiddle {
  Fx r, i;
};
void fx_twiddles(int n, int count, FxTwiddle* out);

// Constants of the fixed-point Green's pass (fftx.cu).
struct GreenFx {
  int is3d, n0, n1, n2, nh;  // is3d: the grid has an axis 0 (n0 > 1), whatever its components
  int kb;            // headroom of the operator: the largest input is below 2^(61 - kb)
  int lams;          // lam and c1 carry 2^(64 - lams)
  Fx lam;            // lambda / (2 mu)
  Fx c1;             // (1 - alpha) lambda / mu, alpha = (lambda + mu) / (lambda + 2 mu)
  Fx al2;            // 2 alpha, x 2^60
  int64_t inv[3];    // 2^61 / n0, n1, n2
};
void fx_green_constants(int n0, int n1, int n2, double lambda, double mu, GreenFx* g);

}  // namespace stz
