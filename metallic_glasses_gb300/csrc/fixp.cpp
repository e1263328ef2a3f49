// fixp.cpp -- host side of the fixed-point forms: the exponential's table, the
// transforms' twiddles and the constants of a context.
#include "fixp.cuh"

#include <algorithm>
#include <cmath>
#include <vector>

#include "stz_internal.h"

namespace stz {
namespace {

typedef unsigned __int128 u128;

// a b 2^-126 for a, b below 2^127
u128 mul_q126(u128 a, u128 b) {
  const uint64_t ah = (uint64_t)(a >> 64), al = (uint64_t)a, bh = (uint64_t)(b >> 64), bl = (uint64_t)b;
  const u128 hh = (u128)ah * bh, hl = (u128)ah * bl, lh = (u128)al * bh, ll = (u128)al * bl;
  const u128 mid = (ll >> 64) + (uint64_t)hl + (uint64_t)lh;
  const u128 hi = hh + (hl >> 64) + (lh >> 64) + (mid >> 64);
  return (hi << 2) | ((uint64_t)mid >> 62);
}

// 2^(2^-i) 2^126 for i = 1 .. 12 (repeated square roots of 2)
const uint64_t kRoots[12][2] = {
    {0x5a827999fcef3242, 0x2cbec4d9baa55f50}, {0x4c1bf828c6dc54b7, 0xa356918c17217b7b},
    {0x45cae0f1f545eb73, 0x7df23143ac529e48}, {0x42d561b3e6243d8a, 0x62e4adc610aa60d9},
    {0x4166c34c5615d0eb, 0x9f1523ada3290600}, {0x40b268f9de0183b9, 0xbdf2b293de8a6f7a},
    {0x4058f6a7ecccd5b6, 0x1299ab8cdb737e90}, {0x402c6be96af2fb58, 0x4a6ac4fb04772551},
    {0x4016321b687027a8, 0x7fc674a533cbd9e7}, {0x400b18178ba33b14, 0x1b486ff22688e804},
    {0x40058bce410147e8, 0x4a2f2a71570c7978}, {0x4002c5d7bff71dae, 0x8e38c59c72a4e5ca}};
// ln 2 2^126
const uint64_t kLn2[2] = {0x2c5c85fdf473de6a, 0xf278ece600fcbdac};

constexpr long double kLog2e = 1.44269504088896340735992468100189214L;

int64_t fixed(long double v, int s) { return (int64_t)std::llrint(std::ldexp(v, s)); }

}  // namespace

void fx_exp_table(FxExp* t) {
  const u128 ln2 = (u128)kLn2[0] << 64 | kLn2[1];
  for (int j = 0; j < kFxExpCells; j++) {
    u128 v = (u128)1 << 126;
    const int h = 2 * j + 1;  // the 12 bits of (j + 1/2) / 2048
    for (int i = 0; i < 12; i++)
      if (h >> (11 - i) & 1) v = mul_q126(v, (u128)kRoots[i][0] << 64 | kRoots[i][1]);
    t[j].t = (int64_t)((uint64_t)(v >> 64) + ((uint64_t)(v >> 63) & 1));
    const Fx s = fx_split((int64_t)((mul_q126(v, ln2) + ((u128)1 << 74)) >> 75));
    t[j].ph = s.h;
    t[j].pl = s.l;
  }
}

namespace {

// pi / 4 2^126
const uint64_t kPi4[2] = {0x3243f6a8885a308d, 0x313198a2e0370734};

// 2^126 / m! for m = from, from + 2, ...
struct Factorials {
  u128 c[14];
  constexpr explicit Factorials(int from) : c() {
    u128 v = (u128)1 << 126;
    for (int m = 2; m <= from; m++) v /= (unsigned)m;
    for (int j = 0; j < 14; j++) {
      c[j] = v;
      v = v / (unsigned)(from + 2 * j + 1) / (unsigned)(from + 2 * j + 2);
    }
  }
};
constexpr Factorials kCos(0), kSin(1);

// The alternating series in y (y below 0.62; the 14th term is below 2^-97)
u128 series(const Factorials& f, u128 y) {
  u128 s = f.c[13];
  for (int j = 12; j >= 0; j--) s = f.c[j] - mul_q126(y, s);
  return s;
}

}  // namespace

void fx_twiddles(int n, int count, FxTwiddle* out) {
  // Cosine and sine of an eighth of a turn times num / n, each fraction formed
  // once: the angles are folded to it, so that exact values stay exact,
  // symmetric values are equal, and a table takes its series for n/8 of them
  // (long double functions took 1.1 us a value on the host of a GB300, 160 us of
  // every stand-alone solve of 48 x 54 x 36).
  struct CS {
    int64_t c = 0, s = 0;
  };
  std::vector<CS> seen((size_t)n + 1);
  const u128 pi4 = (u128)kPi4[0] << 64 | kPi4[1], q = pi4 / (unsigned)n, r = pi4 % (unsigned)n;
  auto round62 = [](u128 v) { return (int64_t)((uint64_t)(v >> 64) + ((uint64_t)(v >> 63) & 1)); };
  auto cs = [&](long long num) {
    CS& e = seen[(size_t)num];
    if (e.c == 0) {  // a cosine is at least sqrt(1/2)
      const u128 x = q * (unsigned)num + r * (unsigned)num / (unsigned)n, y = mul_q126(x, x);
      e.c = round62(series(kCos, y));
      e.s = round62(mul_q126(x, series(kSin, y)));
    }
    return e;
  };
  for (int k = 0; k < count; k++) {
    const int k8 = (int)((8LL * k / n) & 7);
    const long long num = 8LL * k - (long long)k8 * n;  // within the octant
    const CS v = cs(k8 & 1 ? n - num : num);
    int64_t re, im;
    switch (k8) {
      case 0: re = v.c; im = v.s; break;
      case 1: re = v.s; im = v.c; break;
      case 2: re = -v.s; im = v.c; break;
      case 3: re = -v.c; im = v.s; break;
      case 4: re = -v.c; im = -v.s; break;
      case 5: re = -v.s; im = -v.c; break;
      case 6: re = v.s; im = -v.c; break;
      default: re = v.c; im = -v.s; break;
    }
    auto fix = [](int64_t w) {
      Fx f = fx_split(w);
      if (f.l == INT32_MIN) f.l++;  // so that the halves can be negated
      return f;
    };
    out[k] = FxTwiddle{fix(re), fix(-im)};
  }
}

void fx_green_constants(int n0, int n1, int n2, double lambda, double mu, GreenFx* g) {
  GreenFx& ga = *g;
  ga.is3d = n0 > 1;
  ga.n0 = n0; ga.n1 = n1; ga.n2 = n2; ga.nh = n2 / 2 + 1;
  const long double lam = lambda, m = mu, al = (lam + m) / (lam + 2 * m);
  const long double l2 = lam / (2 * m), c1 = (1 - al) * lam / m;
  // constants at most 2^62; the operator's growth (1 + 3 |lambda| / (2 mu) for
  // tau, then three more bits) as headroom
  const long double big = std::max(std::fabs(l2), std::fabs(c1));
  ga.lams = 2;
  while (std::ldexp(1.0L, ga.lams - 2) < big) ga.lams++;
  ga.lam = fx_split(fixed(l2, 64 - ga.lams));
  ga.c1 = fx_split(fixed(c1, 64 - ga.lams));
  ga.al2 = fx_split(fixed(2 * al, 60));
  ga.kb = 3;
  while (std::ldexp(1.0L, ga.kb) < 8 * (1 + 3 * std::fabs(l2))) ga.kb++;
  const int nn[3] = {n0, n1, n2};
  for (int i = 0; i < 3; i++) ga.inv[i] = fixed(1.0L / nn[i], 61);
}

// The constants of an FP64 context (see RateFx); on = 0 when they do not fit.
void rate_fx_constants(const KParams& kp, RateFx* x) {
  x->on = 0;
  const bool d2 = kp.model == STZ_MODEL_REF2D;
  const long double kT = kp.kT, w = (long double)kp.V0 * 1e-18L * (long double)kJInEv / (2 * kT) * kLog2e;
  const long double b = kLog2e / kT, c = std::log2((long double)kp.vt) + 1022;
  if (!(b > 1e-15L && b < 1e15L) || !(w > 1e-15L && w < 1e15L) || !(c > 600 && c < 1440)) return;
  if (d2) {
    const int LW = (int)std::ceil(std::log2(w));
    x->sw = 48 + LW;
    x->w2 = fx_split(fixed(w, 60 - LW));
    x->l2e = fx_split(fixed(kLog2e, 61));
    const long double ft[3] = {0.1L, 0.01L, 0.9L};
    for (int t = 0; t < 3; t++)
      for (int m = 0; m < STZ_MODES; m++) x->ftp[t][m] = fx_split(fixed(std::pow(ft[t], (long double)(m + 2)), 62));
    x->decayed = 746 * kp.t_temp;
  } else {
    long double M[STZ_MODES][5], smax = 0;
    for (int m = 0; m < STZ_MODES; m++) {
      const double* d = kp.modes[m];
      M[m][0] = w * d[0];
      M[m][1] = w * d[1];
      for (int k = 2; k < 5; k++) M[m][k] = 2 * w * d[k + 1];
      long double s = 0;
      for (int k = 0; k < 5; k++) s += std::fabs(M[m][k]);
      if (!(s <= 1e15L)) return;
      smax = std::max(smax, s);
    }
    if (!(smax > 1e-15L)) return;
    const int L = (int)std::ceil(std::log2(smax));
    x->sw = 51 + L;
    for (int m = 0; m < STZ_MODES; m++) {
      for (int k = 0; k < 5; k++) x->m[m][k] = fx_split(fixed(M[m][k], 61 - L));
      const double* d = kp.modes[m];
      const long double t = std::ldexp(w * ((long double)d[0] + d[1] + d[2]), 61 - L);
      if (!(std::fabs(t) < 2e9L)) return;  // a trace far beyond rounding
      x->mt[m] = (int32_t)std::llrint(t);
    }
  }
  const int LB = (int)std::ceil(std::log2(b));
  x->sq = 51 + LB;
  x->nb = fx_split(fixed(-b, 61 - LB));
  const uint64_t c53 = (uint64_t)fixed(c - 1024, 53) + ((uint64_t)1024 << 53);  // c 2^53 may exceed 2^63
  x->c_hh = (int64_t)(c53 >> kFxRateShift);
  x->c_mid = (int64_t)(c53 & ((1u << kFxRateShift) - 1)) << (32 - kFxRateShift);
  x->neg = c53;
  if (!(0.33L * b < 500)) return;
  x->mark = c53 - (uint64_t)fixed(0.33L * b, 53);
  x->on = 1;
}

}  // namespace stz
