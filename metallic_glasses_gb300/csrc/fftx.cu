// fftx.cu -- the Green's-function solve (fft.cu) in 64-bit fixed point.
//
// The FP64 passes are bound by the FP64 pipe, which issues a warp instruction
// in 19 SM clocks: a complex product takes 76, a radix-8 butterfly 1500. Here a
// pass converts its tile of lines to 64-bit integers at a scale of the tile's
// own, runs the transform on the integer pipe (a complex product is twelve
// 32 x 32 bit multiply-adds, an addition two instructions), and converts the
// result back; what lies in memory between the passes stays FP64.
//
// Scale. Every partial sum of a transform of a line is bounded by the line's
// sum of |re| + |im|. Each line takes that sum (in FP32, rounded up) and the
// scale that puts it below 2^61 (R2C, whose last step doubles it), 2^62 (column
// passes) or 2^60 (C2R: 2^62 for the doubled pairs of its half spectrum), so no
// sum reaches 2^63 and no stage needs a scale of its own. A dense line of n
// values keeps them some 59.5 - log2(n) bits above the integers' unit (53 at
// n = 64, 50 at 512), but each value is rounded at that unit three or four times
// in a pass where an FP64 transform rounds it relative to itself at every
// operation; sparse lines keep more. Roundings are to nearest. Green's operator
// works at a scale per wave number. A line with an infinity or a NaN becomes NaN.
// The mean strain's uniform stress C:<eps> is added to the result in FP64
// instead of entering the k = 0 term, which it would dominate.
//
// Measured, solve with host overhead: 422 -> 157 us at 64^3, 2530 -> 800 us at
// 128^3, 250 -> 90 us at 512^2 (tuned tiles and threads on both sides). The
// result's error against wider arithmetic (relative L2, random eigenstrain, FP64
// passes before): 8.9e-16 -> 1.6e-16 at 64^3, 1.1e-15 -> 3.4e-16 at 512^2; below
// FP64 passes' for sparse, smooth, banded and nearly uniform fields too. The
// passes are bound by integer issue and their phases between barriers: about
// 500, 300, 640, 300 and 680 instructions per complex value at 64^3, of which a
// radix-8 stage is 36 to 71.
#include "fftx.cuh"

#include <algorithm>
#include <cmath>

#include "fft.cuh"

namespace stz {

FxSched fx_sched(const Sched& s) {
  FxSched o;
  o.n = s.n;
  o.nst = s.nst;
  int ns = 1;
  auto quo = [](int d) { return d > 1 ? (unsigned)(((1ull << 32) + d - 1) / d) : 0u; };
  for (int i = 0; i < s.nst; i++) {
    FxStage& t = o.st[i];
    t.R = s.r[i];
    t.m = s.n / t.R;
    t.ns = ns;
    t.step = s.n / (ns * t.R);
    t.mq = quo(t.m);
    t.nsq = quo(ns);
    ns *= t.R;
  }
  return o;
}

namespace {

constexpr int kMaxTh = 256;
constexpr unsigned FULL = 0xffffffffu;

struct __align__(16) cx {  // a complex fixed-point value
  int64_t x, y;
};
__device__ __forceinline__ cx operator+(cx a, cx b) { return cx{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ cx operator-(cx a, cx b) { return cx{a.x - b.x, a.y - b.y}; }

__device__ __forceinline__ FxTwiddle tw_load(const FxTwiddle* __restrict__ t, int k) {
  const int4 v = __ldg(reinterpret_cast<const int4*>(t + k));
  return FxTwiddle{Fx{v.x, v.y}, Fx{v.z, v.w}};
}
// half a unit of the products' last place, held in a register pair (as a literal
// the compiler moves it into one at every use)
__device__ __forceinline__ int64_t half_unit() {
  int64_t h;
  asm volatile("mov.b64 %0, 0x20000000;" : "=l"(h));
  return h;
}
// a w / 2^62, rounded to nearest
__device__ __forceinline__ cx cmul(cx a, FxTwiddle w, int64_t half) {
  const Fx ax = fx_split(a.x), ay = fx_split(a.y), ni = Fx{-w.i.h, -w.i.l};
  FxAcc re{0, half}, im{0, half};
  fx_mad(re, ax, w.r);
  fx_mad(re, ay, ni);
  fx_mad(im, ax, w.i);
  fx_mad(im, ay, w.r);
  return cx{fx_value<2>(re), fx_value<2>(im)};
}
// v c / 2^62
__device__ __forceinline__ int64_t rmul(int64_t v, Fx c, int64_t half) {
  FxAcc a{0, half};
  fx_mad(a, fx_split(v), c);
  return fx_value<2>(a);
}
// v c / 2^(64 - s) for a constant of scale 2^(64 - s), 2 <= s < 32; halves, which
// constants like 1/2 or 3/2 make frequent, away from zero
__device__ __forceinline__ int64_t rmul_s(int64_t v, Fx c, int s) {
  FxAcc a{0, (1ll << (31 - s)) + (v >> 63)};
  fx_mad(a, fx_split(v), c);
  return (int64_t)((uint64_t)a.hh << s) + (a.mid >> (32 - s));
}
__device__ __forceinline__ int64_t fmul(Fx v, Fx c) {
  FxAcc a{0, 1 << 29};
  fx_mad(a, v, c);
  return fx_value<2>(a);
}
// v 2^-sh to nearest, halves away from zero (rounding halves up instead would
// bias every value of a spectrum alike, which adds up at the first site)
__device__ __forceinline__ int64_t shift_round(int64_t v, int sh) { return (v + (1ll << (sh - 1)) + (v >> 63)) >> sh; }

// sqrt(1/2) and sqrt(3/4), x 2^62
__device__ __forceinline__ Fx c_r2() { return Fx{0x2d413ccd, -0x18866df}; }
__device__ __forceinline__ Fx c_r3() { return Fx{0x376cf5d1, -0x4f66ab19}; }

// Forward butterflies (w = exp(-2 pi i / R)). An inverse transform is the
// forward one with real and imaginary parts exchanged before and after.
__device__ __forceinline__ cx mul_mi(cx a) { return cx{a.y, -a.x}; }  // -i a
__device__ __forceinline__ void dft4(cx& v0, cx& v1, cx& v2, cx& v3) {
  const cx a0 = v0 + v2, a1 = v0 - v2, a2 = v1 + v3, b3 = mul_mi(v1 - v3);
  v0 = a0 + a2;
  v2 = a0 - a2;
  v1 = a1 + b3;
  v3 = a1 - b3;
}
template <int R>
__device__ __forceinline__ void dft(cx* v, int64_t half) {
  if (R == 2) {
    const cx a = v[0], b = v[1];
    v[0] = a + b;
    v[1] = a - b;
  } else if (R == 3) {
    const cx t = v[1] + v[2], u = v[1] - v[2];
    const cx m = cx{v[0].x - ((t.x - (t.x >> 63)) >> 1), v[0].y - ((t.y - (t.y >> 63)) >> 1)};
    const cx q = cx{rmul(u.y, c_r3(), half), -rmul(u.x, c_r3(), half)};
    v[0] = v[0] + t;
    v[1] = m + q;
    v[2] = m - q;
  } else if (R == 4) {
    dft4(v[0], v[1], v[2], v[3]);
  } else {
    dft4(v[0], v[2], v[4], v[6]);
    dft4(v[1], v[3], v[5], v[7]);
    // the odd half's outputs times exp(-i pi k / 4)
    const Fx r = c_r2();
    const cx p0 = v[1], p1 = cx{rmul(v[3].x + v[3].y, r, half), rmul(v[3].y - v[3].x, r, half)}, p2 = mul_mi(v[5]),
             p3 = cx{rmul(v[7].y - v[7].x, r, half), rmul(-v[7].x - v[7].y, r, half)};
    const cx e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    v[0] = e0 + p0;
    v[4] = e0 - p0;
    v[1] = e1 + p1;
    v[5] = e1 - p1;
    v[2] = e2 + p2;
    v[6] = e2 - p2;
    v[3] = e3 + p3;
    v[7] = e3 - p3;
  }
}

__device__ __forceinline__ int pad(int i) { return i + (i >> 3); }
__device__ __forceinline__ int quot(int i, int d, unsigned q) { return d == 1 ? i : (int)__umulhi((unsigned)i, q); }

// x 2^s rounded to nearest (halves away from zero), |x 2^s| < 2^62. Zeros and
// subnormals shift out like every value below 2^-62 of the scale.
__device__ __forceinline__ int64_t to_fix(double x, int s) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  // significand m x 2^10 (its implicit bit 62); the value is m 2^(e - 1075)
  const uint64_t m = ((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32 | lo) << 10;
  const int r = min(1084 - s - (int)((hi >> 20) & 0x7ffu), 63);  // one bit short of the shift, for the rounding
  const int64_t v = (int64_t)(((m >> r) + 1) >> 1);
  const int64_t sg = (int64_t)(int)hi >> 31;
  return (v ^ sg) - sg;
}
// v 2^sh as a double, rounded to nearest: the conversion instruction (16 SM
// clocks per warp on a pipe the transform leaves idle, against 25 integer
// instructions) and an addition to the exponent, which stays in range for the
// scales of line_scale
__device__ __forceinline__ double to_f64(int64_t v, int sh) {
  const double d = __ll2double_rn(v);
  const int hi = __double2hiint(d);
  return __hiloint2double(v == 0 ? hi : hi + (sh << 20), __double2loint(d));
}

// Running bound of the values a thread brings into the tile: their sum of
// magnitudes in FP32, rounded up, and the largest high word (the exponent when
// FP32's range does not hold the sum; a NaN or an infinity shows in it).
struct Mag {
  float s = 0.f;
  unsigned hi = 0;
  __device__ __forceinline__ void add(double x) {
    const unsigned a = (unsigned)((unsigned long long)__double_as_longlong(x) >> 32) & 0x7fffffffu;
    hi = max(hi, a);
    // the high word as a float, one unit of its last place up; 0 below 2^-126
    const unsigned f = a < (897u << 20) ? 0u : ((a - (896u << 20)) << 3) + 8u;
    s += __uint_as_float(f);
  }
};
// A line's scale from its sum and largest high word: the s with sum 2^s <= 2^top,
// terms the number of its values (for magnitudes out of FP32's range), at most
// 900 (values below 2^-960 vanish). kBad: not finite, or beyond 2^960.
constexpr int kBad = 1 << 20;
__device__ __forceinline__ int line_scale(float sum, unsigned hi, int terms, int top) {
  if (hi >= (1983u << 20)) return kBad;
  if (hi < (1123u << 20) && hi > (923u << 20)) {  // 2^-100 < largest < 2^100
    const int e = (int)(__float_as_uint(sum * 1.001f) >> 23) - 127;
    return top - 1 - e;
  }
  if (hi == 0) return 0;
  const int e = (int)(hi >> 20) - 1023 + (32 - __clz(terms));
  return min(top - 2 - e, 900);
}

// Scales of the lines of a tile whose line is threadIdx.x % L (L a power of two
// up to 32): NC lines share one (the largest of their sums). Sums in a fixed
// order; every thread of the block calls it.
template <int NC>
__device__ __forceinline__ void column_scales(float* s, unsigned hi, int L, int terms, int top, int* lsc) {
  __shared__ float ps[kMaxTh / 32][NC][32];
  __shared__ unsigned ph[kMaxTh / 32][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int off = 16; off >= L; off >>= 1) {
#pragma unroll
    for (int c = 0; c < NC; c++) s[c] += __shfl_xor_sync(FULL, s[c], off);
    hi = max(hi, __shfl_xor_sync(FULL, hi, off));
  }
  if (lane < L) {
#pragma unroll
    for (int c = 0; c < NC; c++) ps[w][c][lane] = s[c];
    ph[w][lane] = hi;
  }
  __syncthreads();
  if (threadIdx.x < L) {
    float m = 0.f;
    unsigned h = 0;
    for (int k = 0; k < nw; k++) h = max(h, ph[k][lane]);
#pragma unroll
    for (int c = 0; c < NC; c++) {
      float t = 0.f;
      for (int k = 0; k < nw; k++) t += ps[k][c][lane];
      m = fmaxf(m, t);
    }
    lsc[lane] = line_scale(m, h, terms, top);
  }
  __syncthreads();
}

// A raw complex double of the tile to fixed point at scale s (zero on a line
// that is not finite), with SWAP its parts exchanged.
template <bool SWAP>
__device__ __forceinline__ cx convert(double2 d, int s) {
  if (s == kBad) return cx{0, 0};
  return SWAP ? cx{to_fix(d.y, s), to_fix(d.x, s)} : cx{to_fix(d.x, s), to_fix(d.y, s)};
}
__device__ __forceinline__ double2 unscale(cx v, int sh, bool bad) {
  const double nan = __longlong_as_double(0x7ff8000000000000LL);
  return bad ? make_double2(nan, nan) : make_double2(to_f64(v.x, sh), to_f64(v.y, sh));
}

template <int R>
__device__ __forceinline__ void stage(const cx* __restrict__ src, cx* __restrict__ dst, const FxStage st, int L, int ld,
                                      const FxTwiddle* __restrict__ tw) {
  const int total = L * st.m;
  const int64_t half = half_unit();
  for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
    const int line = quot(idx, st.m, st.mq), j = idx - line * st.m;
    const int jb = quot(j, st.ns, st.nsq), jm = j - jb * st.ns;
    const cx* s = src + line * ld;
    cx v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = s[pad(j + r * st.m)];
    if (st.ns > 1) {
#pragma unroll
      for (int r = 1; r < R; r++) v[r] = cmul(v[r], tw_load(tw, jm * r * st.step), half);
    }
    dft<R>(v, half);
    cx* d = dst + line * ld;
    const int base = jb * st.ns * R + jm;
#pragma unroll
    for (int r = 0; r < R; r++) d[pad(base + r * st.ns)] = v[r];
  }
}

// Forward transform of L lines in a, b scratch; the result's buffer. Called by
// the whole block with a visible.
__device__ __noinline__ cx* lines(cx* a, cx* b, int L, int ld, const FxSched& sc, const FxTwiddle* tw) {
  cx *src = a, *dst = b;
  for (int s = 0; s < sc.nst; s++) {
    const FxStage& st = sc.st[s];
    if (st.R == 8) stage<8>(src, dst, st, L, ld, tw);
    else if (st.R == 4) stage<4>(src, dst, st, L, ld, tw);
    else if (st.R == 3) stage<3>(src, dst, st, L, ld, tw);
    else stage<2>(src, dst, st, L, ld, tw);
    __syncthreads();
    cx* t = src;
    src = dst;
    dst = t;
  }
  return src;
}

// Row tiles (R2C, C2R). `lpr` lanes (a power of two up to 32) share a row, in
// groups of R rows whose loads are in flight together, U values a lane held in
// registers between the load and the conversion (U R = 8). U = 0: rows of more
// than 256 values, a warp per row, through shared memory.
template <int U>
struct RowMap {
  static constexpr int R = U == 0 ? 1 : 8 / U;
};

// ---------------------------------------------------------------- R2C, axis 2
template <int U>
__device__ __forceinline__ void r2c_tile(int tile, const double* __restrict__ in, double2* __restrict__ out, int h,
                                         int nh, long long rows, long long N, long long Nk, int L, int lgp,
                                         const FxSched& sh, const FxTwiddle* __restrict__ tw_h,
                                         const FxTwiddle* __restrict__ tw_p) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int ld = fx_ld(h);
  cx* a = reinterpret_cast<cx*>(smraw);
  cx* b = a + L * ld;
  int* lsc = reinterpret_cast<int*>(b + L * ld);
  const int c = blockIdx.y;
  const long long r0 = (long long)tile * L;
  const int Lr = (int)min((long long)L, rows - r0);
  const int lpr = 1 << lgp, j0 = threadIdx.x & (lpr - 1), g0 = threadIdx.x >> lgp, ng = blockDim.x >> lgp;
  const double2* src = reinterpret_cast<const double2*>(in + (long long)c * N) + r0 * h + j0;
  constexpr int R = RowMap<U>::R;
  for (int lb = 0; lb < L; lb += ng * R) {
    double2 v[R][U > 0 ? U : 1];
    Mag g[R];
#pragma unroll
    for (int i = 0; i < R; i++) {
      const int l = lb + i * ng + g0;
      if (U > 0) {
#pragma unroll
        for (int u = 0; u < U; u++) {
          const bool on = l < Lr && j0 + u * lpr < h;
          v[i][u] = on ? __ldg(src + l * h + u * lpr) : make_double2(0.0, 0.0);
        }
      } else {
        for (int j = 0; j0 + j < h; j += lpr) {
          const double2 w = l < Lr ? __ldg(src + l * h + j) : make_double2(0.0, 0.0);
          g[i].add(w.x);
          g[i].add(w.y);
          if (l < L) reinterpret_cast<double2*>(a)[l * ld + pad(j0 + j)] = w;
        }
      }
    }
#pragma unroll
    for (int i = 0; i < R; i++) {
      const int l = lb + i * ng + g0;
#pragma unroll
      for (int u = 0; u < U; u++) {
        g[i].add(v[i][u].x);
        g[i].add(v[i][u].y);
      }
      for (int off = lpr >> 1; off; off >>= 1) {
        g[i].s += __shfl_xor_sync(FULL, g[i].s, off);
        g[i].hi = max(g[i].hi, __shfl_xor_sync(FULL, g[i].hi, off));
      }
      const int sc = line_scale(g[i].s, g[i].hi, 2 * h, 61);
      if (l < L) {
        if (j0 == 0) lsc[l] = sc;
        if (U > 0) {
#pragma unroll
          for (int u = 0; u < U; u++)
            if (j0 + u * lpr < h) a[l * ld + pad(j0 + u * lpr)] = convert<false>(v[i][u], sc);
        } else {
          for (int j = j0; j < h; j += lpr) {
            cx* p = a + l * ld + pad(j);
            *p = convert<false>(*reinterpret_cast<double2*>(p), sc);
          }
        }
      }
    }
  }
  __syncthreads();
  const cx* res = lines(a, b, L, ld, sh, tw_h);
  double2* dst = out + (long long)c * Nk + r0 * nh;
  for (int l = g0; l < Lr; l += ng) {
    const int sc = lsc[l];
    for (int k = j0; k < h; k += lpr) {
      const cx zk = res[l * ld + pad(k)];
      cx zc = res[l * ld + pad(k == 0 ? 0 : h - k)];
      zc.y = -zc.y;
      const cx sum = zk + zc, wd = cmul(zk - zc, tw_load(tw_p, k), half_unit());
      dst[l * nh + k] = unscale(cx{sum.x + wd.y, sum.y - wd.x}, -sc - 1, sc == kBad);
    }
  }
  for (int l = threadIdx.x; l < Lr; l += blockDim.x) {  // k = h: Re z0 - Im z0
    const cx z = res[l * ld];
    dst[l * nh + h] = unscale(cx{z.x - z.y, 0}, -lsc[l], lsc[l] == kBad);
  }
}

// A launch of fewer blocks than tiles (a gated solve that rarely runs) takes
// the tiles in turns; so do the other passes.
template <int U>
__global__ void __launch_bounds__(kMaxTh) k_r2c_fx(const double* __restrict__ in, double2* __restrict__ out, int h,
                                                   int nh, long long rows, long long N, long long Nk, int L, int lgp,
                                                   FxSched sh, const FxTwiddle* __restrict__ tw_h,
                                                   const FxTwiddle* __restrict__ tw_p, int tiles, const int* gate) {
  if (gate && *gate == 0) return;
  for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
    if (t != (int)blockIdx.x) __syncthreads();
    r2c_tile<U>(t, in, out, h, nh, rows, N, Nk, L, lgp, sh, tw_h, tw_p);
  }
}

// ------------------------------------------------------- C2C along axis 1
// Columns are numbered through all planes (q = i0 nh + k2), so that a tile may
// straddle two of them: nh is one past a multiple of the tile, and a tile per
// plane's remainder would leave up to half of the lanes idle. U values of a
// column per thread, held in registers between load and conversion.
template <bool INV, int U>
__device__ __forceinline__ void c2c_tile(int tile, double2* __restrict__ data, int n, int nh, int columns, long long Nk,
                                         int L, int lgL, const FxSched& sc, const FxTwiddle* __restrict__ tw) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ int lsc[32];
  const int ld = fx_ld(n);
  cx* a = reinterpret_cast<cx*>(smraw);
  cx* b = a + L * ld;
  const int c = blockIdx.y;
  const int l = threadIdx.x & (L - 1), p0 = threadIdx.x >> lgL, dp = blockDim.x >> lgL;
  const int q = tile * L + l;
  const int o = (int)((unsigned)q / (unsigned)nh);
  const int pe = q < columns ? n : 0;  // columns past the last hold nothing
  double2* base = data + (long long)c * Nk + (long long)o * n * nh + (q - o * nh) + (long long)p0 * nh;
  const long long step = (long long)dp * nh;
  double2 v[U];
  Mag g;
#pragma unroll
  for (int u = 0; u < U; u++) v[u] = p0 + u * dp < pe ? base[u * step] : make_double2(0.0, 0.0);
#pragma unroll
  for (int u = 0; u < U; u++) {
    g.add(v[u].x);
    g.add(v[u].y);
  }
  column_scales<1>(&g.s, g.hi, L, 2 * n, 62, lsc);
  const int s = lsc[l];
  cx* at = a + l * ld;
#pragma unroll
  for (int u = 0; u < U; u++)
    if (p0 + u * dp < n) at[pad(p0 + u * dp)] = convert<INV>(v[u], s);
  __syncthreads();
  const cx* res = lines(a, b, L, ld, sc, tw) + l * ld;
#pragma unroll
  for (int u = 0; u < U; u++)
    if (p0 + u * dp < pe) {
      const cx r = res[pad(p0 + u * dp)];
      base[u * step] = unscale(INV ? cx{r.y, r.x} : r, -s, s == kBad);
    }
}

template <bool INV, int U>
__global__ void __launch_bounds__(kMaxTh) k_c2c_fx(double2* __restrict__ data, int n, int nh, int columns, long long Nk,
                                                   int L, int lgL, FxSched sc, const FxTwiddle* __restrict__ tw,
                                                   int tiles, const int* gate) {
  if (gate && *gate == 0) return;
  for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
    if (t != (int)blockIdx.x) __syncthreads();
    c2c_tile<INV, U>(t, data, n, nh, columns, Nk, L, lgL, sc, tw);
  }
}

// ------------------------------------------------------------- Green's pass
// Unit wave vector of the wave numbers (k0, k1, k2), x 2^62, in axis order
// 2, 1, 0: f_a = w_a / n_a (w_a wrapped, Nyquist to -n/2) scaled by a power of
// two to 1/4 <= max|f| < 1/2, then times 1/|f|: an FP32 estimate and two Newton
// steps y += y (1 - F y^2) / 2 in fixed point (to 2^-58).
__device__ __forceinline__ void unit_wave_fx(int k0, int k1, int k2, const GreenFx& ga, Fx* g) {
  const int w2 = 2 * k2 < ga.n2 ? k2 : k2 - ga.n2, w1 = 2 * k1 < ga.n1 ? k1 : k1 - ga.n1,
            w0 = ga.is3d ? (2 * k0 < ga.n0 ? k0 : k0 - ga.n0) : 0;
  const int64_t f[3] = {(int64_t)w2 * ga.inv[2], (int64_t)w1 * ga.inv[1], (int64_t)w0 * ga.inv[0]};  // x 2^61
  uint64_t m = 0;
#pragma unroll
  for (int i = 0; i < 3; i++) m |= (uint64_t)(f[i] < 0 ? -f[i] : f[i]);
  const int z = __clzll((long long)m) - 3;  // to 2^60 <= max < 2^61, as x 2^62 (max is at most 2^60 before)
  Fx fx[3];
#pragma unroll
  for (int i = 0; i < 3; i++) fx[i] = fx_split(f[i] << z);
  FxAcc F2{0, 1 << 29};
#pragma unroll
  for (int i = 0; i < 3; i++) fx_mad(F2, fx[i], fx[i]);
  const int64_t F = fx_value<2>(F2);  // |f|^2 x 2^62, in [2^58, 2^61.6)
  const Fx Fs = fx_split(F);
  // y = 1/|f| in (1.1, 4], x 2^60
  const float yf = rsqrtf((float)(int32_t)(F >> 32) * 0x1p-30f);
  int64_t y = (int64_t)(int32_t)(yf * 0x1p28f) << 32;
#pragma unroll 1
  for (int it = 0; it < 2; it++) {
    const Fx ys = fx_split(y);
    FxAcc q{0, 0}, d{0, 0};
    fx_mad(q, fx_split(fmul(ys, Fs)), ys);                     // y^2 F x 2^120
    fx_mad(d, ys, fx_split((1ll << 60) - fx_value<4>(q)));     // y (1 - F y^2) x 2^120
    y += fx_value<3>(d);
  }
  const Fx ys = fx_split(y);
#pragma unroll
  for (int i = 0; i < 3; i++) {
    FxAcc d{0, 0};
    fx_mad(d, fx[i], ys);                                      // x 2^122
    int64_t v = fx_value<4>(d);
    const int64_t one = 1ll << 62;
    v = v > one ? one : (v < -one ? -one : v);
    g[i] = fx_split(v);
    if (g[i].l == INT32_MIN) g[i].l++;  // so that the halves can be negated
  }
}

// sigma / (2 mu) of one part (real or imaginary) of the eigenstrain spectrum e
// (with its headroom): t = tau / (2 mu) = e + lambda tr(e) / (2 mu) I, F = t g,
// G = g F, sigma / (2 mu) = F g + g F - 2 alpha G g g + c1 G I - t.
template <int NC>
__device__ __forceinline__ void green_part(const GreenFx& ga, const Fx* g, const int64_t* t, int64_t* sig) {
  constexpr int ND = NC == 3 ? 2 : 3;
  Fx T[NC];
#pragma unroll
  for (int c = 0; c < NC; c++) T[c] = fx_split(t[c]);
  constexpr int I3[3][3] = {{0, 5, 4}, {5, 1, 3}, {4, 3, 2}}, I2[3][3] = {{0, 2, 0}, {2, 1, 0}, {0, 0, 0}};
  Fx F[ND];
#pragma unroll
  for (int a = 0; a < ND; a++) {
    FxAcc q{0, 1 << 29};
#pragma unroll
    for (int b = 0; b < ND; b++) fx_mad(q, T[NC == 3 ? I2[a][b] : I3[a][b]], g[b]);
    F[a] = fx_split(fx_value<2>(q));
  }
  FxAcc gq{0, 1 << 29};
#pragma unroll
  for (int a = 0; a < ND; a++) fx_mad(gq, F[a], g[a]);
  const int64_t G = fx_value<2>(gq);
  const int64_t cG = rmul_s(G, ga.c1, ga.lams);
  const Fx A = fx_split(-rmul_s(G, ga.al2, 4));  // -2 alpha G
#pragma unroll
  for (int c = 0; c < NC; c++) {
    const int a = NC == 3 ? (c == 2 ? 0 : c) : (c < 3 ? c : (c == 3 ? 1 : 0));
    const int b = NC == 3 ? (c == 0 ? 0 : 1) : (c < 3 ? c : (c == 5 ? 1 : 2));
    FxAcc q{0, 1 << 29};
    fx_mad(q, F[a], g[b]);
    fx_mad(q, F[b], g[a]);
    fx_mad(q, A, fx_split(fmul(g[a], g[b])));
    sig[c] = fx_value<2>(q) - t[c] + (c < ND ? cG : 0);
  }
}

// U values per thread of each component's line in registers between load and
// conversion (0: through shared memory).
template <int NC, int U>
__device__ __forceinline__ void green_tile(int tile, double2* __restrict__ spec, int n, int stride, int inner,
                                           long long Nk, int L, int lgL, const FxSched& sc,
                                           const FxTwiddle* __restrict__ tw, const GreenFx& ga) {
  constexpr int ND = NC == 3 ? 2 : 3;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ int lsc[32], lsh[32];
  const int ld = fx_ld(n);
  cx* a = reinterpret_cast<cx*>(smraw);
  cx* b = a + NC * L * ld;
  const int q0 = tile * L;
  const int l = threadIdx.x & (L - 1), p0 = threadIdx.x >> lgL, dp = blockDim.x >> lgL;
  const int q = q0 + l;
  const bool in = q < inner;
  unsigned hi = 0;
  float cs[NC];
  const int pe = in ? n : 0;
  double2* base = spec + q + (long long)p0 * stride;
  const long long step = (long long)dp * stride;
  if (U > 0) {
    double2 v[NC][U > 0 ? U : 1];
#pragma unroll
    for (int c = 0; c < NC; c++)
#pragma unroll
      for (int u = 0; u < U; u++) v[c][u] = p0 + u * dp < pe ? base[c * Nk + u * step] : make_double2(0.0, 0.0);
#pragma unroll
    for (int c = 0; c < NC; c++) {
      Mag g;
#pragma unroll
      for (int u = 0; u < U; u++) {
        g.add(v[c][u].x);
        g.add(v[c][u].y);
      }
      cs[c] = g.s;
      hi = max(hi, g.hi);
    }
    column_scales<NC>(cs, hi, L, 2 * n, 62, lsc);  // the NC lines of a column share a scale
    const int s = lsc[l];
#pragma unroll
    for (int c = 0; c < NC; c++)
#pragma unroll
      for (int u = 0; u < U; u++)
        if (p0 + u * dp < n) a[(c * L + l) * ld + pad(p0 + u * dp)] = convert<false>(v[c][u], s);
  } else {
#pragma unroll
    for (int c = 0; c < NC; c++) {
      Mag g;
      for (int p = p0; p < n; p += dp) {
        const double2 v = in ? spec[c * Nk + (long long)p * stride + q] : make_double2(0.0, 0.0);
        g.add(v.x);
        g.add(v.y);
        reinterpret_cast<double2*>(a)[(c * L + l) * ld + pad(p)] = v;
      }
      cs[c] = g.s;
      hi = max(hi, g.hi);
    }
    column_scales<NC>(cs, hi, L, 2 * n, 62, lsc);
    const int s = lsc[l];
#pragma unroll 1
    for (int c = 0; c < NC; c++)
      for (int p = p0; p < n; p += dp) {
        cx* e = a + (c * L + l) * ld + pad(p);
        *e = convert<false>(*reinterpret_cast<double2*>(e), s);
      }
  }
  __syncthreads();
  cx* res = lines(a, b, NC * L, ld, sc, tw);
  // The operator in place, both parts of a wave number by one thread (its unit
  // vector is the larger half of the work), exchanged for the inverse
  // transform; the lines' new sums of magnitudes. Each wave number is worked on
  // at a shift z of its own, which leaves the operator kb bits of headroom above
  // its largest component, so that its error is relative to itself and not to
  // the column's largest wave number: with one shift per column a field of
  // mostly uniform eigenstrain (10% of spread, 512^2) was off by 6.1e-16 of the
  // stress, and FP64 passes by 1.8e-16.
  // the shifts, in the buffer that is free until the inverse transform (a kilobyte
  // of their own cost the second block per SM at lines of 1024: 288 us for 251)
  signed char* ex = reinterpret_cast<signed char*>(res == a ? b : a);
  float ns[NC];
#pragma unroll
  for (int c = 0; c < NC; c++) ns[c] = 0.f;
  {
    const int items = n << lgL;
    for (int i = threadIdx.x; i < items; i += blockDim.x) {
      const int l1 = i & (L - 1), p = i >> lgL, q1 = q0 + l1;
      if (q1 >= inner) continue;
      int k0, k1, k2;
      if (NC == 6 && ga.is3d) {
        k0 = p;
        k1 = q1 / ga.nh;
        k2 = q1 - k1 * ga.nh;
      } else {
        k0 = 0;
        k1 = p;
        k2 = q1;
      }
      cx* at = res + l1 * ld + pad(p);
      const int cstep = L * ld;
      int64_t t[2][NC], sg[2][NC];
      int m = 0;
#pragma unroll
      for (int c = 0; c < NC; c++) {
        const cx v = at[c * cstep];
        t[0][c] = v.x;
        t[1][c] = v.y;
        const int hx = (int)(v.x >> 32), hy = (int)(v.y >> 32);
        m |= (hx ^ (hx >> 31)) | (hy ^ (hy >> 31));
      }
      // magnitudes are below 2^(32 + bits of m): to below 2^(61 - kb)
      const int z = 29 - ga.kb - (32 - __clz(m));
      ex[i] = (signed char)z;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        int64_t tr = 0;
#pragma unroll
        for (int c = 0; c < NC; c++) {
          t[h][c] = z < 0 ? shift_round(t[h][c], -z) : (int64_t)((uint64_t)t[h][c] << z);
          if (c < ND) tr += t[h][c];
        }
        const int64_t lt = rmul_s(tr, ga.lam, ga.lams);
#pragma unroll
        for (int c = 0; c < ND; c++) t[h][c] += lt;
      }
      if ((k0 | k1 | k2) == 0) {
        // -C:eps_hat; the mean strain's part is added by the last pass
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int c = 0; c < NC; c++) sg[h][c] = -t[h][c];
      } else {
        Fx g[3];
        unit_wave_fx(k0, k1, k2, ga, g);
        // on a Nyquist plane the average over the signs of the Nyquist
        // components (3D: every choice; 2D: all of them together, the
        // reference's real part)
        const int ny = (2 * k2 == ga.n2 ? 1 : 0) | (2 * k1 == ga.n1 ? 2 : 0) | (NC == 6 && 2 * k0 == ga.n0 ? 4 : 0);
#pragma unroll
        for (int c = 0; c < NC; c++) sg[0][c] = sg[1][c] = 0;
        int nv = 0;
#pragma unroll 1
        for (int f = 0; f <= ny; f++) {
          if ((f & ~ny) || (NC == 3 && f != 0 && f != ny)) continue;
          Fx gm[3];
#pragma unroll
          for (int k = 0; k < 3; k++) gm[k] = (f >> k & 1) ? Fx{-g[k].h, -g[k].l} : g[k];
#pragma unroll
          for (int h = 0; h < 2; h++) {
            int64_t s1[NC];
            green_part<NC>(ga, gm, t[h], s1);
#pragma unroll
            for (int c = 0; c < NC; c++) sg[h][c] += s1[c];
          }
          nv++;
        }
        if (nv > 1) {
          const int sh = nv == 2 ? 1 : (nv == 4 ? 2 : 3);
#pragma unroll
          for (int h = 0; h < 2; h++)
#pragma unroll
            for (int c = 0; c < NC; c++) sg[h][c] = shift_round(sg[h][c], sh);
        }
      }
#pragma unroll
      for (int c = 0; c < NC; c++) {
        at[c * cstep] = cx{sg[1][c], sg[0][c]};
        // in units of 2^32, rounded up
        ns[c] += ((float)(abs((int)(sg[0][c] >> 32)) + 1) + (float)(abs((int)(sg[1][c] >> 32)) + 1)) *
                 __uint_as_float((unsigned)(127 - z) << 23);
      }
    }
  }
  // sums in units of 2^32: a top of 30 puts them below 2^62. A column of zeros
  // has the largest shift.
  column_scales<NC>(ns, 0x3ff00000u, L, 2 * n, 30, lsh);
  if (threadIdx.x < L) lsh[threadIdx.x] = min(lsh[threadIdx.x], 62);
  __syncthreads();
  {
    const int sh = lsh[l];
    for (int p = p0; p < pe; p += dp) {
      const int z = ex[p * L + l] - sh;  // to the line's own scale
#pragma unroll
      for (int c = 0; c < NC; c++) {
        cx* e = res + (c * L + l) * ld + pad(p);
        const cx v = *e;
        *e = z > 0 ? cx{shift_round(v.x, z), shift_round(v.y, z)}
                   : cx{(int64_t)((uint64_t)v.x << min(-z, 62)), (int64_t)((uint64_t)v.y << min(-z, 62))};
      }
    }
  }
  __syncthreads();
  const cx* res2 = lines(res, res == a ? b : a, NC * L, ld, sc, tw);
  const int s = lsc[l], so = -s - lsh[l];
  if (in)
#pragma unroll 1
    for (int c = 0; c < NC; c++)
      for (int p = p0; p < n; p += dp) {
        const cx v = res2[(c * L + l) * ld + pad(p)];
        spec[c * Nk + (long long)p * stride + q] = unscale(cx{v.y, v.x}, so, s == kBad);
      }
}

template <int NC, int U>
__global__ void __launch_bounds__(kMaxTh, 2) k_green_fx(double2* __restrict__ spec, int n, int stride, int inner,
                                                        long long Nk, int L, int lgL, FxSched sc,
                                                        const FxTwiddle* __restrict__ tw, GreenFx ga, int tiles,
                                                        const int* gate) {
  if (gate && *gate == 0) return;
  for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
    if (t != (int)blockIdx.x) __syncthreads();
    green_tile<NC, U>(t, spec, n, stride, inner, Nk, L, lgL, sc, tw, ga);
  }
}

// ---------------------------------------------------------------- C2R, axis 2
// Rows of one component (blockIdx.y), the block's sum of the component to msum.
// The factor 2 mu / N of the solve and the mean strain's uniform stress are
// applied here, in FP64 (three operations per value on an otherwise idle pipe).
template <int U>
__device__ __forceinline__ void c2r_tile(int tile, int tiles, const double2* __restrict__ in, int nc, int h, int nh,
                                         long long rows, long long N, long long Nk, int L, int lgp, const FxSched& sh,
                                         const FxTwiddle* __restrict__ tw_h, const FxTwiddle* __restrict__ tw_p,
                                         double factor, const double* __restrict__ ebar, double lambda, double mu,
                                         double* __restrict__ sig, double* __restrict__ msum) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ double red[kMaxTh / 32];
  const int ld = fx_ld(h + 1);
  cx* a = reinterpret_cast<cx*>(smraw);
  cx* b = a + L * ld;
  int* lsc = reinterpret_cast<int*>(b + L * ld);
  const int c = blockIdx.y;
  const long long r0 = (long long)tile * L;
  const int Lr = (int)min((long long)L, rows - r0);
  const int lpr = 1 << lgp, j0 = threadIdx.x & (lpr - 1), g0 = threadIdx.x >> lgp, ng = blockDim.x >> lgp;
  // C:<eps> of this component
  const int nd = nc == 3 ? 2 : 3;
  double cs = 0;
  if (ebar) {
    double tr = 0;
    for (int k = 0; k < nd; k++) tr += ebar[k];
    cs = (c < nd ? lambda * tr : 0.0) + 2.0 * mu * ebar[c];
  }
  const double2* src = in + (long long)c * Nk + r0 * nh;
  constexpr int R = RowMap<U>::R;
  for (int lb = 0; lb < L; lb += ng * R) {
    double2 v[R][U > 0 ? U : 1], x[R];
    Mag g[R];
#pragma unroll
    for (int i = 0; i < R; i++) {
      const int l = lb + i * ng + g0;
      // value h with the row's first lane
      x[i] = l < Lr && j0 == 0 ? __ldg(src + l * nh + h) : make_double2(0.0, 0.0);
      if (U > 0) {
#pragma unroll
        for (int u = 0; u < U; u++) {
          const bool on = l < Lr && j0 + u * lpr < h;
          v[i][u] = on ? __ldg(src + l * nh + j0 + u * lpr) : make_double2(0.0, 0.0);
        }
      } else {
        for (int j = j0; j < h; j += lpr) {
          const double2 w = l < Lr ? __ldg(src + l * nh + j) : make_double2(0.0, 0.0);
          g[i].add(w.x);
          g[i].add(w.y);
          if (l < L) reinterpret_cast<double2*>(a)[l * ld + pad(j)] = w;
        }
      }
    }
#pragma unroll
    for (int i = 0; i < R; i++) {
      const int l = lb + i * ng + g0;
      g[i].add(x[i].x);
      g[i].add(x[i].y);
#pragma unroll
      for (int u = 0; u < U; u++) {
        g[i].add(v[i][u].x);
        g[i].add(v[i][u].y);
      }
      for (int off = lpr >> 1; off; off >>= 1) {
        g[i].s += __shfl_xor_sync(FULL, g[i].s, off);
        g[i].hi = max(g[i].hi, __shfl_xor_sync(FULL, g[i].hi, off));
      }
      // four times the half spectrum's sum bounds every partial sum of Z
      const int sc = line_scale(g[i].s, g[i].hi, 2 * nh, 60);
      if (l < L) {
        if (j0 == 0) {
          lsc[l] = sc;
          a[l * ld + pad(h)] = convert<false>(x[i], sc);
        }
        if (U > 0) {
#pragma unroll
          for (int u = 0; u < U; u++)
            if (j0 + u * lpr < h) a[l * ld + pad(j0 + u * lpr)] = convert<false>(v[i][u], sc);
        } else {
          for (int j = j0; j < h; j += lpr) {
            cx* p = a + l * ld + pad(j);
            *p = convert<false>(*reinterpret_cast<double2*>(p), sc);
          }
        }
      }
    }
  }
  __syncthreads();
  // Z = E + i O, its parts exchanged (inverse transform)
  for (int l = g0; l < L; l += ng) {
    const cx* row = a + l * ld;
    for (int k = j0; k < h; k += lpr) {
      const cx xk = row[pad(k)];
      cx xc = row[pad(h - k)];
      xc.y = -xc.y;
      FxTwiddle t = tw_load(tw_p, k);
      t.i = Fx{-t.i.h, -t.i.l};
      const cx e = xk + xc, od = cmul(xk - xc, t, half_unit());
      b[l * ld + pad(k)] = cx{e.y + od.x, e.x - od.y};
    }
  }
  __syncthreads();
  const cx* res = lines(b, a, L, ld, sh, tw_h);
  double part = 0;
  double2* out = reinterpret_cast<double2*>(sig + (long long)c * N) + r0 * h;
  for (int l = g0; l < Lr; l += ng) {
    const int sc = lsc[l];
    for (int j = j0; j < h; j += lpr) {
      const cx z = res[l * ld + pad(j)];
      const double2 d = unscale(cx{z.y, z.x}, -sc, sc == kBad);
      const double x = __fma_rn(d.x, factor, cs), y = __fma_rn(d.y, factor, cs);
      out[l * h + j] = make_double2(x, y);
      part += x + y;
    }
  }
  if (msum) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int off = 16; off > 0; off >>= 1) part += __shfl_xor_sync(FULL, part, off);
    if (lane == 0) red[w] = part;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0;
      for (int k = 0; k < (int)(blockDim.x >> 5); k++) t += red[k];
      msum[(long long)c * tiles + tile] = t;
    }
  }
}

template <int U>
__global__ void __launch_bounds__(kMaxTh) k_c2r_fx(const double2* __restrict__ in, int nc, int h, int nh,
                                                   long long rows, long long N, long long Nk, int L, int lgp,
                                                   FxSched sh, const FxTwiddle* __restrict__ tw_h,
                                                   const FxTwiddle* __restrict__ tw_p, double factor,
                                                   const double* __restrict__ ebar, double lambda, double mu,
                                                   double* __restrict__ sig, double* __restrict__ msum, int tiles,
                                                   const int* gate) {
  if (gate && *gate == 0) return;
  for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
    if (t != (int)blockIdx.x) __syncthreads();
    c2r_tile<U>(t, tiles, in, nc, h, nh, rows, N, Nk, L, lgp, sh, tw_h, tw_p, factor, ebar, lambda, mu, sig, msum);
  }
}

int ilog2(int v) {
  int l = 0;
  while ((1 << l) < v) l++;
  return l;
}
int warps32(long long t) { return (int)std::max<long long>(32, std::min<long long>(kMaxTh, (t + 31) / 32 * 32)); }

// Row passes: lanes per row, values per lane (0: more than eight), threads for
// a tile of L rows (about `each` values a thread).
struct RowLaunch {
  int lgp, U, threads;
};
RowLaunch row_launch(int h, int L, int each) {
  RowLaunch r;
  r.lgp = std::min(5, ilog2(h));
  const int u = (h + (1 << r.lgp) - 1) >> r.lgp;
  r.U = u <= 1 ? 1 : u <= 2 ? 2 : u <= 4 ? 4 : u <= 8 ? 8 : 0;
  r.threads = warps32((long long)L * h / each);
  return r;
}
// Column passes: threads for L columns of n (about `each` values a thread, at
// most eight) and the values a thread then holds.
struct ColLaunch {
  int U, threads;
};
ColLaunch col_launch(int n, int L, int each) {
  ColLaunch c;
  c.threads = std::max(warps32((long long)L * n / each), L);
  const int u = (n * L + c.threads - 1) / c.threads;
  c.U = u <= 1 ? 1 : u <= 2 ? 2 : u <= 4 ? 4 : u <= 8 ? 8 : 0;
  return c;
}

template <typename F>
void raise_limit(F* k, int optin) {
  cudaFuncAttributes fa;
  if (cudaFuncGetAttributes(&fa, (const void*)k) != cudaSuccess) { (void)cudaGetLastError(); return; }
  const int bytes = optin - (int)fa.sharedSizeBytes;
  if (bytes > 0 &&
      cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess)
    (void)cudaGetLastError();
}

// Blocks of a pass over `tiles` tiles of `comps` components. A block each; for a
// gated solve that rarely runs, two blocks per SM in all: a grid whose blocks
// return at once takes 6 to 7 us with 2000 blocks of 100 KB, 1.5 us then.
dim3 fx_grid(const SolveArgs& a, int tiles, int comps) {
  const int most = 304 / comps;
  return dim3((unsigned)(a.rare && tiles > most ? most : tiles), (unsigned)comps);
}

// The kernels of a pass by the values a thread holds.
auto r2c_kernel(int U) {
  return U == 1 ? k_r2c_fx<1> : U == 2 ? k_r2c_fx<2> : U == 4 ? k_r2c_fx<4> : U == 8 ? k_r2c_fx<8> : k_r2c_fx<0>;
}
auto c2r_kernel(int U) {
  return U == 1 ? k_c2r_fx<1> : U == 2 ? k_c2r_fx<2> : U == 4 ? k_c2r_fx<4> : U == 8 ? k_c2r_fx<8> : k_c2r_fx<0>;
}
template <bool INV>
auto c2c_kernel(int U) {
  return U == 1 || U == 2 ? k_c2c_fx<INV, 2> : U == 4 ? k_c2c_fx<INV, 4> : k_c2c_fx<INV, 8>;
}
auto green_kernel(int nc, int U) {
  if (nc == 6) return U == 1 ? k_green_fx<6, 1> : U == 2 ? k_green_fx<6, 2> : k_green_fx<6, 0>;
  return U == 1 ? k_green_fx<3, 1> : U == 2 ? k_green_fx<3, 2> : k_green_fx<3, 0>;
}

// Green's pass over n values and `inner` columns: along axis 0, or along axis 1
// of a grid without axis 0 (with three components or six).
void launch_green(const FFTPlan& p, int n, int inner, const SolveArgs& a, const FxSched& x, const FxTwiddle* tw,
                  const GreenFx& ga, cudaStream_t st) {
  const ColLaunch c = col_launch(n, p.x.Lg, p.x.eg);
  const int tiles = (inner + p.x.Lg - 1) / p.x.Lg;
  const dim3 grid = fx_grid(a, tiles, 1);
  const auto k = green_kernel(p.nc, c.U);
  k<<<grid, c.threads, p.x.smem_g, st>>>(reinterpret_cast<double2*>(a.spec), n, inner, inner, p.Nk, p.x.Lg, ilog2(p.x.Lg), x,
                                        tw, ga, tiles, a.gate);
}

template <bool INV>
void launch_c2c(const FFTPlan& p, const SolveArgs& a, const FxSched& x, cudaStream_t st) {
  const ColLaunch c = col_launch(p.n1, p.x.Ly, p.x.ey);
  const int columns = p.n0 * p.nh, tiles = (columns + p.x.Ly - 1) / p.x.Ly;
  const dim3 grid = fx_grid(a, tiles, p.nc);
  const auto k = c2c_kernel<INV>(c.U);
  k<<<grid, c.threads, p.x.smem_y, st>>>(reinterpret_cast<double2*>(a.spec), p.n1, p.nh, columns, p.Nk, p.x.Ly,
                                        ilog2(p.x.Ly), x, p.x.tw_1, tiles, a.gate);
}

}  // namespace

bool fftx_fits(int n2, double lambda, double mu) {
  if (n2 > kFxLongest || !(mu > 0) || !std::isfinite(lambda) || !std::isfinite(mu)) return false;
  const double l = std::fabs(lambda) / mu, al = (lambda + mu) / (lambda + 2 * mu);
  return l <= 256 && std::fabs(al) <= 1.5;
}

// Every kernel that a schedule of a grid may take (each pass by the values a
// thread holds), or with `plan` those of its solve: some calls prepare one solve
// and cannot afford a look at every kernel (two runtime calls each).
void fftx_init(const FFTPlan* plan) {
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess || optin <= 0)
    optin = 227 * 1024;
  if (plan) {
    const FFTPlan& p = *plan;
    const int ux = row_launch(p.h, p.x.Lx, p.x.ex).U;
    raise_limit(r2c_kernel(ux), optin);
    raise_limit(c2r_kernel(ux), optin);
    raise_limit(green_kernel(p.nc, col_launch(p.n0 > 1 ? p.n0 : p.n1, p.x.Lg, p.x.eg).U), optin);
    if (p.n0 > 1) {
      const int uy = col_launch(p.n1, p.x.Ly, p.x.ey).U;
      raise_limit(c2c_kernel<false>(uy), optin);
      raise_limit(c2c_kernel<true>(uy), optin);
    }
    return;
  }
  for (int u : {0, 1, 2, 4, 8}) {
    raise_limit(r2c_kernel(u), optin);
    raise_limit(c2r_kernel(u), optin);
  }
  for (int u : {2, 4, 8}) {
    raise_limit(c2c_kernel<false>(u), optin);
    raise_limit(c2c_kernel<true>(u), optin);
  }
  for (int nc : {3, 6})
    for (int u : {0, 1, 2}) raise_limit(green_kernel(nc, u), optin);
}

void fftx_spectrum(const FFTPlan& p, const SolveArgs& a, cudaStream_t st, int64_t* launches) {
  double2* spec = reinterpret_cast<double2*>(a.spec);
  const long long rows = (long long)p.n0 * p.n1;
  const FxSched xh = fx_sched(p.x.sh), x1 = fx_sched(p.x.s1), x0 = fx_sched(p.x.s0);
  const int tiles = (int)((rows + p.x.Lx - 1) / p.x.Lx);
  const dim3 gx = fx_grid(a, tiles, p.nc);
  const RowLaunch r = row_launch(p.h, p.x.Lx, p.x.ex);
  const auto k = r2c_kernel(r.U);
  k<<<gx, r.threads, p.x.smem_x, st>>>(a.eps, spec, p.h, p.nh, rows, p.N, p.Nk, p.x.Lx, r.lgp, xh, p.x.tw_h, p.x.tw_p, tiles,
                                      a.gate);
  GreenFx ga;
  fx_green_constants(p.n0, p.n1, p.n2, a.lambda, a.mu, &ga);
  if (p.n0 > 1) {
    launch_c2c<false>(p, a, x1, st);
    launch_green(p, p.n0, p.n1 * p.nh, a, x0, p.x.tw_0, ga, st);
    launch_c2c<true>(p, a, x1, st);
  } else {
    launch_green(p, p.n1, p.nh, a, x1, p.x.tw_1, ga, st);
  }
  if (launches) *launches += p.n0 > 1 ? 4 : 2;
}

double fftx_factor(const FFTPlan& p, double mu) { return (double)(2 * (long double)mu / (long double)p.N); }

void fftx_c2r(const FFTPlan& p, const SolveArgs& a, cudaStream_t st, int64_t* launches) {
  const long long rows = (long long)p.n0 * p.n1;
  const int tiles = (int)((rows + p.x.Lx - 1) / p.x.Lx);
  const dim3 gx = fx_grid(a, tiles, p.nc);
  const RowLaunch r = row_launch(p.h, p.x.Lx, p.x.ex);
  const auto k = c2r_kernel(r.U);
  k<<<gx, r.threads, p.x.smem_x, st>>>(reinterpret_cast<const double2*>(a.spec), p.nc, p.h, p.nh, rows, p.N, p.Nk, p.x.Lx,
                                      r.lgp, fx_sched(p.x.sh), p.x.tw_h, p.x.tw_p, fftx_factor(p, a.mu), a.ebar, a.lambda, a.mu,
                                      a.sig64, a.msum, tiles, a.gate);
  if (launches) *launches += 1;
}

}  // namespace stz
