// fft.cu -- hand-written mixed-radix FFT and the fused Green's-operator pass.
//
// Layout: a real field is [N] with s = (i0*n1 + i1)*n2 + i2; its half
// spectrum is [n0][n1][nh] complex with nh = n2/2 + 1 (R2C along axis 2).
// A 3D solve is five passes:
//   R2C along axis 2  ->  C2C along axis 1  ->  [C2C axis 0, Green, inverse C2C
//   axis 0] in one kernel  ->  inverse C2C along axis 1  ->  C2R along axis 2
// and a 2D solve (n0 == 1) three: R2C axis 2 -> [axis 1, Green, inverse] -> C2R.
// Every pass stages a tile of lines in shared memory and runs a Stockham
// autosort FFT over it with radix-8/4/3/2 butterflies in registers.
//
// Green's operator (elastic.c:802-809, generalised to 3D): with g the unit
// wave vector of Grad() (init.c:112-140; wrap s - round(s), Nyquist -> -1/2),
// tau = C:eps*, F = tau.g, G = g.F,
//   eps_ij = (F_i g_j + F_j g_i)/(2 mu) - (alpha/mu) G g_i g_j,
//   alpha = (lambda + mu)/(lambda + 2 mu),
// and the pass writes the stress spectrum C:(eps - eps*) directly; the k = 0
// term is C:(N <eps> - eps*_hat(0)). The reference transforms complex fields
// and keeps the real part of the inverse; on a Nyquist plane its operator at k
// and at -k differ (g picks -1/2 for both), so the real part it keeps is the
// result of the average of the two operators. This pass applies that average
// explicitly, which keeps the spectrum Hermitian and the C2R exact. In 3D,
// where the reference has no code, wave vectors with Nyquist components use the
// average over every sign choice of those components; this differs from the
// two-operator average only where two or more components sit on a Nyquist
// plane, and makes the discrete Green's function symmetric under the
// reflection of each axis (the incremental solver relies on that).
#include <cmath>
#include <cstdio>
#include <cstring>
#include <algorithm>
#include <array>
#include <map>
#include <mutex>
#include <vector>

#include "fft.cuh"
#include "fftx.cuh"
#include "kmc.cuh"

namespace stz {
namespace {

// FP32 pair: the unevaluated sum hi + lo of two floats (|lo| <= half an ulp of
// hi), about 48 significant bits, with error-free FP32 transformations
// (Knuth's TwoSum, Dekker's product through an FMA). GB300 issues FP64 at 1/64
// of its FP32 rate, and an FFT pass in FP64 is bound by that rate; in pairs the
// same pass runs on the FP32 pipes. A pair and a complex pair take 8 and 16
// bytes, as a double and a double2 do, so every layout is shared.
struct dfl {
  float hi, lo;
  dfl() = default;
  __host__ __device__ constexpr dfl(float h, float l) : hi(h), lo(l) {}
  __host__ __device__ dfl(double x) : hi((float)x), lo((float)(x - (double)(float)x)) {}
  __host__ __device__ explicit operator double() const { return (double)hi + (double)lo; }
};
__device__ __forceinline__ dfl df_norm(float s, float e) {
  const float h = __fadd_rn(s, e);
  return dfl(h, __fsub_rn(e, __fsub_rn(h, s)));
}
__device__ __forceinline__ dfl operator+(dfl a, dfl b) {
  const float s = __fadd_rn(a.hi, b.hi);
  const float bp = __fsub_rn(s, a.hi);
  const float e = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bp)), __fsub_rn(b.hi, bp));
  return df_norm(s, __fadd_rn(e, __fadd_rn(a.lo, b.lo)));
}
__device__ __forceinline__ dfl operator-(dfl a) { return dfl(-a.hi, -a.lo); }
__device__ __forceinline__ dfl operator-(dfl a, dfl b) { return a + (-b); }
__device__ __forceinline__ dfl operator*(dfl a, dfl b) {
  const float p = __fmul_rn(a.hi, b.hi);
  const float e = __fmaf_rn(a.hi, b.hi, -p);
  return df_norm(p, __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.lo, b.hi, e)));
}
__device__ __forceinline__ dfl operator/(dfl a, dfl b) {
  const float q1 = __fdiv_rn(a.hi, b.hi);
  const dfl r = a - dfl(q1, 0.f) * b;
  return df_norm(q1, __fdiv_rn(r.hi, b.hi));
}
struct __align__(16) df2 {
  dfl x, y;
};

template <typename T> struct VT;
template <> struct VT<double> { using V = double2; };
template <> struct VT<float> { using V = float2; };
template <> struct VT<dfl> { using V = df2; };

// An FP64 value as a pair without FP64 instructions (GB300 issues FP64 at
// 1/64 of its FP32 rate, and the conversions of dfl(double) run there): hi is
// x with its significand cut to 24 bits, built from the bit fields; the 29
// bits cut off are exactly r * 2^(e - 1075) and are rounded to a float; the
// pair is then renormalised (|x - hi - lo| <= 2^-48 |x|). Below 2^-74 in
// magnitude lo is dropped, below 2^-126 the value becomes a signed zero
// (absolute errors under 2^-98 and 2^-126); beyond the float range it becomes
// the infinity of its sign, and a NaN stays a NaN. Every case is integer work:
// an FP64 conversion in a rarely taken branch is still executed for every
// value once the compiler turns the branch into a select.
__device__ __forceinline__ dfl split_f64(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned hw = (unsigned)(b >> 32), lw = (unsigned)b;
  const int e = (int)((hw >> 20) & 0x7ffu);
  const unsigned sg = hw & 0x80000000u;
  if (e > 1023 + 127) {
    const bool nan = e == 2047 && ((hw & 0xfffffu) | lw) != 0u;
    return dfl(__uint_as_float(nan ? 0x7fc00000u : (sg | 0x7f800000u)), 0.f);
  }
  if (e < 1023 - 126) return dfl(__uint_as_float(sg), 0.f);
  const float h = __uint_as_float(sg | ((unsigned)(e - 1023 + 127) << 23) | ((hw & 0xfffffu) << 3) | (lw >> 29));
  float l = 0.f;
  if (e >= 1075 - 126) {
    const float scale = __uint_as_float((unsigned)(e - 1075 + 127) << 23);
    l = __uint_as_float(__float_as_uint(__fmul_rn(__uint2float_rn(lw & 0x1fffffffu), scale)) | sg);
  }
  const float s = __fadd_rn(h, l);
  return dfl(s, __fsub_rn(l, __fsub_rn(s, h)));
}
template <typename T> __device__ __forceinline__ T from_f64(double x) { return (T)x; }
template <> __device__ __forceinline__ dfl from_f64<dfl>(double x) { return split_f64(x); }

template <typename V> __device__ __forceinline__ V vadd(V a, V b) { return V{a.x + b.x, a.y + b.y}; }
template <typename V> __device__ __forceinline__ V vsub(V a, V b) { return V{a.x - b.x, a.y - b.y}; }
template <typename V> __device__ __forceinline__ V vmul(V a, V b) {
  return V{a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x};
}
// S * i * a
template <int S, typename V> __device__ __forceinline__ V vmuli(V a) {
  return S > 0 ? V{-a.y, a.x} : V{a.y, -a.x};
}

template <typename V, int S> __device__ __forceinline__ void dft2(V* v) {
  V a = v[0], b = v[1];
  v[0] = vadd(a, b);
  v[1] = vsub(a, b);
}
template <typename V, int S> __device__ __forceinline__ void dft4(V* v) {
  V a0 = vadd(v[0], v[2]), a1 = vsub(v[0], v[2]);
  V a2 = vadd(v[1], v[3]), a3 = vsub(v[1], v[3]);
  V b3 = vmuli<S>(a3);
  v[0] = vadd(a0, a2);
  v[2] = vsub(a0, a2);
  v[1] = vadd(a1, b3);
  v[3] = vsub(a1, b3);
}
template <typename V, int S> __device__ __forceinline__ void dft3(V* v) {
  using T = decltype(v[0].x);
  const T c = (T)-0.5;
  const T s = (T)(S * 0.86602540378443864676);
  V t = vadd(v[1], v[2]), u = vsub(v[1], v[2]);
  V y0 = vadd(v[0], t);
  V m = V{v[0].x + c * t.x, v[0].y + c * t.y};
  V q = V{-s * u.y, s * u.x};
  v[0] = y0;
  v[1] = vadd(m, q);
  v[2] = vsub(m, q);
}
template <typename V, int S> __device__ __forceinline__ void dft8(V* v) {
  using T = decltype(v[0].x);
  const T r = (T)0.70710678118654752440;
  V e[4] = {v[0], v[2], v[4], v[6]};
  V o[4] = {v[1], v[3], v[5], v[7]};
  dft4<V, S>(e);
  dft4<V, S>(o);
  o[1] = V{r * (o[1].x - S * o[1].y), r * (S * o[1].x + o[1].y)};
  o[2] = vmuli<S>(o[2]);
  o[3] = V{r * (-o[3].x - S * o[3].y), r * (S * o[3].x - o[3].y)};
#pragma unroll
  for (int k = 0; k < 4; k++) {
    v[k] = vadd(e[k], o[k]);
    v[k + 4] = vsub(e[k], o[k]);
  }
}

template <typename V, int R, int S>
__device__ __forceinline__ void stage(const V* __restrict__ src, V* __restrict__ dst, int n, int L, int ld,
                                      int ns, const V* __restrict__ tw, int tid, int nth) {
  const int m = n / R;
  const int step = n / (ns * R);
  const int total = L * m;
  for (int idx = tid; idx < total; idx += nth) {
    const int line = idx / m;
    const int j = idx - line * m;
    const int jm = j % ns;
    const V* s = src + line * ld;
    V v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = s[j + r * m];
    if (jm != 0) {
#pragma unroll
      for (int r = 1; r < R; r++) {
        V w = tw[jm * r * step];
        if (S > 0) w.y = -w.y;
        v[r] = vmul(v[r], w);
      }
    }
    if (R == 2) dft2<V, S>(v);
    else if (R == 3) dft3<V, S>(v);
    else if (R == 4) dft4<V, S>(v);
    else dft8<V, S>(v);
    V* d = dst + line * ld;
    const int base = (j / ns) * ns * R + jm;
#pragma unroll
    for (int r = 0; r < R; r++) d[base + r * ns] = v[r];
  }
}

// FFT of L lines of length sc.n stored with leading dimension ld in a; b is
// scratch of the same size. Returns the buffer that holds the result. Must be
// called by the whole block with the input visible (after __syncthreads).
template <typename V, int S>
__device__ V* fft_lines(V* a, V* b, int L, int ld, const Sched& sc, const V* tw) {
  V* src = a;
  V* dst = b;
  int ns = 1;
  for (int s = 0; s < sc.nst; s++) {
    const int R = sc.r[s];
    if (R == 8) stage<V, 8, S>(src, dst, sc.n, L, ld, ns, tw, threadIdx.x, blockDim.x);
    else if (R == 4) stage<V, 4, S>(src, dst, sc.n, L, ld, ns, tw, threadIdx.x, blockDim.x);
    else if (R == 3) stage<V, 3, S>(src, dst, sc.n, L, ld, ns, tw, threadIdx.x, blockDim.x);
    else stage<V, 2, S>(src, dst, sc.n, L, ld, ns, tw, threadIdx.x, blockDim.x);
    __syncthreads();
    V* t = src;
    src = dst;
    dst = t;
    ns *= R;
  }
  return src;
}

// ---------------------------------------------------------------- R2C, axis 2
template <typename T>
__global__ void __launch_bounds__(256) k_r2c_x(const double* __restrict__ in, typename VT<T>::V* __restrict__ out,
                                               int n2, int h, int nh, long long rows, long long N, long long Nk,
                                               int L, Sched sh, const typename VT<T>::V* __restrict__ tw_h,
                                               const typename VT<T>::V* __restrict__ tw_p, const int* gate) {
  using V = typename VT<T>::V;
  if (gate && *gate == 0) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int ld = h + 1;
  V* a = reinterpret_cast<V*>(smraw);
  V* b = a + L * ld;
  const int c = blockIdx.y;
  const long long r0 = (long long)blockIdx.x * L;
  const double2* src = reinterpret_cast<const double2*>(in + (long long)c * N);
  for (int idx = threadIdx.x; idx < L * h; idx += blockDim.x) {
    const int l = idx / h, j = idx - l * h;
    const long long r = r0 + l;
    V z = V{0, 0};
    if (r < rows) {
      double2 v = src[(r * n2) / 2 + j];
      z = V{from_f64<T>(v.x), from_f64<T>(v.y)};
    }
    a[l * ld + j] = z;
  }
  __syncthreads();
  V* res = fft_lines<V, -1>(a, b, L, ld, sh, tw_h);
  V* dst = out + (long long)c * Nk;
  for (int idx = threadIdx.x; idx < L * nh; idx += blockDim.x) {
    const int l = idx / nh, k = idx - l * nh;
    const long long r = r0 + l;
    if (r >= rows) continue;
    V zk = res[l * ld + (k == h ? 0 : k)];
    V zc = res[l * ld + (k == 0 ? 0 : h - k)];
    zc.y = -zc.y;
    V sum = vadd(zk, zc), dif = vsub(zk, zc);
    V wd = vmul(tw_p[k], dif);
    dst[r * nh + k] = V{(T)0.5 * (sum.x + wd.y), (T)0.5 * (sum.y - wd.x)};
  }
}

// ------------------------------------------------------- C2C along axis 1 / 0
template <typename T, int S>
__global__ void __launch_bounds__(256) k_c2c_axis(typename VT<T>::V* __restrict__ data, int n, long long stride,
                                                  long long inner, long long outer_stride, int ntile,
                                                  long long Nk, int L, Sched sc,
                                                  const typename VT<T>::V* __restrict__ tw, const int* gate) {
  using V = typename VT<T>::V;
  if (gate && *gate == 0) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int ld = n + 1;
  V* a = reinterpret_cast<V*>(smraw);
  V* b = a + L * ld;
  const int c = blockIdx.y;
  const long long o = blockIdx.x / ntile;
  const long long q0 = (long long)(blockIdx.x % ntile) * L;
  V* base = data + (long long)c * Nk + o * outer_stride;
  for (int idx = threadIdx.x; idx < n * L; idx += blockDim.x) {
    const int p = idx / L, l = idx - p * L;
    const long long q = q0 + l;
    a[l * ld + p] = q < inner ? base[p * stride + q] : V{0, 0};
  }
  __syncthreads();
  V* res = fft_lines<V, S>(a, b, L, ld, sc, tw);
  for (int idx = threadIdx.x; idx < n * L; idx += blockDim.x) {
    const int p = idx / L, l = idx - p * L;
    const long long q = q0 + l;
    if (q < inner) base[p * stride + q] = res[l * ld + p];
  }
}

// ------------------------------------------------------------- Green's pass
struct GreenArgs {
  int nc, is3d, n0, n1, n2, nh;
  int disp;  // write the displacement spectrum (components 0 .. dim-1) instead of the stress
  double lambda, mu;
  double Ntot;
  // the same constants as FP32 pairs (hi, lo) for the pair transforms:
  // lambda, mu, alpha = (lambda + mu) / (lambda + 2 mu), 1/n0, 1/n1, 1/n2
  float pr[6][2];
};

// A constant of GreenArgs in the transform's arithmetic: the double, or its
// pair made on the host.
template <typename T> __device__ __forceinline__ T green_const(double d, const float* pr) { return (T)d; }
template <> __device__ __forceinline__ dfl green_const<dfl>(double d, const float* pr) { return dfl(pr[0], pr[1]); }

// stress = C:(e), Voigt with tensor shear; nc = 3 (xx yy xy) or 6 (xx yy zz yz xz xy)
template <typename T, typename V>
__device__ __forceinline__ void apply_C(int nc, T lam, T mu, const V* e, V* out) {
  const int nd = nc == 3 ? 2 : 3;
  V tr = V{0, 0};
  for (int c = 0; c < nd; c++) tr = vadd(tr, e[c]);
  for (int c = 0; c < nc; c++) {
    V v = V{(T)2 * mu * e[c].x, (T)2 * mu * e[c].y};
    if (c < nd) v = V{v.x + lam * tr.x, v.y + lam * tr.y};
    out[c] = v;
  }
}

// sigma_hat = C:(Gamma(g):C:e - e) for one unit wave vector g (x, y, z);
// h = 1/(2 mu), am = -alpha/mu with alpha = (lambda + mu)/(lambda + 2 mu)
template <typename T, typename V>
__device__ __forceinline__ void green_op(int nc, T lam, T mu, T h, T am, const T* g, const V* e, V* sig) {
  V tau[6];
  apply_C<T, V>(nc, lam, mu, e, tau);
  // tensor form of tau
  V t[3][3];
  if (nc == 3) {
    t[0][0] = tau[0]; t[1][1] = tau[1]; t[0][1] = t[1][0] = tau[2];
    t[2][2] = t[0][2] = t[2][0] = t[1][2] = t[2][1] = V{0, 0};
  } else {
    t[0][0] = tau[0]; t[1][1] = tau[1]; t[2][2] = tau[2];
    t[1][2] = t[2][1] = tau[3];
    t[0][2] = t[2][0] = tau[4];
    t[0][1] = t[1][0] = tau[5];
  }
  V F[3];
  for (int a = 0; a < 3; a++) {
    F[a] = V{t[a][0].x * g[0] + t[a][1].x * g[1] + t[a][2].x * g[2],
             t[a][0].y * g[0] + t[a][1].y * g[1] + t[a][2].y * g[2]};
  }
  V G = V{g[0] * F[0].x + g[1] * F[1].x + g[2] * F[2].x, g[0] * F[0].y + g[1] * F[1].y + g[2] * F[2].y};
  const int ia3[6] = {0, 1, 2, 1, 0, 0}, ib3[6] = {0, 1, 2, 2, 2, 1};
  const int ia2[3] = {0, 1, 0}, ib2[3] = {0, 1, 1};
  V d[6];
  for (int c = 0; c < nc; c++) {
    const int a = nc == 3 ? ia2[c] : ia3[c];
    const int b = nc == 3 ? ib2[c] : ib3[c];
    const T gg = g[a] * g[b];
    V ep = V{h * (F[a].x * g[b] + F[b].x * g[a]) + am * (G.x * gg),
             h * (F[a].y * g[b] + F[b].y * g[a]) + am * (G.y * gg)};
    d[c] = vsub(ep, e[c]);
  }
  apply_C<T, V>(nc, lam, mu, d, sig);
}

// Displacement of the same solution, u_hat = -i (F - alpha G g) / (mu |k|) for
// each axis a < dim (HomogeneousStressSolver with uflag 2, elastic.c:873-900:
// HadamardSumnSProd then HadamardSiDivd with g2 = |k|; DispField, io.c:187-205,
// is the same formula); F and G as in green_op, inv_k = 1/|k|.
template <typename T, typename V>
__device__ __forceinline__ void disp_op(int nc, T lam, T mu, T alpha, const T* g, T inv_k, const V* e, V* u) {
  V tau[6];
  apply_C<T, V>(nc, lam, mu, e, tau);
  V t[3][3];
  if (nc == 3) {
    t[0][0] = tau[0]; t[1][1] = tau[1]; t[0][1] = t[1][0] = tau[2];
    t[2][2] = t[0][2] = t[2][0] = t[1][2] = t[2][1] = V{0, 0};
  } else {
    t[0][0] = tau[0]; t[1][1] = tau[1]; t[2][2] = tau[2];
    t[1][2] = t[2][1] = tau[3];
    t[0][2] = t[2][0] = tau[4];
    t[0][1] = t[1][0] = tau[5];
  }
  V F[3];
  for (int a = 0; a < 3; a++) {
    F[a] = V{t[a][0].x * g[0] + t[a][1].x * g[1] + t[a][2].x * g[2],
             t[a][0].y * g[0] + t[a][1].y * g[1] + t[a][2].y * g[2]};
  }
  V G = V{g[0] * F[0].x + g[1] * F[1].x + g[2] * F[2].x, g[0] * F[0].y + g[1] * F[1].y + g[2] * F[2].y};
  const T s = inv_k / mu;
  const int dim = nc == 3 ? 2 : 3;
  for (int a = 0; a < dim; a++) {
    const V w = V{F[a].x - alpha * G.x * g[a], F[a].y - alpha * G.y * g[a]};
    u[a] = V{s * w.y, -s * w.x};
  }
}

__device__ __forceinline__ double wrapf(int k, int n) {
  double s = (double)k * (1.0 / n);
  return s - round(s);
}

// Unit wave vector g (axis order 2, 1, 0) of the wave numbers (k0, k1, k2):
// f_a = wrapf(k_a, n_a), g = f / |f|, in FP64 for FP64 transforms.
template <typename T>
__device__ __forceinline__ void unit_wave(int k0, int k1, int k2, const GreenArgs& ga, T* g) {
  const double f2 = wrapf(k2, ga.n2), f1 = wrapf(k1, ga.n1), f0 = ga.is3d ? wrapf(k0, ga.n0) : 0.0;
  const double gn = sqrt(f2 * f2 + f1 * f1 + f0 * f0);
  g[0] = (T)(f2 / gn);
  g[1] = (T)(f1 / gn);
  g[2] = (T)(f0 / gn);
}
// For pair transforms without FP64 instructions: the wrapped wave number w
// (the Nyquist number maps to -n/2, as in wrapf) times the pair 1/n, then
// 1/|f| by Newton's iteration for the reciprocal square root,
// y <- y + y (1 - F y^2) / 2, two steps in pairs from the FP32 estimate
// (relative error near the pairs' 2^-47).
__device__ __forceinline__ dfl wrap_pair(int k, int n, const float* inv) {
  const int w = 2 * k < n ? k : k - n;
  return dfl((float)w, 0.f) * dfl(inv[0], inv[1]);
}
template <>
__device__ __forceinline__ void unit_wave<dfl>(int k0, int k1, int k2, const GreenArgs& ga, dfl* g) {
  const dfl f2 = wrap_pair(k2, ga.n2, ga.pr[5]), f1 = wrap_pair(k1, ga.n1, ga.pr[4]);
  const dfl f0 = ga.is3d ? wrap_pair(k0, ga.n0, ga.pr[3]) : dfl(0.f, 0.f);
  const dfl F = f2 * f2 + f1 * f1 + f0 * f0;
  dfl y(rsqrtf(F.hi), 0.f);
#pragma unroll
  for (int it = 0; it < 2; it++) {
    const dfl e = dfl(1.f, 0.f) - F * (y * y);
    y = y + y * e * dfl(0.5f, 0.f);
  }
  g[0] = f2 * y;
  g[1] = f1 * y;
  g[2] = f0 * y;
}

template <typename T>
__global__ void __launch_bounds__(256) k_green(typename VT<T>::V* __restrict__ spec, int n, long long stride,
                                               long long inner, long long Nk, int L, Sched sc,
                                               const typename VT<T>::V* __restrict__ tw, GreenArgs ga,
                                               const double* __restrict__ ebar, const int* gate) {
  using V = typename VT<T>::V;
  if (gate && *gate == 0) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int nc = ga.nc;
  const int ld = n + 1;
  V* a = reinterpret_cast<V*>(smraw);
  V* b = a + nc * L * ld;
  const long long q0 = (long long)blockIdx.x * L;
  for (int idx = threadIdx.x; idx < nc * n * L; idx += blockDim.x) {
    const int c = idx / (n * L);
    const int rem = idx - c * n * L;
    const int p = rem / L, l = rem - p * L;
    const long long q = q0 + l;
    a[(c * L + l) * ld + p] = q < inner ? spec[c * Nk + p * stride + q] : V{0, 0};
  }
  __syncthreads();
  V* res = fft_lines<V, -1>(a, b, nc * L, ld, sc, tw);
  const T lam = green_const<T>(ga.lambda, ga.pr[0]), mu = green_const<T>(ga.mu, ga.pr[1]);
  const T alpha = green_const<T>((ga.lambda + ga.mu) / (ga.lambda + 2.0 * ga.mu), ga.pr[2]);
  const T hm = (T)0.5 / mu, am = -alpha / mu;
  for (int idx = threadIdx.x; idx < n * L; idx += blockDim.x) {
    const int p = idx / L, l = idx - p * L;
    const long long q = q0 + l;
    if (q >= inner) continue;
    int k0, k1, k2;
    if (ga.is3d) {
      k0 = p;
      k1 = (int)(q / ga.nh);
      k2 = (int)(q - (long long)k1 * ga.nh);
    } else {
      k0 = 0;
      k1 = p;
      k2 = (int)q;
    }
    V e[6], sig[6];
    for (int c = 0; c < nc; c++) e[c] = res[(c * L + l) * ld + p];
    if (ga.disp) {
      // displacement components 0 .. dim-1; zero at k = 0
      for (int c = 0; c < nc; c++) sig[c] = V{0, 0};
      if (k0 != 0 || k1 != 0 || k2 != 0) {
        const double f2 = wrapf(k2, ga.n2), f1 = wrapf(k1, ga.n1), f0 = ga.is3d ? wrapf(k0, ga.n0) : 0.0;
        const double gn = sqrt(f2 * f2 + f1 * f1 + f0 * f0);
        T g[3] = {(T)(f2 / gn), (T)(f1 / gn), (T)(f0 / gn)};
        const T inv_k = (T)(1.0 / (6.28318530717958647692 * gn));
        const bool ny2 = (ga.n2 % 2 == 0) && (2 * k2 == ga.n2);
        const bool ny1 = (ga.n1 % 2 == 0) && (2 * k1 == ga.n1);
        const bool ny0 = ga.is3d && (ga.n0 % 2 == 0) && (2 * k0 == ga.n0);
        // the Hermitian part of the reference's operator: the average over
        // the sign choices of the Nyquist components, as for the stress
        int nv = 0;
        for (int sg = 0; sg < 8; sg++) {
          if (((sg & 1) && !ny2) || ((sg & 2) && !ny1) || ((sg & 4) && !ny0)) continue;
          if (nc == 3 && sg != 0 && sg != ((ny2 ? 1 : 0) | (ny1 ? 2 : 0))) continue;  // 2D: all flipped together
          T gm[3] = {(sg & 1) ? -g[0] : g[0], (sg & 2) ? -g[1] : g[1], (sg & 4) ? -g[2] : g[2]};
          V u2[3];
          disp_op<T, V>(nc, lam, mu, alpha, gm, inv_k, e, u2);
          for (int c = 0; c < (nc == 3 ? 2 : 3); c++) sig[c] = vadd(sig[c], u2[c]);
          nv++;
        }
        const T inv = (T)1 / (T)nv;
        for (int c = 0; c < nc; c++) sig[c] = V{sig[c].x * inv, sig[c].y * inv};
      }
    } else if (k0 == 0 && k1 == 0 && k2 == 0) {
      V d[6];
      for (int c = 0; c < nc; c++) {
        const T eb = ebar ? (T)(ga.Ntot * ebar[c]) : (T)0;
        d[c] = V{eb - e[c].x, -e[c].y};
      }
      apply_C<T, V>(nc, lam, mu, d, sig);
    } else {
      T g[3];
      unit_wave<T>(k0, k1, k2, ga, g);
      const bool ny2 = (ga.n2 % 2 == 0) && (2 * k2 == ga.n2);
      const bool ny1 = (ga.n1 % 2 == 0) && (2 * k1 == ga.n1);
      const bool ny0 = ga.is3d && (ga.n0 % 2 == 0) && (2 * k0 == ga.n0);
      green_op<T, V>(nc, lam, mu, hm, am, g, e, sig);
      if (ny2 || ny1 || ny0) {
        if (nc == 3) {
          // 2D: the reference's real part of a complex transform, i.e. the
          // average of the operators at k and -k
          T gm[3] = {ny2 ? -g[0] : g[0], ny1 ? -g[1] : g[1], ny0 ? -g[2] : g[2]};
          V s2[6];
          green_op<T, V>(nc, lam, mu, hm, am, gm, e, s2);
          for (int c = 0; c < nc; c++) sig[c] = V{(T)0.5 * (sig[c].x + s2[c].x), (T)0.5 * (sig[c].y + s2[c].y)};
        } else {
          // 3D: average over every sign choice of the Nyquist components,
          // which keeps the discrete Green's function symmetric under the
          // reflection of each axis
          int nv = 1;
          for (int sg = 1; sg < 8; sg++) {
            if (((sg & 1) && !ny2) || ((sg & 2) && !ny1) || ((sg & 4) && !ny0)) continue;
            T gm[3] = {(sg & 1) ? -g[0] : g[0], (sg & 2) ? -g[1] : g[1], (sg & 4) ? -g[2] : g[2]};
            V s2[6];
            green_op<T, V>(nc, lam, mu, hm, am, gm, e, s2);
            for (int c = 0; c < nc; c++) sig[c] = vadd(sig[c], s2[c]);
            nv++;
          }
          const T inv = (T)1 / (T)nv;
          for (int c = 0; c < nc; c++) sig[c] = V{sig[c].x * inv, sig[c].y * inv};
        }
      }
    }
    for (int c = 0; c < nc; c++) res[(c * L + l) * ld + p] = sig[c];
  }
  __syncthreads();
  V* other = (res == a) ? b : a;
  V* res2 = fft_lines<V, +1>(res, other, nc * L, ld, sc, tw);
  for (int idx = threadIdx.x; idx < nc * n * L; idx += blockDim.x) {
    const int c = idx / (n * L);
    const int rem = idx - c * n * L;
    const int p = rem / L, l = rem - p * L;
    const long long q = q0 + l;
    if (q < inner) spec[c * Nk + p * stride + q] = res2[(c * L + l) * ld + p];
  }
}

// ---------------------------------------------------------------- C2R, axis 2
// Deviatoric coordinates of a Voigt stress (tensor shear) in the orthonormal
// basis (xx-yy)/sqrt2, (2zz-xx-yy)/sqrt6, sqrt2*yz, sqrt2*xz, sqrt2*xy, in the
// transform's arithmetic.
template <typename T>
__device__ __forceinline__ void dev_coords(const T* s, T* d) {
  const T r2 = (T)0.70710678118654752440, r6 = (T)0.40824829046386301637, s2 = (T)1.41421356237309504880;
  d[0] = (s[0] - s[1]) * r2;
  d[1] = ((T)2.0 * s[2] - s[0] - s[1]) * r6;
  d[2] = s2 * s[3];
  d[3] = s2 * s[4];
  d[4] = s2 * s[5];
}
// The nearest float of a value, a float as a value, and the accumulator of the
// error norms of the deviatoric epilogue: FP64 for FP64 transforms; FP32 per
// thread for pairs (norms of a difference of order 1e-6 of the field; the
// block totals are added in FP64).
__device__ __forceinline__ float to_f32(double x) { return (float)x; }
__device__ __forceinline__ float to_f32(float x) { return x; }
__device__ __forceinline__ float to_f32(dfl x) { return __fadd_rn(x.hi, x.lo); }
template <typename T> __device__ __forceinline__ T from_f32(float v) { return (T)v; }
template <> __device__ __forceinline__ dfl from_f32<dfl>(float v) { return dfl(v, 0.f); }
template <typename T> struct ErrAcc { using A = float; };
template <> struct ErrAcc<double> { using A = double; };
__device__ __forceinline__ double acc_of(double x) { return x; }
__device__ __forceinline__ double amax(double a, double b) { return fmax(a, b); }
__device__ __forceinline__ float amax(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ float acc_of(float x) { return x; }
__device__ __forceinline__ float acc_of(dfl x) { return to_f32(x); }

template <typename T, int OUT>
__global__ void __launch_bounds__(256) k_c2r_x(const typename VT<T>::V* __restrict__ in, int nc, int n2, int h,
                                               int nh, long long rows, long long N, long long Nk, int L, Sched sh,
                                               const typename VT<T>::V* __restrict__ tw_h,
                                               const typename VT<T>::V* __restrict__ tw_p, double invN,
                                               double* __restrict__ sig64, float* __restrict__ sig32,
                                               float* __restrict__ sdev, const double* __restrict__ uadd,
                                               double* __restrict__ err, double* __restrict__ msum,
                                               const int* gate) {
  using V = typename VT<T>::V;
  if (gate && *gate == 0) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int ld = h + 2;
  V* a = reinterpret_cast<V*>(smraw);
  V* b = a + L * ld;
  T* o = reinterpret_cast<T*>(b + L * ld);  // [nc][L][n2] for the deviatoric epilogue
  const long long r0 = (long long)blockIdx.x * L;
  const T invNT = OUT == kOutDev32 ? (T)invN : (T)0;
  __shared__ double msred[8];
  for (int c = 0; c < nc; c++) {
    double part = 0;
    const V* src = in + (long long)c * Nk;
    for (int idx = threadIdx.x; idx < L * nh; idx += blockDim.x) {
      const int l = idx / nh, k = idx - l * nh;
      const long long r = r0 + l;
      a[l * ld + k] = r < rows ? src[r * nh + k] : V{0, 0};
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < L * h; idx += blockDim.x) {
      const int l = idx / h, k = idx - l * h;
      V xk = a[l * ld + k];
      V xc = a[l * ld + (h - k)];
      xc.y = -xc.y;
      V e = vadd(xk, xc), d = vsub(xk, xc);
      V w = tw_p[k];
      w.y = -w.y;
      V od = vmul(w, d);
      // Z = E + i O
      b[l * ld + k] = V{e.x - od.y, e.y + od.x};
    }
    __syncthreads();
    V* res = fft_lines<V, +1>(b, a, L, ld, sh, tw_h);
    for (int idx = threadIdx.x; idx < L * h; idx += blockDim.x) {
      const int l = idx / h, j = idx - l * h;
      const long long r = r0 + l;
      if (r >= rows) continue;
      V z = res[l * ld + j];
      const double x0 = (double)z.x * invN, x1 = (double)z.y * invN;
      if (OUT == kOutSig64) {
        reinterpret_cast<double2*>(sig64 + (long long)c * N)[(r * n2) / 2 + j] = make_double2(x0, x1);
        part += x0 + x1;
      } else if (OUT == kOutSig32) {
        reinterpret_cast<float2*>(sig32 + (long long)c * N)[(r * n2) / 2 + j] = make_float2((float)x0, (float)x1);
      } else {
        o[(c * L + l) * n2 + 2 * j] = z.x * invNT;
        o[(c * L + l) * n2 + 2 * j + 1] = z.y * invNT;
      }
    }
    if (OUT == kOutSig64 && msum) {
      // deterministic block sum of this component (mean stress, AvgStress)
      for (int off = 16; off > 0; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
      if ((threadIdx.x & 31) == 0) msred[threadIdx.x >> 5] = part;
      __syncthreads();
      if (threadIdx.x == 0) {
        double t = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) t += msred[k];
        msum[(long long)c * gridDim.x + blockIdx.x] = t;
      }
    }
    __syncthreads();
  }
  if (OUT == kOutDev32) {
    using A = typename ErrAcc<T>::A;
    T ua[6];
    for (int c = 0; c < 6; c++) ua[c] = uadd ? (T)uadd[c] : (T)0.0;
    A mxa = 0, ssa = 0, sra = 0, mra = 0;
    for (int idx = threadIdx.x; idx < L * n2; idx += blockDim.x) {
      const int l = idx / n2, i = idx - l * n2;
      const long long r = r0 + l;
      if (r >= rows) continue;
      const long long s = r * n2 + i;
      T sv[6], d[5];
      for (int c = 0; c < 6; c++) sv[c] = o[(c * L + l) * n2 + i] + ua[c];
      dev_coords<T>(sv, d);
      A e2 = 0, n2s = 0;
      for (int k = 0; k < 5; k++) {
        const float old = sdev[k * N + s];
        const A dd = acc_of(from_f32<T>(old) - d[k]);
        const A dk = acc_of(d[k]);
        e2 += dd * dd;
        n2s += dk * dk;
        sdev[k * N + s] = to_f32(d[k]);
      }
      mxa = mxa > e2 ? mxa : e2;
      mra = mra > n2s ? mra : n2s;
      ssa += e2;
      sra += n2s;
    }
    double mx = (double)mxa, ss = (double)ssa, sr = (double)sra, mr = (double)mra;
    // block reduction
    for (int off = 16; off > 0; off >>= 1) {
      mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      mr = fmax(mr, __shfl_xor_sync(0xffffffffu, mr, off));
      ss += __shfl_xor_sync(0xffffffffu, ss, off);
      sr += __shfl_xor_sync(0xffffffffu, sr, off);
    }
    __shared__ double red[4][8];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) { red[0][w] = mx; red[1][w] = ss; red[2][w] = sr; red[3][w] = mr; }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int k = 1; k < (int)(blockDim.x >> 5); k++) {
        mx = fmax(mx, red[0][k]);
        ss += red[1][k];
        sr += red[2][k];
        mr = fmax(mr, red[3][k]);
      }
      // non-negative doubles order like their bit patterns
      atomicMax(reinterpret_cast<unsigned long long*>(&err[0]), (unsigned long long)__double_as_longlong(mx));
      atomicAdd(&err[1], ss);
      atomicAdd(&err[2], sr);
      atomicMax(reinterpret_cast<unsigned long long*>(&err[3]), (unsigned long long)__double_as_longlong(mr));
    }
  }
}

// C2R of all six components of L rows in one batch of 6 L lines (the block's
// threads busy in every stage), then the deviatoric epilogue read straight
// from the transform's buffer (its complex entry j of a row holds the reals
// 2j and 2j + 1): the stored FP32 coordinates are replaced and the error
// norms of the old ones accumulated (kOutDev32 of k_c2r_x).
template <typename T>
__global__ void __launch_bounds__(256) k_c2r_dev(const typename VT<T>::V* __restrict__ in, int n2, int h, int nh,
                                                 long long rows, long long N, long long Nk, int L, Sched sh,
                                                 const typename VT<T>::V* __restrict__ tw_h,
                                                 const typename VT<T>::V* __restrict__ tw_p, double invN,
                                                 float* __restrict__ sdev, const double* __restrict__ uadd,
                                                 double* __restrict__ err, const int* gate,
                                                 const double* __restrict__ ebar, double lambda, double mu) {
  using V = typename VT<T>::V;
  if (gate && *gate == 0) return;
  constexpr int NC = 6;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int ld = h + 2;
  V* a = reinterpret_cast<V*>(smraw);
  V* b = a + NC * L * ld;
  const long long r0 = (long long)blockIdx.x * L;
  // the old FP32 coordinates of this thread's sites (the epilogue's only
  // global reads; beyond L2 at large grids), loaded now so that the transform
  // hides their latency; threads with more than kPre sites read the rest late
  constexpr int kPre = 4;
  float pre[kPre][5];
#pragma unroll
  for (int q = 0; q < kPre; q++) {
    const int idx = threadIdx.x + q * blockDim.x;
    const int l = idx / n2, i = idx - l * n2;
    const long long r = r0 + l;
    const bool ok = idx < L * n2 && r < rows;
#pragma unroll
    for (int k = 0; k < 5; k++) pre[q][k] = ok ? sdev[k * N + r * n2 + i] : 0.f;
  }
  for (int idx = threadIdx.x; idx < NC * L * nh; idx += blockDim.x) {
    const int c = idx / (L * nh), rem = idx - c * L * nh;
    const int l = rem / nh, k = rem - l * nh;
    const long long r = r0 + l;
    a[(c * L + l) * ld + k] = r < rows ? in[(long long)c * Nk + r * nh + k] : V{0, 0};
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < NC * L * h; idx += blockDim.x) {
    const int line = idx / h, k = idx - line * h;
    V xk = a[line * ld + k];
    V xc = a[line * ld + (h - k)];
    xc.y = -xc.y;
    V e = vadd(xk, xc), d = vsub(xk, xc);
    V w = tw_p[k];
    w.y = -w.y;
    V od = vmul(w, d);
    b[line * ld + k] = V{e.x - od.y, e.y + od.x};  // Z = E + i O
  }
  __syncthreads();
  const V* res = fft_lines<V, +1>(b, a, NC * L, ld, sh, tw_h);
  const T invNT = from_f64<T>(invN);
  using A = typename ErrAcc<T>::A;
  T ua[NC];
  for (int c = 0; c < NC; c++) ua[c] = uadd ? from_f64<T>(uadd[c]) : (T)0.0;
  if (ebar)
    for (int c = 0; c < NC; c++)
      ua[c] = ua[c] + from_f64<T>((c < 3 ? lambda * (ebar[0] + ebar[1] + ebar[2]) : 0.0) + 2.0 * mu * ebar[c]);
  A mxa = 0, ssa = 0, sra = 0, mra = 0;
  for (int idx = threadIdx.x, q = 0; idx < L * n2; idx += blockDim.x, q++) {
    const int l = idx / n2, i = idx - l * n2;
    const long long r = r0 + l;
    if (r >= rows) continue;
    const long long s = r * n2 + i;
    T sv[NC], d[5];
    for (int c = 0; c < NC; c++) {
      const V z = res[(c * L + l) * ld + (i >> 1)];
      sv[c] = ((i & 1) ? z.y : z.x) * invNT + ua[c];
    }
    dev_coords<T>(sv, d);
    A e2 = 0, n2s = 0;
#pragma unroll
    for (int k = 0; k < 5; k++) {
      float old = 0.f;
#pragma unroll
      for (int qq = 0; qq < kPre; qq++)
        if (qq == q) old = pre[qq][k];
      if (q >= kPre) old = sdev[k * N + s];
      const A dd = acc_of(from_f32<T>(old) - d[k]);
      const A dk = acc_of(d[k]);
      e2 += dd * dd;
      n2s += dk * dk;
      sdev[k * N + s] = to_f32(d[k]);
    }
    mxa = mxa > e2 ? mxa : e2;
    mra = mra > n2s ? mra : n2s;
    ssa += e2;
    sra += n2s;
  }
  // warp totals in the accumulator's type, block totals in FP64
  for (int off = 16; off > 0; off >>= 1) {
    mxa = amax(mxa, __shfl_xor_sync(0xffffffffu, mxa, off));
    mra = amax(mra, __shfl_xor_sync(0xffffffffu, mra, off));
    ssa += __shfl_xor_sync(0xffffffffu, ssa, off);
    sra += __shfl_xor_sync(0xffffffffu, sra, off);
  }
  double mx = (double)mxa, ss = (double)ssa, sr = (double)sra, mr = (double)mra;
  __shared__ double red[4][8];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) { red[0][w] = mx; red[1][w] = ss; red[2][w] = sr; red[3][w] = mr; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < (int)(blockDim.x >> 5); k++) {
      mx = fmax(mx, red[0][k]);
      ss += red[1][k];
      sr += red[2][k];
      mr = fmax(mr, red[3][k]);
    }
    // non-negative doubles order like their bit patterns
    atomicMax(reinterpret_cast<unsigned long long*>(&err[0]), (unsigned long long)__double_as_longlong(mx));
    atomicAdd(&err[1], ss);
    atomicAdd(&err[2], sr);
    atomicMax(reinterpret_cast<unsigned long long*>(&err[3]), (unsigned long long)__double_as_longlong(mr));
  }
}

// ------------------------------------------------------------ filter (GRF)
template <typename T>
__global__ void k_gauss_filter(typename VT<T>::V* spec, int n0, int n1, int n2, int nh, double corr, long long Nk) {
  using V = typename VT<T>::V;
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= Nk) return;
  const int k2 = (int)(i % nh);
  const int k1 = (int)((i / nh) % n1);
  const int k0 = (int)(i / ((long long)nh * n1));
  const double f0 = n0 > 1 ? wrapf(k0, n0) : 0.0, f1 = wrapf(k1, n1), f2 = wrapf(k2, n2);
  const double k2s = 4 * 3.14159265358979323846 * 3.14159265358979323846 * (f0 * f0 + f1 * f1 + f2 * f2);
  double w = exp(-0.25 * k2s * corr * corr);
  if (i == 0) w = 0;
  V v = spec[i];
  spec[i] = V{(T)(v.x * w), (T)(v.y * w)};
}

// ------------------------------------------------------------------- host
Sched make_sched(int n) {
  Sched s;
  s.n = n;
  int m = n;
  while (m % 8 == 0 && m > 8) { s.r[s.nst++] = 8; m /= 8; }
  if (m == 8) { s.r[s.nst++] = 8; m = 1; }
  while (m % 4 == 0) { s.r[s.nst++] = 4; m /= 4; }
  while (m % 2 == 0) { s.r[s.nst++] = 2; m /= 2; }
  while (m % 3 == 0) { s.r[s.nst++] = 3; m /= 3; }
  if (m != 1) s.nst = -1;
  return s;
}

// Alternative orders of the same factors: radix 4 first (more, simpler
// stages), and the default's stages reversed (small radices first).
Sched make_sched_r4(int n) {
  Sched s;
  s.n = n;
  int m = n;
  while (m % 4 == 0) { s.r[s.nst++] = 4; m /= 4; }
  while (m % 2 == 0) { s.r[s.nst++] = 2; m /= 2; }
  while (m % 3 == 0) { s.r[s.nst++] = 3; m /= 3; }
  if (m != 1) s.nst = -1;
  return s;
}
Sched make_sched_rev(int n) {
  Sched d = make_sched(n), s = d;
  for (int i = 0; i < d.nst; i++) s.r[i] = d.r[d.nst - 1 - i];
  return s;
}

int upload_twiddles(int n, int count, double2** d64, float2** d32, float4** dpair, FxTwiddle** dfx) {
  std::vector<double2> h(count > 0 ? count : 1);
  std::vector<float2> hf(h.size());
  std::vector<float4> hp(h.size());
  std::vector<FxTwiddle> hx(h.size());
  fx_twiddles(n, count, hx.data());
  for (int k = 0; k < count; k++) {
    double ang = -2.0 * M_PI * (double)k / (double)n;
    h[k] = make_double2(std::cos(ang), std::sin(ang));
    hf[k] = make_float2((float)h[k].x, (float)h[k].y);
    const dfl x(h[k].x), y(h[k].y);
    hp[k] = make_float4(x.hi, x.lo, y.hi, y.lo);
  }
  if (cudaMalloc(d64, sizeof(double2) * h.size()) != cudaSuccess) return STZ_ERR_NOMEM;
  if (cudaMalloc(d32, sizeof(float2) * h.size()) != cudaSuccess) return STZ_ERR_NOMEM;
  if (cudaMalloc(dpair, sizeof(float4) * h.size()) != cudaSuccess) return STZ_ERR_NOMEM;
  if (cudaMalloc(dfx, sizeof(FxTwiddle) * h.size()) != cudaSuccess) return STZ_ERR_NOMEM;
  cudaMemcpy(*dfx, hx.data(), sizeof(FxTwiddle) * h.size(), cudaMemcpyHostToDevice);
  cudaMemcpy(*d64, h.data(), sizeof(double2) * h.size(), cudaMemcpyHostToDevice);
  cudaMemcpy(*d32, hf.data(), sizeof(float2) * h.size(), cudaMemcpyHostToDevice);
  cudaMemcpy(*dpair, hp.data(), sizeof(float4) * h.size(), cudaMemcpyHostToDevice);
  return STZ_OK;
}

// The dynamic shared-memory limit is a property of each kernel, shared by
// every plan in the process: raise it once to the device's opt-in maximum
// (requests below it cost nothing) instead of per plan.
template <typename K>
void raise_smem_limit(K kernel, int optin) {
  cudaFuncAttributes fa;
  if (cudaFuncGetAttributes(&fa, kernel) != cudaSuccess) { (void)cudaGetLastError(); return; }
  int bytes = optin - (int)fa.sharedSizeBytes;
  // a refusal here is not sticky; clear it so that it is not reported as a
  // launch failure later (a launch that needs more then fails on its own)
  if (bytes > 0 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess)
    (void)cudaGetLastError();
}

template <typename T>
void set_smem_attrs_max(int optin) {
  raise_smem_limit(k_r2c_x<T>, optin);
  raise_smem_limit(k_c2c_axis<T, -1>, optin);
  raise_smem_limit(k_c2c_axis<T, +1>, optin);
  raise_smem_limit(k_green<T>, optin);
  raise_smem_limit(k_c2r_x<T, kOutSig64>, optin);
  raise_smem_limit(k_c2r_x<T, kOutSig32>, optin);
  raise_smem_limit(k_c2r_x<T, kOutDev32>, optin);
  raise_smem_limit(k_c2r_dev<T>, optin);
}

template <typename T>
void set_smem_attrs(size_t sx, size_t sy, size_t sg, size_t sc) {
  (void)sx; (void)sy; (void)sg; (void)sc;
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess || optin <= 0)
    optin = 227 * 1024;
  set_smem_attrs_max<T>(optin);
}

template <typename T>
struct Tw;
template <>
struct Tw<double> {
  static const double2* h(const FFTPlan& p) { return p.tw_h; }
  static const double2* a1(const FFTPlan& p) { return p.tw_1; }
  static const double2* a0(const FFTPlan& p) { return p.tw_0; }
  static const double2* post(const FFTPlan& p) { return p.tw_p; }
};
template <>
struct Tw<float> {
  static const float2* h(const FFTPlan& p) { return p.tw_hf; }
  static const float2* a1(const FFTPlan& p) { return p.tw_1f; }
  static const float2* a0(const FFTPlan& p) { return p.tw_0f; }
  static const float2* post(const FFTPlan& p) { return p.tw_pf; }
};
template <>
struct Tw<dfl> {
  static const df2* h(const FFTPlan& p) { return reinterpret_cast<const df2*>(p.tw_hd); }
  static const df2* a1(const FFTPlan& p) { return reinterpret_cast<const df2*>(p.tw_1d); }
  static const df2* a0(const FFTPlan& p) { return reinterpret_cast<const df2*>(p.tw_0d); }
  static const df2* post(const FFTPlan& p) { return reinterpret_cast<const df2*>(p.tw_pd); }
};

// The C2R pass of a kOutDev32 solve; factor multiplies its sums (1 / N). With
// ebar, the uniform stress C:ebar is added (a spectrum without its mean part).
template <typename T>
void c2r_dev(const FFTPlan& p, const SolveArgs& a, int L, double factor, const double* ebar, cudaStream_t st,
             int64_t* launches) {
  using V = typename VT<T>::V;
  const long long rows = (long long)p.n0 * p.n1;
  // the deviatoric epilogue stages the block's six real rows: a row tile of
  // its own, kept within 72 KB of shared memory so that several blocks share
  // an SM (the tuned tile is timed without this staging)
  auto dev_smem = [&](int l) { return 2 * (size_t)p.nc * l * (p.h + 2) * sizeof(V); };
  while (L > 1 && dev_smem(L) > 72 * 1024) L /= 2;
  k_c2r_dev<T><<<(unsigned)((rows + L - 1) / L), 256, dev_smem(L), st>>>(
      reinterpret_cast<const V*>(a.spec), p.n2, p.h, p.nh, rows, p.N, p.Nk, L, p.sh, Tw<T>::h(p), Tw<T>::post(p), factor,
      a.sdev, a.uadd, a.err, a.gate, ebar, a.lambda, a.mu);
  if (launches) *launches += 1;
}

template <typename T>
int solve_t(const FFTPlan& p, const SolveArgs& a, cudaStream_t st, int64_t* launches) {
  using V = typename VT<T>::V;
  V* spec = reinterpret_cast<V*>(a.spec);
  const long long rows = (long long)p.n0 * p.n1;
  const int TH = 256;
  // R2C along axis 2
  dim3 gx((unsigned)((rows + p.L_x - 1) / p.L_x), (unsigned)p.nc);
  k_r2c_x<T><<<gx, TH, p.smem_x, st>>>(a.eps, spec, p.n2, p.h, p.nh, rows, p.N, p.Nk, p.L_x, p.sh, Tw<T>::h(p),
                                        Tw<T>::post(p), a.gate);
  int nl = 1;
  GreenArgs ga;
  ga.nc = p.nc;
  ga.is3d = p.n0 > 1;
  ga.n0 = p.n0; ga.n1 = p.n1; ga.n2 = p.n2; ga.nh = p.nh;
  ga.lambda = a.lambda; ga.mu = a.mu;
  ga.Ntot = (double)p.N;
  ga.disp = a.disp;
  {
    const double cst[6] = {a.lambda, a.mu, (a.lambda + a.mu) / (a.lambda + 2.0 * a.mu), 1.0 / p.n0, 1.0 / p.n1,
                           1.0 / p.n2};
    for (int i = 0; i < 6; i++) {
      ga.pr[i][0] = (float)cst[i];
      ga.pr[i][1] = (float)(cst[i] - (double)ga.pr[i][0]);
    }
  }
  // components left for the inverse passes: the displacement has one per axis
  const int nco = a.disp ? (p.n0 > 1 ? 3 : 2) : p.nc;
  if (p.n0 > 1) {
    // axis 1, forward
    const long long inner = p.nh;
    const int ntile = (int)((inner + p.L_y - 1) / p.L_y);
    dim3 gy((unsigned)(ntile * p.n0), (unsigned)p.nc);
    k_c2c_axis<T, -1><<<gy, TH, p.smem_y, st>>>(spec, p.n1, p.nh, inner, (long long)p.n1 * p.nh, ntile, p.Nk,
                                                  p.L_y, p.s1, Tw<T>::a1(p), a.gate);
    // axis 0 with Green
    const long long inner0 = (long long)p.n1 * p.nh;
    dim3 gg((unsigned)((inner0 + p.L_g - 1) / p.L_g));
    k_green<T><<<gg, TH, p.smem_g, st>>>(spec, p.n0, inner0, inner0, p.Nk, p.L_g, p.s0, Tw<T>::a0(p), ga, a.ebar,
                                          a.gate);
    // axis 1, inverse
    k_c2c_axis<T, +1><<<dim3(gy.x, (unsigned)nco), TH, p.smem_y, st>>>(spec, p.n1, p.nh, inner,
                                                                         (long long)p.n1 * p.nh, ntile, p.Nk, p.L_y,
                                                                         p.s1, Tw<T>::a1(p), a.gate);
    nl += 3;
  } else {
    const long long inner = p.nh;
    dim3 gg((unsigned)((inner + p.L_g - 1) / p.L_g));
    k_green<T><<<gg, TH, p.smem_g, st>>>(spec, p.n1, p.nh, inner, p.Nk, p.L_g, p.s1, Tw<T>::a1(p), ga, a.ebar,
                                          a.gate);
    nl += 1;
  }
  const double invN = 1.0 / (double)p.N;
  const size_t sc = p.smem_c2r;
  if (a.out == kOutSig64)
    k_c2r_x<T, kOutSig64><<<gx.x, TH, sc, st>>>(spec, nco, p.n2, p.h, p.nh, rows, p.N, p.Nk, p.L_x, p.sh,
                                               Tw<T>::h(p), Tw<T>::post(p), invN, a.sig64, nullptr, nullptr,
                                               nullptr, nullptr, a.msum, a.gate);
  else if (a.out == kOutSig32)
    k_c2r_x<T, kOutSig32><<<gx.x, TH, sc, st>>>(spec, p.nc, p.n2, p.h, p.nh, rows, p.N, p.Nk, p.L_x, p.sh,
                                               Tw<T>::h(p), Tw<T>::post(p), invN, nullptr, a.sig32, nullptr,
                                               nullptr, nullptr, nullptr, a.gate);
  else if (p.nc == 6)
    c2r_dev<T>(p, a, p.L_x, invN, nullptr, st, nullptr);
  else
    k_c2r_x<T, kOutDev32><<<gx.x, TH, p.smem_c2r + sizeof(double) * (size_t)p.nc * p.L_x * p.n2, st>>>(
        spec, p.nc, p.n2, p.h, p.nh, rows, p.N, p.Nk, p.L_x, p.sh, Tw<T>::h(p), Tw<T>::post(p), invN, nullptr,
        nullptr, a.sdev, a.uadd, a.err, nullptr, a.gate);
  nl += 1;
  if (launches) *launches += nl;
  return STZ_OK;
}

}  // namespace

// Tiles (lines per block) of the three kinds of floating-point pass and their
// shared memory in FP64 (the FP32 and pair transforms use the same tiles);
// false if a pass, or the C2R pass beside the real rows of all components,
// would not fit.
static bool plan_set_tiles(FFTPlan* p, int Lx, int Ly, int Lg, size_t limit = 200 * 1024, bool staging = true) {
  const size_t cz = sizeof(double2);
  const int ng = p->n0 > 1 ? p->n0 : p->n1;
  const size_t sx = 2 * (size_t)Lx * (p->h + 1) * cz, sc = 2 * (size_t)Lx * (p->h + 2) * cz;
  const size_t sy = 2 * (size_t)Ly * (p->n1 + 1) * cz, sg = 2 * (size_t)p->nc * Lg * (ng + 1) * cz;
  if (Lx < 1 || Ly < 1 || Lg < 1) return false;
  if (sc + (staging ? sizeof(double) * p->nc * Lx * p->n2 : 0) > limit || sy > limit || sg > limit) return false;
  p->L_x = Lx;
  p->L_y = Ly;
  p->L_g = Lg;
  p->smem_x = sx;
  p->smem_c2r = sc;
  p->smem_y = sy;
  p->smem_g = sg;
  return true;
}

// The same of the fixed-point passes (padded lines; a thread holds at most eight
// values of a column). Row tiles of more than 9600 values of all components are
// left out: the descent takes twice the default rows with four values a thread
// and then misses the better small tiles with eight (128^3 815 us, 797 without
// them; 64x128x256 785 and 758).
static bool plan_set_fx_tiles(FFTPlan* p, int Lx, int Ly, int Lg, size_t limit = 200 * 1024) {
  const size_t cz = sizeof(double2);
  const int ng = p->n0 > 1 ? p->n0 : p->n1;
  const size_t rx = 2 * (size_t)Lx * fx_ld(p->h + 1) * cz + sizeof(int) * Lx, ry = 2 * (size_t)Ly * fx_ld(p->n1) * cz,
               rg = 2 * (size_t)p->nc * Lg * fx_ld(ng) * cz;
  if (Lx < 1 || Ly < 1 || Lg < 1 || (Ly > 1 && Ly * p->n1 > 2048)) return false;
  if (Lx > 1 && Lx * p->h * p->nc > 9600) return false;
  if (rx > limit || ry > limit || rg > limit) return false;
  FxPasses& x = p->x;
  x.Lx = Lx;
  x.Ly = Ly;
  x.Lg = Lg;
  x.smem_x = rx;
  x.smem_y = ry;
  x.smem_g = rg;
  return true;
}

// The schedule a plan starts with: radices of make_sched, 1024 complex values of
// rows, eight lines of the other axes (four or fewer where shared memory asks
// for it).
static bool default_schedule(FFTPlan* p) {
  p->sh = p->x.sh = make_sched(p->h);
  p->s1 = p->x.s1 = make_sched(p->n1);
  p->s0 = p->x.s0 = make_sched(p->n0);
  if (p->sh.nst < 0 || p->s1.nst < 0 || p->s0.nst < 0) return false;
  const size_t cz = sizeof(double2), most = 200 * 1024;
  const int ng = p->n0 > 1 ? p->n0 : p->n1, nc = p->nc;
  int Lx = std::max(1, 1024 / p->h), Ly = 8, Lg = 8;
  while (Lx > 1 && 2 * (size_t)Lx * (p->h + 2) * cz + sizeof(double) * nc * Lx * p->n2 > most) Lx /= 2;
  while (Ly > 1 && 2 * (size_t)Ly * (p->n1 + 1) * cz > 100 * 1024) Ly /= 2;
  while (Lg > 1 && 2 * (size_t)nc * Lg * (ng + 1) * cz > most) Lg /= 2;
  // the longest lines (8192 values) leave no room for the staging, which no
  // FP64 output has
  if (!plan_set_tiles(p, Lx, Ly, Lg, 224 * 1024, false)) return false;
  p->x.ex = 4;
  p->x.ey = 4;
  p->x.eg = 2;
  Lx = std::max(1, 1024 / p->h), Ly = 8, Lg = 8;
  while (Ly > 1 && (2 * (size_t)Ly * fx_ld(p->n1) * cz > 100 * 1024 || Ly * p->n1 > 2048)) Ly /= 2;
  while (Lg > 1 && 2 * (size_t)nc * Lg * fx_ld(ng) * cz > most) Lg /= 2;
  return plan_set_fx_tiles(p, Lx, Ly, Lg, 224 * 1024);
}

// Floating-point tiles of a plan that tunes the fixed-point passes and runs the
// others for its displacement: fewer lines a block (two at least) where the grid
// would leave SMs without their two blocks. 256^2 with eight lines (17 blocks
// in Green's pass) took 296 us for a displacement, 123 with two.
static void spread_tiles(FFTPlan* p) {
  const long long rows = (long long)p->n0 * p->n1, columns = p->n0 > 1 ? (long long)p->n1 * p->nh : p->nh;
  int Lx = p->L_x, Ly = p->L_y, Lg = p->L_g;
  while (Lx > 2 && rows / Lx < 304) Lx /= 2;
  while (Ly > 2 && (long long)p->nh * p->n0 * p->nc / Ly < 304) Ly /= 2;
  while (Lg > 2 && columns / Lg < 304) Lg /= 2;
  plan_set_tiles(p, Lx, Ly, Lg, 224 * 1024, false);
}

int fft_plan_create(FFTPlan* p, int n0, int n1, int n2, int nc) {
  std::memset((void*)p, 0, sizeof(*p));
  if (n2 < 2 || n2 % 2 != 0 || n1 < 1 || n0 < 1) return STZ_ERR_INVALID;
  p->n0 = n0; p->n1 = n1; p->n2 = n2; p->nc = nc;
  p->h = n2 / 2;
  p->nh = p->h + 1;
  p->N = (long long)n0 * n1 * n2;
  p->Nk = (long long)n0 * n1 * p->nh;
  if (p->h > 4096 || n1 > 1024 || n0 > 1024 || !default_schedule(p)) return STZ_ERR_INVALID;
  int st;
  if ((st = upload_twiddles(p->h, p->h, &p->tw_h, &p->tw_hf, &p->tw_hd, &p->x.tw_h))) return st;
  if ((st = upload_twiddles(n1, n1, &p->tw_1, &p->tw_1f, &p->tw_1d, &p->x.tw_1))) return st;
  if ((st = upload_twiddles(n0, n0, &p->tw_0, &p->tw_0f, &p->tw_0d, &p->x.tw_0))) return st;
  if ((st = upload_twiddles(n2, p->nh, &p->tw_p, &p->tw_pf, &p->tw_pd, &p->x.tw_p))) return st;
  size_t sc_max = p->smem_c2r + sizeof(double) * nc * p->L_x * n2;
  set_smem_attrs<double>(p->smem_x, p->smem_y, p->smem_g, sc_max);
  set_smem_attrs<float>(p->smem_x, p->smem_y, p->smem_g, sc_max);
  set_smem_attrs<dfl>(p->smem_x, p->smem_y, p->smem_g, sc_max);
  fftx_init();
  return STZ_OK;
}

namespace {
// A tuned schedule: of the fixed-point passes, or tiles and radices of the
// floating-point ones.
struct Tuned {
  int L[3], ev[3];
  Sched sh, s1, s0;
  int rejected;  // candidates whose result differed from the default schedule's
};
bool set_tiles(FFTPlan* p, const int* L) {
  return p->kind == kPassFx ? plan_set_fx_tiles(p, L[0], L[1], L[2]) : plan_set_tiles(p, L[0], L[1], L[2]);
}
Tuned schedule_of(const FFTPlan& p) {
  const FxPasses& x = p.x;
  if (p.kind == kPassFx) return Tuned{{x.Lx, x.Ly, x.Lg}, {x.ex, x.ey, x.eg}, x.sh, x.s1, x.s0, 0};
  return Tuned{{p.L_x, p.L_y, p.L_g}, {0, 0, 0}, p.sh, p.s1, p.s0, 0};
}
// false (and the tiles of before) where other tiles do not fit
bool take_schedule(FFTPlan* p, const Tuned& t) {
  const Tuned now = schedule_of(*p);
  const bool ok = std::equal(t.L, t.L + 3, now.L) || set_tiles(p, t.L);
  if (p->kind == kPassFx) {
    p->x.ex = t.ev[0];
    p->x.ey = t.ev[1];
    p->x.eg = t.ev[2];
    p->x.sh = t.sh;
    p->x.s1 = t.s1;
    p->x.s0 = t.s0;
  } else {
    p->sh = t.sh;
    p->s1 = t.s1;
    p->s0 = t.s0;
  }
  return ok;
}
std::mutex g_tune_mu;
std::map<std::array<int, 6>, Tuned> g_tuned;

// The better of two times of three solves. On small grids they queue behind a
// kernel that holds the stream while the host launches them, so that the events
// bracket device time (without it those took four times twelve solves a
// candidate: 153 ms for the first 64^3 context of a process, 45 so).
float time_solve(const FFTPlan& p, const SolveArgs& a, cudaStream_t st, cudaEvent_t e0, cudaEvent_t e1) {
  float best = 1e30f;
  for (int rep = 0; rep < 2; rep++) {
    if (p.N * p.nc < 1 << 21) launch_hold(40000, st);
    cudaEventRecord(e0, st);
    for (int i = 0; i < 3; i++) fft_solve(p, a, st, nullptr);
    cudaEventRecord(e1, st);
    cudaEventSynchronize(e1);
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    best = std::min(best, ms);
  }
  return best;
}
}  // namespace

int fft_autotune(FFTPlan* p, cudaStream_t st, int* chosen, PassKind kind) {
  p->kind = kind;
  if (kind == kPassFx) spread_tiles(p);
  int dev = 0;
  cudaGetDevice(&dev);
  const std::array<int, 6> key = {dev, p->n0, p->n1, p->n2, p->nc, kind};
  auto take = [&](const Tuned& t) {
    take_schedule(p, t);
    const Tuned now = schedule_of(*p);
    if (chosen) {
      for (int i = 0; i < 3; i++) chosen[i] = now.L[i];
      chosen[3] = t.rejected;
    }
  };
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    auto it = g_tuned.find(key);
    if (it != g_tuned.end()) {
      take(it->second);
      return STZ_OK;
    }
  }
  const size_t n = (size_t)p->nc * p->N, nk = (size_t)p->nc * p->Nk;
  double *eps = nullptr, *ref = nullptr, *out = nullptr;
  double2* spec = nullptr;
  if (cudaMalloc(&eps, n * 8) != cudaSuccess || cudaMalloc(&ref, n * 8) != cudaSuccess ||
      cudaMalloc(&out, n * 8) != cudaSuccess || cudaMalloc(&spec, nk * sizeof(double2)) != cudaSuccess) {
    cudaFree(eps); cudaFree(ref); cudaFree(out); cudaFree(spec);
    (void)cudaGetLastError();
    return STZ_OK;  // no room to tune: keep the default schedule
  }
  // a deterministic eigenstrain with content on every wave vector
  std::vector<double> h(n);
  uint64_t x = 0x9E3779B97F4A7C15ull;
  for (size_t i = 0; i < n; i++) {
    x = x * 6364136223846793005ull + 1442695040888963407ull;
    h[i] = (double)(x >> 11) * (1.0 / 9007199254740992.0) - 0.5;
  }
  cudaMemcpyAsync(eps, h.data(), n * 8, cudaMemcpyHostToDevice, st);
  SolveArgs a{};
  a.eps = eps;
  a.lambda = kind == kPassFp64 ? 1000.0 : 2.0;  // beyond the fixed point's range, or within
  a.mu = 1.0;
  a.out = kOutSig64;
  a.sig64 = ref;
  a.spec = spec;
  a.ortho_mean = 1;
  a.pair = kind == kPassPair;
  fft_solve(*p, a, st, nullptr);
  cudaStreamSynchronize(st);
  std::vector<double> r(n), o(n);
  cudaMemcpy(r.data(), ref, n * 8, cudaMemcpyDeviceToHost);
  double refmax = 0;
  for (double v : r) refmax = std::max(refmax, std::fabs(v));
  a.sig64 = out;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  int rejected = 0;
  // a candidate is timed only if its result equals the default schedule's
  auto valid = [&](const FFTPlan& q) {
    fft_solve(q, a, st, nullptr);
    cudaMemcpyAsync(o.data(), out, n * 8, cudaMemcpyDeviceToHost, st);
    cudaStreamSynchronize(st);
    double err = 0;
    for (size_t i = 0; i < n; i++) err = std::max(err, std::fabs(o[i] - r[i]));
    const bool ok = cudaGetLastError() == cudaSuccess && err <= 1e-10 * std::max(refmax, 1e-300);
    if (!ok) rejected++;
    return ok;
  };
  FFTPlan best = *p;
  float tbest = time_solve(best, a, st, e0, e1);
  auto consider = [&](const Tuned& t) {
    FFTPlan q = best;
    if (!take_schedule(&q, t) || !valid(q)) return;
    const float ms = time_solve(q, a, st, e0, e1);
    if (ms < tbest) { tbest = ms; best = q; }
  };
  // coordinate descent over the tiles of each pass, the radix orders and, of the
  // fixed-point passes, the threads per tile
  const Tuned first = schedule_of(best);
  auto try_tile = [&](int i, int L) {
    Tuned t = schedule_of(best);
    if (L < 1 || L == t.L[i]) return;
    t.L[i] = L;
    consider(t);
  };
  for (int L : {first.L[0] * 2, first.L[0] / 2, first.L[0] / 4}) try_tile(0, L);
  for (int L : {2, 4, 16}) try_tile(1, L);
  if (p->n1 <= 64) try_tile(1, 32);
  if (kind == kPassFx) try_tile(2, 1);
  for (int L : {2, 4, 16}) try_tile(2, L);
  for (int v = 0; v < 2; v++) {
    Tuned t = schedule_of(best);
    t.sh = v ? make_sched_rev(p->h) : make_sched_r4(p->h);
    t.s1 = v ? make_sched_rev(p->n1) : make_sched_r4(p->n1);
    t.s0 = v ? make_sched_rev(p->n0) : make_sched_r4(p->n0);
    if (t.sh.nst > 0 && t.s1.nst > 0 && t.s0.nst > 0) consider(t);
  }
  if (kind == kPassFx)
    for (int i = 0; i < 3; i++)
      for (int ev : {i < 2 ? 2 : 1, i < 2 ? 8 : 4}) {
        Tuned t = schedule_of(best);
        t.ev[i] = ev;
        if (i != 1 || p->n0 > 1) consider(t);
      }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(eps); cudaFree(ref); cudaFree(out); cudaFree(spec);
  Tuned t = schedule_of(best);
  t.rejected = rejected;
  take(t);
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tuned[key] = t;
  }
  return cudaGetLastError() == cudaSuccess ? STZ_OK : STZ_ERR_CUDA;
}

// Plan whose twiddle tables live in caller-provided device storage (for the
// allocation-free entry point). FP64 solves only; no device allocation. The
// tables are those of the passes that fft_solve takes for the medium: FP64 or
// fixed point, 16 bytes a value each.
size_t fft_twiddle_count(int n0, int n1, int n2) { return (size_t)(n2 / 2) + n1 + n0 + (n2 / 2 + 1); }

int fft_plan_init_in(FFTPlan* p, int n0, int n1, int n2, int nc, double lambda, double mu, double2* storage, size_t cap,
                     cudaStream_t st) {
  std::memset((void*)p, 0, sizeof(*p));
  if (n2 < 2 || n2 % 2 != 0 || n1 < 1 || n0 < 1) return STZ_ERR_INVALID;
  p->n0 = n0; p->n1 = n1; p->n2 = n2; p->nc = nc;
  p->h = n2 / 2;
  p->nh = p->h + 1;
  p->N = (long long)n0 * n1 * n2;
  p->Nk = (long long)n0 * n1 * p->nh;
  if (p->h > 4096 || n1 > 1024 || n0 > 1024 || !default_schedule(p)) return STZ_ERR_INVALID;
  if (fft_twiddle_count(n0, n1, n2) > cap) return STZ_ERR_INVALID;
  const bool fx = fftx_fits(n2, lambda, mu);
  const int lens[4] = {p->h, n1, n0, n2};
  const int counts[4] = {p->h, n1, n0, p->nh};
  double2** dst[4] = {&p->tw_h, &p->tw_1, &p->tw_0, &p->tw_p};
  FxTwiddle** dfx[4] = {&p->x.tw_h, &p->x.tw_1, &p->x.tw_0, &p->x.tw_p};
  static_assert(sizeof(FxTwiddle) == sizeof(double2), "one table size");
  std::vector<double2> host(fft_twiddle_count(n0, n1, n2));
  size_t off = 0;
  for (int t = 0; t < 4; t++) {
    if (fx) {
      fx_twiddles(lens[t], counts[t], reinterpret_cast<FxTwiddle*>(host.data() + off));
      *dfx[t] = reinterpret_cast<FxTwiddle*>(storage + off);
    } else {
      for (int k = 0; k < counts[t]; k++) {
        const double ang = -2.0 * M_PI * (double)k / (double)lens[t];
        host[off + k] = make_double2(std::cos(ang), std::sin(ang));
      }
      *dst[t] = storage + off;
    }
    off += counts[t];
  }
  if (cudaMemcpyAsync(storage, host.data(), sizeof(double2) * host.size(), cudaMemcpyHostToDevice, st) !=
      cudaSuccess)
    return STZ_ERR_CUDA;
  if (cudaStreamSynchronize(st) != cudaSuccess) return STZ_ERR_CUDA;
  if (fx) fftx_init(p);
  else set_smem_attrs<double>(p->smem_x, p->smem_y, p->smem_g, p->smem_c2r + sizeof(double) * nc * p->L_x * n2);
  return STZ_OK;
}

int fft_c2r_blocks(const FFTPlan& p) {
  const int L = p.kind == kPassFx ? p.x.Lx : p.L_x;
  return (int)(((long long)p.n0 * p.n1 + L - 1) / L);
}

void fft_plan_destroy(FFTPlan* p) {
  cudaFree(p->tw_h); cudaFree(p->tw_1); cudaFree(p->tw_0); cudaFree(p->tw_p);
  cudaFree(p->tw_hf); cudaFree(p->tw_1f); cudaFree(p->tw_0f); cudaFree(p->tw_pf);
  cudaFree(p->tw_hd); cudaFree(p->tw_1d); cudaFree(p->tw_0d); cudaFree(p->tw_pd);
  cudaFree(p->x.tw_h); cudaFree(p->x.tw_1); cudaFree(p->x.tw_0); cudaFree(p->x.tw_p);
  std::memset((void*)p, 0, sizeof(*p));
}

int fft_solve(const FFTPlan& p, const SolveArgs& a, cudaStream_t st, int64_t* launches) {
  if (a.pair) return solve_t<dfl>(p, a, st, launches);
  // FP64 solves run in fixed point (fftx.cu), but for the displacement (a
  // print-time solve), the longest lines and media whose moduli are out of its
  // range
  if (!a.fp32 && !a.disp && (a.out == kOutSig64 || (a.out == kOutDev32 && p.nc == 6)) &&
      fftx_fits(p.n2, a.lambda, a.mu)) {
    fftx_spectrum(p, a, st, launches);
    if (a.out == kOutSig64) fftx_c2r(p, a, st, launches);
    else c2r_dev<double>(p, a, p.x.Lx, fftx_factor(p, a.mu), a.ebar, st, launches);
    return STZ_OK;
  }
  return a.fp32 ? solve_t<float>(p, a, st, launches) : solve_t<double>(p, a, st, launches);
}

// Gaussian-covariance filter of one real field in place (unit-variance
// renormalisation is done by the caller).
int fft_filter_gaussian(const FFTPlan& p, double* field, double corr_len, void* spec, cudaStream_t st) {
  using V = double2;
  V* sp = reinterpret_cast<V*>(spec);
  const long long rows = (long long)p.n0 * p.n1;
  const int TH = 256;
  dim3 gx((unsigned)((rows + p.L_x - 1) / p.L_x), 1);
  k_r2c_x<double><<<gx, TH, p.smem_x, st>>>(field, sp, p.n2, p.h, p.nh, rows, p.N, p.Nk, p.L_x, p.sh, p.tw_h,
                                             p.tw_p, nullptr);
  const long long inner1 = p.nh;
  const int ntile1 = (int)((inner1 + p.L_y - 1) / p.L_y);
  dim3 gy((unsigned)(ntile1 * p.n0), 1);
  k_c2c_axis<double, -1><<<gy, TH, p.smem_y, st>>>(sp, p.n1, p.nh, inner1, (long long)p.n1 * p.nh, ntile1, p.Nk,
                                                    p.L_y, p.s1, p.tw_1, nullptr);
  const long long inner0 = (long long)p.n1 * p.nh;
  // lines per block along axis 0: those of axis 1, fewer where n0 is the longer
  // (its lines need the shared memory; 32 of 256 values do not fit)
  int L0 = p.L_y;
  while (L0 > 1 && 2 * (size_t)L0 * (p.n0 + 1) * sizeof(V) > 200 * 1024) L0 /= 2;
  const int ntile0 = (int)((inner0 + L0 - 1) / L0);
  const size_t s0 = 2 * (size_t)L0 * (p.n0 + 1) * sizeof(V);
  if (p.n0 > 1) {
    k_c2c_axis<double, -1><<<ntile0, TH, s0, st>>>(sp, p.n0, inner0, inner0, 0, ntile0, p.Nk, L0, p.s0, p.tw_0,
                                                   nullptr);
  }
  k_gauss_filter<double><<<(unsigned)((p.Nk + 255) / 256), 256, 0, st>>>(sp, p.n0, p.n1, p.n2, p.nh, corr_len, p.Nk);
  if (p.n0 > 1)
    k_c2c_axis<double, +1><<<ntile0, TH, s0, st>>>(sp, p.n0, inner0, inner0, 0, ntile0, p.Nk, L0, p.s0, p.tw_0,
                                                   nullptr);
  k_c2c_axis<double, +1><<<gy, TH, p.smem_y, st>>>(sp, p.n1, p.nh, inner1, (long long)p.n1 * p.nh, ntile1, p.Nk,
                                                    p.L_y, p.s1, p.tw_1, nullptr);
  k_c2r_x<double, kOutSig64><<<gx.x, TH, p.smem_c2r, st>>>(sp, 1, p.n2, p.h, p.nh, rows, p.N, p.Nk, p.L_x, p.sh,
                                                          p.tw_h, p.tw_p, 1.0, field, nullptr, nullptr, nullptr,
                                                          nullptr, nullptr, nullptr);
  return cudaGetLastError() == cudaSuccess ? STZ_OK : STZ_ERR_CUDA;
}

}  // namespace stz
