// Shared device code for libdnsb: complex helpers, the shared-memory
// Stockham FFT used by every axis pass, and launch/error plumbing.
//
// FFT conventions follow the reference solver (src/dnsjax/fft.py):
// norm="forward" -- the forward transform divides by the length, the
// inverse applies no factor -- and stored spectral axes omit the Nyquist
// mode.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <type_traits>

#define DNSB_MAX_RADIX 8
#define DNSB_MAX_STAGES 12

namespace dnsb {

__host__ __device__ __forceinline__ double2 cadd(double2 a, double2 b) {
  return make_double2(a.x + b.x, a.y + b.y);
}
__host__ __device__ __forceinline__ double2 csub(double2 a, double2 b) {
  return make_double2(a.x - b.x, a.y - b.y);
}
__host__ __device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__host__ __device__ __forceinline__ double2 cscale(double2 a, double s) {
  return make_double2(a.x * s, a.y * s);
}
__host__ __device__ __forceinline__ double2 cconj(double2 a) {
  return make_double2(a.x, -a.y);
}
// i * k * z for real k, evaluated as numpy evaluates 1j * k * z:
// (0 + k i)(a + b i) = (-k b) + (k a) i.
__host__ __device__ __forceinline__ double2 cik(double k, double2 z) {
  return make_double2(-(k * z.y), k * z.x);
}
// i * z
__host__ __device__ __forceinline__ double2 ci(double2 z) {
  return make_double2(-z.y, z.x);
}

// Single-precision complex (the FP32 form of the Couette RHS passes).
__host__ __device__ __forceinline__ float2 cadd(float2 a, float2 b) {
  return make_float2(a.x + b.x, a.y + b.y);
}
__host__ __device__ __forceinline__ float2 csub(float2 a, float2 b) {
  return make_float2(a.x - b.x, a.y - b.y);
}
__host__ __device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__host__ __device__ __forceinline__ float2 cscale(float2 a, float s) {
  return make_float2(a.x * s, a.y * s);
}

// Complex type <-> real type and constructor.
template <typename C>
struct cplx;
template <>
struct cplx<double2> {
  using real = double;
  __host__ __device__ static double2 make(double x, double y) { return make_double2(x, y); }
};
template <>
struct cplx<float2> {
  using real = float;
  __host__ __device__ static float2 make(float x, float y) { return make_float2(x, y); }
};
template <typename C>
__host__ __device__ __forceinline__ C cmake(typename cplx<C>::real x, typename cplx<C>::real y) {
  return cplx<C>::make(x, y);
}
// FP32 complex whose register DFTs (dft2/3/4/8, dft_3p) carry compensated
// (two-sum) accumulation: the FP32 pass buffers and every other operation
// are those of float2 (same layout); see the compensated DFTs below.
struct __align__(8) cf2 : public float2 {
  cf2() = default;
  __host__ __device__ cf2(float2 v) : float2(v) {}
};
template <>
struct cplx<cf2> {
  using real = float;
  __host__ __device__ static cf2 make(float x, float y) { return cf2(make_float2(x, y)); }
};
// Element types of a pass kernel instantiated on T: double (FP64), float
// (FP32), fcomp (FP32 buffers, compensated butterflies).
struct fcomp {};
template <typename T>
struct pass_types {
  using C = double2;
  using R = double;
};
template <>
struct pass_types<float> {
  using C = float2;
  using R = float;
};
template <>
struct pass_types<fcomp> {
  using C = cf2;
  using R = float;
};

// Conversions between the two precisions.
__host__ __device__ __forceinline__ double2 to_c(double2 z, double2*) { return z; }
__host__ __device__ __forceinline__ float2 to_c(double2 z, float2*) {
  return make_float2((float)z.x, (float)z.y);
}
__host__ __device__ __forceinline__ double2 to_d(double2 z) { return z; }
__host__ __device__ __forceinline__ double2 to_d(float2 z) {
  return make_double2((double)z.x, (double)z.y);
}

// An FFT length L = product of radices (each 2, 3, 4 or 8), applied as
// Stockham auto-sort stages so the output is in natural order.
struct FFTPlan {
  int L;
  int nst;
  int radix[DNSB_MAX_STAGES];
};

// ---- small DFTs in registers; sign = -1 forward, +1 inverse ------------
// Generic over the value type: double2, float2, or cff (the compensated FP32
// pair below); the same operations in each.
// i * sign * v (exact)
template <typename C>
__device__ __forceinline__ C cisign(C v, int sign) {
  return cmake<C>(-sign * v.y, sign * v.x);
}
// c v for a real constant c
template <typename C>
__device__ __forceinline__ C cconst(C v, double c) {
  return cscale(v, (typename cplx<C>::real)c);
}
// (c + i s) v for a constant
template <typename C>
__device__ __forceinline__ C crot(C v, double c, double s) {
  using R = typename cplx<C>::real;
  return cmake<C>(v.x * (R)c - v.y * (R)s, v.x * (R)s + v.y * (R)c);
}

// ---- compensated FP32 values (the cf2 element type) -------------------------
// Each FP32 value is carried as h + l: a sum or difference keeps its exact
// rounding error (Knuth's two-sum) in l, a product by a constant keeps the
// product's rounding error (from an FMA) and the constant's own FP32 rounding
// error; l is folded back (h + l, one rounding) when the DFT stores its
// outputs.  Only the register DFTs are compensated; the twiddle
// multiplications between stages and the pass buffers stay FP32.
struct ffv {
  float h, l;
};
__device__ __forceinline__ ffv ff_two_sum(float a, float b) {
  const float s = a + b;
  const float bb = s - a;
  return {s, (a - (s - bb)) + (b - bb)};
}
__device__ __forceinline__ ffv ff_add(ffv a, ffv b) {
  ffv s = ff_two_sum(a.h, b.h);
  s.l += a.l + b.l;
  return s;
}
__device__ __forceinline__ ffv ff_sub(ffv a, ffv b) {
  ffv s = ff_two_sum(a.h, -b.h);
  s.l += a.l - b.l;
  return s;
}
// a (ch + cl): ch the FP32 constant, cl its rounding error
__device__ __forceinline__ ffv ff_mulc(ffv a, float ch, float cl) {
  const float p = a.h * ch;
  return {p, fmaf(a.h, ch, -p) + (a.h * cl + a.l * ch)};
}
__device__ __forceinline__ ffv ff_mulc(ffv a, double c) {
  return ff_mulc(a, (float)c, (float)(c - (double)(float)c));
}
struct cff {
  ffv x, y;
};
__device__ __forceinline__ cff cff_of(float2 v) { return {{v.x, 0.0f}, {v.y, 0.0f}}; }
__device__ __forceinline__ cf2 cff_fold(cff v) {
  return cf2(make_float2(v.x.h + v.x.l, v.y.h + v.y.l));
}
__device__ __forceinline__ cff cadd(cff a, cff b) { return {ff_add(a.x, b.x), ff_add(a.y, b.y)}; }
__device__ __forceinline__ cff csub(cff a, cff b) { return {ff_sub(a.x, b.x), ff_sub(a.y, b.y)}; }
__device__ __forceinline__ cff cisign(cff a, int sign) {
  const ffv nx = {-a.y.h, -a.y.l};
  return sign > 0 ? cff{nx, a.x} : cff{a.y, {-a.x.h, -a.x.l}};
}
__device__ __forceinline__ cff cconst(cff a, double c) {
  return {ff_mulc(a.x, c), ff_mulc(a.y, c)};
}
__device__ __forceinline__ cff crot(cff a, double c, double s) {
  return {ff_sub(ff_mulc(a.x, c), ff_mulc(a.y, s)), ff_add(ff_mulc(a.x, s), ff_mulc(a.y, c))};
}

template <typename V>
__device__ __forceinline__ void dft2(V* v) {
  const V a = v[0], b = v[1];
  v[0] = cadd(a, b);
  v[1] = csub(a, b);
}

// zero: bit i set where v[i] is known to be zero (one at most)
template <typename V>
__device__ __forceinline__ void dft3(V* v, int sign, unsigned zero = 0) {
  if (zero == 1u || zero == 2u || zero == 4u) {
    const double s3 = 0.86602540378443864676;  // sin(2 pi / 3)
    if (zero == 1u) {
      const V t1 = cadd(v[1], v[2]), t2 = cconst(t1, -0.5);
      const V t3 = cconst(cisign(csub(v[1], v[2]), sign), s3);
      v[0] = t1;
      v[1] = cadd(t2, t3);
      v[2] = csub(t2, t3);
    } else {
      const V x = zero == 2u ? v[2] : v[1];
      const V t2 = csub(v[0], cconst(x, 0.5));
      const V t3 = cconst(cisign(x, zero == 2u ? -sign : sign), s3);
      v[0] = cadd(v[0], x);
      v[1] = cadd(t2, t3);
      v[2] = csub(t2, t3);
    }
    return;
  }
  const V t1 = cadd(v[1], v[2]);
  const V t2 = csub(v[0], cconst(t1, 0.5));
  // sin(2 pi / 3)
  const V t3 = cconst(cisign(csub(v[1], v[2]), sign), 0.86602540378443864676);
  v[0] = cadd(v[0], t1);
  v[1] = cadd(t2, t3);
  v[2] = csub(t2, t3);
}

template <typename V>
__device__ __forceinline__ void dft4(V* v, int sign) {
  const V a = cadd(v[0], v[2]), b = csub(v[0], v[2]);
  const V c = cadd(v[1], v[3]), d = csub(v[1], v[3]);
  const V isd = cisign(d, sign);
  v[0] = cadd(a, c);
  v[2] = csub(a, c);
  v[1] = cadd(b, isd);
  v[3] = csub(b, isd);
}

template <typename V>
__device__ __forceinline__ void dft8(V* v, int sign) {
  const double h = 0.70710678118654752440;  // sqrt(2)/2
  V e[4] = {v[0], v[2], v[4], v[6]};
  V o[4] = {v[1], v[3], v[5], v[7]};
  dft4(e, sign);
  dft4(o, sign);
  // twiddles w8^q = exp(sign 2 pi i q / 8): (1 + sign i) h, sign i, (-1 + sign i) h
  const V t1 = cconst(cadd(o[1], cisign(o[1], sign)), h);
  const V t2 = cisign(o[2], sign);
  const V t3 = cconst(csub(cisign(o[3], sign), o[3]), h);
  v[0] = cadd(e[0], o[0]);
  v[4] = csub(e[0], o[0]);
  v[1] = cadd(e[1], t1);
  v[5] = csub(e[1], t1);
  v[2] = cadd(e[2], t2);
  v[6] = csub(e[2], t2);
  v[3] = cadd(e[3], t3);
  v[7] = csub(e[3], t3);
}

// One Stockham radix-R stage over C columns stored as buf[t * C + c].
template <int R>
__device__ __forceinline__ void fft_stage(const double2* __restrict__ in,
                                          double2* __restrict__ out, int L,
                                          int C, int Ns, int sign,
                                          const double2* __restrict__ tw) {
  const int nb = L / R;
  const int step = L / (Ns * R);
  const int total = nb * C;
  for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
    const int c = idx % C;
    const int j = idx / C;
    const int k = j % Ns;
    double2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = in[(j + r * nb) * C + c];
#pragma unroll
    for (int r = 1; r < R; ++r) {
      double2 w = tw[r * k * step];
      if (sign > 0) w.y = -w.y;
      v[r] = cmul(v[r], w);
    }
    if (R == 2) dft2(v);
    if (R == 3) dft3(v, sign);
    if (R == 4) dft4(v, sign);
    if (R == 8) dft8(v, sign);
    const int base = (j / Ns) * Ns * R + k;
#pragma unroll
    for (int r = 0; r < R; ++r) out[(base + r * Ns) * C + c] = v[r];
  }
}

// Transform C columns of length P.L held in a[t * C + c]; b is scratch of
// the same size.  tw[m] = exp(-2 pi i m / L).  Returns the buffer that
// holds the result.  Ends with __syncthreads().
__device__ inline double2* fft_columns(double2* a, double2* b,
                                       const FFTPlan& P, int C, int sign,
                                       const double2* tw) {
  int Ns = 1;
  double2* in = a;
  double2* out = b;
  for (int s = 0; s < P.nst; ++s) {
    const int R = P.radix[s];
    switch (R) {
      case 2: fft_stage<2>(in, out, P.L, C, Ns, sign, tw); break;
      case 3: fft_stage<3>(in, out, P.L, C, Ns, sign, tw); break;
      case 4: fft_stage<4>(in, out, P.L, C, Ns, sign, tw); break;
      default: fft_stage<8>(in, out, P.L, C, Ns, sign, tw); break;
    }
    __syncthreads();
    double2* t = in;
    in = out;
    out = t;
    Ns *= R;
  }
  return in;
}

// ---- compile-time plans -----------------------------------------------
// Same factorisation rule as make_plan (8s first unless the rest is 8, then
// 4s, 2s, 3s), evaluated at compile time so every stage's stride, twiddle
// step and trip count are constants.
__host__ __device__ constexpr int cplan_radix(int L, int s) {
  int n = L, k = 0;
  while (n % 8 == 0 && n != 8) { if (k == s) return 8; ++k; n /= 8; }
  while (n % 4 == 0 && n > 1) { if (k == s) return 4; ++k; n /= 4; }
  while (n % 2 == 0 && n > 1) { if (k == s) return 2; ++k; n /= 2; }
  while (n % 3 == 0 && n > 1) { if (k == s) return 3; ++k; n /= 3; }
  if (n == 8) { if (k == s) return 8; ++k; }
  return 0;
}
__host__ __device__ constexpr int cplan_nst(int L) {
  int s = 0;
  while (cplan_radix(L, s) != 0) ++s;
  return s;
}

// CT: the complex type of the columns and twiddles (double2, or float2).
template <int L, int R, int C, int NS, int SIGN, int NT, typename CT = double2>
__device__ __forceinline__ void fft_stage_t(const CT* __restrict__ in,
                                            CT* __restrict__ out,
                                            const CT* __restrict__ tw) {
  constexpr int NB = L / R;
  constexpr int STEP = L / (NS * R);
  constexpr int TOTAL = NB * C;
#pragma unroll 2
  for (int idx = threadIdx.x; idx < TOTAL; idx += NT) {
    const int c = idx % C;
    const int j = idx / C;
    const int k = j % NS;
    CT v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = in[(j + r * NB) * C + c];
    if (NS > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) {
        CT w = tw[r * k * STEP];
        if (SIGN > 0) w.y = -w.y;
        v[r] = cmul(v[r], w);
      }
    }
    if (R == 2) dft2(v);
    if (R == 3) dft3(v, SIGN);
    if (R == 4) dft4(v, SIGN);
    if (R == 8) dft8(v, SIGN);
    const int base = (j / NS) * NS * R + k;
#pragma unroll
    for (int r = 0; r < R; ++r) out[(base + r * NS) * C + c] = v[r];
  }
}

template <int L, int C, int SIGN, int NT, int S = 0, int NS = 1, typename CT = double2>
__device__ __forceinline__ CT* fft_stages_t(CT* a, CT* b, const CT* tw) {
  if constexpr (S >= cplan_nst(L)) {
    return a;
  } else {
    constexpr int R = cplan_radix(L, S);
    fft_stage_t<L, R, C, NS, SIGN, NT, CT>(a, b, tw);
    __syncthreads();
    return fft_stages_t<L, C, SIGN, NT, S + 1, NS * R, CT>(b, a, tw);
  }
}

// Compile-time-planned version of fft_columns (blockDim.x must equal NT).
template <int L, int C, int SIGN, int NT, typename CT = double2>
__device__ __forceinline__ CT* fft_columns_t(CT* a, CT* b, const CT* tw) {
  return fft_stages_t<L, C, SIGN, NT, 0, 1, CT>(a, b, tw);
}

// Dispatch: ML > 0 uses the compile-time plan for length ML, ML == 0 the
// runtime plan (FP64 only).
template <int ML, int C, int NT, typename CT = double2>
__device__ __forceinline__ CT* fft_cols(CT* a, CT* b, const FFTPlan& P, int sign,
                                        const CT* tw) {
  if constexpr (ML > 0) {
    if (sign > 0) return fft_columns_t<ML, C, 1, NT, CT>(a, b, tw);
    return fft_columns_t<ML, C, -1, NT, CT>(a, b, tw);
  } else {
    static_assert(std::is_same<CT, double2>::value, "runtime-planned FFTs are FP64");
    return fft_columns(a, b, P, C, sign, tw);
  }
}

// ---- register DFTs of composite size ---------------------------------------
// Modular inverse of a mod m (a, m coprime), by search (compile time).
__host__ __device__ constexpr int inv_mod(int a, int m) {
  int r = 1;
  while ((a * r) % m != 1) ++r;
  return r;
}

// cos(2 pi k / N) for the twiddles inside the 9-, 16- and 27-point DFTs
// (a switch, so an unrolled index folds to the literal).
template <int N>
__host__ __device__ constexpr double cos_turn(int k) {
  static_assert(27 % N == 0 || N == 16, "9, 16 and 27 points");
  k = ((k % N) + N) % N;
  k = k > N / 2 ? N - k : k;
  if (N == 16) {
    switch (k) {
      case 0: return 1.0;
      case 1: return 0.9238795325112867;
      case 2: return 0.7071067811865476;
      case 3: return 0.3826834323650898;
      case 4: return 0.0;
      case 5: return -0.3826834323650898;
      case 6: return -0.7071067811865476;
      case 7: return -0.9238795325112867;
      default: return -1.0;
    }
  }
  switch (k * (27 / N)) {
    case 0: return 1.0;
    case 1: return 0.9730448705798238;
    case 2: return 0.8936326403234123;
    case 3: return 0.766044443118978;
    case 4: return 0.5971585917027862;
    case 5: return 0.39607976603915684;
    case 6: return 0.17364817766693036;
    case 7: return -0.05814482891047583;
    case 8: return -0.28680323271109026;
    case 9: return -0.5;
    case 10: return -0.6862416378687336;
    case 11: return -0.8354878114129364;
    case 12: return -0.9396926207859084;
    default: return -0.993238357741943;
  }
}
// sin(2 pi k / N)
template <int N>
__host__ __device__ constexpr double sin_turn(int k) {
  k = ((k % N) + N) % N;
  const double sg = 2 * k > N ? -1.0 : 1.0;
  k = 2 * k > N ? N - k : k;
  if (N == 16) return sg * cos_turn<16>(k - 4);
  switch (k * (27 / N)) {
    case 0: return 0.0;
    case 1: return sg * 0.23061587074244017;
    case 2: return sg * 0.44879918020046217;
    case 3: return sg * 0.6427876096865394;
    case 4: return sg * 0.8021231927550437;
    case 5: return sg * 0.918216106880274;
    case 6: return sg * 0.984807753012208;
    case 7: return sg * 0.9983081582712682;
    case 8: return sg * 0.9579895123154889;
    case 9: return sg * 0.8660254037844386;
    case 10: return sg * 0.7273736415730487;
    case 11: return sg * 0.549508978070806;
    case 12: return sg * 0.3420201433256687;
    default: return sg * 0.11609291412523023;
  }
}

// Natural-order DFT of N values in registers, SIGN -1 forward, +1 inverse.
// N = A B with A, B coprime: the prime-factor (Good-Thomas) form, no twiddles:
// input n = (B n1 + A n2) mod N, output k = (B (B^-1 mod A) k1 + A (A^-1 mod B)
// k2) mod N.  9, 16 and 27 points: Cooley-Tukey with constant twiddles.
// zero: bit i set where v[i] is known to be zero; folded away once unrolled.
// The 3-point DFTs that see such an input (the padded middle third of an
// inverse transform) skip its operations.
template <int N, int SIGN, typename V>
__device__ __forceinline__ void dft_n(V* v, unsigned zero = 0);

template <int A, int B, int SIGN, typename V>
__device__ __forceinline__ void dft_pfa(V* v, unsigned zero) {
  constexpr int N = A * B;
  constexpr int KA = B * inv_mod(B % A, A), KB = A * inv_mod(A % B, B);
  V a[B][A];
#pragma unroll
  for (int n2 = 0; n2 < B; ++n2) {
    unsigned z = 0;
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) {
      a[n2][n1] = v[(B * n1 + A * n2) % N];
      z |= ((zero >> ((B * n1 + A * n2) % N)) & 1u) << n1;
    }
    dft_n<A, SIGN>(a[n2], z);
  }
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    V b[B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) b[n2] = a[n2][k1];
    dft_n<B, SIGN>(b);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) v[(KA * k1 + KB * k2) % N] = b[k2];
  }
}

template <int A, int B, int SIGN, typename V>
__device__ __forceinline__ void dft_ct(V* v, unsigned zero) {
  constexpr int N = A * B;
  V a[B][A];
#pragma unroll
  for (int b = 0; b < B; ++b) {
    unsigned z = 0;
#pragma unroll
    for (int n = 0; n < A; ++n) {
      a[b][n] = v[B * n + b];
      z |= ((zero >> (B * n + b)) & 1u) << n;
    }
    dft_n<A, SIGN>(a[b], z);
  }
#pragma unroll
  for (int b = 1; b < B; ++b)
#pragma unroll
    for (int k = 1; k < A; ++k) {
      if (N == 16 && b * k == 4) a[b][k] = cisign(a[b][k], SIGN);
      else a[b][k] = crot(a[b][k], cos_turn<N>(b * k), SIGN * sin_turn<N>(b * k));
    }
#pragma unroll
  for (int k = 0; k < A; ++k) {
    V c[B];
#pragma unroll
    for (int b = 0; b < B; ++b) c[b] = a[b][k];
    dft_n<B, SIGN>(c);
#pragma unroll
    for (int b = 0; b < B; ++b) v[k + A * b] = c[b];
  }
}

template <int N, int SIGN, typename V>
__device__ __forceinline__ void dft_n(V* v, unsigned zero) {
  if constexpr (N == 2) dft2(v);
  else if constexpr (N == 3) dft3(v, SIGN, zero);
  else if constexpr (N == 4) dft4(v, SIGN);
  else if constexpr (N == 8) dft8(v, SIGN);
  else if constexpr (N == 9) dft_ct<3, 3, SIGN>(v, zero);
  else if constexpr (N == 16) dft_ct<4, 4, SIGN>(v, zero);
  else if constexpr (N == 27) dft_ct<9, 3, SIGN>(v, zero);
  else if constexpr (N == 18) dft_pfa<9, 2, SIGN>(v, zero);
  else {
    static_assert(N == 6 || N == 12 || N == 24, "no register DFT of this size");
    // 3 points first where they see the zeros, else last (a caller that drops
    // the middle third of the outputs drops one of each three there)
    if (zero) dft_pfa<3, N / 3, SIGN>(v, zero);
    else dft_pfa<N / 3, 3, SIGN>(v, 0);
  }
}

// The same on the pass kernels' element types: cf2 runs it on compensated
// values.
template <int N, int SIGN, typename C>
__device__ __forceinline__ void dft_reg(C* v, unsigned zero = 0) {
  if constexpr (std::is_same<C, cf2>::value) {
    cff w[N];
#pragma unroll
    for (int i = 0; i < N; ++i) w[i] = cff_of(v[i]);
    dft_n<N, SIGN>(w, zero);
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = cff_fold(w[i]);
  } else {
    dft_n<N, SIGN>(v, zero);
  }
}

// The middle third of N inputs: what 3/2 zero-padding leaves zero.
__host__ __device__ constexpr unsigned middle_third(int N) {
  return N % 3 ? 0u : ((1u << (N / 3)) - 1u) << (N / 3);
}

// Stored index -> padded FFT position for a Nyquist-free complex axis of
// n-1 stored modes placed in a length-M transform (zeropad_fft /
// truncate_fft index maps, src/dnsjax/fft.py:41-137).
__device__ __forceinline__ int stored_to_pos(int s, int nstored, int M) {
  const int n = nstored + 1;
  return (s < n / 2) ? s : s + M - n + 1;
}
// Padded position -> stored index, or -1 where the padded array is zero.
__device__ __forceinline__ int pos_to_stored(int t, int nstored, int M) {
  const int n = nstored + 1;
  if (t < n / 2) return t;
  if (t >= M - n / 2 + 1) return t - M + n - 1;
  return -1;
}

// u - grad(inv_lapl div u) of one mode (monochromatic.py:377-385, 516-565), each
// rounding written out: the kernels that project give the same bits whatever
// surrounds the call.
__device__ __forceinline__ void project_mode(double2 (&u)[3], double kx, double ky, double kz,
                                             double inv_lapl) {
  const double k[3] = {kx, ky, kz};
  // div u = i (sx + i sy); p = inv_lapl div u
  const double sx = __fma_rn(kz, u[2].x, __fma_rn(ky, u[1].x, __dmul_rn(kx, u[0].x)));
  const double sy = __fma_rn(kz, u[2].y, __fma_rn(ky, u[1].y, __dmul_rn(kx, u[0].y)));
  const double px = __dmul_rn(sx, inv_lapl), py = __dmul_rn(sy, inv_lapl);
  // - i k (i p) = k p
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    u[q].x = __fma_rn(k[q], px, u[q].x);
    u[q].y = __fma_rn(k[q], py, u[q].y);
  }
}

// Raise a kernel's dynamic shared-memory limit to what is left of max_smem
// after its static shared memory.
inline cudaError_t allow_dynamic_smem(const void* fn, int max_smem) {
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, fn);
  if (e != cudaSuccess) return e;
  const int dyn = max_smem - (int)fa.sharedSizeBytes;
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              dyn > 0 ? dyn : 0);
}

// Copy a global twiddle table of length L into shared memory.
// Asynchronous global -> shared copies (cp.async): a thread issues all of
// its copies before waiting, so their latencies overlap.
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem)
               : "memory");
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem)
               : "memory");
}
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem)
               : "memory");
}
// One complex element, either precision.
__device__ __forceinline__ void cp_async_elem(double2* smem, const double2* gmem) {
  cp_async16(smem, gmem);
}
__device__ __forceinline__ void cp_async_elem(float2* smem, const float2* gmem) {
  cp_async8(smem, gmem);
}
// L2 eviction priority of global accesses: a policy from createpolicy,
// carried by .L2::cache_hint loads, stores and cp.async copies.  l2_keep:
// every line evict_last; l2_keep_half: evict_last on half of the lines
// (address-hashed), the rest unchanged; l2_drop: evict_first.
__device__ __forceinline__ unsigned long long l2_keep() {
  unsigned long long p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;\n" : "=l"(p));
  return p;
}
__device__ __forceinline__ unsigned long long l2_keep_half() {
  unsigned long long p;
  asm volatile("createpolicy.fractional.L2::evict_last.L2::evict_unchanged.b64 %0, 0.5;\n"
               : "=l"(p));
  return p;
}
__device__ __forceinline__ unsigned long long l2_drop() {
  unsigned long long p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(p));
  return p;
}
__device__ __forceinline__ void st_l2(double2* g, double2 v, unsigned long long pol) {
  asm volatile("st.global.L2::cache_hint.v2.f64 [%0], {%1, %2}, %3;\n" ::"l"(g), "d"(v.x),
               "d"(v.y), "l"(pol)
               : "memory");
}
__device__ __forceinline__ void st_l2(float2* g, float2 v, unsigned long long pol) {
  asm volatile("st.global.L2::cache_hint.v2.f32 [%0], {%1, %2}, %3;\n" ::"l"(g), "f"(v.x),
               "f"(v.y), "l"(pol)
               : "memory");
}
__device__ __forceinline__ void st_l2(double* g, double v, unsigned long long pol) {
  asm volatile("st.global.L2::cache_hint.f64 [%0], %1, %2;\n" ::"l"(g), "d"(v), "l"(pol)
               : "memory");
}
__device__ __forceinline__ double ld_l2(const double* g, unsigned long long pol) {
  double v;
  asm volatile("ld.global.L2::cache_hint.f64 %0, [%1], %2;\n"
               : "=d"(v)
               : "l"(g), "l"(pol)
               : "memory");
  return v;
}
__device__ __forceinline__ double2 ld_l2(const double2* g, unsigned long long pol) {
  double2 v;
  asm volatile("ld.global.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;\n"
               : "=d"(v.x), "=d"(v.y)
               : "l"(g), "l"(pol)
               : "memory");
  return v;
}
__device__ __forceinline__ float2 ld_l2(const float2* g, unsigned long long pol) {
  float2 v;
  asm volatile("ld.global.L2::cache_hint.v2.f32 {%0, %1}, [%2], %3;\n"
               : "=f"(v.x), "=f"(v.y)
               : "l"(g), "l"(pol)
               : "memory");
  return v;
}
// A load of data used once: no line allocated in L1.
__device__ __forceinline__ double2 ld_stream(const double2* g) {
  double2 v;
  asm volatile("ld.global.L1::no_allocate.v2.f64 {%0, %1}, [%2];\n"
               : "=d"(v.x), "=d"(v.y)
               : "l"(g));
  return v;
}
__device__ __forceinline__ void cp_async16_l2(void* smem, const void* g, unsigned long long pol) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;\n" ::"r"(s), "l"(g),
               "l"(pol)
               : "memory");
}
__device__ __forceinline__ void cp_async8_l2(void* smem, const void* g, unsigned long long pol) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global.L2::cache_hint [%0], [%1], 8, %2;\n" ::"r"(s), "l"(g),
               "l"(pol)
               : "memory");
}
__device__ __forceinline__ void cp_async_elem_l2(double2* smem, const double2* g,
                                                 unsigned long long pol) {
  cp_async16_l2(smem, g, pol);
}
__device__ __forceinline__ void cp_async_elem_l2(float2* smem, const float2* g,
                                                 unsigned long long pol) {
  cp_async8_l2(smem, g, pol);
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_1() {
  asm volatile("cp.async.wait_group 1;\n" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_2() {
  asm volatile("cp.async.wait_group 2;\n" ::: "memory");
}

// Programmatic dependent launch: a kernel launched by launch_dep with dep != 0
// may be set up while the kernel before it on the stream is finishing; it waits
// here, first thing, for that kernel's results, and lets the next one be set up
// in turn.  Without the launch attribute both are no-ops.
__device__ __forceinline__ void grid_dep_sync() {
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}
template <typename... KA, typename... A>
inline cudaError_t launch_dep(int dep, void (*kernel)(KA...), dim3 grid, int threads,
                              size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = dep ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, KA(args)...);
}

template <typename C>
__device__ __forceinline__ void load_twiddles(C* s, const C* g, int L) {
  for (int i = threadIdx.x; i < L; i += blockDim.x) s[i] = g[i];
}

}  // namespace dnsb
