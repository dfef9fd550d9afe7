// Axis-pass kernels of the 3/2-dealiased transforms.
//
// Index maps follow the reference's pad/truncate helpers
// (src/dnsjax/fft.py:41-190) and transform order (fft.py:193-408); the
// fused products follow src/dnsjax/rhs.py:77-90 (rotational form),
// src/dnsjax/geometries/triply_periodic.py:122-132 (curl),
// src/dnsjax/flows/plane_couette.py:251-271 (FD curl) and
// src/dnsjax/flows/monochromatic.py:366-386 (projection).
#include "passes.cuh"

#include <initializer_list>

namespace dnsb {

// Transform lengths with a compile-time FFT plan; others use the runtime
// plan (template argument 0).
#define DNSB_DISPATCH(L, KERNEL, GRID, SMEM, ST, ...)                         \
  switch (L) {                                                              \
    case 48: KERNEL<48><<<GRID, kPassThreads, SMEM, ST>>>(__VA_ARGS__); break; \
    case 72: KERNEL<72><<<GRID, kPassThreads, SMEM, ST>>>(__VA_ARGS__); break; \
    case 96: KERNEL<96><<<GRID, kPassThreads, SMEM, ST>>>(__VA_ARGS__); break; \
    case 192: KERNEL<192><<<GRID, kPassThreads, SMEM, ST>>>(__VA_ARGS__); break; \
    default: KERNEL<0><<<GRID, kPassThreads, SMEM, ST>>>(__VA_ARGS__); break; \
  }
// Variant 2 (runtime-planned stages) takes KERNEL<0> whatever L is.
#define DNSB_DISPATCH_V(VAR, L, KERNEL, GRID, SMEM, ST, ...)                  \
  do {                                                                      \
    if ((VAR) == 2)                                                         \
      KERNEL<0><<<GRID, kPassThreads, SMEM, ST>>>(__VA_ARGS__);             \
    else                                                                    \
      DNSB_DISPATCH(L, KERNEL, GRID, SMEM, ST, __VA_ARGS__);                \
  } while (0)

FFTPlan make_plan(int L) {
  FFTPlan P{};
  P.L = L;
  P.nst = 0;
  int n = L;
  if (L < 1) return P;
  while (n % 8 == 0 && n != 8 && P.nst < DNSB_MAX_STAGES) {
    P.radix[P.nst++] = 8;
    n /= 8;
  }
  while (n % 4 == 0 && n > 1 && P.nst < DNSB_MAX_STAGES) {
    P.radix[P.nst++] = 4;
    n /= 4;
  }
  while (n % 2 == 0 && n > 1 && P.nst < DNSB_MAX_STAGES) {
    P.radix[P.nst++] = 2;
    n /= 2;
  }
  while (n % 3 == 0 && n > 1 && P.nst < DNSB_MAX_STAGES) {
    P.radix[P.nst++] = 3;
    n /= 3;
  }
  if (n == 8 && P.nst < DNSB_MAX_STAGES) {
    P.radix[P.nst++] = 8;
    n = 1;
  }
  if (n != 1) P.nst = 0;
  return P;
}

// ---------------------------------------------------------------------------
// Generic strided column pass.
// ---------------------------------------------------------------------------
size_t col_pass_smem(int M) {
  return sizeof(double2) * (size_t)(2 * M * kTile + M);
}

template <int ML>
__global__ void __launch_bounds__(kPassThreads)
col_pass_kernel(ColPassArgs a) {
  extern __shared__ double2 sm[];
  const int M = ML > 0 ? ML : a.plan.L;
  const int C = kTile;
  double2* bufA = sm;
  double2* bufB = sm + M * C;
  double2* tw = sm + 2 * M * C;
  const int i0 = blockIdx.x * C;
  const long long o = blockIdx.y;
  const long long f = blockIdx.z;
  const double2* in = a.in + f * a.in_fs + o * a.in_os + i0;
  double2* out = a.out + f * a.out_fs + o * a.out_os + i0;
  const int ni = min(C, a.nI - i0);
  load_twiddles(tw, a.tw, M);
  if (a.inverse) {
    for (int idx = threadIdx.x; idx < M * C; idx += blockDim.x) {
      const int c = idx % C, t = idx / C;
      const int s = pos_to_stored(t, a.nstored, M);
      double2 v = make_double2(0.0, 0.0);
      if (s >= 0 && c < ni) v = in[s * a.in_ts + c];
      bufA[idx] = v;
    }
  } else {
    for (int idx = threadIdx.x; idx < M * C; idx += blockDim.x) {
      const int c = idx % C, t = idx / C;
      double2 v = make_double2(0.0, 0.0);
      if (c < ni) v = in[t * a.in_ts + c];
      bufA[idx] = v;
    }
  }
  __syncthreads();
  const double2* res = fft_cols<ML, C, kPassThreads>(bufA, bufB, a.plan, a.inverse ? 1 : -1, tw);
  if (a.inverse) {
    for (int idx = threadIdx.x; idx < M * C; idx += blockDim.x) {
      const int c = idx % C, t = idx / C;
      if (c < ni) out[t * a.out_ts + c] = res[idx];
    }
  } else {
    const double sc = 1.0 / M;
    for (int idx = threadIdx.x; idx < a.nstored * C; idx += blockDim.x) {
      const int c = idx % C, s = idx / C;
      const int t = stored_to_pos(s, a.nstored, M);
      if (c < ni) out[s * a.out_ts + c] = cscale(res[t * C + c], sc);
    }
  }
}

// ---------------------------------------------------------------------------
// Column pass, two register stages (M = R1 R2): stage 1 (radix R1, Ns = 1)
// loads its inputs from global memory (zero-padding applied on load), stage 2
// (radix R2, Ns = R1) stores its outputs to global memory (truncation applied
// on store); one shared buffer in between.  A CTA takes C columns with one
// thread per stage-1 item.
//
// Shapes: one thread per stage-1 item, 16 columns (256-byte runs), 8 where 16
// would leave two CTAs per SM (M = 288, 384).  What bounds the pass is latency at
// the occupancy its registers allow (DRAM 32-56%, FP64 19-28% busy at M = 192),
// so M = 192 is 12 x 16 with 24 warps per SM, not 24 x 8 with 16: 128^3 periodic
// RHS 359 -> 344 us, Couette 128 RHS 213 -> 203 us (16 x 12: 360, 210).
// Against the Stockham stages with one radix <= 8
// exchange each that the lengths beyond 48, 72, 96 and 192 ran before, one
// shared-memory round trip replaces three to five: the four column passes of a
// 256^3 periodic RHS (M = 384) took 5.3 ms, now 2.0 ms (all the passes of a
// 144 x 192 x 108 predict_and_correct: 3.36 -> 2.25 ms).
// ---------------------------------------------------------------------------
constexpr int col_columns(int L) { return L >= 288 ? 8 : 16; }
template <int M>
struct ColShape {
  static constexpr int R1 = ColRadix<M>::R1, R2 = ColRadix<M>::R2, C = col_columns(M);
  static constexpr int NT = R2 * C;
  // CTAs per SM that the registers are held to: 768 threads' worth where at most 16
  // complex values a thread fit 80 registers (24 warps, 25 at 108 points), else 512
  // (12 to 16 warps)
  static constexpr int MINB = (R1 <= 16 && R2 <= 16 ? 768 : 512) / NT;
  // the same for the Couette z inverse, whose curl takes more
  static constexpr int ZB = M == 36 || M == 54                             ? 5
                            : M == 108 || M == 144 || M == 162 || M == 192 ? 3
                            : M == 216                                     ? 2
                                                                           : 4;
};

size_t col_pass2_smem(int M) {
  return sizeof(double2) * (size_t)(M * col_columns(M) + M);
}

// T: the compute type and the element type of `in` (double, or float for the
// FP32 forms, whose pass buffers hold float2); `out` is complex128, or with
// OUT32 (FP32 only) an FP32 pass buffer.  CURL (inverse): `in` is the FP64
// spectral state and field f of the 6 is u, v, w (f < 3) or the spectral
// curl i (k x u) (triply_periodic.py:122-132), formed in FP64 at the load.
// H = 2 (the work-list kernels): the CTA has twice the shape's NT threads, and each
// half of it runs a block, (bx, by, bz) its own; idle: no block is left for the half.
template <int ML, int SIGN, typename T = double, bool OUT32 = false, bool CURL = false,
          bool SLAB = false, int H = 1>
__device__ __forceinline__ void col_pass2_body(const ColPassArgs& a, int bx, int by, int bz,
                                               bool idle = false) {
  using CT = typename pass_types<T>::C;
  using RT = typename pass_types<T>::R;
  constexpr int M = ML, R1 = ColShape<ML>::R1, R2 = ColShape<ML>::R2, C = ColShape<ML>::C;
  constexpr int NT = ColShape<ML>::NT;
  extern __shared__ double2 sm_[];
  const int half = H == 2 ? threadIdx.x / NT : 0;
  CT* X = reinterpret_cast<CT*>(sm_) + half * (M * C + M);  // [t][C]
  CT* tw = X + M * C;
  const int tid = threadIdx.x - half * NT;
  const int i0 = bx * C;
  const long long o = by;
  const long long f = bz;
  const CT* in = reinterpret_cast<const CT*>(a.in) + f * a.in_fs + o * a.in_os + i0;
  // FP64 output, or (OUT32, FP32 arithmetic) an FP32 pass buffer
  double2* out = a.out + f * a.out_fs + o * a.out_os + i0;
  CT* out_c = reinterpret_cast<CT*>(a.out) + f * a.out_fs + o * a.out_os + i0;
  const int ni = H == 2 && idle ? 0 : min(C, a.nI - i0);
  const unsigned long long drop = l2_drop();
  if constexpr (H == 2) {
    for (int i = tid; i < M; i += NT) tw[i] = reinterpret_cast<const CT*>(a.tw)[i];
  } else {
    load_twiddles(tw, reinterpret_cast<const CT*>(a.tw), M);
  }
  __syncthreads();
  {
    const int c = tid % C, j = tid / C;
    CT v[R1];
#pragma unroll
    for (int i = 0; i < R1; ++i) {
      const int t = j + R2 * i;
      CT z = cmake<CT>(0, 0);
      if (c < ni) {
        if (SIGN > 0) {
          const int sidx = pos_to_stored(t, a.nstored, M);
          if (sidx >= 0) {
            if constexpr (CURL) {
              // f is the same for the whole CTA: load only the components
              // the field needs
              const double2* st = reinterpret_cast<const double2*>(a.in) + o * a.in_os + i0 +
                                  (long long)sidx * a.in_ts + c;
              const long long fs = a.in_fs;
              double2 q;
              switch (f) {
                case 0: q = st[0]; break;
                case 1: q = st[fs]; break;
                case 2: q = st[2 * fs]; break;
                case 3: {
                  const double2 vv = st[fs], w = st[2 * fs];
                  const double ky = a.ky[sidx], kz = a.kz[o];
                  q = ci(make_double2(ky * w.x - kz * vv.x, ky * w.y - kz * vv.y));
                  break;
                }
                case 4: {
                  const double2 u = st[0], w = st[2 * fs];
                  const double kx = a.kx[i0 + c], kz = a.kz[o];
                  q = ci(make_double2(kz * u.x - kx * w.x, kz * u.y - kx * w.y));
                  break;
                }
                default: {
                  const double2 u = st[0], vv = st[fs];
                  const double kx = a.kx[i0 + c], ky = a.ky[sidx];
                  q = ci(make_double2(kx * vv.x - ky * u.x, kx * vv.y - ky * u.y));
                  break;
                }
              }
              z = to_c(q, (CT*)nullptr);
            } else {
              z = in[sidx * a.in_ts + c];
            }
          }
        } else {
          z = ld_l2(in + t * a.in_ts + c, drop);  // the input's last use
        }
      }
      v[i] = z;
    }
    dft_reg<R1, SIGN>(v);
#pragma unroll
    for (int i = 0; i < R1; ++i) X[(j * R1 + i) * C + c] = v[i];
  }
  __syncthreads();
  const double sc = 1.0 / M;
  for (int it = tid; it < R1 * C; it += NT) {
    const int c = it % C, k = it / C;
    CT z[R2];
#pragma unroll
    for (int i = 0; i < R2; ++i) z[i] = X[(k + R1 * i) * C + c];
#pragma unroll
    for (int i = 1; i < R2; ++i) {
      CT w = tw[i * k];
      if (SIGN > 0) w.y = -w.y;
      z[i] = cmul(z[i], w);
    }
    dft_reg<R2, SIGN>(z);
    if (c < ni) {
#pragma unroll
      for (int i = 0; i < R2; ++i) {
        const int t = k + R1 * i;
        if (SIGN > 0) {
          if constexpr (SLAB) {
            // position t belongs to rank t / blk (its padded-z share)
            const int q = t / a.slab.blk;
            a.slab.buf[q][f * a.slab.fs + o * a.out_os + (t - q * a.slab.blk) * a.slab.ts +
                          a.slab.off + i0 + c] = to_d(z[i]);
          } else if (OUT32) {
            out_c[t * a.out_ts + c] = z[i];
          } else {
            out[t * a.out_ts + c] = to_d(z[i]);
          }
        } else {
          const int sidx = pos_to_stored(t, a.nstored, M);
          if (sidx >= 0) {
            if (OUT32) out_c[sidx * a.out_ts + c] = cscale(z[i], (RT)sc);
            else out[sidx * a.out_ts + c] = cscale(to_d(z[i]), sc);
          }
        }
      }
    }
  }
}

// Block (bx, by, bz) = (column tile, outer index, field) of the grid
// ((nI + C - 1) / C, nO, nfields); the work-list ensemble kernels call the body
// with their own block numbering.
template <int ML, int SIGN, typename T = double, bool OUT32 = false, bool CURL = false,
          bool SLAB = false>
__global__ void __launch_bounds__(ColShape<ML>::NT)
col_pass2_kernel(ColPassArgs a) {
  grid_dep_sync();
  if (a.skip && *a.skip) return;
  col_pass2_body<ML, SIGN, T, OUT32, CURL, SLAB>(a, blockIdx.x, blockIdx.y, blockIdx.z);
}

// The FP64 pass with its registers held to ColShape::MINB CTAs per SM: the inverse
// passes, the forward ones with ColPassArgs::held and at the lengths compiled for
// FP64 alone.
template <int ML, int SIGN, bool CURL>
__global__ void __launch_bounds__(ColShape<ML>::NT, ColShape<ML>::MINB)
col_pass2_held_kernel(ColPassArgs a) {
  grid_dep_sync();
  if (a.skip && *a.skip) return;
  if (CURL && a.fields_fast)
    col_pass2_body<ML, SIGN, double, false, CURL, false>(a, blockIdx.y, blockIdx.z, blockIdx.x);
  else
    col_pass2_body<ML, SIGN, double, false, CURL, false>(a, blockIdx.x, blockIdx.y, blockIdx.z);
}

cudaError_t launch_col_pass(const ColPassArgs& a, int nfields, int nO,
                            cudaStream_t st) {
  const int L = a.plan.L;
  if (a.variant == 0 && two_stage_length(L)) {
    const int C = col_columns(L);
    const dim3 g2((a.nI + C - 1) / C, nO, nfields);
    const size_t sm2 = a.fp32 ? col_pass2_smem(L) / 2 : col_pass2_smem(L);
    const bool slab = a.slab.buf[0] != nullptr;
    if ((a.fp32 || slab) && !fp32_length(L)) return cudaErrorInvalidValue;
    if (a.fp32 && a.inverse && !a.out32) return cudaErrorInvalidValue;
    if (slab && (a.fp32 || a.curl || !a.inverse)) return cudaErrorInvalidValue;
    return with_length(L, [&](auto len) {
      constexpr int LL = decltype(len)::value, NT = ColShape<LL>::NT;
      if constexpr (fp32_length(LL)) {
        if (slab)
          launch_dep(a.dep, col_pass2_kernel<LL, 1, double, false, false, true>, g2, NT, sm2, st,
                     a);
        else if (a.curl && a.fp32 == 2)
          launch_dep(a.dep, col_pass2_kernel<LL, 1, fcomp, true, true>, g2, NT, sm2, st, a);
        else if (a.fp32 == 2 && a.inverse)
          launch_dep(a.dep, col_pass2_kernel<LL, 1, fcomp, true>, g2, NT, sm2, st, a);
        else if (a.fp32 == 2 && a.out32)
          launch_dep(a.dep, col_pass2_kernel<LL, -1, fcomp, true>, g2, NT, sm2, st, a);
        else if (a.fp32 == 2)
          launch_dep(a.dep, col_pass2_kernel<LL, -1, fcomp>, g2, NT, sm2, st, a);
        else if (a.curl && a.fp32)
          launch_dep(a.dep, col_pass2_kernel<LL, 1, float, true, true>, g2, NT, sm2, st, a);
        else if (a.fp32 && a.inverse)
          launch_dep(a.dep, col_pass2_kernel<LL, 1, float, true>, g2, NT, sm2, st, a);
        else if (a.fp32 && a.out32)
          launch_dep(a.dep, col_pass2_kernel<LL, -1, float, true>, g2, NT, sm2, st, a);
        else if (a.fp32)
          launch_dep(a.dep, col_pass2_kernel<LL, -1, float>, g2, NT, sm2, st, a);
        else if (!a.inverse && !a.held)
          launch_dep(a.dep, col_pass2_kernel<LL, -1>, g2, NT, sm2, st, a);
        if (slab || a.fp32 || (!a.inverse && !a.held)) return cudaGetLastError();
      }
      if (a.curl) {
        const dim3 gf = a.fields_fast ? dim3(g2.z, g2.x, g2.y) : g2;
        launch_dep(a.dep, col_pass2_held_kernel<LL, 1, true>, gf, NT, sm2, st, a);
      } else if (a.inverse)
        launch_dep(a.dep, col_pass2_held_kernel<LL, 1, false>, g2, NT, sm2, st, a);
      else
        launch_dep(a.dep, col_pass2_held_kernel<LL, -1, false>, g2, NT, sm2, st, a);
      return cudaGetLastError();
    });
  }
  // two-stage compile-time passes only
  if (a.fp32 || a.curl || a.slab.buf[0]) return cudaErrorInvalidValue;
  dim3 grid((a.nI + kTile - 1) / kTile, nO, nfields);
  size_t sm = col_pass_smem(a.plan.L);
  DNSB_DISPATCH_V(a.variant, a.plan.L, col_pass_kernel, grid, sm, st, a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// x pass: two real fields per complex transform (z = a + i b).
// ---------------------------------------------------------------------------
__device__ __forceinline__ long long row_offset(int r, int inner_n,
                                                long long so, long long si) {
  return (long long)(r / inner_n) * so + (long long)(r % inner_n) * si;
}

size_t x_pass_smem(int Mx) {
  return sizeof(double2) * (size_t)(2 * Mx * 3 * kXRows + Mx);
}

template <int ML>
__global__ void __launch_bounds__(kPassThreads)
x_pass_kernel(XPassArgs a) {
  extern __shared__ double2 sm[];
  const int M = ML > 0 ? ML : a.plan.L;
  const int R = kXRows;
  const int CI = 3 * R;  // inverse columns
  const int CF = 2 * R;  // forward columns
  double2* bufA = sm;
  double2* bufB = sm + M * CI;
  double2* tw = sm + 2 * M * CI;
  const int r0 = blockIdx.x * R;
  const int nr = min(R, a.nrows - r0);
  const int nkx = ML > 0 ? ML / 3 : a.nkx;  // launcher guarantees nx/2 = M/3
  __shared__ long long s_off[kXRows];
  __shared__ int s_y[kXRows];
  if (threadIdx.x < R) {
    const int row = r0 + threadIdx.x;
    const int outer = row / a.inner_n, inner = row % a.inner_n;
    s_off[threadIdx.x] = (long long)outer * a.so + (long long)inner * a.si;
    s_y[threadIdx.x] = a.y_outer ? outer : inner;
  }
  load_twiddles(tw, a.tw, M);
  __syncthreads();
  // Stage the 6 half spectra: stage[(f * nkx + k) * R + r] in bufB.
  double2* stage = bufB;
  const int nload = 6 * nkx * R;
  for (int idx = threadIdx.x; idx < nload; idx += blockDim.x) {
    int r, k, f;
    if (a.rows_fast) {
      r = idx % R;
      k = (idx / R) % nkx;
      f = idx / (R * nkx);
    } else {
      k = idx % nkx;
      r = (idx / nkx) % R;
      f = idx / (R * nkx);
    }
    double2 v = make_double2(0.0, 0.0);
    if (r < nr) v = a.in[f * a.in_fs + s_off[r] + k * a.ks];
    stage[(f * nkx + k) * R + r] = v;
  }
  __syncthreads();
  // Build the 3 complex inputs per row: (u_x,u_y), (u_z,w_x), (w_y,w_z).
  for (int idx = threadIdx.x; idx < M * CI; idx += blockDim.x) {
    const int q = idx % CI, t = idx / CI;
    const int r = q / 3, pr = q % 3;
    const int fa = 2 * pr, fb = 2 * pr + 1;
    double2 z = make_double2(0.0, 0.0);
    if (t == 0) {
      z = make_double2(stage[(fa * nkx) * R + r].x, stage[(fb * nkx) * R + r].x);
    } else if (t < nkx) {
      const double2 A = stage[(fa * nkx + t) * R + r];
      const double2 B = stage[(fb * nkx + t) * R + r];
      z = make_double2(A.x - B.y, A.y + B.x);
    } else if (M - t < nkx) {
      const int k = M - t;
      const double2 A = stage[(fa * nkx + k) * R + r];
      const double2 B = stage[(fb * nkx + k) * R + r];
      z = make_double2(A.x + B.y, -A.y + B.x);
    }
    bufA[idx] = z;
  }
  __syncthreads();
  double2* res = fft_cols<ML, CI, kPassThreads>(bufA, bufB, a.plan, 1, tw);
  double2* nl = (res == bufA) ? bufB : bufA;
  // Rotational nonlinear product at every physical point of the rows.
  for (int idx = threadIdx.x; idx < M * R; idx += blockDim.x) {
    const int r = idx % R, t = idx / R;
    double2 o0 = make_double2(0.0, 0.0), o1 = make_double2(0.0, 0.0);
    if (r < nr) {
      const double2 z0 = res[t * CI + 3 * r + 0];
      const double2 z1 = res[t * CI + 3 * r + 1];
      const double2 z2 = res[t * CI + 3 * r + 2];
      const double u0 = z0.x, u1 = z0.y, u2 = z1.x;
      const double w0 = z1.y, w1 = z2.x, w2 = z2.y;
      const int y = s_y[r];
      const int ny = a.ny_grid;
      const double U0 = a.U[y], U1 = a.U[ny + y], U2 = a.U[2 * ny + y];
      const double C0 = a.cU[y], C1 = a.cU[ny + y], C2 = a.cU[2 * ny + y];
      const double N0 = a.nU[y], N1 = a.nU[ny + y], N2 = a.nU[2 * ny + y];
      // u x w
      const double n0 = u1 * w2 - u2 * w1;
      const double n1 = u2 * w0 - u0 * w2;
      const double n2 = u0 * w1 - u1 * w0;
      // u x curl U + U x w + U x curl U
      const double b0 = (u1 * C2 - u2 * C1) + (U1 * w2 - U2 * w1) + N0;
      const double b1 = (u2 * C0 - u0 * C2) + (U2 * w0 - U0 * w2) + N1;
      const double b2 = (u0 * C1 - u1 * C0) + (U0 * w1 - U1 * w0) + N2;
      o0 = make_double2(n0 + b0, n1 + b1);
      o1 = make_double2(n2 + b2, 0.0);
    }
    nl[t * CF + 2 * r + 0] = o0;
    nl[t * CF + 2 * r + 1] = o1;
  }
  __syncthreads();
  double2* other = (nl == bufA) ? bufB : bufA;
  double2* fres = fft_cols<ML, CF, kPassThreads>(nl, other, a.plan, -1, tw);
  // Unpack the real-field spectra, truncate to nkx, scale 1/M, store.
  const double h = 0.5 / M;
  const int nst = 3 * nkx * R;
  for (int idx = threadIdx.x; idx < nst; idx += blockDim.x) {
    int r, k, f;
    if (a.rows_fast) {
      r = idx % R;
      k = (idx / R) % nkx;
      f = idx / (R * nkx);
    } else {
      k = idx % nkx;
      r = (idx / nkx) % R;
      f = idx / (R * nkx);
    }
    if (r >= nr) continue;
    const int col = 2 * r + (f == 2 ? 1 : 0);
    const double2 Z = fres[k * CF + col];
    const double2 Zm = fres[((M - k) % M) * CF + col];
    double2 v;
    if (f == 1) {
      v = make_double2((Z.y + Zm.y) * h, (Zm.x - Z.x) * h);
    } else {
      v = make_double2((Z.x + Zm.x) * h, (Z.y - Zm.y) * h);
    }
    a.out[f * a.out_fs + s_off[r] + k * a.ks] = v;
  }
}

cudaError_t launch_x_pass(const XPassArgs& a, cudaStream_t st) {
  dim3 grid((a.nrows + kXRows - 1) / kXRows);
  // The compile-time variants assume nx/2 = M/3 (3/2 oversampling).
  const int L = (a.nkx * 3 == a.plan.L) ? a.plan.L : -1;
  const bool slab = a.slab.buf[0] != nullptr;
  if (slab && (a.fp32 || a.variant != 0 || L < 0)) return cudaErrorInvalidValue;
  if (a.variant == 0 && two_stage_length(L)) return launch_x_pass2(a, st);
  if (a.fp32) return cudaErrorInvalidValue;  // two-stage compile-time passes only
  DNSB_DISPATCH_V(a.variant, L, x_pass_kernel, grid, x_pass_smem(a.plan.L), st, a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Work-list forms for ensembles (csrc/capi.cu, dnsb_ensemble_*): one launch
// runs the two-stage pass of every member.  Item k covers the member's blocks
// base_k .. base_k + blocks_k - 1 of the flattened grid (bx fastest); every
// CTA walks the virtual blocks blockIdx.x, blockIdx.x + gridDim.x, ... and
// runs the member's body on its block, so each member computes exactly what
// its own launch computes.  Members whose `active` flag is 0 are skipped.
// ---------------------------------------------------------------------------
// CTAs of the widest member's shape: 256 threads where a member is 192 long, else
// 128.  Members of the shorter shape run two of their blocks in a wide CTA: with one
// and half of its threads idle, a step of 24 members of 48 to 192 points took 9.15
// ms, 7.67 so (128 threads for all, 24 x 8 at 192: 8.98); four of 128^3: 9.49 and
// 9.32 ms.
__host__ __device__ constexpr int ens_col_threads(bool wide) {
  return wide ? ColShape<192>::NT : ColShape<96>::NT;
}
static_assert(ColShape<48>::NT == ens_col_threads(false) &&
                  ColShape<72>::NT == ens_col_threads(false) &&
                  ens_col_threads(true) == 2 * ens_col_threads(false),
              "a CTA shape for every member");

// A member's block in this half of the CTA.
template <int ML, int SIGN, bool CURL, bool WIDE>
__device__ __forceinline__ void ens_col_block(const EnsColItem& it, const ColPassArgs& a,
                                              int local) {
  constexpr int H = WIDE && ColShape<ML>::NT < ens_col_threads(true) ? 2 : 1;
  const int b = H == 2 ? 2 * local + threadIdx.x / ColShape<ML>::NT : local;
  const int blk = min(b, it.blocks - 1), gx = it.gx, gy = it.gy;
  col_pass2_body<ML, SIGN, double, false, CURL, false, H>(a, blk % gx, (blk / gx) % gy,
                                                          blk / (gx * gy), b != blk);
}

// Wide: 16 warps per SM (the curl pass without the bound takes 246 registers).
template <int SIGN, bool CURL, bool WIDE>
__global__ void __launch_bounds__(ens_col_threads(WIDE), WIDE ? 2 : 0)
ens_col_pass2_kernel(const EnsColItem* __restrict__ items, const int* __restrict__ base, int n,
                     int total, const int* __restrict__ active) {
  __shared__ int s_k;
  for (int vb = blockIdx.x; vb < total; vb += gridDim.x) {
    if (threadIdx.x == 0) s_k = ens_find(base, n, vb);
    __syncthreads();
    const int k = s_k;
    const int m = items[k].member;
    if (!active || active[m]) {
      const ColPassArgs a = items[k].a;
      const int local = vb - base[k];
      switch (a.plan.L) {
        case 48: ens_col_block<48, SIGN, CURL, WIDE>(items[k], a, local); break;
        case 72: ens_col_block<72, SIGN, CURL, WIDE>(items[k], a, local); break;
        case 96: ens_col_block<96, SIGN, CURL, WIDE>(items[k], a, local); break;
        default:
          if constexpr (WIDE) ens_col_block<192, SIGN, CURL, WIDE>(items[k], a, local);
          break;
      }
    }
    __syncthreads();  // shared memory and s_k are reused by the next block
  }
}

bool ens_pass_supported(int L) { return fp32_length(L); }

int ens_col_blocks(EnsColItem* it, int nO, int nfields, bool wide) {
  const int L = it->a.plan.L, C = col_columns(L);
  it->gx = (it->a.nI + C - 1) / C;
  it->gy = nO;
  it->blocks = it->gx * nO * nfields;
  return wide && L != 192 ? (it->blocks + 1) / 2 : it->blocks;
}

size_t ens_col_smem(int maxL) { return col_pass2_smem(maxL); }

// kind 0: inverse with the curl, 1: inverse, 2: forward (col_pass2); 3: x pass;
// 4: y forward with the projection.  wide: a member is 192 long.
static const void* ens_kernel(int kind, bool wide) {
  switch (kind) {
    case 0:
      return wide ? (const void*)ens_col_pass2_kernel<1, true, true>
                  : (const void*)ens_col_pass2_kernel<1, true, false>;
    case 1:
      return wide ? (const void*)ens_col_pass2_kernel<1, false, true>
                  : (const void*)ens_col_pass2_kernel<1, false, false>;
    case 2:
      return wide ? (const void*)ens_col_pass2_kernel<-1, false, true>
                  : (const void*)ens_col_pass2_kernel<-1, false, false>;
    case 3: return ens_x_kernel();
    default: return ens_y_kernel(wide);
  }
}

static int ens_threads(int kind, bool wide) {
  return kind == 3 ? kEnsXThreads : kind == 4 ? ens_y_threads(wide) : ens_col_threads(wide);
}

// Persistent grid of a work-list pass kernel: resident CTAs per SM x SMs,
// at most `total`; also raises the kernel's dynamic shared-memory limit.
int ens_pass_grid(int kind, bool wide, size_t smem, int total, int max_smem) {
  const void* f = ens_kernel(kind, wide);
  if (allow_dynamic_smem(f, max_smem) != cudaSuccess) return 0;
  int per_sm = 0, dev = 0, nsm = 0;
  const int threads = ens_threads(kind, wide);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, threads, smem) != cudaSuccess)
    return 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 0;
  const int g = per_sm * nsm;
  return g < total ? g : total;
}

cudaError_t launch_ens_pass(int kind, bool wide, const void* items, const int* base, int n,
                            int total, const int* active, int grid, size_t smem,
                            cudaStream_t st) {
  // every kernel's parameters are (items, base, n, total, active)
  void* args[] = {&items, &base, &n, &total, &active};
  return cudaLaunchKernel(ens_kernel(kind, wide), dim3(grid), dim3(ens_threads(kind, wide)), args,
                          smem, st);
}

// x pass to physical values only (spec_to_phys of 3 fields).
size_t x_phys_smem(int Mx) {
  return sizeof(double2) * (size_t)(2 * Mx * 2 * kXRows + Mx);
}

template <int ML>
__global__ void __launch_bounds__(kPassThreads)
x_phys_kernel(XPhysArgs a) {
  extern __shared__ double2 sm[];
  const int M = ML > 0 ? ML : a.plan.L;
  const int R = kXRows;
  const int CI = 2 * R;
  double2* bufA = sm;
  double2* bufB = sm + M * CI;
  double2* tw = sm + 2 * M * CI;
  const int r0 = blockIdx.x * R;
  const int nr = min(R, a.nrows - r0);
  const int nkx = a.nkx;
  load_twiddles(tw, a.tw, M);
  double2* stage = bufB;
  for (int idx = threadIdx.x; idx < 3 * nkx * R; idx += blockDim.x) {
    int r, k, f;
    if (a.rows_fast) {
      r = idx % R;
      k = (idx / R) % nkx;
      f = idx / (R * nkx);
    } else {
      k = idx % nkx;
      r = (idx / nkx) % R;
      f = idx / (R * nkx);
    }
    double2 v = make_double2(0.0, 0.0);
    if (r < nr) {
      const long long off = row_offset(r0 + r, a.inner_n, a.so, a.si);
      v = a.in[f * a.in_fs + off + k * a.ks];
    }
    stage[(f * nkx + k) * R + r] = v;
  }
  // Zero partner of the third field lives past the staged block.
  double2* zeros = stage + 3 * nkx * R;
  for (int idx = threadIdx.x; idx < nkx * R; idx += blockDim.x)
    zeros[idx] = make_double2(0.0, 0.0);
  __syncthreads();
  for (int idx = threadIdx.x; idx < M * CI; idx += blockDim.x) {
    const int q = idx % CI, t = idx / CI;
    const int r = q / 2, pr = q % 2;
    const double2* A = stage + ((2 * pr) * nkx) * R + r;
    const double2* B = (pr == 0) ? stage + (1 * nkx) * R + r : zeros + r;
    double2 z = make_double2(0.0, 0.0);
    if (t == 0) {
      z = make_double2(A[0].x, B[0].x);
    } else if (t < nkx) {
      const double2 Av = A[t * R], Bv = B[t * R];
      z = make_double2(Av.x - Bv.y, Av.y + Bv.x);
    } else if (M - t < nkx) {
      const int k = M - t;
      const double2 Av = A[k * R], Bv = B[k * R];
      z = make_double2(Av.x + Bv.y, -Av.y + Bv.x);
    }
    bufA[idx] = z;
  }
  __syncthreads();
  const double2* res = fft_cols<ML, CI, kPassThreads>(bufA, bufB, a.plan, 1, tw);
  for (int idx = threadIdx.x; idx < M * R * 3; idx += blockDim.x) {
    const int t = idx % M;
    const int r = (idx / M) % R;
    const int f = idx / (M * R);
    if (r >= nr) continue;
    const double2 z = res[t * CI + 2 * r + (f == 2 ? 1 : 0)];
    const double v = (f == 1) ? z.y : z.x;
    const long long off = row_offset(r0 + r, a.inner_n, a.pso, a.psi);
    a.out[f * a.out_fs + off + t] = v;
  }
}

cudaError_t launch_x_phys(const XPhysArgs& a, cudaStream_t st) {
  if (two_stage_length(a.plan.L) && 3 * a.nkx == a.plan.L) return launch_x_phys2(a, st);
  dim3 grid((a.nrows + kXRows - 1) / kXRows);
  DNSB_DISPATCH(a.plan.L, x_phys_kernel, grid, x_phys_smem(a.plan.L), st, a);
  return cudaGetLastError();
}

// Forward x pass from physical values (phys_to_spec of 3 fields): rows of
// real samples at outer*pso + inner*psi -> x half spectra at outer*so +
// inner*si, kx modes ks apart, truncated to nkx, scaled 1/Mx.
template <int ML>
__global__ void __launch_bounds__(kPassThreads)
x_fwd_kernel(XPhysArgs a, const double* phys, double2* spec) {
  extern __shared__ double2 sm[];
  const int M = ML > 0 ? ML : a.plan.L;
  const int R = kXRows;
  const int CF = 2 * R;
  double2* bufA = sm;
  double2* bufB = sm + M * CF;
  double2* tw = sm + 2 * M * CF;
  const int r0 = blockIdx.x * R;
  const int nr = min(R, a.nrows - r0);
  const int nkx = a.nkx;
  load_twiddles(tw, a.tw, M);
  for (int idx = threadIdx.x; idx < M * CF; idx += blockDim.x) {
    const int t = idx % M;
    const int q = idx / M;
    const int r = q / 2, pr = q % 2;
    double re = 0.0, im = 0.0;
    if (r < nr) {
      const long long off = row_offset(r0 + r, a.inner_n, a.pso, a.psi);
      if (pr == 0) {
        re = phys[0 * a.out_fs + off + t];
        im = phys[1 * a.out_fs + off + t];
      } else {
        re = phys[2 * a.out_fs + off + t];
      }
    }
    bufA[t * CF + q] = make_double2(re, im);
  }
  __syncthreads();
  const double2* fres = fft_cols<ML, CF, kPassThreads>(bufA, bufB, a.plan, -1, tw);
  const double h = 0.5 / M;
  for (int idx = threadIdx.x; idx < 3 * nkx * R; idx += blockDim.x) {
    int r, k, f;
    if (a.rows_fast) {
      r = idx % R;
      k = (idx / R) % nkx;
      f = idx / (R * nkx);
    } else {
      k = idx % nkx;
      r = (idx / nkx) % R;
      f = idx / (R * nkx);
    }
    if (r >= nr) continue;
    const int col = 2 * r + (f == 2 ? 1 : 0);
    const double2 Z = fres[k * CF + col];
    const double2 Zm = fres[((M - k) % M) * CF + col];
    double2 v;
    if (f == 1) {
      v = make_double2((Z.y + Zm.y) * h, (Zm.x - Z.x) * h);
    } else {
      v = make_double2((Z.x + Zm.x) * h, (Z.y - Zm.y) * h);
    }
    const long long off = row_offset(r0 + r, a.inner_n, a.so, a.si);
    spec[f * a.in_fs + off + k * a.ks] = v;
  }
}

size_t x_fwd_smem(int Mx) {
  return sizeof(double2) * (size_t)(2 * Mx * 2 * kXRows + Mx);
}

cudaError_t launch_x_fwd(const XPhysArgs& a, const double* phys, double2* spec,
                         cudaStream_t st) {
  if (two_stage_length(a.plan.L) && 3 * a.nkx == a.plan.L) return launch_x_fwd2(a, phys, spec, st);
  dim3 grid((a.nrows + kXRows - 1) / kXRows);
  DNSB_DISPATCH(a.plan.L, x_fwd_kernel, grid, x_fwd_smem(a.plan.L), st, a, phys, spec);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Periodic first inverse pass (y) with the spectral curl fused.
// ---------------------------------------------------------------------------
// FP32 form (a Stockham variant chosen for the FP64 passes before the precision was
// set): the state columns and the curl stay FP64 (su); the transform buffers,
// twiddles and the output pass buffer are FP32.
size_t yinv_smem(int My, int NY1, int fp32) {
  const size_t cb = fp32 ? sizeof(float2) : sizeof(double2);
  return sizeof(double2) * (size_t)(3 * NY1 * kTile) + cb * (size_t)(2 * My * kTile + My);
}

template <int ML, typename T = double>
__global__ void __launch_bounds__(kPassThreads)
yinv_kernel(YInvArgs a) {
  using CT = typename pass_types<T>::C;
  using RT = typename pass_types<T>::R;
  extern __shared__ double2 sm[];
  const int M = ML > 0 ? ML : a.plan.L;
  const int C = kTile;
  const int NY1 = a.NY1, NZ1 = a.NZ1, NKX = a.NKX;
  double2* su = sm;                       // [3][NY1][C]
  CT* bufA = reinterpret_cast<CT*>(su + 3 * NY1 * C);
  CT* bufB = bufA + M * C;
  CT* tw = bufB + M * C;
  const int i0 = blockIdx.x * C;
  const int iz = blockIdx.y;
  const int ni = min(C, NKX - i0);
  const long long cs = (long long)NY1 * NZ1 * NKX;
  load_twiddles(tw, reinterpret_cast<const CT*>(a.tw), M);
  for (int idx = threadIdx.x; idx < 3 * NY1 * C; idx += blockDim.x) {
    const int c = idx % C, s = (idx / C) % NY1, comp = idx / (C * NY1);
    double2 v = make_double2(0.0, 0.0);
    if (c < ni) v = a.u[comp * cs + ((long long)s * NZ1 + iz) * NKX + i0 + c];
    su[idx] = v;
  }
  __syncthreads();
  const double kz = a.kz[iz];
  const int nf = a.curl ? 6 : 3;
  const long long fs = (long long)M * NZ1 * NKX;
  for (int f = 0; f < nf; ++f) {
    for (int idx = threadIdx.x; idx < M * C; idx += blockDim.x) {
      const int c = idx % C, t = idx / C;
      const int s = pos_to_stored(t, NY1, M);
      double2 v = make_double2(0.0, 0.0);
      if (s >= 0 && c < ni) {
        const double2 u = su[(0 * NY1 + s) * C + c];
        const double2 vv = su[(1 * NY1 + s) * C + c];
        const double2 w = su[(2 * NY1 + s) * C + c];
        const double kx = a.kx[i0 + c], ky = a.ky[s];
        switch (f) {
          case 0: v = u; break;
          case 1: v = vv; break;
          case 2: v = w; break;
          // curl = 1j * (k x u), triply_periodic.py:122-132
          case 3: v = ci(make_double2(ky * w.x - kz * vv.x, ky * w.y - kz * vv.y)); break;
          case 4: v = ci(make_double2(kz * u.x - kx * w.x, kz * u.y - kx * w.y)); break;
          default: v = ci(make_double2(kx * vv.x - ky * u.x, kx * vv.y - ky * u.y)); break;
        }
      }
      bufA[idx] = to_c(v, (CT*)nullptr);
    }
    __syncthreads();
    const CT* res = fft_cols<ML, C, kPassThreads, CT>(bufA, bufB, a.plan, 1, tw);
    CT* out = reinterpret_cast<CT*>(a.out) + f * fs + (long long)iz * NKX + i0;
    for (int idx = threadIdx.x; idx < M * C; idx += blockDim.x) {
      const int c = idx % C, t = idx / C;
      if (c < ni) out[(long long)t * NZ1 * NKX + c] = res[idx];
    }
    __syncthreads();
  }
}

cudaError_t launch_yinv(const YInvArgs& a, cudaStream_t st) {
  dim3 grid((a.NKX + kTile - 1) / kTile, a.NZ1);
  if (a.fp32 == 2) return cudaErrorInvalidValue;  // compensated: two-stage passes only
  if (a.fp32) {
    const size_t sm = yinv_smem(a.plan.L, a.NY1, 1);
    switch (a.plan.L) {
      case 48: yinv_kernel<48, float><<<grid, kPassThreads, sm, st>>>(a); break;
      case 72: yinv_kernel<72, float><<<grid, kPassThreads, sm, st>>>(a); break;
      case 96: yinv_kernel<96, float><<<grid, kPassThreads, sm, st>>>(a); break;
      case 192: yinv_kernel<192, float><<<grid, kPassThreads, sm, st>>>(a); break;
      default: return cudaErrorInvalidValue;  // compile-time sizes only
    }
    return cudaGetLastError();
  }
  DNSB_DISPATCH_V(a.variant, a.plan.L, yinv_kernel, grid, yinv_smem(a.plan.L, a.NY1, 0), st, a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Periodic last forward pass (y) with the pressure projection fused.
// ---------------------------------------------------------------------------
// FP32 form: the input pass buffer, transform buffers and twiddles are
// FP32; the transformed rows are scaled into FP64 (snl) and the projection
// and the output RHS are FP64.
size_t yfwd_smem(int My, int NY1, int fp32) {
  const size_t cb = fp32 ? sizeof(float2) : sizeof(double2);
  return sizeof(double2) * (size_t)(3 * NY1 * kTile) + cb * (size_t)(2 * My * kTile + My);
}

template <int ML, typename T = double>
__global__ void __launch_bounds__(kPassThreads)
yfwd_kernel(YFwdArgs a) {
  using CT = typename pass_types<T>::C;
  using RT = typename pass_types<T>::R;
  extern __shared__ double2 sm[];
  const int M = ML > 0 ? ML : a.plan.L;
  const int C = kTile;
  const int NY1 = a.NY1, NZ1 = a.NZ1, NKX = a.NKX;
  double2* snl = sm;  // [3][NY1][C]
  CT* bufA = reinterpret_cast<CT*>(snl + 3 * NY1 * C);
  CT* bufB = bufA + M * C;
  CT* tw = bufB + M * C;
  const int i0 = blockIdx.x * C;
  const int iz = blockIdx.y;
  const int ni = min(C, NKX - i0);
  load_twiddles(tw, reinterpret_cast<const CT*>(a.tw), M);
  const long long fs = (long long)M * NZ1 * NKX;
  const double sc = 1.0 / M;
  for (int f = 0; f < 3; ++f) {
    const CT* in = reinterpret_cast<const CT*>(a.in) + f * fs + (long long)iz * NKX + i0;
    for (int idx = threadIdx.x; idx < M * C; idx += blockDim.x) {
      const int c = idx % C, t = idx / C;
      CT v = cmake<CT>(0, 0);
      if (c < ni) v = in[(long long)t * NZ1 * NKX + c];
      bufA[idx] = v;
    }
    __syncthreads();
    const CT* res = fft_cols<ML, C, kPassThreads, CT>(bufA, bufB, a.plan, -1, tw);
    for (int idx = threadIdx.x; idx < NY1 * C; idx += blockDim.x) {
      const int c = idx % C, s = idx / C;
      const int t = stored_to_pos(s, NY1, M);
      snl[(f * NY1 + s) * C + c] = cscale(to_d(res[t * C + c]), sc);
    }
    __syncthreads();
  }
  const long long cs = (long long)NY1 * NZ1 * NKX;
  const double kz = a.kz[iz];
  for (int idx = threadIdx.x; idx < NY1 * C; idx += blockDim.x) {
    const int c = idx % C, s = idx / C;
    if (c >= ni) continue;
    const double2 n0 = snl[(0 * NY1 + s) * C + c];
    const double2 n1 = snl[(1 * NY1 + s) * C + c];
    const double2 n2 = snl[(2 * NY1 + s) * C + c];
    const long long off = ((long long)s * NZ1 + iz) * NKX + i0 + c;
    double2 r0 = n0, r1 = n1, r2 = n2;
    if (a.project) {
      const double kx = a.kx[i0 + c], ky = a.ky[s];
      // NL - grad(inv_lapl * div NL), monochromatic.py:377-385
      const double2 div = cadd(cadd(cik(kx, n0), cik(ky, n1)), cik(kz, n2));
      const double il = a.inv_lapl[off];
      const double2 p = cscale(div, il);
      r0 = csub(n0, cik(kx, p));
      r1 = csub(n1, cik(ky, p));
      r2 = csub(n2, cik(kz, p));
    }
    a.out[off] = r0;
    a.out[cs + off] = r1;
    a.out[2 * cs + off] = r2;
  }
}

cudaError_t launch_yfwd(const YFwdArgs& a, cudaStream_t st) {
  dim3 grid((a.NKX + kTile - 1) / kTile, a.NZ1);
  if (a.fp32 == 2) return cudaErrorInvalidValue;  // compensated: two-stage passes only
  if (a.fp32) {
    const size_t sm = yfwd_smem(a.plan.L, a.NY1, 1);
    switch (a.plan.L) {
      case 48: yfwd_kernel<48, float><<<grid, kPassThreads, sm, st>>>(a); break;
      case 72: yfwd_kernel<72, float><<<grid, kPassThreads, sm, st>>>(a); break;
      case 96: yfwd_kernel<96, float><<<grid, kPassThreads, sm, st>>>(a); break;
      case 192: yfwd_kernel<192, float><<<grid, kPassThreads, sm, st>>>(a); break;
      default: return cudaErrorInvalidValue;  // compile-time sizes only
    }
    return cudaGetLastError();
  }
  DNSB_DISPATCH_V(a.variant, a.plan.L, yfwd_kernel, grid, yfwd_smem(a.plan.L, a.NY1, 0), st, a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Couette first inverse pass (z) with the FD curl fused.
// ---------------------------------------------------------------------------
size_t zinv_curl_smem(int Mz, int NZ1, int span_max) {
  (void)NZ1;
  (void)span_max;
  return sizeof(double2) * (size_t)(2 * Mz * kZTile + Mz);
}

// D1 along y of column x (complex, stride 1) at row y: sum_m w[m] x[j0 + m].
// Up to kD1Unroll taps are unrolled (predicated), so the loads of several
// rows can be in flight together; wider stencils take the plain loop.
constexpr int kD1Unroll = 9;

__device__ __forceinline__ double2 d1_row(const double2* x, const ZInvCurlArgs& a, int y) {
  const int j0 = a.d1_j0[y];
  const double* w = a.d1_wT + y;  // tap m at w[m * Ny]: consecutive y contiguous
  const int Ny = a.Ny;
  double2 d = make_double2(0.0, 0.0);
  if (a.s1 <= kD1Unroll) {
#pragma unroll
    for (int m = 0; m < kD1Unroll; ++m) {
      if (m < a.s1) {
        const double2 q = x[j0 + m];
        d.x += w[m * Ny] * q.x;
        d.y += w[m * Ny] * q.y;
      }
    }
  } else {
    for (int m = 0; m < a.s1; ++m) {
      const double2 q = x[j0 + m];
      d.x += w[m * Ny] * q.x;
      d.y += w[m * Ny] * q.y;
    }
  }
  return d;
}

// Field F of the z-inverse input at stored z mode s (column base b) and row
// y: 0 u, 1 v, 2 w, 3 dy w - dz v, 4 dz u - dx w, 5 dx v - dy u
// (plane_couette.py:251-271).
template <int F>
__device__ __forceinline__ double2 zinv_field(const ZInvCurlArgs& a, const double2* U,
                                              const double2* V, const double2* Wc,
                                              long long b, int s, int y, double kx) {
  if (F == 0) return U[b + y];
  if (F == 1) return V[b + y];
  if (F == 2) return Wc[b + y];
  const double kz = a.kz[s];
  if (F == 3) return csub(d1_row(Wc + b, a, y), cik(kz, V[b + y]));
  if (F == 4) return csub(cik(kz, U[b + y]), cik(kx, Wc[b + y]));
  return csub(cik(kx, V[b + y]), d1_row(U + b, a, y));
}

// Fill buf[t][c] with field F over the tile.  Every element of a thread is
// computed into registers before any is stored, so the global loads of all
// of a thread's elements are in flight together.
template <int M, int F>
__device__ __forceinline__ void zinv_fill(const ZInvCurlArgs& a, double2* buf,
                                          const double2* U, const double2* V,
                                          const double2* Wc, long long sstride,
                                          int y0, int y1, double kx) {
  constexpr int C = kZTile;
  constexpr int NE = (M * C + kPassThreads - 1) / kPassThreads;
  double2 v[NE];
#pragma unroll
  for (int e = 0; e < NE; ++e) {
    const int idx = threadIdx.x + e * kPassThreads;
    const int c = idx % C, t = idx / C;
    const int s = (idx < M * C) ? pos_to_stored(t, a.NZ1, M) : -1;
    const int y = y0 + c;
    v[e] = make_double2(0.0, 0.0);
    if (s >= 0 && y < y1) v[e] = zinv_field<F>(a, U, V, Wc, s * sstride, s, y, kx);
  }
#pragma unroll
  for (int e = 0; e < NE; ++e) {
    const int idx = threadIdx.x + e * kPassThreads;
    if (idx < M * C) buf[idx] = v[e];
  }
}

// Runtime-length variant of the fill (no compile-time plan).
__device__ __forceinline__ void zinv_fill_rt(const ZInvCurlArgs& a, double2* buf, int M, int f,
                                             const double2* U, const double2* V,
                                             const double2* Wc, long long sstride,
                                             int y0, int y1, double kx) {
  const int C = kZTile;
  for (int idx = threadIdx.x; idx < M * C; idx += kPassThreads) {
    const int c = idx % C, t = idx / C;
    const int s = pos_to_stored(t, a.NZ1, M);
    const int y = y0 + c;
    double2 v = make_double2(0.0, 0.0);
    if (s >= 0 && y < y1) {
      const long long b = s * sstride;
      switch (f) {
        case 0: v = zinv_field<0>(a, U, V, Wc, b, s, y, kx); break;
        case 1: v = zinv_field<1>(a, U, V, Wc, b, s, y, kx); break;
        case 2: v = zinv_field<2>(a, U, V, Wc, b, s, y, kx); break;
        case 3: v = zinv_field<3>(a, U, V, Wc, b, s, y, kx); break;
        case 4: v = zinv_field<4>(a, U, V, Wc, b, s, y, kx); break;
        default: v = zinv_field<5>(a, U, V, Wc, b, s, y, kx); break;
      }
    }
    buf[idx] = v;
  }
}

// Fills read the spectral state straight from global memory (the y-stencil
// neighbours of a tile come from L1/L2), so only the FFT buffers occupy
// shared memory and four CTAs fit per SM.
template <int ML>
__global__ void __launch_bounds__(kPassThreads)
zinv_curl_kernel(ZInvCurlArgs a, int span_max) {
  (void)span_max;
  extern __shared__ double2 sm[];
  const int M = ML > 0 ? ML : a.plan.L;
  const int C = kZTile;
  const int NZ1 = a.NZ1;
  const int NKX = a.NKX, Ny = a.Ny;
  double2* bufA = sm;
  double2* bufB = bufA + M * C;
  double2* tw = bufB + M * C;
  const int y0 = blockIdx.x * C;
  const int ix = blockIdx.y;
  const int y1 = min(y0 + C, Ny);
  const long long cs = (long long)NZ1 * NKX * Ny;
  const double2* U = a.u + (long long)ix * Ny;
  const double2* V = U + cs;
  const double2* Wc = U + 2 * cs;
  const long long sstride = (long long)NKX * Ny;
  load_twiddles(tw, a.tw, M);
  const double kx = a.kx[ix];
  const int nf = a.curl ? 6 : 3;
  const long long fs = (long long)M * NKX * Ny;
  for (int f = 0; f < nf; ++f) {
    if (ML > 0) {
      constexpr int MC = ML > 0 ? ML : 1;
      switch (f) {
        case 0: zinv_fill<MC, 0>(a, bufA, U, V, Wc, sstride, y0, y1, kx); break;
        case 1: zinv_fill<MC, 1>(a, bufA, U, V, Wc, sstride, y0, y1, kx); break;
        case 2: zinv_fill<MC, 2>(a, bufA, U, V, Wc, sstride, y0, y1, kx); break;
        case 3: zinv_fill<MC, 3>(a, bufA, U, V, Wc, sstride, y0, y1, kx); break;
        case 4: zinv_fill<MC, 4>(a, bufA, U, V, Wc, sstride, y0, y1, kx); break;
        default: zinv_fill<MC, 5>(a, bufA, U, V, Wc, sstride, y0, y1, kx); break;
      }
    } else {
      zinv_fill_rt(a, bufA, M, f, U, V, Wc, sstride, y0, y1, kx);
    }
    __syncthreads();
    const double2* res = fft_cols<ML, C, kPassThreads>(bufA, bufB, a.plan, 1, tw);
    double2* out = a.out + f * fs + (long long)ix * Ny + y0;
    for (int idx = threadIdx.x; idx < M * C; idx += kPassThreads) {
      const int c = idx % C, t = idx / C;
      if (y0 + c < y1) out[(long long)t * NKX * Ny + c] = res[idx];
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Couette z-inverse pass, two register stages (M = R1 R2, the shapes of the
// column pass): a CTA takes C consecutive (kx, y) columns -- contiguous in the
// (nz-1, nx/2, ny) layout -- fills each field's zero-padded z column into
// shared memory (all of a thread's loads of a batch in flight together), runs
// the inverse radix-R1 stage in registers, exchanges once through shared
// memory, and stores the inverse radix-R2 stage's outputs straight to global
// memory.
// ---------------------------------------------------------------------------
size_t zinv_curl2_smem(int M) { return col_pass2_smem(M); }

template <int M, int F, typename CT>
__device__ __forceinline__ void zinv2_fill(const ZInvCurlArgs& a, CT* X,
                                           const double2* U, const double2* V,
                                           const double2* Wc, long long sstride,
                                           int y, double kx, bool live) {
  constexpr int C = ColShape<M>::C, NT = ColShape<M>::NT;
  constexpr int NE = M * C / NT;  // elements per thread (= R1)
  constexpr int B = (NE % 6 == 0) ? 6 : ((NE % 3 == 0) ? 3 : 1);
  const int tid = threadIdx.x;
  for (int e0 = 0; e0 < NE; e0 += B) {
    double2 v[B];
#pragma unroll
    for (int e = 0; e < B; ++e) {
      const int t = (tid + (e0 + e) * NT) / C;
      const int s = pos_to_stored(t, a.NZ1, M);
      v[e] = make_double2(0.0, 0.0);
      if (live && s >= 0) v[e] = zinv_field<F>(a, U, V, Wc, s * sstride, s, y, kx);
    }
#pragma unroll
    for (int e = 0; e < B; ++e) X[tid + (e0 + e) * NT] = to_c(v[e], (CT*)nullptr);
  }
}

// T: the compute type and the element type of the output pass buffer
// (double, or float for the FP32 form of the Couette RHS); the state is
// read, and the curl's fill computed, in FP64.
template <int ML, typename T = double, bool SLAB = false>
__global__ void __launch_bounds__(ColShape<ML>::NT,
                                  std::is_same<T, float>::value ? 768 / ColShape<ML>::NT
                                                              : ColShape<ML>::ZB)
zinv_curl2_kernel(ZInvCurlArgs a) {
  grid_dep_sync();
  if (a.skip && *a.skip) return;
  using CT = typename pass_types<T>::C;
  using RT = typename pass_types<T>::R;
  constexpr int M = ML, R1 = ColShape<ML>::R1, R2 = ColShape<ML>::R2, C = ColShape<ML>::C;
  constexpr int NT = ColShape<ML>::NT;
  extern __shared__ double2 sm_[];
  CT* X = reinterpret_cast<CT*>(sm_);  // [t][C]
  CT* tw = X + M * C;
  const CT* gtw = reinterpret_cast<const CT*>(a.tw);
  CT* gout = reinterpret_cast<CT*>(a.out);
  const int tid = threadIdx.x;
  const int NZ1 = a.NZ1, NKX = a.NKX, Ny = a.Ny;
  const long long ncol = (long long)NKX * Ny;
  const long long q0 = (long long)(a.fields_fast ? blockIdx.y : blockIdx.x) * C;
  const int nq = (int)min((long long)C, ncol - q0);
  const long long cs = (long long)NZ1 * ncol;
  for (int i = tid; i < M; i += NT) cp_async_elem(tw + i, gtw + i);
  cp_async_commit();
  // The fill column of this thread (the same for all its elements).
  const int cf = tid % C;
  const bool live = cf < nq;
  const long long q = q0 + (live ? cf : 0);
  const int ix = (int)(q / Ny), y = (int)(q % Ny);
  const double kx = a.kx[ix];
  const double2* U = a.u + (long long)ix * Ny;
  const double2* V = U + cs;
  const double2* Wc = U + 2 * cs;
  const long long fs = (long long)M * ncol;
  // Half of the pass buffer's lines stay in L2 for the x pass that reads
  // them next (all of them would not fit beside the rest).
  const unsigned long long keep = l2_keep_half();
  const int f = a.fields_fast ? blockIdx.x : blockIdx.y;  // one field per CTA
  {
    switch (f) {
      case 0: zinv2_fill<M, 0>(a, X, U, V, Wc, ncol, y, kx, live); break;
      case 1: zinv2_fill<M, 1>(a, X, U, V, Wc, ncol, y, kx, live); break;
      case 2: zinv2_fill<M, 2>(a, X, U, V, Wc, ncol, y, kx, live); break;
      case 3: zinv2_fill<M, 3>(a, X, U, V, Wc, ncol, y, kx, live); break;
      case 4: zinv2_fill<M, 4>(a, X, U, V, Wc, ncol, y, kx, live); break;
      default: zinv2_fill<M, 5>(a, X, U, V, Wc, ncol, y, kx, live); break;
    }
    cp_async_wait_all();  // twiddles
    __syncthreads();
    // Stage 1: inverse radix R1 (Ns = 1) on positions t = j + R2 i of column c.
    {
      const int c = tid % C, j = tid / C;
      CT v[R1];
#pragma unroll
      for (int i = 0; i < R1; ++i) v[i] = X[(j + R2 * i) * C + c];
      dft_reg<R1, 1>(v);
      __syncthreads();  // every read done before the in-place writes
#pragma unroll
      for (int i = 0; i < R1; ++i) X[(j * R1 + i) * C + c] = v[i];
    }
    __syncthreads();
    // Stage 2: inverse radix R2 (Ns = R1) -> positions t = k + R1 i.
    for (int it = tid; it < R1 * C; it += NT) {
      const int c = it % C, k = it / C;
      CT z[R2];
#pragma unroll
      for (int i = 0; i < R2; ++i) z[i] = X[(k + R1 * i) * C + c];
#pragma unroll
      for (int i = 1; i < R2; ++i) {
        CT w = tw[i * k];
        w.y = -w.y;
        z[i] = cmul(z[i], w);
      }
      dft_reg<R2, 1>(z);
      if (c < nq) {
#pragma unroll
        for (int i = 0; i < R2; ++i) {
          if constexpr (SLAB) {
            // position t belongs to rank t / blk (its padded-z share)
            const int t = k + R1 * i, r = t / a.slab.blk;
            a.slab.buf[r][f * a.slab.fs + (long long)(t - r * a.slab.blk) * a.slab.ts +
                          a.slab.off + q0 + c] = to_d(z[i]);
          } else {
            st_l2(gout + f * fs + (long long)(k + R1 * i) * ncol + q0 + c, z[i], keep);
          }
        }
      }
    }
  }
}

cudaError_t launch_zinv_curl(const ZInvCurlArgs& a, int span_max,
                             cudaStream_t st) {
  const int L = a.plan.L;
  const bool slab = a.slab.buf[0] != nullptr;
  if (slab && (a.fp32 || a.variant != 0 || !fp32_length(L))) return cudaErrorInvalidValue;
  if (a.variant == 0 && two_stage_length(L)) {
    if (a.fp32 && !fp32_length(L)) return cudaErrorInvalidValue;
    const long long ncol = (long long)a.NKX * a.Ny;
    const int C = col_columns(L);
    const unsigned tiles = (unsigned)((ncol + C - 1) / C), nf = a.curl ? 6 : 3;
    const dim3 grid = a.fields_fast ? dim3(nf, tiles) : dim3(tiles, nf);
    const size_t sm = a.fp32 ? zinv_curl2_smem(L) / 2 : zinv_curl2_smem(L);
    return with_length(L, [&](auto len) {
      constexpr int LL = decltype(len)::value, NT = ColShape<LL>::NT;
      if constexpr (fp32_length(LL)) {
        if (slab) launch_dep(a.dep, zinv_curl2_kernel<LL, double, true>, grid, NT, sm, st, a);
        else if (a.fp32 == 2) launch_dep(a.dep, zinv_curl2_kernel<LL, fcomp>, grid, NT, sm, st, a);
        else if (a.fp32) launch_dep(a.dep, zinv_curl2_kernel<LL, float>, grid, NT, sm, st, a);
        if (slab || a.fp32) return cudaGetLastError();
      }
      launch_dep(a.dep, zinv_curl2_kernel<LL>, grid, NT, sm, st, a);
      return cudaGetLastError();
    });
  }
  if (a.fp32) return cudaErrorInvalidValue;  // two-stage compile-time passes only
  dim3 grid((a.Ny + kZTile - 1) / kZTile, a.NKX);
  DNSB_DISPATCH_V(a.variant, a.plan.L, zinv_curl_kernel, grid,
                  zinv_curl_smem(a.plan.L, a.NZ1, span_max), st, a, span_max);
  return cudaGetLastError();
}

// Raises the dynamic shared-memory limit of every pass kernel that needs more
// than the default 48 KB.
cudaError_t set_pass_attributes(int max_smem) {
  cudaError_t e = cudaSuccess;
  auto allow = [&](std::initializer_list<const void*> fns) {
    for (const void* f : fns) {
      const cudaError_t r = allow_dynamic_smem(f, max_smem);
      if (r != cudaSuccess) e = r;
    }
  };
#define DNSB_STOCKHAM(N)                                                               \
  {(const void*)col_pass_kernel<N>, (const void*)x_pass_kernel<N>,                     \
   (const void*)x_phys_kernel<N>, (const void*)x_fwd_kernel<N>,                        \
   (const void*)yinv_kernel<N>, (const void*)yfwd_kernel<N>, (const void*)zinv_curl_kernel<N>}
  allow(DNSB_STOCKHAM(0));
  for_each_length([&](auto len) {
    constexpr int LL = decltype(len)::value;
    if constexpr (fp32_length(LL)) {
      allow(DNSB_STOCKHAM(LL));
      if constexpr (LL > 72)
        allow({(const void*)yinv_kernel<LL, float>, (const void*)yfwd_kernel<LL, float>});
    }
    if (col_pass2_smem(LL) <= kDefaultSmem) return;
    allow({(const void*)col_pass2_held_kernel<LL, 1, true>,
           (const void*)col_pass2_held_kernel<LL, 1, false>,
           (const void*)col_pass2_held_kernel<LL, -1, false>,
           (const void*)zinv_curl2_kernel<LL>});
    if constexpr (fp32_length(LL))
      allow({(const void*)zinv_curl2_kernel<LL, double, true>,
             (const void*)col_pass2_kernel<LL, -1>,
             (const void*)col_pass2_kernel<LL, 1, double, false, false, true>});
  });
#undef DNSB_STOCKHAM
  for (cudaError_t r : {set_x_pass_attributes(max_smem), set_x_transform_attributes(max_smem),
                        set_yfwd_project_attributes(max_smem)})
    if (r != cudaSuccess) e = r;
  return e;
}

}  // namespace dnsb
