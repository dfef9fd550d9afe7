// x passes of the plain dealiased transforms (no product), in register stages:
// half spectra -> physical rows (spec_to_phys) and physical rows -> truncated
// half spectra (phys_to_spec), src/dnsjax/fft.py:140-190 and 193-408.
//
// Two real fields share one complex transform.  A CTA takes NR rows: (u, v) of
// each row, and w of two rows, fill 3 NR / 2 columns (the Stockham form paired w
// with zero, four transforms in place of three).  Stages as in the x pass of the
// RHS (csrc/x_pass.cu, M = R1 RM RB); physical values go straight from the last
// inverse stage to global memory and straight from global memory into the first
// forward one, consecutive x on consecutive lanes.
//
// Bound: memory (128 x 129 x 128 spec_to_phys moves 315 MB in this pass).
// Measured against the Stockham stages that ran before: whole 128 x 129 x 128
// spec_to_phys 160 -> 82 us, 144^3 phys_to_spec 522 -> 205 us (with its y pass
// in register stages too).
#include "passes.cuh"
#include "x_shape.cuh"

namespace dnsb {

namespace {

template <int M>
struct TLayout {
  using S = XShape<M>;
  static constexpr int NKX = M / 3, PB = M / S::RB, NR = 2 * S::R, C = 3 * S::R, NT = S::NT;
  // staged spectra [field][row][NS]: rows or modes fastest without conflicts
  static constexpr int NS = NR == 8 ? (NKX | 1) : NKX + ((2 - NKX % 8) + 8) % 8;
  // stage-A output [column][XS] with a skew of SK per block of R1 positions,
  // so that consecutive j fall on other banks
  static constexpr int SK = S::R1 % 2 == 0 ? 1 : 0, XS = M + SK * (M / S::R1);
  static constexpr int SZ_S = 3 * NR * NS, SZ_X = C * XS, SZ_I = SZ_S > SZ_X ? SZ_S : SZ_X;
  // forward: stage-1 output [column][i][PK], final spectra [column][FS]
  static constexpr int PK = PB | 1, YS = S::RB * PK, FS = M | 1;
  static constexpr int SZ_F = C * (YS > FS ? YS : FS);
  static constexpr size_t inv_bytes = sizeof(double2) * (size_t)(SZ_I + M);
  static constexpr size_t fwd_bytes = sizeof(double2) * (size_t)(SZ_F + M);
};

// Rows of a column's two fields: column < NR is (u, v) of row `column`, the
// others w of rows 2 (column - NR) and the next.
struct ColumnRows {
  int fa, ra, fb, rb;
};
template <int NR>
__device__ __forceinline__ ColumnRows column_rows(int col) {
  if (col < NR) return {0, col, 1, col};
  return {2, 2 * (col - NR), 2, 2 * (col - NR) + 1};
}

template <int NR>
__device__ __forceinline__ int row_offsets(const XPhysArgs& a, long long* s_spec,
                                           long long* s_phys) {
  const int r0 = blockIdx.x * NR;
  if (threadIdx.x < NR) {
    const int row = r0 + threadIdx.x;
    const long long outer = row / a.inner_n, inner = row % a.inner_n;
    s_spec[threadIdx.x] = outer * a.so + inner * a.si;
    s_phys[threadIdx.x] = outer * a.pso + inner * a.psi;
  }
  return min(NR, a.nrows - r0);
}

template <int ML>
__global__ void __launch_bounds__(XShape<ML>::NT)
x_phys2_kernel(XPhysArgs a) {
  using SH = XShape<ML>;
  using LY = TLayout<ML>;
  constexpr int M = ML, R1 = SH::R1, RM = SH::RM, RB = SH::RB, NT = SH::NT;
  constexpr int NKX = LY::NKX, PB = LY::PB, NR = LY::NR, C = LY::C, NS = LY::NS;
  constexpr int XS = LY::XS, SK = LY::SK;
  extern __shared__ double2 sm[];
  double2* tw = sm + LY::SZ_I;
  __shared__ long long s_spec[NR], s_phys[NR];
  const int tid = threadIdx.x;
  const int nr = row_offsets<NR>(a, s_spec, s_phys);
  for (int i = tid; i < M; i += NT) cp_async16(tw + i, a.tw + i);
  __syncthreads();
  const unsigned long long drop = l2_drop();
  for (int idx = tid; idx < 3 * NKX * NR; idx += NT) {
    int r, k, f;
    if (a.rows_fast) {
      r = idx % NR;
      k = (idx / NR) % NKX;
    } else {
      k = idx % NKX;
      r = (idx / NKX) % NR;
    }
    f = idx / (NR * NKX);
    double2* dst = sm + (f * NR + r) * NS + k;
    if (r < nr) cp_async16_l2(dst, a.in + f * a.in_fs + s_spec[r] + k * a.ks, drop);
    else *dst = make_double2(0.0, 0.0);
  }
  cp_async_commit();
  cp_async_wait_all();
  __syncthreads();
  {  // Stage A
    constexpr int NJ = M / R1, TOT = NJ * C, Q = (TOT + NT - 1) / NT;
    double2 v[Q][R1];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int it = tid + q * NT, j = it % NJ;
      if (TOT % NT == 0 || it < TOT) {
        const ColumnRows cr = column_rows<NR>(it / NJ);
        const double2* A = sm + (cr.fa * NR + cr.ra) * NS;
        const double2* B = sm + (cr.fb * NR + cr.rb) * NS;
#pragma unroll
        for (int i = 0; i < R1; ++i) {
          const int t = j + NJ * i;
          double2 z = make_double2(0.0, 0.0);
          if (t == 0) {
            z = make_double2(A[0].x, B[0].x);
          } else if (t < NKX) {
            z = make_double2(A[t].x - B[t].y, A[t].y + B[t].x);
          } else if (M - t < NKX) {
            const double2 av = A[M - t], bv = B[M - t];
            z = make_double2(av.x + bv.y, -av.y + bv.x);
          }
          v[q][i] = z;
        }
      }
    }
    __syncthreads();  // the spectra are read before they are overwritten
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int it = tid + q * NT, j = it % NJ;
      if (TOT % NT == 0 || it < TOT) {
        dft_reg<R1, 1>(v[q], middle_third(R1));
        double2* X = sm + (it / NJ) * XS + j * (R1 + SK);
#pragma unroll
        for (int i = 0; i < R1; ++i) X[i] = v[q][i];
      }
    }
  }
  __syncthreads();
  if constexpr (RM > 1) {  // Stage A'
    constexpr int NJ = M / RM, TOT = NJ * C, Q = (TOT + NT - 1) / NT;
    double2 v[Q][RM];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int it = tid + q * NT, j = it % NJ;
      if (TOT % NT == 0 || it < TOT) {
        const double2* X = sm + (it / NJ) * XS + j + SK * (j / R1);
#pragma unroll
        for (int i = 0; i < RM; ++i) v[q][i] = X[(NJ + SK * (NJ / R1)) * i];
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int it = tid + q * NT, j = it % NJ, k = j % R1;
      if (TOT % NT == 0 || it < TOT) {
#pragma unroll
        for (int i = 1; i < RM; ++i) {
          double2 w = tw[i * k * RB];
          w.y = -w.y;
          v[q][i] = cmul(v[q][i], w);
        }
        dft_reg<RM, 1>(v[q]);
        double2* X = sm + (it / NJ) * XS + (j / R1) * PB + k;
#pragma unroll
        for (int i = 0; i < RM; ++i) X[i * R1] = v[q][i];
      }
    }
    __syncthreads();
  }
  // Stage B: physical values at t = k + PB i, straight out.
  constexpr int XB = RM > 1 ? 0 : SK;
  for (int it = tid; it < PB * C; it += NT) {
    const int col = it / PB, k = it % PB;
    const double2* X = sm + col * XS + k;
    double2 z[RB];
#pragma unroll
    for (int i = 0; i < RB; ++i) z[i] = X[(PB + XB) * i];
#pragma unroll
    for (int i = 1; i < RB; ++i) {
      double2 w = tw[i * k];
      w.y = -w.y;
      z[i] = cmul(z[i], w);
    }
    dft_reg<RB, 1>(z);
    const ColumnRows cr = column_rows<NR>(col);
    double* pa = a.out + cr.fa * a.out_fs + s_phys[cr.ra] + k;
    double* pb = a.out + cr.fb * a.out_fs + s_phys[cr.rb] + k;
    const bool la = cr.ra < nr, lb = cr.rb < nr;
#pragma unroll
    for (int i = 0; i < RB; ++i) {
      if (la) pa[PB * i] = z[i].x;
      if (lb) pb[PB * i] = z[i].y;
    }
  }
}

template <int ML>
__global__ void __launch_bounds__(XShape<ML>::NT)
x_fwd2_kernel(XPhysArgs a, const double* __restrict__ phys, double2* __restrict__ spec) {
  using SH = XShape<ML>;
  using LY = TLayout<ML>;
  constexpr int M = ML, R1 = SH::R1, RM = SH::RM, RB = SH::RB, NT = SH::NT;
  constexpr int NKX = LY::NKX, PB = LY::PB, NR = LY::NR, C = LY::C;
  constexpr int PK = LY::PK, YS = LY::YS, FS = LY::FS;
  extern __shared__ double2 sm[];
  double2* tw = sm + LY::SZ_F;
  __shared__ long long s_spec[NR], s_phys[NR];
  const int tid = threadIdx.x;
  const int nr = row_offsets<NR>(a, s_spec, s_phys);
  for (int i = tid; i < M; i += NT) cp_async16(tw + i, a.tw + i);
  cp_async_commit();
  cp_async_wait_all();
  __syncthreads();
  // Stage B: radix RB over t = k + PB i, twiddles exp(-2 pi i i k / M).
  for (int it = tid; it < PB * C; it += NT) {
    const int col = it / PB, k = it % PB;
    const ColumnRows cr = column_rows<NR>(col);
    const double* pa = phys + cr.fa * a.out_fs + s_phys[cr.ra] + k;
    const double* pb = phys + cr.fb * a.out_fs + s_phys[cr.rb] + k;
    const bool la = cr.ra < nr, lb = cr.rb < nr;
    double2 z[RB];
#pragma unroll
    for (int i = 0; i < RB; ++i)
      z[i] = make_double2(la ? pa[PB * i] : 0.0, lb ? pb[PB * i] : 0.0);
    dft_reg<RB, -1>(z);
    double2* Y = sm + col * YS + k;
    Y[0] = z[0];
#pragma unroll
    for (int i = 1; i < RB; ++i) Y[i * PK] = cmul(z[i], tw[i * k]);
  }
  __syncthreads();
  if constexpr (RM > 1) {
    // Stage C': radix RM over k = k1 + R1 m; an item writes where it read.
    constexpr int TOT = R1 * RB * C;
    for (int it = tid; it < TOT; it += NT) {
      const int k1 = it % R1, i = (it / R1) % RB;
      double2* Y = sm + (it / (R1 * RB)) * YS + i * PK + k1;
      double2 v[RM];
#pragma unroll
      for (int m = 0; m < RM; ++m) v[m] = Y[R1 * m];
      dft_reg<RM, -1>(v);
#pragma unroll
      for (int m = 1; m < RM; ++m) v[m] = cmul(v[m], tw[m * k1 * RB]);
#pragma unroll
      for (int m = 0; m < RM; ++m) Y[R1 * m] = v[m];
    }
    __syncthreads();
  }
  {  // Stage C: radix R1, natural order, the truncated third dropped
    constexpr int TOT = RM * RB * C, Q = (TOT + NT - 1) / NT;
    double2 v[Q][R1];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int it = tid + q * NT, i = it % RB, m = (it / RB) % RM;
      if (TOT % NT == 0 || it < TOT) {
        const double2* Y = sm + (it / (RB * RM)) * YS + i * PK + m * R1;
#pragma unroll
        for (int n = 0; n < R1; ++n) v[q][n] = Y[n];
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int it = tid + q * NT, i = it % RB, m = (it / RB) % RM;
      if (TOT % NT == 0 || it < TOT) {
        dft_reg<R1, -1>(v[q]);
        double2* X = sm + (it / (RB * RM)) * FS + i + RB * m;
#pragma unroll
        for (int n = 0; n < R1; ++n) {
          constexpr int step = RB * RM;
          if (step * n >= NKX && step * n + step - 1 <= M - NKX) continue;
          X[step * n] = v[q][n];
        }
      }
    }
  }
  __syncthreads();
  // Unpack the two real fields of each column, scale 1/M, store.
  const double h = 0.5 / M;
  for (int idx = tid; idx < NKX * C; idx += NT) {
    const int col = a.rows_fast ? idx % C : idx / NKX;
    const int k = a.rows_fast ? idx / C : idx % NKX;
    const ColumnRows cr = column_rows<NR>(col);
    const double2 Z = sm[col * FS + k], Zm = sm[col * FS + (M - k) % M];
    if (cr.ra < nr)
      spec[cr.fa * a.in_fs + s_spec[cr.ra] + k * a.ks] =
          make_double2((Z.x + Zm.x) * h, (Z.y - Zm.y) * h);
    if (cr.rb < nr)
      spec[cr.fb * a.in_fs + s_spec[cr.rb] + k * a.ks] =
          make_double2((Z.y + Zm.y) * h, (Zm.x - Z.x) * h);
  }
}

}  // namespace

cudaError_t launch_x_phys2(const XPhysArgs& a, cudaStream_t st) {
  return with_length(a.plan.L, [&](auto len) {
    using LY = TLayout<decltype(len)::value>;
    const dim3 grid((a.nrows + LY::NR - 1) / LY::NR);
    x_phys2_kernel<decltype(len)::value><<<grid, LY::NT, LY::inv_bytes, st>>>(a);
    return cudaGetLastError();
  });
}

cudaError_t launch_x_fwd2(const XPhysArgs& a, const double* phys, double2* spec,
                          cudaStream_t st) {
  return with_length(a.plan.L, [&](auto len) {
    using LY = TLayout<decltype(len)::value>;
    const dim3 grid((a.nrows + LY::NR - 1) / LY::NR);
    x_fwd2_kernel<decltype(len)::value><<<grid, LY::NT, LY::fwd_bytes, st>>>(a, phys, spec);
    return cudaGetLastError();
  });
}

cudaError_t set_x_transform_attributes(int max_smem) {
  cudaError_t e = cudaSuccess;
  for_each_length([&](auto len) {
    constexpr int LL = decltype(len)::value;
    using LY = TLayout<LL>;
    if (LY::inv_bytes > kDefaultSmem) {
      const cudaError_t r = allow_dynamic_smem((const void*)x_phys2_kernel<LL>, max_smem);
      if (r != cudaSuccess) e = r;
    }
    if (LY::fwd_bytes > kDefaultSmem) {
      const cudaError_t r = allow_dynamic_smem((const void*)x_fwd2_kernel<LL>, max_smem);
      if (r != cudaSuccess) e = r;
    }
  });
  return e;
}

}  // namespace dnsb
