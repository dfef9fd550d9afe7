// x pass of the dealiased RHS with the rotational product, in register stages.
//
// Two real fields share one complex transform (z = a + i b).  M = R1 RM RB:
//   A   inverse radix R1 (Ns = 1) straight from the staged half spectra
//   A'  inverse radix RM (Ns = R1), only where RM > 1
//   B   inverse radix RB: a thread holds the physical values at k + PB i
//       (PB = M / RB) of its row's three pairs; the product there
//       (src/dnsjax/rhs.py:77-90); the forward radix-RB DFT over the same i and
//       its twiddles exp(-2 pi i i k / M) -- the conjugates of the inverse
//       twiddles the thread has just used, so the forward stages after it read
//       no twiddle table of length M
//   C'  forward radix RM over k = k1 + R1 m, twiddles of length PB (RM > 1)
//   C   forward radix R1, the outputs of kept modes only
// and the real-field unpack with truncation (src/dnsjax/fft.py:140-190).
//
// One work region holds, in turn, the staged half spectra and every stage's
// output: each stage reads its input into registers, waits for every thread,
// then writes its output over it.
//
// Bound (128^3 Kolmogorov, M = 192, 132 us cold): latency.  Nothing is saturated at
// the 15 warps per SM that 128 registers leave: shared-memory data pipe 56% busy, FP64
// pipe 40%, issue slots 44%, DRAM 24% (the 340 MB it moves would take 51 us); a warp
// waits on shared-memory loads, fixed latencies and barriers alike.  FP32 (8 CTAs per
// SM, 85 us): shared memory 67%, issue 69%.
// Twiddles applied where they are already at hand (they had cost stage C 23
// loads a thread beside its 24 values), the zero-padded third left out of the
// inverse DFTs and the truncated third out of the forward ones, the third
// component's spectrum kept as that of a real field: 144 -> 134 us a pass (RHS
// 367 -> 356 us; FP32 243 -> 228 us).  At the lengths beyond 48, 72, 96 and 192
// the pass ran Stockham stages: 256^3 (M = 384) 5.79 -> 1.3 ms.
#include "passes.cuh"
#include "x_shape.cuh"

namespace dnsb {

namespace {

// Shared-memory layouts, free of bank conflicts for 16-byte (FP64, 8 lanes per
// 128-byte wavefront) and 8-byte (FP32, 16 lanes) elements:
//  * the stage-A output carries a skew of XS slots per block of R1 positions,
//    so that consecutive j of one pair's rows fall on other banks;
//  * the stage-B output of block k, entry (i, column), lives in blocks of YB
//    slots (a multiple of 16, so the banks depend on the skew alone);
//  * row t of the final spectra starts at slot XR t, which the unpack reads
//    without conflicts, rows or modes fastest.
template <int M>
struct XLayout {
  using S = XShape<M>;
  static constexpr int NKX = M / 3, PB = M / S::RB;
  static constexpr int CI = 3 * S::R, CF = 2 * S::R;
  static constexpr int XS = (((S::R == 4 ? 4 : 6) - CI * S::R1) % 8 + 8) % 8;
  static constexpr int YB = (S::RB * CF + 16) & ~15;
  static constexpr int XR = CF + 1;
  static constexpr int SZ_S = 6 * NKX * S::R, SZ_Y = PB * YB, SZ_X = M * CI + XS * (M / S::R1);
  static constexpr int SZ_SY = SZ_S > SZ_Y ? SZ_S : SZ_Y;
  static constexpr int SZ = SZ_SY > SZ_X ? SZ_SY : SZ_X;
  static_assert(XR * M <= SZ, "the final spectra fit the work region");
  static_assert(S::R == 2 || S::R == 4, "lane maps");
  static_assert(YB >= S::RB * CF + (S::R == 4 ? 9 : 5), "stage-B blocks hold their skew");
  static_assert(PB * S::R <= S::NT, "one stage-B item per thread");
  static constexpr size_t bytes = sizeof(double2) * (size_t)(SZ + M);
};
template <int R>
__device__ __forceinline__ int y_skew(int k) {
  return (k & 1) + (R == 4 ? 8 : 4) * ((k >> 1) & 1);
}

// Forward DFT of 8 real values (re[i]): half the operations of the complex one.
template <typename C, typename T>
__device__ __forceinline__ void dft8_real(const T* re, C* g) {
  const T h = (T)0.70710678118654752440;
  const T a0 = re[0] + re[4], a1 = re[0] - re[4], a2 = re[2] + re[6], a3 = re[2] - re[6];
  const T b0 = re[1] + re[5], b1 = re[1] - re[5], b2 = re[3] + re[7], b3 = re[3] - re[7];
  const T e0 = a0 + a2, o0 = b0 + b2, p = b1 - b3, q = b1 + b3;
  g[0] = cmake<C>(e0 + o0, 0);
  g[4] = cmake<C>(e0 - o0, 0);
  g[2] = cmake<C>(a0 - a2, b2 - b0);
  g[6] = cmake<C>(a0 - a2, b0 - b2);
  g[1] = cmake<C>(a1 + h * p, -(a3 + h * q));
  g[7] = cmake<C>(a1 + h * p, a3 + h * q);
  g[3] = cmake<C>(a1 - h * p, a3 - h * q);
  g[5] = cmake<C>(a1 - h * p, h * q - a3);
}

// A shared-memory load that is not merged with an earlier one of the address.
__device__ __forceinline__ double2 ld_shared_again(const double2* p) {
  double2 v;
  asm volatile("ld.volatile.shared.v2.f64 {%0, %1}, [%2];\n"
               : "=d"(v.x), "=d"(v.y)
               : "r"((unsigned)__cvta_generic_to_shared(p)));
  return v;
}
__device__ __forceinline__ float2 ld_shared_again(const float2* p) {
  float2 v;
  asm volatile("ld.volatile.shared.v2.f32 {%0, %1}, [%2];\n"
               : "=f"(v.x), "=f"(v.y)
               : "r"((unsigned)__cvta_generic_to_shared(p)));
  return v;
}

// T: the compute type and the element type of the pass buffer (double, float
// for the FP32 forms, fcomp with compensated butterflies).
template <int ML, typename T, bool SLAB = false>
__device__ __forceinline__ void x_pass2_body(const XPassArgs& a, int bx) {
  using CT = typename pass_types<T>::C;
  using RT = typename pass_types<T>::R;
  using SH = XShape<ML>;
  using LY = XLayout<ML>;
  constexpr int M = ML, R1 = SH::R1, RM = SH::RM, RB = SH::RB, R = SH::R, NT = SH::NT;
  constexpr int NKX = LY::NKX, PB = LY::PB, CI = LY::CI, CF = LY::CF, XS = LY::XS, YB = LY::YB;
  // FP32 rows unpacked rows fastest: slots of CF measured 1% faster; the
  // mapping is fixed per launch
  const int xr = (sizeof(CT) == 16 || !a.rows_fast) ? LY::XR : CF;
  extern __shared__ double2 sm_[];
  CT* sm = reinterpret_cast<CT*>(sm_);  // the work region
  CT* tw = sm + LY::SZ;
  const CT* gin = reinterpret_cast<const CT*>(a.in);
  const CT* gtw = reinterpret_cast<const CT*>(a.tw);
  CT* gout = reinterpret_cast<CT*>(a.out);
  const int tid = threadIdx.x;
  const int r0 = bx * R;
  const int nr = min(R, a.nrows - r0);
  __shared__ long long s_off[R];
  __shared__ long long s_doff[R];  // SLAB: the row in the destination layout
  __shared__ int s_y[R];
  if (tid < R) {
    const int row = r0 + tid;
    const int outer = row / a.inner_n, inner = row % a.inner_n;
    s_off[tid] = (long long)outer * a.so + (long long)inner * a.si;
    s_y[tid] = a.y_outer ? outer : inner;
    if (SLAB)
      s_doff[tid] = (long long)(outer + a.slab.oo) * a.slab.so +
                    (long long)(inner + a.slab.io) * a.slab.si;
  }
  for (int i = tid; i < M; i += NT) cp_async_elem(tw + i, gtw + i);
  __syncthreads();
  // The input's last use (evict_first); the output is the next pass's input
  // (evict_last).
  const unsigned long long drop = l2_drop(), keep = l2_keep();
  // Staged half spectra, S[(f * NKX + k) * R + r].
  for (int idx = tid; idx < 6 * NKX * R; idx += NT) {
    int r, k, f;
    if (a.rows_fast) {
      r = idx % R;
      k = (idx / R) % NKX;
      f = idx / (R * NKX);
    } else {
      k = idx % NKX;
      r = (idx / NKX) % R;
      f = idx / (R * NKX);
    }
    CT* dst = sm + (f * NKX + k) * R + r;
    if (r < nr) cp_async_elem_l2(dst, gin + f * a.in_fs + s_off[r] + k * a.ks, drop);
    else *dst = cmake<CT>(0, 0);
  }
  cp_async_commit();
  cp_async_wait_all();
  __syncthreads();
  // Stage A on Z = A + iB, built on the fly; positions t = j + (M / R1) i.
  {
    constexpr int NJ = M / R1, TOT = NJ * CI, Q = (TOT + NT - 1) / NT;
    // lanes: rows fastest, then JL values of j of one pair
    constexpr int JL = NJ % 4 == 0 && (R == 2 || (R1 * CI + XS) % 16 != 0) ? 4 : 2;
    CT v[Q][R1];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int it = tid + q * NT;
      const int r = it % R, rest = it / (R * JL);
      const int pr = rest % 3, j = (it / R) % JL + JL * (rest / 3);
      if (TOT % NT == 0 || it < TOT) {
        const CT* A = sm + (2 * pr) * NKX * R + r;
        const CT* B = sm + (2 * pr + 1) * NKX * R + r;
#pragma unroll
        for (int i = 0; i < R1; ++i) {
          const int t = j + NJ * i;
          CT z = cmake<CT>(0, 0);
          if (t == 0) {
            z = cmake<CT>(A[0].x, B[0].x);
          } else if (t < NKX) {
            const CT av = A[t * R], bv = B[t * R];
            z = cmake<CT>(av.x - bv.y, av.y + bv.x);
          } else if (M - t < NKX) {
            const CT av = A[(M - t) * R], bv = B[(M - t) * R];
            z = cmake<CT>(av.x + bv.y, -av.y + bv.x);
          }
          v[q][i] = z;
        }
      }
    }
    __syncthreads();  // the spectra are read by every thread before they are overwritten
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int it = tid + q * NT;
      const int r = it % R, rest = it / (R * JL);
      const int pr = rest % 3, j = (it / R) % JL + JL * (rest / 3);
      if (TOT % NT == 0 || it < TOT) {
        dft_reg<R1, 1>(v[q], middle_third(R1));
#pragma unroll
        for (int i = 0; i < R1; ++i) sm[(j * R1 + i) * CI + 3 * r + pr + XS * j] = v[q][i];
      }
    }
  }
  __syncthreads();
  if constexpr (RM > 1) {  // Stage A'
    constexpr int NJ = M / RM, TOT = NJ * CI, Q = (TOT + NT - 1) / NT;
    static_assert(NJ % R1 == 0, "stage-A' inputs fall on whole stage-A blocks");
    CT v[Q][RM];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int it = tid + q * NT;
      const int r = it % R, j = (it / R) % NJ, pr = it / (R * NJ);
      if (TOT % NT == 0 || it < TOT) {
#pragma unroll
        for (int i = 0; i < RM; ++i)
          v[q][i] = sm[(j + NJ * i) * CI + 3 * r + pr + XS * (j / R1 + (NJ / R1) * i)];
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int it = tid + q * NT;
      const int r = it % R, j = (it / R) % NJ, pr = it / (R * NJ);
      if (TOT % NT == 0 || it < TOT) {
        const int k = j % R1;
#pragma unroll
        for (int i = 1; i < RM; ++i) {
          CT w = tw[i * k * RB];
          w.y = -w.y;
          v[q][i] = cmul(v[q][i], w);
        }
        dft_reg<RM, 1>(v[q]);
        const int base = (j / R1) * PB + k;
#pragma unroll
        for (int i = 0; i < RM; ++i) sm[(base + i * R1) * CI + 3 * r + pr] = v[q][i];
      }
    }
    __syncthreads();
  }
  // Stage B: physical values at t = k + PB i, the product, the forward DFT.
  {
    constexpr int XB = RM > 1 ? 0 : XS;  // the stage-A skew, gone after A'
    const bool act = tid < PB * R;
    const int r = tid % R, k = tid / R;
    CT F0[RB], F1[RB];
    if (act) {
      CT z[3][RB];
#pragma unroll
      for (int pr = 0; pr < 3; ++pr) {
#pragma unroll
        for (int i = 0; i < RB; ++i) z[pr][i] = sm[(k + PB * i) * CI + 3 * r + pr + XB * i];
#pragma unroll
        for (int i = 1; i < RB; ++i) {
          CT w = tw[i * k];
          w.y = -w.y;
          z[pr][i] = cmul(z[pr][i], w);
        }
        dft_reg<RB, 1>(z[pr]);
      }
      const bool live = r < nr;
      const int y = s_y[r];
      const int ny = a.ny_grid;
      const RT U0 = live ? (RT)a.U[y] : RT(0), U1 = live ? (RT)a.U[ny + y] : RT(0),
              U2 = live ? (RT)a.U[2 * ny + y] : RT(0);
      const RT C0 = live ? (RT)a.cU[y] : RT(0), C1 = live ? (RT)a.cU[ny + y] : RT(0),
              C2 = live ? (RT)a.cU[2 * ny + y] : RT(0);
      const RT N0 = live ? (RT)a.nU[y] : RT(0), N1 = live ? (RT)a.nU[ny + y] : RT(0),
              N2 = live ? (RT)a.nU[2 * ny + y] : RT(0);
      RT third[RB];
#pragma unroll
      for (int i = 0; i < RB; ++i) {
        const RT u0 = z[0][i].x, u1 = z[0][i].y, u2 = z[1][i].x;
        const RT w0 = z[1][i].y, w1 = z[2][i].x, w2 = z[2][i].y;
        const RT n0 = u1 * w2 - u2 * w1;
        const RT n1 = u2 * w0 - u0 * w2;
        const RT n2 = u0 * w1 - u1 * w0;
        const RT b0 = (u1 * C2 - u2 * C1) + (U1 * w2 - U2 * w1) + N0;
        const RT b1 = (u2 * C0 - u0 * C2) + (U2 * w0 - U0 * w2) + N1;
        const RT b2 = (u0 * C1 - u1 * C0) + (U0 * w1 - U1 * w0) + N2;
        F0[i] = live ? cmake<CT>(n0 + b0, n1 + b1) : cmake<CT>(0, 0);
        third[i] = live ? n2 + b2 : RT(0);
      }
      dft_reg<RB, -1>(F0);
      if constexpr (RB == 8 && !std::is_same<T, fcomp>::value) {
        dft8_real(third, F1);
      } else {
#pragma unroll
        for (int i = 0; i < RB; ++i) F1[i] = cmake<CT>(third[i], 0);
        dft_reg<RB, -1>(F1);
      }
#pragma unroll
      for (int i = 1; i < RB; ++i) {
        // read again: held across the product, the twiddles spill
        const CT w = CT(ld_shared_again(tw + i * k));
        F0[i] = cmul(F0[i], w);
        F1[i] = cmul(F1[i], w);
      }
    }
    __syncthreads();  // every value read before the region is written over
    if (act) {
      CT* yk = sm + k * YB + y_skew<R>(k);
#pragma unroll
      for (int i = 0; i < RB; ++i) {
        yk[i * CF + 2 * r] = F0[i];
        yk[i * CF + 2 * r + 1] = F1[i];
      }
    }
  }
  __syncthreads();
  if constexpr (RM > 1) {  // Stage C': blocks k = k1 + R1 m of entry (i, column)
    constexpr int TOT = R1 * RB * CF, Q = (TOT + NT - 1) / NT;
    CT v[Q][RM];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int it = tid + q * NT;
      const int e = it % (RB * CF), k1 = it / (RB * CF);
      if (TOT % NT == 0 || it < TOT) {
#pragma unroll
        for (int m = 0; m < RM; ++m) {
          const int k = k1 + R1 * m;
          v[q][m] = sm[k * YB + y_skew<R>(k) + e];
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int it = tid + q * NT;
      const int e = it % (RB * CF), k1 = it / (RB * CF);
      if (TOT % NT == 0 || it < TOT) {
        dft_reg<RM, -1>(v[q]);
#pragma unroll
        for (int m = 1; m < RM; ++m) v[q][m] = cmul(v[q][m], tw[m * k1 * RB]);
#pragma unroll
        for (int m = 0; m < RM; ++m) sm[(m * R1 + k1) * RB * CF + e] = v[q][m];
      }
    }
    __syncthreads();
  }
  // Stage C: forward radix R1, positions j + RB (m + RM i) in natural order;
  // those of no kept mode (the middle third) are dropped.
  {
    constexpr int TOT = RM * RB * CF, Q = (TOT + NT - 1) / NT;
    CT v[Q][R1];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int it = tid + q * NT;
      const int e = it % (RB * CF), m = it / (RB * CF);  // e = entry j, column
      if (TOT % NT == 0 || it < TOT) {
#pragma unroll
        for (int i = 0; i < R1; ++i)
          v[q][i] = RM > 1 ? sm[(m * R1 + i) * RB * CF + e] : sm[i * YB + y_skew<R>(i) + e];
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int it = tid + q * NT;
      const int e = it % (RB * CF), m = it / (RB * CF);
      if (TOT % NT == 0 || it < TOT) {
        const int col = e % CF, j = e / CF;
        dft_reg<R1, -1>(v[q]);
#pragma unroll
        for (int i = 0; i < R1; ++i) {
          constexpr int step = RB * RM;
          if (step * i >= NKX && step * i + step - 1 <= M - NKX) continue;
          sm[xr * (j + RB * m + step * i) + col] = v[q][i];
        }
      }
    }
  }
  __syncthreads();
  // Unpack the real-field spectra, truncate to NKX, scale 1/M, store: the
  // first two components from the packed pair (Z, Z of -k), the third, whose
  // partner is zero, from its own spectrum.
  const RT h = (RT)0.5 / M;
  for (int idx = tid; idx < NKX * R; idx += NT) {
    const int r = a.rows_fast ? idx % R : idx / NKX;
    const int k = a.rows_fast ? idx / R : idx % NKX;
    if (r >= nr) continue;
    const CT Z = sm[xr * k + 2 * r];
    const CT Zm = sm[xr * ((M - k) % M) + 2 * r];
    const CT W = sm[xr * k + 2 * r + 1];
    const CT v0 = cmake<CT>((Z.x + Zm.x) * h, (Z.y - Zm.y) * h);
    const CT v1 = cmake<CT>((Z.y + Zm.y) * h, (Zm.x - Z.x) * h);
    const CT v2 = cmake<CT>(W.x * (2 * h), W.y * (2 * h));
    if constexpr (SLAB) {
      // mode k belongs to rank k / blk (its kx share)
      const int q = k / a.slab.blk;
      double2* d = a.slab.buf[q] + s_doff[r] + (k - q * a.slab.blk) * a.slab.ks;
      d[0] = to_d(v0);
      d[a.slab.fs] = to_d(v1);
      d[2 * a.slab.fs] = to_d(v2);
    } else {
      CT* d = gout + s_off[r] + k * a.ks;
      st_l2(d, v0, keep);
      st_l2(d + a.out_fs, v1, keep);
      st_l2(d + 2 * a.out_fs, v2, keep);
    }
  }
}

template <int ML, typename T = double, bool SLAB = false>
__global__ void __launch_bounds__(XShape<ML>::NT,
                                  std::is_same<T, float>::value ? 8 : XShape<ML>::MINB)
x_pass2_kernel(XPassArgs a) {
  grid_dep_sync();
  if (a.skip && *a.skip) return;
  x_pass2_body<ML, T, SLAB>(a, blockIdx.x);
}

// Work-list form for ensembles (csrc/capi.cu, dnsb_ensemble_*): one launch runs
// the x pass of every member.  Item k covers the member's blocks base_k ..
// base_k + blocks_k - 1; every CTA walks the virtual blocks blockIdx.x,
// blockIdx.x + gridDim.x, ... and runs the member's body on its block, so each
// member computes exactly what its own launch computes.  Members whose
// `active` flag is 0 are skipped.
static_assert(XShape<48>::NT == kEnsXThreads && XShape<72>::NT == kEnsXThreads &&
                  XShape<96>::NT == kEnsXThreads && XShape<192>::NT == kEnsXThreads,
              "one CTA shape for every member");
__global__ void __launch_bounds__(kEnsXThreads)
ens_x_pass2_kernel(const EnsXItem* __restrict__ items, const int* __restrict__ base, int n,
                   int total, const int* __restrict__ active) {
  __shared__ int s_k;
  for (int vb = blockIdx.x; vb < total; vb += gridDim.x) {
    if (threadIdx.x == 0) s_k = ens_find(base, n, vb);
    __syncthreads();
    const int k = s_k;
    const int m = items[k].member;
    if (!active || active[m]) {
      const XPassArgs a = items[k].a;
      const int bx = vb - base[k];
      switch (a.plan.L) {
        case 48: x_pass2_body<48, double>(a, bx); break;
        case 72: x_pass2_body<72, double>(a, bx); break;
        case 96: x_pass2_body<96, double>(a, bx); break;
        default: x_pass2_body<192, double>(a, bx); break;
      }
    }
    __syncthreads();
  }
}

}  // namespace

cudaError_t launch_x_pass2(const XPassArgs& a, cudaStream_t st) {
  const bool slab = a.slab.buf[0] != nullptr;
  if ((a.fp32 || slab) && !fp32_length(a.plan.L)) return cudaErrorInvalidValue;
  return with_length(a.plan.L, [&](auto len) {
    constexpr int LL = decltype(len)::value;
    constexpr int R = XShape<LL>::R, NT = XShape<LL>::NT;
    const dim3 grid((a.nrows + R - 1) / R);
    const size_t sm = a.fp32 ? XLayout<LL>::bytes / 2 : XLayout<LL>::bytes;
    if constexpr (fp32_length(LL)) {
      if (slab) launch_dep(a.dep, x_pass2_kernel<LL, double, true>, grid, NT, sm, st, a);
      else if (a.fp32 == 2) launch_dep(a.dep, x_pass2_kernel<LL, fcomp>, grid, NT, sm, st, a);
      else if (a.fp32) launch_dep(a.dep, x_pass2_kernel<LL, float>, grid, NT, sm, st, a);
      if (slab || a.fp32) return cudaGetLastError();
    }
    launch_dep(a.dep, x_pass2_kernel<LL>, grid, NT, sm, st, a);
    return cudaGetLastError();
  });
}

cudaError_t set_x_pass_attributes(int max_smem) {
  cudaError_t e = cudaSuccess;
  for_each_length([&](auto len) {
    constexpr int LL = decltype(len)::value;
    if (XLayout<LL>::bytes <= kDefaultSmem) return;
    const cudaError_t r = allow_dynamic_smem((const void*)x_pass2_kernel<LL>, max_smem);
    if (r != cudaSuccess) e = r;
    static_assert(!fp32_length(LL) || XLayout<LL>::bytes <= kDefaultSmem,
                  "the FP32 and slab forms stay within the default");
  });
  return e;
}

int ens_x_blocks(const XPassArgs& a) {
  constexpr int R = XShape<192>::R;
  return (a.nrows + R - 1) / R;
}

size_t ens_x_smem(int maxL) {
  return maxL == 48   ? XLayout<48>::bytes
         : maxL == 72 ? XLayout<72>::bytes
         : maxL == 96 ? XLayout<96>::bytes
                      : XLayout<192>::bytes;
}

const void* ens_x_kernel() { return (const void*)ens_x_pass2_kernel; }

}  // namespace dnsb
