// Periodic y forward transform with truncation and the pressure projection
// NL - grad(inv_lapl div NL) (src/dnsjax/flows/monochromatic.py:366-386), in
// register stages: a CTA takes 8 (kz, kx) columns of all three components, a
// third of its threads each.  The transformed columns stay in shared memory
// until every component of a mode is there.
//
// As two kernels, the transform wrote the RHS and the projection read and wrote
// it again: 100 of 125 + 100 MB at 128^3, and one launch more, which is what
// counts on small grids.  8 columns leave room for 2 CTAs per SM at every
// length up to 288 (3 components x M x 8 columns), 16 would leave one.
// Measured: 32^3 time step 183 -> 175 us, 24 x 36 x 48 predict_and_correct 85 ->
// 81 us, 256^3 RHS 3.35 -> 3.28 ms, 128^3 as before (FP32 229 -> 225 us).
#include "passes.cuh"

namespace dnsb {

namespace {

// Radices (M = R1 R2) of the column pass; 8 columns, so NF threads per
// component and R1 items per thread group of R2.
template <int M, typename T>
struct YShape {
  static constexpr int C = 8;  // of every length and type
  static constexpr bool F32 = !std::is_same_v<T, double>;
  // FP32 at 192: 24 x 8 in 192 threads (128^3 RHS 213.8 us; 12 x 16: 215.6)
  static constexpr int R1 = F32 && M == 192 ? 24 : ColRadix<M>::R1, R2 = M / R1;
  static constexpr int NF = R2 * C, NT = 3 * NF;
  // registers: held to as many whole CTAs as 768 threads hold where at most 16 FP64
  // values a thread fit (192 points: 2 CTAs, 24 warps per SM, against 12 warps of 24 x
  // 8: 128^3 RHS 328.1 -> 320.2 us; 108 points: 3 CTAs, 21 warps: 96 x 72 x 144 RHS
  // 179.5 -> 176.8 us; 144 points: 2 CTAs, 18 warps).  CTAs of up to 192 threads need
  // no more than 2 asked for: at 72 points 90 registers are better, 48 x 48 x 96 RHS
  // 55.4 us against 56.1
  static constexpr int MINB = NT <= 192 ? 2 : !F32 && R1 <= 16 ? 768 / NT : 1;
};

// H = 2: two blocks in a CTA of twice the shape's NT threads, as col_pass2_body
// (csrc/passes.cu).
template <int ML, typename T, int H = 1>
__device__ __forceinline__ void yfwd_project_body(const YProjArgs& a, int bx, int iz,
                                                  bool idle = false) {
  using CT = typename pass_types<T>::C;
  using SH = YShape<ML, T>;
  constexpr int M = ML, R1 = SH::R1, R2 = SH::R2, C = SH::C, NF = SH::NF, NT = SH::NT;
  extern __shared__ double2 sm_[];
  const int half = H == 2 ? threadIdx.x / NT : 0;
  CT* sm = reinterpret_cast<CT*>(sm_) + half * 3 * M * C;  // [component][t][C]
  const CT* __restrict__ tw = reinterpret_cast<const CT*>(a.tw);
  const int tid = threadIdx.x - half * NT, f = tid / NF, t0 = tid % NF;
  const int NY1 = a.NY1, NZ1 = a.NZ1, NKX = a.NKX;
  const int i0 = bx * C;
  const int ni = H == 2 && idle ? 0 : min(C, NKX - i0);
  CT* X = sm + f * M * C;
  const long long row = (long long)NZ1 * NKX;  // stride of y
  {
    const int c = t0 % C, j = t0 / C;
    const CT* in = reinterpret_cast<const CT*>(a.in) + (long long)f * M * row +
                   (long long)iz * NKX + i0 + c;
    const unsigned long long drop = l2_drop();
    CT v[R1];
#pragma unroll
    for (int i = 0; i < R1; ++i)
      v[i] = c < ni ? CT(ld_l2(in + (j + R2 * i) * row, drop)) : cmake<CT>(0, 0);
    dft_reg<R1, -1>(v);
#pragma unroll
    for (int i = 0; i < R1; ++i) X[(j * R1 + i) * C + c] = v[i];
  }
  __syncthreads();
  for (int it = t0; it < R1 * C; it += NF) {
    const int c = it % C, k = it / C;
    CT z[R2];
#pragma unroll
    for (int i = 0; i < R2; ++i) z[i] = X[(k + R1 * i) * C + c];
#pragma unroll
    for (int i = 1; i < R2; ++i) z[i] = cmul(z[i], CT(tw[i * k]));
    dft_reg<R2, -1>(z);
    // position k + R1 i: where the item read
#pragma unroll
    for (int i = 0; i < R2; ++i) X[(k + R1 * i) * C + c] = z[i];
  }
  __syncthreads();
  const double sc = 1.0 / M;
  const double kz = a.kz[iz];
  const long long cs = (long long)NY1 * row;
  for (int idx = tid; idx < NY1 * C; idx += NT) {
    const int c = idx % C, s = idx / C;
    if (c >= ni) continue;
    const int t = stored_to_pos(s, NY1, M) * C + c;
    double2 u[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      // rounded before the projection, as where the transform stores it (the
      // work-list ensemble's kernels give the same bits)
      const double2 z = to_d(sm[q * M * C + t]);
      u[q] = make_double2(__dmul_rn(z.x, sc), __dmul_rn(z.y, sc));
    }
    const long long off = s * row + (long long)iz * NKX + i0 + c;
    project_mode(u, a.kx[i0 + c], a.ky[s], kz, a.inv_lapl[off]);
#pragma unroll
    for (int q = 0; q < 3; ++q) a.out[q * cs + off] = u[q];
  }
}

template <int ML, typename T>
__global__ void __launch_bounds__(YShape<ML, T>::NT, YShape<ML, T>::MINB)
yfwd_project_kernel(YProjArgs a) {
  grid_dep_sync();
  if (a.skip && *a.skip) return;
  yfwd_project_body<ML, T>(a, blockIdx.x, blockIdx.y);
}

// Work-list form for ensembles: as ens_x_pass2_kernel (csrc/x_pass.cu), two blocks of
// a shorter member in a wide CTA as ens_col_pass2_kernel (csrc/passes.cu).  Wide: 24
// warps per SM as the plain kernel at 192 (308 bytes of spills; with 12 warps a step
// of four 128^3 members took 9.55 ms, 9.32 so).
__host__ __device__ constexpr int ens_y_shape(bool wide) {
  return wide ? YShape<192, double>::NT : YShape<96, double>::NT;
}
static_assert(YShape<48, double>::NT == ens_y_shape(false) &&
                  YShape<72, double>::NT == ens_y_shape(false) &&
                  ens_y_shape(true) == 2 * ens_y_shape(false),
              "a CTA shape for every member");
template <int ML, bool WIDE>
__device__ __forceinline__ void ens_y_block(const EnsYItem& it, const YProjArgs& a, int local) {
  constexpr int NT = YShape<ML, double>::NT, H = WIDE && NT < ens_y_shape(true) ? 2 : 1;
  const int b = H == 2 ? 2 * local + threadIdx.x / NT : local;
  const int blk = min(b, it.blocks - 1);
  yfwd_project_body<ML, double, H>(a, blk % it.gx, blk / it.gx, b != blk);
}
template <bool WIDE>
__global__ void __launch_bounds__(ens_y_shape(WIDE), WIDE ? 2 : 0)
ens_yfwd_project_kernel(const EnsYItem* __restrict__ items, const int* __restrict__ base, int n,
                        int total, const int* __restrict__ active) {
  __shared__ int s_k;
  for (int vb = blockIdx.x; vb < total; vb += gridDim.x) {
    if (threadIdx.x == 0) s_k = ens_find(base, n, vb);
    __syncthreads();
    const int k = s_k;
    const int m = items[k].member;
    if (!active || active[m]) {
      const YProjArgs a = items[k].a;
      const int local = vb - base[k];
      switch (items[k].L) {
        case 48: ens_y_block<48, WIDE>(items[k], a, local); break;
        case 72: ens_y_block<72, WIDE>(items[k], a, local); break;
        case 96: ens_y_block<96, WIDE>(items[k], a, local); break;
        default:
          if constexpr (WIDE) ens_y_block<192, WIDE>(items[k], a, local);
          break;
      }
    }
    __syncthreads();
  }
}

template <int ML>
constexpr size_t yproj_smem() {
  return sizeof(double2) * (size_t)(3 * ML * YShape<ML, double>::C);
}

}  // namespace

cudaError_t launch_yfwd_project(const YProjArgs& a, int L, cudaStream_t st) {
  if (a.fp32 && !fp32_length(L)) return cudaErrorInvalidValue;
  return with_length(L, [&](auto len) {
    constexpr int LL = decltype(len)::value;
    const dim3 grid((a.NKX + YShape<LL, double>::C - 1) / YShape<LL, double>::C, a.NZ1);
    const size_t sm = a.fp32 ? yproj_smem<LL>() / 2 : yproj_smem<LL>();
    if constexpr (fp32_length(LL)) {
      constexpr int NT = YShape<LL, float>::NT;
      if (a.fp32 == 2) launch_dep(a.dep, yfwd_project_kernel<LL, fcomp>, grid, NT, sm, st, a);
      else if (a.fp32) launch_dep(a.dep, yfwd_project_kernel<LL, float>, grid, NT, sm, st, a);
      if (a.fp32) return cudaGetLastError();
    }
    launch_dep(a.dep, yfwd_project_kernel<LL, double>, grid, YShape<LL, double>::NT, sm, st, a);
    return cudaGetLastError();
  });
}

int ens_y_blocks(EnsYItem* it, bool wide) {
  it->gx = (it->a.NKX + YShape<192, double>::C - 1) / YShape<192, double>::C;
  it->blocks = it->gx * it->a.NZ1;
  return wide && it->L != 192 ? (it->blocks + 1) / 2 : it->blocks;
}

size_t ens_y_smem(int maxL) {
  return sizeof(double2) * (size_t)(3 * maxL * YShape<192, double>::C);
}

int ens_y_threads(bool wide) { return ens_y_shape(wide); }

const void* ens_y_kernel(bool wide) {
  return wide ? (const void*)ens_yfwd_project_kernel<true>
              : (const void*)ens_yfwd_project_kernel<false>;
}

cudaError_t set_yfwd_project_attributes(int max_smem) {
  cudaError_t e = cudaSuccess;
  for_each_length([&](auto len) {
    constexpr int LL = decltype(len)::value;
    if (yproj_smem<LL>() <= kDefaultSmem) return;
    const cudaError_t r =
        allow_dynamic_smem((const void*)yfwd_project_kernel<LL, double>, max_smem);
    if (r != cudaSuccess) e = r;
    static_assert(!fp32_length(LL) || yproj_smem<LL>() / 2 <= kDefaultSmem,
                  "the FP32 forms stay within the default");
  });
  return e;
}

}  // namespace dnsb
