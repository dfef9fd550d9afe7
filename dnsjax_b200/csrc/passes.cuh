// Axis-pass kernels of the dealiased transforms (declarations + arg blocks).
//
// A 3/2-dealiased transform is a sequence of axis passes; each pass reads
// one layout from HBM, transforms a tile of columns in shared memory and
// writes the next layout.  Zero-padding (inverse) and truncation (forward)
// happen on load/store, and the curl, the rotational nonlinear product and
// the pressure projection are fused into the passes that already hold the
// data they need.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace dnsb {

constexpr int kTile = 8;     // columns per CTA in the column passes
constexpr int kXRows = 4;    // physical rows per CTA in the x pass
constexpr int kPassThreads = 256;

// Padded lengths with two-stage register passes in FP64: those of 3/2 padding from 24
// to 256 modes (3 x 2^a 3^b points; odd lengths, 81 and 243, are refused) but 324 (216
// modes); the others run Stockham stages (216^3 RHS 7.75 ms).  The FP32, slab
// and work-list forms are compiled for fp32_length alone.
__host__ __device__ constexpr bool fp32_length(int L) {
  return L == 48 || L == 72 || L == 96 || L == 192;
}
__host__ __device__ constexpr bool two_stage_length(int L) {
  return fp32_length(L) || L == 36 || L == 54 || L == 108 || L == 144 || L == 162 ||
         L == 216 || L == 288 || L == 384;
}

// f(std::integral_constant<int, L>) for a two-stage length L, or for each.
#define DNSB_LENGTHS(X) \
  X(36) X(48) X(54) X(72) X(96) X(108) X(144) X(162) X(192) X(216) X(288) X(384)
template <typename F>
inline cudaError_t with_length(int L, F&& f) {
  switch (L) {
#define DNSB_LEN(LL) \
  case LL: return f(std::integral_constant<int, LL>{});
    DNSB_LENGTHS(DNSB_LEN)
#undef DNSB_LEN
    default: return cudaErrorInvalidValue;
  }
}
template <typename F>
inline void for_each_length(F&& f) {
#define DNSB_LEN(LL) f(std::integral_constant<int, LL>{});
  DNSB_LENGTHS(DNSB_LEN)
#undef DNSB_LEN
}
// Two radices of a column transform, M = R1 R2.
template <int M>
struct ColRadix;
#define DNSB_COL_RADIX(M_, R1_, R2_)                       \
  template <>                                              \
  struct ColRadix<M_> {                                    \
    static constexpr int R1 = R1_, R2 = R2_;               \
    static_assert(R1 * R2 == M_, "two radices");           \
  };
DNSB_COL_RADIX(36, 6, 6)
DNSB_COL_RADIX(48, 6, 8)
DNSB_COL_RADIX(54, 9, 6)
DNSB_COL_RADIX(72, 9, 8)
DNSB_COL_RADIX(96, 12, 8)
DNSB_COL_RADIX(108, 12, 9)
DNSB_COL_RADIX(144, 12, 12)
DNSB_COL_RADIX(162, 18, 9)
DNSB_COL_RADIX(192, 12, 16)
DNSB_COL_RADIX(216, 18, 12)
DNSB_COL_RADIX(288, 24, 12)
DNSB_COL_RADIX(384, 24, 16)
#undef DNSB_COL_RADIX

// Shared memory a kernel may use without raising its limit (less a margin for
// its static arrays).
constexpr size_t kDefaultSmem = 47 * 1024;

// Slab exchange (the reference's slab scheme over several GPUs): a pass
// that feeds the other layout stores each output straight into the
// buffer of the rank that owns it, through that rank's pointer (peer
// memory, or a buffer of this GPU when the ranks are emulated on one).
constexpr int kMaxRanks = 8;
struct SlabDest {
  double2* buf[kMaxRanks];  // receive buffer of each rank (null: no slab store)
  int blk;                  // extent of the split coordinate per rank
  long long fs, ts;         // destination field / split-coordinate strides
  long long off;            // offset of this rank's share in every destination
  long long so, si;         // x pass: destination row (outer + oo, inner + io)
  int oo, io;
  long long ks;             // x pass: destination kx stride
};

// Generic strided column pass: element (f, o, t, i) at
// base + f*fs + o*os + t*ts + i, with i the contiguous inner index.
struct ColPassArgs {
  const double2* in;
  double2* out;
  long long in_fs, out_fs, in_os, out_os, in_ts, out_ts;
  int nI;        // inner extent
  int nstored;   // stored (Nyquist-free) modes on the spectral side
  int inverse;   // 1: spectral -> padded, inverse FFT; 0: forward, truncate
  FFTPlan plan;  // transform length M = plan.L
  const double2* tw;
  int fp32;            // `in` and arithmetic in FP32 (compile-time sizes)
  int out32;           // with fp32: `out` is an FP32 pass buffer (always for inverse)
  int variant;         // 0: two-stage register pass when compiled for L, 1: Stockham
                       // stages (compile-time plan when compiled for L), 2: runtime plan
  // curl (inverse only, two-stage pass): `in` is the FP64 spectral state
  // [3][nstored][nO][nI] (component stride in_fs) and the 6 output fields are
  // u, v, w and i (k x u) with k = (kx[inner], ky[stored], kz[outer])
  int curl;
  const double* kx;
  const double* ky;
  const double* kz;
  // curl in FP64: the blocks of a column tile's six fields next to one another, so
  // that the components that several fields read come from L2
  int fields_fast;
  int held;  // FP64 two-stage forward pass at fp32_length with its registers held
  // Slab store (inverse, FP64 two-stage pass): position t goes to
  // slab.buf[t / blk] + f*fs + o*out_os + (t % blk)*ts + off + i, instead of
  // out + f*out_fs + o*out_os + t*out_ts + i.
  SlabDest slab;
  // Unrolled step-graph iterations: when non-null and *skip != 0 (the
  // corrector loop ended earlier in the step), the kernel returns at once.
  const int* skip = nullptr;
  int dep = 0;  // launch_dep
};

// x pass.  Rows are (outer, inner) pairs; row r = outer * inner_n + inner
// starts at outer*so + inner*si and its kx modes are ks apart.
struct XPassArgs {
  const double2* in;   // 6 fields (u, omega) of x-half-spectra
  double2* out;        // 3 fields of the forward x-transformed product
  long long in_fs, out_fs;
  int nrows, inner_n;
  long long so, si, ks;
  int nkx;             // stored kx modes (nx/2)
  int y_outer;         // y index = outer (1) or inner (0)
  int rows_fast;       // load mapping: rows contiguous (1) or kx (0)
  const double* U;     // base flow [3][ny_grid]
  const double* cU;    // curl of base flow
  const double* nU;    // U x curl U
  int ny_grid;
  FFTPlan plan;        // Mx
  const double2* tw;   // float2 table when fp32
  int fp32;            // pass buffer and arithmetic in FP32 (compile-time sizes)
  int variant;         // 0: two-stage register pass when compiled for L, 1: Stockham
                       // stages (compile-time plan when compiled for L), 2: runtime plan
  // Slab store (FP64 two-stage pass): mode k of field f of row (outer,
  // inner) goes to slab.buf[k / blk] + f*fs + (outer + oo)*so +
  // (inner + io)*si + (k % blk)*ks, instead of into `out`.
  SlabDest slab;
  // Unrolled step-graph iterations: when non-null and *skip != 0 (the
  // corrector loop ended earlier in the step), the kernel returns at once.
  const int* skip = nullptr;
  int dep = 0;  // launch_dep
};

// x pass to physical space only (3 fields -> real [c] at row offsets
// outer*pso + inner*psi, x contiguous).
struct XPhysArgs {
  const double2* in;
  double* out;
  long long in_fs, out_fs;
  int nrows, inner_n;
  long long so, si, ks, pso, psi;
  int nkx;
  int rows_fast;
  FFTPlan plan;
  const double2* tw;
};

// Periodic first inverse pass (y), curl fused: spectral u [3][NY1][NZ1][NKX]
// -> 6 (or 3) fields [f][My][NZ1][NKX].
struct YInvArgs {
  const double2* u;
  double2* out;
  int NY1, NZ1, NKX;
  int curl;
  const double* kx;
  const double* ky;
  const double* kz;
  FFTPlan plan;
  const double2* tw;
  int fp32;  // FP32 transform and output pass buffer (tw: float2 table)
  int variant;  // 0 / 1: compile-time plan when compiled for L, 2: runtime plan
};

// Periodic last forward pass (y), projection fused: [3][My][NZ1][NKX] ->
// spectral [3][NY1][NZ1][NKX].
struct YFwdArgs {
  const double2* in;
  double2* out;
  int NY1, NZ1, NKX;
  int project;
  const double* kx;
  const double* ky;
  const double* kz;
  const double* inv_lapl;  // [NY1][NZ1][NKX]
  FFTPlan plan;
  const double2* tw;
  int fp32;  // FP32 input pass buffer and transform (tw: float2 table)
  int variant;  // 0 / 1: compile-time plan when compiled for L, 2: runtime plan
};

// Periodic last forward pass (y) with the projection, two-stage lengths
// (csrc/y_project.cu): in [3][My][NZ1][NKX] -> spectral [3][NY1][NZ1][NKX].
struct YProjArgs {
  const double2* in;
  double2* out;
  int NY1, NZ1, NKX;
  const double* kx;
  const double* ky;
  const double* kz;
  const double* inv_lapl;  // [NY1][NZ1][NKX]
  const double2* tw;       // float2 table when fp32
  int fp32;                // FP32 input pass buffer and transform
  const int* skip = nullptr;  // as ColPassArgs::skip
  int dep = 0;                // launch_dep
};
cudaError_t launch_yfwd_project(const YProjArgs& a, int L, cudaStream_t st);
// Its work-list form for ensembles (see EnsColItem).
struct EnsYItem {
  YProjArgs a;
  int L, gx, blocks, member;
};
int ens_y_blocks(EnsYItem* it, bool wide);
size_t ens_y_smem(int maxL);
int ens_y_threads(bool wide);
const void* ens_y_kernel(bool wide);
cudaError_t set_yfwd_project_attributes(int max_smem);

// Couette first inverse pass (z), FD curl fused: spectral
// [3][NZ1][NKX][Ny] -> 6 (or 3) fields [f][Mz][NKX][Ny].
struct ZInvCurlArgs {
  const double2* u;
  double2* out;
  int NZ1, NKX, Ny;
  int curl;
  int fields_fast;     // two-stage pass: as ColPassArgs::fields_fast (any field count)
  int s1;              // D1 stencil width (p + 1)
  const int* d1_j0;    // [Ny]
  const double* d1_w;  // [Ny][s1]
  const double* d1_wT; // [s1][Ny] (the same weights, tap-major)
  const double* kx;
  const double* kz;
  FFTPlan plan;
  const double2* tw;   // float2 table when fp32
  int fp32;            // output pass buffer and FFT in FP32 (compile-time sizes)
  int variant;         // 0: two-stage register pass when compiled for L, 1: Stockham
                       // stages (compile-time plan when compiled for L), 2: runtime plan
  // Slab store (FP64 two-stage pass): position t of column q goes to
  // slab.buf[t / blk] + f*fs + (t % blk)*ts + off + q.
  SlabDest slab;
  // Unrolled step-graph iterations: when non-null and *skip != 0 (the
  // corrector loop ended earlier in the step), the kernel returns at once.
  const int* skip = nullptr;
  int dep = 0;  // launch_dep
};

constexpr int kZTile = 8;  // y values per CTA in the Couette z passes

size_t col_pass_smem(int M);
size_t x_pass_smem(int Mx);
size_t x_phys_smem(int Mx);
size_t yinv_smem(int My, int NY1, int fp32);
size_t yfwd_smem(int My, int NY1, int fp32);
size_t zinv_curl_smem(int Mz, int NZ1, int span_max);
size_t zinv_curl2_smem(int M);

cudaError_t launch_col_pass(const ColPassArgs& a, int nfields, int nO,
                            cudaStream_t st);
cudaError_t launch_x_pass(const XPassArgs& a, cudaStream_t st);
// The register-stage x pass (csrc/x_pass.cu): two_stage_length(plan.L) with
// nkx = plan.L / 3.
cudaError_t launch_x_pass2(const XPassArgs& a, cudaStream_t st);
cudaError_t set_x_pass_attributes(int max_smem);
// The register-stage x passes of the plain transforms (csrc/x_transform.cu),
// same lengths.
cudaError_t launch_x_phys2(const XPhysArgs& a, cudaStream_t st);
cudaError_t launch_x_fwd2(const XPhysArgs& a, const double* phys, double2* spec,
                          cudaStream_t st);
cudaError_t set_x_transform_attributes(int max_smem);

// Work lists of the ensemble form (one launch per pass for every member;
// FP64 two-stage passes, padded lengths 48, 72, 96, 192).
struct EnsColItem {
  ColPassArgs a;
  int gx, gy;  // the member's grid (gx, gy, nfields), flattened bx fastest
  int blocks;  // gx gy nfields
  int member;
};
struct EnsXItem {
  XPassArgs a;
  int member;
};
bool ens_pass_supported(int L);
// Fill an item's grid; CTAs that its blocks take (wide: see ens_pass_grid).
int ens_col_blocks(EnsColItem* it, int nO, int nfields, bool wide);
int ens_x_blocks(const XPassArgs& a);
constexpr int kEnsXThreads = 96;
const void* ens_x_kernel();
// Item of virtual block vb: the last k with base[k] <= vb.
__device__ __forceinline__ int ens_find(const int* __restrict__ base, int n, int vb) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (base[mid] <= vb) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}
size_t ens_col_smem(int maxL);
size_t ens_x_smem(int maxL);
// kind 0: inverse pass with the spectral curl, 1: inverse, 2: forward
// (column passes); 3: the x pass; 4: the y forward pass with the projection.
// wide: a member's padded length is 192.  base[k]: first virtual block of item k.
int ens_pass_grid(int kind, bool wide, size_t smem, int total, int max_smem);
cudaError_t launch_ens_pass(int kind, bool wide, const void* items, const int* base, int n,
                            int total, const int* active, int grid, size_t smem,
                            cudaStream_t st);
cudaError_t launch_x_phys(const XPhysArgs& a, cudaStream_t st);
// Forward x pass from physical rows (uses XPhysArgs with in_fs = spectral
// field stride, out_fs = physical field stride).
cudaError_t launch_x_fwd(const XPhysArgs& a, const double* phys, double2* spec,
                         cudaStream_t st);
size_t x_fwd_smem(int Mx);
cudaError_t set_pass_attributes(int max_smem);
cudaError_t launch_yinv(const YInvArgs& a, cudaStream_t st);
cudaError_t launch_yfwd(const YFwdArgs& a, cudaStream_t st);
cudaError_t launch_zinv_curl(const ZInvCurlArgs& a, int span_max,
                             cudaStream_t st);

FFTPlan make_plan(int L);  // host; L.nst == 0 when L is not 2^a 3^b

}  // namespace dnsb
