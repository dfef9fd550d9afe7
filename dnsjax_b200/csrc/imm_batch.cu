// Plane Couette influence-matrix iteration as five bandwidth-shaped kernels.
//
// Follows src/dnsjax/flows/plane_couette.py:376-504 (six stages) and the
// dgbtrs-'N' substitution of src/dnsjax/geometries/cartesian.py:360-441.
//
//   stages 0-1   one warp per (kz, kx) mode: d_hat = div u^n, then f_hat
//   (+ 3)        (D1 / D2 along y) -> F, and in the same pass the part of
//                stage 3 that does not need p_P, Q = H_k^- u^n + c N_j + (1-c)
//                N_n -> R, so u^n, N_j and N_n are read once per call
//   L_k solve    p_P = L_k^-1 f_hat in place in F: a CTA per tile of 16 items,
//                one warp per component, lane = side * 16 + item (side 1 is the
//                mirror mode (nz-1-s, kx) of item (s, kx) when it shares the
//                item's factors), each lane one complex column
//   stage 3      R -= grad p_P on the interior rows
//   H_k solve    as the L_k solve, three components, in place in R
//   stages 4-6   one warp per mode: wall divergence, influence-matrix
//                weights, u^{j+1}, the correction and its Simpson norm
//
// The workspaces F and R[3] are laid out for the substitutions, [tile][y][32
// lanes]: a row of a tile is 512 contiguous bytes, so the rows that enter a
// block of substitution steps are one bulk copy and every result row one
// coalesced store.  (As [mode][y], which the kernels ran on before, each lane's
// 16 bytes were a sector of their own, read and written twice per solve: the
// L_k / H_k launches took 38 / 68 us at 128 x 129 x 128, now 30 / 36.  What is
// left is the dependent chain of a step, about 220 cycles, on a warp that has its
// scheduler to itself; real and imaginary columns on a warp each made the whole
// corrector slower, 201 -> 214 us, as the lanes' 8-byte stores were 16 apart; with
// a warp per side, lane = (item, re or im), they are contiguous.)  The stage kernels
// transpose through shared memory, four modes (64 bytes of a row) at a time.
//
// The LU factors are repacked once, when the operators are bound, into
// 16-item tiles whose rows are contiguous (layout below), so a block of
// substitution steps of one tile is one bulk copy into shared memory.
// An item is mode (s, kx) with s <= (nz-1)/2; when the factors of (s, kx)
// and its mirror (nz-1-s, kx) are bit-identical (same k^2; checked at bind
// time) the mirror reads the item's records, else every mode is an item.
#include <algorithm>
#include <vector>

#include "imm_solve.cuh"
#include "solver.cuh"

namespace dnsb {

namespace {

constexpr int kStageWarps = 4;  // modes per CTA in the stage kernels

// L2 residency of the workspaces F and R (K Ny and 3 K Ny complex, 67 MB at
// 128x129x128, each touched about three times per call): their writes carry an
// evict_last policy, and the last read of R (stage 6) evict_first, so the
// streamed inputs do not push them out of the 126 MB L2 between the kernels of
// one call (l2_keep / l2_drop and the hinted accesses are in common.cuh).

// Tile and lane of mode m: item p on side 0, or the mirror of item p on side 1.
struct ModeSlot {
  long long tile;
  int lane;
};
__device__ __forceinline__ ModeSlot mode_slot(int m, int NKX, int NZ1, int paired) {
  const int s = m / NKX, ix = m % NKX;
  const bool mirror = paired && s >= (NZ1 + 1) / 2;
  const int p = mirror ? (NZ1 - s) * NKX + ix : m;
  return {p / kTile, (mirror ? kTile : 0) + p % kTile};
}

}  // namespace

// ---------------------------------------------------------------------------
// Bind time: repack one operator's factors into 16-item tiles, each tile's
// rows contiguous so a block of substitution steps is one contiguous copy:
//   facL[tile][j][i/2][16][2]       (rows j < Ny, then W zero rows)  L
//                                   multipliers of rows j+1..j+kl
//   facU[tile][j + WB][i/2][16][2]  (WB zero rows first; NUP = NU+1 rounded
//                                   up to even) i = 0: 1/U_jj, i > 0:
//                                   U_{j-i,j}, over U_jj where `scaled`
//   dp[tile][j][16]            ipiv[j] - j, validated (a bad pivot is flagged
//                              and replaced by 0)
// Item p is mode p (modes (s, kx) with s <= (nz-1)/2 when mirrors share
// factors).  The arrays must be zeroed before the call (padding rows and
// items).
// ---------------------------------------------------------------------------
__global__ void imm_repack_kernel(const double* __restrict__ ab, const int* __restrict__ piv,
                                  int Ny, int kl, int nu, int row0, int NP, int scaled,
                                  double* facL, double* facU, unsigned char* dp, int* status) {
  const int rows = 3 * kl + 1, kuu = 2 * kl, W = kl + 1, WB = nu + 1;
  const int nup = (nu + 2) & ~1;  // U record length, even
  const long long NyF = Ny + W, NyB = Ny + WB;
  const long long n = (long long)NP * Ny;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < n;
       idx += (long long)gridDim.x * blockDim.x) {
    const int p = (int)(idx % NP), j = (int)(idx / NP);
    const int tile = p / kTile, it = p % kTile;
    const double* abm = ab + (long long)p * rows * Ny;
    const double r = 1.0 / abm[(long long)kuu * Ny + j];
    // element i of row j: [tile][j][i / 2][it][i % 2]
    double* L = facL + (tile * NyF + j) * kl * kTile + 2 * it;
    for (int i = 1; i <= kl; ++i) {
      const int e = i - 1;
      L[(e >> 1) * 2 * kTile + (e & 1)] = abm[(long long)(kuu + i) * Ny + j];
    }
    double* U = facU + (tile * NyB + j + WB) * nup * kTile + 2 * it;
    U[0] = r;
    for (int i = 1; i <= nu; ++i) {
      const int row = kuu - i;
      const double u = (row >= row0) ? abm[(long long)row * Ny + j] : 0.0;
      U[(i >> 1) * 2 * kTile + (i & 1)] = scaled ? u * r : u;
    }
    int d = piv[(long long)p * Ny + j] - j;
    if (d < 0 || d > kl || j + d >= Ny) {  // never follow a bad pivot
      atomicOr(status, 1);
      d = 0;
    }
    dp[(tile * NyF + j) * kTile + it] = (unsigned char)d;
  }
}

cudaError_t launch_imm_repack(const double* ab, const int* piv, int Ny, int kl, int nu,
                              int row0, int NP, int scaled, double* facL, double* facU,
                              unsigned char* dp, int* status, cudaStream_t st) {
  imm_repack_kernel<<<592, 256, 0, st>>>(ab, piv, Ny, kl, nu, row0, NP, scaled, facL, facU,
                                         dp, status);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Stages 0-1 and the pressure-free part of stage 3.  One warp per mode, lane l
// the YM consecutive rows y = YM l + o, four modes per CTA.
//
// With N = c N_j + (1-c) N_n, f_hat = d/dt + div N + (1-c) nu (D2 - k2) d and
// Q = u/dt + (1-c) nu (D2 - k2) u + N.  A lane walks the W = S2 + YM - 1 rows its
// YM rows' stencils reach, adding each row to the YM sums it belongs to: one
// shared-memory read per row of the window instead of one per tap and row, and
// 2 YM or more independent sums in flight.  The weights come window-relative
// ([o][W][32 lanes], zero outside the stencil), so rows whose stencils are
// shifted at the walls run the same code.  YM is odd, so lanes YM rows apart
// read without bank conflicts.  All rows live in place in 7 Ny complex values a
// mode (3 CTAs per SM at 129 rows): Q_u, Q_v, Q_w over N, f over d.  Bound by
// latency and the weights' L1 reads: 71 us cold at 128 x 129 x 128 for 33 us of
// memory time (72 with one read per tap and row-major workspaces; 80 with the
// window in registers, 55 against 43 at 96 x 193 x 72).
// ---------------------------------------------------------------------------
// Values per mode in shared memory: 7 Ny, rounded so that the four modes of a
// row fall on other banks when the CTA writes it out.
__host__ __device__ constexpr int stage_stride(int Ny) { return ((7 * Ny + 5) / 8) * 8 + 2; }

__device__ __forceinline__ void axpy(double2& acc, double w, double2 x) {
  acc.x += w * x.x;
  acc.y += w * x.y;
}

template <int KL, int YM>
__global__ void __launch_bounds__(32 * kStageWarps, YM == 5 ? 3 : 1)
imm_stage013_kernel(ImmArgs a, int paired, const double* __restrict__ w1x,
                    const double* __restrict__ w2x, const int* __restrict__ base,
                    const double2* __restrict__ vel_n, const double2* __restrict__ nl_n,
                    const double2* __restrict__ nl_j, double2* __restrict__ F,
                    double2* __restrict__ R, long long cs) {
  grid_dep_sync();
  if (a.skip && *a.skip) return;
  constexpr int W = KL + 2 + YM - 1;
  extern __shared__ double2 sm[];
  __shared__ long long s_dst[kStageWarps];
  const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5;
  const int NKX = a.NKX, Ny = a.Ny, NM = a.NZ1 * a.NKX;
  const int m = blockIdx.x * kStageWarps + wq;
  const bool act = m < NM;
  const int SS = stage_stride(Ny);
  if (act) {
    double2* T = sm + wq * SS;  // u, v, w, N_u, N_v, N_w, d
    double2 *Nr = T + 3 * Ny, *D = T + 6 * Ny;
    const long long CS = (long long)NM * Ny, mo = (long long)m * Ny;
    if (lane == 0) {
      const ModeSlot ms = mode_slot(m, NKX, a.NZ1, paired);
      s_dst[wq] = ms.tile * Ny * kLanes + ms.lane;
    }
    for (int y = lane; y < Ny; y += 32) {
#pragma unroll
      for (int c = 0; c < 3; ++c) cp_async16(T + c * Ny + y, vel_n + c * CS + mo + y);
    }
    cp_async_commit();
    const int iz = m / NKX, ix = m % NKX;
    const double kx = a.kx[ix], kz = a.kz[iz];
    const double k2 = kx * kx + kz * kz;
    const double c = a.c, omc = 1.0 - c, omc_nu = omc * a.nu, idt = 1.0 / a.dt;
    {
      double2 nj[3][YM], nn[3][YM];
#pragma unroll
      for (int k = 0; k < YM; ++k) {
        const int y = lane + 32 * k;
        if (y < Ny) {
#pragma unroll
          for (int cpt = 0; cpt < 3; ++cpt) {
            // streamed once: keep the weights in L1
            nj[cpt][k] = ld_stream(nl_j + cpt * CS + mo + y);
            nn[cpt][k] = ld_stream(nl_n + cpt * CS + mo + y);
          }
        }
      }
#pragma unroll
      for (int k = 0; k < YM; ++k) {
        const int y = lane + 32 * k;
        if (y < Ny) {
#pragma unroll
          for (int cpt = 0; cpt < 3; ++cpt)
            Nr[cpt * Ny + y] = cadd(cscale(nj[cpt][k], c), cscale(nn[cpt][k], omc));
        }
      }
    }
    cp_async_wait_all();
    __syncwarp();
    const int y0 = YM * lane, b = base[lane];
    const double *w1 = w1x + lane, *w2 = w2x + lane;
    double2 f[YM], qv[YM];
    {
      // d_hat = div u^n, Q, and div N but for D1 N_v
      double2 su[YM], sv[YM], sw[YM], dv[YM];
#pragma unroll
      for (int o = 0; o < YM; ++o) su[o] = sv[o] = sw[o] = dv[o] = make_double2(0.0, 0.0);
#pragma unroll 2
      for (int i = 0; i < W; ++i) {
        const int r = min(b + i, Ny - 1);
        const double2 xu = T[r], xv = T[Ny + r], xw = T[2 * Ny + r];
#pragma unroll
        for (int o = 0; o < YM; ++o) {
          const double c1 = w1[(o * W + i) * 32], c2 = w2[(o * W + i) * 32];
          axpy(dv[o], c1, xv);
          axpy(su[o], c2, xu);
          axpy(sv[o], c2, xv);
          axpy(sw[o], c2, xw);
        }
      }
#pragma unroll
      for (int o = 0; o < YM; ++o) {
        const int y = y0 + o;
        if (y < Ny) {
          const bool in = y > 0 && y < Ny - 1;
          const double2 zero = make_double2(0.0, 0.0);
          const double2 u = T[y], v = T[Ny + y], w = T[2 * Ny + y];
          const double2 nu = Nr[y], nv = Nr[Ny + y], nw = Nr[2 * Ny + y];
          D[y] = cadd(cadd(cik(kx, u), dv[o]), cik(kz, w));
          f[o] = cadd(cik(kx, nu), cik(kz, nw));
          const double2 hu = cadd(cscale(u, idt), cscale(csub(su[o], cscale(u, k2)), omc_nu));
          const double2 hv = cadd(cscale(v, idt), cscale(csub(sv[o], cscale(v, k2)), omc_nu));
          const double2 hw = cadd(cscale(w, idt), cscale(csub(sw[o], cscale(w, k2)), omc_nu));
          Nr[y] = in ? cadd(hu, nu) : zero;
          qv[o] = in ? cadd(hv, nv) : zero;
          Nr[2 * Ny + y] = in ? cadd(hw, nw) : zero;
        }
      }
    }
    __syncwarp();  // every D row written
    {
      double2 dn[YM], sd[YM];
#pragma unroll
      for (int o = 0; o < YM; ++o) dn[o] = sd[o] = make_double2(0.0, 0.0);
#pragma unroll 2
      for (int i = 0; i < W; ++i) {
        const int r = min(b + i, Ny - 1);
        const double2 xn = Nr[Ny + r], xd = D[r];
#pragma unroll
        for (int o = 0; o < YM; ++o) {
          axpy(dn[o], w1[(o * W + i) * 32], xn);
          axpy(sd[o], w2[(o * W + i) * 32], xd);
        }
      }
#pragma unroll
      for (int o = 0; o < YM; ++o) {
        const int y = y0 + o;
        if (y < Ny) {
          const double2 d = D[y];
          const double2 Lkd = csub(sd[o], cscale(d, k2));
          f[o] = cadd(cadd(cscale(d, idt), cadd(f[o], dn[o])), cscale(Lkd, omc_nu));
        }
      }
    }
    __syncwarp();  // every D and N_v row read
#pragma unroll
    for (int o = 0; o < YM; ++o) {
      const int y = y0 + o;
      if (y < Ny) {
        D[y] = (y > 0 && y < Ny - 1) ? f[o] : make_double2(0.0, 0.0);
        Nr[Ny + y] = qv[o];
      }
    }
  }
  __syncthreads();
  // Out to the tiles, four modes of a row at a time.
  const unsigned long long keep = l2_keep();
  const int nm = min(kStageWarps, NM - (int)blockIdx.x * kStageWarps);
  const int q = threadIdx.x & 3;
  if (q < nm) {
    const double2* src = sm + q * SS + 3 * Ny;
    const long long dst = s_dst[q];
    for (int y = threadIdx.x >> 2; y < Ny; y += 8 * kStageWarps) {
      const long long d = dst + (long long)y * kLanes;
#pragma unroll
      for (int cpt = 0; cpt < 3; ++cpt) st_l2(R + cpt * cs + d, src[cpt * Ny + y], keep);
      st_l2(F + d, src[3 * Ny + y], keep);
    }
  }
}

// ---------------------------------------------------------------------------
// Stage 3's pressure gradient: R -= grad p_P on the interior rows (the wall
// rows of R stay zero), p_P = L_k^-1 f_hat from the L_k substitution in F.
// Thread = (row, lane) of a tile: every access is a whole tile row, and the
// rows of p that a block's stencils share come from L1.
// ---------------------------------------------------------------------------
constexpr int kGradRows = 8;

template <int KL>
__global__ void __launch_bounds__(kLanes * kGradRows)
imm_grad_kernel(ImmArgs a, int paired, int NP, const double2* __restrict__ P,
                double2* __restrict__ R, long long cs) {
  grid_dep_sync();
  if (a.skip && *a.skip) return;
  constexpr int S1 = KL + 1;
  const int lane = threadIdx.x & 31, side = lane / kTile, Ny = a.Ny;
  const int y = blockIdx.x * kGradRows + (threadIdx.x >> 5) + 1;
  if (y >= Ny - 1) return;
  const long long t0 = (long long)blockIdx.y * Ny * kLanes + lane;
  const int p = blockIdx.y * kTile + lane % kTile, s = p / a.NKX;
  const bool live = p < NP && (side == 0 || (paired && s != 0));
  if (!live) return;
  const double kx = a.kx[p % a.NKX], kz = a.kz[side ? a.NZ1 - s : s];
  const unsigned long long keep = l2_keep();
  double2* r = R + t0 + (long long)y * kLanes;
  const double2 r0 = ld_l2(r, keep), r1 = ld_l2(r + cs, keep), r2 = ld_l2(r + 2 * cs, keep);
  const double2 pc = P[t0 + (long long)y * kLanes];
  const double2* pw = P + t0 + (long long)a.d1_j0[y] * kLanes;
  double2 dp = make_double2(0.0, 0.0);
#pragma unroll
  for (int i = 0; i < S1; ++i) {
    const double w = a.d1_w[y * S1 + i];
    const double2 v = pw[i * kLanes];
    dp.x += w * v.x;
    dp.y += w * v.y;
  }
  st_l2(r, csub(r0, cik(kx, pc)), keep);
  st_l2(r + cs, csub(r1, dp), keep);
  st_l2(r + 2 * cs, csub(r2, cik(kz, pc)), keep);
}

// ---------------------------------------------------------------------------
// Stages 4-6: vel_new, correction, per-mode norm partial.  One warp per mode,
// y over the lanes; R comes out of the tiles through shared memory, four modes
// of a row at a time.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int assemble_stride(int Ny) { return ((3 * Ny + 5) / 8) * 8 + 2; }

// YM: rows per lane whose inputs are held in registers (all in flight at once;
// Ny <= 32 YM), or 0: read where they are used.
template <int KL, int YM>
__global__ void __launch_bounds__(32 * kStageWarps)
imm_stage6_kernel(ImmArgs a, int paired, const double2* __restrict__ R, long long cs,
                  const double2* vel_j, double2* vel_new, double2* __restrict__ corr_out,
                  double* __restrict__ partials) {
  grid_dep_sync();
  if (a.skip && *a.skip) return;
  constexpr int S1 = KL + 1, YR = YM > 0 ? YM : 1;
  extern __shared__ double2 sm[];
  const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5;
  const int NKX = a.NKX, Ny = a.Ny, NM = a.NZ1 * a.NKX, SS = assemble_stride(Ny);
  const int m = blockIdx.x * kStageWarps + wq;
  const unsigned long long drop = l2_drop();
  {
    const int q = threadIdx.x & 3, mq = blockIdx.x * kStageWarps + q;
    if (mq < NM) {
      const ModeSlot ms = mode_slot(mq, NKX, a.NZ1, paired);
      const double2* src = R + ms.tile * Ny * kLanes + ms.lane;
      for (int y = threadIdx.x >> 2; y < Ny; y += 8 * kStageWarps) {
#pragma unroll
        for (int cpt = 0; cpt < 3; ++cpt)
          cp_async16_l2(sm + q * SS + cpt * Ny + y, src + cpt * cs + (long long)y * kLanes, drop);
      }
    }
    cp_async_commit();
  }
  const bool act = m < NM;
  const long long CS = (long long)NM * Ny, mo = (long long)m * Ny;
  const int iz = m / NKX, ix = m % NKX;
  double2 vj[3][YR];
  double c1[YR], c2[YR], e1[YR], e2[YR];
  auto load = [&](int k, int y) {
#pragma unroll
    for (int cpt = 0; cpt < 3; ++cpt) vj[cpt][k] = vel_j[cpt * CS + mo + y];
    c1[k] = a.v1[mo + y];
    c2[k] = a.v2[mo + y];
    e1[k] = a.q1[mo + y];
    e2[k] = a.q2[mo + y];
  };
#pragma unroll
  for (int k = 0; k < YM; ++k) {
    const int y = lane + 32 * k;
    if (act && y < Ny) load(k, y);
  }
  cp_async_wait_all();
  __syncthreads();
  if (!act) return;  // no CTA-wide barrier below
  const double kx = a.kx[ix], kz = a.kz[iz];
  const double k2 = kx * kx + kz * kz;
  const double2 *ra = sm + wq * SS, *va = ra + Ny;
  // Stages 4-5: wall divergence and influence-matrix weights
  double2 dw0 = make_double2(0.0, 0.0), dw1 = dw0;
#pragma unroll
  for (int i = 0; i < S1; ++i) {
    const double b0 = a.d1_w[i], b1 = a.d1_w[(Ny - 1) * S1 + i];
    const double2 x0 = va[a.d1_j0[0] + i], x1 = va[a.d1_j0[Ny - 1] + i];
    dw0.x += b0 * x0.x;
    dw0.y += b0 * x0.y;
    dw1.x += b1 * x1.x;
    dw1.y += b1 * x1.y;
  }
  if (k2 == 0.0) dw0 = make_double2(0.0, 0.0);
  const double* Mi = a.M_inv + (long long)m * 4;
  const double2 a1 = make_double2(-(Mi[0] * dw0.x + Mi[1] * dw1.x),
                                  -(Mi[0] * dw0.y + Mi[1] * dw1.y));
  const double2 a2 = make_double2(-(Mi[2] * dw0.x + Mi[3] * dw1.x),
                                  -(Mi[2] * dw0.y + Mi[3] * dw1.y));
  // Stage 6: assemble, store, correction norm
  const double km = (ix == 0 && a.kx0) ? 1.0 : 2.0;
  const int nk = YM > 0 ? YM : (Ny + 31) / 32;
  double acc = 0.0;
#pragma unroll
  for (int kk = 0; kk < nk; ++kk) {
    const int y = lane + 32 * kk, k = YM > 0 ? kk : 0;
    if (y >= Ny) continue;
    if (YM == 0) load(0, y);
    const double2 vnew = cadd(cadd(va[y], cscale(a1, c1[k])), cscale(a2, c2[k]));
    const double2 qq = cadd(cscale(a1, e1[k]), cscale(a2, e2[k]));
    const double2 unew = csub(ra[y], cik(kx, qq));
    const double2 wnew = csub(ra[2 * Ny + y], cik(kz, qq));
    const double2 cu = csub(unew, vj[0][k]);
    const double2 cv = csub(vnew, vj[1][k]);
    const double2 cw = csub(wnew, vj[2][k]);
    vel_new[mo + y] = unew;
    vel_new[CS + mo + y] = vnew;
    vel_new[2 * CS + mo + y] = wnew;
    if (corr_out) {
      corr_out[mo + y] = cu;
      corr_out[CS + mo + y] = cv;
      corr_out[2 * CS + mo + y] = cw;
    }
    acc += a.simpson[y] * km *
           ((cu.x * cu.x + cu.y * cu.y) + (cv.x * cv.x + cv.y * cv.y) +
            (cw.x * cw.x + cw.y * cw.y));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if (lane == 0 && partials) partials[m] = acc;
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
size_t imm_batch_stage_smem(int Ny) {
  return sizeof(double2) * (size_t)(stage_stride(Ny) * kStageWarps);
}

static size_t imm_batch_assemble_smem(int Ny) {
  return sizeof(double2) * (size_t)(assemble_stride(Ny) * kStageWarps);
}

// Rows per lane of the stage kernel (odd): 32 lanes cover Ny rows.  17 rows (289 to
// 512 points) do not fit the registers (255, 1.9 KB of spills); the iteration is still
// far ahead of the single-kernel form there: 64 x 301 x 64 at order 6 2487 -> 573 us, 48
// x 401 x 48 at order 4 2390 -> 432, 24 x 511 x 24 at order 4 1302 -> 327.
constexpr int kMaxNy = 512;  // four modes' rows fit in shared memory
// Back substitution with pre-scaled U (see the substitution kernel's comment).
constexpr int kMaxScaled = 160;
bool imm_batch_scaled(int Ny) { return Ny <= kMaxScaled; }
int imm_batch_rows(int Ny) {
  return Ny <= 96 ? 3 : Ny <= 160 ? 5 : Ny <= 224 ? 7 : Ny <= 288 ? 9 : 17;
}

bool imm_batch_supported(int kl, int ny) {
  return (kl == 2 || kl == 4 || kl == 6 || kl == 8) && ny <= kMaxNy;
}

// First row of lane l's window of W = (p + 2) + YM - 1 rows.
static int window_base(int Ny, int p, const int* j01, const int* j02, int l) {
  const int YM = imm_batch_rows(Ny), W = p + 2 + YM - 1, y = std::min(YM * l, Ny - 1);
  return std::max(0, std::min(std::min(j01[y], j02[y]), Ny - W));
}

// Window-relative stencil weights of the stage kernel: base[l] = window_base, and
// w1x / w2x[(o W + i) 32 + l] is the weight of window row i in D1 / D2 of row YM l + o
// (0 outside the stencil and past the last row).
void imm_batch_windows(int Ny, int p, const int* j01, const double* w1, const int* j02,
                       const double* w2, std::vector<int>* base, std::vector<double>* w1x,
                       std::vector<double>* w2x) {
  const int YM = imm_batch_rows(Ny), S1 = p + 1, S2 = p + 2, W = S2 + YM - 1;
  base->assign(32, 0);
  w1x->assign((size_t)YM * W * 32, 0.0);
  w2x->assign((size_t)YM * W * 32, 0.0);
  for (int l = 0; l < 32; ++l) {
    const int b = window_base(Ny, p, j01, j02, l);
    (*base)[l] = b;
    for (int o = 0; o < YM && YM * l + o < Ny; ++o) {
      const int y = YM * l + o;
      for (int m = 0; m < S1; ++m)
        (*w1x)[(size_t)(o * W + j01[y] + m - b) * 32 + l] = w1[y * S1 + m];
      for (int m = 0; m < S2; ++m)
        (*w2x)[(size_t)(o * W + j02[y] + m - b) * 32 + l] = w2[y * S2 + m];
    }
  }
}

// Every stencil of a lane's rows lies in its window: true where D1's start a row
// after D2's or with them, as they do centred in the interior (D2's even width
// either way) and shifted to stay inside the walls.
bool imm_batch_windows_ok(int Ny, int p, const int* j01, const int* j02) {
  const int YM = imm_batch_rows(Ny), S1 = p + 1, S2 = p + 2, W = S2 + YM - 1;
  for (int y = 0; y < Ny; ++y) {
    const int b = window_base(Ny, p, j01, j02, y / YM);
    if (j01[y] < b || j02[y] < b || j01[y] + S1 > b + W || j02[y] + S2 > b + W) return false;
  }
  return true;
}

// Ring slot bytes of one substitution launch: the larger of a forward block
// (factors, pivots) and a back-substitution block (U records), plus the
// entering rows of every component; and the ring depth that fits.
static int solve_slot_bytes(int kl, int nu, int ncomp) {
  const int W = kl + 1, WB = nu + 1, nup = (nu + 2) & ~1;
  const int MW = W > WB ? W : WB;
  const int f = W * kl * kTile * 8 + W * kTile;
  const int b = WB * nup * kTile * 8;
  return (((f > b ? f : b) + 127) & ~127) + ncomp * MW * kLanes * 16;
}

static int solve_ring(int kl, int nu, int ncomp, int max_smem) {
  const int sb = solve_slot_bytes(kl, nu, ncomp);
  if (3 * sb <= max_smem && 3 * sb <= 100 * 1024) return 3;
  if (2 * sb <= max_smem) return 2;
  return 0;
}

bool imm_batch_fits(int kl, int nu, int max_smem) {
  return solve_ring(kl, nu, 3, max_smem) > 0 && solve_ring(kl, nu, 1, max_smem) > 0;
}

template <int KL>
static cudaError_t solve_launch(const ImmBatch& bt, int op, double2* X, long long cs, int ncomp,
                                int Ny, const int* skip, cudaStream_t st) {
  SolveArgs s{};
  s.skip = skip;
  s.facL = bt.facL[op];
  s.facU = bt.facU[op];
  s.dp = bt.dp[op];
  s.X = X;
  s.cs = cs;
  s.status = bt.status;
  s.Ny = Ny;
  s.ncomp = ncomp;
  s.ring = solve_ring(KL, bt.nu, ncomp, bt.max_smem);
  s.slot_bytes = solve_slot_bytes(KL, bt.nu, ncomp);
  s.wait_limit = bt.wait_limit;
  if (s.ring == 0) return cudaErrorInvalidValue;
  const size_t sm = (size_t)s.ring * s.slot_bytes;
  const int grid = (bt.NP + kTile - 1) / kTile;
  // Never dependent on the kernel before: the one or two CTAs an SM has room for
  // would gather on the SMs that finish first (96 x 71 x 108 corrector: 97 us
  // so, 110 us with dependent substitutions).
  // Real and imaginary columns on lanes of their own shorten a step's chain but
  // run twice the warps: faster for the wide bands while every CTA has an SM to
  // itself (corrector, kl = 6: 48 x 49 x 48 49.5 -> 45.4 us, 64 x 65 x 64 62.5 ->
  // 59.8, 96 x 97 x 96 113.1 -> 109.3; kl = 8, 64 x 65 x 64: 70.0 -> 63.1).  On more
  // tiles it loses (128 x 129 x 128 193.7 -> 195.1 us), as it does at kl = 4 (32 x
  // 53 x 36 predict_and_correct 131.4 -> 133.7 us).
  constexpr int SC = kSplitCols<KL>;
  const bool split = SC == 1 && grid <= bt.sms;
  const int threads = 32 * ((split ? 2 : 1) * ncomp + 1);
  const void* kernel = imm_batch_scaled(Ny) ? imm_solve_fn<true>(KL, bt.nu, split)
                                            : imm_solve_plain(KL, bt.nu, split);
  void* args[] = {&s};
  return cudaLaunchKernel(kernel, dim3(grid), dim3(threads), args, sm, st);
}

template <int K>
static cudaError_t pipeline(const ImmArgs& a, const ImmBatch& bt, const double2* vel_n,
                           const double2* vel_j, const double2* nl_n, const double2* nl_j,
                           double2* vel_new, double2* corr_out, double* partials,
                           cudaStream_t st) {
  const int NM = a.NZ1 * a.NKX, Ny = a.Ny;
  const int grid = (NM + kStageWarps - 1) / kStageWarps, threads = 32 * kStageWarps;
  const int tiles = (bt.NP + kTile - 1) / kTile;
  const long long cs = (long long)tiles * Ny * kLanes;
  const size_t sm = imm_batch_stage_smem(Ny), sm6 = imm_batch_assemble_smem(Ny);
  cudaError_t e;
#define DNSB_STAGE013(YM)                                                              \
  case YM:                                                                             \
    launch_dep(a.dep, imm_stage013_kernel<K, YM>, grid, threads, sm, st, a, bt.paired, \
               bt.w1x, bt.w2x, bt.base, vel_n, nl_n, nl_j, bt.F, bt.R, cs);            \
    break;
  switch (imm_batch_rows(Ny)) {
    DNSB_STAGE013(3) DNSB_STAGE013(5) DNSB_STAGE013(7) DNSB_STAGE013(9) DNSB_STAGE013(17)
  }
#undef DNSB_STAGE013
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  e = solve_launch<K>(bt, 0, bt.F, 0, 1, Ny, a.skip, st);
  if (e != cudaSuccess) return e;
  const dim3 gg((Ny - 2 + kGradRows - 1) / kGradRows, tiles);
  launch_dep(a.dep, imm_grad_kernel<K>, gg, kLanes * kGradRows, 0, st, a, bt.paired, bt.NP, bt.F,
             bt.R, cs);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  e = solve_launch<K>(bt, 1, bt.R, cs, 3, Ny, a.skip, st);
  if (e != cudaSuccess) return e;
  auto* stage6 = Ny <= 96    ? imm_stage6_kernel<K, 3>
                 : Ny <= 160 ? imm_stage6_kernel<K, 5>
                             : imm_stage6_kernel<K, 0>;
  launch_dep(a.dep, stage6, grid, threads, sm6, st, a, bt.paired, bt.R, cs, vel_j, vel_new,
             corr_out, partials);
  return cudaGetLastError();
}

// Five launches: stages 0-1, L_k solve, stage 3, H_k solve, stages 4-6.
cudaError_t launch_imm_batch(const ImmArgs& a, const ImmBatch& bt, const double2* vel_n,
                             const double2* vel_j, const double2* nl_n,
                             const double2* nl_j, double2* vel_new, double2* corr_out,
                             double* partials, cudaStream_t st) {
  switch (a.kl) {
    case 2: return pipeline<2>(a, bt, vel_n, vel_j, nl_n, nl_j, vel_new, corr_out, partials, st);
    case 4: return pipeline<4>(a, bt, vel_n, vel_j, nl_n, nl_j, vel_new, corr_out, partials, st);
    case 6: return pipeline<6>(a, bt, vel_n, vel_j, nl_n, nl_j, vel_new, corr_out, partials, st);
    case 8: return pipeline<8>(a, bt, vel_n, vel_j, nl_n, nl_j, vel_new, corr_out, partials, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t set_imm_batch_attributes(int max_smem, int Ny) {
  cudaError_t e = cudaSuccess;
  auto allow = [&](const void* f) {
    const cudaError_t r = allow_dynamic_smem(f, max_smem);
    if (r != cudaSuccess) e = r;
  };
#define DNSB_IMM_STAGES(K)                                                            \
  for (const void* f :                                                                \
       {(const void*)imm_stage013_kernel<K, 3>, (const void*)imm_stage013_kernel<K, 5>, \
        (const void*)imm_stage013_kernel<K, 7>, (const void*)imm_stage013_kernel<K, 9>, \
        (const void*)imm_stage013_kernel<K, 17>, (const void*)imm_stage6_kernel<K, 0>}) \
    allow(f);
  DNSB_IMM_STAGES(2) DNSB_IMM_STAGES(4) DNSB_IMM_STAGES(6) DNSB_IMM_STAGES(8)
#undef DNSB_IMM_STAGES
  for (int kl : {2, 4, 6, 8})
    for (int nu : {kl + 1, 2 * kl})
      for (bool split : {false, true})
        allow(imm_batch_scaled(Ny) ? imm_solve_fn<true>(kl, nu, split)
                                   : imm_solve_plain(kl, nu, split));
  return e;
}

}  // namespace dnsb
