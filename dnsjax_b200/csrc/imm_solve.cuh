// The influence-matrix iteration's batched banded substitution kernel, in two
// translation units (csrc/imm_batch.cu, csrc/imm_solve_plain.cu).
#pragma once

#include "common.cuh"

namespace dnsb {

namespace {

constexpr int kTile = 16;       // items per substitution CTA (two sides per item)
constexpr int kLanes = 2 * kTile;  // lanes of a tile row (two sides)
constexpr int kRowDoubles = 2 * kLanes;
// Real columns of a substitution lane on few tiles, by bandwidth (see solve_launch).
template <int KL>
constexpr int kSplitCols = KL >= 6 ? 1 : 2;

}  // namespace

// ---------------------------------------------------------------------------
// Batched banded substitution: one CTA per tile of 16 items, one warp per
// component (1 for L_k: p_P; 3 for H_k) and one copying warp; lane = (side,
// item) (lanes 0-15 the items' own modes, 16-31 their mirrors), and each thread
// solves both real columns (re, im) of its mode's component as two recurrences
// sharing every factor load, or, on few tiles of wide bands, one of them (COLS
// below); the warps share the tile's factor stream.  Lane 0
// of the copying warp streams each block of steps -- its factors and pivots and,
// per component, the right-hand-side rows that enter the windows during the
// block, each one contiguous bulk copy -- into a ring of shared-memory slots
// (`full` barriers, by bytes); the component warps hand a slot back one by one
// (`empty` barriers), so no warp waits for another but for the data.  Lanes of
// no mode (padding items, the mirror side of s = 0 or of unpaired items) run on
// the workspace's zeros.
//
// Forward elimination (dgbtrs 'N'): windows b[j..j+KL] in registers,
// slot(o, ph) = (o + ph) % W, W = KL + 1; the row interchange is chosen per
// block for the warp: none, with the next row only (two selects), or
// general (switch).  Back substitution: windows b[j-NU..j], slot(o, ph) =
// (o - ph) mod WB, WB = NU + 1.  Its rows are the forward results, read back by
// bulk copies: every lane fences its stores towards the copies' proxy before the
// copying warp is told.
//
// Up to 160 points U is pre-scaled by 1/U_jj, so that a step is one FMA deep (128 x
// 129 x 128 corrector 191.9 us; plain 195.4).  Above, x_j = b_j / U_jj is formed
// first and multiplies the plain U, as dgbtrs and the single-kernel form do: it
// costs nothing there (96 x 193 x 72 predict_and_correct 622 us either way), and
// L_k, whose condition grows with the points, shows the rounding.  Its share of a
// corrector update's error in the mean mode against an 80-bit solution, over
// heights of 161 to 257 points and kl 4 and 6 (emulated, 98 matrices): pre-scaled
// 1.15-1.17 times dgbtrs', plain 1.02; whole updates on the GPU (36, geometric
// mean): dgbtrs 1.7e-14, plain 1.9e-14, pre-scaled 2.9e-14.
// A wait that does not complete within its bound sets bit 2 of the status word
// and the CTA stops computing.
// ---------------------------------------------------------------------------

struct SolveArgs {
  const double* facL;
  const double* facU;
  const unsigned char* dp;
  double2* X;    // [ncomp][tiles][Ny][32]
  long long cs;  // component stride of X
  int* status;
  int Ny, ncomp, ring, slot_bytes;
  int wait_limit;  // polls before a wait gives up (the drain after it uses kDrainPolls)
  const int* skip;  // non-null and *skip != 0: return at once (ImmArgs::skip)
};

__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
// Global -> shared bulk copy (this GPU's memory, no multicast).
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes,
                                         unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
      ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait for a ring slot: false if it did not complete within
// `limit` polls.
constexpr int kDrainPolls = 1 << 20;
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity, int limit) {
  for (int it = 0; it < limit; ++it)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

// Row interchange of step ph (pivot offset d) on one window.
template <int KL, int MODE>
__device__ __forceinline__ double pivot_take(double (&w)[KL + 1], int ph, int d) {
  constexpr int W = KL + 1;
  double bpj = w[ph % W];
  if (MODE == 1) {
    const double x1 = w[(1 + ph) % W];
    const bool p = d != 0;
    w[(1 + ph) % W] = p ? bpj : x1;
    bpj = p ? x1 : bpj;
  } else if (MODE == 2) {
    switch (d) {
#define DNSB_PIV(I)                  \
  case I:                            \
    if (I <= KL) {                   \
      bpj = w[(I + ph) % W];         \
      w[(I + ph) % W] = w[ph % W];   \
    }                                \
    break;
      DNSB_PIV(1) DNSB_PIV(2) DNSB_PIV(3) DNSB_PIV(4)
      DNSB_PIV(5) DNSB_PIV(6) DNSB_PIV(7) DNSB_PIV(8)
#undef DNSB_PIV
      default: break;
    }
  }
  return bpj;
}

// A lane's element of a tile row, re and im or one of them, as COLS doubles.
__device__ __forceinline__ void put(double* g, const double (&v)[2], unsigned long long pol) {
  st_l2(reinterpret_cast<double2*>(g), make_double2(v[0], v[1]), pol);
}
__device__ __forceinline__ void put(double* g, const double (&v)[1], unsigned long long pol) {
  st_l2(g, v[0], pol);
}
template <int N>
__device__ __forceinline__ void get(double (&w)[2][N], int i, const double2 v) {
  w[0][i] = v.x;
  w[1][i] = v.y;
}
template <int N>
__device__ __forceinline__ void get(double (&w)[1][N], int i, double v) {
  w[0][i] = v;
}
template <int COLS>
using lane_elem = std::conditional_t<COLS == 2, double2, double>;

template <int KL, int MODE, bool TAIL, int COLS>
__device__ __forceinline__ void tile_fwd_block(double* col, int j0, int nsteps, int Ny,
                                               double (&w)[COLS][KL + 1], const double2* Lp,
                                               const int (&dr)[KL + 1], const double* ent,
                                               unsigned long long pol) {
  constexpr int W = KL + 1;
  using E = lane_elem<COLS>;
#pragma unroll
  for (int ph = 0; ph < W; ++ph) {
    const int j = j0 + ph;
    if (!TAIL || j < nsteps) {
      double L[KL];
#pragma unroll
      for (int i2 = 0; i2 < KL / 2; ++i2) {
        const double2 t = Lp[(ph * (KL / 2) + i2) * kTile];
        L[2 * i2] = t.x;
        L[2 * i2 + 1] = t.y;
      }
      double bp[COLS];
#pragma unroll
      for (int c = 0; c < COLS; ++c) bp[c] = pivot_take<KL, MODE>(w[c], ph, dr[ph]);
      put(col + j * kRowDoubles, bp, pol);
#pragma unroll
      for (int c = 0; c < COLS; ++c) {
#pragma unroll
        for (int i = 1; i <= KL; ++i) w[c][(i + ph) % W] -= L[i - 1] * bp[c];
      }
      // b[j+W] enters at offset KL (0 past the last row)
      get(w, ph % W, j + W < Ny ? *reinterpret_cast<const E*>(ent + ph * kRowDoubles) : E{});
    }
  }
}

template <int NU, bool TAIL, int COLS, bool SCALED>
__device__ __forceinline__ void tile_bwd_block(double* col, int j0, double (&w)[COLS][NU + 1],
                                               const double2* Up, const double* ent,
                                               unsigned long long pol) {
  using E = lane_elem<COLS>;
  constexpr int WB = NU + 1, NUP = (NU + 2) & ~1;
#pragma unroll
  for (int ph = 0; ph < WB; ++ph) {
    const int j = j0 - ph;
    if (!TAIL || j >= 0) {
      const double2* u = Up + (WB - 1 - ph) * (NUP / 2) * kTile;
      double U[NUP];
#pragma unroll
      for (int i2 = 0; i2 < NUP / 2; ++i2) {
        const double2 t = u[i2 * kTile];
        U[2 * i2] = t.x;
        U[2 * i2 + 1] = t.y;
      }
      const int st = ((NU - ph) % WB + WB) % WB;
      double bj[COLS], x[COLS];
#pragma unroll
      for (int c = 0; c < COLS; ++c) {
        bj[c] = w[c][st];
        x[c] = bj[c] * U[0];
      }
      put(col + j * kRowDoubles, x, pol);
#pragma unroll
      for (int i = 1; i <= NU; ++i) {
        const int si = ((NU - i - ph) % WB + WB) % WB;
#pragma unroll
        for (int c = 0; c < COLS; ++c) w[c][si] -= U[i] * (SCALED ? bj[c] : x[c]);
      }
      // b[j-WB] enters at offset 0 (0 below row 0); rows in ascending order
      get(w, st,
          j - WB >= 0 ? *reinterpret_cast<const E*>(ent + (WB - 1 - ph) * kRowDoubles) : E{});
    }
  }
}

constexpr int kMaxRing = 4;

// COLS: real columns of a lane, 2 (one warp per component, lane = (side, item)) or
// 1 (two warps per component, one for each side, lane = (item, re or im)).
// SCALED: facU is pre-scaled (imm_batch_scaled).
template <int KL, int NU, int COLS, bool SCALED>
__global__ void __launch_bounds__(COLS == 2 ? 128 : 224)
imm_solve_kernel(SolveArgs a) {
  if (a.skip && *a.skip) return;  // before any barrier is set up
  constexpr int W = KL + 1, WB = NU + 1, NUP = (NU + 2) & ~1;
  constexpr int LB = W * KL * kTile * 8, PB = W * kTile, UB = WB * NUP * kTile * 8;
  constexpr int MW = W > WB ? W : WB;  // entering rows of a component in a slot
  constexpr int RB = kLanes * 16;      // bytes of a tile row
  extern __shared__ __align__(128) unsigned char ring[];
  __shared__ __align__(8) unsigned long long full[kMaxRing], empty[kMaxRing], fwd_done;
  __shared__ int s_fail;
  constexpr int WPC = 3 - COLS;  // warps per component
  using E = lane_elem<COLS>;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cw = warp / WPC;
  const int it = COLS == 2 ? lane & (kTile - 1) : lane >> 1;
  const long long tile = blockIdx.x;
  const int Ny = a.Ny, R = a.ring, SB = a.slot_bytes, nc = a.ncomp;
  const int E0 = SB - nc * MW * RB;  // entering rows, at the slot's end
  const long long NyF = Ny + W, NyB = Ny + WB;
  const int nsteps = Ny - 1;
  const int nbf = (nsteps + W - 1) / W;  // forward blocks
  const int nbb = (Ny + WB - 1) / WB;    // back-substitution blocks
  const int nblk = nbf + nbb;
  double2* X = a.X + tile * Ny * kLanes;

  if (tid == 0) {
    for (int r = 0; r < R; ++r) {
      mbar_init(&full[r], 1);
      mbar_init(&empty[r], WPC * nc);
    }
    mbar_init(&fwd_done, WPC * nc);
    mbar_fence_init();
    s_fail = 0;
  }
  __syncthreads();
  volatile int* fail = &s_fail;

  if (warp == WPC * nc) {
    if (lane != 0) return;
    // Blocks 0 .. nblk-1 into slot g % R: forward blocks hold the factors and
    // pivots of steps j0 .. j0+W-1 and rows j0+W .. j0+2W-1; back-substitution
    // blocks U records j0-WB+1 .. j0 and rows j0-2WB+1 .. j0-WB, those that
    // exist.
    int g = 0;
    bool ok = true;
    for (; g < nblk; ++g) {
      if (g >= R) ok = mbar_wait(&empty[g % R], (g / R - 1) & 1, a.wait_limit);
      if (ok && g == nbf) ok = mbar_wait(&fwd_done, 0, a.wait_limit);
      if (!ok || *fail) break;
      unsigned char* slot = ring + (g % R) * SB;
      unsigned long long* bar = &full[g % R];
      const bool fwd = g < nbf;
      const int j0 = fwd ? g * W : Ny - 1 - (g - nbf) * WB;
      const int first = fwd ? j0 + W : j0 - 2 * WB + 1;  // row of the slot's first entry
      const int lo = max(first, 0), hi = min(fwd ? j0 + 2 * W : j0 - WB + 1, Ny);
      const int rows = max(hi - lo, 0);
      mbar_arrive_tx(bar, (fwd ? LB + PB : UB) + rows * RB * nc);
      if (fwd) {
        bulk_g2s(slot, a.facL + (tile * NyF + j0) * KL * kTile, LB, bar);
        bulk_g2s(slot + LB, a.dp + (tile * NyF + j0) * kTile, PB, bar);
      } else {
        bulk_g2s(slot, a.facU + (tile * NyB + j0 + 1) * NUP * kTile, UB, bar);
      }
      if (rows > 0)
        for (int c = 0; c < nc; ++c)
          bulk_g2s(slot + E0 + (c * MW + lo - first) * RB, X + c * a.cs + (long long)lo * kLanes,
                   rows * RB, bar);
    }
    if (!ok) {
      *fail = 1;
      atomicOr(a.status, 2);
    }
    // Leave no bulk copy in flight, whether the other warps take them or gave
    // up: wait for the blocks issued last (a slot's earlier blocks were taken
    // before it was filled again).
    for (int h = max(g - R, 0); h < g; ++h) mbar_wait(&full[h % R], (h / R) & 1, kDrainPolls);
    return;
  }

  const unsigned long long keep = l2_keep();
  const int at = (warp % WPC) * kLanes + lane * COLS;  // the lane's double in a tile row
  double* col = reinterpret_cast<double*>(X + cw * a.cs) + at;
  int g = 0;
  bool ok = true;
  auto take = [&] {  // wait for block g
    ok = mbar_wait(&full[g % R], (g / R) & 1, a.wait_limit) && !*fail;
    ok = __all_sync(0xffffffffu, ok);
    if (!ok && lane == 0) {
      *fail = 1;
      atomicOr(a.status, 2);
    }
    return ok;
  };
  auto give = [&] {  // block g's slot back
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[g % R]);
  };

  // ---- forward elimination, steps j = 0 .. Ny-2 ----
  {
    double w[COLS][W];
#pragma unroll
    for (int o = 0; o < W; ++o)
      get(w, o, o < Ny ? ld_l2(reinterpret_cast<const E*>(col + o * kRowDoubles), keep) : E{});
    for (int k = 0; k < nbf; ++k, ++g) {
      if (!take()) break;
      const unsigned char* slot = ring + (g % R) * SB;
      const double2* Lp = reinterpret_cast<const double2*>(slot) + it;
      const unsigned char* Ps = slot + LB;
      const double* ent = reinterpret_cast<const double*>(slot + E0 + cw * MW * RB) + at;
      int dr[W];
      int dm = 0;
#pragma unroll
      for (int ph = 0; ph < W; ++ph) {
        dr[ph] = Ps[ph * kTile + it];
        dm = max(dm, dr[ph]);
      }
      dm = __reduce_max_sync(0xffffffffu, dm);
      const int j0 = k * W;
      if (j0 + W > nsteps)
        tile_fwd_block<KL, 2, true, COLS>(col, j0, nsteps, Ny, w, Lp, dr, ent, keep);
      else if (dm == 0)
        tile_fwd_block<KL, 0, false, COLS>(col, j0, nsteps, Ny, w, Lp, dr, ent, keep);
      else if (dm == 1)
        tile_fwd_block<KL, 1, false, COLS>(col, j0, nsteps, Ny, w, Lp, dr, ent, keep);
      else
        tile_fwd_block<KL, 2, false, COLS>(col, j0, nsteps, Ny, w, Lp, dr, ent, keep);
      give();
    }
    // b[Ny-1] sits at offset 0 after the last step: slot nsteps % W.
    const int last = nsteps % W;
    double v[COLS];
#pragma unroll
    for (int c = 0; c < COLS; ++c) {
      v[c] = w[c][0];
#pragma unroll
      for (int t = 1; t < W; ++t)
        if (last == t) v[c] = w[c][t];
    }
    if (ok) {
      put(col + (Ny - 1) * kRowDoubles, v, keep);
      // the forward results are read back by bulk copies (async proxy)
      asm volatile("fence.proxy.async;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&fwd_done);
    }
  }

  // ---- back substitution, rows j = Ny-1 .. 0 ----
  if (ok) {
    double w[COLS][WB];
#pragma unroll
    for (int o = 0; o < WB; ++o) {
      const int idx = Ny - 1 - NU + o;
      get(w, o, idx >= 0 ? ld_l2(reinterpret_cast<const E*>(col + idx * kRowDoubles), keep) : E{});
    }
    for (int k = 0; k < nbb; ++k, ++g) {
      if (!take()) break;
      const unsigned char* slot = ring + (g % R) * SB;
      const double2* Up = reinterpret_cast<const double2*>(slot) + it;
      const double* ent = reinterpret_cast<const double*>(slot + E0 + cw * MW * RB) + at;
      const int j0 = Ny - 1 - k * WB;
      if (j0 - WB + 1 < 0)
        tile_bwd_block<NU, true, COLS, SCALED>(col, j0, w, Up, ent, keep);
      else
        tile_bwd_block<NU, false, COLS, SCALED>(col, j0, w, Up, ent, keep);
      give();
    }
  }
}

// The kernel of a bandwidth, stored superdiagonals (kl + 1 or 2 kl) and lanes
// (split: kSplitCols<KL> columns a lane).
template <int KL, bool SCALED>
const void* imm_solve_fn(int nu, bool split) {
  constexpr int SC = kSplitCols<KL>;
  if (nu == KL + 1)
    return split ? (const void*)imm_solve_kernel<KL, KL + 1, SC, SCALED>
                 : (const void*)imm_solve_kernel<KL, KL + 1, 2, SCALED>;
  return split ? (const void*)imm_solve_kernel<KL, 2 * KL, SC, SCALED>
               : (const void*)imm_solve_kernel<KL, 2 * KL, 2, SCALED>;
}
template <bool SCALED>
const void* imm_solve_fn(int kl, int nu, bool split) {
  switch (kl) {
    case 2: return imm_solve_fn<2, SCALED>(nu, split);
    case 4: return imm_solve_fn<4, SCALED>(nu, split);
    case 6: return imm_solve_fn<6, SCALED>(nu, split);
    case 8: return imm_solve_fn<8, SCALED>(nu, split);
    default: return nullptr;
  }
}
// imm_solve_fn<false> (csrc/imm_solve_plain.cu).
const void* imm_solve_plain(int kl, int nu, bool split);

}  // namespace dnsb
