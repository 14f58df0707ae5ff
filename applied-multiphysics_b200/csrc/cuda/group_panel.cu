// Group panel of the FP64 factors (the FP32 ones': group_panel_f32.cu; Cholesky, LDL^T with static pivot perturbation,
// LDL^T with Bunch-Kaufman pivots inside each pivot block): the pivot blocks of a group of 64-column blocks of a front
// factored in one dataflow launch -- POTRF of each pivot block, TRSM of the rows below it, and the update of the group's
// remaining columns. The products run on the FP64 tensor cores (mma.sync m8n8k4).
//
// What bounds it: the chain through the pivot blocks of the large fronts (POTRF of block b, then block b + 1's rows
// against it, then their update and POTRF), one CTA at a time, so a block's latency is what counts: per block POTRF
// 11,200 clocks, the flag and the loads behind it 3,300, TRSM 2,500, the block's own update 1,600 (FP64; 33,700 / - /
// 10,400 / 7,100 with FMA tiles and a four-thread substitution per row). A 4,096-row front's group of two blocks takes
// 32 us (66 before), eight of them at once 63 us (110). The split: warp w
// of a strip owns 8 rows (row group rg(w)) of every 64 x 64 product, so a strip's TRSM runs inside each warp without a
// barrier -- the C fragment of a solved 8 x 8 tile is the A fragment of the next product (its two registers are the k
// indices 2 t and 2 t + 1, and the B fragment takes the same pair with one 16-byte load).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "../host/plan.hpp"
#include "devplan.cuh"
#include "launch.hpp"
#include "panel_blocks.cuh"
#include "pivot_steps.cuh"

namespace amp {

namespace {

// Rows [i0, i0 + nr) x columns [j0, j0 + ncol) of a front's column-major block (ld m) into S; lower: only the entries
// on and below the diagonal. The rest is zero, and with pad the diagonal entries from ncol on are one. Read through
// L2 (another CTA of the running launch may have written them). 8 rows x 4 columns per warp access.
__device__ __forceinline__ void load_block(double *S, const double *L, int m, int i0, int nr, int j0, int ncol, bool lower,
                                           bool pad) {
  const int lane = threadIdx.x & 31, i = 8 * (threadIdx.x >> 5) + (lane >> 2), t = lane & 3;
  double v[16];
#pragma unroll
  for (int e = 0; e < 16; e++) {
    const int c = 4 * e + t;
    v[e] = (i < nr && c < ncol && (!lower || c <= i)) ? __ldcg(L + (int64_t)(j0 + c) * m + i0 + i) : 0.0;
  }
#pragma unroll
  for (int e = 0; e < 16; e++) {
    const int c = 4 * e + t;
    S[sw(i, c)] = pad && i == c && i >= ncol ? 1.0 : v[e];
  }
}

// Pivot block: POTRF (or LDL^T) of the 64 x 64 diagonal block of a front, called by all 256 threads of a CTA.
// Ds: the updated block (lower part; identity from column w on), left unchanged; Lp: the block's
// (0, 0) entry in the front (ld m), where the factor is written; w <= 64 its columns; scr: 11 step buffers; Linv:
// the inverses of the eight 8 x 8 diagonal blocks of L (64 doubles each, row-major), for the strips' TRSM.
// Right-looking on the unscaled columns in steps of eight. Step k: (1) the first two warps, one row per lane, factor the
// 8 x 8 diagonal tile redundantly in registers -- so no value of the pivot chain crosses lanes -- and eliminate their
// own row with it, publishing -a and a / d; (2) after a barrier the warps of the row groups below (C fragments of their
// trailing tiles in registers) update their tile of the next eight columns and hand it over; (3) after a second barrier
// they update the rest of the triangle while the first two warps go on with step k + 1. The chain per column is one
// reciprocal (the hardware estimate and three dependent products) and two products, 58 clocks (FP64); a step's FP64
// issue in a panel warp takes 790 clocks alone and 1,050-1,200 beside the trailing products. The pivots are tested, the
// columns scaled and everything written after the last step. A block takes 11,200 clocks
// (33,700 with 4 x 4 register tiles, a diagonal thread per step and two barriers per four columns).
// Cholesky tests d > 0 (sparse.mjs:1151-1156); LDL^T (ldlt.mjs:450-562) perturbs |d| < tau to +-tau by the sign of d (a
// non-finite small pivot fails) and counts negative and perturbed pivots. Cholesky L = a / sqrt(d) with sqrt(d) on the
// diagonal, LDL^T L = a / d with a unit diagonal (D to ld.D). Returns 0, or 1 (status set for the first failing column
// f + c0 + k, nothing written) when a pivot failed. LB (the Bunch-Kaufman fast path): returns 2, writing nothing, when
// a multiplier |L(i, k)| of the block exceeds lbound or a pivot was perturbed.
template <bool LDLT, bool LB>
__device__ int potrf_block(const double *Ds, double *scr, double *Lp, double *Linv, int m, int w, int f, int c0, int s,
                           unsigned long long *status, const LdltArgs<double> &ld, double lbound) {
  constexpr int CL = kColLd, kStepBuf = kPanel * CL;
  __shared__ double scale[kPanel], diag[kPanel];
  __shared__ int failAt, redo, nNeg, nPert, inexact;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3, rg = row_group(warp);
  const int nk = (w + 7) >> 3;  // steps: the columns from w on are the identity's
  const double tau = LDLT ? ld.scal[1] : 0.0;
  double *R = scr, *Q = R + kStepBuf, *P = R + 3 * kStepBuf;  // Q: two buffers; P: -a of every step
  const int myRow = (8 * rg + g) * CL + 2 * t;
  auto tile = [&](int cb, double(&c)[2]) {  // this warp's tile (rg, cb) of the block
    const double2 v = pair_at(Ds, 8 * rg + g, 8 * cb + 2 * t);
    c[0] = v.x;
    c[1] = v.y;
  };
  auto hand_over = [&](const double(&c)[2]) {
    double2 v;
    v.x = c[0];
    v.y = c[1];
    *reinterpret_cast<double2 *>(R + myRow) = v;
  };
  auto panel = [&](auto exact) {  // the first two warps, a row per lane
    bool fine = true;
    for (int k = 0; k < nk; k++) {
      if (8 * k + 32 * warp < kPanel)
        fine &= eliminate8<decltype(exact)::value, LDLT, false>(R, P + k * kStepBuf, Q + (k & 1) * kStepBuf, 8 * k,
                                                               min(8 * k + 32 * warp + lane, kPanel - 1), 8, tau);
      __syncthreads();
      if (k == 0 && warp == 1) {  // row group 1's only trailing tile
        double c[2];
        tile(1, c);
        step_tile(c, P + 8 * CL, Q + 8 * CL, CL, g, t);
        hand_over(c);
      }
      __syncthreads();
    }
    if (!fine) inexact = 1;
  };
  auto trailing = [&]() {  // the other warps
    double c[7][2];  // at step k: the tiles (rg, k + 1), (rg, k + 2), ...
#pragma unroll
    for (int j = 0; j < 7; j++) {
      c[j][0] = c[j][1] = 0.0;
      if (j < rg) tile(j + 1, c[j]);
    }
    for (int k = 0; k < nk; k++) {
      __syncthreads();
      const double *Pk = P + k * kStepBuf + 8 * rg * CL, *Qk = Q + (k & 1) * kStepBuf;
      if (rg > k) {
        step_tile(c[0], Pk, Qk + 8 * (k + 1) * CL, CL, g, t);
        hand_over(c[0]);
      }
      __syncthreads();
      if (rg > k + 1) {
#pragma unroll
        for (int j = 1; j < 7; j++) {
          if (k + 1 + j <= rg) step_tile(c[j], Pk, Qk + 8 * (k + 1 + j) * CL, CL, g, t);
          c[j - 1][0] = c[j][0];
          c[j - 1][1] = c[j][1];
        }
      }
    }
  };
  for (int pass = 0; pass < 2; pass++) {
    double first[2];
    tile(0, first);
    hand_over(first);
    if (tid == 0) {
      failAt = kPanel;  // none
      redo = nNeg = nPert = inexact = 0;
    }
    __syncthreads();
    if (warp >= 2)
      trailing();
    else if (pass == 0)
      panel(std::false_type());
    else
      panel(std::true_type());
    __syncthreads();
    if (!inexact) break;  // (the second pass sets it never)
    __syncthreads();
  }
  // the pivots: test and count, the columns' scales
  if (tid < kPanel) {
    double d = -P[(tid >> 3) * kStepBuf + tid * CL + (tid & 7)];
    bool bad = false, small = false;
    if (LDLT) {
      small = tid < w && !(fabs(d) >= tau);
      bad = small && !isfinite(d);
      if (small) d = d < 0.0 ? -tau : tau;
      const int neg = __popc(__ballot_sync(0xffffffffu, tid < w && d < 0.0));
      const int pert = __popc(__ballot_sync(0xffffffffu, small));
      if (lane == 0) {
        atomicAdd(&nNeg, neg);
        atomicAdd(&nPert, pert);
        if (LB && pert) redo = 1;
      }
    } else {
      bad = tid < w && !(d > 0.0);
    }
    const unsigned mask = __ballot_sync(0xffffffffu, bad);
    if (lane == 0 && mask) atomicMin(&failAt, 32 * warp + __ffs(mask) - 1);
    const double dl = LDLT ? d : sqrt(d);
    diag[tid] = dl;
    scale[tid] = 1.0 / dl;
  }
  __syncthreads();
  if (LB) {  // the multipliers a / d of the strictly lower part (a failed pivot exceeds the bound too)
    for (int e = tid; e < kPanel * kPanel; e += 256) {
      const int r = e & (kPanel - 1), j = e >> 6;
      if (r > j && r < w && !(fabs(P[(j >> 3) * kStepBuf + r * CL + (j & 7)]) <= lbound * fabs(diag[j]))) redo = 1;
    }
    __syncthreads();
    if (redo) return 2;
  }
  if (failAt < kPanel) {
    if (tid == 0) atomicMin(status, status_word(f + c0 + failAt, LDLT ? 2 : 1, s));
    return 1;
  }
  if (warp >= 2) {  // the columns: a lane per row, eight columns at a time
    const int r = tid & (kPanel - 1);
    for (int p = (tid >> 6) - 1; p < 8; p += 3) {
      if (r < 8 * p || r >= w) continue;
      const double *Pr = P + p * kStepBuf + r * CL;
      double *dst = Lp + (int64_t)(8 * p) * m + r;
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; u += 2) {
        const double2 a = *reinterpret_cast<const double2 *>(Pr + u);
        v[u] = -a.x * scale[8 * p + u];
        v[u + 1] = -a.y * scale[8 * p + u + 1];
      }
#pragma unroll
      for (int u = 0; u < 8; u++)
        if (r >= 8 * p + u) dst[(int64_t)u * m] = r > 8 * p + u ? v[u] : LDLT ? 1.0 : diag[r];
    }
  } else {  // column j of inv(L_pp): forward substitution with the unit block, rows over the diagonal
    const int p = min(tid >> 3, nk - 1), j = tid & 7;  // (the strips use the first nk blocks)
    const double *Pp = P + p * kStepBuf + 8 * p * CL;
    double x[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      double v = 0.0;
#pragma unroll
      for (int u = 0; u < i; u++) {
        const double sc = scale[8 * p + u];
        v += (Pp[i * CL + u] * (LDLT ? sc : sc * sc)) * x[u];
      }
      x[i] = i < j ? 0.0 : i == j ? 1.0 : v;  // (P holds -a)
    }
    double r2 = 0.0;  // squared norm of row j of the scaled block
#pragma unroll
    for (int u = 0; u < 7; u++) {
      const double a = u < j ? Pp[j * CL + u] : 0.0, l = a * scale[8 * p + u];
      r2 += LDLT ? fabs(a * l) : l * l;
    }
    r2 += LDLT ? fabs(diag[8 * p + j]) : diag[8 * p + j] * diag[8 * p + j];
    unsigned top = 0;  // high word of the largest X(i, j)^2 / |d_i| (Cholesky: |X(i, j)|); above all numbers for NaN
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const double sc = scale[8 * p + i], z = LDLT ? x[i] : x[i] * sc;
      Linv[64 * p + 8 * i + j] = z;
      top = max(top, (unsigned)__double2hiint(LDLT ? z * (z * sc) : z) & 0x7fffffffu);
    }
    const double z2 = __hiloint2double((int)top, 0);
    const bool wild = !((LDLT ? z2 : z2 * z2) * r2 <= kInvBound * kInvBound);
    put_wild(Linv, 1, wild);
  }
  if (LDLT) {
    if (tid < w) ld.D[f + c0 + tid] = diag[tid];
    if (tid == 0) {
      atomicAdd(ld.counts, nNeg);
      atomicAdd(ld.counts + 1, nPert);
    }
  }
  return 0;
}

// |x| as an integer of the same order, 0 for what is not a number
__device__ __forceinline__ unsigned long long mag_key(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
  return b <= 0x7ff0000000000000ull ? b : 0ull;
}
// the largest of the lanes' keys
__device__ __forceinline__ unsigned long long warp_max_key(unsigned long long v) {
  const unsigned hi = (unsigned)(v >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)v : 0u);
  return (unsigned long long)mh << 32 | ml;
}
// 1 / d from the reciprocal estimate (two roundings), or the quotient where the estimate has no range; the same d in every
// lane
__device__ __forceinline__ double fast_recip(double d) {
  double x, f;
  return recip_parts<false>(d, x, f) ? x * f : 1.0 / d;
}

// Bunch-Kaufman LDL^T of a pivot block, the pivot search restricted to the block's w columns (so the supernode
// partition and every row structure stay the reference's): at column k, with colmax = max_{i>k} |B(i, k)| (row r),
// a 1 x 1 pivot k when |B(k, k)| >= alpha colmax or |B(k, k)| rowmax >= alpha colmax^2 (rowmax = max_{j != r}
// |B(r, j)|), a 1 x 1 pivot r when |B(r, r)| >= alpha rowmax, else the 2 x 2 pivot (k, r); alpha = (1 + sqrt 17) / 8
// (Bunch and Kaufman, Math. Comp. 31, 1977). Each interchange is applied to the block's whole rows, the L columns
// already computed included, so that P B P^T = L D L^T with L unit lower triangular (L(k + 1, k) = 0 inside a 2 x 2
// pivot, whose off-diagonal is D(k + 1, k)). A column with no entry at or above tau keeps the reference's static
// perturbation (|d| < tau -> -+tau, a non-finite one fails; ldlt.mjs:513-522).
// S: 64 x 65 doubles of shared workspace (a full symmetric copy, S[j][i] = B(i, j)); Ds: the updated block (lower part),
// overwritten by L. Writes L to Lp (ld m), D, Doff and piv, adds the inertia (a 2 x 2 pivot with a
// negative determinant has one negative eigenvalue, with a positive one two when its diagonal is negative) and the
// perturbed count. Returns false (status set) on a non-finite pivot; nothing is written then. Called by every thread.
//
// What bounds it is the latency of a column's step, so a step has two barriers: the rows stay where they are and only
// their positions in the pivot order change (two rows per lane, in every warp), every warp finds the pivot by itself, and a
// pivot's columns stay unscaled in S once they are chosen. Thread (i, q) holds the entries S[q + 4 u][i] in registers and
// stores those that the step has changed. With physical interchanges, one warp choosing and five barriers per column, the
// panels of the edge-element system with 13 elements per edge took 4.49 ms, now 2.56 ms (a full block 67,000 clocks).
__device__ bool bk_block(double *Ds, double (*S)[kPanel + 1], double *Lp, double *Linv, int m, int w, int f, int c0, int s,
                         unsigned long long *status, const LdltArgs<double> &ld) {
  __shared__ int sPerm[kPanel];
  __shared__ double sD[kPanel], sE[kPanel];
  __shared__ double sT[kPanel], sG[kPanel];  // 1 x 1: 1 / d, -; 2 x 2 (k, k + 1): t / e twice, c and a
  const int tid = threadIdx.x, lane = tid & 31, i = tid & (kPanel - 1), q = tid >> 6;
  const double tau = ld.scal[1];
  const double alpha = 0.64038820320220756;  // (1 + sqrt(17)) / 8
  constexpr unsigned kAll = 0xffffffffu;
  double v[16];
#pragma unroll
  for (int u = 0; u < 16; u++) {
    const int j = q + 4 * u;
    v[u] = (i < w && j < w) ? (i >= j ? Ds[sw(i, j)] : Ds[sw(j, i)]) : 0.0;
    S[j][i] = v[u];
  }
  // positions of the rows lane and lane + 32 in the pivot order (-1: not a row of the block)
  int p0 = lane < w ? lane : -1, p1 = lane + 32 < w ? lane + 32 : -1;
  auto row_at = [&](int pos) {
    const unsigned a = __ballot_sync(kAll, p0 == pos), b = __ballot_sync(kAll, p1 == pos);
    return a ? __ffs(a) - 1 : 31 + __ffs(b);
  };
  auto exchange = [&](int pa, int pb) {  // the rows at positions pa and pb
    p0 = p0 == pa ? pb : p0 == pb ? pa : p0;
    p1 = p1 == pa ? pb : p1 == pb ? pa : p1;
  };
  int failAt = -1, nNeg = 0, nPert = 0;
  __syncthreads();
  for (int k = 0; k < w;) {
    const int c = row_at(k);
    const unsigned long long x0 = p0 > k ? mag_key(S[c][lane]) : 0ull, x1 = p1 > k ? mag_key(S[c][lane + 32]) : 0ull;
    const unsigned long long xm = warp_max_key(max(x0, x1));
    const double colmax = __longlong_as_double((long long)xm), absakk = fabs(S[c][c]);
    int step = 1, r = c, posR = k;  // r: the row of the larger pivot, at position posR
    if (colmax > 0.0 && !(absakk >= alpha * colmax)) {  // (a NaN diagonal goes on too, and fails at its own turn)
      const unsigned at0 = (p0 > k && x0 == xm) ? (unsigned)p0 : ~0u, at1 = (p1 > k && x1 == xm) ? (unsigned)p1 : ~0u;
      posR = (int)__reduce_min_sync(kAll, min(at0, at1));  // the first in the pivot order
      r = row_at(posR);
      const unsigned long long y0 = (p0 >= k && lane != r) ? mag_key(S[lane][r]) : 0ull;
      const unsigned long long y1 = (p1 >= k && lane + 32 != r) ? mag_key(S[lane + 32][r]) : 0ull;
      const double rm = __longlong_as_double((long long)warp_max_key(max(y0, y1)));
      if (absakk * rm >= alpha * colmax * colmax)
        r = c, posR = k;
      else if (!(fabs(S[r][r]) >= alpha * rm))
        step = 2;
    }
    exchange(k + step - 1, posR);
    const int k1 = k + step;
    const unsigned long long live =  // the rows still to be eliminated
        (unsigned long long)__ballot_sync(kAll, p0 >= k1) | ((unsigned long long)__ballot_sync(kAll, p1 >= k1) << 32);
    // bit 4 u: entry u of this thread changes (what is computed for the others is not read again)
    const unsigned long long store = live >> i & 1 ? live >> q : 0ull;
    if (step == 1) {
      double d = S[r][r];
      const double ci = S[r][i];
      const bool small = !(fabs(d) >= tau);
      if (small && isfinite(d)) d = d < 0.0 ? -tau : tau;
      if (tid == 0) {
        sD[k] = d;
        sE[k] = 0.0;
      }
      if (!isfinite(d)) {  // the same for every thread
        failAt = k;
        break;
      }
      nNeg += d < 0.0 ? 1 : 0;
      nPert += small ? 1 : 0;
      const double inv = fast_recip(d);  // L takes the exact quotient below
      double cj[16];
#pragma unroll
      for (int u = 0; u < 16; u++) cj[u] = S[r][q + 4 * u] * inv;
      __syncthreads();  // every warp has chosen
#pragma unroll
      for (int u = 0; u < 16; u++) {
        v[u] -= ci * cj[u];
        if (store >> (4 * u) & 1) S[q + 4 * u][i] = v[u];
      }
    } else {
      // D_k = e [[a, 1], [1, c]], D_k^-1 = (t / e) [[c, -1], [-1, a]] with a = d11 / e, c = d22 / e, t = 1 / (a c - 1)
      const double d11 = S[c][c], e21 = S[c][r], d22 = S[r][r];
      const double ci0 = S[c][i], ci1 = S[r][i];
      const double ie = fast_recip(e21), aa = d11 * ie, cc = d22 * ie, te = fast_recip(aa * cc - 1.0) * ie;
      if (tid == 0) {
        sD[k] = d11;
        sD[k + 1] = d22;
        sE[k] = e21;
        sE[k + 1] = 0.0;
      }
      if (!(isfinite(te) && isfinite(aa) && isfinite(cc))) {
        failAt = k;
        break;
      }
      nNeg += aa * cc - 1.0 < 0.0 ? 1 : (d11 < 0.0 ? 2 : 0);
      __syncthreads();  // every warp has chosen
      const double l1 = te * (cc * ci0 - ci1), l2 = te * (aa * ci1 - ci0);
#pragma unroll
      for (int u = 0; u < 16; u++) v[u] -= l1 * S[c][q + 4 * u] + l2 * S[r][q + 4 * u];
#pragma unroll
      for (int u = 0; u < 16; u++)
        if (store >> (4 * u) & 1) S[q + 4 * u][i] = v[u];
    }
    __syncthreads();
    k = k1;
  }
  if (failAt >= 0) {
    if (tid == 0) atomicMin(status, status_word(f + c0 + failAt, 2, s));
    return false;
  }
  if (tid < 32) {
    if (p0 >= 0) sPerm[p0] = lane;
    if (p1 >= 0) sPerm[p1] = lane + 32;
  } else if (tid >= 64 && tid < 64 + w) {
    const int j = tid - 64;
    const double en = sE[j], ep = j > 0 ? sE[j - 1] : 0.0;
    if (en != 0.0 || ep != 0.0) {
      const int a = en != 0.0 ? j : j - 1;
      const double aa = sD[a] / sE[a], cc = sD[a + 1] / sE[a];
      sT[j] = (1.0 / (aa * cc - 1.0)) / sE[a];
      sG[j] = a == j ? cc : aa;
    } else {
      sT[j] = 1.0 / sD[j];
    }
  }
  __syncthreads();
  // L in the pivot order, thread (i, q) columns q + 4 u (entries of the pivots' unscaled columns); to Ds as [column][row]
  const int ri = i < w ? sPerm[i] : 0;
#pragma unroll
  for (int u = 0; u < 16; u++) {
    const int j = q + 4 * u;
    double x = i == j ? 1.0 : 0.0;
    if (i < w && j < i) {
      const double en = sE[j], ep = j > 0 ? sE[j - 1] : 0.0;
      if (en != 0.0 || ep != 0.0) {
        const int o = en != 0.0 ? j + 1 : j - 1;  // the 2 x 2 pivot's other column
        x = i == o ? 0.0 : sT[j] * (sG[j] * S[sPerm[j]][ri] - S[sPerm[o]][ri]);
      } else {
        x = S[sPerm[j]][ri] * sT[j];
      }
    }
    if (i < w && j <= i) Lp[(int64_t)j * m + i] = x;
    Ds[kPanel * j + i] = x;
  }
  __syncthreads();
  if (tid < kPanel) {  // the inverses of the diagonal 8 x 8 blocks of the unit L, for the strips' TRSM
    const int p = tid >> 3, j = tid & 7;
    double x[8];
#pragma unroll
    for (int ii = 0; ii < 8; ii++) {
      double z = 0.0;
#pragma unroll
      for (int u = 0; u < ii; u++) z += Ds[kPanel * (8 * p + u) + 8 * p + ii] * x[u];
      x[ii] = ii < j ? 0.0 : ii == j ? 1.0 : -z;
      Linv[64 * p + 8 * ii + j] = x[ii];
    }
    // multipliers are bounded here, so the block itself stands for its scaled form
    double r2 = 1.0;
    bool wild = false;
#pragma unroll
    for (int u = 0; u < 7; u++) {
      const double l = u < j ? Ds[kPanel * (8 * p + u) + 8 * p + j] : 0.0;
      r2 += l * l;
    }
#pragma unroll
    for (int ii = 0; ii < 8; ii++) wild |= !(x[ii] * x[ii] * r2 <= kInvBound * kInvBound);
    put_wild(Linv, 1, wild);
  }
  if (tid < w) {
    ld.D[f + c0 + tid] = sD[tid];
    ld.Doff[f + c0 + tid] = sE[tid];
    ld.piv[f + c0 + tid] = sPerm[tid];
  }
  if (tid == 0) {
    atomicAdd(ld.counts, nNeg);
    atomicAdd(ld.counts + 1, nPert);
  }
  return true;
}

// C(8 x 64 of this warp) += N S^T: N the warp's A fragments (8 x 64), S a block in shared memory. Eight independent
// accumulators between two products of one.
__device__ __forceinline__ void update_row_group(double (&c)[8][2], const double (&n)[8][2], const double *S, int g,
                                                 int t) {
#pragma unroll
  for (int q = 0; q < 8; q++) {
    double2 v[8];
#pragma unroll
    for (int p = 0; p < 8; p++) v[p] = pair_at(S, 8 * p + g, 8 * q + 2 * t);
#pragma unroll
    for (int p = 0; p < 8; p++) mma884(c[p], n[q][0], v[p].x);
#pragma unroll
    for (int p = 0; p < 8; p++) mma884(c[p], n[q][1], v[p].y);
  }
}

// Row g of w = c L_pp^-T by substitution, L_pp the p-th 8 x 8 diagonal block of the pivot block Ls, 1 / L(k, k) on the
// diagonal of its inverse; lane t of the row holds entries 2 t and 2 t + 1.
__device__ __forceinline__ void substitute8(const double (&c)[2], double (&w)[2], const double *Ls, const double *Li, int p,
                                            int g, int t) {
  double x0 = c[0], x1 = c[1];
#pragma unroll 1
  for (int k = 0; k < 8; k++) {
    const double v = __shfl_sync(0xffffffffu, k & 1 ? x1 : x0, 4 * g + (k >> 1)) * Li[64 * p + 9 * k];
    if (2 * t == k) w[0] = v;
    if (2 * t + 1 == k) w[1] = v;
    x0 -= v * Ls[sw(8 * p + 2 * t, 8 * p + k)];  // (nothing reads an entry after its own step)
    x1 -= v * Ls[sw(8 * p + 2 * t + 1, 8 * p + k)];
  }
}

// One group of pivot blocks [g0, g1) of a front, a strip of up to 64 rows per CTA, CTAs ordered by an atomic ticket
// (the diagonal strips of every item first, then the strips below the group). A strip takes the group's pivot blocks b
// in order (a diagonal strip those before its own), left-looking:
//   its rows of block b receive the earlier blocks q: C -= sum W_q X_q^T (summed by itself, as the own block's update below:
//   products added to C one by one would each be rounded at C's size), with W_q its own solved rows and X_q the rows of
//   diagonal strip b, waited for by D[b] >= q + 1 (the last W_q is still in registers, earlier ones are read back);
//   then, after P[b], they are solved against the pivot block: W = C L_bb^-T by 8 x 8 blocks with the inverses of its
//   diagonal blocks (Cholesky X = W; LDL^T with the unit L_bb, X = W D^-1; Bunch-Kaufman the columns in the block's
//   pivot order first, then the 1 x 1 and 2 x 2 inverses of D).
// A diagonal strip keeps its own pivot block in shared memory from the start, publishes D[j] = b + 1 after each solve,
// subtracts W X^T from the block's lower part, and after its last solve factors it and publishes P[j].
// Every wait is on a strip with a smaller ticket, which runs to completion without waiting on a larger one, so the
// launch cannot deadlock whatever the number of resident CTAs. The columns right of the group receive the group's
// update afterwards (k_update / k_update_mx, K = the group). Failure (a pivot, a bounded wait) sets the status and
// releases P[b], so every waiter leaves.
constexpr int kBlockElems = kPanel * kPanel;
constexpr int kGroupSmem = 3 * kBlockElems * (int)sizeof(double);  // two CTAs per SM
template <bool LDLT, bool BK>
__global__ void __launch_bounds__(256, 2) k_group_panel(const GroupItem *__restrict__ items,
                                                        const StripTask *__restrict__ strips, int nstrips, int *ticket,
                                                        int *flags, DevPlan P, double *__restrict__ Lx,
                                                        double *__restrict__ Linv, unsigned long long *status,
                                                        LdltArgs<double> ld) {
  extern __shared__ __align__(16) unsigned char gp_raw[];
  double *Ls = reinterpret_cast<double *>(gp_raw);  // pivot block, rows of another diagonal strip, POTRF step buffers
  double *Xs = Ls + kBlockElems;                    // this strip's solved rows (Bunch-Kaufman: column exchange)
  double *Ds = Xs + kBlockElems;                    // a diagonal strip's own pivot block
  __shared__ __align__(16) double Li[8 * 64];
  __shared__ double dv[kPanel], dinv[kPanel];
  __shared__ double dB[BK ? kPanel : 1];
  __shared__ int dP[BK ? kPanel : 1], sPiv[BK ? kPanel : 1];
  __shared__ int sTicket, sWild;
  if (threadIdx.x == 0) sTicket = factor_failed(status) ? nstrips : atomicAdd(ticket, 1);
  __syncthreads();
  const int tk = sTicket;
  if (tk >= nstrips) return;
  const StripTask st = strips[tk];
  const GroupItem it = items[st.item];
  const int s = it.s, g0 = it.g0, g1 = it.g1;
  const int f = P.snF[s], m = P.snM[s];
  const int nb = (g1 - g0 + kPanel - 1) / kPanel;
  const int r0 = st.r0, r1 = st.r1, jd = st.diag;
  const int bmax = jd >= 0 ? jd : nb;  // pivot blocks whose rows below include this strip
  const int64_t lxp = P.snLxp[s];
  double *L = Lx + lxp;
  int *Pf = flags + it.flag0, *Df = Pf + nb;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int lr = 8 * row_group(warp) + g, row = r0 + lr;  // this lane's row of every fragment
  const bool act = row < r1;
  if (jd >= 0) load_block(Ds, L, m, r0, r1 - r0, r0, r1 - r0, true, true);
  double nx[8][2];  // -W of the block solved last
#pragma unroll
  for (int p = 0; p < 8; p++) nx[p][0] = nx[p][1] = 0.0;
  for (int b = 0; b < bmax; b++) {
    const int c0 = g0 + b * kPanel, w = min(kPanel, g1 - c0);
    double x[8][2];  // the strip's rows of block b
    const double *src = L + (int64_t)(c0 + 2 * t) * m + row;
#pragma unroll
    for (int p = 0; p < 8; p++)
#pragma unroll
      for (int u = 0; u < 2; u++)
        x[p][u] = act && 8 * p + 2 * t + u < w ? __ldcg(src + (int64_t)(8 * p + u) * m) : 0.0;
    for (int q = 0; q < b; q++) {
      const int cq = g0 + q * kPanel;
      if (b > 1) {  // read the strip's solved rows back (with one earlier block they are still in registers)
#pragma unroll
        for (int p = 0; p < 8; p++)
#pragma unroll
          for (int u = 0; u < 2; u++) {
            const int cc = cq + 8 * p + 2 * t + u;  // (every pivot block before the last of a group is full)
            double v = 0.0;
            if (act) {
              const int64_t at = (int64_t)cc * m + row;
              v = BK ? __ldcg(ld.W + lxp + at) : __ldcg(L + at);
              if (LDLT && !BK) v *= __ldcg(ld.D + f + cc);
            }
            nx[p][u] = -v;
          }
      }
      if (!panel_wait(Df + b, q + 1, status, P.spin)) return;
      if (q == 0) {  // the products are summed by themselves (see above); after the wait's barrier nobody reads Xs any more
#pragma unroll
        for (int p = 0; p < 8; p++) {
          set_pair(Xs, lr, 8 * p + 2 * t, x[p][0], x[p][1]);
          x[p][0] = x[p][1] = 0.0;
        }
      }
      load_block(Ls, L, m, c0, w, cq, kPanel, false, false);
      __syncthreads();
      update_row_group(x, nx, Ls, g, t);
    }
    if (b > 0) {
#pragma unroll
      for (int p = 0; p < 8; p++) {
        const double2 v = pair_at(Xs, lr, 8 * p + 2 * t);
        x[p][0] += v.x;
        x[p][1] += v.y;
      }
    }
    if (!panel_wait(Pf + b, 1, status, P.spin)) return;  // (its barrier: every warp is done with Ls)
    load_block(Ls, L, m, c0, w, c0, w, true, true);
    if (tid < kPanel) {
      if constexpr (BK) {
        double a = 1.0, bb = 0.0;
        int pc = tid;
        if (tid < w) {
          const double *D = ld.D + f + c0, *E = ld.Doff + f + c0;
          const double d = __ldcg(D + tid), en = __ldcg(E + tid), ep = tid > 0 ? __ldcg(E + tid - 1) : 0.0;
          if (en != 0.0 || ep != 0.0) {  // 2 x 2 pivot (tid, tid + 1) or (tid - 1, tid): the inverse as in bk_block
            const bool first = en != 0.0;
            const double e = first ? en : ep;
            const double d11 = first ? d : __ldcg(D + tid - 1), d22 = first ? __ldcg(D + tid + 1) : d;
            const double aa = d11 / e, cc = d22 / e, te = (1.0 / (aa * cc - 1.0)) / e;
            a = te * (first ? cc : aa);
            bb = -te;
            pc = first ? tid + 1 : tid - 1;
          } else {
            a = 1.0 / d;
          }
        }
        dinv[tid] = a;
        dB[tid] = bb;
        dP[tid] = pc;
        sPiv[tid] = tid < w ? __ldcg(ld.piv + f + c0 + tid) : tid;
      } else if constexpr (LDLT) {
        const double d = tid < w ? __ldcg(ld.D + f + c0 + tid) : 1.0;
        dv[tid] = d;
        dinv[tid] = 1.0 / d;
      }
    }
    const double *Lb = Linv + ((int64_t)(it.flag0 / 2) + b) * linv_stride(1);
    *reinterpret_cast<double2 *>(Li + 2 * tid) = __ldcg(reinterpret_cast<const double2 *>(Lb + 2 * tid));
    if (tid == 0) sWild = wild_blocks(Lb, 1);
    __syncthreads();
    if constexpr (BK) {  // the strip's columns in the block's pivot order (each warp exchanges its own rows)
#pragma unroll
      for (int p = 0; p < 8; p++) set_pair(Xs, lr, 8 * p + 2 * t, x[p][0], x[p][1]);
      __syncwarp();
#pragma unroll
      for (int p = 0; p < 8; p++)
#pragma unroll
        for (int u = 0; u < 2; u++) x[p][u] = Xs[sw(lr, sPiv[8 * p + 2 * t + u])];
      __syncwarp();
    }
    // W = C L_bb^-T, right-looking over the 8-column blocks: solved with the block's inverse (by substitution where that is
    // large), then subtracted from the later ones
    auto solve = [&](auto some, const int wild) {
#pragma unroll
      for (int p = 0; p < 8; p++) {
        if (8 * p >= w) break;  // x is zero from column w on
        double wv[2] = {0.0, 0.0};
        if (decltype(some)::value && wild >> p & 1) {
          substitute8(x[p], wv, Ls, Li, p, g, t);
        } else {
          const double2 iv = *reinterpret_cast<const double2 *>(Li + 64 * p + 8 * g + 2 * t);
          mma884(wv, x[p][0], iv.x);
          mma884(wv, x[p][1], iv.y);
        }
        x[p][0] = wv[0];
        x[p][1] = wv[1];
#pragma unroll
        for (int p2 = p + 1; p2 < 8; p2++) {
          if (8 * p2 >= w) break;
          const double2 l = pair_at(Ls, 8 * p2 + g, 8 * p + 2 * t);
          mma884(x[p2], -wv[0], l.x);
          mma884(x[p2], -wv[1], l.y);
        }
      }
    };
    if (sWild == 0)
      solve(std::false_type(), 0);
    else
      solve(std::true_type(), sWild);
    if constexpr (BK) {
#pragma unroll
      for (int p = 0; p < 8; p++) set_pair(Xs, lr, 8 * p + 2 * t, x[p][0], x[p][1]);
      __syncwarp();
    }
    // x := L21's entries; nx := -W (W = x D for LDL^T)
#pragma unroll
    for (int p = 0; p < 8; p++)
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int cc = 8 * p + 2 * t + u;
        const double wv = x[p][u];
        double xv = wv;
        if constexpr (BK)
          xv = dinv[cc] * wv + dB[cc] * Xs[sw(lr, dP[cc])];
        else if constexpr (LDLT)
          xv = wv * dinv[cc];
        x[p][u] = xv;
        nx[p][u] = BK ? -wv : LDLT ? -x[p][u] * dv[cc] : -x[p][u];
        if (BK && act && cc < w) ld.W[lxp + (int64_t)(c0 + cc) * m + row] = wv;
      }
    if constexpr (BK) __syncwarp();
#pragma unroll
    for (int p = 0; p < 8; p++) set_pair(Xs, lr, 8 * p + 2 * t, x[p][0], x[p][1]);
    __syncthreads();
    // written column by column, a warp's lanes on consecutive rows (the fragments hold 8-row pieces of a column)
    for (int cc = warp; cc < w; cc += 8) {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int r = lane + 32 * h;
        if (r0 + r >= r1) continue;
        const double xv = Xs[sw(r, cc)];
        const int64_t at = (int64_t)(c0 + cc) * m + r0 + r;
        L[at] = xv;
        if (LDLT && !BK && ld.W) ld.W[lxp + at] = xv * dv[cc];
      }
    }
    if (jd < 0) continue;
    panel_release(Df + jd, b + 1);
    // the strip's own pivot block: tiles (rg, 0 .. rg) of D -= W X^T, two at a time
    for (int nt = 0; nt <= lr >> 3; nt += 2) {
      const bool two = nt + 1 <= lr >> 3;
      const int nb2 = two ? nt + 1 : nt;
      double ca[2] = {0.0, 0.0}, cb[2] = {0.0, 0.0};
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const double2 xa = pair_at(Xs, 8 * nt + g, 8 * q + 2 * t), xb = pair_at(Xs, 8 * nb2 + g, 8 * q + 2 * t);
        mma884(ca, nx[q][0], xa.x);
        if (two) mma884(cb, nx[q][0], xb.x);
        mma884(ca, nx[q][1], xa.y);
        if (two) mma884(cb, nx[q][1], xb.y);
      }
      const double2 va = pair_at(Ds, lr, 8 * nt + 2 * t), vb = pair_at(Ds, lr, 8 * nb2 + 2 * t);
      set_pair(Ds, lr, 8 * nt + 2 * t, va.x + ca[0], va.y + ca[1]);
      if (two) set_pair(Ds, lr, 8 * nt + 8 + 2 * t, vb.x + cb[0], vb.y + cb[1]);
    }
  }
  if (jd >= 0) {  // this strip's own pivot block, fully updated: factor it and publish it (also after a failure)
    const int c0 = g0 + jd * kPanel, w = min(kPanel, g1 - c0);
    double *Lp = L + (int64_t)c0 * m + c0;
    double *Lb = Linv + ((int64_t)(it.flag0 / 2) + jd) * linv_stride(1);
    __syncthreads();  // Ds complete (also when the strip had no earlier pivot block); Ls and Xs free
    if constexpr (BK) {
      // Bunch-Kaufman keeps every pivot of the block in place exactly when each multiplier is at most 1 / alpha in
      // magnitude and no pivot needs the perturbation: try the unpivoted LDL^T first, else redo the block with pivots
      // from its untouched entries
      const int r = potrf_block<true, true>(Ds, Ls, Lp, Lb, m, w, f, c0, s, status, ld, 1.0 / 0.64038820320220756);
      if (r == 2) {
        bk_block(Ds, reinterpret_cast<double(*)[kPanel + 1]>(gp_raw), Lp, Lb, m, w, f, c0, s, status, ld);
      } else if (r == 0 && tid < w) {  // the identity pivot order, 1 x 1 pivots
        ld.piv[f + c0 + tid] = tid;
        ld.Doff[f + c0 + tid] = 0.0;
      }
    } else {
      potrf_block<LDLT, false>(Ds, Ls, Lp, Lb, m, w, f, c0, s, status, ld, -1.0);
    }
    panel_release(Pf + jd, 1);
  }
}

}  // namespace

template <bool LDLT, bool BK>
static cudaError_t init_one() {
  return cudaFuncSetAttribute(k_group_panel<LDLT, BK>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGroupSmem);
}
cudaError_t init_group_panel_attributes() {
  cudaError_t e = init_one<false, false>();
  if (e == cudaSuccess) e = init_one<true, false>();
  if (e == cudaSuccess) e = init_one<true, true>();
  return e;
}

void launch_group_panel(const GroupItem *items, const StripTask *strips, int nstrips, int *ticket, int *flags,
                        const DevPlan &P, double *Lx, double *Linv, unsigned long long *status, const LdltArgs<double> &ld,
                        cudaStream_t st) {
  if (nstrips <= 0) return;
  auto run = [&](auto kernel) {
    kernel<<<(unsigned)nstrips, 256, kGroupSmem, st>>>(items, strips, nstrips, ticket, flags, P, Lx, Linv, status, ld);
  };
  if (ld.piv)
    run(k_group_panel<true, true>);  // Bunch-Kaufman pivot blocks
  else if (ld.scal)
    run(k_group_panel<true, false>);
  else
    run(k_group_panel<false, false>);
}

}  // namespace amp
