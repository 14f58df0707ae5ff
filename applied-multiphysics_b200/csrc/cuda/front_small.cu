// Small fronts: one warp (m <= 32, four or eight fronts per CTA) or one CTA (32 < m <= 128) per front does all of the
// front's work for its level, in one launch per level and size class:
//   zero the front, add A's entries of the pivot columns (sparse.mjs:965-973), extend-add the children's update
//   matrices in the reference's child order (sparse.mjs:974-985), factor the nc pivot columns right-looking over the
//   whole trailing triangle (Cholesky sparse.mjs:995-1098; LDL^T with static pivot perturbation ldlt.mjs:450-562, or
//   with Bunch-Kaufman pivots inside each 64-column block of the pivot columns), and
//   write the first nc columns to L (the reference layout) and the rest to the update matrix U (the arena).
// Such fronts dominate 2D problems (the batched heat set: median m = 5, 97% with m <= 32), where the general path's
// 64 x 64 pivot-block kernels and 128-row tiles would spend almost all of their work on padding, one launch per step.
// What bounds them is the latency of one front, level after level: a 99-row root front took 144 us with a barrier and
// two quotients per pivot column, 17 us now; a 76-row front with 15 pivots and two children 39 us, 17 now (about 5 us of
// it the launch); the small fronts of a 64 x 64 heat problem 1,344 us, 620 now.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "../host/plan.hpp"
#include "devplan.cuh"
#include "launch.hpp"
#include "pivot_steps.cuh"
#include "small_fronts.cuh"
#include "sync.cuh"

namespace amp {

// entries per lane in flight during the assembly, and CTAs per SM that the registers are held to: the m <= 16 class is
// bound by the warps in flight (157,000 leaves of a batch: 262 us at 98 registers and two CTAs per SM)
template <int MAXM>
constexpr int tiny_batch() {
  return MAXM <= kTinyMid ? 8 : 16;
}
template <int MAXM>
constexpr int tiny_ctas() {
  return MAXM <= kTinyMid ? 4 : 5;
}

// The children's row maps as well; a map's entries are front positions below 128
struct ChildMaps : ChildMeta {
  unsigned char map[kChildChunk][kSmallFront];
};

// The latency of a front's assembly is its chain of dependent loads (the children's metadata, their maps, their update
// matrices, one child after another), so the update matrices are read a batch ahead: while a batch of entries is
// added to the front, the next one (of the same child or of the next) is in flight, up to 16 entries per lane.

// Zero F (m x m, column-major), add A's entries of the pivot columns and the children's update matrices in the
// reference's order. One warp, m <= 32: a lane per row of the child.
template <int kBatch>
__device__ void assemble_warp(int s, const DevPlan &P, const double *__restrict__ values, const double *__restrict__ U,
                              double *F, int lane) {
  const int f = P.snF[s], nc = P.snNc[s], m = P.snM[s];
  const int q0 = P.chPtr[s], nch = P.chPtr[s + 1] - q0;
  const int p0 = P.asmColPtr[f], p1 = P.asmColPtr[f + nc];
  for (int e = lane; e < m * m; e += 32) F[e] = 0.0;
  __syncwarp();
  // A's entries of all nc pivot columns (one contiguous CSR range): slot dst = j m + i of the L panel, each (i, j) once
  for (int p = p0 + lane; p < p1; p += 32) F[P.asmDst[p]] += __ldg(values + P.asmSrc[p]);
  __syncwarp();  // other lanes add the children to these entries
  pdl_wait();  // the children's level
  for (int qb = 0; qb < nch; qb += 32) {  // the metadata of up to 32 children, one per lane
    const int nq = min(32, nch - qb);
    int muc = 0;
    int64_t ea = 0, uo = 0;
    if (lane < nq) {
      const int c = P.chList[q0 + qb + lane];
      muc = P.snM[c] - P.snNc[c];
      ea = P.eaPtr[c];
      uo = P.snUoff[c];
    }
    // batch (q, b0): columns [b0, b0 + kBatch) of child q, row a = lane; pos: the child row's front position
    auto fetch = [&](int q, int b0, double(&v)[kBatch], int &mq, int &pos) {
      mq = __shfl_sync(0xffffffffu, muc, q);
      const int64_t eq = __shfl_sync(0xffffffffu, ea, q), uq = __shfl_sync(0xffffffffu, uo, q);
      pos = lane < mq ? P.eaMap[eq + lane] : 0;
      const double *Uc = U + uq;
#pragma unroll
      for (int i = 0; i < kBatch; i++)
        v[i] = lane < mq && b0 + i <= lane ? Uc[(b0 + i) * mq + lane] : 0.0;
    };
    double v[kBatch], vn[kBatch];
    int mq = 0, pos = 0, mn = 0, pn = 0;
    fetch(0, 0, v, mq, pos);
    for (int q = 0, b0 = 0; q < nq;) {
      const int qn = b0 + kBatch < mq ? q : q + 1, bn = qn == q ? b0 + kBatch : 0;
      if (qn < nq) fetch(qn, bn, vn, mn, pn);
#pragma unroll
      for (int i = 0; i < kBatch; i++) {
        const int col = __shfl_sync(0xffffffffu, pos, min(b0 + i, 31));
        if (lane < mq && b0 + i <= lane) F[col * m + pos] += v[i];
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < kBatch; i++) v[i] = vn[i];
      mq = mn;
      pos = pn;
      q = qn;
      b0 = bn;
    }
  }
  __syncwarp();
}

// The same by a CTA of NT threads (m <= 128): warps over the child's columns, lanes over its rows. Ends with a barrier;
// false (in every thread) when the factorization has failed.
template <int NT>
__device__ bool assemble_cta(int s, const DevPlan &P, const double *__restrict__ values, const double *__restrict__ U,
                             double *F, ChildMaps *cm, const unsigned long long *status) {
  constexpr int NW = NT / 32;
  constexpr int kBatch = 16;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int f = P.snF[s], nc = P.snNc[s], m = P.snM[s];
  const int q0 = P.chPtr[s], nch = P.chPtr[s + 1] - q0;
  const int p0 = P.asmColPtr[f], p1 = P.asmColPtr[f + nc];
  auto metadata = [&](int qb, int nq) {
    if (t < nq) {
      const int c = P.chList[q0 + qb + t];
      cm->muc[t] = P.snM[c] - P.snNc[c];
      cm->ea[t] = P.eaPtr[c];
      cm->uo[t] = P.snUoff[c];
    }
  };
  metadata(0, min(kChildChunk, nch));
  for (int e = t; e < m * m; e += NT) F[e] = 0.0;
  __syncthreads();
  for (int p = p0 + t; p < p1; p += NT) F[P.asmDst[p]] += __ldg(values + P.asmSrc[p]);
  pdl_wait();  // the children's level
  const bool bad = t == 0 && factor_failed(status);  // one read for the CTA (sync.cuh), in time for the last barrier
  for (int qb = 0; qb < nch; qb += kChildChunk) {
    const int nq = min(kChildChunk, nch - qb);
    if (qb > 0) {
      metadata(qb, nq);  // (the last chunk's data is consumed: barrier below)
      __syncthreads();
    }
    // batch (q, i): rows [128 i' ..) of 4 of the warp's columns of child q: columns b = warp + NW (4 i + j), j < 4, rows
    // b + lane + 32 h, h < 4
    auto fetch = [&](int q, int i, double(&v)[kBatch]) {
      const int mq = cm->muc[q];
      const double *Uc = U + cm->uo[q];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int b = warp + NW * (4 * i + j);
#pragma unroll
        for (int h = 0; h < 4; h++) {
          const int a = b + lane + 32 * h;
          v[4 * j + h] = a < mq ? Uc[b * mq + a] : 0.0;
        }
      }
    };
    double v[kBatch], vn[kBatch];
    fetch(0, 0, v);
    for (int e = t; e < nq * kSmallFront; e += NT) {
      const int q = e / kSmallFront, a = e % kSmallFront;
      if (a < cm->muc[q]) cm->map[q][a] = (unsigned char)P.eaMap[cm->ea[q] + a];
    }
    __syncthreads();  // the maps; A's entries
    for (int q = 0, i = 0; q < nq;) {
      const int mq = cm->muc[q];
      const int qn = 4 * NW * (i + 1) < mq ? q : q + 1, in = qn == q ? i + 1 : 0;
      if (qn < nq) fetch(qn, in, vn);
      const unsigned char *map = cm->map[q];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int b = warp + NW * (4 * i + j);
        if (b >= mq) continue;
        double *col = F + map[b] * m;
#pragma unroll
        for (int h = 0; h < 4; h++) {
          const int a = b + lane + 32 * h;
          if (a < mq) col[map[a]] += v[4 * j + h];
        }
      }
      if (qn != q) __syncthreads();  // the next child adds to the same entries from other warps
#pragma unroll
      for (int j = 0; j < kBatch; j++) v[j] = vn[j];
      q = qn;
      i = in;
    }
  }
  return !__syncthreads_or(bad);
}

// The whole front of supernode s by one warp (m <= 32) over the shared m x m column-major tile F.
//
// Column k of the elimination is one phase with one barrier: every lane reads the pivot F(k, k) (final since the
// previous barrier), computes the same pivot decision and scale, writes its share of L's column k straight to Lx and
// updates its share of the trailing triangle from the unscaled column k, which nobody writes in the phase. The
// arithmetic is the column-scaled form's: l_i = F(i, k) / r (Cholesky, r = sqrt F(k, k)) or F(i, k) / d (LDL^T), and
// F(i, j) -= l_i (l_j d) with d = 1 for Cholesky.
template <int MAXM>
__device__ void factor_front_warp(int s, const DevPlan &P, const double *__restrict__ values, double *__restrict__ Lx,
                                  double *__restrict__ U, double *F, unsigned long long *status, const LdltArgs<double> &la,
                                  int lane) {
  const int f = P.snF[s], nc = P.snNc[s], m = P.snM[s], mu = m - nc;
  const bool ldlt = la.scal != nullptr;
  const double tau = ldlt ? la.scal[1] : 0.0;
  assemble_warp<tiny_batch<MAXM>()>(s, P, values, U, F, lane);
  if (warp_failed(status)) return;
  int neg = 0, pert = 0;  // lane 0
  double *Lp = Lx + P.snLxp[s];
  for (int k = 0; k < nc; k++) {
    double d = F[k * m + k], inv, dk, diag;
    if (ldlt) {
      int n1 = 0, p1 = 0;
      const bool ok = small_ldlt_pivot(d, tau, n1, p1);
      if (!ok) {
        if (lane == 0) atomicMin(status, status_word(f + k, 2, s));
        return;  // warp-uniform: every lane saw the same pivot
      }
      if (lane == 0) {
        neg += n1;
        pert += p1;
        la.D[f + k] = d;
      }
      dk = d;
      inv = 1.0 / d;
      diag = 1.0;
    } else {
      if (!(d > 0.0)) {
        if (lane == 0) atomicMin(status, status_word(f + k, 1, s));
        return;  // warp-uniform
      }
      const double r = sqrt(d);
      dk = 1.0;
      inv = 1.0 / r;
      diag = r;
    }
    const double *Fk = F + k * m;
    const int i = lane;  // the lane's row
    const double li = i < m ? Fk[i] * inv : 0.0;
    if (i >= k && i < m) Lp[(int64_t)k * m + i] = i == k ? diag : li;
#pragma unroll 4
    for (int j = k + 1; j < m; j++) {
      const double lj = __shfl_sync(0xffffffffu, li, j) * dk;
      if (i >= j && i < m) F[j * m + i] -= li * lj;
    }
    __syncwarp();
  }
  if (ldlt && lane == 0 && (neg | pert)) {
    atomicAdd(la.counts, neg);
    atomicAdd(la.counts + 1, pert);
  }
  double *Up = U + P.snUoff[s];
  for (int jj = 0; jj < mu; jj++) {
    const int ii = jj + lane;
    if (ii < mu) Up[(int64_t)jj * mu + ii] = F[(nc + jj) * m + nc + ii];
  }
}

// The whole front of supernode s (32 < m <= MAXM, 64 or 128) by one CTA. The front is assembled in
// shared memory and then held in registers, as C fragments of its 8 x 8 tiles: eight warps own the row groups (w, and
// for 128 rows also 15 - w), MAXM / 32 more warps take the pivot columns, a row per lane (pivot_steps.cuh). Eight pivot
// columns per step with two barriers: the panel warps eliminate them; the others update their tiles of the next eight
// columns and hand them over, then the rest of the triangle while the panel warps go on. What bounds it is latency: a
// step takes about 1,300 clocks, where a barrier and a rank-1 update of the shared front per column took 2,000 each.
// The steps' columns stay in shared memory (over the front, which is dead by then) until they are scaled and written.
template <int MAXM>
constexpr int small_threads() { return 32 * (8 + MAXM / 32); }
// shared memory (entries) for fronts of at most m rows and nc pivot columns: the front, or the steps' columns over
// it, and three step buffers
__host__ __device__ constexpr int small_main(int m, int nc) {
  const int f = m * m, p = (nc + 7) / 8 * ((m + 7) / 8 * 8) * kColLd;
  return ((f > p ? f : p) + 3) & ~3;
}
constexpr int small_elems(int m, int nc) { return small_main(m, nc) + 3 * ((m + 7) / 8 * 8) * kColLd; }

template <bool LDLT, int MAXM>
__global__ void __launch_bounds__(small_threads<MAXM>(), MAXM == 64 ? 2 : 1)
    k_front_small(const int *__restrict__ fronts, int mainElems, DevPlan P, const double *__restrict__ values,
                  double *__restrict__ Lx, double *__restrict__ U, unsigned long long *status, LdltArgs<double> la) {
  constexpr int NT = small_threads<MAXM>(), NP = MAXM / 32, CL = kColLd, NG = MAXM / 64;
  extern __shared__ __align__(16) unsigned char fs_dyn[];
  __shared__ ChildMaps cm;
  __shared__ double scale[MAXM], diag[MAXM];
  __shared__ int failAt, inexact, nNeg, nPert;
  pdl_next();
  const int s = fronts[blockIdx.x];
  const int f = P.snF[s], nc = P.snNc[s], m = P.snM[s], mu = m - nc;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int rows = (m + 7) & ~7, RB = rows / 8, steps = (nc + 7) / 8, pst = rows * CL;
  double *F = reinterpret_cast<double *>(fs_dyn), *R = F + mainElems, *Q = R + pst, *Pc = F;  // Pc: -a of every step
  double *Lp = Lx + P.snLxp[s];
  double *Up = U + (mu > 0 ? P.snUoff[s] : 0);
  const double tau = LDLT ? la.scal[1] : 0.0;
  if (!assemble_cta<NT>(s, P, values, U, F, &cm, status)) return;
  // the front's tiles: row group rg[h], tile column cb
  const int rg[2] = {warp, NG == 2 ? 15 - warp : -1};
  auto tile = [&](int rb, int cb, double(&c)[2]) {
    const int i = 8 * rb + g;
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const int j = 8 * cb + 2 * t + u;
      c[u] = i < m && j <= i ? F[j * m + i] : i == j ? 1.0 : 0.0;
    }
  };
  auto hand_over = [&](int rb, const double(&c)[2]) {
    double2 v;
    v.x = c[0];
    v.y = c[1];
    *reinterpret_cast<double2 *>(R + (8 * rb + g) * CL + 2 * t) = v;
  };
  if (warp < 8) {
#pragma unroll
    for (int h = 0; h < NG; h++) {
      double c0[2];
      if (rg[h] < RB) {
        tile(rg[h], 0, c0);
        hand_over(rg[h], c0);
      }
    }
  }
  if (tid == 0) {
    failAt = 0x7fffffff;
    inexact = nNeg = nPert = 0;
  }
  if (warp >= 8) {
    __syncthreads();  // the front is in registers: Pc may overwrite it
    for (int k = 0; k < steps; k++) {
      double *Pk = Pc + k * pst, *Qk = Q + (k & 1) * pst;
      const int r = min(8 * k + 32 * (warp - 8) + lane, rows - 1), w = nc - 8 * k;
      const bool mine = 8 * k + 32 * (warp - 8) < rows;
      if (mine) {
        const bool fine = w >= 8 ? eliminate8<false, LDLT, false>(R, Pk, Qk, 8 * k, r, 8, tau)
                                 : eliminate8<false, LDLT, true>(R, Pk, Qk, 8 * k, r, w, tau);
        if (!fine) inexact = 1;
      }
      __syncthreads();
      if (inexact) {  // R is unchanged: the step again with exact quotients
        if (mine) eliminate8<true, LDLT, true>(R, Pk, Qk, 8 * k, r, w, tau);
        __syncthreads();
        if (tid == 256) inexact = 0;
      }
      __syncthreads();
    }
  } else {
    double ca[7][2], cb[NG == 2 ? 15 : 1][2];  // at step k: the tiles (rg[h], k + 1), (rg[h], k + 2), ...
#pragma unroll
    for (int j = 0; j < 7; j++)
      if (rg[0] < RB && j < rg[0]) tile(rg[0], j + 1, ca[j]);
    if constexpr (NG == 2) {
#pragma unroll
      for (int j = 0; j < 15; j++)
        if (rg[1] < RB && j < rg[1]) tile(rg[1], j + 1, cb[j]);
    }
    __syncthreads();
    for (int k = 0; k < steps; k++) {
      __syncthreads();
      if (inexact) __syncthreads();
      const double *Pk = Pc + k * pst, *Qk = Q + (k & 1) * pst;
      const bool on0 = rg[0] > k && rg[0] < RB, on1 = NG == 2 && rg[1] > k && rg[1] < RB;
      if (on0) {
        step_tile(ca[0], Pk + 8 * rg[0] * CL, Qk + 8 * (k + 1) * CL, CL, g, t);
        hand_over(rg[0], ca[0]);
      }
      if (on1) {
        step_tile(cb[0], Pk + 8 * rg[1] * CL, Qk + 8 * (k + 1) * CL, CL, g, t);
        hand_over(rg[1], cb[0]);
      }
      __syncthreads();
      const bool last = k + 1 == steps;  // the tiles from column k + 1 on are then the update block's
      if (on0) {
#pragma unroll
        for (int j = 1; j < 7; j++)
          if (k + 1 + j <= rg[0]) step_tile(ca[j], Pk + 8 * rg[0] * CL, Qk + 8 * (k + 1 + j) * CL, CL, g, t);
        if (!last) {
#pragma unroll
          for (int j = 1; j < 7; j++) {
            ca[j - 1][0] = ca[j][0];
            ca[j - 1][1] = ca[j][1];
          }
        }
      }
      if constexpr (NG == 2) {
        if (on1) {
#pragma unroll
          for (int j = 1; j < 15; j++)
            if (k + 1 + j <= rg[1]) step_tile(cb[j], Pk + 8 * rg[1] * CL, Qk + 8 * (k + 1 + j) * CL, CL, g, t);
          if (!last) {
#pragma unroll
            for (int j = 1; j < 15; j++) {
              cb[j - 1][0] = cb[j][0];
              cb[j - 1][1] = cb[j][1];
            }
          }
        }
      }
    }
    // the update block (of a failed front too: nobody reads it)
    auto put = [&](int rb, int tc, const double(&c)[2]) {
      const int i = 8 * rb + g;
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int j = 8 * tc + 2 * t + u;
        if (i < m && j <= i) Up[(int64_t)(j - nc) * mu + i - nc] = c[u];
      }
    };
    if (rg[0] < RB) {
#pragma unroll
      for (int j = 0; j < 7; j++)
        if (steps + j <= rg[0]) put(rg[0], steps + j, ca[j]);
    }
    if constexpr (NG == 2) {
      if (rg[1] < RB) {
#pragma unroll
        for (int j = 0; j < 15; j++)
          if (steps + j <= rg[1]) put(rg[1], steps + j, cb[j]);
      }
    }
  }
  // the pivots: test and count, the columns' scales
  if (tid < MAXM) {
    double d = tid < nc ? -Pc[(tid >> 3) * pst + tid * CL + (tid & 7)] : 1.0;
    bool bad = false, small = false;
    if (LDLT) {
      small = tid < nc && !(fabs(d) >= tau);
      bad = small && !isfinite(d);
      if (small) d = d < 0.0 ? -tau : tau;
      const int neg = __popc(__ballot_sync(0xffffffffu, tid < nc && d < 0.0));
      const int pert = __popc(__ballot_sync(0xffffffffu, small));
      if (lane == 0) {
        atomicAdd(&nNeg, neg);
        atomicAdd(&nPert, pert);
      }
    } else {
      bad = tid < nc && !(d > 0.0);
    }
    const unsigned mask = __ballot_sync(0xffffffffu, bad);
    if (lane == 0 && mask) atomicMin(&failAt, 32 * warp + __ffs(mask) - 1);
    const double dl = LDLT ? d : sqrt(d);
    diag[tid] = dl;
    scale[tid] = 1.0 / dl;
  }
  __syncthreads();
  if (failAt < MAXM) {
    if (tid == 0) atomicMin(status, status_word(f + failAt, LDLT ? 2 : 1, s));
    return;  // block-uniform
  }
  {  // L, and the update block's part of the last step's columns: a lane per row, eight columns at a time
    const int r = tid & (MAXM - 1);
    for (int p = tid / MAXM; p < steps && tid < NT / MAXM * MAXM; p += NT / MAXM) {
      if (r < 8 * p || r >= m) continue;
      const double *Pr = Pc + p * pst + r * CL;
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; u += 2) {
        const double2 x = *reinterpret_cast<const double2 *>(Pr + u);
        v[u] = -x.x;
        v[u + 1] = -x.y;
      }
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const int col = 8 * p + u;
        if (r < col) continue;
        if (col < nc)
          Lp[(int64_t)col * m + r] = r == col ? (LDLT ? 1.0 : diag[col]) : v[u] * scale[col];
        else
          Up[(int64_t)(col - nc) * mu + r - nc] = v[u];
      }
    }
  }
  if (LDLT) {
    if (tid < nc) la.D[f + tid] = diag[tid];
    if (tid == 0 && (nNeg | nPert)) {
      atomicAdd(la.counts, nNeg);
      atomicAdd(la.counts + 1, nPert);
    }
  }
}

// (value, index) of the largest value over the warp, the smallest index on ties (every lane gets the result)
__device__ __forceinline__ void front_warp_argmax(double &v, int &i) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double ov = __shfl_xor_sync(0xffffffffu, v, o);
    const int oi = __shfl_xor_sync(0xffffffffu, i, o);
    if (ov > v || (ov == v && oi < i)) {
      v = ov;
      i = oi;
    }
  }
}

// The whole front with Bunch-Kaufman pivots inside each 64-column block of its pivot columns (AMP_LDLT_BK; the rule,
// the 2 x 2 inverse and the outputs of bk_block in group_panel.cu), FP64 arithmetic. At column k of block [c0, c1):
// colmax and rowmax over the block's rows only, computed by every warp with shuffles (the same values in the same
// order, so every thread takes the same decision without sharing it); the interchange applied in lower storage to
// the block's earlier columns (their rows) and to the whole trailing triangle (rows below the pivot columns
// included); the rank-1 or rank-2 update of the trailing triangle from the unscaled column(s); then the column(s)
// scaled in place to L. Three barriers per step, one more where row im is searched (its entries belong to the triangle that
// a faster warp goes on to interchange and update). A block's L columns go to Lx once the block is done (its later steps may
// still interchange their rows), with its pivot order; D and D(k + 1, k) as they are decided. A column with no usable entry
// in its block keeps the static perturbation to +-tau (counted); a non-finite pivot fails.
template <int G>
__device__ void factor_front_bk(int s, const DevPlan &P, const double *__restrict__ values, double *__restrict__ Lx,
                                double *__restrict__ U, double *F, unsigned long long *status, const LdltArgs<double> &la,
                                int t, ChildMaps *cm) {
  constexpr int NW = G / 32;
  const int warp = t >> 5, lane = t & 31;
  const int f = P.snF[s], nc = P.snNc[s], m = P.snM[s], mu = m - nc;
  const double tau = la.scal[1];
  const double alpha = 0.64038820320220756;  // (1 + sqrt(17)) / 8
  if constexpr (G == 32) {
    assemble_warp<16>(s, P, values, U, F, t);
    if (warp_failed(status)) return;
  } else {
    if (!assemble_cta<G>(s, P, values, U, F, cm, status)) return;
  }
  auto at = [&](int i, int j) -> double & { return F[j * m + i]; };  // entry (i, j), i >= j
  int neg = 0, pert = 0;  // thread 0
  int perm[64];           // thread 0: the current block's pivot order
  double *Lp = Lx + P.snLxp[s];
  for (int c0 = 0; c0 < nc; c0 += 64) {
    const int c1 = min(nc, c0 + 64);
    if (t == 0)
      for (int i = 0; i < c1 - c0; i++) perm[i] = i;
    for (int k = c0; k < c1;) {
      double cmx = -1.0;
      int im = -1;
      for (int i = k + 1 + lane; i < c1; i += 32) {
        const double a = fabs(at(i, k));
        if (a > cmx) {
          cmx = a;
          im = i;
        }
      }
      front_warp_argmax(cmx, im);
      const double colmax = cmx > 0.0 ? cmx : 0.0, absakk = fabs(at(k, k));
      int step = 1, kp = k;
      if (colmax > 0.0 && !(absakk >= alpha * colmax)) {
        double rm = 0.0;
        for (int j = k + lane; j < c1; j += 32)
          if (j != im) rm = fmax(rm, fabs(j > im ? at(j, im) : at(im, j)));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) rm = fmax(rm, __shfl_xor_sync(0xffffffffu, rm, o));
        if (absakk * rm >= alpha * colmax * colmax) {
          kp = k;
        } else if (fabs(at(im, im)) >= alpha * rm) {
          kp = im;
        } else {
          step = 2;
          kp = im;
        }
        group_sync<G>();  // every warp has read row im before anyone changes the trailing triangle
      }
      const int kk = k + step - 1;
      if (kp != kk) {  // interchange p = kk and r = kp (p < r), lower storage
        const int p = kk, r = kp, nBelow = m - r - 1, nMid = r - p - 1, nLeft = p - c0;
        for (int e = t; e < 1 + nBelow + nMid + nLeft; e += G) {
          double *x, *y;
          if (e == 0) {
            x = &at(p, p);
            y = &at(r, r);
          } else if (e <= nBelow) {
            x = &at(r + e, p);
            y = &at(r + e, r);
          } else if (e <= nBelow + nMid) {
            const int i = p + (e - nBelow);
            x = &at(i, p);
            y = &at(r, i);
          } else {
            const int j = c0 + (e - nBelow - nMid - 1);
            x = &at(p, j);
            y = &at(r, j);
          }
          const double tmp = *x;
          *x = *y;
          *y = tmp;
        }
        if (t == 0) {
          const int tmp = perm[p - c0];
          perm[p - c0] = perm[r - c0];
          perm[r - c0] = tmp;
        }
        group_sync<G>();
      }
      if (step == 1) {
        double d = at(k, k);
        const bool small = !(fabs(d) >= tau);
        if (small && isfinite(d)) d = d < 0.0 ? -tau : tau;
        if (!isfinite(d)) {
          if (t == 0) atomicMin(status, status_word(f + k, 2, s));
          return;  // group-uniform
        }
        if (t == 0) {
          neg += d < 0.0 ? 1 : 0;
          pert += small ? 1 : 0;
          la.D[f + k] = d;
          la.Doff[f + k] = 0.0;
        }
        const double inv = 1.0 / d;
        for (int jj = warp; jj < m - k - 1; jj += NW) {
          const int j = k + 1 + jj;
          const double lj = at(j, k);
          for (int i = j + lane; i < m; i += 32) at(i, j) -= (at(i, k) * inv) * lj;
        }
        group_sync<G>();
        for (int i = k + 1 + t; i < m; i += G) at(i, k) *= inv;  // L(i, k)
        group_sync<G>();
      } else {
        // D_k = e [[a, 1], [1, c]], D_k^-1 = (t / e) [[c, -1], [-1, a]] with a = d11 / e, c = d22 / e, t = 1 / (a c - 1)
        const double d11 = at(k, k), e21 = at(k + 1, k), d22 = at(k + 1, k + 1);
        const double a = d11 / e21, c = d22 / e21, te = (1.0 / (a * c - 1.0)) / e21;
        if (!(isfinite(te) && isfinite(a) && isfinite(c))) {
          if (t == 0) atomicMin(status, status_word(f + k, 2, s));
          return;  // group-uniform
        }
        if (t == 0) {
          neg += a * c - 1.0 < 0.0 ? 1 : (d11 < 0.0 ? 2 : 0);
          la.D[f + k] = d11;
          la.D[f + k + 1] = d22;
          la.Doff[f + k] = e21;
          la.Doff[f + k + 1] = 0.0;
        }
        for (int jj = warp; jj < m - k - 2; jj += NW) {
          const int j = k + 2 + jj;
          const double pj = at(j, k), qj = at(j, k + 1);
          for (int i = j + lane; i < m; i += 32) {
            const double pi = at(i, k), qi = at(i, k + 1);
            at(i, j) -= te * (c * pi - qi) * pj + te * (a * qi - pi) * qj;
          }
        }
        group_sync<G>();
        for (int i = k + 2 + t; i < m; i += G) {
          const double pi = at(i, k), qi = at(i, k + 1);
          at(i, k) = te * (c * pi - qi);      // L(i, k)
          at(i, k + 1) = te * (a * qi - pi);  // L(i, k + 1)
        }
        if (t == 0) at(k + 1, k) = 0.0;  // L(k + 1, k)
        group_sync<G>();
      }
      k += step;
    }
    for (int j = c0; j < c1; j++)  // the block's L columns, unit diagonal, rows in the block's pivot order
      for (int i = j + t; i < m; i += G) Lp[(int64_t)j * m + i] = i == j ? 1.0 : at(i, j);
    if (t == 0)
      for (int i = 0; i < c1 - c0; i++) la.piv[f + c0 + i] = perm[i];
  }
  if (t == 0 && (neg | pert)) {
    atomicAdd(la.counts, neg);
    atomicAdd(la.counts + 1, pert);
  }
  if (mu > 0) {
    double *Up = U + P.snUoff[s];
    for (int e = t; e < mu * mu; e += G) {
      const int jj = e / mu, ii = e - jj * mu;
      if (ii >= jj) Up[e] = F[(nc + jj) * m + nc + ii];
    }
  }
}

// m <= MAXM (16 or 32): one warp per front, tiny_warps<MAXM>() fronts per CTA
// BK: Bunch-Kaufman pivots (FP64 factors with la.piv set)
template <int MAXM, bool BK>
__global__ void __launch_bounds__(32 * tiny_warps<MAXM>(), BK ? 1 : tiny_ctas<MAXM>())
    k_front_tiny(const int *__restrict__ fronts, int count, DevPlan P, const double *__restrict__ values,
                 double *__restrict__ Lx, double *__restrict__ U, unsigned long long *status, LdltArgs<double> la) {
  constexpr int W = tiny_warps<MAXM>();
  __shared__ double F[W][MAXM * MAXM];
  pdl_next();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int idx = blockIdx.x * W + warp;
  if (idx >= count) return;  // warp-uniform; no CTA-wide barrier follows
  if constexpr (BK)
    factor_front_bk<32>(fronts[idx], P, values, Lx, U, F[warp], status, la, lane, nullptr);
  else
    factor_front_warp<MAXM>(fronts[idx], P, values, Lx, U, F[warp], status, la, lane);
}

// 32 < m <= 128 with Bunch-Kaufman pivots: one CTA per front; dynamic shared memory = the launch's largest m squared
__global__ void __launch_bounds__(256) k_front_small_bk(const int *__restrict__ fronts, DevPlan P,
                                                        const double *__restrict__ values, double *__restrict__ Lx,
                                                        double *__restrict__ U, unsigned long long *status,
                                                        LdltArgs<double> la) {
  extern __shared__ __align__(16) unsigned char fs_dyn[];
  __shared__ ChildMaps cm;
  pdl_next();
  factor_front_bk<256>(fronts[blockIdx.x], P, values, Lx, U, reinterpret_cast<double *>(fs_dyn), status, la,
                          threadIdx.x, &cm);
}

template <bool LDLT>
static cudaError_t init_small() {
  const int bytes = small_elems(kSmallFront, kSmallFront) * (int)sizeof(double);
  cudaError_t e = cudaFuncSetAttribute(k_front_small<LDLT, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       bytes);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_front_small<LDLT, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  return e;
}
cudaError_t init_front_small_attributes() {
  cudaError_t e = init_small<false>();
  if (e == cudaSuccess) e = init_small<true>();
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_front_small_bk, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kSmallFront * kSmallFront * (int)sizeof(double));
  return e;
}

// after: the launch before it on the stream is the one of the level below, alone (SmallFronts): it then starts before that
// one has ended, and assembles A's entries meanwhile
template <class... KA, class... A>
static void launch_level(void (*kernel)(KA...), bool after, int grid, int threads, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3((unsigned)threads);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = after ? 1 : 0;
  cudaLaunchKernelEx(&c, kernel, KA(args)...);
}

template <int MAXM, bool BK>
static int launch_tiny(bool after, const int *fronts, int count, const DevPlan &P, const double *values, double *Lx,
                       double *U, unsigned long long *status, const LdltArgs<double> &la, cudaStream_t st) {
  constexpr int W = tiny_warps<MAXM>();
  if (count <= 0) return 0;
  launch_level(k_front_tiny<MAXM, BK>, after, (count + W - 1) / W, 32 * W, 0, st, fronts, count, P, values, Lx, U, status,
               la);
  return 1;
}

template <bool LDLT, int MAXM>
static int launch_small(bool after, const SmallClass &c, const DevPlan &P, const double *values, double *Lx, double *U,
                        unsigned long long *status, const LdltArgs<double> &la, cudaStream_t st) {
  if (c.count <= 0) return 0;
  launch_level(k_front_small<LDLT, MAXM>, after, c.count, small_threads<MAXM>(),
               small_elems(c.maxM, c.maxNc) * sizeof(double), st, c.sn, small_main(c.maxM, c.maxNc), P, values, Lx, U,
               status, la);
  return 1;
}
template <bool LDLT, bool BK>
static int launch_fronts_tc(const SmallFronts &fr, const DevPlan &P, const double *values, double *Lx, double *U,
                            unsigned long long *status, const LdltArgs<double> &la, cudaStream_t st) {
  // a class of its own only where the GPU would otherwise not hold the level's fronts at once: two launches one after
  // the other take twice a front's latency
  const int mid = fr.ntiny <= num_sms() * tiny_warps<kTinyFront>() ? 0 : fr.ntinyMid;
  SmallClass half = fr.half, full = fr.full;
  if (half.count + full.count <= num_sms() && half.count > 0 && full.count > 0) {  // (the two lists are one)
    full = SmallClass{half.sn, half.count + full.count, full.maxM, std::max(half.maxNc, full.maxNc)};
    half.count = 0;
  }
  int k = launch_tiny<kTinyMid, BK>(fr.after, fr.tiny, mid, P, values, Lx, U, status, la, st);
  k += launch_tiny<kTinyFront, BK>(fr.after, fr.tiny + mid, fr.ntiny - mid, P, values, Lx, U, status, la, st);
  if constexpr (BK) {
    for (const SmallClass &c : {half, full})
      if (c.count > 0) {
        launch_level(k_front_small_bk, fr.after, c.count, 256, (size_t)c.maxM * c.maxM * sizeof(double), st, c.sn, P, values,
                     Lx, U, status, la);
        k++;
      }
  } else {
    k += launch_small<LDLT, 64>(fr.after, half, P, values, Lx, U, status, la, st);
    k += launch_small<LDLT, 128>(fr.after, full, P, values, Lx, U, status, la, st);
  }
  return k;
}
template <>
int launch_fronts_small<double>(const SmallFronts &fr, const DevPlan &P, const double *values, double *Lx, double *U,
                                unsigned long long *status, const LdltArgs<double> &la, cudaStream_t st) {
  if (la.piv != nullptr)  // Bunch-Kaufman pivots (FP64)
      return launch_fronts_tc<true, true>(fr, P, values, Lx, U, status, la, st);
  if (la.scal != nullptr)  // LDL^T: FP64 arithmetic whatever the storage
    return launch_fronts_tc<true, false>(fr, P, values, Lx, U, status, la, st);
  return launch_fronts_tc<false, false>(fr, P, values, Lx, U, status, la, st);
}

}  // namespace amp
