// Group panel of the FP32 factors of the mixed-precision path: POTRF (or LDL^T) of each 64 x 64 pivot block, TRSM of the rows
// below it and the update of the group's remaining columns, in FP32, in one dataflow launch as group_panel.cu. An FP32
// factor is used on its own too (a solve without refinement), where the order of its FP32 operations is what the caller
// sees: the FP64 tensor-core panel of the FP64 factors, correct to the last FP32 bit as it is, moves such a solution by 5e-6
// (its distance from the exact one is 9e-6 either way). It took 32 against 39 us per group of two blocks of a 4,096-row front.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cfloat>

#include "../host/plan.hpp"
#include "devplan.cuh"
#include "launch.hpp"
#include "panel_blocks.cuh"

namespace amp {

namespace {

__device__ __forceinline__ double ldcg_v(const double *p) { return __ldcg(p); }
__device__ __forceinline__ float ldcg_v(const float *p) { return __ldcg(p); }
__device__ __forceinline__ double pivot_mag(double d) { return fabs(d); }
__device__ __forceinline__ double pivot_mag(float d) { return fabs((double)d); }
template <class TC>
__device__ __forceinline__ bool chol_pivot_ok(TC d) { return d > TC(0); }
template <class TC>
__device__ __forceinline__ TC chol_sqrt(TC d) { return sqrt(d); }
__device__ __forceinline__ double recip_nr(double d) {
  const double a = fabs(d);
  if (!(a > 1e-30 && a < 1e30)) return 1.0 / d;  // outside the float range of the first approximation
  double x = (double)__frcp_rn((float)d);
  double e = fma(-d, x, 1.0);
  x = fma(x, e, x);
  e = fma(-d, x, 1.0);
  x = fma(x, e, x);
  e = fma(-d, x, 1.0);
  return fma(x, e, x);
}

// Static pivot perturbation of LDL^T (ldlt.mjs:513-522): |d| < tau (or NaN) becomes -tau / +tau by the sign of d,
// a non-finite small pivot fails the factorization. flags: bit 0 negative pivot, bit 1 perturbed. false = failure.
template <class TC>
__device__ __forceinline__ bool ldlt_pivot(TC &d, TC tau, unsigned char &flags) {
  flags = 0;
  if (!(fabs(d) >= tau)) {
    if (!isfinite(d)) return false;
    d = d < TC(0) ? -tau : tau;
    flags = 2;
  }
  if (d < TC(0)) flags |= 1;
  return true;
}
__device__ __forceinline__ double fast_recip(double d) { return recip_nr(d); }
__device__ __forceinline__ float fast_recip(float d) { return __fdividef(1.0f, d); }

// Pivot block: POTRF (or LDL^T) of the 64 x 64 diagonal block of a front, called by all 256 threads of a CTA, the
// block in registers, in TC. src: the updated block in
// shared memory, entry (i, j) at src[j lds + i]; Lp: the block's (0, 0) entry in the front (ld m), where the factor is
// written; w <= 64 its columns. Thread t < 136 owns the 4 x 4 tile (ti, tj), ti >= tj, of the lower triangle.
// Right-looking on the unscaled columns, four columns per step kb with two barriers: (1) the diagonal tile eliminates
// its four columns (settling the pivots) and publishes them; (2) the tiles below it in column block kb eliminate the
// same four columns against it and publish theirs; then every tile right of the block applies the rank-4 update
// S(i, j) -= sum S(i, k) S(j, k) / d_k. Cholesky tests d > 0 (sparse.mjs:1151-1156); LDL^T (ld.scal != null,
// ldlt.mjs:450-562) perturbs |d| < tau to +-tau and counts negative and perturbed pivots. At the end the columns are
// scaled: Cholesky L = a / sqrt(d) with sqrt(d) on the diagonal, LDL^T L = a / d with a unit diagonal (D to ld.D).
// Returns false (status set for the first failing column f + c0 + k) when a pivot failed; the block is then not
// written back.
template <class TC>
__device__ int potrf_core(const float *src, int lds, float *Lp, int m, int w, int f, int c0, int s,
                          unsigned long long *status, const LdltArgs<float> &ld, double promoteBelow) {
  __shared__ TC col[2][4][kPanel];  // per 4-column block (double-buffered): the block's unscaled columns, by row
  __shared__ TC pd[kPanel], piv[2][4];
  __shared__ unsigned char pflag[kPanel];
  __shared__ int fail, promote;
  const int tid = threadIdx.x;
  const bool ldlt = ld.scal != nullptr;
  const TC tau = ldlt ? (TC)ld.scal[1] : TC(0);
  // tile of this thread: row block ti, column block tj (ti >= tj), from tid by the triangular numbering
  int ti = 0;
  while ((ti + 1) * (ti + 2) / 2 <= tid) ti++;
  const int tj = tid - ti * (ti + 1) / 2;
  const bool owner = tid < 136;
  int myFail = -1;  // diagonal tiles only
  TC a[4][4];
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const int i = 4 * ti + r, j = 4 * tj + c;
      a[r][c] = !owner || i < j ? TC(0) : (i < w ? (TC)src[j * lds + i] : (i == j ? TC(1) : TC(0)));
    }
  if (tid == 0) {
    fail = kPanel;  // none
    promote = 0;
  }
  for (int kb = 0; kb < (w + 3) / 4; kb++) {  // the columns from w on are the identity's
    const int buf = kb & 1;
    if (owner && ti == kb && tj == kb) {
#pragma unroll
      for (int kk = 0; kk < 4; kk++) {
        const int k = 4 * kb + kk;
        TC d = a[kk][kk];
        unsigned char fl = 0;
        const bool bad = k < w && (ldlt ? !ldlt_pivot(d, tau, fl) : !chol_pivot_ok(d));
        if (bad && myFail < 0) myFail = k;  // first failing pivot of this diagonal tile
        const TC iv = fast_recip(d);          // the update scale only; L is scaled with the exact 1 / d at the end
        pd[k] = d;
        pflag[k] = fl;
        piv[buf][kk] = iv;
#pragma unroll
        for (int r = kk + 1; r < 4; r++)
#pragma unroll
          for (int c = kk + 1; c <= r; c++) a[r][c] -= a[r][kk] * (a[c][kk] * iv);
      }
#pragma unroll
      for (int kk = 0; kk < 4; kk++)
#pragma unroll
        for (int r = 0; r < 4; r++) col[buf][kk][4 * kb + r] = a[r][kk];
    }
    __syncthreads();
    if (owner && tj == kb && ti > kb) {
#pragma unroll
      for (int kk = 0; kk < 4; kk++) {
        const TC iv = piv[buf][kk];
#pragma unroll
        for (int c = kk + 1; c < 4; c++) {
          const TC cj = col[buf][kk][4 * kb + c] * iv;
#pragma unroll
          for (int r = 0; r < 4; r++) a[r][c] -= a[r][kk] * cj;
        }
      }
#pragma unroll
      for (int kk = 0; kk < 4; kk++)
#pragma unroll
        for (int r = 0; r < 4; r++) col[buf][kk][4 * ti + r] = a[r][kk];
    }
    __syncthreads();
    if (owner && tj > kb) {
#pragma unroll
      for (int kk = 0; kk < 4; kk++) {
        const TC iv = piv[buf][kk];
        TC ci[4], cj[4];
#pragma unroll
        for (int r = 0; r < 4; r++) ci[r] = col[buf][kk][4 * ti + r];
#pragma unroll
        for (int c = 0; c < 4; c++) cj[c] = col[buf][kk][4 * tj + c] * iv;
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
          for (int c = 0; c < 4; c++)
            if (ti > tj || c <= r) a[r][c] -= ci[r] * cj[c];
      }
    }
  }
  if (myFail >= 0) atomicMin(&fail, myFail);
  if (promoteBelow > 0.0 && tid < w && !(pivot_mag(pd[tid]) >= promoteBelow)) promote = 1;
  __syncthreads();
  if (promote) return 2;  // the caller redoes the block in higher precision (nothing written)
  if (fail < kPanel) {
    if (tid == 0) atomicMin(status, status_word(f + c0 + fail, ldlt ? 2 : 1, s));
    return 1;
  }
  if (owner) {
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const int j = 4 * tj + c;
      const TC d = pd[j];
      const TC lj = ldlt ? d : chol_sqrt(d);
      const TC inv = TC(1) / lj;
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const int i = 4 * ti + r;
        if (i >= j && i < w && j < w) Lp[(int64_t)j * m + i] = (float)(i == j ? (ldlt ? TC(1) : lj) : a[r][c] * inv);
      }
    }
  }
  if (ldlt) {
    if (tid < w) ld.D[f + c0 + tid] = (double)pd[tid];
    if (tid == 0) {
      int neg = 0, pert = 0;
      for (int k = 0; k < w; k++) neg += pflag[k] & 1, pert += pflag[k] >> 1;
      atomicAdd(ld.counts, neg);
      atomicAdd(ld.counts + 1, pert);
    }
  }
  return 0;
}

// POTRF / LDL^T of a pivot block (potrf_core in the factor's precision). An FP32 LDL^T block with a pivot of
// magnitude below FLT_EPSILON x max_i |A(i, i)| (a pivot with no correct FP32 digit left) is factored again from the
// same entries (src is left unchanged) in FP64 arithmetic (stored FP32): the small-pivot blocks of the mixed-precision
// indefinite factor get FP64 pivots. Returns false when a pivot failed (status set).
__device__ bool potrf_block(const float *src, int lds, float *Lp, int m, int w, int f, int c0, int s,
                            unsigned long long *status, const LdltArgs<float> &ld) {
  if (ld.scal == nullptr) return potrf_core<float>(src, lds, Lp, m, w, f, c0, s, status, ld, -1.0) == 0;
  const double amax = ld.scal[0] > 0.0 ? ld.scal[1] / ld.scal[0] : 0.0;
  const int r = potrf_core<float>(src, lds, Lp, m, w, f, c0, s, status, ld, amax * (double)FLT_EPSILON);
  if (r != 2) return r == 0;
  return potrf_core<double>(src, lds, Lp, m, w, f, c0, s, status, ld, -1.0) == 0;
}

// TRSM of up to 64 rows [r0, r1) of a front (L: its column-major block, ld m) against its factored pivot block
// [c0, c0 + w): x_k = (a_k - sum_{c<k} x_c M(k, c)) / M(k, k). Four threads per row, thread (row, q) holds columns
// 16 q .. 16 q + 15 in registers. Phase p: the threads of quarter p solve their 16 columns (the earlier quarters'
// contributions already applied) and publish them; after a barrier the threads of the later quarters subtract
// quarter p's contribution (16 x 16 products) from theirs. Cholesky: M = L11, x = L21. LDL^T: M(k, c) = L11(k, c) d_c,
// M(k, k) = d_k, x = L21, and w = x D = L21 D (the update's A operand, written to ld.W for the FP64 factor). The rows
// are also written as BF16 hi / lo pairs (hi = bf16(x), lo = bf16(x - hi)) into the split columns of the tensor-core
// update (mixed precision). The pivot block and D come from another CTA of the launch: read through L2 (__ldcg).
// x: this thread's 16 entries of its row (row r0 + tid % 64, columns c0 + 16 (tid / 64) + u), loaded by the caller
// before it waited for the pivot block (the strip's own rows are final by then).
// On return Ws[c][r] holds this strip's update operand (x, or x D for LDL^T) and M[c][r] the solved rows x
// (c < w, r < r1 - r0; zero elsewhere): a diagonal strip's X_c for its own column block.
__device__ void trsm_strip(float *L, int m, int f, int c0, int w, int r0, int r1, int64_t lxp, int64_t sp,
                           __nv_bfloat16 *Shi, __nv_bfloat16 *Slo, const LdltArgs<float> &ld, float (*M)[kPanel + 1],
                           float (*Ws)[kPanel + 1], float *invd, float *dv, float (&x)[16]) {
  const bool ldlt = ld.scal != nullptr;
  const int tid = threadIdx.x, r = tid & (kPanel - 1), q = tid >> 6;
  {  // the pivot block: thread (r, q) loads row r of columns 16 q .. 16 q + 15 (times their pivots for LDL^T), and
     // thread r < 64 the pivot of column r, in one round trip
    float v[16];
#pragma unroll
    for (int u = 0; u < 16; u++) {
      const int c = 16 * q + u;
      v[u] = (r < w && c < r) ? ldcg_v(L + (int64_t)(c0 + c) * m + c0 + r) : 0.0f;
    }
    if (ldlt) {
#pragma unroll
      for (int u = 0; u < 16; u++) {
        const int c = 16 * q + u;
        v[u] = v[u] * (c < w ? (float)ldcg_v(ld.D + f + c0 + c) : 1.0f);
      }
    }
    if (tid < kPanel) {
      const float d = tid < w ? (ldlt ? (float)ldcg_v(ld.D + f + c0 + tid) : ldcg_v(L + (int64_t)(c0 + tid) * m + c0 + tid))
                               : 1.0f;
      dv[tid] = d;
      invd[tid] = 1.0f / d;
    }
#pragma unroll
    for (int u = 0; u < 16; u++) M[r][16 * q + u] = v[u];
  }
  const int row = r0 + r;
  const bool active = row < r1;
  __syncthreads();
  for (int p = 0; p < (w + 15) / 16; p++) {  // (zero from column w on)
    if (q == p) {  // solve this quarter
#pragma unroll
      for (int u = 0; u < 16; u++) {
        const int c = 16 * p + u;
        x[u] *= invd[c];
#pragma unroll
        for (int u2 = u + 1; u2 < 16; u2++) x[u2] -= x[u] * M[16 * p + u2][c];
      }
#pragma unroll
      for (int u = 0; u < 16; u++) Ws[16 * p + u][r] = x[u];
    }
    __syncthreads();
    if (q > p) {  // subtract quarter p's contribution
#pragma unroll 4
      for (int kk = 0; kk < 16; kk++) {
        const int k = 16 * p + kk;
        const float xk = Ws[k][r];
#pragma unroll
        for (int u = 0; u < 16; u++) x[u] -= xk * M[16 * q + u][k];
      }
    }
  }
  __syncthreads();  // every quarter read Ws: overwrite it with the update operand
  const int ld8 = (m + 7) & ~7;
#pragma unroll
  for (int u = 0; u < 16; u++) {
    const int cc = 16 * q + u;
    float xv = x[u];
    float wv = ldlt ? xv * dv[cc] : xv;
    Ws[cc][r] = active && cc < w ? wv : 0.0f;
    M[cc][r] = active && cc < w ? xv : 0.0f;  // the pivot block in M is no longer read
    if (!active || cc >= w) continue;
    L[(int64_t)(c0 + cc) * m + row] = xv;
    if (ldlt && ld.W) ld.W[lxp + (int64_t)(c0 + cc) * m + row] = wv;
    if (Shi) {
      const int64_t g = sp + (int64_t)(c0 + cc) * ld8 + row;
      const __nv_bfloat16 hi = __float2bfloat16_rn((float)xv);
      Shi[g] = hi;
      Slo[g] = __float2bfloat16_rn((float)xv - __bfloat162float(hi));
      if (ldlt) {
        const __nv_bfloat16 whi = __float2bfloat16_rn((float)wv);
        ld.Whi[g] = whi;
        ld.Wlo[g] = __float2bfloat16_rn((float)wv - __bfloat162float(whi));
      }
    }
  }
  __syncthreads();
}


// One group of pivot blocks [g0, g1) of a front, a strip of up to 64 rows per CTA, CTAs ordered by an atomic ticket
// (the diagonal strips of every item first, then the strips below the group). Per pivot block b of the group:
//   the diagonal strip of block b (rows [c0, c0 + w)) factors it once its own updates are done and publishes P[b];
//   every strip with rows below block b waits for P[b], solves its rows against the block (TRSM) and, when it is a
//   diagonal strip, publishes D[j] = b + 1; then it updates its rows of the group's remaining columns [c0 + w, g1)
//   with block b (C -= W_r X_c^T, K = w; X_c: the rows of those columns, from the diagonal strips' TRSM, waited for
//   by D[j] >= b + 1; a diagonal strip updates only the lower part, columns up to its own rows).
// Every wait is on a strip with a smaller ticket, which runs to completion without waiting on a larger one, so the
// launch cannot deadlock whatever the number of resident CTAs. The columns right of the group receive the group's
// update afterwards (k_update / k_update_mx, K = the group). Failure (a pivot, a bounded wait) sets the status and
// releases P[b], so every waiter leaves.
constexpr int kGroupSmem32 = 3 * kPanel * (kPanel + 1) * (int)sizeof(float);
// two CTAs per SM (registers capped at 128)
__global__ void __launch_bounds__(256, 2) k_group_panel_f32(const GroupItem *__restrict__ items,
                                                     const StripTask *__restrict__ strips, int nstrips, int *ticket,
                                                     int *flags, DevPlan P, float *__restrict__ Lx,
                                                     unsigned long long *status, __nv_bfloat16 *__restrict__ Shi,
                                                     __nv_bfloat16 *__restrict__ Slo, LdltArgs<float> ld) {
  extern __shared__ __align__(16) unsigned char gp_raw[];
  float(*M)[kPanel + 1] = reinterpret_cast<float(*)[kPanel + 1]>(gp_raw);  // pivot block (TRSM), then the X_c chunk
  float(*Ws)[kPanel + 1] = reinterpret_cast<float(*)[kPanel + 1]>(gp_raw + kPanel * (kPanel + 1) * sizeof(float));
  float(*Ds)[kPanel + 1] = reinterpret_cast<float(*)[kPanel + 1]>(gp_raw + 2 * kPanel * (kPanel + 1) * sizeof(float));
  __shared__ float invd[kPanel], dv[kPanel];
  __shared__ int sTicket;
  if (threadIdx.x == 0) sTicket = factor_failed(status) ? nstrips : atomicAdd(ticket, 1);
  __syncthreads();
  const int t = sTicket;
  if (t >= nstrips) return;
  const StripTask st = strips[t];
  const GroupItem it = items[st.item];
  const int s = it.s, g0 = it.g0, g1 = it.g1;
  const int f = P.snF[s], m = P.snM[s];
  const int nb = (g1 - g0 + kPanel - 1) / kPanel;
  const int r0 = st.r0, r1 = st.r1, jd = st.diag;
  const int bmax = jd >= 0 ? jd : nb;  // pivot blocks whose rows below include this strip
  float *L = Lx + P.snLxp[s];
  int *Pf = flags + it.flag0, *Df = Pf + nb;
  const int tid = threadIdx.x, tr = tid & 15, tc = tid >> 4;
  // A diagonal strip keeps its own pivot block (columns [r0, r1), lower part) in shared memory while it updates it
  // (Ds[j][i] = block (i, j)), and its POTRF reads it from there: no round trip through the front.
  if (jd >= 0) {
    for (int e = tid; e < kPanel * kPanel; e += blockDim.x) {
      const int i = e & 63, j = e >> 6;
      Ds[j][i] = (r0 + i < r1 && j <= i) ? L[(int64_t)(r0 + j) * m + r0 + i] : 0.0f;
    }
  }
  for (int b = 0; b < bmax; b++) {
    const int c0 = g0 + b * kPanel, w = min(kPanel, g1 - c0), c1 = c0 + w;
    float x[16];  // this thread's part of the strip's rows of block b, loaded while the pivot block is not yet ready
    {
      const int xr = r0 + (tid & (kPanel - 1)), xq = tid >> 6;
#pragma unroll
      for (int u = 0; u < 16; u++) {
        const int c = 16 * xq + u;
        x[u] = xr < r1 && c < w ? L[(int64_t)(c0 + c) * m + xr] : 0.0f;
      }
    }
    if (!panel_wait(Pf + b, 1, status, P.spin)) return;
    trsm_strip(L, m, f, c0, w, r0, r1, P.snLxp[s], P.snSp[s], Shi, Slo, ld, M, Ws, invd, dv, x);
    if (jd >= 0) panel_release(Df + jd, b + 1);
    // Update with block b (C -= W_r X_c^T, K = w): a diagonal strip first its own pivot block (X_c = its solved rows,
    // left in M by the TRSM; into Ds), then the blocks between block b and its own; a strip below every remaining
    // column block of the group.
    const int hi = jd >= 0 ? r0 : g1, nown = jd >= 0 ? 1 : 0;
    const int nchunk = nown + (hi > c1 ? (hi - c1 + kPanel - 1) / kPanel : 0);
    for (int ch = 0; ch < nchunk; ch++) {
      const bool own = ch < nown;
      const int cb = own ? r0 : c1 + (ch - nown) * kPanel, ncol = own ? r1 - r0 : min(kPanel, hi - cb);
      if (!own) {
        if (!panel_wait(Df + (cb - g0) / kPanel, b + 1, status, P.spin)) return;
        for (int e = tid; e < kPanel * kPanel; e += blockDim.x) {  // X_c[k][jj] = L(cb + jj, c0 + k)
          const int k = e >> 6, jj = e & 63;
          M[k][jj] = (k < w && jj < ncol) ? ldcg_v(L + (int64_t)(c0 + k) * m + cb + jj) : 0.0f;
        }
        __syncthreads();
      }
      float acc[4][4];
#pragma unroll
      for (int a = 0; a < 4; a++)
#pragma unroll
        for (int bb = 0; bb < 4; bb++) acc[a][bb] = 0.0f;
      for (int k = 0; k < w; k++) {
        float wv[4], xv[4];
#pragma unroll
        for (int a = 0; a < 4; a++) wv[a] = Ws[k][tr + 16 * a];
#pragma unroll
        for (int bb = 0; bb < 4; bb++) xv[bb] = M[k][tc + 16 * bb];
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
          for (int bb = 0; bb < 4; bb++) acc[a][bb] += wv[a] * xv[bb];
      }
#pragma unroll
      for (int a = 0; a < 4; a++)
#pragma unroll
        for (int bb = 0; bb < 4; bb++) {
          const int i = tr + 16 * a, jj = tc + 16 * bb;
          if (own) {
            if (jj <= i) Ds[jj][i] -= acc[a][bb];
          } else if (r0 + i < r1 && jj < ncol) {
            float *cptr = L + (int64_t)(cb + jj) * m + r0 + i;
            *cptr = *cptr - acc[a][bb];
          }
        }
      __syncthreads();  // M is reloaded by the next chunk, or by the next TRSM
    }
  }
  if (jd >= 0) {  // this strip's own pivot block, fully updated: factor it and publish it (also after a failure)
    const int c0 = g0 + jd * kPanel, w = min(kPanel, g1 - c0);
    __syncthreads();  // Ds complete (also when the strip had no earlier pivot block)
    potrf_block(&Ds[0][0], kPanel + 1, L + (int64_t)c0 * m + c0, m, w, f, c0, s, status, ld);
    panel_release(Pf + jd, 1);
  }
}


}  // namespace

cudaError_t init_group_panel_f32_attributes() {
  return cudaFuncSetAttribute(k_group_panel_f32, cudaFuncAttributeMaxDynamicSharedMemorySize, kGroupSmem32);
}

void launch_group_panel(const GroupItem *items, const StripTask *strips, int nstrips, int *ticket, int *flags,
                        const DevPlan &P, float *Lx, unsigned long long *status, __nv_bfloat16 *Shi, __nv_bfloat16 *Slo,
                        const LdltArgs<float> &ld, cudaStream_t st) {
  if (nstrips > 0)
    k_group_panel_f32<<<(unsigned)nstrips, 256, kGroupSmem32, st>>>(items, strips, nstrips, ticket, flags, P, Lx,
                                                                          status, Shi, Slo, ld);
}

}  // namespace amp
