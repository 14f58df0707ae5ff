// Solves and the refinement residual of the complex-symmetric LDL^T (the reference's ComplexSupernodalLDLT.solve and
// complexSolveRefined, ldlt.mjs:802-900): A = L D L^T with L unit lower (no conjugation), D complex diagonal.
//
// The sweeps go level by level over the supernodal tree, one launch per level and direction, a cluster of 1 to 8 CTAs
// per supernode, in 64-column blocks. Both directions are left-looking:
//   forward   y_b - (rows of block b times the earlier blocks' values): the CTAs of the cluster take the earlier blocks in
//             turn and read one another's partial sums through distributed shared memory; then every CTA solves the block's
//             unit lower triangle by itself (one warp, two rows per lane, the column's value by shuffle), so that the
//             result needs no hand-off. At the end the rows of the ancestors take their products by atomic subtraction
//             (the ancestors run at later levels), 64 rows per CTA in turn;
//   diagonal  y_j = y_j / D_j, written as the reference writes it ((a dr + b di) / den, (b dr - a di) / den);
//   backward  levels top-down, blocks last to first, the same with the rows below the block (later blocks, ancestors) in
//             place of the earlier columns, and the triangle L11^T.
// What bounds a sweep is the chain of blocks up the tree, at one system of a few thousand unknowns some 40 blocks each way,
// a latency each. Hence: triangles by cp.async one block ahead, the next block's first operand in registers before the
// triangle is solved, and each launch reads its first operands while the level before it still runs (programmatic
// dependent launch; the factor is constant, the values are read after the wait). One CTA per supernode, with the
// triangle's columns read from memory one after the other, took 2.9 ms for both sweeps of the edge-element system with 10
// elements per edge (6,130 unknowns, 20 levels); now 0.58 ms.
// Sums run in a different order from the reference's sequential loops (atomic subtraction in the forward sweep,
// partial sums in both), so results agree with it to round-off, not bit for bit.
#include <cuda_runtime.h>

#include <cstdint>

#include "cp_async.cuh"
#include "cplx.cuh"
#include "devplan.cuh"
#include "launch.hpp"
#include "sync.cuh"

namespace amp {

__device__ __forceinline__ cplx cld(const cplx *p) {
  const double2 v = *reinterpret_cast<const double2 *>(p);
  return cplx(v.x, v.y);
}
__device__ __forceinline__ cplx warp_sum(cplx v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v.re += __shfl_down_sync(0xffffffffu, v.re, o);
    v.im += __shfl_down_sync(0xffffffffu, v.im, o);
  }
  return v;
}

// y (permuted order, complex) = b[perm[i]] from the planar right-hand side (br, bi)
__global__ void k_cpermute_in(int n, const double *__restrict__ br, const double *__restrict__ bi,
                              const int *__restrict__ perm, cplx *__restrict__ y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = cplx(br[perm[i]], bi[perm[i]]);
}
// x[perm[i]] = y[i], planar
__global__ void k_cpermute_out(int n, const cplx *__restrict__ y, const int *__restrict__ perm,
                               double *__restrict__ xr, double *__restrict__ xi) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    xr[perm[i]] = y[i].re;
    xi[perm[i]] = y[i].im;
  }
}
// interleave the planar values (re, im) of the CSR slots
__global__ void k_cpack(int64_t nnz, const double *__restrict__ re, const double *__restrict__ im,
                        cplx *__restrict__ out) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p < nnz) out[p] = cplx(re[p], im[p]);
}

__device__ __forceinline__ cplx cldcg(const cplx *p) {
  const double2 v = __ldcg(reinterpret_cast<const double2 *>(p));
  return cplx(v.x, v.y);
}
// a -= b c, the product rounded by itself (its two parts, subtracted one by one, would each be rounded at a's size)
__device__ __forceinline__ void csubmul(cplx &a, cplx b, cplx c) {
  a.re -= fma(b.re, c.re, -(b.im * c.im));
  a.im -= fma(b.re, c.im, b.im * c.re);
}
// a += b c
__device__ __forceinline__ void caddmul(cplx &a, cplx b, cplx c) {
  a.re = fma(b.re, c.re, a.re);
  a.im = fma(b.re, c.im, a.im);
  a.re = fma(-b.im, c.im, a.re);
  a.im = fma(b.im, c.re, a.im);
}
__device__ __forceinline__ cplx cshfl(cplx v, int src) {
  return cplx(__shfl_sync(0xffffffffu, v.re, src), __shfl_sync(0xffffffffu, v.im, src));
}
// CTA of its cluster, CTAs per cluster; barrier of the cluster (global and shared writes before it are seen after it)
__device__ __forceinline__ int cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return (int)r;
}
__device__ __forceinline__ int cluster_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return (int)r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// *p of CTA k's shared memory
__device__ __forceinline__ cplx cluster_ld(const cplx *p, int k) {
  unsigned a;
  cplx v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(k));
  asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.re), "=d"(v.im) : "r"(a) : "memory");
  return v;
}
constexpr int kCB = 64;  // columns of a block

// the strictly lower part of a block's pivot triangle (columns [p0, p0 + w)) to T[c * ld + r]
__device__ __forceinline__ void stage_triangle(cplx *T, int ld, const cplx *__restrict__ L, int m, int p0, int w) {
  for (int e = threadIdx.x; e < w * kCB; e += blockDim.x) {
    const int c = e >> 6, r = e & (kCB - 1);
    if (r > c && r < w)
      cp_async<16>(T + c * ld + r, L + (int64_t)(p0 + c) * m + p0 + r);
  }
  cp_async_commit();
}
__device__ __forceinline__ void staged(bool newer) {  // all but the newest staging (newer), or all
  if (newer)
    cp_async_wait<1>();
  else
    cp_async_wait<0>();
}
// forward operand: row `row` of columns c0 + q + 4 u (below c0 + w); ok: the row exists
__device__ __forceinline__ void load_row(cplx (&v)[16], const cplx *__restrict__ L, int m, int row, bool ok, int c0, int w,
                                         int q) {
#pragma unroll
  for (int u = 0; u < 16; u++) {
    const int c = q + 4 * u;
    v[u] = (ok && c < w) ? cld(L + (int64_t)(c0 + c) * m + row) : cplx(0.0);
  }
}

// ld: leading dimension of a staged triangle; tri: its entries (two buffers when the level has a supernode of more than
// one block)
__global__ void __launch_bounds__(256) k_cfwd_level(const int *__restrict__ sn, const __grid_constant__ DevPlan P,
                                                    const cplx *__restrict__ Lx, cplx *__restrict__ y, int ld, int tri) {
  extern __shared__ __align__(16) unsigned char cs_raw[];
  cplx *T = reinterpret_cast<cplx *>(cs_raw);
  __shared__ cplx yb[kCB], ys[kCB], qs[4][kCB], pbuf[2][kCB];
  const int rank = cluster_rank(), C = cluster_size();
  const int s = sn[blockIdx.x / C];
  const int f = P.snF[s], nc = P.snNc[s], m = P.snM[s];
  const cplx *L = Lx + P.snLxp[s];
  const int *rows = P.Si + P.Sp[s];
  const int tid = threadIdx.x, lane = tid & 31, r = tid & (kCB - 1), q = tid >> 6;
  const int nblk = (nc + kCB - 1) / kCB;
  stage_triangle(T, ld, L, m, 0, min(kCB, nc));
  cplx v[16];
  const int ra = nc + kCB * rank + r;  // this CTA's first rows of ancestors
  if (nblk == 1) load_row(v, L, m, ra, ra < m, 0, nc, q);
  pdl_wait();
  pdl_next();
  for (int b = 0; b < nblk; b++) {
    const int p0 = b * kCB, w = min(kCB, nc - p0);
    cplx yin(0.0);
    if (tid < w) yin = cldcg(y + f + p0 + tid);  // rank 0 overwrites it after a barrier
    if (b == 0) {
      if (C > 1) cluster_arrive();
    } else {
      cplx acc(0.0);
      for (int i = rank; i < b; i += C) {  // column block b - 1 - i; the newest (i = 0) is in yb
        const int j = b - 1 - i;
        if (i != rank) load_row(v, L, m, p0 + r, r < w, j * kCB, kCB, q);
#pragma unroll
        for (int u = 0; u < 16; u++) {
          const int c = q + 4 * u;
          caddmul(acc, v[u], i == 0 ? yb[c] : i == rank ? ys[c] : cldcg(y + f + j * kCB + c));
        }
      }
      qs[q][r] = acc;
      __syncthreads();
      if (tid < kCB) pbuf[b & 1][tid] = (qs[0][tid] + qs[1][tid]) + (qs[2][tid] + qs[3][tid]);
      cluster_arrive();
      cluster_wait();
      if (tid < w)
        for (int k = 0; k < min(C, b); k++) yin -= cluster_ld(&pbuf[b & 1][tid], k);
    }
    if (tid < w) yb[tid] = yin;
    const bool more = b + 1 < nblk;
    if (more) {
      stage_triangle(T + ((b + 1) & 1) * tri, ld, L, m, p0 + kCB, min(kCB, nc - p0 - kCB));
      if (rank <= b) load_row(v, L, m, p0 + kCB + r, p0 + kCB + r < nc, (b - rank) * kCB, kCB, q);
    } else if (nblk > 1) {
      load_row(v, L, m, ra, ra < m, p0, w, q);
    }
    staged(more);
    __syncthreads();
    if (tid < 32) {  // the block's unit lower triangle
      const cplx *Tb = T + (b & 1) * tri;
      cplx a0 = lane < w ? yb[lane] : cplx(0.0), a1 = lane + 32 < w ? yb[lane + 32] : cplx(0.0);
      const int w0 = min(w, 32);
#pragma unroll 4
      for (int c = 0; c < w0; c++) {
        const cplx yc = cshfl(a0, c);
        if (lane > c && lane < w) csubmul(a0, Tb[c * ld + lane], yc);
        if (lane + 32 < w) csubmul(a1, Tb[c * ld + lane + 32], yc);
      }
#pragma unroll 4
      for (int c = 32; c < w; c++) {
        const cplx yc = cshfl(a1, c - 32);
        if (lane + 32 > c && lane + 32 < w) csubmul(a1, Tb[c * ld + lane + 32], yc);
      }
      if (lane < w) yb[lane] = a0;
      if (lane + 32 < w) yb[lane + 32] = a1;
    } else if (tid >= 64 && tid < 128 && more && rank > 0 && rank <= b) {
      ys[tid - 64] = cldcg(y + f + (b - rank) * kCB + tid - 64);
    }
    __syncthreads();
    if (b == 0 && C > 1) cluster_wait();
    if (rank == 0 && tid < w) y[f + p0 + tid] = yb[tid];
  }
  // the rows of ancestors: the last block's values in yb, the others' final in y since the last barrier of the cluster
  for (int k0 = nc + kCB * rank; k0 < m; k0 += kCB * C) {
    const int row = k0 + r;
    const bool ok = row < m;
    const int dst = (ok && tid < kCB) ? rows[row] : 0;
    const int pl = (nblk - 1) * kCB;
    if (k0 != nc + kCB * rank) load_row(v, L, m, row, ok, pl, nc - pl, q);
    cplx acc(0.0);
#pragma unroll
    for (int u = 0; u < 16; u++)
      if (q + 4 * u < nc - pl) caddmul(acc, v[u], yb[q + 4 * u]);
    for (int b = nblk - 2; b >= 0; b--) {
      load_row(v, L, m, row, ok, b * kCB, kCB, q);
#pragma unroll
      for (int u = 0; u < 16; u++) caddmul(acc, v[u], cldcg(y + f + b * kCB + q + 4 * u));
    }
    qs[q][r] = acc;
    __syncthreads();
    if (tid < kCB && ok) {
      const cplx t = (qs[0][tid] + qs[1][tid]) + (qs[2][tid] + qs[3][tid]);
      double *d = reinterpret_cast<double *>(y + dst);
      atomicAdd(d, -t.re);
      atomicAdd(d + 1, -t.im);
    }
    __syncthreads();
  }
  if (C > 1 && nblk > 1) {  // the others may still read this CTA's partial sums
    cluster_arrive();
    cluster_wait();
  }
}

__global__ void k_cdiag(int n, const cplx *__restrict__ D, cplx *__restrict__ y) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const double ar = D[j].re, ai = D[j].im, den = ar * ar + ai * ai, a = y[j].re, b = y[j].im;
  y[j] = cplx((a * ar + b * ai) / den, (b * ar - a * ai) / den);
}

// sum over the lanes of eight values each; lane l returns the sum of value l / 4
__device__ __forceinline__ cplx warp_sum8(cplx (&a)[8], int lane) {
#pragma unroll
  for (int o = 16, n = 4; o >= 4; o >>= 1, n >>= 1) {
    const bool hi = lane & o;
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (k < n) {
        const cplx mine = hi ? a[k + n] : a[k], other = hi ? a[k] : a[k + n];
        a[k] = cplx(mine.re + __shfl_xor_sync(0xffffffffu, other.re, o),
                    mine.im + __shfl_xor_sync(0xffffffffu, other.im, o));
      }
  }
#pragma unroll
  for (int o = 2; o > 0; o >>= 1)
    a[0] = cplx(a[0].re + __shfl_xor_sync(0xffffffffu, a[0].re, o), a[0].im + __shfl_xor_sync(0xffffffffu, a[0].im, o));
  return a[0];
}
// backward operand: rows r0 + lane and r0 + lane + 32 (below r1) of columns p0 + warp + 8 u (below p0 + w)
__device__ __forceinline__ void load_cols(cplx (&v)[8][2], const cplx *__restrict__ L, int m, int r0, int r1, int p0, int w,
                                          int warp, int lane) {
#pragma unroll
  for (int u = 0; u < 8; u++) {
    const int c = warp + 8 * u;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int row = r0 + lane + 32 * h;
      v[u][h] = (c < w && row < r1) ? cld(L + (int64_t)(p0 + c) * m + row) : cplx(0.0);
    }
  }
}

__global__ void __launch_bounds__(256) k_cbwd_level(const int *__restrict__ sn, const __grid_constant__ DevPlan P,
                                                    const cplx *__restrict__ Lx, cplx *__restrict__ y, int ld, int tri) {
  extern __shared__ __align__(16) unsigned char cs_raw[];
  cplx *T = reinterpret_cast<cplx *>(cs_raw);
  __shared__ cplx yb[kCB], ys[kCB], pbuf[2][kCB];
  const int rank = cluster_rank(), C = cluster_size();
  const int s = sn[blockIdx.x / C];
  const int f = P.snF[s], nc = P.snNc[s], m = P.snM[s];
  const cplx *L = Lx + P.snLxp[s];
  const int *rows = P.Si + P.Sp[s];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nblk = (nc + kCB - 1) / kCB, nanc = (m - nc + kCB - 1) / kCB;
  // the 64-row pieces below block b: nin = nblk - 1 - b of later blocks, then nanc of ancestors. [r0, r1) of piece i
  auto piece = [&](int b, int i, int &r0, int &r1) {
    const int nin = nblk - 1 - b;
    r0 = i < nin ? (b + 1 + i) * kCB : nc + (i - nin) * kCB;
    r1 = min(r0 + kCB, i < nin ? nc : m);
  };
  // value of row `row`: later blocks' values, or an ancestor's
  auto value = [&](int row) { return cldcg(y + (row < nc ? f + row : rows[row])); };
  cplx v[8][2];
  int r0, r1;
  stage_triangle(T + ((nblk - 1) & 1) * tri, ld, L, m, (nblk - 1) * kCB, nc - (nblk - 1) * kCB);
  piece(nblk - 1, rank, r0, r1);
  if (rank < nanc) load_cols(v, L, m, r0, r1, (nblk - 1) * kCB, nc - (nblk - 1) * kCB, warp, lane);
  pdl_wait();
  pdl_next();
  if (rank < nanc && tid < r1 - r0) ys[tid] = value(r0 + tid);
  __syncthreads();
  for (int b = nblk - 1; b >= 0; b--) {
    const int p0 = b * kCB, w = min(kCB, nc - p0), nin = nblk - 1 - b, np = nin + nanc;
    cplx yin(0.0);
    if (tid < w) yin = cldcg(y + f + p0 + tid);  // rank 0 overwrites it after the barrier
    cplx acc[8];
#pragma unroll
    for (int u = 0; u < 8; u++) acc[u] = cplx(0.0);
    for (int i = rank; i < np; i += C) {  // piece i; the newest block's values (i = 0 < nin) are in yb
      piece(b, i, r0, r1);
      if (i != rank) load_cols(v, L, m, r0, r1, p0, w, warp, lane);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int t = lane + 32 * h;
        cplx x(0.0);
        if (t < r1 - r0) x = i != rank ? value(r0 + t) : (i == 0 && nin > 0) ? yb[t] : ys[t];
#pragma unroll
        for (int u = 0; u < 8; u++) caddmul(acc[u], v[u][h], x);
      }
    }
    if (rank < np) {
      const cplx t = warp_sum8(acc, lane);
      if ((lane & 3) == 0) pbuf[b & 1][warp + 8 * (lane >> 2)] = t;
    }
    cluster_arrive();
    cluster_wait();
    if (tid < w) {
      for (int k = 0; k < min(C, np); k++) yin -= cluster_ld(&pbuf[b & 1][tid], k);
      yb[tid] = yin;
    }
    const bool more = b > 0;
    if (more) {
      stage_triangle(T + ((b - 1) & 1) * tri, ld, L, m, p0 - kCB, kCB);
      piece(b - 1, rank, r0, r1);
      if (rank < np + 1) load_cols(v, L, m, r0, r1, p0 - kCB, kCB, warp, lane);
    }
    staged(more);
    __syncthreads();
    if (tid < 32) {  // the block's unit upper triangle L11^T, last column first
      const cplx *Tb = T + (b & 1) * tri;
      cplx a0 = lane < w ? yb[lane] : cplx(0.0), a1 = lane + 32 < w ? yb[lane + 32] : cplx(0.0);
#pragma unroll 4
      for (int c = w - 1; c >= 32; c--) {
        const cplx xc = cshfl(a1, c - 32);
        csubmul(a0, Tb[lane * ld + c], xc);
        if (lane + 32 < c) csubmul(a1, Tb[(lane + 32) * ld + c], xc);
      }
#pragma unroll 4
      for (int c = min(w, 32) - 1; c > 0; c--) {
        const cplx xc = cshfl(a0, c);
        if (lane < c) csubmul(a0, Tb[lane * ld + c], xc);
      }
      if (lane < w) yb[lane] = a0;
      if (lane + 32 < w) yb[lane + 32] = a1;
    } else if (tid >= 64 && tid < 128 && more && rank > 0 && rank < np + 1 && tid - 64 < r1 - r0) {
      ys[tid - 64] = value(r0 + tid - 64);
    }
    __syncthreads();
    if (rank == 0 && tid < w) y[f + p0 + tid] = yb[tid];
  }
  if (C > 1) {  // the others may still read this CTA's partial sums
    cluster_arrive();
    cluster_wait();
  }
}

// r = b - A x (complex values on the CSR slots), norms[0] += ||r||^2, norms[1] += ||b||^2. One warp per row.
__global__ void __launch_bounds__(256) k_cresidual(int n, const int *__restrict__ rowptr, const int *__restrict__ colidx,
                                                   const cplx *__restrict__ val, const cplx *__restrict__ x,
                                                   const cplx *__restrict__ b, cplx *__restrict__ r,
                                                   double *__restrict__ norms) {
  const int lane = threadIdx.x & 31;
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (row >= n) return;
  cplx t(0.0);
  for (int p = rowptr[row] + lane; p < rowptr[row + 1]; p += 32) t += cld(val + p) * cld(x + colidx[p]);
  t = warp_sum(t);
  if (lane == 0) {
    const cplx bi = b[row], ri = bi - t;
    r[row] = ri;
    atomicAdd(norms, ri.re * ri.re + ri.im * ri.im);
    atomicAdd(norms + 1, bi.re * bi.re + bi.im * bi.im);
  }
}

__global__ void k_cpermute_vec(int n, const cplx *__restrict__ src, const int *__restrict__ perm, cplx *__restrict__ dst,
                               int gather) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (gather)
    dst[i] = src[perm[i]];
  else
    dst[perm[i]] = src[i];
}
__global__ void k_caxpy(int n, cplx *__restrict__ x, const cplx *__restrict__ dx) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] += dx[i];
}

// planar copy of a complex vector
__global__ void k_cunpack(int n, const cplx *__restrict__ x, double *__restrict__ xr, double *__restrict__ xi) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    xr[i] = x[i].re;
    xi[i] = x[i].im;
  }
}

// tau = pivotTol * max_i hypot(A(i, i)) (1 when that maximum is 0 or not a number; diagScale, ldlt.mjs:419-424)
__global__ void __launch_bounds__(1024) k_ctau(const cplx *__restrict__ values, const int *__restrict__ diagSlot, int n,
                                               double *scal) {
  __shared__ double red[32];
  double mx = 0.0;
  bool nan = false;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const cplx a = values[diagSlot[i]];
    const double h = hypot(a.re, a.im);
    if (h != h) nan = true;
    mx = fmax(mx, h);
  }
  nan = __syncthreads_or(nan);
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); w++) mx = fmax(mx, red[w]);
    scal[1] = scal[0] * ((mx > 0.0 && !nan) ? mx : 1.0);
  }
}

static unsigned nblocks(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

void launch_cunpack(int n, const cplx *x, double *xr, double *xi, cudaStream_t st) {
  if (n > 0) k_cunpack<<<nblocks(n, 256), 256, 0, st>>>(n, x, xr, xi);
}
void launch_ctau(const cplx *values, const DevPlan &P, double *scal, cudaStream_t st) {
  k_ctau<<<1, 1024, 0, st>>>(values, P.diagSlot, P.n, scal);
}

void launch_cpack(int64_t nnz, const double *re, const double *im, cplx *out, cudaStream_t st) {
  if (nnz > 0) k_cpack<<<nblocks(nnz, 256), 256, 0, st>>>(nnz, re, im, out);
}
void launch_cpermute_in(int n, const double *br, const double *bi, const int *perm, cplx *y, cudaStream_t st) {
  if (n > 0) k_cpermute_in<<<nblocks(n, 256), 256, 0, st>>>(n, br, bi, perm, y);
}
void launch_cpermute_out(int n, const cplx *y, const int *perm, double *xr, double *xi, cudaStream_t st) {
  if (n > 0) k_cpermute_out<<<nblocks(n, 256), 256, 0, st>>>(n, y, perm, xr, xi);
}
void launch_cpermute_vec(int n, const cplx *src, const int *perm, cplx *dst, bool gather, cudaStream_t st) {
  if (n > 0) k_cpermute_vec<<<nblocks(n, 256), 256, 0, st>>>(n, src, perm, dst, gather ? 1 : 0);
}
void launch_caxpy(int n, cplx *x, const cplx *dx, cudaStream_t st) {
  if (n > 0) k_caxpy<<<nblocks(n, 256), 256, 0, st>>>(n, x, dx);
}
// Kernel attributes of the level sweeps (per device)
cudaError_t init_csolve() {
  constexpr int most = 2 * kCB * (kCB + 1) * (int)sizeof(cplx);
  cudaError_t e = cudaFuncSetAttribute(k_cfwd_level, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  return e != cudaSuccess ? e : cudaFuncSetAttribute(k_cbwd_level, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
}
// The launch of a level: its widest supernode sets the shared memory, its tallest the CTAs per supernode: one per 64 rows up
// to 8, as long as the level is at most four CTAs per SM (more would only wait for one another). A solve with two, four and
// eight per SM: 642, 641 and 644 us for the edge-element system with 10 elements per edge, 1,169, 1,191 and 1,211 with 14.
CSolveLevel csolve_level(int first, int count, int maxNc, int maxM) {
  CSolveLevel v{first, count, 1, 0, 0, 0};
  while (v.cluster < 8 && v.cluster * kCB < maxM && 2 * v.cluster * (int64_t)count <= 4 * num_sms()) v.cluster *= 2;
  const int w = maxNc < kCB ? maxNc : kCB;
  v.ld = w | 1;  // odd: conflict-free by rows and by columns
  v.tri = w * v.ld;
  v.smem = (maxNc > kCB ? 2 : 1) * v.tri * (int)sizeof(cplx);
  return v;
}
template <class K>
static void launch_level(K *kernel, const CSolveLevel &v, bool after, const DevPlan &P, const cplx *L, cplx *y,
                         cudaStream_t st) {
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)v.cluster;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3((unsigned)(v.count * v.cluster));
  c.blockDim = dim3(256);
  c.dynamicSmemBytes = (size_t)v.smem;
  c.stream = st;
  c.attrs = at;
  c.numAttrs = after ? 2 : 1;
  cudaLaunchKernelEx(&c, kernel, (const int *)(P.lvlSn + v.first), P, L, y, v.ld, v.tri);
}
// y (permuted, complex) := A^-1 y: forward levels leaves first, the diagonal, backward levels top-down. A sweep's first
// launch waits for all work before it, the others only for the level before (after).
int launch_csolve_permuted(const DevPlan &P, const std::vector<CSolveLevel> &levels, const cplx *L, const cplx *D, cplx *y,
                           cudaStream_t st) {
  for (size_t i = 0; i < levels.size(); i++) launch_level(k_cfwd_level, levels[i], i > 0, P, L, y, st);
  k_cdiag<<<nblocks(P.n, 256), 256, 0, st>>>(P.n, D, y);
  for (size_t i = levels.size(); i-- > 0;) launch_level(k_cbwd_level, levels[i], i + 1 < levels.size(), P, L, y, st);
  return 2 * (int)levels.size() + 1;
}
void launch_cresidual(int n, const int *rowptr, const int *colidx, const cplx *val, const cplx *x, const cplx *b,
                      cplx *r, double *norms, cudaStream_t st) {
  if (n > 0) k_cresidual<<<nblocks((int64_t)n * 32, 256), 256, 0, st>>>(n, rowptr, colidx, val, x, b, r, norms);
}

}  // namespace amp
