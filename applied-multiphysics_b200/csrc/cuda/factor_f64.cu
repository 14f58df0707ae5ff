// Multifrontal numeric factorization on sm_100a: assembly, the FP64 and complex updates.
//
// Per level of the supernodal tree (leaves first):
//   k_assemble  zero the front, scatter A's entries (sparse.mjs:965-973) and extend-add the children's update
//               matrices in the reference's child order (sparse.mjs:974-985). One CTA owns a block of 8 front
//               columns, so every entry has a single writer and the summation order is the reference's.
//   per group of up to kGroup pivot blocks of 64 columns:
//     k_group_panel  (group_panel.cu, cgroup_panel.cu for the complex factor) one dataflow launch: POTRF (or LDL^T)
//                    of each 64 x 64 pivot block, the rows below it against it (TRSM, 64-row strips, one CTA each) and
//                    the update of the group's remaining columns, ordered by flags between the strips of the launch.
//     k_update       FP64 update F -= A B^T of the columns right of the group (A = L21, or L21 D for LDL^T; B = L21;
//                    K = the group) on 128 x 64 tiles with the FP64 tensor-core MMA (mma.sync m16n8k16), covering
//                    the remaining pivot columns (in Lx) and the update block (in the U arena). The mixed-precision
//                    update is k_update_mx (update_bf16x3.cu).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "cp_async.cuh"
#include "devplan.cuh"
#include "launch.hpp"
#include "pivot_steps.cuh"
#include "sync.cuh"
#include "../host/plan.hpp"

namespace amp {

template <class T>
__device__ __forceinline__ T *front_addr(T *Lp, T *Up, int m, int nc, int i, int j) {
  // front entry (i, j), i >= j: first nc columns in the L panel (ld m), the rest in the U block (ld mu)
  return j < nc ? Lp + (int64_t)j * m + i : Up + (int64_t)(j - nc) * (m - nc) + (i - nc);
}

__device__ __forceinline__ double ldg_v(const double *p) { return __ldg(p); }
__device__ __forceinline__ cplx ldg_v(const cplx *p) {
  const double2 v = __ldg(reinterpret_cast<const double2 *>(p));
  return cplx(v.x, v.y);
}

// tau = pivotTol * max |A(i, i)| (1 when that maximum is 0 or not a number, ldlt.mjs:419-424). One CTA.
__global__ void __launch_bounds__(1024) k_ldlt_tau(const double *__restrict__ values, const int *__restrict__ diagSlot,
                                                    int n, double *scal) {
  __shared__ double red[32];
  double mx = 0.0;
  bool nan = false;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double a = fabs(values[diagSlot[i]]);
    if (a != a) nan = true;
    mx = fmax(mx, a);
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

// ---------------------------------------------------------------------------------------------------------------
// Assembly + extend-add
// ---------------------------------------------------------------------------------------------------------------
constexpr int kAsmChildren = 64;  // children whose column ranges an assembly CTA stages in shared memory up front
// extend-add entries per lane and read-modify-write step; as many are read ahead
template <class T>
constexpr int asm_step() { return sizeof(T) == 4 ? 8 : 4; }

// What bounds it is memory latency: an entry's map and value, then the front's entry behind the map. With four entries per
// lane and nothing read ahead the large fronts' children came in at 2.4 TB/s; now the next entries (eight FP32, four
// wider) are read while the current ones are added, four CTAs per SM (64 registers; with three or five the launches are
// slower). 40^3 elasticity, FP32 fronts: 3.29 -> 2.73 ms (3 CTAs 3.05, 5 CTAs 3.33), FP64 4.59 -> 4.29; quadratic heat
// with 32 elements per edge 4.38 -> 3.53 ms.
// ranges[t.ch0 + q]: the columns of child q's update matrix that map into the task's front columns (computed with
// the schedule, so a CTA starts without searching the children's maps)
template <class T>
__global__ void __launch_bounds__(256, 4) k_assemble(const AsmTask *__restrict__ tasks, const ChildRange *__restrict__ ranges,
                                                  DevPlan P, const value_of<T> *__restrict__ values, T *__restrict__ Lx,
                                                  T *__restrict__ U, const unsigned long long *status) {
  if (cta_failed(status)) return;
  const AsmTask t = tasks[blockIdx.x];
  const int s = t.s, j0 = t.j0;
  const int f = P.snF[s], nc = P.snNc[s], m = P.snM[s];
  const int jend = min(j0 + kAsmCols, m);
  T *Lp = Lx + P.snLxp[s];
  T *Up = (m > nc) ? U + P.snUoff[s] : nullptr;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  // 0. the child columns mapping into [j0, jend) (one range per child, the first kAsmChildren children staged in
  // shared memory while the columns are zeroed)
  __shared__ ChildRange chRange[kAsmChildren];
  const int q0 = P.chPtr[s], nch = P.chPtr[s + 1] - q0;
  const ChildRange *rg = ranges + t.ch0;
  if ((int)threadIdx.x < min(nch, kAsmChildren)) chRange[threadIdx.x] = rg[threadIdx.x];
  // 1. zero the lower part of the owned columns
  for (int j = j0 + warp; j < jend; j += nwarps)
    for (int i = j + lane; i < m; i += 32) *front_addr(Lp, Up, m, nc, i, j) = T(0);
  __syncthreads();
  // 2. A's entries of the owned pivot columns (each (row, col) once); 4 entries per lane in flight
  for (int j = j0 + warp; j < min(jend, nc); j += nwarps) {
    const int p0 = P.asmColPtr[f + j], p1 = P.asmColPtr[f + j + 1];
    for (int p = p0 + lane; p < p1; p += 128) {
      int dst[4];
      T v[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int pp = p + 32 * u;
        dst[u] = pp < p1 ? P.asmDst[pp] : -1;
        v[u] = pp < p1 ? (T)ldg_v(values + P.asmSrc[pp]) : T(0);
      }
      T cur[4];
#pragma unroll
      for (int u = 0; u < 4; u++) cur[u] = dst[u] >= 0 ? Lp[dst[u]] : T(0);
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (dst[u] >= 0) Lp[dst[u]] = cur[u] + v[u];
    }
  }
  __syncthreads();
  // 3. children, one after another (stack order of the reference)
  constexpr int N = asm_step<T>();
  for (int q = 0; q < nch; q++) {
    const int c = P.chList[q0 + q];
    const int muc = P.snM[c] - P.snNc[c];
    if (muc <= 0) continue;  // block-uniform
    const int *map = P.eaMap + P.eaPtr[c];
    const T *Uc = U + P.snUoff[c];
    const ChildRange br = q < kAsmChildren ? chRange[q] : rg[q];
    for (int b = br.b0 + warp; b < br.b1; b += nwarps) {
      const int jj = map[b];
      const T *col = Uc + (int64_t)b * muc;
      T *to = jj < nc ? Lp + (int64_t)jj * m : Up + (int64_t)(jj - nc) * (m - nc) - nc;  // row i of front column jj
      int dst[N], dn[N];
      T v[N], vn[N];
      auto fetch = [&](int a, int(&d)[N], T(&x)[N]) {
#pragma unroll
        for (int u = 0; u < N; u++) {
          const int aa = a + 32 * u;
          d[u] = aa < muc ? __ldg(map + aa) : -1;
          x[u] = aa < muc ? col[aa] : T(0);
        }
      };
      fetch(b + lane, dst, v);
      for (int a = b + lane; a - lane < muc; a += 32 * N) {
        fetch(a + 32 * N, dn, vn);
        T cur[N];
#pragma unroll
        for (int u = 0; u < N; u++) cur[u] = dst[u] >= 0 ? to[dst[u]] : T(0);
#pragma unroll
        for (int u = 0; u < N; u++)
          if (dst[u] >= 0) to[dst[u]] = cur[u] + v[u];
#pragma unroll
        for (int u = 0; u < N; u++) {
          dst[u] = dn[u];
          v[u] = vn[u];
        }
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Trailing update: F[i0:i0+128, j0:j0+64] -= A B^T with A = panel rows i, B = panel rows j, K = the task's pivot columns.
// The product runs on the FP64 tensor cores with mma.sync m16n8k16 (fragment layouts of the SM90 FP64 MMA atoms:
// A (m = g + 8 (v & 1), k = t + 4 (v >> 1)), B (n = g, k = t + 4 v), C (m = g + 8 (v >> 1), n = 2 t + (v & 1)),
// g = lane / 4, t = lane % 4), the panel rows in shared memory by cp.async.
// What bounds it: the FP64 pipe (36.5 TFLOP/s on 148 SMs), when something else issues the loads meanwhile. A thread's
// panel rows come in 8-byte copies (a column of the front starts on any 8-byte boundary), so the copies of a chunk are
// hundreds of instructions, and with one CTA of 8 warps per SM the pipe idled while all of them copied: 24 TFLOP/s in
// the largest launches. Hence CTAs of 4 warps, two or three per SM, that copy while another one multiplies: 28 TFLOP/s
// there (40^3 elasticity, 84 GFLOP: 3.51 -> 3.00 ms). Issuing the copies between a warp's own products was slower (25
// TFLOP/s: a warp that has issued a product issues nothing else until the pipe takes the next one).
// The front's entries of a tile come into L2 while its last two chunks are multiplied (128-row CTAs only; in launches of few
// tiles it costs more than it gives): 40^3 elasticity, all updates 36.0 -> 35.6 ms.
// ROWS = 128: warps of 64 x 32; 64: half a task per CTA, warps of 32 x 32, for launches of few tasks (see launch_update).
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void dmma_16x8x16(double (&c)[4], const double (&a)[8], const double (&b)[4]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7,%8,%9,%10,%11}, "
      "{%12,%13,%14,%15}, {%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]), "d"(b[0]), "d"(b[1]),
        "d"(b[2]), "d"(b[3]));
}

constexpr int kChunk = 32;  // pivot columns per pipeline stage
// leading dimensions in shared memory: 4 mod 16 doubles, conflict-free fragment loads
template <int ROWS>
constexpr int upd_stage() { return kChunk * (ROWS + 4) + kChunk * (kTile + 4); }  // doubles
template <int ROWS>
constexpr int upd_smem() { return 2 * upd_stage<ROWS>() * (int)sizeof(double); }

// Rows [i0, i0 + R) of the front's columns [k0, k0 + kChunk) into dst (column-major, ld R + 4), zero past m rows or kend.
template <int R>
__device__ __forceinline__ void stage_rows(double *dst, const double *src, int m, int i0, int k0, int kend) {
  constexpr int STEP = 128 / R;
  const int i = threadIdx.x & (R - 1), kb = threadIdx.x / R, r = i0 + i;
  const bool rowok = r < m;
  const double *p = src + (int64_t)(k0 + kb) * m + (rowok ? r : 0);
#pragma unroll 8
  for (int k = kb; k < kChunk; k += STEP, p += (int64_t)STEP * m) {
    const bool ok = rowok && k0 + k < kend;
    cp_async<8>(dst + k * (R + 4) + i, ok ? p : src, ok);
  }
}

// Persistent CTAs walk (tile, chunk) items; the next item's panel rows stream into the other stage while the current one
// runs; the C tile is read and written once, after the tile's last chunk.
template <int ROWS>
__global__ void __launch_bounds__(128, ROWS == 128 ? 2 : 3)
    k_update(const TileTask *__restrict__ tasks, int ntasks, double *__restrict__ Lx, double *__restrict__ U,
             const double *__restrict__ W, const unsigned long long *status) {
  if (cta_failed(status)) return;
  constexpr int SPLIT = kTileM / ROWS, MA = ROWS / 32;  // CTA tiles per task; 16-row fragments per warp
  const double *Ax = W ? W : Lx;                        // LDL^T: A = L21 D
  extern __shared__ double smem_upd[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wr = (warp >> 1) * (ROWS / 2), wc = (warp & 1) * 32;
  const int g = lane >> 2, t4 = lane & 3;
  const int nitems = ntasks * SPLIT;
  int t = blockIdx.x;
  // the item's task with its own rows; an item past the front's last row or above its diagonal has none
  auto item = [&](int x, TileTask &k) {
    k = tasks[x / SPLIT];
    k.i0 += (x % SPLIT) * ROWS;
  };
  auto empty = [&](const TileTask &k) { return k.i0 >= k.m || k.i0 + ROWS <= k.j0; };
  TileTask cur;
  for (;; t += gridDim.x) {
    if (t >= nitems) return;
    item(t, cur);
    if (!empty(cur)) break;
  }
  auto loads = [&](const TileTask &k, int chunk, double *stage) {
    const int k0 = k.c0 + chunk * kChunk, kend = k.c0 + k.w;
    stage_rows<ROWS>(stage, Ax + k.lp, k.m, k.i0, k0, kend);
    stage_rows<kTile>(stage + kChunk * (ROWS + 4), Lx + k.lp, k.m, k.j0, k0, kend);
  };
  int stage = 0;
  loads(cur, 0, smem_upd);
  cp_async_commit();
  while (true) {
    TileTask next = cur;
    int tn = t + gridDim.x;
    for (; tn < nitems; tn += gridDim.x) {
      item(tn, next);
      if (!empty(next)) break;
    }
    const int m = cur.m, nc = cur.nc, nch = (cur.w + kChunk - 1) / kChunk;
    const bool active = cur.i0 + wr < m && cur.i0 + wr + ROWS / 2 > cur.j0 + wc;  // the warp's part has entries
    double acc[MA][4][4];
#pragma unroll
    for (int a = 0; a < MA; a++)
#pragma unroll
      for (int b = 0; b < 4; b++)
#pragma unroll
        for (int v = 0; v < 4; v++) acc[a][b][v] = 0.0;
    for (int chunk = 0; chunk < nch; chunk++) {
      const bool more = chunk + 1 < nch || tn < nitems;
      if (more)
        loads(chunk + 1 < nch ? cur : next, chunk + 1 < nch ? chunk + 1 : 0, smem_upd + (stage ^ 1) * upd_stage<ROWS>());
      cp_async_commit();
      if (ROWS == 128 && chunk == max(nch - 2, 0)) {  // the tile's entries of the front into L2, 16 rows of a column per thread and step
        double *Lp = Lx + cur.lp;
        double *Up = cur.up >= 0 ? U + cur.up : Lp;
#pragma unroll
        for (int e = tid; e < ROWS / 16 * kTile; e += 128) {
          const int i = cur.i0 + 16 * (e % (ROWS / 16)), j = cur.j0 + e / (ROWS / 16);
          if (i < m && j < cur.jend && i + 15 >= j) {
            const double *to = j < nc ? Lp + (int64_t)j * m + i : Up + (int64_t)(j - nc) * (m - nc) + max(i - nc, 0);
            asm volatile("prefetch.global.L2 [%0];\n" ::"l"(to));
          }
        }
      }
      if (more) cp_async_wait<1>(); else cp_async_wait<0>();
      __syncthreads();
      if (active) {
        const double *As = smem_upd + stage * upd_stage<ROWS>() + wr + g;
        const double *Bs = smem_upd + stage * upd_stage<ROWS>() + kChunk * (ROWS + 4) + wc + g;
        const int kw = min(kChunk, cur.w - chunk * kChunk);
#pragma unroll
        for (int kk = 0; kk < kChunk; kk += 16) {
          if (kk >= kw) break;
          const double *Ak = As + (kk + t4) * (ROWS + 4), *Bk = Bs + (kk + t4) * (kTile + 4);
          double bf[4][4];
#pragma unroll
          for (int b = 0; b < 4; b++)
#pragma unroll
            for (int v = 0; v < 4; v++) bf[b][v] = Bk[4 * v * (kTile + 4) + 8 * b];
#pragma unroll
          for (int a = 0; a < MA; a++) {
            double af[8];
#pragma unroll
            for (int v = 0; v < 8; v++) af[v] = Ak[4 * (v >> 1) * (ROWS + 4) + 16 * a + 8 * (v & 1)];
#pragma unroll
            for (int b = 0; b < 4; b++) dmma_16x8x16(acc[a][b], af, bf[b]);
          }
        }
      }
      __syncthreads();  // this stage is free for the item after next
      stage ^= 1;
    }
    if (active) {  // C -= the product: half of the warp's rows at a time, their entries in flight together
      double *Lp = Lx + cur.lp;
      double *Up = cur.up >= 0 ? U + cur.up : Lp;
      constexpr int H = MA / 2;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        double cv[H][4][4];
#pragma unroll
        for (int pass = 0; pass < 2; pass++)
#pragma unroll
          for (int b = 0; b < 4; b++)
#pragma unroll
            for (int u = 0; u < 2; u++) {
              const int j = cur.j0 + wc + 8 * b + 2 * t4 + u;
              double *col = j < nc ? Lp + (int64_t)j * m : Up + (int64_t)(j - nc) * (m - nc) - nc;
#pragma unroll
              for (int a = 0; a < H; a++)
#pragma unroll
                for (int v = 0; v < 2; v++) {
                  const int i = cur.i0 + wr + 16 * (h * H + a) + g + 8 * v;
                  if (i >= m || i < j || j >= cur.jend) continue;
                  if (pass == 0)
                    cv[a][b][2 * v + u] = col[i];
                  else
                    col[i] = cv[a][b][2 * v + u] - acc[h * H + a][b][2 * v + u];
                }
            }
      }
    }
    if (tn >= nitems) return;
    t = tn;
    cur = next;
  }
}


// Complex-symmetric update tiles (no conjugation): F[i0:i0+128, j0:j0+64] -= W B^T with W = L21 D (the A operand of
// the LDL^T update) and B = L21, K = the task's pivot columns, four FP64 tensor-core products (mma.sync m8n8k4) per complex
// one. A task is split into TS x TS squares of its tile, one CTA of 4 warps (2 x 2, TS / 2 rows and columns each) per square;
// the operands come through a ring of four cp.async stages of 16 pivot columns. What bounds it at the sizes of complex
// systems is the latency of one square (the launches of a front's groups follow one another and have few tasks): 128 x 64
// per CTA, 8 columns at a time copied and then multiplied, took 66 us per launch for the edge-element system with 10
// elements per edge, now 15 us.
constexpr int kCK = 16, kCStages = 4;
template <int TS>
constexpr int cupd_ld() { return TS + 2; }  // 2 mod 8 entries of 16 bytes: conflict-free fragment loads
template <int TS>
constexpr int cupd_smem() { return kCStages * 2 * kCK * cupd_ld<TS>() * (int)sizeof(cplx); }
template <int TS>
__global__ void __launch_bounds__(128) k_update_c(const TileTask *__restrict__ tasks, cplx *__restrict__ Lx,
                                                  cplx *__restrict__ U, const cplx *__restrict__ W,
                                                  const unsigned long long *status) {
  constexpr int LD = cupd_ld<TS>(), PER = (kTileM / TS) * (kTile / TS), ROWS = kTileM / TS, MT = TS / 16;
  extern __shared__ __align__(16) cplx cu_raw[];
  const TileTask t = tasks[blockIdx.x / PER];
  const int sub = blockIdx.x % PER, i0 = t.i0 + TS * (sub % ROWS), j0 = t.j0 + TS * (sub / ROWS);
  const int m = t.m, nc = t.nc, jend = t.jend;
  if (i0 >= m || j0 >= jend || i0 + TS <= j0) return;
  __shared__ int sOk;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  if (tid == 0) sOk = !factor_failed(status);
  const cplx *Ap = W + t.lp + (int64_t)t.c0 * m, *Bp = Lx + t.lp + (int64_t)t.c0 * m;
  const int nchunk = (t.w + kCK - 1) / kCK;
  auto stage = [&](int ch) {
    cplx *As = cu_raw + (ch % kCStages) * 2 * kCK * LD, *Bs = As + kCK * LD;
    if (ch < nchunk) {
      const int i = tid & (TS - 1);
#pragma unroll
      for (int k = tid / TS; k < kCK; k += 128 / TS) {
        const int c = ch * kCK + k;
        const bool okA = c < t.w && i0 + i < m, okB = c < t.w && j0 + i < m;
        cp_async<16>(As + k * LD + i, Ap + (okA ? (int64_t)c * m + i0 + i : 0), okA);
        cp_async<16>(Bs + k * LD + i, Bp + (okB ? (int64_t)c * m + j0 + i : 0), okB);
      }
    }
    cp_async_commit();
  };
  for (int ch = 0; ch < kCStages - 1; ch++) stage(ch);
  __syncthreads();
  if (!sOk) {
    cp_async_wait<0>();
    return;
  }
  const int wr = TS / 2 * (warp & 1), wc = TS / 2 * (warp >> 1);
  double re[MT][MT][2], im[MT][MT][2];
#pragma unroll
  for (int a = 0; a < MT; a++)
#pragma unroll
    for (int b = 0; b < MT; b++) re[a][b][0] = re[a][b][1] = im[a][b][0] = im[a][b][1] = 0.0;
  for (int ch = 0; ch < nchunk; ch++) {
    cp_async_wait<kCStages - 2>();
    __syncthreads();  // chunk ch has arrived, and everyone is done with chunk ch - 1
    stage(ch + kCStages - 1);
    const cplx *As = cu_raw + (ch % kCStages) * 2 * kCK * LD, *Bs = As + kCK * LD;
#pragma unroll
    for (int k = 0; k < kCK; k += 4) {
      cplx av[MT], bv[MT];
#pragma unroll
      for (int a = 0; a < MT; a++) av[a] = As[(k + q) * LD + wr + 8 * a + g];
#pragma unroll
      for (int b = 0; b < MT; b++) bv[b] = Bs[(k + q) * LD + wc + 8 * b + g];
#pragma unroll
      for (int a = 0; a < MT; a++) {
        const double ni = -av[a].im;
#pragma unroll
        for (int b = 0; b < MT; b++) mma884(re[a][b], av[a].re, bv[b].re);
#pragma unroll
        for (int b = 0; b < MT; b++) mma884(im[a][b], av[a].re, bv[b].im);
#pragma unroll
        for (int b = 0; b < MT; b++) mma884(re[a][b], ni, bv[b].im);
#pragma unroll
        for (int b = 0; b < MT; b++) mma884(im[a][b], av[a].im, bv[b].re);
      }
    }
  }
  cp_async_wait<0>();
  cplx *Lp = Lx + t.lp;
  cplx *Up = t.up >= 0 ? U + t.up : Lp;
#pragma unroll
  for (int b = 0; b < MT; b++) {  // C -= the product, a column of squares' entries in flight together
    cplx cv[MT][2];
#pragma unroll
    for (int pass = 0; pass < 2; pass++)
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int j = j0 + wc + 8 * b + 2 * q + u;
        cplx *col = j < nc ? Lp + (int64_t)j * m : Up + (int64_t)(j - nc) * (m - nc) - nc;
#pragma unroll
        for (int a = 0; a < MT; a++) {
          const int i = i0 + wr + 8 * a + g;
          if (i >= m || i < j || j >= jend) continue;
          if (pass == 0)
            cv[a][u] = col[i];
          else
            col[i] = cplx(cv[a][u].re - re[a][b][u], cv[a][u].im - im[a][b][u]);
        }
      }
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Solves. Vectors: q right-hand sides stored one after another (y[k n + i]) in the permuted order.
// ---------------------------------------------------------------------------------------------------------------
__global__ void k_permute_in(const double *__restrict__ b, double *__restrict__ y, const int *__restrict__ perm, int n,
                             int q) {
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)n * q) return;
  int k = (int)(idx / n), i = (int)(idx % n);
  y[idx] = b[(int64_t)k * n + perm[i]];
}

__global__ void k_permute_out(const double *__restrict__ y, double *__restrict__ x, const int *__restrict__ perm, int n,
                              int q) {
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)n * q) return;
  int k = (int)(idx / n), i = (int)(idx % n);
  x[(int64_t)k * n + perm[i]] = y[idx];
}

// ---------------------------------------------------------------------------------------------------------------
// Launchers (host side)
// ---------------------------------------------------------------------------------------------------------------
static int g_num_sms = 148;

cudaError_t init_group_panel_attributes();
cudaError_t init_cgroup_panel_attributes();
cudaError_t init_group_panel_f32_attributes();
cudaError_t init_front_small_f32_attributes();
cudaError_t init_mixed_attributes();
cudaError_t init_solve_attributes();
cudaError_t init_solve_multi_attributes();
cudaError_t init_front_small_attributes();
cudaError_t init_kernel_attributes() {
  // function attributes belong to the current device's context: the caller runs this once per device
  cudaError_t e = init_group_panel_attributes();
  if (e == cudaSuccess) e = init_cgroup_panel_attributes();
  if (e == cudaSuccess) e = init_group_panel_f32_attributes();
  if (e == cudaSuccess) e = init_front_small_f32_attributes();
  if (e == cudaSuccess) e = init_mixed_attributes();
  if (e == cudaSuccess) e = init_solve_attributes();
  if (e == cudaSuccess) e = init_solve_multi_attributes();
  if (e == cudaSuccess) e = init_front_small_attributes();
  if (e == cudaSuccess) e = init_csolve();
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_update<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, upd_smem<128>());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_update<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, upd_smem<64>());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_update_c<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, cupd_smem<32>());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_update_c<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, cupd_smem<64>());
  int dev = 0;
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
  return e;
}

template <class T>
void launch_assemble(const AsmTask *tasks, const ChildRange *ranges, int64_t ntasks, const DevPlan &P,
                     const value_of<T> *values, T *Lx, T *U, const unsigned long long *status, cudaStream_t st) {
  if (ntasks > 0) k_assemble<T><<<(unsigned)ntasks, 256, 0, st>>>(tasks, ranges, P, values, Lx, U, status);
}
template void launch_assemble<double>(const AsmTask *, const ChildRange *, int64_t, const DevPlan &, const double *,
                                      double *, double *, const unsigned long long *, cudaStream_t);
template void launch_assemble<float>(const AsmTask *, const ChildRange *, int64_t, const DevPlan &, const double *,
                                     float *, float *, const unsigned long long *, cudaStream_t);
template void launch_assemble<cplx>(const AsmTask *, const ChildRange *, int64_t, const DevPlan &, const cplx *,
                                    cplx *, cplx *, const unsigned long long *, cudaStream_t);
void launch_update_c(const TileTask *tasks, int64_t ntasks, cplx *Lx, cplx *U, const cplx *W,
                     const unsigned long long *status, cudaStream_t st) {
  if (ntasks <= 0) return;
  // squares of 32 while the tasks' squares of 64 are fewer than two per SM: a quarter of a square's latency, and four times
  // the CTAs; beyond that squares of 64, which read each operand half as often
  if (2 * ntasks <= 2 * g_num_sms)
    k_update_c<32><<<(unsigned)(8 * ntasks), 128, cupd_smem<32>(), st>>>(tasks, Lx, U, W, status);
  else
    k_update_c<64><<<(unsigned)(2 * ntasks), 128, cupd_smem<64>(), st>>>(tasks, Lx, U, W, status);
}
void launch_ldlt_tau(const double *values, const DevPlan &P, double *scal, cudaStream_t st) {
  k_ldlt_tau<<<1, 1024, 0, st>>>(values, P.diagSlot, P.n, scal);
}
int num_sms() { return g_num_sms; }
void launch_update(const TileTask *tasks, int64_t ntasks, const DevPlan &P, double *Lx, double *U, const double *W,
                   const unsigned long long *status, cudaStream_t st) {
  (void)P;
  if (ntasks <= 0) return;
  // 64-row CTAs when they all fit at once (three per SM): twice the CTAs for a launch that would leave SMs idle, and a
  // tile's latency halved on the chain through a front's groups. With more tasks the 128-row CTAs copy a quarter less
  // per product: 28 against 27 TFLOP/s in the largest launches.
  if (2 * ntasks <= 3 * g_num_sms)
    k_update<64><<<(unsigned)(2 * ntasks), 128, upd_smem<64>(), st>>>(tasks, (int)ntasks, Lx, U, W, status);
  else
    k_update<128><<<(unsigned)std::min<int64_t>(ntasks, 2 * g_num_sms), 128, upd_smem<128>(), st>>>(
        tasks, (int)ntasks, Lx, U, W, status);
}
void launch_permute_in(const double *b, double *y, const int *perm, int n, int q, cudaStream_t st) {
  int64_t tot = (int64_t)n * q;
  if (tot > 0) k_permute_in<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(b, y, perm, n, q);
}
void launch_permute_out(const double *y, double *x, const int *perm, int n, int q, cudaStream_t st) {
  int64_t tot = (int64_t)n * q;
  if (tot > 0) k_permute_out<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(y, x, perm, n, q);
}
}  // namespace amp
