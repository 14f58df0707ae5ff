// Supernodal triangular solves with several right-hand sides at once (sparse.mjs solveNumericMulti :1261-1310,
// ldlt.mjs solveMany :595-643): the same task lists and ticket order as the one-vector sweeps (solve.cu), every task
// moving a slice of up to 16 of the q <= 64 vectors.
//
// Vectors are interleaved: entry i of vector k sits at y[i q + k] (and likewise the front vectors V and the pass-up
// buffers T), so a row of the solution is q contiguous doubles and the gathers through the extend-add maps and the
// row lists move whole rows.
//
// Vector slices of 16 (ns = ceil(q / 16)), each with its own ready flags (flags[slice * nflags + block]) and done
// counters (done[slice * nsuper + s]): the host expands the block tasks into ns consecutive tasks, one per slice (int4 .w
// = the slice), so the slices' dependency chains run on different CTAs. The expanded order keeps every wait on a task with a
// smaller ticket, and a task never computes on absent vectors. The small supernodes (kind 2, one warp each, not expanded)
// solve all q vectors and count/release every slice.
//
// A task is a small GEMM on the FP64 tensor cores (mma.sync m16n8k16): out (64 rows x 16 vectors) = sum over a
// reduction index of A (64 rows x a chunk, FP32 factors widened as they are read) times B (chunk x 16), 8 warps as 4
// 16-row blocks x 2 vector halves, each with the whole reduction of its tile (no sum over warps).
// Forward: A = L[block rows, pivot columns so far], B = y[those columns]. Backward: A = the block's columns of L over
// the rows below the block, B = x[those rows]. Then the 64 x 64 inverse of the diagonal block, prefetched into shared
// memory by cp.async when the task starts, is applied the same way.
//
// What bounds a task is latency, not bandwidth: the factor's chunks, the flags, the values behind the flags and the
// children's rows were read one after the other, each a trip to L2 or HBM. So A streams through a ring of four
// cp.async stages (16 FP64 or 32 FP32 columns each; two in flight while one is multiplied, small enough for three
// CTAs per SM), the flags of up to 32 blocks (8 ancestor chunks) are polled at once, the values are read one block
// ahead of the products, and the children's rows are read ahead of their maps (solve_small.cuh). 16 vectors
// of the quadratic heat system with 32 elements per edge (FP32 factors), five sweeps each way: forward 15.4 -> 11.6 ms,
// backward 10.4 -> 8.7 ms; FP64 LDL^T factors of the edge-element system with 24: 5.25 -> 3.82 and 3.73 -> 3.20 ms.
//
// Forward, supernodes with one pivot block and at most kWholeMulti rows are one task per slice (kind 3, run_whole) in the
// levels that have more tasks than there are CTAs (expand_slices in capi.cpp has the rule and its times).
//
// Backward order: the rows below the supernode are summed from the last chunk down, each chunk after the flags of the
// ancestor blocks that hold its rows (rowBlk), so a task works while its ancestors are still being solved (the
// highest ancestors, which hold the last rows, finish first); then the supernode's own later blocks, each after its
// flag.
#include <cuda_runtime.h>

#include <cstdint>

#include "../host/plan.hpp"
#include "cp_async.cuh"
#include "devplan.cuh"
#include "solve_small.cuh"
#include "sync.cuh"

namespace amp {

constexpr int kMB = 64;   // rows of a block task
constexpr int kQS = 16;   // vectors per slice (one slice per task)
constexpr int kMQ = 64;   // vectors per pass (the host splits larger sets)
// A operands stream through a ring of stages, a chunk of the reduction index each: 16 FP64 or 32 FP32 columns
template <class TL>
constexpr int chunk_k() { return sizeof(TL) == 8 ? 16 : 32; }
constexpr int kStages = 4;
constexpr int kLdKM = kMB + 4;  // a chunk stored [k][m] (m contiguous): 4 mod 16 doubles, 4 mod 32 floats
template <class TL>
constexpr int ld_mk() { return chunk_k<TL>() + 4; }  // a chunk stored [m][k]: 20 doubles, 36 floats (conflict-free)
constexpr int kLdB = kQS + 4;  // B and R stored [k][n]: 20
constexpr int kMultiThreads = 256;
constexpr int kMultiCtas = 3;  // resident CTAs per SM of the persistent sweeps (registers capped at 80)
constexpr int kWholeMulti = 256;  // the most rows of a whole-supernode task (kind 3)
constexpr int kRingBytes = kStages * kMB * ld_mk<double>() * (int)sizeof(double);  // the largest stage: FP64 [m][k]
static_assert(kMB * ld_mk<float>() * 4 <= kMB * ld_mk<double>() * 8 && chunk_k<double>() * kLdKM <= kMB * ld_mk<double>() &&
                  chunk_k<float>() * kLdKM * 4 <= kMB * ld_mk<double>() * 8,
              "ring stage");
static_assert(kWholeMulti * kLdB * 8 <= kRingBytes && 2 * chunk_k<double>() * kLdKM * 8 <= 2 * kMB * kLdB * 8 &&
                  2 * chunk_k<float>() * kLdKM * 4 <= 2 * kMB * kLdB * 8,
              "whole-supernode tasks: the front vector in the ring, two stages in Bs");
int whole_multi_rows() { return kWholeMulti; }
// front vectors of one warp of a kind 2 task of `count` supernodes (more than kSolveGroup: m <= kTinyMid)
__host__ __device__ constexpr int small_stride(int count) { return (count > kSolveGroup ? kTinyMid : kTinyFront) * kMQ; }
constexpr int multi_smem() {
  const int own = kRingBytes + 3 * kMB * kLdB * (int)sizeof(double);
  const int small = kSolveGroup * small_stride(kSolveGroup) * (int)sizeof(double);
  static_assert(kSolveWarps * small_stride(kSolveWarps) <= kSolveGroup * small_stride(kSolveGroup), "kind 2 tasks");
  return own > small ? own : small;
}

__device__ __forceinline__ void dmma16816(double (&c)[4], const double (&a)[8], const double (&b)[4]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7,%8,%9,%10,%11}, "
      "{%12,%13,%14,%15}, {%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]), "d"(b[0]), "d"(b[1]),
        "d"(b[2]), "d"(b[3]));
}

// Fragment layouts of the m16n8k16 FP64 MMA (g = lane / 4, t = lane % 4): A (m = g + 8 (v & 1), k = t + 4 (v >> 1)),
// B (n = g, k = t + 4 v), C (m = g + 8 (v >> 1), n = 2 t + (v & 1)).
// One chunk: c += A[16 mw .. +16, 0 .. K) B[0 .. K, 8 nv .. 8 nv + 8) with K = chunk_k; A element (m, k) at A[k * kLdKM + m]
// (KM) or A[m * ld_mk + k], widened to FP64 as it is read; B element (k, n) at B[k * kLdB + n]. 8 warps: mw = warp % 4 the
// 16-row blocks, nv = warp / 4 the vector halves, so a tile needs no sum over warps.
template <bool KM, class TL>
__device__ __forceinline__ void mma_chunk(const TL *__restrict__ A, const double *__restrict__ B, int warp, int lane,
                                          double (&c)[4]) {
  const int g = lane >> 2, t = lane & 3, m0 = 16 * (warp & 3), n = 8 * (warp >> 2) + g;
#pragma unroll
  for (int k0 = 0; k0 < chunk_k<TL>(); k0 += 16) {
    double a[8], b[4];
#pragma unroll
    for (int v = 0; v < 8; v++) {
      const int m = m0 + g + 8 * (v & 1), k = k0 + t + 4 * (v >> 1);
      a[v] = (double)(KM ? A[k * kLdKM + m] : A[m * ld_mk<TL>() + k]);
    }
#pragma unroll
    for (int v = 0; v < 4; v++) b[v] = B[(k0 + t + 4 * v) * kLdB + n];
    dmma16816(c, a, b);
  }
}

// sum += c, c = 0. The long sums over FP64 factors are taken in pieces of kFold chunks (64 columns), so that a product is
// rounded at its piece's size. One sum over the whole reduction left the residual of solves without refinement 19% larger than
// the two halves that the products were once split into, pieces leave it 3 to 8% larger (elasticity, quadratic heat) to 33%
// smaller (Bunch-Kaufman), for 1 to 2% of a solve's time; pieces of one chunk took 3 to 6%, of eight no less than of four. An
// FP32 factor's own error hides the difference (equal to four digits), so its sums stay whole.
constexpr int kFold = 4;
__device__ __forceinline__ void fold(double (&sum)[4], double (&c)[4]) {
#pragma unroll
  for (int v = 0; v < 4; v++) {
    sum[v] += c[v];
    c[v] = 0.0;
  }
}

// row / vector of accumulator element v of this lane
__device__ __forceinline__ int acc_row(int warp, int lane, int v) { return 16 * (warp & 3) + (lane >> 2) + 8 * (v >> 1); }
__device__ __forceinline__ int acc_vec(int warp, int lane, int v) { return 8 * (warp >> 2) + 2 * (lane & 3) + (v & 1); }

__device__ __forceinline__ void cp_async_all() {
  cp_async_commit();
  cp_async_wait<0>();
}

// persistent ticket loop shared by both sweeps
template <class Run>
__device__ __forceinline__ void ticket_loop(int *ticket, int ntasks, Run &&run) {
  __shared__ int tk;
  for (;;) {
    if (threadIdx.x == 0) tk = atomicAdd(ticket, 1);
    __syncthreads();
    const int mine = tk;
    __syncthreads();
    if (mine >= ntasks || !run(mine)) return;
  }
}

// This task's rows [r0, r0 + rows) of the front vector v_s = [y(f .. f + nc); 0] + the children's pass-up vectors (rb:
// their 64-row block), vectors [vb, vb + qs) of q, into Rs (row r at Rs[r kLdB], kQS columns; zero outside): the
// pivot rows from y, then each child's entries that map into these rows (the schedule's gatherRange), in the
// reference's child order. Up to kGatherCh children at a time, one per thread, are waited for (their pass-up vectors of
// slice sl), so the waits of all children overlap; a child's entries are read while the one before it is added. Every task of the supernode gathers its own rows in parallel. false: a wait gave up.
constexpr int kGatherCh = 64;
// whole: rb is not used, the rows are the whole front (r0 = 0) and every child's vector is taken whole. Rs is cleared up
// to the next multiple of kMB rows.
__device__ __forceinline__ bool gather_front_rows(const DevPlan &P, int s, bool whole, int rb, int r0, int rows,
                                                  const double *__restrict__ y, const double *__restrict__ T, int *done,
                                                  int sl, int q, int vb, int qs, unsigned long long *status, double *Rs) {
  __shared__ int2 chA[kGatherCh];
  __shared__ int64_t chMap[kGatherCh], chT[kGatherCh];
  constexpr int N = 4;  // entries per thread read ahead
  const int tid = threadIdx.x, f = P.snF[s], nc = P.snNc[s];
  for (int e = tid; e < (rows + kMB - 1) / kMB * kMB * kQS; e += blockDim.x) {
    const int row = e / kQS, k = e % kQS;
    Rs[row * kLdB + k] = (row < rows && k < qs && r0 + row < nc) ? y[(int64_t)(f + r0 + row) * q + vb + k] : 0.0;
  }
  const int q0 = P.chPtr[s], q1 = P.chPtr[s + 1];
  const int64_t range0 = P.gatherOff[s] + (int64_t)rb * (q1 - q0);
  for (int qb = q0; qb < q1; qb += kGatherCh) {
    const int nq = min(kGatherCh, q1 - qb);
    if (qb > q0) __syncthreads();  // the previous chunk's ranges are consumed
    int ok = 1;
    if (tid < nq) {
      const int c = P.chList[qb + tid];
      const int muc = P.snM[c] - P.snNc[c];
      chA[tid] = whole ? make_int2(0, muc) : P.gatherRange[range0 + qb - q0 + tid];
      chMap[tid] = P.eaPtr[c];
      chT[tid] = P.snTOff[c];
      ok = wait_count(done + (int64_t)sl * P.nsuper + c, (muc + kMB - 1) / kMB, status, s, P.spin);
    }
    if (!__syncthreads_and(ok)) return false;  // block-uniform
    // the first N entries per thread of child qq (row a0 + e / kQS of its vector, vector e % kQS), and where they go
    auto fetch = [&](int qq, double(&v)[N], int(&dst)[N]) {
      const int a0 = chA[qq].x, na = chA[qq].y - a0;
#pragma unroll
      for (int u = 0; u < N; u++) {
        const int e = tid + (int)blockDim.x * u, a = a0 + e / kQS, k = e % kQS;
        dst[u] = -1;
        v[u] = 0.0;
        if (e < na * kQS && k < qs) {
          dst[u] = (P.eaMap[chMap[qq] + a] - r0) * kLdB + k;
          v[u] = __ldcg(T + (chT[qq] + a) * q + vb + k);
        }
      }
    };
    double v[N], vn[N];
    int dst[N], dn[N];
    fetch(0, v, dst);
    for (int qq = 0; qq < nq; qq++) {
      if (qq + 1 < nq) fetch(qq + 1, vn, dn);
#pragma unroll
      for (int u = 0; u < N; u++)
        if (dst[u] >= 0) Rs[dst[u]] += v[u];
      const int a0 = chA[qq].x, na = chA[qq].y - a0;
      for (int e = tid + (int)blockDim.x * N; e < na * kQS; e += blockDim.x) {
        const int a = a0 + e / kQS, k = e % kQS;
        if (k < qs) Rs[(P.eaMap[chMap[qq] + a] - r0) * kLdB + k] += __ldcg(T + (chT[qq] + a) * q + vb + k);
      }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < N; u++) {
        v[u] = vn[u];
        dst[u] = dn[u];
      }
    }
  }
  if (q0 == q1) __syncthreads();
  return true;
}

// ---- forward ------------------------------------------------------------------------------------------------------
// task (s, blk, below) of slice sl: as k_fwd_blocks. Diagonal: y[block] = X (v[block] - L[block, 0:blk 64] y[0:blk 64]);
// below: T[block] = v[block] - L[block, 0:nc] y[0:nc], where v[block] is the task's rows of the front vector, gathered
// by the task itself (gather_front_rows). With the chain matrices of a Cholesky factor (Mch, see k_chain_mats), a
// diagonal task b >= 1 forms W = X (v[block] - L[block, 0:(b-1) 64] y) before its last wait and then, after block
// b - 1's flag, y[block] = W - M_b y[block b - 1]: one 64 x 64 product per chain step instead of the block's last
// chunk, the reduction and the inverse product.
template <class TL>
__global__ void __launch_bounds__(kMultiThreads, kMultiCtas) k_fwd_multi(const int4 *__restrict__ tasks, int ntasks, int ns,
                                                                int *__restrict__ ticket, const __grid_constant__ DevPlan P,
                                                                const TL *__restrict__ Lx, const TL *__restrict__ Inv,
                                                                const TL *__restrict__ Mch, double *__restrict__ y,
                                                                double *__restrict__ T, int *__restrict__ flags,
                                                                int nflags, int epoch, int *__restrict__ done, int q,
                                                                unsigned long long *status) {
  extern __shared__ double msm[];
  constexpr int KC = chunk_k<TL>(), PB = kMB / KC;  // reduction chunk, chunks per 64-column block
  TL *ring = reinterpret_cast<TL *>(msm);
  double *Bs = msm + kRingBytes / sizeof(double), *Rs = Bs + 2 * kMB * kLdB;  // two blocks of y values; v_s, then R
  __shared__ int waitOk, sReady;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  auto bail = [] {  // a wait gave up: drain this thread's copies into shared memory before the CTA leaves
    cp_async_all();
    return false;
  };
  // one block task for vector slice sl
  auto run_slice = [&](const int4 t, const int sl) -> bool {
    const int s = t.x, blk = t.y, below = t.z;
    const int f = P.snF[s], nc = P.snNc[s], m = P.snM[s], mu = m - nc;
    const int vb = sl * kQS, qs = min(kQS, q - vb);
    const int r0 = below ? nc + blk * kMB : blk * kMB;
    const int rows = below ? min(kMB, mu - blk * kMB) : min(kMB, nc - blk * kMB);
    const bool chain = Mch != nullptr && !below && blk > 0;  // block b - 1 enters through M_b after the last wait
    const int ncols = below ? nc : (chain ? blk - 1 : blk) * kMB;
    int *myflags = flags + (int64_t)sl * nflags + P.blkOff[s];
    int *mydone = done + (int64_t)sl * P.nsuper;
    // The task's A operands, chunk after chunk: L[block rows, the columns summed], then (diagonal) the block's inverse X
    // and M_b. None depends on another task of the sweep, so they stream through the ring kStages - 1 chunks ahead.
    const int nL = (ncols + KC - 1) / KC, nX = below ? 0 : (rows + KC - 1) / KC, nM = chain ? PB : 0;
    const TL *Lb = Lx + P.snLxp[s] + r0;
    const TL *Xb = Inv + (below ? 0 : P.invOff[P.blkOff[s] + blk]);
    const TL *Mb = chain ? Mch + (int64_t)(P.blkOff[s] - s + blk - 1) * kMB * kMB : Xb;
    auto issue = [&](int i) {  // [k][m]: chunk i's element (row, column k0 + cc) at [cc kLdKM + row]
      const bool isL = i < nL, isX = !isL && i < nL + nX;
      const TL *src = isL ? Lb : isX ? Xb : Mb;
      const int ld = isL ? m : isX ? rows : kMB, lim = isL ? ncols : isX ? rows : kMB;
      const int k0 = (isL ? i : isX ? i - nL : i - nL - nX) * KC;
      TL *dst = ring + (i % kStages) * (KC * kLdKM);
      if (i < nL + nX + nM) {
#pragma unroll
        for (int u = 0; u < KC * kMB / kMultiThreads; u++) {
          const int e = tid + kMultiThreads * u, row = e & (kMB - 1), cc = e >> 6;
          const bool ok = row < rows && k0 + cc < lim;
          cp_async<sizeof(TL)>(dst + cc * kLdKM + row, ok ? src + (int64_t)(k0 + cc) * ld + row : src, ok);
        }
      }
      cp_async_commit();
    };
    for (int i = 0; i < kStages - 1; i++) issue(i);
    // this task's rows of v_s (this slice) into Rs, gathered by every task of the supernode in parallel
    if (!gather_front_rows(P, s, false, (below ? (nc + kMB - 1) / kMB : 0) + blk, r0, rows, y, T, done, sl, q, vb,
                                      qs, status, Rs))
      return bail();
    double c[4] = {0.0, 0.0, 0.0, 0.0}, sum[4] = {0.0, 0.0, 0.0, 0.0};
    // y values of a pivot block (64 x 16, four per thread): read one block ahead when that block is known final. ready:
    // the leading blocks known final, found for up to 32 blocks at a time.
    double yr[4];
    auto load_y = [&](int cb) {
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int e = tid + kMultiThreads * u, k = e >> 4, n = e & (kQS - 1);
        yr[u] = (cb + k < ncols && n < qs) ? __ldcg(y + (int64_t)(f + cb + k) * q + vb + n) : 0.0;
      }
    };
    int ready = 0;
    bool ahead = false;
    for (int i = 0; i < nL; i++) {
      const int cb = i * KC, j = cb / kMB;
      const bool first = (cb & (kMB - 1)) == 0;
      double *Bj = Bs + (j & 1) * kMB * kLdB;
      if (first) {
        if (!ahead) {
          if (ready <= j) {
            if (warp == 0) {
              const bool fin = (j + lane) * kMB < ncols && ld_acquire(myflags + j + lane) == epoch;
              int run = __ffs(~__ballot_sync(0xffffffffu, fin)) - 1;
              if (run < 0) run = 32;
              if (run == 0) {
                int ok = 1;
                if (lane == 0) ok = wait_flag(myflags + j, epoch, status, s, P.spin);
                run = __shfl_sync(0xffffffffu, ok, 0) ? 1 : -1;
              }
              if (lane == 0) sReady = run < 0 ? -1 : j + run;
            }
            __syncthreads();
            ready = sReady;
            if (ready < 0) return bail();
          }
          load_y(cb);
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int e = tid + kMultiThreads * u;
          Bj[(e >> 4) * kLdB + (e & (kQS - 1))] = yr[u];
        }
      }
      cp_async_wait<kStages - 2>();
      __syncthreads();  // chunk i and its y values have arrived; every warp is done with chunk i - 1
      if (first) {
        ahead = ready > j + 1 && cb + kMB < ncols;
        if (ahead) load_y(cb + kMB);
      }
      issue(i + kStages - 1);
      if (sizeof(TL) == 8 && i % kFold == 0) fold(sum, c);
      mma_chunk<true>(ring + (i % kStages) * (KC * kLdKM), Bj + (cb & (kMB - 1)) * kLdB, warp, lane, c);
    }
    fold(sum, c);
    // R = v[block] - the sum (the task's rows of v in Rs)
    if (below) {
      double *to = T + (P.snTOff[s] + (int64_t)blk * kMB) * q + vb;
#pragma unroll
      for (int v = 0; v < 4; v++) {
        const int row = acc_row(warp, lane, v), n = acc_vec(warp, lane, v);
        if (row < rows && n < qs) to[(int64_t)row * q + n] = Rs[row * kLdB + n] - sum[v];
      }
      __syncthreads();
      if (tid == 0) red_release_add(mydone + s, 1);
      return true;
    }
#pragma unroll
    for (int v = 0; v < 4; v++) {
      const int at = acc_row(warp, lane, v) * kLdB + acc_vec(warp, lane, v);
      Rs[at] = (acc_row(warp, lane, v) < rows && acc_vec(warp, lane, v) < qs) ? Rs[at] - sum[v] : 0.0;
    }
    // y[block] = X R
    for (int i = nL; i < nL + nX; i++) {
      cp_async_wait<kStages - 2>();
      __syncthreads();
      issue(i + kStages - 1);
      mma_chunk<true>(ring + (i % kStages) * (KC * kLdKM), Rs + (i - nL) * KC * kLdB, warp, lane, c);
    }
    if (chain) {  // y[block] = W - M_b y[block b - 1]; M_b's chunks all fit the ring now
      double wv[4];
#pragma unroll
      for (int v = 0; v < 4; v++) {
        wv[v] = c[v];
        c[v] = 0.0;
      }
      __syncthreads();  // every warp is done with X
      for (int i = nL + nX + kStages - 1; i < nL + nX + nM; i++) issue(i);
      if (tid == 0) waitOk = wait_flag(myflags + blk - 1, epoch, status, s, P.spin);
      __syncthreads();
      if (!waitOk) return bail();
      const int cp = (blk - 1) * kMB;  // block b - 1: 64 columns (not the last block)
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int e = tid + kMultiThreads * u, k = e >> 4, n = e & (kQS - 1);
        Bs[k * kLdB + n] = n < qs ? __ldcg(y + (int64_t)(f + cp + k) * q + vb + n) : 0.0;
      }
      cp_async_wait<0>();
      __syncthreads();
#pragma unroll
      for (int i = 0; i < PB; i++)
        mma_chunk<true>(ring + ((nL + nX + i) % kStages) * (KC * kLdKM), Bs + i * KC * kLdB, warp, lane, c);
#pragma unroll
      for (int v = 0; v < 4; v++) c[v] = wv[v] - c[v];
    }
#pragma unroll
    for (int v = 0; v < 4; v++) {
      const int row = acc_row(warp, lane, v), n = acc_vec(warp, lane, v);
      if (row < rows && n < qs) y[(int64_t)(f + r0 + row) * q + vb + n] = c[v];
    }
    __syncthreads();
    if (tid == 0) st_release(myflags + blk, epoch);
    return true;
  };
  // kind 3: the whole supernode s (nc <= 64, m <= kWholeMulti) for vector slice sl: its front vector v (all m rows) where
  // the ring is, y = X v[0:nc), then u = v - L[rows below, :] y in 64-row blocks: in place of a diagonal task and up to four
  // below it, each with its ticket, gather and flag.
  auto run_whole = [&](const int s, const int sl) -> bool {
    const int f = P.snF[s], nc = P.snNc[s], m = P.snM[s], mu = m - nc;
    const int vb = sl * kQS, qs = min(kQS, q - vb);
    double *V = msm;
    TL *stage = reinterpret_cast<TL *>(Bs);
    const int nK = (nc + KC - 1) / KC, nbel = (mu + kMB - 1) / kMB, total = nK + nbel * nK;
    const TL *Lb = Lx + P.snLxp[s] + nc, *Xb = Inv + P.invOff[P.blkOff[s]];
    auto issue = [&](int i) {  // chunk i: of X, then of each block of rows below; [k][m]
      if (i < total) {
        const int j = i / nK - 1, k0 = (i % nK) * KC;  // j < 0: X
        const TL *src = j < 0 ? Xb : Lb + kMB * j;
        const int ld = j < 0 ? nc : m, rows = j < 0 ? nc : min(kMB, mu - kMB * j);
        TL *dst = stage + (i & 1) * (KC * kLdKM);
#pragma unroll
        for (int u = 0; u < KC * kMB / kMultiThreads; u++) {
          const int e = tid + kMultiThreads * u, row = e & (kMB - 1), cc = e >> 6;
          const bool ok = row < rows && k0 + cc < nc;
          cp_async<sizeof(TL)>(dst + cc * kLdKM + row, ok ? src + (int64_t)(k0 + cc) * ld + row : src, ok);
        }
      }
      cp_async_commit();
    };
    issue(0);
    if (!gather_front_rows(P, s, true, 0, 0, m, y, T, done, sl, q, vb, qs, status, V)) return bail();
    for (int e = tid; e < kMB * kQS; e += kMultiThreads) {  // R = v[0:nc)
      const int row = e >> 4, n = e & (kQS - 1);
      Rs[row * kLdB + n] = row < nc ? V[row * kLdB + n] : 0.0;
    }
    double c[4] = {0.0, 0.0, 0.0, 0.0};
    for (int i = 0; i < total; i++) {
      const int j = i / nK - 1, kk = i % nK;
      cp_async_wait<0>();
      __syncthreads();  // chunk i has arrived (and R, or y, is complete); every warp is done with chunk i - 1
      issue(i + 1);
      mma_chunk<true>(stage + (i & 1) * (KC * kLdKM), Rs + kk * KC * kLdB, warp, lane, c);
      if (kk + 1 < nK) continue;
      if (j < 0) {  // y: to memory, and over R for the products below
        __syncthreads();  // every warp is done with R
#pragma unroll
        for (int v = 0; v < 4; v++) {
          const int row = acc_row(warp, lane, v), n = acc_vec(warp, lane, v);
          Rs[row * kLdB + n] = row < nc ? c[v] : 0.0;
          if (row < nc && n < qs) y[(int64_t)(f + row) * q + vb + n] = c[v];
          c[v] = 0.0;
        }
      } else {
        double *to = T + (P.snTOff[s] + (int64_t)j * kMB) * q + vb;
        const double *Vj = V + (nc + j * kMB) * kLdB;
#pragma unroll
        for (int v = 0; v < 4; v++) {
          const int row = acc_row(warp, lane, v), n = acc_vec(warp, lane, v);
          if (row < mu - j * kMB && n < qs) to[(int64_t)row * q + n] = Vj[row * kLdB + n] - c[v];
          c[v] = 0.0;
        }
      }
    }
    __syncthreads();
    if (tid == 0) {  // after the barrier: the CTA's stores of y and T are ordered before both
      st_release(flags + (int64_t)sl * nflags + P.blkOff[s], epoch);
      if (nbel > 0) red_release_add(done + (int64_t)sl * P.nsuper + s, nbel);
    }
    return true;
  };
  auto run = [&](const int tkv) -> bool {
    const int4 t = tasks[tkv];
    if (t.z == 2) {  // up to kSolveGroup supernodes with m <= 32, or kSolveWarps with m <= 16, one warp each, all vectors
      if (tid == 0) waitOk = 1;
      __syncthreads();
      if (warp < t.y && !small_fwd_warp_multi<TL>(P.solveSmall[t.x + warp], P, Lx, y, T, done, q, ns, status,
                                                  msm + small_stride(t.y) * warp))
        waitOk = 0;
      __syncthreads();
      return waitOk != 0;
    }
    if (t.z == 3) return run_whole(t.x, t.w);
    return run_slice(t, t.w);
  };
  ticket_loop(ticket, ntasks, run);
}

// ---- backward -----------------------------------------------------------------------------------------------------
// task (s, blk) of slice sl: x[block] = X^T (y[block] (/ D for LDL^T) - L[rows below the block, block columns]^T
// x[those rows]). With the chain matrices of a Cholesky factor (Gch), block b + 1 is left out of the sum and enters
// after its flag as x[block] = W - G_b^T x[block b + 1], W = X^T (y[block] - the other rows' terms).
template <class TL>
__global__ void __launch_bounds__(kMultiThreads, kMultiCtas) k_bwd_multi(const int4 *__restrict__ tasks, int ntasks, int ns,
                                                                int *__restrict__ ticket, const __grid_constant__ DevPlan P,
                                                                const TL *__restrict__ Lx, const TL *__restrict__ Inv,
                                                                const TL *__restrict__ Gch,
                                                                const double *__restrict__ Dpiv,
                                                                double *__restrict__ y, int *__restrict__ flags,
                                                                int nflags, int epoch, int q,
                                                                unsigned long long *status) {
  extern __shared__ double msm[];
  constexpr int KC = chunk_k<TL>(), PB = kMB / KC, LD = ld_mk<TL>();  // reduction chunk, chunks per block, [m][k] stride
  constexpr int NY = KC * kQS / kMultiThreads;                          // x values per thread and chunk
  TL *ring = reinterpret_cast<TL *>(msm);
  double *Bs = msm + kRingBytes / sizeof(double), *Rs = Bs + 2 * kMB * kLdB;  // x values; R
  __shared__ int waitOk, sReady, sFin[8];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  auto bail = [] {  // a wait gave up: drain this thread's copies into shared memory before the CTA leaves
    cp_async_all();
    return false;
  };
  // one block task for vector slice sl
  auto run_slice = [&](const int4 t, const int sl) -> bool {
    const int s = t.x, blk = t.y;
    const int f = P.snF[s], nc = P.snNc[s], m = P.snM[s];
    const int vb = sl * kQS, qs = min(kQS, q - vb);
    const int *rowsOf = P.Si + P.Sp[s];
    const int c0 = blk * kMB, w = min(kMB, nc - c0), nb = (nc + kMB - 1) / kMB;
    int *sflags = flags + (int64_t)sl * nflags;
    int *myflags = sflags + P.blkOff[s];
    // chunks of the reduction: the rows below the supernode [nc, m) in KC steps from the last down, then pivot blocks
    // nb - 1 .. blk + 1 (PB chunks each), then X^T and G_b^T; none of these A operands depends on another task of the
    // sweep, so they stream through the ring kStages - 1 chunks ahead
    const bool chain = Gch != nullptr && blk + 1 < nb;  // block b + 1 enters through G_b after its flag
    const int nanc = (m - nc + KC - 1) / KC;
    const int nS = nanc + (nb - 1 - blk - (chain ? 1 : 0)) * PB;  // summed chunks
    const int nX = (w + KC - 1) / KC, nG = chain ? PB : 0;
    const int rn = (blk + 1) * kMB, wn = chain ? min(kMB, nc - rn) : 0;  // the next pivot block
    auto chunk_rows = [&](int ch, int &rb, int &rw) {
      if (ch < nanc) {
        rb = nc + (nanc - 1 - ch) * KC;
        rw = min(KC, m - rb);
      } else {
        const int p = ch - nanc, pb = nb - 1 - p / PB;  // pivot block, from the last down
        rb = pb * kMB + (p % PB) * KC;
        rw = max(0, min(KC, nc - rb));
      }
    };
    const TL *Lb = Lx + P.snLxp[s] + (int64_t)c0 * m;
    const TL *Xb = Inv + P.invOff[P.blkOff[s] + blk];
    const TL *Gb = chain ? Gch + (int64_t)(P.blkOff[s] - s + blk) * kMB * kMB : Xb;
    auto issue = [&](int i) {  // [m][k]: chunk i's element (k0 + rr, column cc) at [cc LD + rr]
      if (i < nS + nX + nG) {
        const TL *src = Lb;
        int ld = m, k0, lim;
        if (i < nS) {
          int rw;
          chunk_rows(i, k0, rw);
          lim = k0 + rw;
        } else if (i < nS + nX) {
          src = Xb;
          ld = lim = w;
          k0 = (i - nS) * KC;
        } else {
          src = Gb;
          ld = kMB;
          lim = wn;
          k0 = (i - nS - nX) * KC;
        }
        TL *dst = ring + (i % kStages) * (kMB * LD);
#pragma unroll
        for (int u = 0; u < KC * kMB / kMultiThreads; u++) {
          const int e = tid + kMultiThreads * u, rr = e % KC, cc = e / KC;
          const bool ok = cc < w && k0 + rr < lim;
          cp_async<sizeof(TL)>(dst + cc * LD + rr, ok ? src + (int64_t)cc * ld + k0 + rr : src, ok);
        }
      }
      cp_async_commit();
    };
    for (int i = 0; i < kStages - 1; i++) issue(i);
    double c[4] = {0.0, 0.0, 0.0, 0.0}, sum[4] = {0.0, 0.0, 0.0, 0.0};
    // x values of a chunk (KC x 16): read one chunk ahead when its rows are known final (ready: the chunks known final,
    // found for up to eight chunks of ancestors' rows, a warp each, or 32 pivot blocks at a time); ix: the row numbers of
    // the chunk to be read next, themselves read when the one before it was
    double yr[NY];
    int ix[NY];
    auto row_index = [&](int ch) {
      int rb, rw;
      chunk_rows(ch, rb, rw);
#pragma unroll
      for (int u = 0; u < NY; u++) {
        const int rr = (tid + kMultiThreads * u) >> 4;
        ix[u] = rr >= rw ? -1 : ch < nanc ? rowsOf[rb + rr] : f + rb + rr;
      }
    };
    auto load_x = [&]() {
#pragma unroll
      for (int u = 0; u < NY; u++) {
        const int n = tid & (kQS - 1);
        yr[u] = ix[u] >= 0 && n < qs ? __ldcg(y + (int64_t)ix[u] * q + vb + n) : 0.0;
      }
    };
    int ready = 0;
    bool ahead = false;
    if (nS > 0) row_index(0);
    for (int i = 0; i < nS; i++) {
      if (!ahead) {
        if (ready <= i) {
          if (i < nanc) {
            const int ch = i + warp;
            int rb, rw;
            bool fin = false;
            if (ch < nanc) {
              chunk_rows(ch, rb, rw);
              fin = lane >= rw || ld_acquire(sflags + P.rowBlk[rowsOf[rb + lane]]) == epoch;
            }
            fin = __all_sync(0xffffffffu, fin);
            if (lane == 0) sFin[warp] = fin;
            __syncthreads();
            if (warp == 0) {
              const unsigned bits = __ballot_sync(0xffffffffu, lane < 8 && sFin[lane & 7]);
              int run = __ffs(~bits) - 1;
              if (run == 0) {  // the ancestor blocks of this chunk's rows: one lane per row, each distinct block once
                chunk_rows(i, rb, rw);
                const int fb = lane < rw ? P.rowBlk[rowsOf[rb + lane]] : -1;
                const int prev = __shfl_up_sync(0xffffffffu, fb, 1);
                int ok = 1;
                if (fb >= 0 && (lane == 0 || fb != prev)) ok = wait_flag(sflags + fb, epoch, status, s, P.spin);
                run = __all_sync(0xffffffffu, ok) ? 1 : -1;
              }
              if (lane == 0) sReady = run < 0 ? -1 : i + run;
            }
          } else if (warp == 0) {  // pivot blocks from pb down
            const int p = i - nanc, pb = nb - 1 - p / PB;
            const bool fin = pb - lane > blk && ld_acquire(myflags + pb - lane) == epoch;
            int run = __ffs(~__ballot_sync(0xffffffffu, fin)) - 1;
            if (run < 0) run = 32;
            if (run == 0) {
              int ok = 1;
              if (lane == 0) ok = wait_flag(myflags + pb, epoch, status, s, P.spin);
              run = __shfl_sync(0xffffffffu, ok, 0) ? 1 : -1;
            }
            if (lane == 0) sReady = run < 0 ? -1 : i - p % PB + run * PB;
          }
          __syncthreads();
          ready = sReady;
          if (ready < 0) return bail();
        }
        load_x();
        if (i + 1 < nS) row_index(i + 1);
      }
      double *Bi = Bs + (i & 1) * kMB * kLdB;
#pragma unroll
      for (int u = 0; u < NY; u++) {
        const int e = tid + kMultiThreads * u;
        Bi[(e >> 4) * kLdB + (e & (kQS - 1))] = yr[u];
      }
      cp_async_wait<kStages - 2>();
      __syncthreads();  // chunk i and its x values have arrived; every warp is done with chunk i - 1
      ahead = i + 1 < nS && ready > i + 1;
      if (ahead) {
        load_x();
        if (i + 2 < nS) row_index(i + 2);
      }
      issue(i + kStages - 1);
      if (sizeof(TL) == 8 && i % kFold == 0) fold(sum, c);
      mma_chunk<false>(ring + (i % kStages) * (kMB * LD), Bi, warp, lane, c);
    }
    fold(sum, c);
    // R = y[block] (/ D) - the sum
#pragma unroll
    for (int v = 0; v < 4; v++) {
      const int cc = acc_row(warp, lane, v), n = acc_vec(warp, lane, v);
      double r = 0.0;
      if (cc < w && n < qs) {
        const double yv = y[(int64_t)(f + c0 + cc) * q + vb + n];
        r = (Dpiv ? yv / Dpiv[f + c0 + cc] : yv) - sum[v];  // LDL^T: y /= D before the backward sweep (ldlt.mjs:629)
      }
      Rs[cc * kLdB + n] = r;
    }
    // x[block] = X^T R
    for (int i = nS; i < nS + nX; i++) {
      cp_async_wait<kStages - 2>();
      __syncthreads();
      issue(i + kStages - 1);
      mma_chunk<false>(ring + (i % kStages) * (kMB * LD), Rs + (i - nS) * KC * kLdB, warp, lane, c);
    }
    if (chain) {  // x[block] = W - G_b^T x[block b + 1]; G_b's chunks all fit the ring now
      double wv[4];
#pragma unroll
      for (int v = 0; v < 4; v++) {
        wv[v] = c[v];
        c[v] = 0.0;
      }
      __syncthreads();  // every warp is done with X^T
      for (int i = nS + nX + kStages - 1; i < nS + nX + nG; i++) issue(i);
      if (tid == 0) waitOk = wait_flag(myflags + blk + 1, epoch, status, s, P.spin);
      __syncthreads();
      if (!waitOk) return bail();
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int e = tid + kMultiThreads * u, r = e >> 4, n = e & (kQS - 1);
        Bs[r * kLdB + n] = (r < wn && n < qs) ? __ldcg(y + (int64_t)(f + rn + r) * q + vb + n) : 0.0;
      }
      cp_async_wait<0>();
      __syncthreads();
#pragma unroll
      for (int i = 0; i < PB; i++)
        mma_chunk<false>(ring + ((nS + nX + i) % kStages) * (kMB * LD), Bs + i * KC * kLdB, warp, lane, c);
#pragma unroll
      for (int v = 0; v < 4; v++) c[v] = wv[v] - c[v];
    }
#pragma unroll
    for (int v = 0; v < 4; v++) {
      const int cc = acc_row(warp, lane, v), n = acc_vec(warp, lane, v);
      if (cc < w && n < qs) y[(int64_t)(f + c0 + cc) * q + vb + n] = c[v];
    }
    __syncthreads();
    if (tid == 0) st_release(myflags + blk, epoch);
    return true;
  };
  auto run = [&](const int tkv) -> bool {
    const int4 t = tasks[tkv];
    if (t.z == 2) {  // up to kSolveGroup supernodes with m <= 32, or kSolveWarps with m <= 16, one warp each, all vectors
      if (tid == 0) waitOk = 1;
      __syncthreads();
      if (warp < t.y && !small_bwd_warp_multi<TL>(P.solveSmall[t.x + warp], P, Lx, Dpiv, y, flags, nflags, epoch, q,
                                                  ns, status, msm + small_stride(t.y) * warp))
        waitOk = 0;
      __syncthreads();
      return waitOk != 0;
    }
    return run_slice(t, t.w);
  };
  ticket_loop(ticket, ntasks, run);
}

// ---- layout and vector kernels -------------------------------------------------------------------------------------
// Yil[i q + k] = B[k n + i] through 32 x 32 shared tiles (both sides coalesced)
__global__ void k_to_interleaved(const double *__restrict__ B, double *__restrict__ Yil, int n, int q) {
  __shared__ double t[32][33];
  const int i0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int k = k0 + r, i = i0 + threadIdx.x;
    if (k < q && i < n) t[r][threadIdx.x] = B[(int64_t)k * n + i];
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int i = i0 + r, k = k0 + threadIdx.x;
    if (i < n && k < q) Yil[(int64_t)i * q + k] = t[threadIdx.x][r];
  }
}
// X[k n + i] = Xil[i q + k]
__global__ void k_from_interleaved(const double *__restrict__ Xil, double *__restrict__ X, int n, int q) {
  __shared__ double t[32][33];
  const int i0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int i = i0 + r, k = k0 + threadIdx.x;
    if (i < n && k < q) t[r][threadIdx.x] = Xil[(int64_t)i * q + k];
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int k = k0 + r, i = i0 + threadIdx.x;
    if (k < q && i < n) X[(int64_t)k * n + i] = t[threadIdx.x][r];
  }
}
// row gather / scatter of interleaved rows: y[i] = b[perm[i]] (in), x[perm[i]] = y[i] (out)
__global__ void k_rows_permute(const double *__restrict__ src, double *__restrict__ dst, const int *__restrict__ perm,
                               int n, int q, int scatter) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (int64_t)n * q) return;
  const int i = (int)(e / q), k = (int)(e - (int64_t)i * q);
  const int p = perm[i];
  if (scatter)
    dst[(int64_t)p * q + k] = src[e];
  else
    dst[e] = src[(int64_t)p * q + k];
}

// r = b - A x for q interleaved vectors, with the squared norms of r and b summed per (row group, vector):
// norms[2 (g q + k)] += ||r_k restricted to group g||^2, norms[2 (g q + k) + 1] += the same for b (zeroed by the
// caller). rowGroup == nullptr: one group. One warp per row, lane l holds vectors l and l + 32.
//   one group: rows grid-strided over the warps; the squares stay in registers and each block adds its sums with one
//              atomic pair per vector;
//   groups:    each warp takes a contiguous range of rows and adds its sums whenever the group changes.
__global__ void __launch_bounds__(256) k_residual_multi(int n, const int *__restrict__ rowptr,
                                                        const int *__restrict__ colidx, const double *__restrict__ val,
                                                        const double *__restrict__ x, const double *__restrict__ b,
                                                        double *__restrict__ r, double *__restrict__ norms, int q,
                                                        const int *__restrict__ rowGroup) {
  __shared__ double red[8][2 * kMQ];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k0 = lane, k1 = lane + 32;
  const bool v0 = k0 < q, v1 = k1 < q;
  double rr0 = 0.0, rr1 = 0.0, bb0 = 0.0, bb1 = 0.0;
  auto row = [&](int64_t i) {
    double s0 = 0.0, s1 = 0.0;
    const int p1 = rowptr[i + 1];
#pragma unroll 4
    for (int p = rowptr[i]; p < p1; p++) {
      const double a = val[p];
      const double *xr = x + (int64_t)colidx[p] * q;
      if (v0) s0 = fma(a, xr[k0], s0);
      if (v1) s1 = fma(a, xr[k1], s1);
    }
    if (v0) {
      const double bi = b[i * q + k0], ri = bi - s0;
      r[i * q + k0] = ri;
      rr0 += ri * ri;
      bb0 += bi * bi;
    }
    if (v1) {
      const double bi = b[i * q + k1], ri = bi - s1;
      r[i * q + k1] = ri;
      rr1 += ri * ri;
      bb1 += bi * bi;
    }
  };
  if (rowGroup) {
    const int64_t nw = (int64_t)gridDim.x * 8, gw = (int64_t)blockIdx.x * 8 + warp;
    const int64_t per = (n + nw - 1) / nw, i0 = gw * per, i1 = min((int64_t)n, i0 + per);
    int g = i0 < i1 ? rowGroup[i0] : 0;
    auto flush = [&] {
      double *nb = norms + 2 * (int64_t)g * q;
      if (v0) {
        atomicAdd(nb + 2 * k0, rr0);
        atomicAdd(nb + 2 * k0 + 1, bb0);
      }
      if (v1) {
        atomicAdd(nb + 2 * k1, rr1);
        atomicAdd(nb + 2 * k1 + 1, bb1);
      }
      rr0 = rr1 = bb0 = bb1 = 0.0;
    };
    for (int64_t i = i0; i < i1; i++) {
      const int gi = rowGroup[i];
      if (gi != g) {
        flush();
        g = gi;
      }
      row(i);
    }
    if (i0 < i1) flush();
    return;
  }
  for (int64_t i = (int64_t)blockIdx.x * 8 + warp; i < n; i += (int64_t)gridDim.x * 8) row(i);
  red[warp][2 * k0] = rr0;
  red[warp][2 * k0 + 1] = bb0;
  red[warp][2 * k1] = rr1;
  red[warp][2 * k1 + 1] = bb1;
  __syncthreads();
  if (threadIdx.x < 2 * q) {
    double a = 0.0;
    for (int w = 0; w < 8; w++) a += red[w][threadIdx.x];
    atomicAdd(norms + threadIdx.x, a);
  }
}

template <class TL>
static cudaError_t set_multi_smem() {
  cudaError_t e =
      cudaFuncSetAttribute(k_fwd_multi<TL>, cudaFuncAttributeMaxDynamicSharedMemorySize, multi_smem());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_bwd_multi<TL>, cudaFuncAttributeMaxDynamicSharedMemorySize, multi_smem());
  return e;
}
cudaError_t init_solve_multi_attributes() {
  const cudaError_t e = set_multi_smem<double>();
  return e == cudaSuccess ? set_multi_smem<float>() : e;
}

int num_sms();
int multi_max_vectors() { return kMQ; }
int multi_slices(int q) { return (q + kQS - 1) / kQS; }
int multi_resident() { return kMultiCtas * num_sms(); }
static int multi_grid(int64_t ntasks) { return ntasks < multi_resident() ? (int)ntasks : multi_resident(); }

template <class TL>
void launch_fwd_multi(const int4 *tasks, int ntasks, int *ticket, const DevPlan &P, const TL *Lx,
                      const TL *Inv, const TL *Mch, double *y, double *T, int *flags, int nflags, int epoch, int *done,
                      int q, unsigned long long *status, cudaStream_t st) {
  const int ns = multi_slices(q);
  if (ntasks <= 0) return;
  k_fwd_multi<TL><<<multi_grid(ntasks), kMultiThreads, multi_smem(), st>>>(tasks, ntasks, ns, ticket, P, Lx, Inv, Mch, y, T,
                                                                  flags, nflags, epoch, done, q, status);
}
template <class TL>
void launch_bwd_multi(const int4 *tasks, int ntasks, int *ticket, const DevPlan &P, const TL *Lx,
                      const TL *Inv, const TL *Gch, const double *Dpiv, double *y, int *flags, int nflags, int epoch,
                      int q, unsigned long long *status, cudaStream_t st) {
  const int ns = multi_slices(q);
  if (ntasks <= 0) return;
  k_bwd_multi<TL><<<multi_grid(ntasks), kMultiThreads, multi_smem(), st>>>(tasks, ntasks, ns, ticket, P, Lx, Inv, Gch, Dpiv, y,
                                                                  flags, nflags, epoch, q, status);
}
void launch_to_interleaved(const double *B, double *Yil, int n, int q, cudaStream_t st) {
  if (n > 0 && q > 0) k_to_interleaved<<<dim3((n + 31) / 32, (q + 31) / 32), dim3(32, 8), 0, st>>>(B, Yil, n, q);
}
void launch_from_interleaved(const double *Xil, double *X, int n, int q, cudaStream_t st) {
  if (n > 0 && q > 0) k_from_interleaved<<<dim3((n + 31) / 32, (q + 31) / 32), dim3(32, 8), 0, st>>>(Xil, X, n, q);
}
void launch_rows_permute(const double *src, double *dst, const int *perm, int n, int q, bool scatter, cudaStream_t st) {
  const int64_t tot = (int64_t)n * q;
  if (tot > 0) k_rows_permute<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(src, dst, perm, n, q, scatter ? 1 : 0);
}
void launch_residual_multi(int n, const int *rowptr, const int *colidx, const double *val, const double *x,
                           const double *b, double *r, double *norms, int q, const int *rowGroup, cudaStream_t st) {
  if (n <= 0 || q <= 0) return;
  const int64_t want = ((int64_t)n + 7) / 8;
  const int grid = (int)(want < 8 * num_sms() ? want : 8 * num_sms());
  k_residual_multi<<<grid, 256, 0, st>>>(n, rowptr, colidx, val, x, b, r, norms, q, rowGroup);
}
template void launch_fwd_multi<double>(const int4 *, int, int *, const DevPlan &, const double *,
                                       const double *, const double *, double *, double *, int *, int, int, int *, int,
                                       unsigned long long *, cudaStream_t);
template void launch_fwd_multi<float>(const int4 *, int, int *, const DevPlan &, const float *, const float *,
                                      const float *, double *, double *, int *, int, int, int *, int,
                                      unsigned long long *, cudaStream_t);
template void launch_bwd_multi<double>(const int4 *, int, int *, const DevPlan &, const double *,
                                       const double *, const double *, const double *, double *, int *, int, int, int,
                                       unsigned long long *, cudaStream_t);
template void launch_bwd_multi<float>(const int4 *, int, int *, const DevPlan &, const float *, const float *,
                                      const float *, const double *, double *, int *, int, int, int,
                                      unsigned long long *, cudaStream_t);

}  // namespace amp
