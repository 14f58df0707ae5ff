// Small fronts of the FP32 factors of the mixed-precision path (front_small.cu has the FP64 factors'): one warp (m <= 32) or
// one CTA (32 < m <= 128) per front, a column per phase in shared memory, in FP32 (FP64 for LDL^T, rounded once when stored).
// As with the FP32 group panel, the order of the FP32 operations is what a caller of an unrefined solve sees; the
// eight-column register tiles of the FP64 kernels have another.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "../host/plan.hpp"
#include "devplan.cuh"
#include "launch.hpp"
#include "small_fronts.cuh"
#include "sync.cuh"

namespace amp {

namespace {

// Zero F (m x m), add A's entries of the pivot columns and the children's update matrices in the reference's order.
template <class TC, int G>
__device__ void assemble_front(int s, const DevPlan &P, const double *__restrict__ values, const float *__restrict__ U,
                               TC *F, int t, ChildMeta *cm) {
  const int warp = t >> 5, lane = t & 31;
  const int f = P.snF[s], nc = P.snNc[s], m = P.snM[s];
  for (int e = t; e < m * m; e += G) F[e] = TC(0);
  group_sync<G>();
  // A's entries of all nc pivot columns (one contiguous CSR range): slot dst = j m + i of the L panel, each (i, j) once
  {
    const int p0 = P.asmColPtr[f], p1 = P.asmColPtr[f + nc];
    for (int p = p0 + t; p < p1; p += G) F[P.asmDst[p]] += (TC)(float)__ldg(values + P.asmSrc[p]);
  }
  group_sync<G>();
  // children's update matrices, one after another (the map is injective within a child); the metadata of up to
  // kChildChunk children is fetched at once, one child per thread
  const int q0 = P.chPtr[s], q1 = P.chPtr[s + 1];
  for (int qb = q0; qb < q1; qb += kChildChunk) {
    const int nq = min(kChildChunk, q1 - qb);
    int muc = 0;
    int64_t ea = 0, uo = 0;
    if (warp == 0 && lane < nq) {
      const int c = P.chList[qb + lane];
      muc = P.snM[c] - P.snNc[c];
      ea = P.eaPtr[c];
      uo = P.snUoff[c];
    }
    if constexpr (G > 32) {
      if (qb > q0) __syncthreads();  // the previous chunk's metadata is read by all warps before it is replaced
      if (warp == 0 && lane < nq) {
        cm->muc[lane] = muc;
        cm->ea[lane] = ea;
        cm->uo[lane] = uo;
      }
      __syncthreads();
    }
    for (int q = 0; q < nq; q++) {
      int mq;
      int64_t eq, uq;
      if constexpr (G == 32) {
        mq = __shfl_sync(0xffffffffu, muc, q);
        eq = __shfl_sync(0xffffffffu, ea, q);
        uq = __shfl_sync(0xffffffffu, uo, q);
      } else {
        mq = cm->muc[q];
        eq = cm->ea[q];
        uq = cm->uo[q];
      }
      if (mq <= 0) continue;  // group-uniform
      const int *map = P.eaMap + eq;
      const float *Uc = U + uq;
      for (int e = t; e < mq * mq; e += G) {
        const int b = e / mq, a = e - b * mq;
        if (a >= b) F[map[b] * m + map[a]] += (TC)Uc[e];
      }
      group_sync<G>();
    }
  }
}

// The whole front of supernode s by a group of G threads (thread t) over the shared m x m column-major tile F, in the
// compute type TC (FP32 as L and U, or FP64: an FP32 LDL^T factor's small fronts are computed in FP64
// and rounded once when stored, since the indefinite factor's pivots cancel). cm: the group's child metadata (G > 32;
// a warp passes its child metadata by shuffles).
//
// Column k of the elimination is one phase with one barrier: every thread reads the pivot F(k, k) (final since the
// previous barrier), computes the same pivot decision and scale, writes its share of L's column k straight to Lx and
// updates its share of the trailing triangle from the unscaled column k, which nobody writes in the phase. The
// arithmetic is the column-scaled form's: l_i = F(i, k) / r (Cholesky, r = sqrt F(k, k)) or F(i, k) / d (LDL^T), and
// F(i, j) -= l_i (l_j d) with d = 1 for Cholesky.
template <class TC, int G>
__device__ void factor_front(int s, const DevPlan &P, const double *__restrict__ values, float *__restrict__ Lx,
                             float *__restrict__ U, TC *F, unsigned long long *status, const LdltArgs<float> &la, int t,
                             ChildMeta *cm) {
  constexpr int NW = G / 32;
  const int warp = t >> 5, lane = t & 31;
  const int f = P.snF[s], nc = P.snNc[s], m = P.snM[s], mu = m - nc;
  const bool ldlt = la.scal != nullptr;
  const TC tau = ldlt ? (TC)(float)la.scal[1] : TC(0);
  assemble_front<TC, G>(s, P, values, U, F, t, cm);
  // partial factorization of the nc pivot columns, one barrier per column; warps over the trailing columns j, lanes
  // over the rows i >= j
  int neg = 0, pert = 0;  // thread 0
  float *Lp = Lx + P.snLxp[s];
  for (int k = 0; k < nc; k++) {
    TC d = F[k * m + k], inv, dk, diag;
    if (ldlt) {
      int n1 = 0, p1 = 0;
      const bool ok = small_ldlt_pivot(d, tau, n1, p1);
      if (!ok) {
        if (t == 0) atomicMin(status, status_word(f + k, 2, s));
        return;  // group-uniform: every thread saw the same pivot
      }
      if (t == 0) {
        neg += n1;
        pert += p1;
        la.D[f + k] = (double)(float)d;
      }
      dk = d;
      inv = TC(1) / d;
      diag = TC(1);
    } else {
      if (!(d > TC(0))) {
        if (t == 0) atomicMin(status, status_word(f + k, 1, s));
        return;  // group-uniform
      }
      const TC r = sqrt(d);
      dk = TC(1);
      inv = TC(1) / r;
      diag = r;
    }
    const TC *Fk = F + k * m;
    float *Lk = Lp + (int64_t)k * m;
    for (int i = k + t; i < m; i += G) Lk[i] = (float)(i == k ? diag : Fk[i] * inv);
    const int w = m - k - 1;
    for (int jj = warp; jj < w; jj += NW) {
      const int j = k + 1 + jj;
      const TC lj = (Fk[j] * inv) * dk;
      TC *Fj = F + j * m;
      for (int i = j + lane; i < m; i += 32) Fj[i] -= (Fk[i] * inv) * lj;
    }
    group_sync<G>();
  }
  if (ldlt && t == 0 && (neg | pert)) {
    atomicAdd(la.counts, neg);
    atomicAdd(la.counts + 1, pert);
  }
  if (mu > 0) {
    float *Up = U + P.snUoff[s];
    for (int e = t; e < mu * mu; e += G) {
      const int jj = e / mu, ii = e - jj * mu;
      if (ii >= jj) Up[e] = (float)F[(nc + jj) * m + nc + ii];
    }
  }
}


// m <= MAXM (16 or 32): one warp per front, tiny_warps<MAXM>() fronts per CTA
template <class TC, int MAXM>
__global__ void __launch_bounds__(32 * tiny_warps<MAXM>()) k_front_tiny_f32(const int *__restrict__ fronts, int count,
                                                                         DevPlan P, const double *__restrict__ values,
                                                                         float *__restrict__ Lx, float *__restrict__ U,
                                                                         unsigned long long *status, LdltArgs<float> la) {
  constexpr int W = tiny_warps<MAXM>();
  __shared__ TC F[W][MAXM * MAXM];
  if (warp_failed(status)) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int idx = blockIdx.x * W + warp;
  if (idx >= count) return;  // warp-uniform; no CTA-wide barrier follows
  factor_front<TC, 32>(fronts[idx], P, values, Lx, U, F[warp], status, la, lane, nullptr);
}

// 32 < m <= 128: one CTA per front; dynamic shared memory = the launch's largest m squared
template <class TC>
__global__ void __launch_bounds__(256) k_front_small_f32(const int *__restrict__ fronts, int count, DevPlan P,
                                                     const double *__restrict__ values, float *__restrict__ Lx,
                                                     float *__restrict__ U, unsigned long long *status,
                                                     LdltArgs<float> la) {
  extern __shared__ __align__(16) unsigned char fs_dyn[];
  __shared__ ChildMeta cm;
  if (cta_failed(status)) return;
  factor_front<TC, 256>(fronts[blockIdx.x], P, values, Lx, U, reinterpret_cast<TC *>(fs_dyn), status, la,
                             threadIdx.x, &cm);
}

template <class TC>
int launch_f32(const SmallFronts &fr, const DevPlan &P, const double *values, float *Lx, float *U,
               unsigned long long *status, const LdltArgs<float> &la, cudaStream_t st) {
  int k = 0;
  auto tiny = [&](auto kernel, const int *fronts, int count, int warps) {
    if (count <= 0) return;
    kernel<<<(count + warps - 1) / warps, 32 * warps, 0, st>>>(fronts, count, P, values, Lx, U, status, la);
    k++;
  };
  tiny(k_front_tiny_f32<TC, kTinyMid>, fr.tiny, fr.ntinyMid, tiny_warps<kTinyMid>());
  tiny(k_front_tiny_f32<TC, kTinyFront>, fr.tiny + fr.ntinyMid, fr.ntiny - fr.ntinyMid, tiny_warps<kTinyFront>());
  const int small = fr.half.count + fr.full.count;  // (the two lists are one)
  if (small > 0) {
    const int maxM = fr.full.count > 0 ? fr.full.maxM : fr.half.maxM;
    k_front_small_f32<TC><<<small, 256, (size_t)maxM * maxM * sizeof(TC), st>>>(fr.half.sn, small, P, values, Lx, U,
                                                                                       status, la);
    k++;
  }
  return k;
}

}  // namespace

cudaError_t init_front_small_f32_attributes() {
  cudaError_t e = cudaFuncSetAttribute(k_front_small_f32<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       kSmallFront * kSmallFront * (int)sizeof(float));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_front_small_f32<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kSmallFront * kSmallFront * (int)sizeof(double));
  return e;
}

template <>
int launch_fronts_small<float>(const SmallFronts &fr, const DevPlan &P, const double *values, float *Lx, float *U,
                               unsigned long long *status, const LdltArgs<float> &la, cudaStream_t st) {
  if (la.scal != nullptr)  // LDL^T: FP64 arithmetic whatever the storage
    return launch_f32<double>(fr, P, values, Lx, U, status, la, st);
  return launch_f32<float>(fr, P, values, Lx, U, status, la, st);
}

}  // namespace amp
