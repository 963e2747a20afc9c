// Device bodies of the two assembly kernels, shared by the single-GEP launches (assemble.cu) and the
// batched persistent launch over many GEPs (assemble_batch.cu), so both compute every value with the
// same operations in the same order.
#pragma once
#include <cuda_runtime.h>

#include "gep.h"
#include "shape.cuh"

namespace fem2d {
namespace {

// kind -> (family of the outer Elem at the scaled points, family of the inner Elem)
__device__ __forceinline__ int2 kind_families(int kind) {
  switch (kind) {
    case 0: return make_int2(0, 0);   // N  N
    case 1: return make_int2(3, 3);   // T' T'
    case 2: return make_int2(2, 2);   // T  T
    case 3: return make_int2(0, 3);   // N  T'
    default: return make_int2(3, 0);  // T' N
  }
}

// One (interval, axis, kind) table of 1-D contractions, P x P entries, strided over the block's threads:
//   G[a][b] = sum_m w_m X_a(s x_m + o) Y_b(x_m)            (glq.rs:19-32 restricted to one axis)
// The shape functions are tabulated per chunk of points first (up to kTabP of them; evaluating two of them
// per term, each a recurrence of FP64 operations, took 254 us for KOLeg tables of order 7 and 418 us for
// order 8, against 0.2 and 2.6 ms of the values themselves).
constexpr int kTabP = 24, kTabPts = 16, kTabThreads = 128;
__device__ __forceinline__ void contract1d_table(int basis, int P, int nivl, int iv, int axis, int kind,
                                                 const double* __restrict__ ivl, const double* __restrict__ glq,
                                                 int nq_u, int nq_v, double* __restrict__ tables) {
  __shared__ double tx[kTabPts][kTabP], ty[kTabPts][kTabP];
  const int nq = axis == 0 ? nq_u : nq_v;
  const double* xs = axis == 0 ? glq : glq + 2 * nq_u;
  const double* ws = xs + nq;
  const double s = ivl[2 * iv], o = ivl[2 * iv + 1];
  const int2 fam = kind_families(kind);
  double* out = tables + (((size_t)axis * nivl + iv) * 5 + kind) * P * P;
  if (P > kTabP) {   // uniform
    for (int t = threadIdx.x; t < P * P; t += blockDim.x) {
      const int a = t / P, b = t % P;
      double acc = 0.0;
      for (int m = 0; m < nq; m++) {
        const double x = xs[m];
        acc += ws[m] * shape(basis, fam.x, a, s * x + o) * shape(basis, fam.y, b, x);
      }
      out[t] = acc;
    }
    return;
  }
  constexpr int kOut = (kTabP * kTabP + kTabThreads - 1) / kTabThreads;   // entries per thread (kTabThreads of them)
  double acc[kOut];
#pragma unroll
  for (int i = 0; i < kOut; i++) acc[i] = 0.0;
  for (int m0 = 0; m0 < nq; m0 += kTabPts) {
    const int mc = min(kTabPts, nq - m0);
    if (m0 > 0) __syncthreads();
    for (int t = threadIdx.x; t < 2 * mc * P; t += blockDim.x) {
      const bool second = t >= mc * P;
      const int r = second ? t - mc * P : t, m = r / P, a = r - m * P;
      const double x = xs[m0 + m];
      if (second) ty[m][a] = shape(basis, fam.y, a, x);
      else tx[m][a] = shape(basis, fam.x, a, s * x + o);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kOut; i++) {
      const int t = threadIdx.x + i * kTabThreads;
      if (t >= P * P) break;
      const int a = t / P, b = t % P;
      for (int m = 0; m < mc; m++) acc[i] += ws[m0 + m] * tx[m][a] * ty[m][b];
    }
  }
#pragma unroll
  for (int i = 0; i < kOut; i++) {
    const int t = threadIdx.x + i * kTabThreads;
    if (t < P * P) out[t] = acc[i];
  }
}

// v, with +0 for -0 (in integers: these kernels have no FP64 operation to spare)
__device__ __forceinline__ double positive_zero(double v) {
  const long long bits = __double_as_longlong(v);
  return (bits << 1) == 0 ? 0.0 : v;
}

// The value of one upper-triangle entry of A and B: the sum of its visits k0..k1-1, each the product C * Gu * Gv that
// equals the reference's 2-D Gauss sum (integrals.rs:26-92, 292-354). The FP64 pipe bounds the kernels that
// call this (79% busy): the four direction pairs share one sequence of products, with the tables chosen by
// index, since a warp of mixed pairs would run each branch's products, and the first visit is not added to
// zero (nearly every entry has one visit). A sum that starts from zero is never -0, and the values are written to
// files bit for bit, so a first visit of -0 (a zero table entry times a negative coefficient) is stored as +0.
__device__ __forceinline__ void entry_values(int64_t k0, int64_t k1, const uint64_t* __restrict__ codes,
                                             const GBlock* __restrict__ blocks, const uint32_t* __restrict__ specs,
                                             const double* __restrict__ tables, int P, int nivl, double& out_a,
                                             double& out_b) {
  const int PP = P * P;
  const size_t axis_stride = (size_t)nivl * 5 * PP;
  double sa = 0.0, sb = 0.0;
  for (int64_t k = k0; k < k1; k++) {
    const uint64_t code = __ldg(codes + k);
    const GBlock* bl = blocks + (code >> 32);
    const int2 sp = __ldg(reinterpret_cast<const int2*>(bl));
    const int2 iv = __ldg(reinterpret_cast<const int2*>(bl) + 1);
    const uint32_t p = __ldg(specs + sp.x + (int)((code >> 16) & 0xffff));
    const uint32_t q = __ldg(specs + sp.y + (int)(code & 0xffff));
    const int pi = p & 0xff, pj = (p >> 8) & 0xff, pd = (p >> 16) & 0xff;
    const int qi = q & 0xff, qj = (q >> 8) & 0xff, qd = (q >> 16) & 0xff;
    const double* gu = tables + (size_t)iv.x * 5 * PP + pi * P + qi;
    const double* gv = tables + axis_stride + (size_t)iv.y * 5 * PP + pj * P + qj;
    const int dd = pd * 2 + qd;   // 0 UU, 1 UV, 2 VU, 3 VV
    // curl-curl: UU (NN, DD), UV (ND, DN), VU (DN, ND), VV (DD, NN); mass: UU (NN, TT), VV (TT, NN)
    const int ku = dd == 0 ? G_NN : dd == 1 ? G_ND : dd == 2 ? G_DN : G_DD;
    const int kv = dd == 0 ? G_DD : dd == 1 ? G_DN : dd == 2 ? G_ND : G_NN;
    const double va = __ldg(bl->ca + dd) * __ldg(gu + ku * PP) * __ldg(gv + kv * PP);
    double vb = 0.0;
    if (pd == qd)
      vb = __ldg(bl->cb + pd) * __ldg(gu + (pd ? G_TT : G_NN) * PP) * __ldg(gv + (pd ? G_NN : G_TT) * PP);
    if (k == k0) {
      sa = va;
      sb = vb;
    } else {
      sa += va;
      sb += vb;
    }
  }
  out_a = positive_zero(sa);
  out_b = positive_zero(sb);
}

// the value of an upper entry into the full CSR
__device__ __forceinline__ void store_entry(EntryPos q, double va, double vb, double* __restrict__ A,
                                            double* __restrict__ B) {
  A[q.own] = va;
  B[q.own] = vb;
  if (q.mirror != q.own) {
    A[q.mirror] = va;
    B[q.mirror] = vb;
  }
}

}  // namespace
}  // namespace fem2d
