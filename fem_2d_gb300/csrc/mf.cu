// Numeric multifrontal factorization and block solves on the device (plan: mf.h, mf_symbolic.cpp).
//
// Fronts are dense and column-major, processed level by level. A front that fits one CTA's shared memory is
// assembled there from the CSR values of c_a*A + c_b*B and its children's Schur complements, its first p columns
// are eliminated by a blocked LU with partial pivoting restricted to the fully-summed rows (or without
// pivoting for SPD shifts), and it is written back once with its pivot square inverted (mf_front_kernel).
// Larger fronts stay in global memory: assembly, extend-add of the children one after the other, then eight
// columns per launch, a CTA per 8-column strip (mf_strip_kernel), and the inverses by strips
// (mf_inverse_kernel, mf_partinv_kernel). The trailing (f-p)x(f-p) block left in place is the update matrix
// for the parent.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cstring>
#include <mutex>

namespace cg = cooperative_groups;

#include "dmma.h"
#include "mfdev.h"

namespace fem2d {

namespace {

// the solve workspace holds one row of kLdW values per front row (row-major, one right-hand side per
// column), so a row that a parent gathers from a child is one contiguous read
constexpr int kLdW = 32;

constexpr int MAXKIDS = 4;   // binary dissection nodes; Elem nodes have 2 (U/V) or 4 (T) children

struct FrontDesc {   // device copy of the per-front scalars
  int32_t f, p, parent;
  int32_t kid[MAXKIDS];
  int64_t off, dptr, aptr, aend, eptr;
  int64_t prow;   // tiled fronts: the front's first pull record (one per row)
  int64_t aux;    // fronts factored in global memory: offset of the p x p scratch square of their inverses
};

// the CSR values of the listed fronts to their positions row * f + col: `by_rows` keeps the fronts row-major (one
// dense front, inverted in that layout), otherwise they are column-major like all fronts. (The scaled pencil is
// symmetric up to rounding only, and the solves are to be those of the matrix that the products multiply with.)
__global__ void mf_assemble_kernel(const int32_t* __restrict__ lf, const FrontDesc* __restrict__ fd,
                                   const int64_t* __restrict__ apos, const int64_t* __restrict__ acsr,
                                   const double* __restrict__ va, const double* __restrict__ vb, double ca, double cb,
                                   int by_rows, double* __restrict__ F) {
  const FrontDesc d = fd[lf[blockIdx.y]];
  for (int64_t k = d.aptr + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < d.aend;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = acsr[k], pos = apos[k], row = pos / d.f;
    F[d.off + (by_rows ? pos : (pos - row * d.f) * d.f + row)] = ca * va[c] + cb * vb[c];
  }
}

// add the children's trailing blocks (rows/cols >= p_child) into the parent at mapped positions, in slot
// order; a CTA owns kExtendCols columns of the parent and takes the child columns that map there
constexpr int kExtendCols = 16;
__global__ void __launch_bounds__(256) mf_extend_add_kernel(const int32_t* __restrict__ lf,
                                                            const FrontDesc* __restrict__ fd,
                                                            const int32_t* __restrict__ emap, double* __restrict__ F) {
  const FrontDesc par = fd[lf[blockIdx.y]];
  const int j0 = blockIdx.x * kExtendCols;
  if (j0 >= par.f) return;
  __shared__ int from[kExtendCols], count;   // child column of each parent column (-1: none), any at all
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int slot = 0; slot < MAXKIDS; slot++) {
    const int32_t ch = par.kid[slot];
    if (ch < 0) continue;   // uniform across the CTA
    const FrontDesc c = fd[ch];
    const int s = c.f - c.p;
    const int32_t* m = emap + c.eptr;
    __syncthreads();   // one child after the other: the sums keep their order
    if (threadIdx.x < kExtendCols) from[threadIdx.x] = -1;
    if (threadIdx.x == 0) count = 0;
    __syncthreads();
    for (int j = threadIdx.x; j < s; j += 256) {
      const int to = m[j] - j0;
      if (to >= 0 && to < kExtendCols) {
        from[to] = j;
        count = 1;
      }
    }
    __syncthreads();
    if (count == 0) continue;
    for (int q = warp; q < kExtendCols; q += 8) {
      const int j = from[q];
      if (j < 0) continue;
      const double* src = F + c.off + (int64_t)(c.p + j) * c.f + c.p;
      double* dst = F + par.off + (int64_t)(j0 + q) * par.f;
#pragma unroll 4
      for (int i = lane; i < s; i += 32) dst[m[i]] += src[i];
    }
  }
}

// ------------------------------------------------------------------ fronts in shared memory
// A front of up to kFusedF rows is factored by one CTA in one pass (mf_front_kernel): assembled from the
// CSR values and the children's Schur complements into shared memory, factored there, its inverted
// diagonal blocks (and, where the solves want them, L21' and U12') formed there, and written once. What
// bounds it is the FP64 pipe: updates and inverses run as FP64 MMAs on 8 x 8 tiles, a pivot column costs
// one or two barriers, and pivots are compared as integers (a double comparison takes a slot of the FP64
// pipe). Passing each front through global memory seven times per 32 columns (assembly, extend-adds, panel,
// triangular solve, update, inverse, with 20 to 400 us per panel whatever its size) took 0.59 ms per
// factorization at 832 DoFs, 3.7 at 29k, 7.0 at 83k and 59 at 1M; now 0.24, 2.5, 4.1 and 33.
// Larger fronts, and those above kFusedNarrowF rows of levels that would leave SMs idle, stay in global
// memory and are factored by many CTAs each (mf_strip_kernel): a front of 160 rows keeps one SM's FP64 pipe
// busy for half a millisecond. (Lines at 32 to 128 rows were within 10% of each other at 5k to 83k DoFs;
// at 832 DoFs 32 rows cost a third more.)
constexpr int kFusedF = 164;
constexpr int kFusedNarrowF = 64;   // on levels of at most one front per SM
constexpr int kFusedSmallF = 64;   // fronts up to here: 128 threads
constexpr size_t kFusedStatic = 4096, kSmemPerSM = 227 * 1024;   // static shared memory of a CTA (at most), an SM's

// fronts that the solves may give one CTA (see there)
constexpr int kSmallP = 160;
constexpr int kSmallF = 512;

constexpr int strip_smem(int rows) { return (int)sizeof(double) * 8 * (rows | 1); }

struct FactorArgs {
  const FrontDesc* fd;
  const int64_t *apos, *acsr;
  const double *va, *vb;
  double ca, cb;
  const int32_t *emap, *dofs;
  const int64_t* piv_off;
  double* F;
  int32_t *piv, *perm, *iperm;
  int* flags;
  int32_t* weak;
  int* nweak;
  int weak_cap;
  int pivoting;
};

// A column whose largest fully-summed entry is below kWeakPivot times its largest entry in the rows of
// the front's other (not yet summed) DoFs has no stable pivot here: its DoF is recorded, and the solver
// moves its elimination to the parent front and refactors (delayed pivoting).
constexpr double kWeakPivot = 1e-3;

// |a| as an integer that orders like |a| (0 for NaN)
__device__ __forceinline__ unsigned long long mag_key(double a) {
  const unsigned long long k = (unsigned long long)__double_as_longlong(a) & 0x7FFFFFFFFFFFFFFFull;
  return k > 0x7FF0000000000000ull ? 0ull : k;
}

template <int NT>
struct LuScratch {   // double-buffered by column parity, so that a column costs one barrier
  unsigned long long key[2][NT / 32], other[2][NT / 32];   // per warp: largest candidate, largest other entry
  int row[2][NT / 32];
  double cand[2][NT / 32][8];   // the candidates' rows of the micro-panel
  double top[2][8];             // row k
  double inv[2];
};

// largest key of the warp and, among equal keys, the smallest row
__device__ __forceinline__ unsigned long long warp_max_key(unsigned long long key) {
  const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32));
  const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32) == hi ? (unsigned)key : 0u);
  return ((unsigned long long)hi << 32) | lo;
}

// A micro-panel: w <= 8 pivot columns k0 .. of the nr-row block, carried in registers (thread: the rows
// k0 + tid + NT m) with `nc` >= w columns, so that columns past the pivots are solved and updated with them.
// Rows below pr are pivot candidates; A points at column k0, pv[k] gets the row swapped with row k. Bound by
// its chain per column: a warp reduction, one barrier, a division (some 700 clocks on this FP64 pipe) and
// the row update.
template <int NT, int RPT>
__device__ __forceinline__ void micro_panel(double* A, int ld, int k0, int nr, int nc, int w, int pr,
                                            const FactorArgs& a, const int32_t* col_dof, bool has_parent, int32_t* pv,
                                            LuScratch<NT>& sc) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool pivoting = a.pivoting != 0;
  const bool one_divides = nr - k0 > 128;   // else every warp with rows does, without a second barrier
  double x[RPT][8];
#pragma unroll
  for (int m = 0; m < RPT; m++) {
    const int i = k0 + tid + NT * m;
#pragma unroll
    for (int c = 0; c < 8; c++) x[m][c] = (i < nr && c < nc) ? A[c * ld + i] : 0.0;
  }
#pragma unroll
  for (int jj = 0; jj < 8; jj++) {
    if (jj >= w) break;   // uniform
    const int k = k0 + jj, par = jj & 1;
    if (pivoting) {
      unsigned long long bk = 0, ok = 0;
      int bi = INT32_MAX;
#pragma unroll
      for (int m = 0; m < RPT; m++) {
        const int i = k0 + tid + NT * m;
        if (i < k || i >= nr) continue;
        const unsigned long long q = mag_key(x[m][jj]);
        if (i >= pr) ok = max(ok, q);
        else if (bi == INT32_MAX || q > bk) {
          bk = q;
          bi = i;
        }
      }
      const unsigned long long best = warp_max_key(bk);
      const int row = __reduce_min_sync(0xffffffffu, bk == best ? bi : INT32_MAX);
      ok = warp_max_key(ok);
      if (lane == 0) {
        sc.key[par][warp] = best;
        sc.row[par][warp] = row;
        sc.other[par][warp] = ok;
      }
#pragma unroll
      for (int m = 0; m < RPT; m++)
        if (k0 + tid + NT * m == row) {
#pragma unroll
          for (int c = 0; c < 8; c++) sc.cand[par][warp][c] = x[m][c];
        }
    }
#pragma unroll
    for (int m = 0; m < RPT; m++)
      if (k0 + tid + NT * m == k) {
#pragma unroll
        for (int c = 0; c < 8; c++) sc.top[par][c] = x[m][c];
      }
    __syncthreads();
    int best = k;
    const double* ur = sc.top[par];
    if (pivoting) {
      unsigned long long bk = 0, ok = 0;
      int bw = 0;
      best = INT32_MAX;
#pragma unroll
      for (int q = 0; q < NT / 32; q++) {
        const unsigned long long kq = sc.key[par][q];
        const int rq = sc.row[par][q];
        ok = max(ok, sc.other[par][q]);
        if (kq > bk || (kq == bk && rq < best)) {
          bk = kq;
          best = rq;
          bw = q;
        }
      }
      ur = sc.cand[par][bw];
      if (tid == 0 && has_parent && bk < ok &&   // (the factor is below 1)
          __longlong_as_double((long long)bk) < kWeakPivot * __longlong_as_double((long long)ok)) {
        const int slot = atomicAdd(a.nweak, 1);
        if (slot < a.weak_cap) a.weak[slot] = col_dof[k];
      }
    }
    double u[8];
#pragma unroll
    for (int c = 0; c < 8; c++) u[c] = ur[c];
    const long long ub = __double_as_longlong(u[jj]);
    const unsigned long long uk = mag_key(u[jj]);   // 0: zero or NaN
    if (uk == 0 || (!pivoting && ub < 0)) {
      if (tid == 0) atomicOr(a.flags, pivoting ? 1 : 2);   // 1: zero pivot (perturbed), 2: not positive definite
      if ((ub & 0x7FFFFFFFFFFFFFFFll) == 0) u[jj] = 1e-300;
    }
    if (tid == 0) pv[k] = best;
    double inv = 0.0;
    if (one_divides) {
      if (warp == 0) {
        inv = 1.0 / u[jj];
        if (lane == 0) sc.inv[par] = inv;
      }
      __syncthreads();
      inv = sc.inv[par];
    } else if (k0 + 32 * warp < nr) {
      inv = 1.0 / u[jj];
    }
#pragma unroll
    for (int m = 0; m < RPT; m++) {
      const int i = k0 + tid + NT * m;
      if (i == k) {
#pragma unroll
        for (int c = 0; c < 8; c++) x[m][c] = u[c];
      } else if (i > k && i < nr) {
        if (i == best) {
#pragma unroll
          for (int c = 0; c < 8; c++) x[m][c] = sc.top[par][c];
        }
        const double l = x[m][jj] * inv;
        x[m][jj] = l;
#pragma unroll
        for (int c = jj + 1; c < 8; c++) x[m][c] -= l * u[c];
      }
    }
  }
#pragma unroll
  for (int m = 0; m < RPT; m++) {
    const int i = k0 + tid + NT * m;
#pragma unroll
    for (int c = 0; c < 8; c++)
      if (i < nr && c < nc) A[c * ld + i] = x[m][c];
  }
}

// The same on rows left in memory, any number of them (fronts of more than 2048 rows, which no mesh measured
// here has)
__device__ __forceinline__ void micro_panel_memory(double* A, int64_t ld, int k0, int nr, int nc, int w, int pr,
                                                   const FactorArgs& a, const int32_t* col_dof, bool has_parent,
                                                   int32_t* pv, LuScratch<256>& sc) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool pivoting = a.pivoting != 0;
  for (int jj = 0; jj < w; jj++) {
    const int k = k0 + jj;
    double* ck = A + jj * ld;
    __syncthreads();
    int best = k;
    if (pivoting) {
      unsigned long long bk = 0, ok = 0;
      int bi = INT32_MAX;
      for (int i = k + tid; i < nr; i += 256) {
        const unsigned long long q = mag_key(ck[i]);
        if (i >= pr) ok = max(ok, q);
        else if (bi == INT32_MAX || q > bk) {
          bk = q;
          bi = i;
        }
      }
      const unsigned long long wk = warp_max_key(bk);
      const int row = __reduce_min_sync(0xffffffffu, bk == wk ? bi : INT32_MAX);
      ok = warp_max_key(ok);
      if (lane == 0) {
        sc.key[0][warp] = wk;
        sc.row[0][warp] = row;
        sc.other[0][warp] = ok;
      }
      __syncthreads();
      bk = 0;
      best = INT32_MAX;
      for (int q = 0; q < 8; q++) {
        ok = max(ok, sc.other[0][q]);
        if (sc.key[0][q] > bk || (sc.key[0][q] == bk && sc.row[0][q] < best)) {
          bk = sc.key[0][q];
          best = sc.row[0][q];
        }
      }
      if (tid == 0 && has_parent &&
          __longlong_as_double((long long)bk) < kWeakPivot * __longlong_as_double((long long)ok)) {
        const int slot = atomicAdd(a.nweak, 1);
        if (slot < a.weak_cap) a.weak[slot] = col_dof[k];
      }
      __syncthreads();
    }
    if (tid < nc && best != k) {
      const double x = A[tid * ld + k];
      A[tid * ld + k] = A[tid * ld + best];
      A[tid * ld + best] = x;
    }
    __syncthreads();
    if (tid == 0) {
      pv[k] = best;
      double dk = ck[k];
      if (!(fabs(dk) > 0.0) || (!pivoting && !(dk > 0.0))) {
        atomicOr(a.flags, pivoting ? 1 : 2);
        if (dk == 0.0) ck[k] = dk = 1e-300;
      }
      sc.inv[0] = 1.0 / dk;
    }
    __syncthreads();
    const double inv = sc.inv[0];
    for (int i = k + 1 + tid; i < nr; i += 256) {
      const double l = ck[i] * inv;
      ck[i] = l;
      for (int c = jj + 1; c < nc; c++) A[c * ld + i] -= l * A[c * ld + k];
    }
  }
  __syncthreads();
}

// U12 = L11^-1 A12 for one column c (rows k0 ..) after the micro-panel's row swaps; L11 unit lower, at A
__device__ __forceinline__ void swap_solve8(double* c, const double* A, int64_t ld, int k0, int w, const int32_t* pv,
                                            bool solve) {
  for (int k = k0; k < k0 + w; k++) {
    const int r = pv[k];
    if (r != k) {
      const double x = c[k];
      c[k] = c[r];
      c[r] = x;
    }
  }
  if (!solve) return;
  double x[8];
#pragma unroll
  for (int r = 0; r < 8; r++) x[r] = r < w ? c[k0 + r] : 0.0;
#pragma unroll
  for (int q = 0; q < 7; q++)
#pragma unroll
    for (int r = q + 1; r < 8; r++)
      if (r < w) x[r] -= A[q * ld + k0 + r] * x[q];
#pragma unroll
  for (int r = 0; r < 8; r++)
    if (r < w) c[k0 + r] = x[r];
}

// LU of the first np columns of the f x f column-major block A in shared memory (leading dimension ld)
template <int NT>
__device__ __forceinline__ void lu_shared(double* A, int ld, int f, int np, const FactorArgs& a,
                                          const int32_t* col_dof, bool has_parent, int32_t* pv, LuScratch<NT>& sc) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int k0 = 0; k0 < np; k0 += 8) {
    const int w = min(8, np - k0);
    micro_panel<NT, 1>(A + k0 * ld, ld, k0, f, w, w, np, a, col_dof, has_parent, pv, sc);
    __syncthreads();
    for (int j = tid; j < f; j += NT)
      if (j < k0 || j >= k0 + w) swap_solve8(A + j * ld, A + k0 * ld, ld, k0, w, pv, j > k0);
    __syncthreads();
    // A22 -= L21 U12
    const int b0 = k0 + w, tr = (f - b0 + 7) >> 3;
    const int g = lane >> 2, kl = lane & 3;
    for (int q = warp; q < tr * tr; q += NT / 32) {
      const int rt = q % tr, ct = q / tr;
      const int i = b0 + 8 * rt + g, j = b0 + 8 * ct + g;
      const bool ri = i < f, cj = j < f;
      const double a0 = (ri && kl < w) ? -A[(k0 + kl) * ld + i] : 0.0;
      const double a1 = (ri && 4 + kl < w) ? -A[(k0 + 4 + kl) * ld + i] : 0.0;
      const double u0 = (cj && kl < w) ? A[j * ld + k0 + kl] : 0.0;
      const double u1 = (cj && 4 + kl < w) ? A[j * ld + k0 + 4 + kl] : 0.0;
      const int jc = b0 + 8 * ct + 2 * kl;
      double* o = A + jc * ld + i;
      double c[2] = {(ri && jc < f) ? o[0] : 0.0, (ri && jc + 1 < f) ? o[ld] : 0.0};
      dmma(c, a0, u0);
      if (w > 4) dmma(c, a1, u1);
      if (ri && jc < f) o[0] = c[0];
      if (ri && jc + 1 < f) o[ld] = c[1];
    }
    __syncthreads();
  }
}

// element (r, c) of the unit lower / upper triangular factor in the LU square of order p, 0 outside
__device__ __forceinline__ double lower_at(const double* A, int ld, int p, int r, int c) {
  return (r >= p || c > r) ? 0.0 : (c == r ? 1.0 : A[c * ld + r]);
}
__device__ __forceinline__ double upper_at(const double* A, int ld, int p, int r, int c) {
  return (c >= p || c < r) ? 0.0 : A[c * ld + r];
}

// The LU square of order p (the first p rows and columns of A) overwritten by (unit lower L11^-1, U11^-1):
// the 8 x 8 diagonal blocks by substitution, then block row by block row
//   X_ij = -L_ii^-1 sum_{j <= k < i} L_ik X_kj        (and the same for U, from the last block row up).
// scr: 64 doubles per warp; p <= MAXP.
template <int NT, int MAXP>
__device__ __forceinline__ void invert_square(double* A, int ld, int p, double* scr) {
  constexpr int NW = NT / 32, MAXT = (2 * ((MAXP + 7) / 8 - 1) + NW - 1) / NW;   // tiles per warp and step
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, kl = lane & 3;
  const int nb = (p + 7) >> 3;
  for (int t0 = 0; t0 < 16 * nb; t0 += NT) {   // one column of one diagonal block's inverse per thread
    const int t = t0 + tid, blk = t >> 4, c = t & 7, d0 = 8 * blk, w = min(8, p - d0);
    const bool up = (t & 8) != 0, on = t < 16 * nb && c < w;
    double x[8];
#pragma unroll
    for (int r = 0; r < 8; r++) x[r] = 0.0;
    if (on) {
      if (!up) {
#pragma unroll
        for (int r = 0; r < 8; r++) {
          double s = r == c ? 1.0 : 0.0;
#pragma unroll
          for (int k = 0; k < r; k++)
            if (k >= c && r < w) s -= A[(d0 + k) * ld + d0 + r] * x[k];
          x[r] = r >= c ? s : 0.0;
        }
      } else {
#pragma unroll
        for (int r = 7; r >= 0; r--) {
          if (r > c || r >= w) continue;
          double s = r == c ? 1.0 : 0.0;
#pragma unroll
          for (int k = r + 1; k < 8; k++)
            if (k <= c) s -= A[(d0 + k) * ld + d0 + r] * x[k];
          x[r] = s / A[(d0 + r) * ld + d0 + r];
        }
      }
    }
    __syncthreads();   // a block's columns are read by its own 16 threads only, all in this pass
    if (on) {
#pragma unroll
      for (int r = 0; r < 8; r++)
        if (r < w && (up ? r <= c : r > c)) A[(d0 + c) * ld + d0 + r] = x[r];
    }
  }
  __syncthreads();
  double* ws = scr + 64 * warp;
  for (int st = 1; st < nb; st++) {
    // block row st of L^-1 (tiles j < st) and block row nb - 1 - st of U^-1 (tiles j > nb - 1 - st)
    const int iu = nb - 1 - st;
    double out[MAXT][2];
#pragma unroll
    for (int m = 0; m < MAXT; m++) {
      const int q = warp + m * NW;   // tiles 0 .. st - 1 of L, then st tiles of U
      out[m][0] = out[m][1] = 0.0;
      if (q >= 2 * st) continue;   // uniform per warp
      const bool up = q >= st;
      const int j = up ? iu + 1 + (q - st) : q, i = up ? iu : st;
      double s[2] = {0.0, 0.0};
      if (!up) {
        for (int k = j; k < i; k++)
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int kk = 8 * k + 4 * h + kl;
            const int r = 8 * i + g;
            dmma(s, r < p ? A[kk * ld + r] : 0.0, lower_at(A, ld, p, kk, 8 * j + g));
          }
      } else {
        for (int k = i + 1; k <= j; k++)
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int kk = 8 * k + 4 * h + kl, c = 8 * j + g;
            dmma(s, kk < p ? A[kk * ld + 8 * i + g] : 0.0, kk < p ? upper_at(A, ld, p, kk, c) : 0.0);
          }
      }
      ws[(2 * kl) * 8 + g] = s[0];   // column-major 8 x 8
      ws[(2 * kl + 1) * 8 + g] = s[1];
      __syncwarp();
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int kk = 4 * h + kl;
        const double x = up ? upper_at(A, ld, p, 8 * i + g, 8 * i + kk) : lower_at(A, ld, p, 8 * i + g, 8 * i + kk);
        dmma(out[m], -x, ws[g * 8 + kk]);
      }
      __syncwarp();
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < MAXT; m++) {
      const int q = warp + m * NW;
      if (q >= 2 * st) continue;
      const bool up = q >= st;
      const int j = up ? iu + 1 + (q - st) : q, i = up ? iu : st;
      const int r = 8 * i + g, c = 8 * j + 2 * kl;
      if (r < p && c < p) A[c * ld + r] = out[m][0];
      if (r < p && c + 1 < p) A[(c + 1) * ld + r] = out[m][1];
    }
    __syncthreads();
  }
}

// L21 -> -L21 L11^-1 (8-row strips, tiles left to right: a tile needs the strip's columns from its own on)
// and U12 -> -U11^-1 U12 (8-column strips, tiles downwards), in place, one warp per strip
template <int NT>
__device__ __forceinline__ void partinv_shared(double* A, int ld, int f, int p) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, kl = lane & 3;
  const int nb = (p + 7) >> 3, ns = (f - p + 7) >> 3;
  for (int q = warp; q < 2 * ns; q += NT / 32) {
    const bool up = q >= ns;
    const int s0 = p + 8 * (up ? q - ns : q);
    for (int t = 0; t < nb; t++) {
      double s[2] = {0.0, 0.0};
      for (int k = t; k < nb; k++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int kk = 8 * k + 4 * h + kl;
          if (!up) {
            const double b = (kk < p && s0 + g < f) ? A[kk * ld + s0 + g] : 0.0;
            dmma(s, b, lower_at(A, ld, p, kk, 8 * t + g));
          } else {
            const double b = (kk < p && s0 + g < f) ? A[(s0 + g) * ld + kk] : 0.0;
            dmma(s, 8 * t + g < p ? upper_at(A, ld, p, 8 * t + g, kk) : 0.0, b);
          }
        }
      __syncwarp();
      if (!up) {
        const int r = s0 + g, c = 8 * t + 2 * kl;
        if (r < f && c < p) A[c * ld + r] = -s[0];
        if (r < f && c + 1 < p) A[(c + 1) * ld + r] = -s[1];
      } else {
        const int r = 8 * t + g, c = s0 + 2 * kl;
        if (r < p && c < f) A[c * ld + r] = -s[0];
        if (r < p && c + 1 < f) A[(c + 1) * ld + r] = -s[1];
      }
      __syncwarp();
    }
  }
}

__host__ __device__ constexpr size_t fused_smem(int f, int nt) {
  return sizeof(double) * ((size_t)f * (f | 1) + 2 * nt);
}

// one front (f <= MAXF) per CTA: see above. partinv: the solves use L21' and U12' too.
template <int NT, int MAXF>
__global__ void __launch_bounds__(NT, 768 / NT) mf_front_kernel(const int32_t* __restrict__ lf, FactorArgs a, int partinv) {
  extern __shared__ double A[];
  __shared__ int32_t pv[kFusedF], pm[kFusedF];
  __shared__ LuScratch<NT> sc;
  const int fr = lf[blockIdx.x], tid = threadIdx.x;
  const FrontDesc d = a.fd[fr];
  const int f = d.f, p = d.p, ld = f | 1;
  double* scr = A + f * ld;
  for (int t = tid; t < f * ld; t += NT) A[t] = 0.0;
  __syncthreads();
#pragma unroll 4
  for (int64_t k = d.aptr + tid; k < d.aend; k += NT) {
    const int pos = (int)__ldg(a.apos + k), i = pos / f;   // row i, column pos - i f
    const int64_t c = __ldg(a.acsr + k);
    A[(pos - i * f) * ld + i] = a.ca * __ldg(a.va + c) + a.cb * __ldg(a.vb + c);
  }
  for (int slot = 0; slot < MAXKIDS; slot++) {
    const int ch = d.kid[slot];
    if (ch < 0) continue;   // uniform across the CTA
    const FrontDesc cd = a.fd[ch];
    const int s = cd.f - cd.p;
    const int32_t* m = a.emap + cd.eptr;
    const double* C = a.F + cd.off + (int64_t)cd.p * cd.f + cd.p;
    __syncthreads();
    for (int t0 = tid; t0 < s * s; t0 += 4 * NT) {   // four entries (distinct targets) in flight per thread
      double v[4];
      int to[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int t = t0 + q * NT, j = t / s, i = t - j * s;
        to[q] = t < s * s ? __ldg(m + j) * ld + __ldg(m + i) : -1;
        v[q] = t < s * s ? C[(int64_t)j * cd.f + i] : 0.0;
      }
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (to[q] >= 0) A[to[q]] += v[q];
    }
  }
  __syncthreads();
  lu_shared<NT>(A, ld, f, p, a, a.dofs + d.dptr, d.parent >= 0, pv, sc);
  if (tid == 0) {   // the row swaps as a gather permutation
    for (int i = 0; i < p; i++) pm[i] = i;
    for (int k = 0; k < p; k++) {
      const int r = pv[k], x = pm[k];
      pm[k] = pm[r];
      pm[r] = x;
    }
  }
  __syncthreads();
  invert_square<NT, MAXF>(A, ld, p, scr);
  if (partinv) partinv_shared<NT>(A, ld, f, p);
  __syncthreads();
  double* out = a.F + d.off;
  for (int t = tid; t < f * f; t += NT) {
    const int j = t / f;
    out[t] = A[j * ld + (t - j * f)];
  }
  const int64_t po = a.piv_off[fr];
  for (int i = tid; i < p; i += NT) {
    a.piv[po + i] = pv[i];
    a.perm[po + i] = pm[i];
    a.iperm[po + pm[i]] = i;
  }
}

// Fronts factored in global memory advance eight columns per launch, one CTA per 8-column strip (blockIdx.x)
// and front (blockIdx.y): step s applies the micro-panel 8 (s - 1) to the strip -- its row swaps, U12, and the
// update of the rows below -- and the CTA of strip s then factors that strip, the next micro-panel, while the
// other strips are still being updated. A strip of f rows costs a few microseconds, so a narrow level of
// large fronts is spread over the chip instead of being bound by one SM's FP64 rate per front; 32-column
// panels by one CTA, whose own update is nearly all of it on one SM's FP64 pipe, took 85 to 170 us each at 1M DoFs,
// a strip step 20 to 80.
// RPT: rows of the strip per thread in the micro-panel; 0: the front has more rows than fit, the strip stays
// in global memory.
template <int NT, int RPT>
__global__ void __launch_bounds__(NT) mf_strip_kernel(const int32_t* __restrict__ lf, FactorArgs a, int s) {
  extern __shared__ double S[];
  __shared__ int32_t pv[16];
  __shared__ LuScratch<NT> sc;
  const int fr = lf[blockIdx.y], tid = threadIdx.x;
  const FrontDesc d = a.fd[fr];
  const int f = d.f, p = d.p, q = blockIdx.x, kp = 8 * (s - 1), j0 = 8 * q;
  if (j0 >= f || kp >= p || (s > 0 ? q == s - 1 : q != 0)) return;
  double* G = a.F + d.off;
  const int nc = min(8, f - j0);
  const int w = s > 0 ? min(8, p - kp) : 0;
  const int rb = s > 0 ? kp : 0, nr = f - rb, ld = RPT > 0 ? (nr | 1) : f;   // rows from rb on
  double* C = RPT > 0 ? S : G + (int64_t)j0 * f + rb;
  int32_t* piv = a.piv + a.piv_off[fr];
  if (tid < w) pv[tid] = piv[kp + tid] - rb;
  if (s > 0 && q < s - 1) {   // left of the micro-panel: row swaps only
    __syncthreads();
    if (tid < nc) swap_solve8(G + (int64_t)(j0 + tid) * f + rb, nullptr, 0, 0, w, pv, false);
    return;
  }
  if (RPT > 0) {
    for (int t = tid; t < nr * nc; t += NT) {
      const int c = t / nr, i = t - c * nr;
      S[c * ld + i] = G[(int64_t)(j0 + c) * f + rb + i];
    }
  }
  __syncthreads();
  if (s > 0) {
    const double* P = G + (int64_t)kp * f + rb;   // the micro-panel's columns, rows from rb on
    if (tid < nc) swap_solve8(C + (int64_t)tid * ld, P, f, 0, w, pv, true);
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, kl = lane & 3;
    const double u0 = (g < nc && kl < w) ? C[(int64_t)g * ld + kl] : 0.0;
    const double u1 = (g < nc && 4 + kl < w) ? C[(int64_t)g * ld + 4 + kl] : 0.0;
    for (int i0 = w + 8 * warp; i0 < nr; i0 += NT / 4) {
      const int i = i0 + g;
      const bool ri = i < nr;
      const double a0 = (ri && kl < w) ? -P[(int64_t)kl * f + i] : 0.0;
      const double a1 = (ri && 4 + kl < w) ? -P[(int64_t)(4 + kl) * f + i] : 0.0;
      double* o = C + (int64_t)(2 * kl) * ld + i;
      double c[2] = {(ri && 2 * kl < nc) ? o[0] : 0.0, (ri && 2 * kl + 1 < nc) ? o[ld] : 0.0};
      dmma(c, a0, u0);
      dmma(c, a1, u1);
      if (ri && 2 * kl < nc) o[0] = c[0];
      if (ri && 2 * kl + 1 < nc) o[ld] = c[1];
    }
    __syncthreads();
  }
  if (q == s && j0 < p) {   // the next micro-panel (its columns past the pivots are solved with it)
    const int k0 = j0 - rb, wn = min(8, p - j0);
    if constexpr (RPT > 0)
      micro_panel<NT, RPT>(C, ld, k0, nr, nc, wn, p - rb, a, a.dofs + d.dptr + rb, d.parent >= 0, pv, sc);
    else
      micro_panel_memory(C, ld, k0, nr, nc, wn, p - rb, a, a.dofs + d.dptr + rb, d.parent >= 0, pv, sc);
    __syncthreads();
    if (tid < wn) piv[j0 + tid] = pv[k0 + tid] + rb;
  }
  if (RPT > 0) {
    for (int t = tid; t < nr * nc; t += NT) {
      const int c = t / nr, i = t - c * nr;
      G[(int64_t)(j0 + c) * f + rb + i] = S[c * ld + i];
    }
  }
}

// ------------------------------------------------------------------ cluster block solves
// One 8-CTA thread-block cluster per front. Rows are owned in interleaved 32-row chunks
// (chunk q belongs to CTA q % 8). The triangular factors are walked in 32-column blocks: every CTA
// solves the 32 x nb diagonal block itself (from the rows finalised before the last cluster barrier),
// then updates the rows it owns; cluster.sync() separates the blocks. The solved block is written
// back after the barrier, when no CTA reads those rows any more.
constexpr int CL = 8;

// sequential LAPACK-style row swaps -> gather permutation (v'[i] = v[perm[i]])
__global__ void mf_perm_kernel(int nl, const int32_t* __restrict__ lf, const FrontDesc* __restrict__ fd,
                               const int32_t* __restrict__ piv, const int64_t* __restrict__ piv_off, int32_t* __restrict__ perm,
                               int32_t* __restrict__ iperm) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nl) return;
  const int fr = lf[q];
  const int p = fd[fr].p;
  const int32_t* pv = piv + piv_off[fr];
  int32_t* pm = perm + piv_off[fr];
  for (int i = 0; i < p; i++) pm[i] = i;
  for (int k = 0; k < p; k++) {
    const int r = pv[k];
    const int32_t t = pm[k];
    pm[k] = pm[r];
    pm[r] = t;
  }
  int32_t* ip = iperm + piv_off[fr];
  for (int i = 0; i < p; i++) ip[pm[i]] = i;
}

__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(256)
    mf_forward_cluster_kernel(const int32_t* __restrict__ lf, const FrontDesc* __restrict__ fd,
                              const int32_t* __restrict__ dofs, const int32_t* __restrict__ emap,
                              const int32_t* __restrict__ perm, const int32_t* __restrict__ iperm,
                              const int64_t* __restrict__ piv_off,
                              const int64_t* __restrict__ woff, const double* __restrict__ F,
                              const double* __restrict__ B, int64_t ldb, int nb, double* __restrict__ W) {
  cg::cluster_group cluster = cg::this_cluster();
  const int r = (int)cluster.block_rank();
  const int fr = lf[blockIdx.x / CL];
  const FrontDesc d = fd[fr];
  const int f = d.f, p = d.p;
  double* v = W + woff[fr];
  const int32_t* D = dofs + d.dptr;
  const int32_t* pm = perm + piv_off[fr];
  const int32_t* ipm = iperm + piv_off[fr];
  const int nchunk = (f + 31) / 32;
  for (int q = r; q < nchunk; q += CL)
    for (int t = threadIdx.x; t < 32 * nb; t += blockDim.x) {
      const int i = q * 32 + (t & 31), c = t >> 5;
      if (i < f) v[(int64_t)i * kLdW + c] = i < p ? B[(int64_t)D[pm[i]] * ldb + c] : 0.0;
    }
  __syncthreads();
  for (int slot = 0; slot < MAXKIDS; slot++) {
    const int ch = d.kid[slot];
    if (ch < 0) continue;
    const FrontDesc cd = fd[ch];
    const int s = cd.f - cd.p;
    const double* cw = W + woff[ch];
    const int32_t* m = emap + cd.eptr;
    for (int t = threadIdx.x; t < s * nb; t += blockDim.x) {
      const int i = t % s, c = t / s;
      const int row = m[i] < p ? ipm[m[i]] : m[i];   // pivot rows are stored permuted
      if (((row >> 5) % CL) == r) v[(int64_t)row * kLdW + c] += cw[(int64_t)(cd.p + i) * kLdW + c];
    }
    __syncthreads();
  }
  cluster.sync();
  __shared__ double ys[32][33];
  __shared__ double Ld[32][33];
  for (int jb = 0; jb < p; jb += 32) {
    const int bw = min(32, p - jb);
    for (int t = threadIdx.x; t < 32 * nb; t += blockDim.x) {
      const int u = t & 31, c = t >> 5;
      ys[u][c] = u < bw ? v[(int64_t)(jb + u) * kLdW + c] : 0.0;
    }
    for (int t = threadIdx.x; t < 32 * 32; t += blockDim.x) {
      const int u = t & 31, k = t >> 5;   // row jb+u, col jb+k
      Ld[u][k] = (u < bw && k < bw) ? F[d.off + (int64_t)(jb + k) * f + jb + u] : 0.0;
    }
    __syncthreads();
    if (threadIdx.x < nb) {
      const int c = threadIdx.x;
      for (int u = 0; u < bw; u++) {
        double s = ys[u][c];
        for (int k = 0; k < u; k++) s -= Ld[u][k] * ys[k][c];
        ys[u][c] = s;
      }
    }
    __syncthreads();
    // update owned rows below the block
    const int first = jb + bw;
    for (int q = r; q < nchunk; q += CL) {
      if (q * 32 + 31 < first) continue;
      for (int t = threadIdx.x; t < 32 * nb; t += blockDim.x) {
        const int i = q * 32 + (t & 31), c = t >> 5;
        if (i < first || i >= f) continue;
        double acc = 0.0;
        for (int u = 0; u < bw; u++) acc += F[d.off + (int64_t)(jb + u) * f + i] * ys[u][c];
        v[(int64_t)i * kLdW + c] -= acc;
      }
    }
    cluster.sync();
    // the owner stores the solved block (rows jb.. are read by nobody after the barrier)
    if (((jb >> 5) % CL) == r)
      for (int t = threadIdx.x; t < 32 * nb; t += blockDim.x) {
        const int u = t & 31, c = t >> 5;
        if (u < bw) v[(int64_t)(jb + u) * kLdW + c] = ys[u][c];
      }
    __syncthreads();
  }
}

__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(256)
    mf_backward_cluster_kernel(const int32_t* __restrict__ lf, const FrontDesc* __restrict__ fd,
                               const int32_t* __restrict__ dofs, const int64_t* __restrict__ woff,
                               const double* __restrict__ F, double* __restrict__ W, int nb, double* __restrict__ X,
                               int64_t ldx) {
  cg::cluster_group cluster = cg::this_cluster();
  const int r = (int)cluster.block_rank();
  const int fr = lf[blockIdx.x / CL];
  const FrontDesc d = fd[fr];
  const int f = d.f, p = d.p;
  if (p == 0) return;   // uniform across the cluster
  double* v = W + woff[fr];
  const int32_t* D = dofs + d.dptr;
  const int nchunk = (p + 31) / 32;
  // y -= U12 x_struct on owned rows
  for (int q = r; q < nchunk; q += CL)
    for (int t = threadIdx.x; t < 32 * nb; t += blockDim.x) {
      const int i = q * 32 + (t & 31), c = t >> 5;
      if (i >= p) continue;
      double s = v[(int64_t)i * kLdW + c];
      for (int j = p; j < f; j++) s -= F[d.off + (int64_t)j * f + i] * X[(int64_t)D[j] * ldx + c];
      v[(int64_t)i * kLdW + c] = s;
    }
  cluster.sync();
  __shared__ double xs[32][33];
  __shared__ double Ud[32][33];
  const int last = ((p - 1) / 32) * 32;
  for (int jb = last; jb >= 0; jb -= 32) {
    const int bw = min(32, p - jb);
    for (int t = threadIdx.x; t < 32 * nb; t += blockDim.x) {
      const int u = t & 31, c = t >> 5;
      xs[u][c] = u < bw ? v[(int64_t)(jb + u) * kLdW + c] : 0.0;
    }
    for (int t = threadIdx.x; t < 32 * 32; t += blockDim.x) {
      const int u = t & 31, k = t >> 5;
      Ud[u][k] = (u < bw && k < bw) ? F[d.off + (int64_t)(jb + k) * f + jb + u] : 0.0;
    }
    __syncthreads();
    if (threadIdx.x < nb) {
      const int c = threadIdx.x;
      for (int u = bw - 1; u >= 0; u--) {
        double s = xs[u][c];
        for (int k = u + 1; k < bw; k++) s -= Ud[u][k] * xs[k][c];
        xs[u][c] = s / Ud[u][u];
      }
    }
    __syncthreads();
    for (int q = r; q * 32 < jb; q += CL)
      for (int t = threadIdx.x; t < 32 * nb; t += blockDim.x) {
        const int i = q * 32 + (t & 31), c = t >> 5;
        if (i >= jb) continue;
        double acc = 0.0;
        for (int u = 0; u < bw; u++) acc += F[d.off + (int64_t)(jb + u) * f + i] * xs[u][c];
        v[(int64_t)i * kLdW + c] -= acc;
      }
    if (((jb >> 5) % CL) == r)
      for (int t = threadIdx.x; t < 32 * nb; t += blockDim.x) {
        const int u = t & 31, c = t >> 5;
        if (u < bw) X[(int64_t)D[jb + u] * ldx + c] = xs[u][c];
      }
    cluster.sync();
  }
}


// ------------------------------------------------------------------ small-front solves
// Fronts with p <= kSmallP and f <= kSmallF (every front of an Elem-level elimination tree at the
// orders this library meets in practice) are solved by one CTA each, with no sequential triangular
// substitution: the factorization leaves (unit lower L11^-1, upper U11^-1) in each such front's p x p
// diagonal square (invert_square, or mf_inverse_kernel), so both solve directions become dense,
// fully parallel products:
//   forward:  y = L11^-1 P b_p,  b_s -= L21 y          (b_s goes to the parent)
//   backward: x_p = U11^-1 (y - U12 x_s)

// One 8-column strip of L11^-1 (kind 0) or U11^-1 (kind 1) of a front factored in global memory, per CTA:
//   X_i = -L_ii^-1 sum_{j <= k < i} L_ik X_k   down from the strip's diagonal block (up from it for U),
// the strip in shared memory, the sums over k split over the four warps. Results go to the scratch square
// (FrontDesc::aux), since the other strips of the front still read the factors.
__global__ void __launch_bounds__(128) mf_inverse_kernel(const int4* __restrict__ items,
                                                         const FrontDesc* __restrict__ fd,
                                                         const double* __restrict__ F, double* __restrict__ sq) {
  extern __shared__ double X[];   // X[n * ldx + row]: column n of the strip
  __shared__ double part[4][64];
  const int4 it = items[blockIdx.x];
  const FrontDesc d = fd[it.x];
  const int p = d.p, f = d.f, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, kl = lane & 3;
  const bool up = it.y != 0;
  const int j = it.z, nb = (p + 7) >> 3, ldx = (8 * nb) | 4;
  const double* A = F + d.off;
  auto at = [&](int r, int c) -> double {   // the triangular factor
    if (r >= p || c >= p) return 0.0;
    if (r == c) return up ? A[(int64_t)c * f + r] : 1.0;
    return (up ? r < c : r > c) ? A[(int64_t)c * f + r] : 0.0;
  };
  for (int t = tid; t < 8 * ldx; t += 128) X[t] = 0.0;
  // the inverses of the diagonal blocks that the strip passes, one column per thread
  const int steps = up ? j + 1 : nb - j, i_lo = up ? 0 : j;
  double* dg = X + 8 * ldx;   // 64 per block, column-major
  for (int t = tid; t < 8 * steps; t += 128) {
    const int c = t & 7, d0 = 8 * (i_lo + (t >> 3));
    double x[8];
#pragma unroll
    for (int r = 0; r < 8; r++) x[r] = 0.0;
    if (d0 + c < p) {
      if (!up) {
#pragma unroll
        for (int r = 0; r < 8; r++) {
          double s = r == c ? 1.0 : 0.0;
#pragma unroll
          for (int k = 0; k < r; k++) s -= at(d0 + r, d0 + k) * x[k];
          x[r] = r >= c ? s : 0.0;
        }
      } else {
#pragma unroll
        for (int r = 7; r >= 0; r--) {
          if (r > c) continue;
          double s = r == c ? 1.0 : 0.0;
#pragma unroll
          for (int k = r + 1; k < 8; k++) s -= at(d0 + r, d0 + k) * x[k];
          x[r] = s / A[(int64_t)(d0 + r) * f + d0 + r];
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 8; r++) dg[8 * t + r] = x[r];
  }
  __syncthreads();
  for (int st = 0; st < steps; st++) {
    const int i = up ? j - st : j + st;
    // S = sum over the block columns between i and j, the strip's rows known so far
    double s[2] = {0.0, 0.0};
    const int klo = up ? i + 1 : j, khi = up ? j + 1 : i;
    for (int k = klo + warp; k < khi; k += 4)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int kk = 8 * k + 4 * h + kl;
        const int r = 8 * i + g;
        dmma(s, (r < p && kk < p) ? A[(int64_t)kk * f + r] : 0.0, X[g * ldx + kk]);
      }
    part[warp][(2 * kl) * 8 + g] = s[0];
    part[warp][(2 * kl + 1) * 8 + g] = s[1];
    __syncthreads();
    if (warp == 0) {
      double o[2] = {0.0, 0.0};
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int kk = 4 * h + kl, e = g * 8 + kk;   // S[kk][g]
        const double sv = i == j ? (kk == g ? -1.0 : 0.0) : (part[0][e] + part[1][e]) + (part[2][e] + part[3][e]);
        dmma(o, -dg[64 * (i - i_lo) + kk * 8 + g], sv);
      }
      X[(2 * kl) * ldx + 8 * i + g] = o[0];
      X[(2 * kl + 1) * ldx + 8 * i + g] = o[1];
    }
    __syncthreads();
  }
  double* out = sq + d.aux;
  const int r_lo = up ? 0 : 8 * j, r_hi = up ? min(p, 8 * j + 8) : p;
  for (int t = tid; t < 8 * (r_hi - r_lo); t += 128) {
    const int n = t / (r_hi - r_lo), r = r_lo + t - n * (r_hi - r_lo), c = 8 * j + n;
    if (c < p && (up ? r <= c : r > c)) out[(int64_t)c * p + r] = X[n * ldx + r];
  }
}

// the scratch squares back into their fronts
__global__ void mf_square_copy_kernel(const int32_t* __restrict__ lf, const FrontDesc* __restrict__ fd,
                                      const double* __restrict__ S, double* __restrict__ F) {
  const FrontDesc d = fd[lf[blockIdx.y]];
  const int64_t pp = (int64_t)d.p * d.p;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < pp; t += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(t % d.p), k = (int)(t / d.p);
    F[d.off + (int64_t)k * d.f + i] = S[d.aux + t];
  }
}

// One 8-row strip of L21' = -L21 L11^-1 (kind 0) or 8-column strip of U12' = -U11^-1 U12 (kind 1) of a front
// factored in global memory, per CTA: the strip in shared memory, its 8 x 8 tiles dealt to four warps; items
// are (front, kind, first row / column past the pivots).
__global__ void __launch_bounds__(128) mf_partinv_kernel(const int4* __restrict__ items,
                                                         const FrontDesc* __restrict__ fd, double* __restrict__ F) {
  extern __shared__ double X[];   // X[n * ldx + k]: pivot row / column k of the strip's n-th column / row
  const int4 it = items[blockIdx.x];
  const FrontDesc d = fd[it.x];
  const int p = d.p, f = d.f, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, kl = lane & 3;
  const bool up = it.y != 0;
  const int s0 = p + it.z, nb = (p + 7) >> 3, ldx = (8 * nb) | 4;
  double* A = F + d.off;
  for (int t = tid; t < 8 * ldx; t += 128) X[t] = 0.0;
  __syncthreads();
  for (int t = tid; t < 8 * p; t += 128) {
    const int n = up ? t / p : t & 7, k = up ? t - n * p : t >> 3;
    if (s0 + n < f) X[n * ldx + k] = up ? A[(int64_t)(s0 + n) * f + k] : A[(int64_t)k * f + s0 + n];
  }
  __syncthreads();
  for (int q = warp; q < nb; q += 4) {
    double s[2] = {0.0, 0.0};
    for (int k = q; k < nb; k++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int kk = 8 * k + 4 * h + kl, e = 8 * q + g;
        if (!up) {
          const double l = (kk >= p || e > kk) ? 0.0 : (e == kk ? 1.0 : A[(int64_t)e * f + kk]);   // L11^-1(kk, e)
          dmma(s, X[g * ldx + kk], l);
        } else {
          const double u = (kk >= p || kk < e) ? 0.0 : A[(int64_t)kk * f + e];   // U11^-1(e, kk)
          dmma(s, u, X[g * ldx + kk]);
        }
      }
    if (!up) {
      const int r = s0 + g, c = 8 * q + 2 * kl;
      if (r < f && c < p) A[(int64_t)c * f + r] = -s[0];
      if (r < f && c + 1 < p) A[(int64_t)(c + 1) * f + r] = -s[1];
    } else {
      const int r = 8 * q + g, c = s0 + 2 * kl;
      if (r < p && c < f) A[(int64_t)c * f + r] = -s[0];
      if (r < p && c + 1 < f) A[(int64_t)(c + 1) * f + r] = -s[1];
    }
  }
}

constexpr size_t inverse_smem(int p) { return sizeof(double) * 8 * (size_t)((((p + 7) / 8 * 8) | 4) + (p + 7) / 8 * 8); }

// sum_{k = 0}^{n - 1} A[k * f] * v[k]; the FP64 pipe issues one warp instruction in some 19 clocks per SM, so
// two accumulators hide its latency and cost one addition per row (four cost three)
__device__ __forceinline__ double col_dot(const double* __restrict__ A, int f, const double* __restrict__ v, int n) {
  double a0 = 0.0, a1 = 0.0;
  int k = 0;
#pragma unroll 4
  for (; k + 2 <= n; k += 2) {
    a0 += A[(int64_t)k * f] * v[k];
    a1 += A[(int64_t)(k + 1) * f] * v[k + 1];
  }
  if (k < n) a0 += A[(int64_t)k * f] * v[k];
  return a0 + a1;
}

// Two rows of a triangle as one loop of n steps: r1 = the first n1 products, r2 = the others. Step j takes
// A[o1 + j s1] v[x1 + j e1] before n1 and A[o2 + j s2] v[x2 + j e2] from n1 on. The rows q and p - 1 - q have
// the same number of products together for every q, so the lanes of a warp stay together although n1 differs:
// with one loop per row a warp issued as many FP64 instructions as its longest rows have products, and
// a fifth of the lanes in them were idle.
__device__ __forceinline__ void pair_dot(const double* __restrict__ A, const double* __restrict__ v, int n, int n1, int o1,
                                         int s1, int x1, int e1, int o2, int s2, int x2, int e2, double& r1,
                                         double& r2) {
  double acc = 0.0;
  r1 = 0.0;
#pragma unroll 4
  for (int j = 0; j < n; j++) {
    r1 = j == n1 ? acc : r1;
    acc = j == n1 ? 0.0 : acc;
    const int o = j < n1 ? o1 : o2, x = j < n1 ? x1 : x2;
    acc += A[o] * v[x];
    o1 += s1, o2 += s2, x1 += e1, x2 += e2;
  }
  r2 = n1 < n ? acc : 0.0;
  r1 = n1 < n ? r1 : acc;
}

// One factorization of the plan and what a solve with it writes. A launch serves one or two of them: the solves of
// one right-hand side with both shifted matrices go level by level together.
struct SolveSet {
  const int32_t *perm, *iperm;
  const double* F;
  double* W;
  double* X;
  int64_t ldx;
};

struct SolveArgs {
  const FrontDesc* fd;
  const int32_t *dofs, *emap;
  const int64_t *piv_off, *woff;
  const double* B;
  int64_t ldb;
  SolveSet set[2];
  int nb;
  int per;          // right-hand sides per CTA
  int sets, parts;  // CTAs per front, one after another: a set (the low bit, when there are two) and a column range
};

// One CTA solves a front for `per` right-hand sides. The kernels are bound by the FP64 pipe (under two
// FMA per clock and SM) where a level fills the chip, and by what is left idle around it elsewhere:
//   - global rows (B, X, the workspace) are read and written with the right-hand sides along the lanes, so
//     a row is one contiguous access; the dot products take the rows along the lanes and read the factor
//     contiguously. Shared columns have odd length, so both orders are free of bank conflicts.
//   - a level's largest fronts go first, and one with few fronts per SM splits the right-hand sides over
//     CTAs: the SMs then
//     finish together, and one CTA's gathers overlap another's dot products.
// At 83k DoFs (1,179 leaf fronts, 24 right-hand sides) the leaf level took 348 / 315 us forward / backward
// with column-major rows and one CTA per front; a whole solve went from 0.99 to 0.70 ms there, from 0.48 to
// 0.31 ms at 29k DoFs and from 5.95 to 4.93 ms at 1M (13 right-hand sides on average), upper levels included.
// With both shifted matrices in one launch it took 542 / 557 us at 95% of the FP64 issue rate; the paired
// triangle rows, two accumulators for four and the order by size brought it to 391 / 393 us (1M: a whole
// solve from 10.8 to 9.5 ms), at 92% of that rate while it runs: what is left is the products themselves.

// the front's gathered right-hand side v[c * ld + i] (pivot rows permuted): the pivot rows' entries of
// B, then each child's update vector added in slot order (rows are distinct within one child, so no
// atomics are needed, and the fixed order makes the sums, and the whole solve, reproducible bit for bit)
__device__ __forceinline__ void gather_front_rhs(const FrontDesc& d, const FrontDesc* __restrict__ fd,
                                                 const int32_t* __restrict__ emap, const int32_t* __restrict__ ipm,
                                                 const double* __restrict__ W, const int64_t* __restrict__ woff,
                                                 const double* __restrict__ B, int64_t ldb,
                                                 const int32_t* __restrict__ D, const int32_t* __restrict__ pm, int c0,
                                                 int w, int ld, double* v) {
  const int f = d.f, p = d.p;
  for (int t = threadIdx.x; t < f * w; t += blockDim.x) {
    const int i = t / w, c = t - i * w;
    v[c * ld + i] = i < p ? B[(int64_t)D[pm[i]] * ldb + c0 + c] : 0.0;
  }
  for (int slot = 0; slot < MAXKIDS; slot++) {
    const int ch = d.kid[slot];
    if (ch < 0) continue;   // uniform across the CTA
    const FrontDesc cd = fd[ch];
    const int sz = cd.f - cd.p;
    const double* cw = W + woff[ch] + (int64_t)cd.p * kLdW + c0;
    const int32_t* m = emap + cd.eptr;
    __syncthreads();
    for (int t = threadIdx.x; t < sz * w; t += blockDim.x) {
      const int i = t / w, c = t - i * w;
      const int mi = m[i];
      const int row = mi < p ? ipm[mi] : mi;   // pivot rows are stored permuted
      v[c * ld + row] += cw[(int64_t)i * kLdW + c];
    }
  }
  __syncthreads();
}

// shared memory of the two kernels in doubles per right-hand side
__host__ __device__ constexpr int forward_cols(int f, int p) { return (f | 1) + (p | 1); }
__host__ __device__ constexpr int backward_cols(int f, int p) { return (p | 1) + ((f - p > p ? f - p : p) | 1); }

// NT threads per front: 256 for wide levels, up to 1024 for narrow ones, where a few fronts occupy the
// GPU and each front's dependent dot products set the level's latency
template <int NT>
__global__ void __launch_bounds__(NT) mf_forward_small_kernel(const int32_t* __restrict__ lf, SolveArgs a) {
  extern __shared__ double sm[];
  const int fr = lf[blockIdx.x / a.parts], part = blockIdx.x % a.parts;
  const SolveSet set = a.set[part & (a.sets - 1)];
  const int c0 = part / a.sets * a.per, w = min(a.per, a.nb - c0);
  const FrontDesc d = a.fd[fr];
  const int f = d.f, p = d.p, lv = f | 1, ly = p | 1;
  double* v = sm;            // v[c * lv + i]
  double* y = sm + lv * w;   // y[c * ly + i]
  const double* A = set.F + d.off;
  gather_front_rhs(d, a.fd, a.emap, set.iperm + a.piv_off[fr], set.W, a.woff, a.B, a.ldb, a.dofs + d.dptr,
                   set.perm + a.piv_off[fr], c0, w, lv, v);
  // the unit lower triangle: row i is a dot product of length i, so a thread takes the rows p - 1 - q and q
  // (p - 1 products together), the first by rising and the second by falling columns: a warp then reads one
  // or two columns in a step
  const int hp = (p + 1) >> 1;
  for (int t = threadIdx.x; t < hp * w; t += blockDim.x) {
    const int c = t / hp, q = t - c * hp, i2 = p - 1 - q;
    const double* vc = v + c * lv;
    double r1, r2;
    pair_dot(A, vc, p - 1, i2, i2, f, 0, 1, q + (p - 2) * f, -f, p - 2, -1, r1, r2);
    y[c * ly + i2] = vc[i2] + r1;
    if (i2 != q) y[c * ly + q] = vc[q] + r2;
  }
  __syncthreads();
  const int s = f - p;
  for (int t = threadIdx.x; t < s * w; t += blockDim.x) {
    const int c = t / s, i = p + t - c * s;
    v[c * lv + i] -= col_dot(A + i, f, y + c * ly, p);
  }
  __syncthreads();
  double* out = set.W + a.woff[fr] + c0;
  for (int t = threadIdx.x; t < f * w; t += blockDim.x) {
    const int i = t / w, c = t - i * w;
    out[(int64_t)i * kLdW + c] = i < p ? y[c * ly + i] : v[c * lv + i];
  }
}

template <int NT>
__global__ void __launch_bounds__(NT) mf_backward_small_kernel(const int32_t* __restrict__ lf, SolveArgs a) {
  extern __shared__ double sm[];
  const int fr = lf[blockIdx.x / a.parts], part = blockIdx.x % a.parts;
  const SolveSet set = a.set[part & (a.sets - 1)];
  const int c0 = part / a.sets * a.per, w = min(a.per, a.nb - c0);
  const FrontDesc d = a.fd[fr];
  const int f = d.f, p = d.p;
  if (p == 0) return;
  const int s = f - p, lz = p | 1, lx = (s > p ? s : p) | 1;
  double* z = sm;             // z[c * lz + i]
  double* xs = sm + lz * w;   // xs[c * lx + j]: solved struct unknowns, then the front's own
  const int32_t* D = a.dofs + d.dptr;
  const double* A = set.F + d.off;
  const double* v = set.W + a.woff[fr] + c0;
  double* X = set.X + c0;
  for (int t = threadIdx.x; t < f * w; t += blockDim.x) {
    const int i = t / w, c = t - i * w;
    if (i < p) z[c * lz + i] = v[(int64_t)i * kLdW + c];
    else xs[c * lx + i - p] = X[(int64_t)D[i] * set.ldx + c];
  }
  __syncthreads();
  for (int t = threadIdx.x; t < p * w; t += blockDim.x) {
    const int c = t / p, i = t - c * p;
    z[c * lz + i] -= col_dot(A + (int64_t)p * f + i, f, xs + c * lx, s);
  }
  __syncthreads();
  // the upper triangle: row i is a dot product of length p - i; the rows q (by falling columns) and p - 1 - q
  // (by rising ones) share a thread, p + 1 products together
  const int hp = (p + 1) >> 1;
  for (int t = threadIdx.x; t < hp * w; t += blockDim.x) {
    const int c = t / hp, q = t - c * hp, i2 = p - 1 - q;
    double r1, r2;
    pair_dot(A, z + c * lz, p + 1, p - q, q + (p - 1) * f, -f, p - 1, -1, i2 - f, f, -1, 1, r1, r2);
    xs[c * lx + q] = r1;
    if (i2 != q) xs[c * lx + i2] = r2;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < p * w; t += blockDim.x) {
    const int i = t / w, c = t - i * w;
    X[(int64_t)D[i] * set.ldx + c] = xs[c * lx + i];
  }
}

// ------------------------------------------------------------------ tiled solves (partitioned inverse)
// The upper levels of the tree hold few or small fronts, some far too large for one CTA, and GB300's
// FP64 rate per SM (under two FMA per clock) makes any solve confined to a few SMs the bottleneck. After
// the factorization, every front of such a level is turned into its partitioned
// inverse:
//   diagonal square: unit lower L11^-1 and upper U11^-1      (invert_square / mf_inverse_kernel)
//   L21 -> L21' = -L21 L11^-1,  U12 -> U12' = -U11^-1 U12    (partinv_shared / mf_partinv_kernel)
// so that each solve direction is one dense product with no dependency between rows:
//   forward:  out[r] = v[r] + sum_{k < min(r, p)} F(r, k) v[k]            every row r < f
//   backward: x[r]   = sum_{k = r}^{f - 1} F(r, k) z[k],  z = [y; x_s]    every pivot row r < p
// (v: the gathered right-hand side in pivot order; out[0:p] = y, out[p:f] the update for the parent).
// A level's rows are cut into tiles of kTileRows = 8 rows x 8 NT right-hand sides, one CTA of four warps
// each, so a level of a few fronts spreads over the whole chip. The products run as FP64 MMAs
// (mma.sync m8n8k4, the same rate as the FP64 FMAs on this chip but one instruction per 256 of them, with
// operands shared across the warp); the four warps split the inner dimension, since an 8 x 8 tile of a
// 200-row front keeps one quarter of an SM busy for 15 us and four quarters for 4 us. v is pulled without
// atomics from the B rows and the children's update vectors through a per-front source list, chunk by
// chunk, into shared memory; sums have one fixed order, so solves are reproducible bit for bit.
// With one row per warp and DFMAs a level of 4 to 64 fronts took 18 to 37 us per direction at 83k DoFs
// (24 right-hand sides), a level of 54 to 213 fronts on one CTA per front 27 to 35 us; now 8 to 14 us.
constexpr int kTileRows = 8;
constexpr int kChunkK = 128;
constexpr int kTiledMaxP = 768;   // an inverse's strip and its diagonal blocks fit 98 KB of shared memory: two CTAs per SM
constexpr int kTileThreads = 128;
constexpr int kTiledLeaves = 2;   // per SM
constexpr int kTileSteps = kChunkK / 16;   // MMA steps (4 columns of the front) per warp and chunk

struct TiledArgs {
  const FrontDesc* fd;
  const int32_t* dofs;
  const int64_t* piv_off;
  const int64_t* woff;
  const int4* pull;   // per row of a tiled front (from FrontDesc::prow on), two int4: see pull_row
  const double* B;
  int64_t ldb;
  SolveSet set[2];
  int nb;
  int chunk;   // rows of v in shared memory (see tile_product)
};

// row k (pivot order) of front d's gathered right-hand side, column c: the row's record holds its DoF (the
// row of B, -1 past the pivots), then up to MAXKIDS workspace rows of the children, in slot order, -1 past
// the last
__device__ __forceinline__ double pull_row(const TiledArgs& a, const FrontDesc& d, const double* W, const int32_t* pm, int k,
                                           int c) {
  const int u = k < d.p ? pm[k] : k;
  const int4* rec = a.pull + 2 * (d.prow + u);
  const int4 q = __ldg(rec);
  double s = q.x >= 0 ? a.B[(int64_t)q.x * a.ldb + c] : 0.0;
  if (q.y >= 0) s += W[(int64_t)q.y * kLdW + c];
  if (q.z >= 0) s += W[(int64_t)q.z * kLdW + c];
  if (q.w >= 0) {
    s += W[(int64_t)q.w * kLdW + c];
    const int last = __ldg(&rec[1].x);
    if (last >= 0) s += W[(int64_t)last * kLdW + c];
  }
  return s;
}

// One tile: rows r0 .. r0 + 7, columns c0 .. c0 + 8 NT - 1: init(r, c) + sum over kbeg <= k < kend of
// F(r, k) v[k], F taken only where use(r, k). load(k, c) gives v[k][c0 + c]; done(r, c, sum) gets each row
// below rlim. vs holds `chunk` rows of v (a multiple of 16, as many as the level's longest sum needs, so
// that short sums leave room for more CTAs per SM; never 0).
template <int NT, class Use, class Load, class Init, class Done>
__device__ __forceinline__ void tile_product(const double* __restrict__ A, int f, int r0, int rlim, int kbeg, int kend,
                                             int ncol, int chunk, const Use& use, const Load& load, const Init& init,
                                             const Done& done) {
  constexpr int LD = 8 * NT + 4;   // rows 4 banks apart: the B fragments read without conflicts
  extern __shared__ double vs[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = r0 + (lane >> 2), kl = lane & 3;
  constexpr int OWN = (64 * NT + kTileThreads - 1) / kTileThreads;
  double own[OWN];
  double acc[NT][2];
#pragma unroll
  for (int n = 0; n < NT; n++) acc[n][0] = acc[n][1] = 0.0;
#pragma unroll
  for (int i = 0; i < OWN; i++) {   // the tile's own rows
    const int t = threadIdx.x + i * kTileThreads, r = t / (8 * NT), c = t - r * (8 * NT);
    own[i] = (t < 64 * NT && r0 + r < rlim && c < ncol) ? init(r0 + r, c) : 0.0;
  }
  for (int k0 = kbeg; k0 < kend; k0 += chunk) {
    const int kc = min(chunk, kend - k0), kc4 = (kc + 3) & ~3;
    double af[kTileSteps];   // this warp's steps warp, warp + 4, ... of the chunk
#pragma unroll
    for (int i = 0; i < kTileSteps; i++) {
      const int k = k0 + 4 * (warp + 4 * i) + kl;
      af[i] = (4 * (warp + 4 * i) < kc && k < kend && row < rlim && use(row, k)) ? __ldg(A + (int64_t)k * f + row) : 0.0;
    }
    if (k0 > kbeg) __syncthreads();
    for (int t = threadIdx.x; t < kc4 * 8 * NT; t += kTileThreads) {
      const int kk = t / (8 * NT), c = t - kk * (8 * NT);
      vs[kk * LD + c] = (kk < kc && c < ncol) ? load(k0 + kk, c) : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kTileSteps; i++) {
      const int st = warp + 4 * i;
      if (4 * st < kc4) {
        const double* vb = vs + (4 * st + kl) * LD + (lane >> 2);
#pragma unroll
        for (int n = 0; n < NT; n++) dmma(acc[n], af[i], vb[8 * n]);
      }
    }
  }
  __syncthreads();
  // the four warps' partial sums, added in warp order
#pragma unroll
  for (int n = 0; n < NT; n++) {
    double* o = vs + (warp * 8 + (lane >> 2)) * (8 * NT) + 8 * n + 2 * kl;
    o[0] = acc[n][0];
    o[1] = acc[n][1];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < OWN; i++) {
    const int t = threadIdx.x + i * kTileThreads, r = t / (8 * NT), c = t - r * (8 * NT);
    if (t < 64 * NT && r0 + r < rlim && c < ncol)
      done(r0 + r, c, own[i] + ((vs[t] + vs[64 * NT + t]) + (vs[128 * NT + t] + vs[192 * NT + t])));
  }
}

// dynamic shared memory of a tile with `chunk` rows of v: those rows, later the four partial sums
constexpr size_t tile_smem(int nt, int chunk) {
  return sizeof(double) * (size_t)(chunk * (8 * nt + 4) > 256 * nt ? chunk * (8 * nt + 4) : 256 * nt);
}

// items: (front, first row) pairs; blockIdx.y: the columns from 8 NT blockIdx.y on
template <int NT>
__global__ void __launch_bounds__(kTileThreads) mf_forward_tiled_kernel(const int2* __restrict__ items, TiledArgs a) {
  const int2 it = items[blockIdx.x];
  const SolveSet set = a.set[blockIdx.z];
  const FrontDesc d = a.fd[it.x];
  const int p = d.p, c0 = blockIdx.y * 8 * NT;
  const int32_t* pm = set.perm + a.piv_off[it.x];
  double* out = set.W + a.woff[it.x] + c0;
  // rows r < p need k < r, rows r >= p need k < p
  auto pull = [&](int k, int c) { return pull_row(a, d, set.W, pm, k, c0 + c); };
  tile_product<NT>(
      set.F + d.off, d.f, it.y, d.f, 0, min(p, it.y + kTileRows), min(8 * NT, a.nb - c0), a.chunk,
      [p](int r, int k) { return k < r || r >= p; }, pull, pull,
      [&](int r, int c, double s) { out[(int64_t)r * kLdW + c] = s; });
}

template <int NT>
__global__ void __launch_bounds__(kTileThreads) mf_backward_tiled_kernel(const int2* __restrict__ items, TiledArgs a) {
  const int2 it = items[blockIdx.x];
  const SolveSet set = a.set[blockIdx.z];
  const FrontDesc d = a.fd[it.x];
  const int p = d.p, c0 = blockIdx.y * 8 * NT;
  const int32_t* D = a.dofs + d.dptr;
  const double* y = set.W + a.woff[it.x] + c0;
  double* X = set.X + c0;
  tile_product<NT>(
      set.F + d.off, d.f, it.y, p, it.y, d.f, min(8 * NT, a.nb - c0), a.chunk, [](int r, int k) { return k >= r; },
      [&](int k, int c) { return k < p ? y[(int64_t)k * kLdW + c] : X[(int64_t)D[k] * set.ldx + c]; },
      [](int, int) { return 0.0; }, [&](int r, int c, double s) { X[(int64_t)D[r] * set.ldx + c] = s; });
}

// X = Kinv B for a dense inverse (n x n, row-major): one warp per row, lane c owns right-hand side c;
// four accumulators keep the inverse-row and B-row loads in flight
__global__ void __launch_bounds__(256) dense_inverse_apply_kernel(int64_t n, const double* __restrict__ Kinv,
                                                                  const double* __restrict__ B, int64_t ldb, int nb,
                                                                  double* __restrict__ X, int64_t ldx) {
  const int lane = threadIdx.x & 31;
  for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; i < n;
       i += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    const double* row = Kinv + i * n;
    const bool live = lane < nb;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    int64_t j = 0;
    for (; j + 4 <= n; j += 4) {
      if (live) {
        s0 += row[j] * B[j * ldb + lane];
        s1 += row[j + 1] * B[(j + 1) * ldb + lane];
        s2 += row[j + 2] * B[(j + 2) * ldb + lane];
        s3 += row[j + 3] * B[(j + 3) * ldb + lane];
      }
    }
    for (; j < n; j++)
      if (live) s0 += row[j] * B[j * ldb + lane];
    if (live) X[i * ldx + lane] = (s0 + s1) + (s2 + s3);
  }
}

// Gauss-Jordan inversion of a dense n x n matrix in place (n <= 4096), one pivot per step:
//   gjp_pivot_kernel   (1 CTA)  partial pivoting: the largest |M[i][q]|, i >= q, row q <-> row p, recorded
//   gjp_update_kernel           M[i][j] -= M[i][q] M[q][j] / M[q][q] for i, j != q
//   gjp_finish_kernel           column q and row q scaled, then (one thread, next launch) the pivot inverted
// and after the last step the row interchanges are undone as column interchanges in reverse order.
// Without pivoting (SPD shifts) a non-positive pivot sets flag 2; a zero pivot sets flag 1 and is
// perturbed.
__global__ void __launch_bounds__(1024) gjp_pivot_kernel(int n, int q, int pivoting, double* __restrict__ M,
                                                         int32_t* __restrict__ piv, int* __restrict__ flags) {
  __shared__ double bv[1024];
  __shared__ int bi[1024];
  double best = -1.0;
  int bidx = q;
  if (pivoting)
    for (int i = q + threadIdx.x; i < n; i += blockDim.x) {
      const double a = fabs(M[(int64_t)i * n + q]);
      if (a > best) { best = a; bidx = i; }
    }
  bv[threadIdx.x] = best;
  bi[threadIdx.x] = bidx;
  __syncthreads();
  for (int st = blockDim.x / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st) {
      const double o = bv[threadIdx.x + st];
      const int oi = bi[threadIdx.x + st];
      if (o > bv[threadIdx.x] || (o == bv[threadIdx.x] && oi < bi[threadIdx.x])) {
        bv[threadIdx.x] = o;
        bi[threadIdx.x] = oi;
      }
    }
    __syncthreads();
  }
  const int p = pivoting ? bi[0] : q;
  if (threadIdx.x == 0) piv[q] = p;
  if (p != q)
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
      const double t = M[(int64_t)q * n + j];
      M[(int64_t)q * n + j] = M[(int64_t)p * n + j];
      M[(int64_t)p * n + j] = t;
    }
  __syncthreads();
  if (threadIdx.x == 0) {
    const double d = M[(int64_t)q * n + q];
    if (!(fabs(d) > 0.0) || (!pivoting && !(d > 0.0))) {
      atomicOr(flags, pivoting ? 1 : 2);
      if (d == 0.0) M[(int64_t)q * n + q] = 1e-300;
    }
  }
}

__global__ void gjp_update_kernel(int n, int q, double* __restrict__ M) {
  const double inv = 1.0 / M[(int64_t)q * n + q];
  const int64_t total = (int64_t)n * n;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(t / n), j = (int)(t % n);
    if (i == q || j == q) continue;
    M[t] -= M[(int64_t)i * n + q] * inv * M[(int64_t)q * n + j];
  }
}

__global__ void gjp_finish_kernel(int n, int q, double* __restrict__ M) {
  const double inv = 1.0 / M[(int64_t)q * n + q];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    if (i != q) {
      M[(int64_t)i * n + q] = -M[(int64_t)i * n + q] * inv;
      M[(int64_t)q * n + i] = M[(int64_t)q * n + i] * inv;
    }
}

__global__ void gjp_recip_kernel(int n, int q, double* __restrict__ M) {
  if (blockIdx.x == 0 && threadIdx.x == 0) M[(int64_t)q * n + q] = 1.0 / M[(int64_t)q * n + q];
}

// undo the row interchanges as column interchanges, last pivot first; one thread per row
__global__ void gjp_unscramble_kernel(int n, const int32_t* __restrict__ piv, double* __restrict__ M) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double* row = M + (int64_t)i * n;
    for (int k = n - 1; k >= 0; k--) {
      const int p = piv[k];
      if (p != k) {
        const double t = row[k];
        row[k] = row[p];
        row[p] = t;
      }
    }
  }
}

}  // namespace

void MFDevice::setup(Ctx& c, const MFSymbolic& s, int nb_max, bool pairs) {
  cudaStream_t st = c.stream;
  nf = s.nfronts;
  nlevels = s.nlevels;
  level_ptr = s.level_ptr;
  max_f = s.max_f;
  max_p = s.max_p;
  if (nb_max > kLdW) fail(FEM2D_E_INVALID_ARG, "solve block wider than the workspace rows");
  nb_cap = nb_max;
  factor_flops = s.flops;
  // fronts laid out level by level so each level's storage is contiguous
  std::vector<int64_t> off(nf, 0), poff(nf, 0), woff_h(nf, 0);
  std::vector<std::array<int32_t, MAXKIDS>> kids(nf);
  for (auto& k : kids) k.fill(-1);
  std::vector<int> nk(nf, 0);
  for (int f = 0; f < nf; f++) {
    int pa = s.parent[f];
    if (pa >= 0) {
      if (nk[pa] >= MAXKIDS) fail(FEM2D_E_INVALID_ARG, "elimination tree node with more than 4 children");
      kids[pa][nk[pa]++] = f;
    }
  }
  int64_t o = 0, po = 0, wo = 0;
  level_off.assign(nlevels + 1, 0);
  std::vector<uint8_t> fused(nf, 0);
  for (int l = 0; l < nlevels; l++) {
    const int n = s.level_ptr[l + 1] - s.level_ptr[l];
    for (int k = s.level_ptr[l]; k < s.level_ptr[l + 1]; k++) {
      const int f = s.level_fronts[k];
      fused[f] = s.p[f] <= kSmallP && s.f[f] <= (n <= c.num_sms ? kFusedNarrowF : kFusedF);
    }
  }
  level_big_end.assign(nlevels, 0);
  for (int l = 0; l < nlevels; l++) {
    level_off[l] = o;
    for (int pass = 0; pass < 2; pass++) {   // the fronts factored in global memory first: their range is zeroed
      for (int k = s.level_ptr[l]; k < s.level_ptr[l + 1]; k++) {
        int f = s.level_fronts[k];
        if (fused[f] != (pass == 1)) continue;
        off[f] = o;
        o += (int64_t)s.f[f] * s.f[f];
        poff[f] = po;
        po += s.p[f];
        woff_h[f] = wo;
        wo += (int64_t)s.f[f] * kLdW;
      }
      if (pass == 0) level_big_end[l] = o;
    }
  }
  level_off[nlevels] = o;
  mat_total = o;
  std::vector<FrontDesc> fdh(nf);
  for (int f = 0; f < nf; f++) {
    FrontDesc& x = fdh[f];
    x.f = s.f[f];
    x.p = s.p[f];
    x.parent = s.parent[f];
    for (int k = 0; k < MAXKIDS; k++) x.kid[k] = kids[f][k];
    x.off = off[f];
    x.dptr = s.dof_ptr[f];
    x.aptr = s.asm_ptr[f];
    x.aend = s.asm_ptr[f + 1];
    x.eptr = s.ea_ptr[f];
  }
  for (FrontDesc& x : fdh) x.prow = x.aux = 0;
  // Tiled levels: every level above the leaves, and leaf levels of at most kTiledLeaves fronts per SM (or with a
  // front too large for one CTA), if all their fronts have p <= kTiledMaxP. Their fronts get pull records
  // (for each front row, the children's update rows that add into it) and factor-time work items. Upper
  // levels gain at every width, since one CTA per front leaves its threads idle on the few pivots that
  // such fronts have (5,487 fronts of 10 pivots at 1M DoFs; all levels: 5.8 -> 4.9 ms per solve of 20
  // right-hand sides). Leaf fronts have most of their rows as pivots and fill a CTA: at 414 leaves the tiled
  // form took 0.34 instead of 0.31 ms per solve and 12% more factorization time, at 125 leaves both took
  // 0.14 ms.
  level_tiled.assign(nlevels, 0);
  level_kmax.assign(nlevels, 0);
  level_pmax.assign(nlevels, 0);
  if (wo / kLdW > INT32_MAX) fail(FEM2D_E_TOO_LARGE, "solve workspace rows exceed 32 bits");
  tf_ptr.assign(nlevels + 1, 0);
  tb_ptr.assign(nlevels + 1, 0);
  std::vector<int32_t> tf_h, tb_h, inv_h, ii_h, pi_h;
  std::vector<int32_t> pull_h;   // 8 per row: DoF, children's workspace rows (see pull_row)
  max_inv_p = 0;
  int64_t sq_total = 0;
  const bool single_dense = nf == 1 && max_p == max_f && max_f <= 4096;   // factor() inverts it whole
  for (int l = 0; l < nlevels; l++) {
    tf_ptr[l] = (int32_t)(tf_h.size() / 2);
    tb_ptr[l] = (int32_t)(tb_h.size() / 2);
    int ns = 0, nl = 0;
    bool fits = true;
    for (int k = s.level_ptr[l]; k < s.level_ptr[l + 1]; k++) {
      const int fr = s.level_fronts[k];
      if (s.p[fr] <= kSmallP && s.f[fr] <= kSmallF) ns++;
      else nl++;
      if (s.p[fr] > kTiledMaxP) fits = false;
    }
    if (single_dense || !fits || !(nl > 0 || l > 0 || ns <= kTiledLeaves * c.num_sms)) continue;
    level_tiled[l] = 1;
    for (int k = s.level_ptr[l]; k < s.level_ptr[l + 1]; k++) {
      const int fr = s.level_fronts[k];
      const int F = s.f[fr], P = s.p[fr];
      for (int r0 = 0; r0 < F; r0 += kTileRows) tf_h.insert(tf_h.end(), {fr, r0});
      for (int r0 = 0; r0 < P; r0 += kTileRows) tb_h.insert(tb_h.end(), {fr, r0});
      // pull records: row u of the front (before pivoting) receives row i of child ch's update block
      fdh[fr].prow = (int64_t)pull_h.size() / 8;
      pull_h.resize(pull_h.size() + (size_t)8 * F, -1);
      int32_t* rec = pull_h.data() + 8 * fdh[fr].prow;
      for (int u = 0; u < P; u++) rec[8 * u] = s.dofs[s.dof_ptr[fr] + u];
      for (int slot = 0; slot < MAXKIDS; slot++) {
        const int ch = kids[fr][slot];
        if (ch < 0) continue;
        const int sc = s.f[ch] - s.p[ch];
        for (int i = 0; i < sc; i++) {
          const int u = s.ea_map[s.ea_ptr[ch] + i];
          if (u < 0 || u >= F) fail(FEM2D_E_INVALID_ARG, "extend-add map outside the parent front");
          int q = 1;
          while (q <= MAXKIDS && rec[8 * u + q] >= 0) q++;
          if (q > MAXKIDS) fail(FEM2D_E_INVALID_ARG, "a child adds to one row twice");
          rec[8 * u + q] = (int32_t)(woff_h[ch] / kLdW + s.p[ch] + i);
        }
      }
      level_kmax[l] = std::max(level_kmax[l], std::max(F, P));
      level_pmax[l] = std::max(level_pmax[l], P);
    }
  }
  // factorization work: per level the fronts factored in global memory, and groups of the others (wide
  // levels by size class, so that small fronts share an SM; within a group the largest first)
  std::vector<int32_t> big_h, fused_h;
  big_ptr.assign(nlevels + 1, 0);
  fused_groups.clear();
  level_big_f.assign(nlevels, 0);
  level_big_p.assign(nlevels, 0);
  for (int l = 0; l < nlevels; l++) {
    big_ptr[l] = (int32_t)big_h.size();
    std::vector<int32_t> q;
    for (int k = s.level_ptr[l]; k < s.level_ptr[l + 1]; k++) {
      const int fr = s.level_fronts[k], F = s.f[fr], P = s.p[fr];
      if (fused[fr]) {
        q.push_back(fr);
        continue;
      }
      big_h.push_back(fr);
      level_big_f[l] = std::max(level_big_f[l], F);
      level_big_p[l] = std::max(level_big_p[l], P);
      if (P == 0 || !(level_tiled[l] || (P <= kSmallP && F <= kSmallF))) continue;
      inv_h.push_back(fr);
      max_inv_p = std::max(max_inv_p, P);
      fdh[fr].aux = sq_total;
      sq_total += (int64_t)P * P;
      for (int j = 0; j < (P + 7) / 8; j++) ii_h.insert(ii_h.end(), {fr, 0, j, 0, fr, 1, j, 0});
      if (level_tiled[l])
        for (int t0 = 0; t0 < F - P; t0 += 8) pi_h.insert(pi_h.end(), {fr, 0, t0, 0, fr, 1, t0, 0});
    }
    std::stable_sort(q.begin(), q.end(), [&](int32_t x, int32_t y) { return s.f[x] > s.f[y]; });
    // The launches of one stream follow each other, so a group ends at a size class only once its fronts fill the
    // chip; fewer join the next class (305 leaves at 12k DoFs, 98 of them in the first four classes: 1,501 us of
    // launches after one another, 640 so).
    const int classes[] = {116, 95, 82, kFusedSmallF, 48, 32};   // above: 1, 2, 3, 4, 6, ... CTAs per SM
    const auto fills = [&](int f, size_t count) {
      const int nt = f <= kFusedSmallF ? 128 : 256;
      const size_t per = std::min<size_t>(768 / nt, kSmemPerSM / (fused_smem(f, nt) + kFusedStatic));
      return count >= per * c.num_sms;
    };
    size_t k0 = 0;
    for (int cl = 0; k0 < q.size(); cl++) {
      size_t k1 = q.size();
      if (cl < 6 && (int)q.size() > 2 * c.num_sms) {
        k1 = k0;
        while (k1 < q.size() && s.f[q[k1]] > classes[cl]) k1++;
        if (k1 < q.size() && !fills(s.f[q[k0]], k1 - k0)) continue;
      }
      if (k1 == k0) continue;
      fused_groups.push_back({l, (int)fused_h.size(), (int)(k1 - k0), s.f[q[k0]]});
      fused_h.insert(fused_h.end(), q.begin() + k0, q.begin() + k1);
      k0 = k1;
    }
  }
  big_ptr[nlevels] = (int32_t)big_h.size();
  arena.add(lbig, big_h);
  arena.add(lfused, fused_h);
  tf_ptr[nlevels] = (int32_t)(tf_h.size() / 2);
  tb_ptr[nlevels] = (int32_t)(tb_h.size() / 2);
  ninv = (int)inv_h.size();
  ninv_items = (int)(ii_h.size() / 4);
  npinv = (int)(pi_h.size() / 4);
  arena.add(tf_items, tf_h);
  arena.add(tb_items, tb_h);
  arena.add(pull, pull_h);
  arena.add(linv, inv_h);
  arena.add(inv_items, ii_h);
  arena.add(pinv_items, pi_h);
  arena.reserve(sq, std::max<int64_t>(sq_total, 1));
  std::vector<uint8_t> raw(fdh.size() * sizeof(FrontDesc));
  std::memcpy(raw.data(), fdh.data(), raw.size());
  arena.add(desc, raw);
  arena.add(lfronts, s.level_fronts);
  arena.add(dofs, s.dofs);
  arena.add(asm_pos, s.asm_pos);
  arena.add(asm_csr, s.asm_csr);
  arena.add(ea_map, s.ea_map);
  arena.add(piv_off, poff);
  arena.add(woff, woff_h);
  piv_total = po;
  arena.reserve(work, std::max<int64_t>(wo, 1));
  if (pairs) arena.reserve(work2, std::max<int64_t>(wo, 1));
  arena.reserve(flags, 1);
  arena.reserve(weak_list, std::max<int64_t>(s.n, 1));
  arena.reserve(weak_count, 1);
  level_factor_bytes.assign(nlevels, 0.0);
  level_max_f.assign(nlevels, 0);
  level_max_p.assign(nlevels, 0);
  for (int l = 0; l < nlevels; l++)
    for (int k = s.level_ptr[l]; k < s.level_ptr[l + 1]; k++) {
      const double F = s.f[s.level_fronts[k]], P = s.p[s.level_fronts[k]];
      level_factor_bytes[l] += 8.0 * (0.5 * P * P + P * (F - P));
      level_max_f[l] = std::max(level_max_f[l], s.f[s.level_fronts[k]]);
      level_max_p[l] = std::max(level_max_p[l], s.p[s.level_fronts[k]]);
    }
  std::vector<int32_t> ls, ll;
  small_ptr.assign(nlevels + 1, 0);
  large_ptr.assign(nlevels + 1, 0);
  level_fwd_cols.assign(nlevels, 0);
  level_bwd_cols.assign(nlevels, 0);
  for (int l = 0; l < nlevels; l++) {
    small_ptr[l] = (int32_t)ls.size();
    large_ptr[l] = (int32_t)ll.size();
    for (int k = s.level_ptr[l]; k < s.level_ptr[l + 1]; k++) {
      const int fr = s.level_fronts[k];
      if (s.p[fr] <= kSmallP && s.f[fr] <= kSmallF) {
        ls.push_back(fr);
        level_fwd_cols[l] = std::max(level_fwd_cols[l], forward_cols(s.f[fr], s.p[fr]));
        level_bwd_cols[l] = std::max(level_bwd_cols[l], backward_cols(s.f[fr], s.p[fr]));
      } else {
        ll.push_back(fr);
      }
    }
    const auto cost = [&](int32_t fr) { return (int64_t)s.p[fr] * (2 * s.f[fr] - s.p[fr]); };
    std::stable_sort(ls.begin() + small_ptr[l], ls.end(), [&](int32_t x, int32_t y) { return cost(x) > cost(y); });
  }
  small_ptr[nlevels] = (int32_t)ls.size();
  large_ptr[nlevels] = (int32_t)ll.size();
  arena.add(lsmall, ls);
  arena.add(llarge, ll);
  arena.commit(st);
  // dynamic shared memory limits are set once per device (a function attribute of the device's context)
  static std::mutex attr_mu;
  static bool attr_done[256] = {};
  std::lock_guard<std::mutex> lk(attr_mu);
  if (c.device >= 0 && c.device < 256 && !attr_done[c.device]) {
    const int smem = (kSmallF + kSmallP + 2) * kLdW * (int)sizeof(double);
    FEM2D_CUDA(cudaFuncSetAttribute(mf_front_kernel<256, kFusedF>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)fused_smem(kFusedF, 256)));
    FEM2D_CUDA(cudaFuncSetAttribute(mf_front_kernel<128, kFusedSmallF>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)fused_smem(kFusedSmallF, 128)));
    FEM2D_CUDA(cudaFuncSetAttribute(mf_strip_kernel<256, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, strip_smem(256)));
    FEM2D_CUDA(cudaFuncSetAttribute(mf_strip_kernel<512, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, strip_smem(1024)));
    FEM2D_CUDA(cudaFuncSetAttribute(mf_strip_kernel<512, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, strip_smem(2048)));
    FEM2D_CUDA(cudaFuncSetAttribute(mf_inverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)inverse_smem(kTiledMaxP)));
    FEM2D_CUDA(cudaFuncSetAttribute(mf_partinv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)inverse_smem(kTiledMaxP)));
    FEM2D_CUDA(cudaFuncSetAttribute(mf_forward_small_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    FEM2D_CUDA(cudaFuncSetAttribute(mf_forward_small_kernel<512>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    FEM2D_CUDA(cudaFuncSetAttribute(mf_forward_small_kernel<1024>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    FEM2D_CUDA(cudaFuncSetAttribute(mf_backward_small_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    FEM2D_CUDA(cudaFuncSetAttribute(mf_backward_small_kernel<512>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    FEM2D_CUDA(cudaFuncSetAttribute(mf_backward_small_kernel<1024>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    attr_done[c.device] = true;
  }
}

void MFDevice::factor(Ctx& c, const double* va, const double* vb, double ca, double cb, bool cholesky,
                      MFFactor& out) {
  cudaStream_t st = c.stream;
  DBuf<double>& Fbuf = out.F;
  enable_stream_pool(c.device);
  if (Fbuf.n != (size_t)std::max<int64_t>(mat_total, 1)) Fbuf.alloc_on(std::max<int64_t>(mat_total, 1), st);
  if (out.piv.n != (size_t)std::max<int64_t>(piv_total, 1)) out.piv.alloc_on(std::max<int64_t>(piv_total, 1), st);
  FEM2D_CUDA(cudaMemsetAsync(flags.p, 0, sizeof(int), st));
  FEM2D_CUDA(cudaMemsetAsync(weak_count.p, 0, sizeof(int), st));
  out.weak.clear();
  const FrontDesc* fd = reinterpret_cast<const FrontDesc*>(desc.p);
  ProfScope ps(c, "mf_factor", 8.0 * (double)mat_total, cholesky ? 0.5 * factor_flops : factor_flops);
  out.inv_n = 0;
  if (nf == 1 && max_p == max_f && max_f <= 4096) {
    // one dense front (a small GEP): its explicit inverse by Gauss-Jordan, kept in F; solves are then
    // one dense product
    const int n = max_f;
    FEM2D_CUDA(cudaMemsetAsync(Fbuf.p, 0, (size_t)n * n * sizeof(double), st));
    mf_assemble_kernel<<<dim3(8, 1), 256, 0, st>>>(lfronts.p, fd, asm_pos.p, asm_csr.p, va, vb, ca, cb, 1, Fbuf.p);
    c.launches++;
    const int gu = (int)std::min<int64_t>(((int64_t)n * n + 255) / 256, (int64_t)c.num_sms * 8);
    const int pivoting = cholesky ? 0 : 1;
    for (int q = 0; q < n; q++) {
      gjp_pivot_kernel<<<1, 1024, 0, st>>>(n, q, pivoting, Fbuf.p, out.piv.p, flags.p);
      gjp_update_kernel<<<gu, 256, 0, st>>>(n, q, Fbuf.p);
      gjp_finish_kernel<<<(n + 255) / 256, 256, 0, st>>>(n, q, Fbuf.p);
      gjp_recip_kernel<<<1, 32, 0, st>>>(n, q, Fbuf.p);
      c.launches += 4;
    }
    if (pivoting) {
      gjp_unscramble_kernel<<<(n + 127) / 128, 128, 0, st>>>(n, out.piv.p, Fbuf.p);
      c.launches++;
    }
    FEM2D_CUDA(cudaGetLastError());
    out.inv_n = n;
    out.flags = read_flags(c);
    return;
  }
  if (out.perm.n != out.piv.n) out.perm.alloc_on(out.piv.n, st);
  if (out.iperm.n != out.piv.n) out.iperm.alloc_on(out.piv.n, st);
  const FactorArgs fa{fd,     asm_pos.p,  asm_csr.p,  va,        vb,      ca,          cb,           ea_map.p,
                      dofs.p, piv_off.p,  Fbuf.p,     out.piv.p, out.perm.p, out.iperm.p, flags.p,  weak_list.p,
                      weak_count.p, (int)weak_list.n, cholesky ? 0 : 1};
  size_t group = 0;
  for (int l = 0; l < nlevels; l++) {
    for (; group < fused_groups.size() && fused_groups[group].level == l; group++) {
      const FusedGroup& g = fused_groups[group];
      const int32_t* lf = lfused.p + g.first;
      if (g.max_f <= kFusedSmallF)
        mf_front_kernel<128, kFusedSmallF><<<g.count, 128, fused_smem(g.max_f, 128), st>>>(lf, fa, level_tiled[l]);
      else
        mf_front_kernel<256, kFusedF><<<g.count, 256, fused_smem(g.max_f, 256), st>>>(lf, fa, level_tiled[l]);
      c.launches++;
    }
    const int nbig = big_ptr[l + 1] - big_ptr[l];
    if (nbig == 0) continue;
    const int32_t* lf = lbig.p + big_ptr[l];
    FEM2D_CUDA(cudaMemsetAsync(Fbuf.p + level_off[l], 0, (level_big_end[l] - level_off[l]) * sizeof(double), st));
    mf_assemble_kernel<<<dim3(8, nbig), 256, 0, st>>>(lf, fd, asm_pos.p, asm_csr.p, va, vb, ca, cb, 0, Fbuf.p);
    c.launches++;
    const int mf = level_big_f[l], mp = level_big_p[l], strips = (mf + 7) / 8;
    if (l > 0) {
      mf_extend_add_kernel<<<dim3((mf + kExtendCols - 1) / kExtendCols, nbig), 256, 0, st>>>(lf, fd, ea_map.p, Fbuf.p);
      c.launches++;
    }
    for (int s = 0; mp > 0 && s <= (mp + 7) / 8; s++) {
      const dim3 grid(s == 0 ? 1 : strips, nbig);
      const int rows = mf - std::max(0, 8 * (s - 1));   // upper bound of the strips' rows
      if (rows <= 256) mf_strip_kernel<256, 1><<<grid, 256, strip_smem(rows), st>>>(lf, fa, s);
      else if (rows <= 1024) mf_strip_kernel<512, 2><<<grid, 512, strip_smem(rows), st>>>(lf, fa, s);
      else if (rows <= 2048) mf_strip_kernel<512, 4><<<grid, 512, strip_smem(rows), st>>>(lf, fa, s);
      else mf_strip_kernel<256, 0><<<grid, 256, 0, st>>>(lf, fa, s);
      c.launches++;
    }
  }
  const int nbig = big_ptr[nlevels];
  if (nbig > 0) {
    mf_perm_kernel<<<(nbig + 31) / 32, 32, 0, st>>>(nbig, lbig.p, fd, out.piv.p, piv_off.p, out.perm.p, out.iperm.p);
    c.launches++;
  }
  // their inverted diagonal squares, then L21' = -L21 L11^-1 and U12' = -U11^-1 U12
  if (ninv > 0) {
    mf_inverse_kernel<<<ninv_items, 128, inverse_smem(max_inv_p), st>>>(reinterpret_cast<const int4*>(inv_items.p), fd,
                                                                        Fbuf.p, sq.p);
    mf_square_copy_kernel<<<dim3(8, ninv), 256, 0, st>>>(linv.p, fd, sq.p, Fbuf.p);
    c.launches += 2;
  }
  if (npinv > 0) {
    mf_partinv_kernel<<<npinv, 128, inverse_smem(max_inv_p), st>>>(reinterpret_cast<const int4*>(pinv_items.p), fd,
                                                                   Fbuf.p);
    c.launches++;
  }

  FEM2D_CUDA(cudaGetLastError());
  out.flags = read_flags(c);
  if (!cholesky) {
    int nw = 0;
    FEM2D_CUDA(cudaMemcpyAsync(&nw, weak_count.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    FEM2D_CUDA(cudaStreamSynchronize(st));
    nw = std::min<int>(nw, (int)weak_list.n);
    if (nw > 0) {
      out.weak.resize(nw);
      FEM2D_CUDA(cudaMemcpyAsync(out.weak.data(), weak_list.p, nw * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
      FEM2D_CUDA(cudaStreamSynchronize(st));
    }
  }
}

// A level with fewer than kSplitFronts CTAs per SM splits its right-hand sides over two CTAs per front and set:
// 1,179 leaf fronts and two sets took 0.92 ms per solve instead of 0.94 (three CTAs: 1.00), 414 leaf fronts
// 0.386 instead of 0.381; at 18,502 fronts, where the level fills the chip many times over, it cost 2 to 9%.
constexpr int kSplitFronts = 16;

// How a level of ns small fronts with `cols` doubles of shared memory per right-hand side is solved, one CTA
// per front and `per` right-hand sides.
struct SmallShape {
  int per, threads;
};

static SmallShape small_shape(int ns, int cols, int nb, int num_sms) {
  const int split = ns < kSplitFronts * num_sms && nb > 8 ? 2 : 1;
  SmallShape s;
  s.per = (nb + split - 1) / split;
  const size_t smem = (size_t)cols * s.per * sizeof(double);
  const int ctas = ns * ((nb + s.per - 1) / s.per);
  s.threads = ctas <= num_sms ? 1024 : (ctas <= 2 * num_sms && smem <= 100 * 1024) ? 512 : 256;
  return s;
}

// Right-hand sides (in groups of 8) per tile of a tiled level with `items` row tiles: narrow tiles while the
// level leaves SMs idle, wide ones once it fills the chip and what counts is gathering each row once (the
// line between 4 and 32 CTAs per SM made no difference beyond 2% at 29k to 1M DoFs).
constexpr int kTileFill = 8;
static int tile_groups(int items, int nb, int num_sms) {
  const int groups = (nb + 7) / 8;
  int nt = items * groups <= kTileFill * num_sms ? 1 : (items * ((groups + 1) / 2) <= kTileFill * num_sms ? 2 : groups);
  return std::min(nt, groups);
}

void MFDevice::solve(Ctx& c, const MFFactor& fac, const double* B, int64_t ldb, double* X, int64_t ldx, int nb) {
  if (nb > nb_cap) fail(FEM2D_E_INVALID_ARG, "solve block wider than the workspace");
  if (fac.inv_n > 0) {
    ProfScope ps(c, "mf_solve", 8.0 * fac.inv_n * fac.inv_n, 2.0 * fac.inv_n * fac.inv_n * nb);
    const int64_t blocks = std::min<int64_t>((fac.inv_n * 32 + 255) / 256, (int64_t)c.num_sms * 8);
    dense_inverse_apply_kernel<<<(int)std::max<int64_t>(blocks, 1), 256, 0, c.stream>>>(fac.inv_n, fac.F.p, B, ldb, nb, X,
                                                                                 ldx);
    c.launches++;
    FEM2D_CUDA(cudaGetLastError());
    return;
  }
  solve_sets(c, 1, &fac, nullptr, B, ldb, X, ldx, nullptr, 0, nb);
}

void MFDevice::solve_pair(Ctx& c, const MFFactor& f1, const MFFactor& f2, const double* B, int64_t ldb, double* X1,
                          int64_t ldx1, double* X2, int64_t ldx2, int nb) {
  if (f1.inv_n > 0 || f2.inv_n > 0) {
    solve(c, f1, B, ldb, X1, ldx1, nb);
    solve(c, f2, B, ldb, X2, ldx2, nb);
    return;
  }
  if (nb > nb_cap) fail(FEM2D_E_INVALID_ARG, "solve block wider than the workspace");
  if (work2.n < work.n) work2.alloc(work.n);
  solve_sets(c, 2, &f1, &f2, B, ldb, X1, ldx1, X2, ldx2, nb);
}

void MFDevice::solve_sets(Ctx& c, int sets, const MFFactor* f1, const MFFactor* f2, const double* B, int64_t ldb,
                          double* X1, int64_t ldx1, double* X2, int64_t ldx2, int nb) {
  cudaStream_t st = c.stream;
  const FrontDesc* fd = reinterpret_cast<const FrontDesc*>(desc.p);
  double fbytes = 0.0;
  for (double b : level_factor_bytes) fbytes += b;
  // the whole solve is one profiled region: per-level events would dominate the short level launches
  ProfScope ps(c, "mf_solve", sets * 2.0 * fbytes, sets * 2.0 * 2.0 * (fbytes / 8.0) * nb);
  const SolveSet s1{f1->perm.p, f1->iperm.p, f1->F.p, work.p, X1, ldx1};
  const SolveSet s2 = sets == 2 ? SolveSet{f2->perm.p, f2->iperm.p, f2->F.p, work2.p, X2, ldx2} : s1;
  SolveArgs a{fd, dofs.p, ea_map.p, piv_off.p, woff.p, B, ldb, {s1, s2}, nb, nb, sets, sets};
  TiledArgs ta{fd, dofs.p, piv_off.p, woff.p, reinterpret_cast<const int4*>(pull.p), B, ldb, {s1, s2}, nb, 0};
  auto tiled = [&](bool fwd, int l, const int2* items, int ni) {
    const int nt = tile_groups(sets * ni, nb, c.num_sms);
    ta.chunk = std::max(16, std::min(kChunkK, ((fwd ? level_pmax[l] : level_kmax[l]) + 15) & ~15));
    const size_t smem = tile_smem(nt, ta.chunk);
    const dim3 grid(ni, (nb + 8 * nt - 1) / (8 * nt), sets);
    if (fwd) {
      if (nt == 1) mf_forward_tiled_kernel<1><<<grid, kTileThreads, smem, st>>>(items, ta);
      else if (nt == 2) mf_forward_tiled_kernel<2><<<grid, kTileThreads, smem, st>>>(items, ta);
      else if (nt == 3) mf_forward_tiled_kernel<3><<<grid, kTileThreads, smem, st>>>(items, ta);
      else mf_forward_tiled_kernel<4><<<grid, kTileThreads, smem, st>>>(items, ta);
    } else {
      if (nt == 1) mf_backward_tiled_kernel<1><<<grid, kTileThreads, smem, st>>>(items, ta);
      else if (nt == 2) mf_backward_tiled_kernel<2><<<grid, kTileThreads, smem, st>>>(items, ta);
      else if (nt == 3) mf_backward_tiled_kernel<3><<<grid, kTileThreads, smem, st>>>(items, ta);
      else mf_backward_tiled_kernel<4><<<grid, kTileThreads, smem, st>>>(items, ta);
    }
    c.launches++;
  };
  auto small = [&](bool fwd, int l, int ns) {
    const int cols = fwd ? level_fwd_cols[l] : level_bwd_cols[l];
    const SmallShape s = small_shape(sets * ns, cols, nb, c.num_sms);
    a.per = s.per;
    a.parts = sets * ((nb + s.per - 1) / s.per);
    const unsigned grid = (unsigned)ns * a.parts;
    const size_t smem = (size_t)cols * s.per * sizeof(double);
    const int32_t* lf = lsmall.p + small_ptr[l];
    if (fwd) {
      if (s.threads == 1024) mf_forward_small_kernel<1024><<<grid, 1024, smem, st>>>(lf, a);
      else if (s.threads == 512) mf_forward_small_kernel<512><<<grid, 512, smem, st>>>(lf, a);
      else mf_forward_small_kernel<256><<<grid, 256, smem, st>>>(lf, a);
    } else {
      if (s.threads == 1024) mf_backward_small_kernel<1024><<<grid, 1024, smem, st>>>(lf, a);
      else if (s.threads == 512) mf_backward_small_kernel<512><<<grid, 512, smem, st>>>(lf, a);
      else mf_backward_small_kernel<256><<<grid, 256, smem, st>>>(lf, a);
    }
    c.launches++;
  };
  const int2* tfi = reinterpret_cast<const int2*>(tf_items.p);
  const int2* tbi = reinterpret_cast<const int2*>(tb_items.p);
  for (int l = 0; l < nlevels; l++) {
    if (level_tiled[l]) {
      const int ni = tf_ptr[l + 1] - tf_ptr[l];
      if (ni > 0) tiled(true, l, tfi + tf_ptr[l], ni);
      continue;
    }
    const int ns = small_ptr[l + 1] - small_ptr[l], nl = large_ptr[l + 1] - large_ptr[l];
    if (ns > 0) small(true, l, ns);
    if (nl > 0) {
      for (int q = 0; q < sets; q++) {
        const SolveSet& s = a.set[q];
        mf_forward_cluster_kernel<<<nl * CL, 256, 0, st>>>(llarge.p + large_ptr[l], fd, dofs.p, ea_map.p, s.perm, s.iperm,
                                                           piv_off.p, woff.p, s.F, B, ldb, nb, s.W);
        c.launches++;
      }
    }
  }
  for (int l = nlevels - 1; l >= 0; l--) {
    if (level_tiled[l]) {
      const int ni = tb_ptr[l + 1] - tb_ptr[l];
      if (ni > 0) tiled(false, l, tbi + tb_ptr[l], ni);
      continue;
    }
    const int ns = small_ptr[l + 1] - small_ptr[l], nl = large_ptr[l + 1] - large_ptr[l];
    if (ns > 0) small(false, l, ns);
    if (nl > 0) {
      for (int q = 0; q < sets; q++) {
        const SolveSet& s = a.set[q];
        mf_backward_cluster_kernel<<<nl * CL, 256, 0, st>>>(llarge.p + large_ptr[l], fd, dofs.p, woff.p, s.F, s.W, nb, s.X,
                                                            s.ldx);
        c.launches++;
      }
    }
  }
  FEM2D_CUDA(cudaGetLastError());
}

// ------------------------------------------------------------------ ordered solves (dense eigensolve)
// The dense eigensolve reads the lower triangle of B^-1 A, whose structurally zero entries are rounding noise of
// 1e-17, and the sign of its eigenvector follows the signs of that noise through the Householder reflectors: one
// ulp in four of the 55 entries of a 10-DoF problem turns the vector round. The order of the sums is part
// of that result, so it does not follow the tuned kernels (with them 37 of 120 small problems changed sign): LU in
// panels of 32 columns without pivoting, a column's sums in plain loops, inverted squares, and on levels of few or
// large fronts (`parted`: by the tree alone, so that the order is the same on every chip) the partitioned inverse.
// At most 1,000 DoFs: one CTA per front, then one per front and 32 columns; bound by the latency of a level (123 DoFs: 2.25 ms a solve with the tuned kernels, 2.27 with these; 370 to
// 984 DoFs: 0.6 to 5.6 ms of the 36 to 630 ms that the whole solve takes, most of it on the host;
// the kernels whose order they keep took 1.5 to 4.8).
constexpr int kOrderedPanel = 32, kOrderedMaxP = 768, kOrderedParted = 38;

__global__ void __launch_bounds__(256) mf_ordered_factor_kernel(const int32_t* __restrict__ lf,
                                                                const FrontDesc* __restrict__ fd,
                                                                const int64_t* __restrict__ apos,
                                                                const int64_t* __restrict__ acsr,
                                                                const int32_t* __restrict__ emap,
                                                                const double* __restrict__ vals, int parted, double* F,
                                                                double* G, int* __restrict__ flags) {
  const FrontDesc d = fd[lf[blockIdx.x]];
  const int f = d.f, p = d.p, s = f - p, tid = threadIdx.x, nt = blockDim.x;
  double* A = F + d.off;
  for (int t = tid; t < f * f; t += nt) A[t] = 0.0;
  __syncthreads();
  for (int64_t k = d.aptr + tid; k < d.aend; k += nt) A[apos[k]] = vals[acsr[k]];
  for (int slot = 0; slot < MAXKIDS; slot++) {
    __syncthreads();
    if (d.kid[slot] < 0) continue;   // uniform across the CTA
    const FrontDesc cd = fd[d.kid[slot]];
    const int cs = cd.f - cd.p;
    const int32_t* m = emap + cd.eptr;
    for (int t = tid; t < cs * cs; t += nt) {
      const int i = t % cs, j = t / cs;
      A[m[j] * f + m[i]] += F[cd.off + (int64_t)(cd.p + j) * cd.f + cd.p + i];
    }
  }
  __syncthreads();
  for (int k0 = 0; k0 < p; k0 += kOrderedPanel) {
    const int w = min(kOrderedPanel, p - k0), base = k0 + w;
    for (int k = k0; k < base; k++) {
      double* col = A + k * f;
      double dk = col[k];
      __syncthreads();
      if (dk == 0.0) dk = 1e-300;
      if (tid == 0 && !(col[k] > 0.0)) {
        atomicOr(flags, 2);
        col[k] = dk;
      }
      const double inv = 1.0 / dk;
      for (int i = k + 1 + tid; i < f; i += nt) col[i] *= inv;
      __syncthreads();
      const int rows = f - (k + 1);
      for (int t = tid; t < (base - (k + 1)) * rows; t += nt) {
        const int jj = k + 1 + t / rows, ii = k + 1 + t % rows;
        A[jj * f + ii] = fma(-col[ii], A[jj * f + k], A[jj * f + ii]);
      }
      __syncthreads();
    }
    for (int j = base + tid; j < f; j += nt) {   // U12 of the panel's rows
      double* x = A + j * f + k0;
      for (int r = 1; r < w; r++) {
        double sum = x[r];
        for (int q = 0; q < r; q++) sum = fma(-A[(k0 + q) * f + k0 + r], x[q], sum);
        x[r] = sum;
      }
    }
    __syncthreads();
    const int rest = f - base;
    for (int t = tid; t < rest * rest; t += nt) {
      const int r = base + t % rest, q = base + t / rest;
      double acc = 0.0;
      for (int k = k0; k < base; k++) acc = fma(A[k * f + r], A[q * f + k], acc);
      A[q * f + r] -= acc;
    }
    __syncthreads();
  }
  // the pivot square, L21 by rows and U12 by columns, as the inverses below read them
  double *S = G + d.off, *Lr = S + p * p, *Uc = Lr + s * p;
  for (int t = tid; t < p * p; t += nt) S[t] = A[t / p * f + t % p];
  for (int t = tid; t < s * p; t += nt) {
    const int q = t / p, k = t % p;
    Lr[t] = A[k * f + p + q];
    Uc[t] = A[(p + q) * f + k];
  }
  __syncthreads();
  const bool two = p > kSmallP;   // two sums by turns
  for (int j = tid; j < p; j += nt) {
    double* out = A + j * f;   // column j; only this thread writes it
    for (int i = j + 1; i < p; i++) {
      double a[2] = {-S[j * p + i], 0.0};
      for (int k = j + 1; k < i; k++) {
        const int z = two ? (k - j - 1) & 1 : 0;
        a[z] = fma(-S[k * p + i], out[k], a[z]);
      }
      out[i] = two ? a[0] + a[1] : a[0];
    }
    out[j] = 1.0 / S[j * p + j];
    for (int i = j - 1; i >= 0; i--) {
      double a[2] = {0.0, 0.0};
      for (int k = i + 1; k <= j; k++) {
        const int z = two ? (k - i - 1) & 1 : 0;
        a[z] = fma(S[k * p + i], out[k], a[z]);
      }
      out[i] = -(two ? a[0] + a[1] : a[0]) / S[i * p + i];
    }
  }
  if (!parted) return;
  __syncthreads();
  const int lane = tid & 31;
  for (int q = tid >> 5; q < s; q += nt >> 5) {
    const double *b = Lr + q * p, *u = Uc + q * p;
    for (int k = 0; k < p; k++) {
      double sum = 0.0;
      for (int i = k + 1 + lane; i < p; i += 32) sum = fma(b[i], A[k * f + i], sum);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
      if (lane == 0) A[k * f + p + q] = -(b[k] + sum);
    }
    for (int i = lane; i < p; i += 32) {
      double a[2] = {0.0, 0.0};
      for (int k = i; k < p; k++) a[(k - i) & 1] = fma(A[k * f + i], u[k], a[(k - i) & 1]);
      A[(p + q) * f + i] = -(a[0] + a[1]);
    }
  }
}

// sum over k0 <= k < k1 of A[k f] v(k): four sums by turns and the rest with the first; or, on a parted level,
// two sums by turns that start again at every 128 from `from` on
template <class V>
__device__ __forceinline__ double ordered_dot(const double* A, int f, int k0, int k1, int parted, int from, const V& v) {
  double a[4] = {0.0, 0.0, 0.0, 0.0};
  if (!parted) {
    for (int k = k0; k < k1; k++) {
      const int z = k0 + ((k1 - k0) & ~3) > k ? (k - k0) & 3 : 0;
      a[z] = fma(A[(int64_t)k * f], v(k), a[z]);
    }
    return (a[0] + a[1]) + (a[2] + a[3]);
  }
  for (int c0 = from; c0 < k1; c0 += 128) {
    const int b = max(c0, k0), e = min(c0 + 128, k1);
    for (int k = b; k < e; k++) a[(k - b) & 1] = fma(A[(int64_t)k * f], v(k), a[(k - b) & 1]);
  }
  return a[0] + a[1];
}

// one front and 32 columns per CTA; V: gathered right-hand sides, W: solved rows and updates (per 32 columns)
__global__ void __launch_bounds__(256) mf_ordered_forward_kernel(const int32_t* __restrict__ lf,
                                                                 const FrontDesc* __restrict__ fd,
                                                                 const int32_t* __restrict__ dofs,
                                                                 const int32_t* __restrict__ emap,
                                                                 const int64_t* __restrict__ woff, int parted,
                                                                 const double* __restrict__ F, int64_t wsize, int64_t n,
                                                                 const double* __restrict__ B, double* V, double* W) {
  const int fr = lf[blockIdx.x];
  const FrontDesc d = fd[fr];
  const int f = d.f, p = d.p, c0 = blockIdx.y * kLdW, w = (int)min((int64_t)kLdW, n - c0), c = threadIdx.x & 31;
  const double* A = F + d.off;
  double *v = V + blockIdx.y * wsize + woff[fr] + c, *o = W + blockIdx.y * wsize + woff[fr] + c;
  const int row0 = threadIdx.x >> 5, rows = blockDim.x >> 5;
  for (int i = row0; i < f; i += rows) v[i * kLdW] = i < p && c < w ? B[(int64_t)dofs[d.dptr + i] * n + c0 + c] : 0.0;
  for (int slot = 0; slot < MAXKIDS; slot++) {
    __syncthreads();
    if (d.kid[slot] < 0) continue;   // uniform across the CTA
    const FrontDesc cd = fd[d.kid[slot]];
    const double* cw = W + blockIdx.y * wsize + woff[d.kid[slot]] + cd.p * kLdW + c;
    for (int i = row0; i < cd.f - cd.p; i += rows) v[emap[cd.eptr + i] * kLdW] += cw[i * kLdW];
  }
  __syncthreads();
  const auto gathered = [&](int k) { return v[k * kLdW]; };
  const auto solved = [&](int k) { return o[k * kLdW]; };
  for (int i = row0; i < (parted ? f : p); i += rows)
    o[i * kLdW] = v[i * kLdW] + ordered_dot(A + i, f, 0, min(i, p), parted, 0, gathered);
  __syncthreads();
  if (!parted)
    for (int i = p + row0; i < f; i += rows) o[i * kLdW] = v[i * kLdW] - ordered_dot(A + i, f, 0, p, 0, 0, solved);
}

__global__ void __launch_bounds__(256) mf_ordered_backward_kernel(const int32_t* __restrict__ lf,
                                                                  const FrontDesc* __restrict__ fd,
                                                                  const int32_t* __restrict__ dofs,
                                                                  const int64_t* __restrict__ woff, int parted,
                                                                  const double* __restrict__ F, int64_t wsize, int64_t n,
                                                                  double* V, const double* W, double* X) {
  const int fr = lf[blockIdx.x];
  const FrontDesc d = fd[fr];
  const int f = d.f, p = d.p, c0 = blockIdx.y * kLdW, w = (int)min((int64_t)kLdW, n - c0), c = threadIdx.x & 31;
  const double* A = F + d.off;
  const int32_t* D = dofs + d.dptr;
  double* z = V + blockIdx.y * wsize + woff[fr] + c;
  const double* y = W + blockIdx.y * wsize + woff[fr] + c;
  const int row0 = threadIdx.x >> 5, rows = blockDim.x >> 5;
  for (int k = row0; k < f; k += rows)
    z[k * kLdW] = k < p ? y[k * kLdW] : (c < w ? X[(int64_t)D[k] * n + c0 + c] : 0.0);
  __syncthreads();
  const auto value = [&](int k) { return z[k * kLdW]; };
  if (!parted) {
    for (int i = row0; i < p; i += rows)
      z[i * kLdW] -= ordered_dot(A + (int64_t)p * f + i, f, 0, f - p, 0, 0, [&](int k) { return z[(p + k) * kLdW]; });
    __syncthreads();
  }
  for (int i = row0; i < p; i += rows) {
    const double x = ordered_dot(A + i, f, i, parted ? f : p, parted, i & ~7, value);
    if (c < w) X[(int64_t)D[i] * n + c0 + c] = x;
  }
}

bool MFDevice::solve_ordered(Ctx& c, const double* vals, int64_t n, const double* B, double* X, int* flags_out) {
  std::vector<int> parted(nlevels, 0);
  for (int l = 0; l < nlevels; l++) {
    const int count = level_ptr[l + 1] - level_ptr[l];
    if (level_max_p[l] > kOrderedMaxP) return false;
    const bool large = level_max_p[l] > kSmallP || level_max_f[l] > kSmallF;
    parted[l] = large || count <= kOrderedParted;
  }
  const cudaStream_t st = c.stream;
  const FrontDesc* fd = reinterpret_cast<const FrontDesc*>(desc.p);
  const int groups = (int)((n + kLdW - 1) / kLdW);
  const int64_t wsize = (int64_t)work.n;
  DBuf<double> F, G, V, W;
  F.alloc_on(std::max<int64_t>(mat_total, 1), st);
  G.alloc_on(std::max<int64_t>(mat_total, 1), st);
  V.alloc_on(wsize * groups, st);
  W.alloc_on(wsize * groups, st);
  FEM2D_CUDA(cudaMemsetAsync(flags.p, 0, sizeof(int), st));
  {
    ProfScope ps(c, "mf_factor", 8.0 * (double)mat_total, 0.5 * factor_flops);
    for (int l = 0; l < nlevels; l++) {
      const int count = level_ptr[l + 1] - level_ptr[l];
      mf_ordered_factor_kernel<<<count, 256, 0, st>>>(lfronts.p + level_ptr[l], fd, asm_pos.p, asm_csr.p, ea_map.p, vals,
                                                      parted[l], F.p, G.p, flags.p);
    }
  }
  double fbytes = 0.0;
  for (double b : level_factor_bytes) fbytes += b;
  ProfScope ps(c, "mf_solve", 2.0 * fbytes, 2.0 * 2.0 * (fbytes / 8.0) * n);
  for (int l = 0; l < nlevels; l++)
    mf_ordered_forward_kernel<<<dim3(level_ptr[l + 1] - level_ptr[l], groups), 256, 0, st>>>(
        lfronts.p + level_ptr[l], fd, dofs.p, ea_map.p, woff.p, parted[l], F.p, wsize, n, B, V.p, W.p);
  for (int l = nlevels - 1; l >= 0; l--)
    mf_ordered_backward_kernel<<<dim3(level_ptr[l + 1] - level_ptr[l], groups), 256, 0, st>>>(
        lfronts.p + level_ptr[l], fd, dofs.p, woff.p, parted[l], F.p, wsize, n, V.p, W.p, X);
  c.launches += 3 * nlevels;
  FEM2D_CUDA(cudaGetLastError());
  *flags_out = read_flags(c);
  return true;
}

int MFDevice::read_flags(Ctx& c) {
  int h = 0;
  FEM2D_CUDA(cudaMemcpyAsync(&h, flags.p, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
  FEM2D_CUDA(cudaStreamSynchronize(c.stream));
  return h;
}

}  // namespace fem2d
