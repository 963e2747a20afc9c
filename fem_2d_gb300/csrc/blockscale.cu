// Block congruence scaling of the pencil over row runs.
//
// The rows of one run (consecutive DoFs with one column list: an Elem's interior functions) keep a
// common pattern, and by symmetry so do their columns. With S = blockdiag(L_g^-1), B_gg = L_g L_g^T
// the Cholesky factor of B's diagonal block of run g, the pencil (S A S^T, S B S^T) has exactly the
// sparsity pattern of (A, B), the same eigenvalues, eigenvectors x = S^T x~, and identity diagonal
// blocks in S B S^T. For high-order monomial (HierPoly) bases this lowers cond(B) by three or more
// orders of magnitude where the diagonal (Jacobi) scaling only normalises the diagonal, and with it
// the digits the shifted factorizations lose. It costs (|g| + |h|) |g| |h| FP64 FMAs per coupled
// block pair, so the solver applies it only when the Jacobi-scaled factorizations are inaccurate.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "blockscale.h"
#include "dmma.h"

namespace fem2d {

namespace {

constexpr int kRun = 64;   // rows per run (the runs of device_upload are at most 64 long)

// per listed run of at most LD rows: Cholesky of B_gg in shared memory, then S_g = L^-1 (row-major, lower) to
// global. Runs of up to kSmallRun rows (60% of them at 1M DoFs) take small CTAs of their own: at the
// 64 KB of the long ones three fit an SM.
constexpr int kSmallRun = 16;
template <int LD>
__global__ void __launch_bounds__(4 * LD) run_cholinv_kernel(const int32_t* __restrict__ list,
                                                          const int32_t* __restrict__ grp,
                                                          const int64_t* __restrict__ rp,
                                                          const int32_t* __restrict__ col,
                                                          const double* __restrict__ vb,
                                                          const int64_t* __restrict__ soff,
                                                          double* __restrict__ S, int* __restrict__ flag) {
  extern __shared__ double csm[];
  double* M = csm;                 // LD x LD
  double* Li = csm + LD * LD;  // LD x LD
  __shared__ int s_off;
  const int g = list[blockIdx.x];
  const int g0 = grp[g], R = grp[g + 1] - g0;
  if (threadIdx.x == 0) {   // position of column g0 in row g0 (every row of the run has the same list)
    int lo = 0, hi = (int)(rp[g0 + 1] - rp[g0]) - 1, at = -1;
    const int32_t* cl = col + rp[g0];
    while (lo <= hi) {
      const int mid = (lo + hi) >> 1;
      if (cl[mid] == g0) { at = mid; break; }
      if (cl[mid] < g0) lo = mid + 1; else hi = mid - 1;
    }
    s_off = at;
    if (at < 0) atomicOr(flag, 2);
  }
  __syncthreads();
  if (s_off < 0) return;
  for (int t = threadIdx.x; t < R * R; t += blockDim.x) {
    const int r = t / R, q = t % R;
    M[r * LD + q] = vb[rp[g0 + r] + s_off + q];
  }
  __syncthreads();
  for (int j = 0; j < R; j++) {   // right-looking Cholesky, lower triangle
    if (threadIdx.x == 0) {
      const double d = M[j * LD + j];
      if (!(d > 0.0)) atomicOr(flag, 1);
      M[j * LD + j] = d > 0.0 ? sqrt(d) : 1.0;
    }
    __syncthreads();
    const double dj = M[j * LD + j];
    for (int i = j + 1 + threadIdx.x; i < R; i += blockDim.x) M[i * LD + j] /= dj;
    __syncthreads();
    for (int t = threadIdx.x; t < (R - j - 1) * (R - j - 1); t += blockDim.x) {
      const int i = j + 1 + t / (R - j - 1), k = j + 1 + t % (R - j - 1);
      if (k <= i) M[i * LD + k] -= M[i * LD + j] * M[k * LD + j];
    }
    __syncthreads();
  }
  // column q of L^-1 per thread: L x = e_q
  for (int q = threadIdx.x; q < R; q += blockDim.x) {
    for (int i = 0; i < q; i++) Li[i * LD + q] = 0.0;
    Li[q * LD + q] = 1.0 / M[q * LD + q];
    for (int i = q + 1; i < R; i++) {
      double s = 0.0;
      for (int k = q; k < i; k++) s += M[i * LD + k] * Li[k * LD + q];
      Li[i * LD + q] = -s / M[i * LD + i];
    }
  }
  __syncthreads();
  double* out = S + soff[g];
  for (int t = threadIdx.x; t < R * R; t += blockDim.x) out[t] = Li[(t / R) * LD + t % R];
}

// Per run g and matrix (blockIdx.y: A, B): block <- S_g block S_h^T for every column run h of its pattern, both
// factors lower triangular, as FP64 MMAs on 8 x 8 tiles: U = S_g block with all operands read straight into
// the fragments (rows of the CSR and of S are contiguous), U kept in shared memory, then U S_h^T. In this order:
// the result multiplies y = S^-T x from the left, so that the rounding of S_g block meets the smooth S_h^T y = x,
// where that of block S_h^T would meet y itself, which is large for a monomial basis (eigenvectors of HierPoly
// pencils at 12,430 DoFs: 1 to 2e-8 from the exact ones, 8 to 9e-8 the other way). The column
// runs go in groups of up to kGroupTiles tiles, so that the many runs of 4 to 8 functions fill the eight warps
// together. One column run at a time through shared memory, with six barriers each, took 31.5 ms at 1M DoFs;
// now 28, of which the FP64 pipe needs 20 (26 with the tiles' padding). Loading whole tiles ahead of their
// products was slower (33 ms).
constexpr int kTransformThreads = 256;
constexpr int kGroupTiles = 12;
constexpr int kUld = 8 * kGroupTiles + 4;   // rows 4 banks apart: fragments read without conflicts
constexpr int kTransformSmem = kRun * kUld * (int)sizeof(double);
__global__ void __launch_bounds__(kTransformThreads) run_transform_kernel(
    const int32_t* __restrict__ grp, const int64_t* __restrict__ rp, const int64_t* __restrict__ seg_ptr,
    const int2* __restrict__ seg, const int64_t* __restrict__ soff, const double* __restrict__ S,
    const double* __restrict__ va, const double* __restrict__ vb, double* __restrict__ sa, double* __restrict__ sb) {
  extern __shared__ double U[];
  __shared__ int64_t tile_s[kGroupTiles];                               // S_h of the tile's column run
  __shared__ int tile_h[kGroupTiles], tile_c[kGroupTiles], tile_j[kGroupTiles];   // its order, first column, tile in it
  __shared__ int ntiles;
  __shared__ int64_t next;
  const double* src = blockIdx.y == 0 ? va : vb;
  double* dst = blockIdx.y == 0 ? sa : sb;
  const int g = blockIdx.x, g0 = grp[g], R = grp[g + 1] - g0, strips = (R + 7) >> 3;
  const double* Sg = S + soff[g];
  const int64_t r0 = rp[g0], len = rp[g0 + 1] - r0;   // the run's rows follow each other, len entries each
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q8 = lane >> 2, kl = lane & 3;
  const int64_t end = seg_ptr[g + 1];
  for (int64_t first = seg_ptr[g]; first < end; first = next) {
    __syncthreads();   // U and the tile list of the previous group are read
    if (threadIdx.x == 0) {
      int n = 0;
      int64_t s = first;
      for (; s < end; s++) {
        const int2 sh = seg[s];
        const int H = grp[sh.x + 1] - grp[sh.x], ht = (H + 7) >> 3;
        if (n + ht > kGroupTiles) break;   // (a column run has at most 8 tiles: every group makes progress)
        for (int j = 0; j < ht; j++, n++) {
          tile_s[n] = soff[sh.x];
          tile_h[n] = H;
          tile_c[n] = sh.y;
          tile_j[n] = j;
        }
      }
      ntiles = n;
      next = s;
    }
    __syncthreads();
    const int nt = ntiles;
    // U = S_g block: tile (strip i, tile j of h) sums the rows of g up to strip i
    for (int w = warp; w < strips * nt; w += kTransformThreads / 32) {
      const int i = w % strips, c = w / strips, H = tile_h[c];
      const int row = 8 * i + q8, col = 8 * tile_j[c] + q8;
      const double* b = src + r0 + tile_c[c] + col;
      double acc[2] = {0.0, 0.0};
      for (int k0 = 0; k0 <= 8 * i + 4; k0 += 4) {
        const int k = k0 + kl;
        const double x = (row < R && k <= row) ? __ldg(Sg + row * R + k) : 0.0;
        const double y = (k < R && col < H) ? __ldg(b + (int64_t)k * len) : 0.0;
        dmma(acc, x, y);
      }
      double* u = U + row * kUld + 8 * c + 2 * kl;
      u[0] = acc[0];
      u[1] = acc[1];
    }
    __syncthreads();
    // out = U S_h^T: tile j sums U's columns of h up to tile j
    for (int w = warp; w < strips * nt; w += kTransformThreads / 32) {
      const int i = w % strips, c = w / strips, H = tile_h[c], j = tile_j[c];
      const double* Sh = S + tile_s[c];
      const int row = 8 * i + q8, scol = 8 * j + q8;
      const double* u = U + row * kUld + 8 * (c - j);
      double acc[2] = {0.0, 0.0};
      for (int k0 = 0; k0 <= 8 * j + 4; k0 += 4) {
        const int k = k0 + kl;
        const double y = (scol < H && k <= scol) ? __ldg(Sh + (int64_t)scol * H + k) : 0.0;   // S_h[scol][k]
        dmma(acc, u[k], y);
      }
      const int col = 8 * j + 2 * kl;
      double* o = dst + r0 + (int64_t)row * len + tile_c[c] + col;
      if (row < R && col < H) o[0] = acc[0];
      if (row < R && col + 1 < H) o[1] = acc[1];
    }
  }
}

// X_g <- S_g^T X_g per run (back to the original basis)
__global__ void __launch_bounds__(256) run_back_kernel(const int32_t* __restrict__ grp,
                                                       const int64_t* __restrict__ soff,
                                                       const double* __restrict__ S, double* __restrict__ X,
                                                       int64_t ldx, int nb) {
  __shared__ double xs[kRun * 32];
  const int g = blockIdx.x;
  const int g0 = grp[g], R = grp[g + 1] - g0;
  for (int t = threadIdx.x; t < R * nb; t += blockDim.x) xs[t] = X[(int64_t)(g0 + t / nb) * ldx + t % nb];
  __syncthreads();
  const double* Sg = S + soff[g];
  for (int t = threadIdx.x; t < R * nb; t += blockDim.x) {
    const int r = t / nb, c = t % nb;
    double s = 0.0;
    for (int k = r; k < R; k++) s += Sg[k * R + r] * xs[k * nb + c];   // (S_g^T)[r][k] = S_g[k][r]
    X[(int64_t)(g0 + r) * ldx + c] = s;
  }
}

}  // namespace

void BlockScale::build(Ctx& c, const HostGEP& h, const DeviceGEP& d, double* sa, double* sb) {
  if (!ready) {
    const int64_t n = h.n;
    // runs exactly as device_upload forms them, their column-run segments, block offsets
    const std::vector<int32_t>& grp = d.grp_h;
    ngrp = (int)grp.size() - 1;
    std::vector<int32_t> run_of(n);
    for (int g = 0; g < ngrp; g++)
      for (int32_t i = grp[g]; i < grp[g + 1]; i++) run_of[i] = g;
    std::vector<int64_t> so(ngrp + 1, 0), sp(ngrp + 1, 0);
    std::vector<int2> sg;
    for (int g = 0; g < ngrp; g++) {
      const int R = grp[g + 1] - grp[g];
      so[g + 1] = so[g] + (int64_t)R * R;
      alg_flops += (double)R * R * R;        // Cholesky (R^3 / 3 FMA) and inverse (R^3 / 6 FMA)
      alg_bytes += 8.0 * 3.0 * R * R;        // B's diagonal block read, S_g written and read back
      const int64_t b = h.row_ptr[grp[g]], e = h.row_ptr[grp[g] + 1];
      int64_t q = b;
      while (q < e) {
        const int32_t hr = run_of[h.col[q]];
        const int H = grp[hr + 1] - grp[hr];
        // a column run appears whole and in order (its columns are consecutive DoFs)
        if (h.col[q] != grp[hr] || q + H > e || h.col[q + H - 1] != grp[hr] + H - 1)
          fail(FEM2D_E_INVALID_ARG, "block scaling: a column run is split in a row pattern");
        sg.push_back(make_int2(hr, (int)(q - b)));
        alg_flops += 2.0 * 2.0 * ((double)R * (R + 1) / 2.0 * H + (double)R * H * (H + 1) / 2.0);
        alg_bytes += 8.0 * (double)H * H;   // S_h read for this block
        q += H;
      }
      sp[g + 1] = (int64_t)sg.size();
    }
    // kept in the GEP's plan across solves: plain (not stream-ordered) allocations
    std::vector<int32_t> runs[2];   // short, long
    for (int g = 0; g < ngrp; g++) runs[grp[g + 1] - grp[g] > kSmallRun].push_back(g);
    nshort = (int)runs[0].size();
    runs[0].insert(runs[0].end(), runs[1].begin(), runs[1].end());
    list.upload(runs[0], c.stream);
    grp_d.upload(grp, c.stream);
    soff.upload(so, c.stream);
    seg_ptr.upload(sp, c.stream);
    seg.upload(sg, c.stream);
    S.alloc(std::max<int64_t>(so[ngrp], 1));
    alg_bytes += 32.0 * (double)h.nnz_full;
    ready = true;
  }
  DBuf<int> flag;
  flag.alloc_on(1, c.stream);
  FEM2D_CUDA(cudaMemsetAsync(flag.p, 0, sizeof(int), c.stream));
  static std::mutex mu;
  static bool attr[256] = {};
  {
    std::lock_guard<std::mutex> lk(mu);
    if (c.device >= 0 && c.device < 256 && !attr[c.device]) {
      FEM2D_CUDA(cudaFuncSetAttribute(run_cholinv_kernel<kRun>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      2 * kRun * kRun * (int)sizeof(double)));
      FEM2D_CUDA(cudaFuncSetAttribute(run_transform_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      kTransformSmem));
      attr[c.device] = true;
    }
  }
  if (nshort > 0) {
    run_cholinv_kernel<kSmallRun><<<nshort, 4 * kSmallRun, 2 * kSmallRun * kSmallRun * sizeof(double), c.stream>>>(
        list.p, grp_d.p, d.row_ptr.p, d.col.p, d.b.p, soff.p, S.p, flag.p);
    c.launches++;
  }
  if (ngrp > nshort) {
    run_cholinv_kernel<kRun><<<ngrp - nshort, 4 * kRun, 2 * kRun * kRun * sizeof(double), c.stream>>>(
        list.p + nshort, grp_d.p, d.row_ptr.p, d.col.p, d.b.p, soff.p, S.p, flag.p);
    c.launches++;
  }
  run_transform_kernel<<<dim3(ngrp, 2), kTransformThreads, kTransformSmem, c.stream>>>(
      grp_d.p, d.row_ptr.p, seg_ptr.p, seg.p, soff.p, S.p, d.a.p, d.b.p, sa, sb);
  c.launches++;
  FEM2D_CUDA(cudaGetLastError());
  int hf = 0;
  FEM2D_CUDA(cudaMemcpyAsync(&hf, flag.p, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
  FEM2D_CUDA(cudaStreamSynchronize(c.stream));
  if (hf & 2) fail(FEM2D_E_INVALID_ARG, "block scaling: a run's diagonal block is missing from the pattern");
  if (hf & 1) fail(FEM2D_E_B_NOT_SPD, "a diagonal block of B is not positive definite");
}

void BlockScale::unscale(Ctx& c, double* X, int64_t ldx, int nb) const {
  if (nb > 32) fail(FEM2D_E_INVALID_ARG, "block unscaling of more than 32 columns");
  run_back_kernel<<<ngrp, 256, 0, c.stream>>>(grp_d.p, soff.p, S.p, X, ldx, nb);
  c.launches++;
  FEM2D_CUDA(cudaGetLastError());
}

}  // namespace fem2d
