// Device side of the multifrontal factorization (mf.cu).
#pragma once
#include <cstring>
#include <memory>
#include <mutex>
#include <vector>

#include "blockscale.h"
#include "device.h"
#include "mf.h"
#include "ozaki.h"

namespace fem2d {

// One numeric factorization: dense fronts and their row pivots.
struct MFFactor {
  DBuf<double> F;
  DBuf<int32_t> piv;
  DBuf<int32_t> perm;    // gather permutation equivalent to the row swaps
  DBuf<int32_t> iperm;   // its inverse
  int flags = 0;   // 1: a zero pivot was perturbed, 2: a non-positive pivot in Cholesky mode
  std::vector<int32_t> weak;   // DoFs whose columns had no stable pivot among their front's fully-summed rows
  // dense single-front plans (small GEPs): F holds the explicit inverse K^-1 (n x n) instead of LU
  // factors (Gauss-Jordan, partial pivoting); solves are then one dense product
  int64_t inv_n = 0;
};

struct MFDevice {
  int nf = 0, nlevels = 0, max_f = 0, max_p = 0, nb_cap = 0;
  int64_t mat_total = 0, piv_total = 0;
  double factor_flops = 0;   // LU flops of all fronts, 2/3 (f^3 - (f - p)^3) each (half for Cholesky)
  std::vector<int32_t> level_ptr, level_max_f, level_max_p;
  std::vector<int64_t> level_off;
  std::vector<int64_t> level_big_end;   // end of the storage of a level's fronts factored in global memory
  std::vector<double> level_factor_bytes;   // L (forward) or U (backward) bytes read per level
  DArena arena;   // holds all of the buffers below
  DBuf<uint8_t> desc;
  DBuf<int32_t> lfronts, dofs, ea_map;
  DBuf<int64_t> asm_pos, asm_csr, piv_off, woff;
  DBuf<double> work, work2;   // workspaces; the second for pairs of solves, where the plan makes them
  DBuf<int> flags;
  DBuf<int32_t> weak_list;   // capacity n: weak-pivot DoFs recorded by the factorization
  DBuf<int> weak_count;
  // per level, the fronts solved by one CTA each (inverted diagonal blocks) and the rest (clusters)
  std::vector<int32_t> small_ptr, large_ptr;   // nlevels + 1 offsets into lsmall / llarge
  std::vector<int32_t> level_fwd_cols, level_bwd_cols;   // shared doubles per right-hand side of their kernels
  DBuf<int32_t> lsmall, llarge;
  // factorization: per level the fronts factored in global memory (lbig), and the groups of fronts factored
  // by one CTA each in shared memory (lfused)
  struct FusedGroup {
    int level, first, count, max_f;
  };
  std::vector<FusedGroup> fused_groups;
  std::vector<int32_t> big_ptr, level_big_f, level_big_p;
  DBuf<int32_t> lbig, lfused;
  // tiled levels (narrow upper levels solved through the fronts' partitioned inverses, rows spread over
  // many CTAs): per level a flag and offsets into the (front, first row) items of each direction
  std::vector<uint8_t> level_tiled;
  std::vector<int32_t> tf_ptr, tb_ptr;
  DBuf<int32_t> tf_items, tb_items;
  DBuf<int32_t> pull;   // pull records of the tiled fronts' right-hand sides (8 per row)
  std::vector<int32_t> level_pmax, level_kmax;   // tiled levels: longest sums of the two directions
  // inverses of the fronts factored in global memory: the fronts, their (front, L or U, column strip) items and
  // scratch squares, then the partitioned-inverse items of those on tiled levels
  DBuf<int32_t> linv, inv_items, pinv_items;
  DBuf<double> sq;
  int ninv = 0, ninv_items = 0, max_inv_p = 0, npinv = 0;

  // pairs: solve_pair will be called (else its first call gets the second workspace, as large as the first)
  void setup(Ctx& c, const MFSymbolic& s, int nb_max, bool pairs);
  // factor c_a*A + c_b*B (values in full-CSR order); Cholesky mode skips pivoting (SPD shifts)
  void factor(Ctx& c, const double* va, const double* vb, double ca, double cb, bool cholesky, MFFactor& out);
  // X = K^-1 B for an n x nb row-major block (nb <= nb_cap); B and X must not alias
  void solve(Ctx& c, const MFFactor& fac, const double* B, int64_t ldb, double* X, int64_t ldx, int nb);
  // X1 = K1^-1 B and X2 = K2^-1 B in one pass over the levels (B may alias neither)
  void solve_pair(Ctx& c, const MFFactor& f1, const MFFactor& f2, const double* B, int64_t ldb, double* X1, int64_t ldx1,
                  double* X2, int64_t ldx2, int nb);
  int read_flags(Ctx& c);
  // X = K^-1 B for all n columns of B (row-major, ld n; X likewise) and K = A's or B's SPD values, every sum in
  // the fixed order of plain loops over each front (see mf_ordered_factor_kernel); false when a front is too
  // large for them. Returns the flags of factor() in *flags_out.
  bool solve_ordered(Ctx& c, const double* vals, int64_t n, const double* B, double* X, int* flags_out);

 private:
  void solve_sets(Ctx& c, int sets, const MFFactor* f1, const MFFactor* f2, const double* B, int64_t ldb, double* X1,
                  int64_t ldx1, double* X2, int64_t ldx2, int nb);
};

// The factorization plan of one GEP: the host symbolic phase and its device copy depend on the
// sparsity pattern only, so they are built on the first solve of a GEP and reused by later solves of
// the same GEP (numeric factorizations are always recomputed). mu serialises solves that share the
// plan's solve workspace.
struct MFPlan {
  std::unique_ptr<MFSymbolic> sym;
  std::unique_ptr<MFDevice> mf;
  bool ready = false;
  bool dense = false;   // a single dense front (chosen when the sparse plan's solves are inaccurate)
  std::vector<uint8_t> lift;   // per DoF: levels its elimination was moved up (delayed pivots)
  int device = -1;
  // pattern-only structures of the eigensolver, built on first use on the plan's device: the row-run
  // block scaling's blocks and segments, the tensor-core operator products' items (their values are
  // recomputed, and the pencil re-sliced, by every solve)
  std::unique_ptr<BlockScale> bsc;
  std::unique_ptr<TcSpmm> tcs;
  int aux_device = -1;
  std::mutex mu;
};

// the plan's MFDevice, building the plan on first use (or after a device change); `pre`, when given, is
// the sparse symbolic analysis already computed for this GEP
MFDevice& mf_plan(MFPlan& p, Ctx& c, const Domain& dom, const HostGEP& h, bool pairs,
                  std::unique_ptr<MFSymbolic> pre = nullptr);
// replace the plan by the dense single-front plan
MFDevice& mf_plan_dense(MFPlan& p, Ctx& c, const HostGEP& h);

}  // namespace fem2d
