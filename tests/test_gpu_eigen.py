"""Device eigensolvers against the reference's known answers and the FP64 oracles.

* nalgebra_solve_gep restated on the device: mesh_a -> 2.6479657 (1e-6, src/lib.rs:65) and agreement
  with the oracle's restatement to 1e-9 relative.
* gpu_solve_gep: mesh_b nearest 1.475 -> test_input/test_eval.dat to 1e-9 relative (src/lib.rs:104), the
  eigenvector against test_input/test_evec.dat (both B-normalised, up to sign), and k pairs against the
  LAPACK / sparse FP64 oracles with eigenvalue relative error <= 1e-9.
"""
import numpy as np
import pytest

import fem_2d_gb300 as fg
from fem_2d_gb300 import configs

pytestmark = pytest.mark.gpu
EIG_TOL = 1e-9


@pytest.fixture(scope="module")
def ctx():
    from fem_2d_gb300 import build

    build.build()
    return fg.Context(0)


def _gep(mesh_json, ops, basis, glq, ctx):
    pm = fg.Mesh.from_json(mesh_json)
    configs.apply_ops(pm, ops)
    dom = fg.Domain.from_mesh(pm)
    bs = fg.KOLeg if basis == 1 else fg.HierPoly
    return fg.galerkin_sample_gep_hcurl(bs, fg.CurlCurl, fg.L2Inner, dom, list(glq), ctx=ctx)


def test_dense_solve_kat_nalg_problem(oracle_lib, kat, ctx):
    gep = _gep(kat["mesh_a"], [("pref", 2, 2, None)], 0, (8, 8), ctx)
    pair = fg.nalgebra_solve_gep(gep, 2.64)
    assert abs(pair.value - 2.6479657) < 1e-6
    A, B = gep.scipy()
    val, vec = oracle_lib.reference_dense_solve(A, B, 2.64)
    assert abs(pair.value - val) <= 1e-9 * abs(val)
    assert len(pair.vector) == gep.dimension
    assert abs(abs(pair.vector @ vec) - 1.0) < 1e-6


def test_dense_solve_waveguide(oracle_lib, ctx):
    w = configs.waveguide_small()
    gep = _gep(w.mesh_json, w.ops, w.basis, w.glq, ctx)
    pair = fg.nalgebra_solve_gep(gep, w.target)
    A, B = gep.scipy()
    val, _ = oracle_lib.reference_dense_solve(A, B, w.target)
    assert abs(pair.value - val) <= 1e-9 * abs(val)


def test_dense_solve_too_large(ctx):
    w = configs.precision(seed=0, nx=4, ny=2)
    gep = _gep(w.mesh_json, w.ops, w.basis, w.glq, ctx)
    assert gep.dimension > 1000
    with pytest.raises(fg.Fem2dError) as e:
        fg.nalgebra_solve_gep(gep, 10.0)
    assert e.value.code == fg.E_TOO_LARGE


def test_gpu_solve_kat_slepc_problem(kat, ctx):
    ops = [("pref", 3, 3, None), ("href", 0, None, -1), ("href", 0, [6, 9, 12], -1)]
    gep = _gep(kat["mesh_b"], ops, 0, (8, 8), ctx)
    pair = fg.gpu_solve_gep(gep, 1.475)
    assert abs(pair.value - kat["slepc_eval"]) <= EIG_TOL * kat["slepc_eval"]
    assert abs(pair.value - 1.4745880937) < 1e-9
    g = np.asarray(kat["slepc_evec"])
    x = pair.vector * np.sign(pair.vector @ g)
    assert np.max(np.abs(x - g)) < 1e-7
    assert pair.residual < 1e-9


@pytest.mark.parametrize("seed,k,dense", [(0, 6, 0), (2, 10, 0), (2, 10, 2)])
def test_gpu_solve_against_lapack(oracle_lib, ctx, seed, k, dense):
    """dense = 2 runs every contraction on the tensor cores at this small size (the default keeps the
    FP64 kernels below 50,000 DoFs)."""
    ref = oracle_lib
    w = configs.precision(seed=seed, nx=4, ny=2)
    gep = _gep(w.mesh_json, w.ops, w.basis, w.glq, ctx)
    res = fg.gpu_solve_gep_n(gep, w.target, k, dense=dense)
    A, B = gep.scipy()
    wd, vd = ref.dense_nearest_physical(A, B, w.target, k)
    assert np.max(np.abs(res.values - wd) / np.abs(wd)) <= EIG_TOL
    assert np.max(res.residuals) < 1e-9
    # B-orthonormal eigenvectors
    G = res.vectors @ (B @ res.vectors.T)
    assert np.max(np.abs(G - np.eye(k))) < 1e-8


def test_gpu_solve_batch_member(oracle_lib, ctx):
    ref = oracle_lib
    w = configs.batch_member(4)
    gep = _gep(w.mesh_json, w.ops, w.basis, w.glq, ctx)
    res = fg.gpu_solve_gep_n(gep, w.target, w.n_pairs)
    A, B = gep.scipy()
    wd, _ = ref.dense_nearest_physical(A, B, w.target, w.n_pairs)
    assert np.max(np.abs(res.values - wd) / np.abs(wd)) <= EIG_TOL


def test_gpu_solve_precision_config(oracle_lib, ctx):
    """The full precision workload (16x8 Elems, KOLeg, ~29k DoFs) against the sparse FP64 oracle."""
    ref = oracle_lib
    w = configs.precision(seed=0)
    gep = _gep(w.mesh_json, w.ops, w.basis, w.glq, ctx)
    res = fg.gpu_solve_gep_n(gep, w.target, w.n_pairs)
    A, B = gep.scipy()
    ws, _, rs = ref.sparse_nearest_physical(A, B, w.target, w.n_pairs)
    assert np.max(np.abs(res.values - ws) / np.abs(ws)) <= EIG_TOL
    assert np.max(res.residuals) < 1e-9


@pytest.mark.parametrize("target,k", [(10.0, 6), (2.6, 1), (30.0, 4), (-3.0, 3)])
@pytest.mark.parametrize("opts", [{}, {"refine": 2}, {"damping": 0.05}, {"damping": 1.0}, {"damping": 4.0, "refine": -1}])
def test_targets_and_dampings(oracle_lib, ctx, target, k, opts):
    """The search operator in both forms: partial fractions (targets above zero), with and without
    refinement and with dampings around |target|, and the product form (below zero, where with a damping of
    one the two shifted matrices coincide)."""
    w = configs.full_scale(seed=4, nx=5, ny=3, rounds=2, fraction=0.4, pmin=3, pmax=5, basis=1)
    w.mesh_json = configs.grid_mesh_json(5, 3, 0.0, 1.87, 0.0, 1.0)
    gep = _gep(w.mesh_json, w.ops, 1, w.glq, ctx)
    A, B = gep.scipy()
    ref, _ = oracle_lib.dense_nearest_physical(A, B, target, k)
    r = fg.gpu_solve_gep_n(gep, target, k, **opts)
    assert np.max(np.abs(r.values - ref) / np.abs(ref)) <= EIG_TOL
    assert np.all(np.abs(np.einsum("ij,ij->i", r.vectors, (B @ r.vectors.T).T) - 1.0) < 1e-9)


@pytest.mark.parametrize("dense", [1, 2])
@pytest.mark.parametrize("nx,ny,rounds,k", [(2, 2, 0, 1), (4, 3, 1, 3), (6, 5, 1, 12)])
def test_block_updates_of_several_operands(oracle_lib, ctx, nx, ny, rounds, k, dense):
    """Updates of one, two and three blocks at once, with the FP64 and the tensor kernels, from GEPs of less
    than one tile of 128 rows to several with a ragged last one, with locked and compressed columns."""
    w = configs.full_scale(seed=nx, nx=nx, ny=ny, rounds=rounds, fraction=0.4, pmin=3, pmax=4, basis=1)
    w.mesh_json = configs.grid_mesh_json(nx, ny, 0.0, 1.87, 0.0, 1.0)
    gep = _gep(w.mesh_json, w.ops, 1, w.glq, ctx)
    A, B = gep.scipy()
    ref, _ = oracle_lib.dense_nearest_physical(A, B, 2.64, k)
    r = fg.gpu_solve_gep_n(gep, 2.64, k, dense=dense)
    assert np.max(np.abs(r.values - ref) / np.abs(ref)) <= EIG_TOL
    assert np.all(np.abs(np.einsum("ij,ij->i", r.vectors, (B @ r.vectors.T).T) - 1.0) < 1e-9)


@pytest.mark.parametrize("nx,ny,p,rounds", [(2, 1, 2, 0), (2, 1, 4, 1), (3, 2, 3, 1), (7, 6, 2, 1), (9, 7, 2, 2),
                                            (6, 4, 4, 0)])
def test_dense_solve_tree_shapes(oracle_lib, ctx, nx, ny, p, rounds):
    """The dense solve on trees of one to several levels, with few fronts (partitioned inverses) and with more
    than the chip's SMs take row by row: the mode nearest the target of the same lower triangle, to rounding
    (n 2^-53 cond(B), below 1e-10 for orders up to 4), and its vector up to the sign."""
    w = configs.full_scale(seed=nx + p, nx=nx, ny=ny, rounds=rounds, fraction=0.3, pmin=p, pmax=p, basis=0)
    w.mesh_json = configs.grid_mesh_json(nx, ny, 0.0, 1.87, 0.0, 1.0)
    gep = _gep(w.mesh_json, w.ops, 0, [8, 8], ctx)
    assert gep.dimension <= 1000
    A, B = (m.toarray() for m in gep.scipy())
    S = np.linalg.solve(B, A)
    val, vec = np.linalg.eigh(np.tril(S) + np.tril(S, -1).T)
    best = np.argmin(np.abs(val - 10.0))
    pair = fg.nalgebra_solve_gep(gep, 10.0)
    assert abs(pair.value - val[best]) <= 1e-10 * np.max(np.abs(val))
    gap = np.min(np.abs(np.delete(val, best) - val[best]))
    assert 1.0 - abs(vec[:, best] @ pair.vector) <= (1e-10 * np.max(np.abs(val)) / gap) ** 2 + 1e-12
