"""The eigensolve on a full-form HierPoly mesh (monomial bases of orders 3..8, four refinement rounds).

HierPoly and KOLeg span the same discrete space on a mesh, so their Galerkin eigenvalues agree up to
rounding: the KOLeg pencil (well conditioned) is an independent check of the HierPoly pencil (cond(B)
orders of magnitude larger), whose attainable relative residual rises with ||A||. The domain is
[0,2]x[0,1] with PEC walls, whose Maxwell eigenvalues are (m pi / 2)^2 + (k pi)^2.
"""
import numpy as np
import pytest

import fem_2d_gb300 as fg
from fem_2d_gb300 import configs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from fem_2d_gb300 import build

    build.build()
    return fg.Context(0)


def _solve(ctx, basis, nx, ny):
    w = configs.full_scale(seed=0, nx=nx, ny=ny, rounds=4, fraction=0.3, basis=basis)
    d = fg.Domain.from_mesh(configs.build_mesh(w))
    g = fg.galerkin_sample_gep_hcurl(fg.KOLeg if basis else fg.HierPoly, fg.CurlCurl, fg.L2Inner, d, [10, 10],
                                     ctx=ctx)
    return g, fg.gpu_solve_gep_n(g, 10.0, 20)


def _analytic(k, target=10.0):
    ana = np.sort([(a * np.pi / 2) ** 2 + (b * np.pi) ** 2 for a in range(40) for b in range(20) if a + b > 0])
    return np.sort(ana[np.argsort(np.abs(ana - target), kind="stable")[:k]])


@pytest.mark.parametrize("nx,ny", [(16, 8), (32, 16)])
def test_hierpoly_matches_koleg(ctx, nx, ny):
    g, hp = _solve(ctx, 0, nx, ny)
    _, ko = _solve(ctx, 1, nx, ny)
    assert hp.stats["converged"] and ko.stats["converged"]
    assert hp.stats["block_scaled"] == 1
    assert hp.stats["max_backward_error"] < 1e-10
    vh, vk = np.sort(hp.values), np.sort(ko.values)
    assert np.max(np.abs(vh - vk) / vk) < 1e-10
    assert np.max(np.abs(vh - _analytic(20)) / _analytic(20)) < 1e-5
    # the eigenvectors: B-normalised, residuals recomputed on the host in the original pencil
    A, B = g.scipy()
    X = hp.vectors.T
    th = hp.values
    R = A @ X - (B @ X) * th
    rel = np.linalg.norm(R, axis=0) / (np.abs(th) * np.linalg.norm(B @ X, axis=0))
    assert np.allclose(rel, hp.residuals, rtol=1e-3, atol=1e-14)
    assert np.allclose(np.einsum("ij,ij->j", X, B @ X), 1.0, atol=1e-8)


def test_hierpoly_repeat_solve_is_stable(ctx):
    g, first = _solve(ctx, 0, 16, 8)
    again = fg.gpu_solve_gep_n(g, 10.0, 20)
    assert again.stats["converged"]
    assert np.allclose(np.sort(first.values), np.sort(again.values), rtol=1e-11, atol=0)


def test_scaling_and_damping_options_agree(ctx):
    """Jacobi and row-run block scaling, and the two damping regimes, reach the same eigenvalues."""
    w = configs.precision(seed=1, nx=8, ny=4)
    d = fg.Domain.from_mesh(configs.build_mesh(w))
    g = fg.galerkin_sample_gep_hcurl(fg.KOLeg, fg.CurlCurl, fg.L2Inner, d, [10, 10], ctx=ctx)
    runs = [fg.gpu_solve_gep_n(g, 10.0, 6, scaling=sc, damping=dm) for sc in (1, 2) for dm in (0.05, 1.0)]
    ref = np.sort(runs[0].values)
    for r in runs:
        assert r.stats["converged"]
        assert np.allclose(np.sort(r.values), ref, rtol=1e-11, atol=0)
    assert [r.stats["block_scaled"] for r in runs] == [0, 0, 1, 1]


@pytest.mark.parametrize("orders", [(1, 1), (2, 3), (4, 4), (6, 5), (8, 8)])
def test_block_scaling_run_lengths(ctx, oracle_lib, orders):
    """Block scaling over runs from one row to 64, short and long in one mesh and column runs that do and do
    not fill tiles of 8: the eigenvalues are those of LAPACK on the unscaled pencil."""
    pm = configs.build_mesh(configs.full_scale(seed=2, nx=3, ny=2, rounds=1, fraction=0.5, pmin=1, pmax=2))
    leaves = [int(e) for e in np.nonzero(pm.elem_info()[:, 0] == 1)[0]]
    pm.set_expansion_on_elems(leaves[:max(1, len(leaves) // 2)], fg.Orders(*orders))
    gep = fg.galerkin_sample_gep_hcurl(fg.KOLeg, fg.CurlCurl, fg.L2Inner, fg.Domain.from_mesh(pm), [10, 10], ctx=ctx)
    A, B = gep.scipy()
    ref, _ = oracle_lib.dense_nearest_physical(A, B, 5.0, 1)
    r = fg.gpu_solve_gep_n(gep, 5.0, 1, scaling=2)
    assert r.stats["block_scaled"] == 1
    assert abs(r.values[0] - ref[0]) <= 1e-9 * abs(ref[0])


def _exact_vector(A, B, value, start):
    """The eigenvector at ``value`` by inverse iteration, its systems refined with long double residuals."""
    import scipy.sparse as sp
    import scipy.sparse.linalg as sla

    L = np.longdouble
    rp, col = A.indptr[:-1], A.indices
    mul = lambda v, x: np.add.reduceat(v * x[col], rp)
    a, b, d = A.data.astype(L), B.data.astype(L), (1.0 / np.sqrt(B.diagonal()))
    shift = value * (1.0 + 1e-4)
    S = sp.diags(d)
    lu = sla.splu((S @ (A - shift * B) @ S).tocsc())
    x, d = start / d, d.astype(L)
    for _ in range(3):   # (each step gains the factor gap / 1e-4 value)
        rhs = d * mul(b, d * x)
        y, r = np.zeros_like(rhs), rhs
        for _ in range(6):
            y = y + lu.solve(r.astype(np.float64))
            r = rhs - d * (mul(a, d * y) - L(shift) * mul(b, d * y))
        assert np.max(np.abs(r)) <= 1e-15 * np.max(np.abs(rhs))
        x = y / np.sqrt((d * y) @ mul(b, d * y))
    return (d * x).astype(np.float64)


@pytest.mark.parametrize("nx,ny,side", [(14, 9, 1.87), (14, 9, 2.13), (20, 9, 1.87)])
def test_products_and_solves_round_alike(ctx, nx, ny, side):
    """The block-scaled pencil is symmetric up to rounding only, and one order of its two products keeps the
    eigenvectors of a monomial basis several times better than the other. Products and factorizations both see
    the better one: the vectors of refined solves, which the products decide, and of unrefined ones, which the
    factorization does, are equally far from the exact vectors of the assembled pencil (at most twice)."""
    w = configs.full_scale(seed=0, nx=nx, ny=ny, rounds=2, fraction=0.35, pmin=2, pmax=8)
    w.mesh_json = configs.grid_mesh_json(nx, ny, 0.0, side, 0.0, 1.0)
    gep = fg.galerkin_sample_gep_hcurl(fg.HierPoly, fg.CurlCurl, fg.L2Inner,
                                       fg.Domain.from_mesh(configs.build_mesh(w)), [10, 10], ctx=ctx)
    assert gep.dimension >= 10000
    A, B = gep.scipy()
    runs = [fg.gpu_solve_gep_n(gep, 10.0, 3, refine=k, dense=1) for k in (-1, 2)]
    err = np.zeros((2, 3))
    for q in range(3):
        exact = _exact_vector(A, B, runs[0].values[q], runs[0].vectors[q])
        for k, r in enumerate(runs):
            v = r.vectors[q] * np.sign(r.vectors[q] @ exact)
            err[k, q] = np.max(np.abs(v - exact)) / np.max(np.abs(exact))
    err = np.max(err, axis=1)
    assert np.max(err) <= 2.0 * np.min(err), err
