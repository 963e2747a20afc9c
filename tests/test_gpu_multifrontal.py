"""The device multifrontal LU of the shifted pencil: residuals of (c_a A + c_b B) X = R (FP64)."""
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


@pytest.mark.parametrize("name,ca,cb,spd", [("kat_b", 1.0, -1.475, False), ("kat_b", 1.0, 0.07, True),
                                            ("prec", 1.0, -10.0, False), ("prec", 0.0, 1.0, True),
                                            ("batch", 1.0, -10.0, False)])
def test_shifted_solve_residual(kat, ctx, name, ca, cb, spd):
    if name == "kat_b":
        mj, ops, basis, glq = kat["mesh_b"], [("pref", 3, 3, None), ("href", 0, None, -1),
                                              ("href", 0, [6, 9, 12], -1)], 0, (8, 8)
    elif name == "prec":
        w = configs.precision(seed=0, nx=6, ny=3)
        mj, ops, basis, glq = w.mesh_json, w.ops, w.basis, w.glq
    else:
        w = configs.batch_member(3)
        mj, ops, basis, glq = w.mesh_json, w.ops, w.basis, w.glq
    pm = fg.Mesh.from_json(mj)
    configs.apply_ops(pm, ops)
    gep = fg.galerkin_sample_gep_hcurl(fg.KOLeg if basis else fg.HierPoly, fg.CurlCurl, fg.L2Inner,
                                       fg.Domain.from_mesh(pm), list(glq), ctx=ctx)
    A, B = gep.scipy()
    K = ca * A + cb * B
    R = np.random.default_rng(0).standard_normal((gep.dimension, 5))
    X = gep.shifted_solve(ca, cb, R, spd=spd)
    rel = np.linalg.norm(K @ X - R, axis=0) / np.linalg.norm(R, axis=0)
    import scipy.sparse.linalg as sla

    Xs = sla.splu(K.tocsc()).solve(R)
    rels = np.linalg.norm(K @ Xs - R, axis=0) / np.linalg.norm(R, axis=0)
    assert np.max(rel) <= max(1e-9, 100 * np.max(rels)), (rel, rels)


@pytest.mark.parametrize("ca,cb,spd", [(1.0, -10.0, False), (1.0, 10.0, True)])
def test_shifted_solve_wide_fronts(ctx, ca, cb, spd):
    """A 389,566-DoF full-form mesh whose top separator fronts have p > 160: the narrow upper levels are
    solved through the fronts' partitioned inverses (the wide ones inverted column-parallel); the
    normwise backward error ||K X - R|| / (||K|| ||X|| + ||R||) stays at the FP64 level."""
    w = configs.full_scale(seed=0, basis=0, nx=64, ny=32, rounds=1, fraction=0.44)
    dom = fg.Domain.from_mesh(configs.build_mesh(w))
    fronts = fg.factor_plan(dom)["fronts"]
    assert np.max(fronts[:, 3]) > 160   # the case the wide inversion covers
    gep = fg.galerkin_sample_gep_hcurl(fg.HierPoly, fg.CurlCurl, fg.L2Inner, dom, list(w.glq), ctx=ctx)
    A, B = gep.scipy()
    K = (ca * A + cb * B).tocsr()
    R = np.random.default_rng(1).standard_normal((gep.dimension, 4))
    X = gep.shifted_solve(ca, cb, R, spd=spd)
    knorm = np.max(np.asarray(abs(K).sum(axis=1)).ravel())
    bwd = np.max(np.abs(K @ X - R), axis=0) / (knorm * np.max(np.abs(X), axis=0) + np.max(np.abs(R), axis=0))
    assert np.all(np.isfinite(X))
    assert np.max(bwd) < 1e-13, bwd


@pytest.mark.parametrize("columns", [1, 7, 8, 9, 16, 23, 32, 33])
@pytest.mark.parametrize("mesh", ["empty_level", "uneven", "leaves"])
def test_shifted_solve_columns(kat, ctx, mesh, columns):
    """Right-hand side counts around the tiles of 8 and the column splits, on trees with a level of fronts
    without pivots (kat_b), with fronts of many sizes on eleven levels, and with more leaf fronts than the
    tiled solve takes: the normwise backward error stays at the FP64 level (450 units of rounding)."""
    if mesh == "empty_level":
        pm = fg.Mesh.from_json(kat["mesh_b"])
        configs.apply_ops(pm, [("pref", 3, 3, None), ("href", 0, None, -1), ("href", 0, [6, 9, 12], -1)])
    elif mesh == "uneven":
        pm = configs.build_mesh(configs.full_scale(seed=5, nx=9, ny=5, rounds=3, fraction=0.4, pmin=2, pmax=7))
    else:
        pm = configs.build_mesh(configs.full_scale(seed=6, nx=23, ny=17, rounds=1, fraction=0.2, pmin=2, pmax=4))
    dom = fg.Domain.from_mesh(pm)
    fronts = fg.factor_plan(dom)["fronts"]
    levels = [fronts[fronts[:, 1] == k] for k in range(fronts[:, 1].max() + 1)]
    assert {"empty_level": min(q[:, 3].max() for q in levels) == 0, "uneven": len(levels) >= 8,
            "leaves": len(levels[0]) > 304}[mesh]
    gep = fg.galerkin_sample_gep_hcurl(fg.KOLeg, fg.CurlCurl, fg.L2Inner, dom, [10, 10], ctx=ctx)
    A, B = gep.scipy()
    for ca, cb, spd in ((1.0, -10.0, False), (1.0, 10.0, True)):
        K = (ca * A + cb * B).tocsr()
        R = np.random.default_rng(columns).standard_normal((gep.dimension, columns))
        X = gep.shifted_solve(ca, cb, R, spd=spd)
        knorm = np.max(np.asarray(abs(K).sum(axis=1)).ravel())
        bwd = np.max(np.abs(K @ X - R), axis=0) / (knorm * np.max(np.abs(X), axis=0) + np.max(np.abs(R), axis=0))
        assert np.max(bwd) < 1e-13, bwd


@pytest.mark.parametrize("orders", [(1, 2), (3, 3), (5, 4), (8, 7), (9, 9), (12, 10)])
@pytest.mark.parametrize("copies", [1, 90])
def test_factor_front_sizes(ctx, orders, copies):
    """Factorizations whose leaf fronts run from a few rows to more than a CTA's shared memory holds (two to
    several hundred rows, pivot counts that are and are not multiples of 8, up to p > 160), on levels
    narrower and wider than the chip: normwise backward errors at the FP64 level (450 units of rounding)."""
    nx, ny = (3, 2) if copies == 1 else (16, 12)
    if copies > 1 and orders[0] * orders[1] > 60:
        nx, ny = 13, 12
    pm = configs.build_mesh(configs.full_scale(seed=3, nx=nx, ny=ny, rounds=1, fraction=0.15, pmin=1, pmax=1))
    leaves = [int(e) for e in np.nonzero(pm.elem_info()[:, 0] == 1)[0]]
    pm.set_expansion_on_elems(leaves[::2], fg.Orders(*orders))
    pm.set_expansion_on_elems(leaves[1::2], fg.Orders(orders[0], max(1, orders[1] - 1)))
    gep = fg.galerkin_sample_gep_hcurl(fg.KOLeg, fg.CurlCurl, fg.L2Inner, fg.Domain.from_mesh(pm), [14, 14], ctx=ctx)
    A, B = gep.scipy()
    for ca, cb, spd in ((1.0, -10.0, False), (1.0, 10.0, True)):
        K = (ca * A + cb * B).tocsr()
        R = np.random.default_rng(7).standard_normal((gep.dimension, 3))
        X = gep.shifted_solve(ca, cb, R, spd=spd)
        knorm = np.max(np.asarray(abs(K).sum(axis=1)).ravel())
        bwd = np.max(np.abs(K @ X - R), axis=0) / (knorm * np.max(np.abs(X), axis=0) + np.max(np.abs(R), axis=0))
        assert np.max(bwd) < 1e-13, bwd


def test_eigensolve_after_shifted_solve(ctx):
    """A plan made by a shifted solve has one workspace; an eigensolve on it, which solves with two matrices at
    once, gives the eigenvalues of an eigensolve on a plan of its own."""
    w = configs.full_scale(seed=5, nx=9, ny=5, rounds=2, fraction=0.4, pmin=2, pmax=6)
    w.mesh_json = configs.grid_mesh_json(9, 5, 0.0, 1.87, 0.0, 1.0)
    dom = fg.Domain.from_mesh(configs.build_mesh(w))
    geps = [fg.galerkin_sample_gep_hcurl(fg.KOLeg, fg.CurlCurl, fg.L2Inner, dom, [10, 10], ctx=ctx) for _ in range(2)]
    geps[0].shifted_solve(1.0, -10.0, np.ones(dom.num_dofs))
    a, b = (fg.gpu_solve_gep_n(g, 10.0, 4).values for g in geps)
    assert np.max(np.abs(a - b) / b) < 1e-11
    x = geps[0].shifted_solve(1.0, -10.0, np.ones(dom.num_dofs))
    A, B = geps[0].scipy()
    assert np.linalg.norm((A - 10.0 * B) @ x - 1.0) <= 1e-9 * np.sqrt(dom.num_dofs)


def _backward_error(K, X, R):
    """Per column ||K X - R|| / (||K|| ||X|| + ||R||) in the infinity norm."""
    knorm = np.max(np.asarray(abs(K).sum(axis=1)).ravel())
    return np.max(np.abs(K @ X - R), axis=0) / (knorm * np.max(np.abs(X), axis=0) + np.max(np.abs(R), axis=0))


@pytest.mark.parametrize("spd", [False, True])
@pytest.mark.parametrize("pivots", [[9], [1, 7, 8, 9, 45], [160, 161, 199], [96, 200, 728], [101, 924], [768, 532],
                                    [769, 531], [103, 700, 700, 545], [96, 801, 1152], [801, 763, 736]],
                         ids=lambda p: "f%d_p%d" % (sum(p), p[0]))
def test_fronts_of_every_size(ctx, pivots, spd):
    """Unrefined solves with a dense matrix in chains of fronts: one front inverted whole, fronts in shared
    memory, fronts of up to 256, 1,024, 2,048 and more rows (a kernel each), pivot counts on both sides of 160 and
    768 (one CTA, tiled and cluster solves) that are and are not multiples of 8. Without spd the large entries
    stand off the diagonal of their front's pivot square, so that every column is pivoted. Normwise backward
    errors below n roundings."""
    n = sum(pivots)
    rng = np.random.default_rng(n + len(pivots))
    G = rng.standard_normal((n, n))
    if spd:
        K = G @ G.T / n + 0.1 * np.eye(n)
    else:
        K, first = G, 0
        for p in pivots:
            K[first + rng.permutation(p), first + np.arange(p)] += 4.0 * np.sqrt(n)
            first += p
    R = rng.standard_normal((n, 33))
    X = fg.fronts_solve(ctx, K, pivots, R, spd=spd)
    assert np.max(_backward_error(K, X, R)) <= n * 2.0 ** -53


@pytest.mark.parametrize("orders", [(1, 2), (3, 3), (5, 4), (8, 7), (9, 9), (12, 10)])
@pytest.mark.parametrize("copies", [1, 90])
def test_unrefined_solves(ctx, orders, copies):
    """The eigensolver's solves as it uses them, without refinement or a dense fallback, singly and in pairs, on the
    meshes of test_factor_front_sizes: the backward errors stay below the 1e-11 at which the eigensolver turns to
    another scaling or plan, and a pair of solves gives the two single ones bit for bit."""
    nx, ny = (3, 2) if copies == 1 else (16, 12)
    if copies > 1 and orders[0] * orders[1] > 60:
        nx, ny = 13, 12
    pm = configs.build_mesh(configs.full_scale(seed=3, nx=nx, ny=ny, rounds=1, fraction=0.15, pmin=1, pmax=1))
    leaves = [int(e) for e in np.nonzero(pm.elem_info()[:, 0] == 1)[0]]
    pm.set_expansion_on_elems(leaves[::2], fg.Orders(*orders))
    pm.set_expansion_on_elems(leaves[1::2], fg.Orders(orders[0], max(1, orders[1] - 1)))
    gep = fg.galerkin_sample_gep_hcurl(fg.KOLeg, fg.CurlCurl, fg.L2Inner, fg.Domain.from_mesh(pm), [14, 14], ctx=ctx)
    A, B = gep.scipy()
    R = np.random.default_rng(7).standard_normal((gep.dimension, 35))
    shifts = [(1.0, -10.0, False), (1.0, 10.0, True)]
    single = [gep.factor_solve([s], R)[0] for s in shifts]
    for (ca, cb, _), X in zip(shifts, single):
        assert np.max(_backward_error((ca * A + cb * B).tocsr(), X, R)) < 1e-11
    for X, Y in zip(single, gep.factor_solve(shifts, R)):
        assert np.array_equal(X, Y)
