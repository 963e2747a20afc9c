"""The work a program has this package do: dense, sparse and batched eigensolves, assembly, shifted
solves, operator products and field evaluation on refinement-by-superposition meshes.

Every case is a dict of plain values. Its mesh is nx x ny base Elems on [0, a] x [0, 1], expansion orders
uniform in pmin..pmax per Elem and direction, and ``rounds`` rounds of T/U/V refinement of ``fraction`` of
the leaves (the package's full-form, precision and batching families). The case fixes the orders and the
refinement; the geometry (the side a and the grid lines) comes from the seed. a is chosen so that the
wanted eigenvalues are simple: eigenvectors are then determined up to their sign, which the solver fixes.
"""
import ctypes
import math

import numpy as np
import torch

import fem_2d_gb300 as fg
from fem_2d_gb300 import configs

TARGET = 10.0
_BASIS = {"hierpoly": fg.HierPoly, "koleg": fg.KOLeg}


def _mesh(nx, ny, pmin, pmax, rounds, fraction):
    return {"nx": nx, "ny": ny, "pmin": pmin, "pmax": pmax, "rounds": rounds, "fraction": fraction}


def listed():
    return [
        # the reference's own smallest use: one mesh, one mode, the dense solve of its nalgebra path
        {"name": "dense_150", "do": "dense", "basis": "hierpoly", "glq": 8, **_mesh(3, 2, 3, 3, 1, 0.4)},
        # one small mesh from its Domain to one mode (the documentation's example sizes)
        {"name": "whole_600", "do": "whole", "basis": "hierpoly", "glq": 8, "pairs": 1, **_mesh(4, 4, 4, 4, 1, 0.4)},
        # a parameter sweep: many small meshes assembled in one launch and solved side by side
        {"name": "batch_24", "do": "batch", "basis": "koleg", "glq": 10, "pairs": 4, "meshes": 24,
         **_mesh(6, 4, 2, 8, 1, 0.3)},
        # a mesh of an adaptive loop, assembled and solved once, mixed orders, odd sizes
        {"name": "whole_7k", "do": "whole", "basis": "koleg", "glq": 10, "pairs": 4, **_mesh(11, 5, 2, 8, 2, 0.3)},
        # the precision workload: assembly and solve on a kept plan
        {"name": "step_29k", "do": "step", "basis": "koleg", "glq": 10, "pairs": 10, "vectors": True,
         **_mesh(16, 8, 6, 6, 3, 0.3)},
        # the same at the size from which the solver's contractions run on the tensor cores
        {"name": "step_83k", "do": "step", "basis": "koleg", "glq": 10, "pairs": 16, "vectors": True,
         **_mesh(32, 16, 5, 7, 2, 0.3)},
        # the full form at about a million DoFs
        {"name": "step_1m", "do": "step", "basis": "koleg", "glq": 10, "pairs": 20, "vectors": False,
         **_mesh(64, 32, 3, 8, 4, 0.44)},
        # the matrices themselves, for a solver on the host
        {"name": "assemble_70k", "do": "assemble", "basis": "hierpoly", "glq": 10, **_mesh(16, 8, 3, 8, 4, 0.44)},
        # new values of A and B into the caller's own device arrays
        {"name": "values_1m", "do": "values", "basis": "hierpoly", "glq": 10, **_mesh(64, 32, 3, 8, 4, 0.44)},
        # one right-hand side block of a caller's own shift-invert iteration
        {"name": "shifted_29k", "do": "shifted", "basis": "koleg", "glq": 10, "columns": 9, **_mesh(16, 8, 6, 6, 3, 0.3)},
        # operator products of a caller's own iteration
        {"name": "spmm_160k", "do": "spmm", "basis": "hierpoly", "glq": 10, "columns": 20,
         **_mesh(24, 13, 3, 8, 4, 0.44)},
        # E_x and E_y of one mode on a grid per leaf, for plotting
        {"name": "fields_70k", "do": "fields", "basis": "hierpoly", "glq": 10, "grid_u": 16, "grid_v": 15,
         **_mesh(16, 8, 3, 8, 4, 0.44)},
    ]


def draw(rng):
    do = rng.choice(["dense", "whole", "whole", "batch", "step", "step", "step", "assemble", "values", "shifted", "spmm",
                     "fields"])
    basis = rng.choice(["hierpoly", "koleg"])

    def size(lo, hi):
        """nx, ny with nx * ny spread over lo..hi on a log scale."""
        n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        r = rng.uniform(1.0, 2.2)
        return max(1, round(math.sqrt(n * r))), max(1, round(math.sqrt(n / r)))

    if do == "dense":
        p = rng.randint(2, 4)
        nx, ny = size(2, 9)
        return {"do": do, "basis": "hierpoly", "glq": 8, **_mesh(nx, ny, p, p, rng.randint(0, 1), 0.3)}
    if do == "batch":
        nx, ny = size(6, 40)
        return {"do": do, "basis": "koleg", "glq": 10, "pairs": rng.randint(1, 4), "meshes": rng.randint(2, 30),
                **_mesh(nx, ny, 2, rng.randint(4, 8), rng.randint(0, 2), 0.3)}
    if do == "whole":
        nx, ny = size(8, 300)
        small = nx * ny < 40
        pmin = rng.randint(2, 4)
        return {"do": do, "basis": "hierpoly" if small else "koleg", "glq": 8 if small else 10,
                "pairs": rng.randint(1, 4 if small else 12),
                **_mesh(nx, ny, pmin, 4 if small else rng.randint(max(4, pmin), 8), rng.randint(0, 2), 0.3)}
    if do == "step":
        if rng.random() < 0.5:
            nx, ny = size(60, 500)
            pmin = rng.randint(3, 6)
            return {"do": do, "basis": "koleg", "glq": 10, "pairs": rng.randint(5, 20), "vectors": True,
                    **_mesh(nx, ny, pmin, rng.randint(max(pmin, 5), 7), rng.randint(1, 2), round(rng.uniform(0.2, 0.35), 2))}
        nx, ny = size(120, 1900)
        return {"do": do, "basis": "koleg", "glq": 10, "pairs": rng.randint(10, 20), "vectors": False,
                **_mesh(nx, ny, 3, rng.randint(6, 8), rng.randint(3, 4), round(rng.uniform(0.3, 0.44), 2))}
    nx, ny = size(12, 1800 if do == "values" else 400)
    m = _mesh(nx, ny, rng.randint(2, 4), rng.randint(5, 8), rng.randint(1, 4), round(rng.uniform(0.2, 0.44), 2))
    case = {"do": do, "basis": "koleg" if do == "shifted" else basis, "glq": 10, **m}
    if do in ("shifted", "spmm"):
        case["columns"] = rng.randint(1, 32)
    if do == "fields":
        case["grid_u"], case["grid_v"] = rng.randint(3, 24), rng.randint(3, 24)
    return case


# ----------------------------------------------------------------------------------------- inputs
def _side(seed, pairs):
    """A side a such that the ``pairs`` eigenvalues pi^2 (m^2 / a^2 + n^2) nearest the target are simple,
    and neither their order nor the last of them is in doubt."""
    rng = configs.SplitMix64(seed + 77)
    best, found = -1.0, 2.1
    m, n = np.meshgrid(np.arange(40.0), np.arange(12.0))
    for _ in range(100):
        a = 1.7 + 0.9 * rng.uniform()
        lam = np.sort((math.pi ** 2 * ((m / a) ** 2 + n ** 2)).ravel())[1:pairs + 12]
        gap = np.minimum(np.diff(lam, prepend=0.0), np.diff(lam, append=1e3))
        dist = np.abs(lam - TARGET)
        near = np.argsort(dist)[:pairs + 1]
        score = min(float(gap[near].min()), 4.0 * float(np.diff(dist[near]).min()))
        if score > best:
            best, found = score, a
    return found


def _domain(case, seed, pairs=1, member=0):
    """The mesh and its Domain (host); ``member`` picks another set of orders and refinements."""
    w = configs.full_scale(seed=member, nx=case["nx"], ny=case["ny"], rounds=case["rounds"], fraction=case["fraction"],
                           pmin=case["pmin"], pmax=case["pmax"])
    w.mesh_json = configs.grid_mesh_json(case["nx"], case["ny"], 0.0, _side(seed, pairs), 0.0, 1.0)
    # grid lines moved by up to a tenth of their distance: no mode has two equal largest coefficients
    rng = np.random.default_rng(seed)
    move = [rng.uniform(-0.1, 0.1, k + 1) / k for k in (case["nx"], case["ny"])]
    for k, node in enumerate(w.mesh_json["Nodes"]):
        i, j = k % (case["nx"] + 1), k // (case["nx"] + 1)
        if 0 < i < case["nx"]:
            node[0] += move[0][i]
        if 0 < j < case["ny"]:
            node[1] += move[1][j]
    mesh = configs.build_mesh(w)
    return mesh, fg.Domain.from_mesh(mesh)


def _sample(case, domain):
    return fg.galerkin_sample_gep_hcurl(_BASIS[case["basis"]], fg.CurlCurl, fg.L2Inner, domain,
                                        [case["glq"], case["glq"]])


def prepare(case, seed):
    do = case["do"]
    s = {"case": case}
    if do == "batch":
        s["domains"] = [_domain(case, 1000 * seed + k, case["pairs"], k)[1] for k in range(case["meshes"])]
        return s
    s["mesh"], s["domain"] = _domain(case, seed, case.get("pairs", 1))
    n = s["domain"].num_dofs
    rng = np.random.default_rng(seed)
    if do in ("step", "values", "shifted", "spmm"):
        s["gep"] = _sample(case, s["domain"])
    if do == "values":
        nnz = s["gep"].dims()[2]
        s["a"] = torch.empty(nnz, dtype=torch.float64, device="cuda")
        s["b"] = torch.empty(nnz, dtype=torch.float64, device="cuda")
    if do == "shifted":
        s["rhs"] = rng.standard_normal((n, case["columns"]))
    if do == "spmm":
        s["x"] = torch.from_numpy(rng.standard_normal((n, case["columns"]))).cuda()
        s["y"] = torch.empty_like(s["x"])
    if do == "fields":
        s["space"] = fg.UniformFieldSpace(s["domain"], (case["grid_u"], case["grid_v"]))
        s["plan"] = s["space"]._device(_BASIS[case["basis"]])
        # a mode's coefficients fall with the order of the function
        spec = s["domain"].basis_specs()
        coef = np.zeros(n)
        coef[spec[:, 5]] = 2.0 ** -(spec[:, 2] + spec[:, 3])
        s["u"] = torch.from_numpy(coef * rng.standard_normal(n)).cuda()
        shape = (s["plan"].num_leaves, case["grid_u"], case["grid_v"])
        s["x"] = torch.empty(shape, dtype=torch.float64, device="cuda")
        s["y"] = torch.empty(shape, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------------------------------- runs
def run(s):
    case = s["case"]
    do = case["do"]
    if do == "dense":
        pair = fg.nalgebra_solve_gep(_sample(case, s["domain"]), TARGET)
        return {"value": pair.value, "vector": pair.vector}
    if do == "whole":
        r = fg.gpu_solve_gep_n(_sample(case, s["domain"]), TARGET, case["pairs"])
        return {"values": r.values, "vectors": r.vectors}
    if do == "step":
        s["gep"].recompute()
        r = fg.gpu_solve_gep_n(s["gep"], TARGET, case["pairs"])
        # a pair is accepted at the backward error that its pencil allows. From some 100k DoFs of mixed
        # orders that settles a vector to about 1e-8 (its eigenvalue to 1e-13), so the vectors there,
        # although computed and downloaded all the same, are not a value to compare
        return {"values": r.values, "vectors": r.vectors} if case["vectors"] else {"values": r.values}
    if do == "batch":
        geps, _ = fg.galerkin_sample_gep_hcurl_batch(_BASIS[case["basis"]], fg.CurlCurl, fg.L2Inner, s["domains"],
                                                     [case["glq"], case["glq"]])
        out = fg.gpu_solve_gep_batch(geps, TARGET, case["pairs"])
        return {"values": [r.values for r in out], "vectors": [r.vectors for r in out]}
    if do == "assemble":
        r, c, a, b = _sample(case, s["domain"]).upper_coo()
        return {"rows": r, "cols": c, "a": a, "b": b}
    if do == "shifted":
        return s["gep"].shifted_solve(1.0, -TARGET, s["rhs"])
    gep = s.get("gep")
    if do == "values":
        fg._check(fg.lib().fem2d_gep_values_noalloc(gep.ctx._h, gep._h, ctypes.c_void_p(s["a"].data_ptr()),
                                                    ctypes.c_void_p(s["b"].data_ptr())))
        return {"a": s["a"], "b": s["b"]}
    if do == "spmm":
        k = case["columns"]
        gep.spmm_device(1.0, -TARGET, s["x"].data_ptr(), k, k, s["y"].data_ptr(), k)
        return s["y"]
    s["plan"].xy_device(s["u"].data_ptr(), s["u"].numel(), s["x"].data_ptr(), s["y"].data_ptr())
    return {"x": s["x"], "y": s["y"]}


# ------------------------------------------------------------------------------------------- work
def work(case):
    """Bytes: the pencil's upper triangles (value pairs) once where the path reads or writes them, and its
    other inputs and outputs once. Flops: the products that the path is defined by."""
    do = case["do"]
    if do == "batch":
        one = work({**case, "do": "whole"})
        return {k: v * case["meshes"] for k, v in one.items()}
    mesh, dom = _domain(case, 1, case.get("pairs", 1))
    n = dom.num_dofs
    upper = len(fg.domain_pattern(dom)[0])
    full = 2 * upper - n
    if do == "dense":
        return {"bytes": 16.0 * upper + 8.0 * n, "flops": 4.0 / 3.0 * n ** 3}
    if do in ("whole", "step"):
        # A and B formed once and read once, the vectors written; one product with each per vector
        return {"bytes": 32.0 * upper + 8.0 * n * case["pairs"], "flops": 4.0 * full * case["pairs"]}
    if do == "assemble":
        return {"bytes": 24.0 * upper, "flops": 6.0 * upper}
    if do == "values":
        return {"bytes": 16.0 * full + 8.0 * upper, "flops": 6.0 * upper}
    if do == "shifted":
        return {"bytes": 16.0 * upper + 16.0 * n * case["columns"], "flops": 2.0 * full * case["columns"]}
    if do == "spmm":
        return {"bytes": 16.0 * upper + 4.0 * upper + 16.0 * n * case["columns"], "flops": 2.0 * full * case["columns"]}
    info = mesh.elem_info()
    points = case["grid_u"] * case["grid_v"]
    specs = np.bincount(dom.basis_specs()[:, 0], minlength=len(info))
    visits, leaves = 0, np.nonzero(info[:, 0] == 1)[0]
    for e in leaves:
        while e >= 0:
            visits += int(specs[e])
            e = info[e, 3]
    return {"bytes": 16.0 * points * len(leaves) + 8.0 * n, "flops": 4.0 * visits * points}


# ------------------------------------------------------------------------------------------ exact
def _shapes(basis, p, x):
    """N, N', T, T' of orders 0..p at the points x, each (p + 1) x len(x)."""
    n, dn = np.ones((p + 1, len(x))), np.zeros((p + 1, len(x)))
    t, dt = np.zeros_like(n), np.zeros_like(n)
    t[0], dt[0], t[1], dt[1] = 1 - x, -1, 1 + x, 1
    if basis == "hierpoly":
        for k in range(1, p + 1):
            n[k], dn[k] = x ** k, k * x ** (k - 1)
        for k in range(2, p + 1):
            t[k], dt[k] = (n[k] - 1, dn[k]) if k % 2 == 0 else (n[k] - x, dn[k] - 1)
        return n, dn, t, dt
    n[1], dn[1] = x, 1
    for k in range(2, p + 1):
        n[k] = ((2 * k - 1) * x * n[k - 1] - (k - 1) * n[k - 2]) / k
        dn[k] = k * n[k - 1] + x * dn[k - 1]
    scale = [0.968246, 2.561738, 0.838525, 4.248161, 0.816397, 5.882766, 0.808509, 1, 1, 1, 1, 1]
    den = [1, 3, 6, 10, 15, 21, 28, 36, 40, 55, 66, 72]
    for k in range(2, p + 1):
        q = k - 2
        w = np.zeros(k + 1)
        w[k % 2:k:2] = [-(2 * j + 1) for j in range(k % 2, k, 2)]
        w[k] = [1, 3, 6, 10, 15, 21, 28, 36, 40, 55, 66, 72][q]
        t[k], dt[k] = scale[q] / den[q] * (w @ n[:k + 1]), scale[q] / den[q] * (w @ dn[:k + 1])
    return n, dn, t, dt


def _chains(mesh, dom):
    """Bounds per Elem, its specs (i, j, dir, dof), and its ancestors from itself to the root."""
    info, bounds, spec = mesh.elem_info(), mesh.elem_bounds(), dom.basis_specs()
    order = np.argsort(spec[:, 0], kind="stable")
    cut = np.searchsorted(spec[order, 0], np.arange(len(info) + 1))
    specs = [spec[order[cut[e]:cut[e + 1]]][:, 2:6] for e in range(len(info))]
    return info, bounds, specs


def _functions(basis, bounds, outer, inner, spec, xu, xv):
    """Values on the tensor grid xu x xv of ``inner`` of the functions of ``outer``: the u and v components
    (zero for the other direction) and the curl, each (functions, len(xu), len(xv))."""
    (x0, y0, x1, y1), (a0, b0, a1, b1) = bounds[outer], bounds[inner]
    u = (2 * (a0 + (a1 - a0) * (xu + 1) / 2) - x0 - x1) / (x1 - x0)
    v = (2 * (b0 + (b1 - b0) * (xv + 1) / 2) - y0 - y1) / (y1 - y0)
    p = int(spec[:, :2].max()) if len(spec) else 1
    nu, _, tu, dtu = _shapes(basis, max(p, 1), u)
    nv, _, tv, dtv = _shapes(basis, max(p, 1), v)
    ju, jv = 2 / (x1 - x0), 2 / (y1 - y0)
    i, j, along_u = spec[:, 0], spec[:, 1], (spec[:, 2] == 0)[:, None, None]
    fu = np.where(along_u, ju * nu[i][:, :, None] * tv[j][:, None, :], 0.0)
    fv = np.where(along_u, 0.0, jv * tu[i][:, :, None] * nv[j][:, None, :])
    curl = np.where(along_u, -ju * jv * nu[i][:, :, None] * dtv[j][:, None, :],
                    ju * jv * dtu[i][:, :, None] * nv[j][:, None, :])
    return fu, fv, curl


def _pencil(case, mesh, dom):
    """A and B as dense matrices: inner products of the functions on nested Elems by Gauss quadrature."""
    info, bounds, specs = _chains(mesh, dom)
    n = dom.num_dofs
    A, B = np.zeros((n, n)), np.zeros((n, n))
    x, w = np.polynomial.legendre.leggauss(case["glq"])
    for e in range(len(info)):
        if not len(specs[e]):
            continue
        jac = (bounds[e][2] - bounds[e][0]) * (bounds[e][3] - bounds[e][1]) / 4
        wt = (w[:, None] * w[None, :] * jac).ravel()
        mine = [f.reshape(len(specs[e]), -1) for f in _functions(case["basis"], bounds, e, e, specs[e], x, x)]
        dofs, o = specs[e][:, 3], e
        while o >= 0:
            if len(specs[o]):
                theirs = [f.reshape(len(specs[o]), -1) for f in _functions(case["basis"], bounds, o, e, specs[o], x, x)]
                a = (mine[2] * wt) @ theirs[2].T
                b = (mine[0] * wt) @ theirs[0].T + (mine[1] * wt) @ theirs[1].T
                at = np.ix_(dofs, specs[o][:, 3])
                np.add.at(A, at, a)
                np.add.at(B, at, b)
                if o != e:
                    at = np.ix_(specs[o][:, 3], dofs)
                    np.add.at(A, at, a.T)
                    np.add.at(B, at, b.T)
            o = info[o, 3]
    return A, B


def _eigenpairs(A, B, pairs):
    """The physical eigenpairs nearest the target: B-normalised, the largest entry positive."""
    a, b = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    d = torch.rsqrt(torch.diagonal(b))
    a, b = a * d[:, None] * d[None, :], b * d[:, None] * d[None, :]
    low = torch.linalg.cholesky(b)
    c = torch.linalg.solve_triangular(low, torch.linalg.solve_triangular(low, a, upper=False).T, upper=False)
    lam, z = torch.linalg.eigh((c + c.T) / 2)
    lam, z = lam.cpu().numpy(), torch.linalg.solve_triangular(low.T, z, upper=True)
    near = [k for k in np.argsort(np.abs(lam - TARGET), kind="stable") if abs(lam[k]) > 0.05][:pairs]
    values, vectors = [], []
    for k in near:
        x, th = z[:, k], float(lam[k])
        lu = torch.linalg.lu_factor(a - th * (1 + 1e-7) * b)
        for _ in range(4):
            x = torch.linalg.lu_solve(*lu, (b @ x)[:, None])[:, 0]
            x = x / torch.sqrt(x @ (b @ x))
        values.append(float(x @ (a @ x)))
        y = (d * x).cpu().numpy()
        vectors.append(y * np.sign(y[np.argmax(np.abs(y))]))
    return np.array(values), np.array(vectors)


def exact(case, seed):
    do = case["do"]
    if do == "batch":
        values, vectors = [], []
        for k in range(case["meshes"]):
            mesh, dom = _domain(case, 1000 * seed + k, case["pairs"], k)
            if dom.num_dofs > 4000 or k >= 3:
                values.append(None)
                vectors.append(None)
                continue
            va, ve = _eigenpairs(*_pencil(case, mesh, dom), case["pairs"])
            values.append(va)
            vectors.append(ve)
        return {"values": values, "vectors": vectors}
    mesh, dom = _domain(case, seed, case.get("pairs", 1))
    n = dom.num_dofs
    if do in ("dense", "whole"):
        if n > 4000:
            return None
        A, B = _pencil(case, mesh, dom)
        if do == "whole":
            values, vectors = _eigenpairs(A, B, case["pairs"])
            return {"values": values, "vectors": vectors}
        # the symmetric matrix that the lower triangle of B^-1 A stands for; the sign of its vector is free
        z = torch.linalg.solve(torch.from_numpy(B), torch.from_numpy(A))
        z = torch.tril(z) + torch.tril(z, -1).T
        lam = torch.linalg.eigvalsh(z)
        return {"value": float(lam[torch.argmin(torch.abs(lam - TARGET))]), "vector": None}
    if do == "fields":
        s = prepare(case, seed)
        info, bounds, specs = _chains(mesh, dom)
        u = s["u"].cpu().numpy()
        xu, xv = np.linspace(-1, 1, case["grid_u"]), np.linspace(-1, 1, case["grid_v"])
        x, y = np.zeros(tuple(s["x"].shape)), np.zeros(tuple(s["y"].shape))
        if len(x) > 12000:
            return None
        for k, e in enumerate(s["plan"].leaves):
            o = e
            while o >= 0:
                if len(specs[o]):
                    fu, fv, _ = _functions(case["basis"], bounds, o, e, specs[o], xu, xv)
                    x[k] += np.tensordot(u[specs[o][:, 3]], fu, 1)
                    y[k] += np.tensordot(u[specs[o][:, 3]], fv, 1)
                o = info[o, 3]
        return {"x": x, "y": y}
    if do in ("spmm", "shifted"):
        # the matrices are the inputs here
        s = prepare(case, seed)
        rp, col, a = s["gep"].csr("A")
        k = torch.sparse_csr_tensor(torch.from_numpy(rp), torch.from_numpy(col.astype(np.int64)),
                                    torch.from_numpy(a - TARGET * s["gep"].csr("B")[2]), size=(n, n))
        if do == "spmm":
            return torch.mv(k, s["x"].cpu()[:, 0])[:, None] if case["columns"] == 1 else k @ s["x"].cpu()
        if n > 12000:
            return None
        k = k.to_dense().cuda()
        lu, rhs = torch.linalg.lu_factor(k), torch.from_numpy(s["rhs"]).cuda()
        x = torch.linalg.lu_solve(*lu, rhs)
        for _ in range(3):
            x = x + torch.linalg.lu_solve(*lu, rhs - k @ x)
        return x.cpu().numpy()
    if n > 2500 or do in ("step",):
        return None
    A, B = _pencil(case, mesh, dom)
    if do == "assemble":
        r, c = fg.domain_pattern(dom)
        return {"rows": None, "cols": None, "a": A[r, c], "b": B[r, c]}
    gep = _sample(case, dom)
    rp, col, _ = gep.csr("A")
    r = np.repeat(np.arange(n), np.diff(rp))
    return {"a": A[r, col], "b": B[r, col]}
