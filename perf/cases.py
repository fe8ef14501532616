"""Work that programs using h2lib_b200 have it do, as cases that can be timed and checked.

A case names a kind of call and its sizes.  The kinds are the public entry points of the boundary
element path: one nearfield block (bem->nearfield), a dense operator (assemble_bem3d_amatrix), the
assembly of H2 matrices, products with them, GMRES solves, a whole Dirichlet problem from mesh to
solution, and the evaluation of the scattered field.  Quadrature orders (2 / 4), leaf size 64,
eta 1.4, interpolation orders 4 and 5, k between 1 and 8, GMRES(50) and GMRES(80) to 1e-8 are those
of the repository's benchmark and tests.  Every seed turns and stretches the mesh, so another seed
is another geometry (other trees and blocks) as well as other vectors.

exact() restates the discretised operators in plain torch: the same quadrature rules and the same
H2 approximation, every sum in 64 bits, from the definitions.
"""
import math

import numpy as np
import torch

Q, Q2, LEAF, ETA = 2, 4, 64, 1.4
KCONST = 0.0795774715459476679  # 1 / (4 pi)
EPS = 1e-8


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------

def listed():
    return [
        # one block of the nearfield callback, as an H-matrix or ACA code asks for them: the smallest
        # call, all latency
        dict(name="block_laplace_ll", kind="block", mesh="sphere", split=16, pde="laplace",
             layer="slp", basis="l", rows=60, cols=57),
        # dense boundary element matrices of small problems: linear basis, complex kernel
        dict(name="dense_helmholtz_ll", kind="dense", mesh="sphere", split=12, pde="helmholtz",
             layer="dlp", basis="l", k=3.0),
        # the dense matrix of the benchmark (8192 triangles, constant basis)
        dict(name="dense_laplace_cc", kind="dense", mesh="sphere", split=32, pde="laplace",
             layer="slp", basis="c"),
        # both operators of the benchmark's interior Dirichlet problem assembled and applied once
        dict(name="assemble_laplace_ll", kind="assemble", mesh="sphere", split=64, pde="laplace",
             basis="l", m=4),
        # both operators of the Brakhage-Werner equation on the benchmark's cube
        dict(name="assemble_helmholtz_cc", kind="assemble", mesh="cube", split=64, pde="helmholtz",
             basis="c", m=5, k=4.0),
        # the greenhybrid farfield (cross approximation) with the reference test's parameters
        dict(name="assemble_green_ll", kind="green", mesh="sphere", split=45, layer="slp",
             basis="l"),
        # one product in FP64, the inner step of every iterative solver a user brings along
        dict(name="matvec_laplace_ll", kind="matvec", mesh="sphere", split=64, pde="laplace",
             layer="slp", basis="l", m=4, nrhs=1),
        # several incident fields at once: products of one complex matrix with five vectors
        dict(name="matvec_helmholtz_5", kind="matvec", mesh="cube", split=64, pde="helmholtz",
             layer="dlp", basis="c", m=5, k=4.0, nrhs=5),
        # a scattering solve: K + M/2 - ikV, the two matrices sharing one structure
        dict(name="solve_helmholtz_bw", kind="solve", mesh="cube", split=32, k=4.0, m=5),
        # many small uneven Dirichlet systems in one call, mixed precision, four sides each
        dict(name="solve_batch_mixed", kind="batch", meshes=24, nrhs=4, top=24, m=4),
        # the whole of a small Dirichlet problem, from the mesh arrays to the Neumann data
        dict(name="dirichlet_small", kind="dirichlet", split=13, m=4),
        # the scattered field at the points of the reference's exterior test
        dict(name="field_400", kind="field", mesh="cube", split=64, basis="c", k=4.0, points=400),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: the kinds above over their range of sizes, operators, bases and waves."""
    kind = rng.choice(["block", "dense", "assemble", "green", "matvec", "matvec", "solve", "batch",
                       "dirichlet", "field"])
    mesh = rng.choice(["sphere", "cube"])
    pde = rng.choice(["laplace", "helmholtz"])
    layer = rng.choice(["slp", "dlp"])
    basis = rng.choice(["c", "l"])
    k = round(rng.uniform(1.0, 8.0), 2)
    if kind == "block":
        c = dict(kind=kind, mesh=mesh, split=_log_int(rng, 8, 48), pde=pde, layer=layer,
                 basis=basis, rows=_log_int(rng, 3, 200), cols=_log_int(rng, 3, 200))
    elif kind == "dense":
        c = dict(kind=kind, mesh=mesh, split=_log_int(rng, 4, 20), pde=pde, layer=layer,
                 basis=basis)
    elif kind == "assemble":
        c = dict(kind=kind, mesh=mesh, split=_log_int(rng, 8, 40), pde=pde, basis=basis,
                 m=rng.choice([3, 4, 5]))
    elif kind == "green":
        return dict(kind=kind, mesh="sphere", split=_log_int(rng, 8, 45), layer=layer, basis=basis)
    elif kind == "matvec":
        c = dict(kind=kind, mesh=mesh, split=_log_int(rng, 8, 44), pde=pde, layer=layer,
                 basis=basis, m=rng.choice([3, 4, 5]), nrhs=rng.choice([1, 1, 2, 4, 7]))
    elif kind == "solve":
        return dict(kind=kind, mesh=mesh, split=_log_int(rng, 6, 28), k=k, m=rng.choice([4, 5]))
    elif kind == "batch":
        return dict(kind=kind, meshes=_log_int(rng, 2, 20), nrhs=rng.choice([1, 2, 4]),
                    top=rng.choice([9, 16, 24]), m=rng.choice([3, 4]))
    elif kind == "dirichlet":
        return dict(kind=kind, split=_log_int(rng, 4, 16), m=rng.choice([3, 4]))
    else:
        return dict(kind=kind, mesh=mesh, split=_log_int(rng, 8, 64), basis=basis, k=k,
                    points=_log_int(rng, 1, 400))
    if pde == "helmholtz":
        c["k"] = k
    return c


def tolerance(case):
    """About four times what separates the results from exact().  Assembled entries, products and
    fields are FP64 sums: up to 2e-15 on the norm at these sizes.  A solve stops at a residual of
    1e-8, and a step more or less moves the answer as far as it is from the solution: 3e-8 for the
    second-kind equation, 4e-6 for the first-kind one.  The greenhybrid cross approximation (accuracy
    5e-3) picks pivots by comparing rounded values, and other pivots are another approximation, as far
    off the operator as the first: 1e-3."""
    kind = case["kind"]
    if kind in ("batch", "dirichlet"):
        return {"rel": 2e-5, "max": 2e-3}
    if kind == "solve":
        return {"rel": 2e-7, "max": 2e-5}
    if kind == "green":
        return {"rel": 4e-3, "max": 0.1}
    return {"rel": 2e-14, "max": 1e-12}


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------

_OCTAHEDRON = (np.array([[0, 0, 1], [1, 0, 0], [0, 0, -1], [-1, 0, 0], [0, 1, 0], [0, -1, 0]],
                        dtype=np.float64),
               np.array([[0, 1, 4], [1, 2, 4], [2, 3, 4], [3, 0, 4],
                         [0, 5, 1], [1, 5, 2], [2, 5, 3], [3, 5, 0]]))
_CUBE = (np.array([[-1, -1, -1], [-1, 1, -1], [-1, -1, 1], [-1, 1, 1],
                   [1, -1, -1], [1, 1, -1], [1, -1, 1], [1, 1, 1]], dtype=np.float64),
         np.array([[1, 0, 3], [3, 0, 2], [4, 5, 7], [4, 7, 6], [3, 2, 6], [3, 6, 7],
                   [4, 0, 1], [4, 1, 5], [0, 6, 2], [4, 6, 0], [1, 3, 7], [1, 7, 5]]))


def _refined(kind, split):
    """The octahedron (points pushed to the unit sphere) or the cube with every face triangle cut
    into split^2: vertices and triangles, equal points joined."""
    P, F = _OCTAHEDRON if kind == "sphere" else _CUBE
    ij = [(i, j) for i in range(split + 1) for j in range(split + 1 - i)]
    at = {p: n for n, p in enumerate(ij)}
    bary = np.array([(split - i - j, i, j) for i, j in ij], dtype=np.float64) / split
    tri = []
    for i in range(split):
        for j in range(split - i):
            tri.append((at[i, j], at[i + 1, j], at[i, j + 1]))
            if i + j < split - 1:
                tri.append((at[i + 1, j], at[i + 1, j + 1], at[i, j + 1]))
    tri = np.array(tri)
    x = np.einsum("pk,fkd->fpd", bary, P[F]).reshape(-1, 3)
    t = (tri[None] + (np.arange(len(F)) * len(ij))[:, None, None]).reshape(-1, 3)
    _, first, inv = np.unique(np.round(x * 1e7).astype(np.int64), axis=0, return_index=True,
                              return_inverse=True)
    x, t = x[first], inv.reshape(-1)[t]
    if kind == "sphere":
        x = x / np.linalg.norm(x, axis=1, keepdims=True)
    return x, t.astype(np.uint32)


_REFINED = {}


def _mesh(kind, split, rng):
    """A refined macro surface, stretched per axis and turned by the seed's generator."""
    if (kind, split) not in _REFINED:
        _REFINED[kind, split] = _refined(kind, split)
    x, t = _REFINED[kind, split]
    axes = rng.uniform(0.7, 1.4, 3)
    qm, r = np.linalg.qr(rng.standard_normal((3, 3)))
    qm = qm * np.sign(np.diag(r))
    if np.linalg.det(qm) < 0:
        qm[:, 0] = -qm[:, 0]
    return (x * axes) @ qm.T, t


def _splits(case):
    """Refinements of a batch's meshes: 4 to `top`, evenly over the logarithm, in mixed order."""
    s = np.exp(np.linspace(math.log(4), math.log(case["top"]), case["meshes"]))
    return [int(v) for v in np.random.default_rng(5).permutation(np.rint(s).astype(int))]


def _inputs(case, seed):
    """Everything the seed decides, as host arrays: shared by prepare() and exact()."""
    rng = np.random.default_rng([int(seed), 20261204])
    kind = case["kind"]
    if kind == "batch":
        meshes, zs = [], []
        for split in _splits(case):
            meshes.append(_mesh("sphere", split, rng))
            v = rng.standard_normal((case["nrhs"], 3))
            zs.append(4.2 * v / np.linalg.norm(v, axis=1, keepdims=True))
        return dict(meshes=meshes, zs=np.stack(zs, axis=1))  # (nrhs, meshes, 3)
    if kind == "dirichlet":
        x, t = _mesh("sphere", case["split"], rng)
        z = rng.standard_normal(3)
        return dict(x=x, t=t, z=3.0 * z / np.linalg.norm(z))
    x, t = _mesh(case["mesh"], case["split"], rng)
    out = dict(x=x, t=t)
    n = len(x) if case.get("basis", "c") == "l" else len(t)
    cx = case.get("pde") == "helmholtz" or kind in ("solve", "field")

    def vec(shape):
        v = rng.standard_normal(shape)
        return v + 1j * rng.standard_normal(shape) if cx else v

    if kind == "block":
        # two neighbouring patches of the surface, as two clusters of a tree are
        pts = x if case["basis"] == "l" else x[t.astype(np.int64)].mean(axis=1)
        a = pts[rng.integers(n)]
        b = pts[np.argsort(((pts - a) ** 2).sum(1))[min(n - 1, 2 * case["rows"])]]
        out["ridx"], out["cidx"] = (
            np.sort(np.argsort(((pts - p) ** 2).sum(1), kind="stable")[:min(n, c)]).astype(np.uint32)
            for p, c in ((a, case["rows"]), (b, case["cols"])))
    elif kind in ("assemble", "green"):
        out["v"] = vec((n, 1))
    elif kind == "matvec":
        out["v"] = vec((n, case["nrhs"]))
    elif kind == "solve":
        d = rng.standard_normal(3)
        out["dir"] = d / np.linalg.norm(d)
    elif kind == "field":
        out["v"] = vec((n,))
        th = rng.uniform(0, 2 * np.pi, case["points"])
        rad = rng.uniform(2.2, 10.0, case["points"])
        out["pts"] = np.stack([rad * np.cos(th), np.zeros_like(th), rad * np.sin(th)], axis=1)
    return out


def _operator(hb, gr, case, layer):
    b = hb.BASIS_LINEAR_BEM3D if case.get("basis", "c") == "l" else hb.BASIS_CONSTANT_BEM3D
    if case.get("pde", "laplace") == "laplace":
        if layer == "slp":
            return hb.new_slp_laplace_bem3d(gr, Q, Q2, b, b)
        return hb.new_dlp_laplace_bem3d(gr, Q, Q2, b, b, 0.5)
    if layer == "slp":
        return hb.new_slp_helmholtz_bem3d(case["k"], gr, Q, Q2, b, b)
    return hb.new_dlp_helmholtz_bem3d(case["k"], gr, Q, Q2, b, b, 0.5)


def _assemble_pair(lib, check, V, K):
    for h in (V, K):
        check(lib.h2b_h2matrix_assemble_row_clusterbasis(h.handle), "row basis")
        check(lib.h2b_h2matrix_assemble_col_clusterbasis(h.handle), "column basis")
        check(lib.h2b_h2matrix_assemble_farfield(h.handle), "coupling")
    check(lib.h2b_h2matrix_assemble_nearfield_pair(V.handle, K.handle), "nearfield")


def _on_gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def prepare(case, seed):
    from h2lib_b200 import bem3d as hb
    from h2lib_b200._lib import check, lib
    st = dict(case=case, hb=hb, lib=lib, check=check, **_inputs(case, seed))
    kind = case["kind"]
    if kind == "dirichlet":
        return st
    if kind == "batch":
        gu, voff, toff = hb.union_surface3d([hb.Surface3d(x, t) for x, t in st["meshes"]])
        b = hb.BASIS_LINEAR_BEM3D
        slp = hb.new_slp_laplace_bem3d(gu, Q, Q2, b, b)
        dlp = hb.new_dlp_laplace_bem3d(gu, Q, Q2, b, b, 0.5)
        forest = hb.build_forest(gu, voff, toff, b, b, LEAF, ETA)
        V = hb.H2Matrix(slp, forest, case["m"])
        K = hb.H2Matrix(dlp, forest, case["m"], like=V)
        _assemble_pair(lib, check, V, K)
        V.make_single()
        gD = hb.project_l2_harmonic_multi(dlp, toff, st["zs"])
        B = np.zeros_like(gD)
        for r in range(case["nrhs"]):
            hb.addeval_h2matrix_avector(1.0, K, gD[r], B[r])
        st.update(V=V, B=B, voff=voff, keep=(gu, slp, dlp, forest))
        return st
    gr = hb.Surface3d(st["x"], st["t"])
    if kind in ("block", "dense"):
        st["op"] = op = _operator(hb, gr, case, case["layer"])
        shape = (len(st["cidx"]), len(st["ridx"])) if kind == "block" else (op.rows, op.rows)
        # column-major matrices: a torch tensor holds the transpose
        st["G"] = torch.zeros(shape, device="cuda",
                              dtype=torch.complex128 if "k" in case else torch.float64)
        return st
    if kind == "field":
        st["op"] = _operator(hb, gr, dict(case, pde="helmholtz"), "slp")
        return st
    helm = dict(case, pde="helmholtz") if kind == "solve" else case
    b = hb.BASIS_LINEAR_BEM3D if case.get("basis", "c") == "l" else hb.BASIS_CONSTANT_BEM3D
    tree = hb.build_tree(gr, b, b, LEAF, ETA)
    st["tree"] = tree
    if kind == "green":
        st["H"] = hb.H2Matrix(_operator(hb, gr, case, case["layer"]), tree, 2,
                              green=(1, 1.0, 5e-3))
    elif kind == "matvec":
        st["H"] = hb.H2Matrix(_operator(hb, gr, case, case["layer"]), tree, case["m"]).assemble()
    else:
        st["V"] = hb.H2Matrix(_operator(hb, gr, helm, "slp"), tree, case["m"])
        st["K"] = hb.H2Matrix(_operator(hb, gr, helm, "dlp"), tree, case["m"], like=st["V"])
    if kind == "solve":
        _assemble_pair(lib, check, st["V"], st["K"])
        st["b"] = hb.integrate_plane_wave(st["V"].bem, case["k"] * st["dir"], coef=-1.0)
    if "v" in st:
        st["X"] = _on_gpu(st["v"].T)  # one vector per row of the tensor
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------

def run(st):
    case, hb = st["case"], st["hb"]
    kind = case["kind"]
    if kind == "block":
        return hb.nearfield(st["op"], st["ridx"], st["cidx"], out=st["G"].T)
    if kind == "dense":
        return hb.assemble_bem3d_amatrix(st["op"], st["G"])
    if kind in ("assemble", "green", "matvec"):
        if kind == "assemble":
            _assemble_pair(st["lib"], st["check"], st["V"], st["K"])
            mats = [st["V"], st["K"]]
        elif kind == "green":
            mats = [st["H"].assemble()]
        else:
            mats = [st["H"]]
        X = st["X"]
        ys = [torch.zeros_like(X) for _ in mats]
        # the library works on streams of its own: its inputs have to be there
        torch.cuda.current_stream().synchronize()
        for h, y in zip(mats, ys):
            if len(X) == 1:
                hb.addeval_h2matrix_avector(1.0, h, X, y)
            else:
                n = X.shape[1]
                st["check"](st["lib"].h2b_h2matrix_addeval_multi(
                    1.0, 0.0, h.handle, len(X), hb._ptr(X), n, hb._ptr(y), n), "addeval_multi")
        return ys
    if kind == "solve":
        u = np.zeros(st["V"].rows, dtype=np.complex128)
        hb.solve_gmres([st["K"], st["V"]], [1.0, -1j * case["k"]], st["b"], u, EPS, 1000, 80,
                       unitary=True)
        return u
    if kind == "batch":
        X = np.zeros_like(st["B"])
        hb.solve_gmres_batch([st["V"]], [1.0], st["voff"], st["B"], X, EPS, 1000, 50,
                             nrhs=case["nrhs"], mixed=True)
        return X
    if kind == "dirichlet":
        gr = hb.Surface3d(st["x"], st["t"])
        b = hb.BASIS_LINEAR_BEM3D
        slp = hb.new_slp_laplace_bem3d(gr, Q, Q2, b, b)
        dlp = hb.new_dlp_laplace_bem3d(gr, Q, Q2, b, b, 0.5)
        tree = hb.build_tree(gr, b, b, LEAF, ETA)
        V = hb.H2Matrix(slp, tree, case["m"])
        K = hb.H2Matrix(dlp, tree, case["m"], like=V)
        _assemble_pair(st["lib"], st["check"], V, K)
        g = hb.project_l2_harmonic(dlp, st["z"])
        rhs = hb.addeval_h2matrix_avector(1.0, K, g, np.zeros(K.rows))
        u = np.zeros(V.rows)
        hb.solve_gmres_h2matrix_avector(V, rhs, u, EPS, 1000, 50)
        return [g, u]
    return hb.eval_brakhage_werner(st["op"], st["v"], st["pts"], case["k"])


# ---------------------------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------------------------

# operations of one kernel value: three differences, the square of the distance, its inverse root;
# the double layer adds the product with the normal; a wave adds its angle and product
_KERNEL_FLOPS = {("laplace", "slp"): 12, ("laplace", "dlp"): 20, ("laplace", "both"): 22,
                 ("helmholtz", "slp"): 18, ("helmholtz", "dlp"): 30, ("helmholtz", "both"): 34}


def _counts(case, x, t, basis):
    """Nearfield entries, admissible blocks, clusters and index count of the block tree."""
    s = _Structure(x, t, basis)
    near = sum(len(s.tree[r]["idx"]) * len(s.tree[c]["idx"]) for r, c in s.near)
    return near, len(s.far), len(s.tree), s.n


def work(case):
    """One pass: inputs read and results written once; the kernel values of the quadrature (16
    points for each distinct pair of triangles), the multiply-adds of the products."""
    kind = case["kind"]
    d = _inputs(case, 0)
    if kind == "batch":
        steps, by, fl = 40, 0.0, 0.0
        for x, t in d["meshes"]:
            near, far, ncl, n = _counts(case, x, t, "l")
            k = case["m"] ** 3
            entries = near + far * k * k
            by += steps * (4.0 * entries + 16.0 * n * case["nrhs"])
            fl += steps * case["nrhs"] * 2.0 * entries
        return {"bytes": by, "flops": fl}
    x, t = d["x"], d["t"]
    nt, basis = len(t), case.get("basis", "l" if kind == "dirichlet" else "c")
    n = len(x) if basis == "l" else nt
    pde = case.get("pde", "helmholtz" if kind in ("solve", "field") else "laplace")
    w = 16 if pde == "helmholtz" else 8
    geometry = 24.0 * len(x) + 44.0 * nt
    if kind == "block":
        e = float(len(d["ridx"]) * len(d["cidx"]))
        tri = 2.0 if basis == "l" else 1.0  # about two triangles for each vertex
        return {"bytes": w * e + 136.0 * tri * (len(d["ridx"]) + len(d["cidx"])),
                "flops": 16.0 * tri * tri * e * _KERNEL_FLOPS[pde, case["layer"]]}
    if kind == "dense":
        return {"bytes": w * float(n) * n + geometry,
                "flops": 16.0 * nt * nt * _KERNEL_FLOPS[pde, case["layer"]]}
    if kind == "field":
        return {"bytes": geometry + 16.0 * n + 40.0 * case["points"],
                "flops": 4.0 * nt * case["points"] * _KERNEL_FLOPS["helmholtz", "both"]}
    near, far, ncl, n = _counts(case, x, t, basis)
    k = 48 if kind == "green" else case["m"] ** 3
    entries = float(near + far * k * k)
    pairs = near * (4.0 if basis == "l" else 1.0)
    if kind == "matvec":
        return {"bytes": w * (entries + 2.0 * n * case["nrhs"]) + 16.0 * n * k,
                "flops": 2.0 * case["nrhs"] * (entries + 2.0 * n * k) * (4 if w == 16 else 1)}
    if kind == "solve":
        steps = 20.0
        return {"bytes": steps * w * (far * k * k + 2.0 * near), "flops": steps * 8 * entries}
    ops = 1 if kind == "green" else 2
    layer = case.get("layer", "both")
    fl = 16.0 * pairs * _KERNEL_FLOPS[pde, layer] + ops * far * k * k * _KERNEL_FLOPS[pde, "slp"]
    by = ops * (w * (entries + 2.0 * n) + 16.0 * n * k) + geometry
    if kind == "dirichlet":
        steps = 50.0
        return {"bytes": by + steps * w * entries, "flops": fl + steps * 2 * entries}
    return {"bytes": by, "flops": fl}


# ---------------------------------------------------------------------------------------------
# the operators in plain torch
# ---------------------------------------------------------------------------------------------

def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return 0.5 + 0.5 * x, 0.5 * w


def _triangle_rule():
    """Points (t, s) of the unit triangle 0 <= s <= t <= 1 and weights: Duffy's map of Gauss x Gauss."""
    g, w = _gauss(Q)
    t, s = np.repeat(g, Q), (g[:, None] * g[None]).ravel()
    return t, s, (w[:, None] * w[None] * g[:, None]).ravel()


def _singular_rule(case):
    """Sauter and Schwab's rules for a common vertex (1), edge (2) or triangle (3): t, s on the
    row triangle, t, s on the column triangle, weight."""
    g, w = _gauss(Q2)
    a, b, c, d = (v.ravel() for v in np.meshgrid(g, g, g, g, indexing="ij"))
    wa = np.einsum("i,j,k,l->ijkl", w, w, w, w).ravel()
    if case == 1:
        ww = wa * d ** 3 * a
        p = [(d, b * d, a * d, a * c * d), (a * d, a * c * d, d, b * d)]
    elif case == 2:
        e1, e2, x1, x2 = a, b, c, d * (1 - c)
        ww = wa * (1 - x1) * x1 ** 2 * e1
        p = [(x1 + x2, x1 * e1 * e2, x1 * (1 - e1) + x2, x1 * (1 - e1)),
             (x1 + x2, x1 * e1, x1 * (1 - e1 * e2) + x2, x1 * (1 - e1 * e2)),
             (x1 + x2, x1, x1 * e1 + x2, x1 * e1 * e2),
             (x1 * (1 - e1 + e1 * e2) + x2, x1 * e1 * e2, x1 + x2, x1),
             (x1 * e1 * e2 + x2, x1 * e1 * e2, x1 + x2, x1 * e1),
             (x1 * e1 + x2, x1 * e1, x1 + x2, x1 * e1 * e2)]
    else:
        eta, x1, x2 = a, b, c * (1 - b)
        x3 = d * (1 - x1 - x2)
        ww = wa * (1 - x1) * (1 - x1 - x2) * x1
        v = x1 * (1 - eta)
        p = [(x1 + x2 + x3, x1 + x2, v + x2 + x3, x2), (v + x2 + x3, v + x2, x1 + x2 + x3, x2),
             (x1 + x2 + x3, x1 * eta + x2, x2 + x3, x2), (v + x2 + x3, x2, x1 + x2 + x3, x1 + x2),
             (x1 + x2 + x3, x2, v + x2 + x3, v + x2), (x2 + x3, x2, x1 + x2 + x3, x1 * eta + x2)]
    return [np.concatenate([q[i] for q in p]) for i in range(4)] + [np.tile(ww, len(p))]


def _nodal(t, s):
    return [1 - t, t - s, s]


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(_dev())


class _Structure:
    """Cluster tree (longest side of the points' box halved) and strictly admissible block leaves."""

    def __init__(self, x, t, basis):
        t = t.astype(np.int64)
        corners = x[t]
        lo, hi = corners.min(axis=1), corners.max(axis=1)
        if basis == "l":
            pts, smin, smax = x, x.copy(), x.copy()
            for j in range(3):
                np.minimum.at(smin, t[:, j], lo)
                np.maximum.at(smax, t[:, j], hi)
        else:
            pts, smin, smax = (corners[:, 0] + corners[:, 1] + corners[:, 2]) / 3.0, lo, hi
        self.n = len(pts)
        self.tree = []
        self._cluster(pts, smin, smax, np.arange(self.n), -1)
        bmin = np.stack([c["lo"] for c in self.tree])
        bmax = np.stack([c["hi"] for c in self.tree])
        diam = (bmax - bmin).max(axis=1)
        sons = np.array([c["sons"] or (-1, -1) for c in self.tree])
        r, c, self.near, self.far = np.zeros(1, int), np.zeros(1, int), [], []
        while len(r):
            gap = np.maximum(np.maximum(bmin[c] - bmax[r], bmin[r] - bmax[c]), 0.0).max(axis=1)
            adm = (diam[r] <= ETA * gap) & (diam[c] <= ETA * gap)
            leaf = ~adm & (sons[r, 0] < 0) & (sons[c, 0] < 0)
            self.far += list(zip(r[adm], c[adm]))
            self.near += list(zip(r[leaf], c[leaf]))
            go = ~adm & ~leaf
            r, c = r[go], c[go]
            rs = np.where(sons[r] >= 0, sons[r], np.stack([r, np.full_like(r, -1)], 1))
            cs = np.where(sons[c] >= 0, sons[c], np.stack([c, np.full_like(c, -1)], 1))
            r, c = (np.concatenate([rs[:, i] for i in (0, 1) for j in (0, 1)]),
                    np.concatenate([cs[:, j] for i in (0, 1) for j in (0, 1)]))
            ok = (r >= 0) & (c >= 0)
            r, c = r[ok], c[ok]

    def _cluster(self, pts, smin, smax, idx, father):
        me = len(self.tree)
        node = dict(idx=idx, father=father, sons=None)
        self.tree.append(node)
        if len(idx) > LEAF:
            p = pts[idx]
            a, b = p.min(axis=0), p.max(axis=0)
            d = int(np.argmax(b - a))
            below = p[:, d] < (b[d] + a[d]) / 2.0
            if below.any() and not below.all():
                node["sons"] = (self._cluster(pts, smin, smax, idx[below], me),
                                self._cluster(pts, smin, smax, idx[~below], me))
                kids = [self.tree[s] for s in node["sons"]]
                node["lo"] = np.minimum(kids[0]["lo"], kids[1]["lo"])
                node["hi"] = np.maximum(kids[0]["hi"], kids[1]["hi"])
                return me
        node["lo"], node["hi"] = smin[idx].min(axis=0), smax[idx].max(axis=0)
        return me


class _Operator:
    """One discretised boundary integral operator: dense rows, or its H2 approximation of order m
    applied to a matrix of columns."""

    def __init__(self, x, t, pde, layer, basis, k=0.0, alpha=0.5):
        t = t.astype(np.int64)
        self.pde, self.layer, self.basis, self.k = pde, layer, basis, k
        self.alpha = alpha if layer == "dlp" else 0.0
        self.xh, self.th = x, t
        A, B, C = x[t[:, 0]], x[t[:, 1]], x[t[:, 2]]
        nn = np.cross(B - A, C - A)
        gram = np.linalg.norm(nn, axis=1)
        self.nt, self.n = len(t), len(x) if basis == "l" else len(t)
        self.gram, self.normal = _cuda(gram), _cuda(nn / gram[:, None])
        self.t, self.corner = _cuda(t), _cuda(x[t])
        tt, ss, w = _triangle_rule()
        nod = np.stack(_nodal(tt, ss))  # (3, q)
        self.qpts = torch.einsum("lq,tld->tqd", _cuda(nod), self.corner)
        self.qw = _cuda(w * nod if basis == "l" else w[None])  # (functions, q)
        # the functions of a triangle and their indices
        self.dof = self.t if basis == "l" else torch.arange(self.nt, device=_dev())[:, None]
        self.dtype = torch.complex128 if pde == "helmholtz" else torch.float64
        self._singular()

    def kernel(self, X, Y, N):
        """(p, 3), (q, 3) and the normals at Y: the (p, q) kernel values without 1 / (4 pi); any
        leading dimensions."""
        d = [X[..., :, None, i] - Y[..., None, :, i] for i in range(3)]
        return self._value(d, None if N is None else [N[..., None, :, i] for i in range(3)])

    def _value(self, d, n):
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        rn = 1.0 / torch.sqrt(r2)
        if n is not None:
            dot = d[0] * n[0] + d[1] * n[1] + d[2] * n[2]
            val = dot * rn * rn * rn
        else:
            val = rn
        if self.pde == "laplace":
            return val
        kr = self.k * (r2 * rn)
        wave = torch.complex(torch.cos(kr), torch.sin(kr))
        if n is not None:
            wave = wave * torch.complex(torch.ones_like(kr), -kr)
        return val * wave

    def _pairs(self):
        """Ordered pairs of triangles with common vertices, and how many they have."""
        v = self.th.ravel()
        tri = np.repeat(np.arange(self.nt), 3)
        order = np.argsort(v, kind="stable")
        v, tri = v[order], tri[order]
        start = np.flatnonzero(np.r_[True, v[1:] != v[:-1]])
        val = np.diff(np.r_[start, len(v)])
        keys = []
        for d in np.unique(val):
            at = start[val == d][:, None] + np.arange(d)[None]
            ring = tri[at]
            keys.append((ring[:, :, None] * self.nt + ring[:, None, :]).ravel())
        key, shared = np.unique(np.concatenate(keys), return_counts=True)
        return key // self.nt, key % self.nt, shared

    def _singular(self):
        """Sparse matrix of the pairs with common vertices and of the identity term."""
        a, b, shared = self._pairs()
        self.pa, self.pb = _cuda(a), _cuda(b)
        rows, cols, vals = [], [], []
        nf = self.qw.shape[0]
        for c in (1, 2, 3):
            pa, pb = a[shared == c], b[shared == c]
            tv, sv = self.th[pa], self.th[pb]
            eq = tv[:, :, None] == sv[:, None, :]
            tp = np.argsort(~eq.any(axis=2), axis=1, kind="stable")
            rank = np.empty_like(tp)
            np.put_along_axis(rank, tp, np.tile(np.arange(3), (len(tp), 1)), axis=1)
            hit = eq.any(axis=1)
            srank = np.where(hit, np.take_along_axis(rank, eq.argmax(axis=1), axis=1),
                             3 + np.arange(3)[None])
            sp = np.argsort(srank, axis=1, kind="stable")
            x0, x1, y0, y1, w = (_cuda(v) for v in _singular_rule(c))
            nx, ny = torch.stack(_nodal(x0, x1)), torch.stack(_nodal(y0, y1))
            wx, wy = (nx, ny) if self.basis == "l" else (torch.ones_like(x0)[None],) * 2
            step = max(1, 1_500_000 // len(w))
            for s in range(0, len(pa), step):
                ta, tb = _cuda(pa[s:s + step]), _cuda(pb[s:s + step])
                pt, ps = _cuda(tp[s:s + step]), _cuda(sp[s:s + step])
                ca = torch.gather(self.corner[ta], 1, pt[:, :, None].expand(-1, -1, 3))
                cb = torch.gather(self.corner[tb], 1, ps[:, :, None].expand(-1, -1, 3))
                # differences from the corners' differences, the common ones exactly zero
                d = [(ca[:, :, i] @ nx) - (cb[:, :, i] @ ny) for i in range(3)]
                nn = self.normal[tb]
                v = self._value(d, None if self.layer == "slp" else [nn[:, i, None] for i in range(3)])
                wxy = torch.einsum("iq,jq,q->ijq", wx, wy, w).reshape(nf * nf, -1).to(self.dtype)
                val = (v @ wxy.T).reshape(-1, nf, nf)
                val = val * (KCONST * self.gram[ta] * self.gram[tb])[:, None, None]
                ia = torch.gather(self.dof[ta], 1, pt) if nf == 3 else self.dof[ta]
                ib = torch.gather(self.dof[tb], 1, ps) if nf == 3 else self.dof[tb]
                rows.append(ia[:, :, None].expand(-1, nf, nf).reshape(-1))
                cols.append(ib[:, None, :].expand(-1, nf, nf).reshape(-1))
                vals.append(val.reshape(-1))
        if self.alpha:
            mass = (torch.eye(3, device=_dev(), dtype=torch.float64) + 1) / 24 if nf == 3 else \
                torch.full((1, 1), 0.5, device=_dev(), dtype=torch.float64)
            rows.append(self.dof[:, :, None].expand(-1, nf, nf).reshape(-1))
            cols.append(self.dof[:, None, :].expand(-1, nf, nf).reshape(-1))
            vals.append((self.alpha * self.gram[:, None, None] * mass).reshape(-1).to(self.dtype))
        self.sr, self.sc, self.sv = torch.cat(rows), torch.cat(cols), torch.cat(vals)

    def _charges(self, tri, X, keep):
        """Weighted point values (len(tri) * q, columns) of the columns X, whose rows outside the
        index set `keep` count as zero."""
        if keep is None:
            Xm = X
        else:
            Xm = torch.zeros_like(X)
            Xm[keep] = X[keep]
        v = torch.einsum("fq,tfc->tqc", self.qw.to(X.dtype), Xm[self.dof[tri]])
        return (v * self.gram[tri][:, None, None]).reshape(-1, X.shape[1])

    def _tested(self, tri, V, out):
        """out += the sums over the functions of `tri` of the point values V."""
        v = V.reshape(len(tri), -1, V.shape[-1]) * self.gram[tri][:, None, None]
        w = torch.einsum("fq,tqc->tfc", self.qw.to(V.dtype), v)
        out.index_add_(0, self.dof[tri].reshape(-1), w.reshape(-1, V.shape[-1]))

    def _regular(self, ta, tb):
        """Kernel values between the points of two lists of triangles, zero for pairs with common
        vertices."""
        p, q = len(ta), len(tb)
        common = torch.zeros(p, q, dtype=torch.bool, device=_dev())
        for i in range(3):
            for j in range(3):
                common |= self.t[ta][:, i, None] == self.t[tb][None, :, j]
        nq = self.qpts.shape[1]
        N = None if self.layer == "slp" else self.normal[tb].repeat_interleave(nq, 0)
        K = self.kernel(self.qpts[ta].reshape(-1, 3), self.qpts[tb].reshape(-1, 3), N)
        mask = common[:, None, :, None].expand(p, nq, q, nq).reshape(p * nq, q * nq)
        return K.masked_fill(mask, 0.0) * KCONST

    def dense(self, rows=None, cols=None):
        """Entries (rows, cols) of the operator."""
        rows = torch.arange(self.n, device=_dev()) if rows is None else rows
        cols = torch.arange(self.n, device=_dev()) if cols is None else cols
        A = torch.zeros(self.n, len(cols), dtype=self.dtype, device=_dev())
        ra, cb = self._touching(rows), self._touching(cols)
        loc = torch.full((self.n,), -1, dtype=torch.int64, device=_dev())
        loc[cols] = torch.arange(len(cols), device=_dev())
        step = max(1, 12_000_000 // (len(cb) * self.qpts.shape[1] ** 2))
        for s in range(0, len(ra), step):
            ta = ra[s:s + step]
            K = self._regular(ta, cb)
            KT = torch.zeros(len(cols) + 1, K.shape[0], dtype=self.dtype, device=_dev())
            v = K.T.reshape(len(cb), -1, K.shape[0]) * self.gram[cb][:, None, None]
            w = torch.einsum("fq,tqc->tfc", self.qw.to(self.dtype), v)
            at = loc[self.dof[cb]].reshape(-1)
            KT.index_add_(0, torch.where(at < 0, len(cols), at), w.reshape(-1, K.shape[0]))
            self._tested(ta, KT[:-1].T.contiguous(), A)
        at = loc[self.sc]
        ok = at >= 0
        A.index_put_((self.sr[ok], at[ok]), self.sv[ok], accumulate=True)
        return A[rows]

    def _touching(self, idx):
        on = torch.zeros(self.n, dtype=torch.bool, device=_dev())
        on[idx] = True
        return torch.nonzero(on[self.dof].any(dim=1)).reshape(-1)

    def apply_dense(self, X):
        """The operator without any approximation of the farfield, applied to columns."""
        X = X.to(self.dtype)
        Y = torch.zeros_like(X)
        everything = torch.arange(self.nt, device=_dev())
        ch = self._charges(everything, X, None)
        step = max(1, 12_000_000 // (self.nt * self.qpts.shape[1] ** 2))
        for s in range(0, self.nt, step):
            ta = everything[s:s + step]
            self._tested(ta, self._regular(ta, everything) @ ch, Y)
        Y.index_add_(0, self.sr, self.sv[:, None] * X[self.sc])
        return Y

    # ---- H2 approximation by Chebyshev interpolation

    def _lagrange(self, nodes, p, dn=None):
        """(m^3, len(p)) values at p of the Lagrange polynomials of the nodes (3, m), or of their
        derivatives along dn."""
        m = nodes.shape[1]
        val, der = [], []
        for d in range(3):
            xi, z = nodes[d], p[:, d]
            v, g = [], []
            for mu in range(m):
                f = [(z - xi[l]) / (xi[mu] - xi[l]) for l in range(m) if l != mu]
                one = torch.ones_like(z)
                prod = one
                for e in f:
                    prod = prod * e
                v.append(prod)
                if dn is not None:
                    s = torch.zeros_like(z)
                    others = [l for l in range(m) if l != mu]
                    for j, l in enumerate(others):
                        q = one / (xi[mu] - xi[l])
                        for i, e in enumerate(f):
                            if i != j:
                                q = q * e
                        s = s + q
                    g.append(s)
            val.append(torch.stack(v))
            if dn is not None:
                der.append(torch.stack(g))
        if dn is None:
            return torch.einsum("ap,bp,cp->abcp", *val).reshape(m ** 3, -1)
        return (torch.einsum("ap,bp,cp->abcp", der[0] * dn[:, 0], val[1], val[2]) +
                torch.einsum("ap,bp,cp->abcp", val[0], der[1] * dn[:, 1], val[2]) +
                torch.einsum("ap,bp,cp->abcp", val[0], val[1], der[2] * dn[:, 2])
                ).reshape(m ** 3, -1)

    def _structure(self, m):
        self.s = s = _Structure(self.xh, self.th, self.basis)
        cheb = np.cos(np.pi * (2 * np.arange(m) + 1) / (2 * m))
        lo, hi = np.stack([c["lo"] for c in s.tree]), np.stack([c["hi"] for c in s.tree])
        flat = hi - lo < 5e-3
        lo, hi = np.where(flat, lo - 5e-3, lo), np.where(flat, hi + 5e-3, hi)
        nodes = (0.5 * (hi + lo))[:, :, None] + (0.5 * (hi - lo))[:, :, None] * cheb
        self.nodes = _cuda(nodes)  # (clusters, 3, m)
        g = np.stack([np.repeat(nodes[:, 0], m * m, 1),
                      np.tile(np.repeat(nodes[:, 1], m, 1), (1, m)),
                      np.tile(nodes[:, 2], (1, m * m))], axis=2)
        self.grid = _cuda(g)  # (clusters, m^3, 3)
        self.index = [_cuda(c["idx"]) for c in s.tree]
        self.up = [None if c["father"] < 0 else self._lagrange(self.nodes[c["father"]], self.grid[i])
                   for i, c in enumerate(s.tree)]
        near = {}
        for r, c in s.near:
            near.setdefault(r, []).append(c)
        self.near = [(r, torch.cat([self.index[c] for c in cs])) for r, cs in near.items()]

    def apply(self, X, m):
        """The H2 matrix of order m applied to the columns of X."""
        if not hasattr(self, "s"):
            self._structure(m)
        X = X.to(self.dtype)
        Y = torch.zeros_like(X)
        k, cols, tree = m ** 3, X.shape[1], self.s.tree
        nq = self.qpts.shape[1]
        xt = torch.zeros(len(tree), k, cols, dtype=self.dtype, device=_dev())
        yt = torch.zeros_like(xt)
        leaves = [i for i, c in enumerate(tree) if c["sons"] is None]
        for i in leaves:
            tri = self._touching(self.index[i])
            dn = self.normal[tri].repeat_interleave(nq, 0) if self.layer == "dlp" else None
            L = self._lagrange(self.nodes[i], self.qpts[tri].reshape(-1, 3), dn)
            xt[i] = L.to(self.dtype) @ self._charges(tri, X, self.index[i])
        for i in range(len(tree) - 1, 0, -1):  # sons after fathers in the list
            xt[tree[i]["father"]] += self.up[i].to(self.dtype) @ xt[i]
        if self.s.far:
            fr = torch.tensor([r for r, _ in self.s.far], device=_dev())
            fc = torch.tensor([c for _, c in self.s.far], device=_dev())
            step = max(1, 30_000_000 // (k * max(k, cols)))
            for s in range(0, len(fr), step):
                r, c = fr[s:s + step], fc[s:s + step]
                S = self.kernel(self.grid[r], self.grid[c], None) * KCONST
                yt.index_add_(0, r, torch.bmm(S, xt[c]))
        for i in range(1, len(tree)):
            yt[i] += self.up[i].T.to(self.dtype) @ yt[tree[i]["father"]]
        for i in leaves:
            tri = self._touching(self.index[i])
            L = self._lagrange(self.nodes[i], self.qpts[tri].reshape(-1, 3))
            part = torch.zeros_like(X)
            self._tested(tri, L.T.to(self.dtype) @ yt[i], part)
            Y[self.index[i]] += part[self.index[i]]
        for r, near in self.near:
            ta, tb = self._touching(self.index[r]), self._touching(near)
            part = torch.zeros_like(X)
            self._tested(ta, self._regular(ta, tb) @ self._charges(tb, X, near), part)
            Y[self.index[r]] += part[self.index[r]]
        # triangles with common vertices lie in inadmissible blocks only
        for s in range(0, len(self.sr), 4_000_000 // min(cols, 256) + 1):
            e = s + 4_000_000 // min(cols, 256) + 1
            Y.index_add_(0, self.sr[s:e], self.sv[s:e, None] * X[self.sc[s:e]])
        return Y

    def h2_dense(self, m):
        """The whole H2 matrix, column panel by column panel."""
        A = torch.empty(self.n, self.n, dtype=self.dtype, device=_dev())
        for s in range(0, self.n, 2048):
            e = min(self.n, s + 2048)
            X = torch.zeros(self.n, e - s, dtype=self.dtype, device=_dev())
            X[torch.arange(s, e, device=_dev()), torch.arange(e - s, device=_dev())] = 1.0
            A[:, s:e] = self.apply(X, m)
        return A

    # ---- data

    def points_sum(self, f):
        """Integrals of f(points) against the functions of the basis; f: (p, 3) -> (p,)."""
        v = f(self.qpts.reshape(-1, 3))[:, None]
        out = torch.zeros(self.n, 1, dtype=v.dtype, device=_dev())
        self._tested(torch.arange(self.nt, device=_dev()), v, out)
        return out[:, 0]

    def projected(self, f):
        """L2 projection of f onto the linear functions."""
        mass = (torch.eye(3, device=_dev(), dtype=torch.float64) + 1) / 24
        M = torch.zeros(self.n, self.n, dtype=torch.float64, device=_dev())
        i = self.t[:, :, None].expand(-1, 3, 3).reshape(-1)
        j = self.t[:, None, :].expand(-1, 3, 3).reshape(-1)
        M.index_put_((i, j), (self.gram[:, None, None] * mass).reshape(-1), accumulate=True)
        return torch.linalg.solve(M, self.points_sum(f))


def _dirichlet(x, t, zs, m):
    """Projected data (n, columns) and Neumann data of the interior problem for sources zs."""
    V, K = (_Operator(x, t, "laplace", layer, "l") for layer in ("slp", "dlp"))
    g = torch.stack([V.projected(lambda p, z=_cuda(z): 1.0 / (p - z).norm(dim=1)) for z in zs], 1)
    return g, torch.linalg.solve(V.h2_dense(m), K.apply(g, m))


def exact(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    if kind == "batch":
        us = [_dirichlet(x, t, d["zs"][:, i], case["m"])[1] for i, (x, t) in enumerate(d["meshes"])]
        return torch.cat(us).T.contiguous()
    if kind == "dirichlet":
        g, u = _dirichlet(d["x"], d["t"], [d["z"]], case["m"])
        return [g[:, 0], u[:, 0]]
    basis = case.get("basis", "c")
    if kind in ("block", "dense", "green", "matvec"):
        op = _Operator(d["x"], d["t"], case.get("pde", "laplace"), case["layer"], basis,
                       case.get("k", 0.0))
        if kind == "block":
            return op.dense(_cuda(d["ridx"].astype(np.int64)), _cuda(d["cidx"].astype(np.int64)))
        if kind == "dense":
            return op.dense().T
        X = _cuda(d["v"])
        # the cross approximation has no other value to meet than the operator itself
        return [(op.apply_dense(X) if kind == "green" else op.apply(X, case["m"])).T.contiguous()]
    if kind == "assemble":
        X, ys = _cuda(d["v"]), []
        for layer in ("slp", "dlp"):
            op = _Operator(d["x"], d["t"], case["pde"], layer, basis, case.get("k", 0.0))
            ys.append(op.apply(X, case["m"]).T.contiguous())
            del op
        return ys
    k = case["k"]
    if kind == "solve":
        V, K = (_Operator(d["x"], d["t"], "helmholtz", layer, "c", k) for layer in ("slp", "dlp"))
        kd = _cuda(k * d["dir"])
        b = -V.points_sum(lambda p: torch.exp(1j * (p @ kd)))
        A = K.h2_dense(case["m"])
        A -= 1j * k * V.h2_dense(case["m"])
        return torch.linalg.solve(A, b)
    # field: the double layer minus i k times the single layer of the density
    op = _Operator(d["x"], d["t"], "helmholtz", "dlp", basis, k)
    ch = op._charges(torch.arange(op.nt, device=_dev()), _cuda(d["v"])[:, None], None)
    Y = op.qpts.reshape(-1, 3)
    N = op.normal.repeat_interleave(op.qpts.shape[1], 0)
    out = []
    for p in _cuda(d["pts"]).split(32):
        G = op.kernel(p, Y, N) - 1j * k * op.kernel(p, Y, None)
        out.append(KCONST * (G @ ch)[:, 0])
    return torch.cat(out)
