"""Products with several columns (h2b_h2matrix_addeval_multi) against products column by column and
against the matrix put together from its exported parts, which reads every coupling block where the
product reads one of two transposed ones.  Sums of at most a few thousand FP64 terms in another
order: 1e-13 on the norm."""
import contextlib
import ctypes as C

import numpy as np
import pytest

from h2lib_b200 import bem3d as hb
from h2lib_b200._lib import check, checkp, lib

pytestmark = pytest.mark.gpu
L, K = hb.BASIS_LINEAR_BEM3D, hb.BASIS_CONSTANT_BEM3D


def matrix(pde, basis, m, rb=None):
    gr = hb.new_ellipsoid_surface3d(13, (1.0, 0.8, 1.3))
    rb = basis if rb is None else rb
    op = (hb.new_dlp_laplace_bem3d(gr, 2, 4, rb, basis, 0.5) if pde == "laplace"
          else hb.new_dlp_helmholtz_bem3d(2.0, gr, 2, 4, rb, basis, 0.5))
    return hb.H2Matrix(op, hb.build_tree(gr, rb, basis, 24, 1.4), m).assemble()


def vectors(H, n, cols, seed=0):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((cols, n))
    return x + 1j * rng.standard_normal((cols, n)) if H.dtype == np.complex128 else x


def multi(H, alpha, n, X, ldx, Y, ldy):
    a = complex(alpha)
    p = [v if isinstance(v, C.c_void_p) else hb._ptr(v) for v in (X, Y)]
    check(lib.h2b_h2matrix_addeval_multi(a.real, a.imag, H.handle, n, p[0], ldx, p[1], ldy), "multi")


def singles(H, alpha, X, Y):
    return np.stack([hb.addeval_h2matrix_avector(alpha, H, x.copy(), y.copy()) for x, y in zip(X, Y)])


def close(a, b, tol=1e-13):
    assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)


@pytest.mark.parametrize("pde,basis,m", [("laplace", L, 2), ("laplace", K, 4), ("helmholtz", K, 3),
                                         ("helmholtz", L, 5)])
def test_columns(pde, basis, m):
    H = matrix(pde, basis, m)
    alpha = 0.7 - 0.2j if pde == "helmholtz" else 0.7
    for cols in (1, 2, 3, 4, 5, 8, 9, 17):
        X, Y = vectors(H, H.cols, cols), vectors(H, H.rows, cols, 1)
        ref = singles(H, alpha, X, Y)
        out = Y.copy()
        multi(H, alpha, cols, X, H.cols, out, H.rows)
        close(out, ref)
    # device arrays with longer columns
    import torch
    ld = H.cols + 5
    X, Y = vectors(H, ld, 6), vectors(H, ld, 6, 1)
    dx, dy = torch.from_numpy(X).cuda(), torch.from_numpy(Y).cuda()
    torch.cuda.synchronize()
    multi(H, alpha, 6, dx, ld, dy, ld)
    out = dy.cpu().numpy()
    close(out[:, :H.rows], singles(H, alpha, X[:, :H.cols], Y[:, :H.rows]))
    assert np.array_equal(out[:, H.rows:], Y[:, H.rows:])


def test_columns_in_place():
    H = matrix("laplace", L, 3)
    X = vectors(H, H.cols, 4)
    ref = singles(H, 1.0, X, X)
    buf = X.copy()
    multi(H, 1.0, 4, buf, H.cols, buf, H.cols)  # y = x
    close(buf, ref)
    # column r of Y is column r + 1 of X: one after the other
    buf = vectors(H, H.cols, 5)
    ref = buf.copy()
    for r in range(4):
        ref[r + 1] = hb.addeval_h2matrix_avector(1.0, H, ref[r].copy(), ref[r + 1].copy())
    multi(H, 1.0, 4, buf, H.cols, C.c_void_p(buf.ctypes.data + buf.strides[0]), H.cols)
    close(buf, ref)


@contextlib.contextmanager
def no_room(left=0):
    """Stream-ordered allocations find `left` pieces of 1 MiB meanwhile: they come from a pool of limited
    size that is full but for these."""
    from cuda.bindings import driver as cu

    def ok(r):
        assert r[0] == cu.CUresult.CUDA_SUCCESS, r[0]
        return r[1] if len(r) > 1 else None
    dev = ok(cu.cuCtxGetDevice())
    props = cu.CUmemPoolProps()
    props.allocType = cu.CUmemAllocationType.CU_MEM_ALLOCATION_TYPE_PINNED
    props.location.type = cu.CUmemLocationType.CU_MEM_LOCATION_TYPE_DEVICE
    props.location.id = int(dev)
    props.maxSize = 32 << 20
    pool, before, held = ok(cu.cuMemPoolCreate(props)), ok(cu.cuDeviceGetMemPool(dev)), []
    while len(held) < 256:
        r = cu.cuMemAllocFromPoolAsync(1 << 20, pool, cu.CUstream(0))
        if r[0] != cu.CUresult.CUDA_SUCCESS:
            break
        held.append(r[1])
    assert r[0] == cu.CUresult.CUDA_ERROR_OUT_OF_MEMORY
    for _ in range(left):
        ok(cu.cuMemFreeAsync(held.pop(), cu.CUstream(0)))
    ok(cu.cuCtxSynchronize())
    ok(cu.cuDeviceSetMemPool(dev, pool))
    try:
        yield
    finally:
        ok(cu.cuDeviceSetMemPool(dev, before))
        for p in held:
            ok(cu.cuMemFreeAsync(p, cu.CUstream(0)))
        ok(cu.cuCtxSynchronize())
        ok(cu.cuMemPoolDestroy(pool))


def test_columns_without_room():
    """Eight columns' work vectors (5 MB) do not fit: one column after the other."""
    H = matrix("helmholtz", K, 5)
    X = vectors(H, H.cols, 8)
    ref = singles(H, 1.0, X, np.zeros_like(X))
    Y = np.zeros_like(X)
    with no_room():
        multi(H, 1.0, 8, X, H.cols, Y, H.rows)
    close(Y, ref)


def test_export_without_room():
    """The coupling matrices of 1472 blocks (368 MB), put out in pieces that fit 4 MiB."""
    H = matrix("helmholtz", K, 5)
    ref = H.export(4)
    with no_room(4):
        out = H.export(4)
    assert np.array_equal(out, ref)


def parts(H):
    """The matrix put together from its exported parts: leaf bases, transfers, every admissible block's
    coupling matrix, nearfield blocks."""
    k = H.info()["rank"]
    rec = H.tree.block_records()
    trees = [H.tree.clusters(s) for s in (0, 1)]
    W = []
    for side, (cl, _, _) in enumerate(trees):
        V, E = H.export(2 * side), H.export(2 * side + 1)
        vo, eo, full = 0, 0, {}
        # pre-order: leaves' V and non-root clusters' E in that order
        info = []
        for i, (off, size, sons) in enumerate(cl):
            if i:
                info.append((i, E[eo:eo + k * k].reshape(k, k).T))
                eo += k * k
            if sons == 0:
                full[i] = V[vo:vo + size * k].reshape(k, size).T
                vo += size * k
        E = dict(info)

        def son_ids(i):
            if cl[i][2] == 0:
                return i + 1
            at = i + 1
            rows = []
            for _ in range(cl[i][2]):
                s = at
                at = son_ids(s)
                rows.append(full[s] @ E[s])
            full[i] = np.concatenate(rows)
            return at
        son_ids(0)
        W.append({(int(cl[i][0]), int(cl[i][1])): full[i] for i in range(len(cl))})
    S, N = H.export(4), H.export(5)
    A = np.zeros((H.rows, H.cols), dtype=H.dtype)
    ri, ci = trees[0][2], trees[1][2]
    so = no = 0
    for r0, rs, c0, cs, adm in rec:
        r, c = ri[r0:r0 + rs], ci[c0:c0 + cs]
        if adm:
            B = W[0][r0, rs] @ S[so:so + k * k].reshape(k, k).T @ W[1][c0, cs].T
            so += k * k
        else:
            B = N[no:no + rs * cs].reshape(cs, rs).T
            no += rs * cs
        A[np.ix_(r, c)] = B
    return A


@pytest.mark.parametrize("rb,cb", [(L, L), (K, K), (K, L)])
@pytest.mark.parametrize("pde,m", [("laplace", 2), ("laplace", 3), ("helmholtz", 5)])
def test_product_against_parts(pde, m, rb, cb):
    """rb != cb: the trees differ and no block stands for two."""
    H = matrix(pde, cb, m, rb)
    A = parts(H)
    X = vectors(H, H.cols, 3)
    Y = np.zeros((3, H.rows), dtype=H.dtype)
    multi(H, 1.0, 3, X, H.cols, Y, H.rows)
    close(Y.T, A @ X.T)
    close(singles(H, 1.0, X, np.zeros_like(Y)).T, A @ X.T)


def flat(tree, blocks):
    """A tree with the same clusters and these blocks (row cluster, column cluster, admissible)."""
    rec, box, idx = tree.clusters()
    b = np.array(blocks, dtype=np.uint32)
    tr = [np.ascontiguousarray(rec[:, j]) for j in range(3)] + [np.ascontiguousarray(box), len(idx), idx]
    handle = lib.h2b_tree_new_flat(len(rec), *tr, len(rec), *tr, len(b), np.ascontiguousarray(b[:, 0]),
                                   np.ascontiguousarray(b[:, 1]),
                                   np.ascontiguousarray(b[:, 2].astype(np.uint8)))
    return hb.Tree(checkp(handle, "h2b_tree_new_flat"))


def block_ids(tree):
    rec, _, _ = tree.clusters()
    ids = {(int(o), int(s)): i for i, (o, s, _) in enumerate(rec)}
    return [(ids[int(r0), int(rs)], ids[int(c0), int(cs)], int(adm))
            for r0, rs, c0, cs, adm in tree.block_records()]


def one_sided(tree, by_row):
    """The same clusters with some of the admissible blocks above the diagonal cut into their sons'
    blocks, so that the blocks across the diagonal from them have no transposed partner.  by_row: the
    blocks of a row cluster one after the other, else the order of the block tree."""
    rec, _, _ = tree.clusters()
    ends = {}

    def walk(i):
        end = i + 1
        for _ in range(int(rec[i][2])):
            end = walk(end)
        ends[i] = end
        return end
    walk(0)
    sons = {i: [i + 1, ends[i + 1]] for i in range(len(rec)) if rec[i][2]}
    blocks = []
    for r, c, adm in block_ids(tree):
        if adm and r < c and r in sons and c in sons and (r + c) % 3:
            blocks += [(a, b, 1) for b in sons[c] for a in sons[r]]
        else:
            blocks.append((r, c, adm))
    if by_row:
        blocks.sort()
    pairs = {(r, c) for r, c, a in blocks if a}
    alone = sum((c, r) not in pairs for r, c in pairs)
    return flat(tree, blocks), alone, len(pairs)


@pytest.mark.parametrize("basis", [L, K])
def test_blocks_listed_twice(basis):
    """A list that has every block twice is the sum of both."""
    gr = hb.new_ellipsoid_surface3d(9, (1.0, 0.8, 1.3))
    tree = hb.build_tree(gr, basis, basis, 24, 1.4)
    blocks = block_ids(tree)
    op = hb.new_dlp_laplace_bem3d(gr, 2, 4, basis, basis, 0.5)
    H = hb.H2Matrix(op, flat(tree, blocks), 3).assemble()
    X = vectors(H, H.cols, 3)
    ref = singles(H, 2.0, X, np.zeros_like(X))
    for twice in (blocks + blocks, [b for b in blocks for _ in range(2)]):
        H2 = hb.H2Matrix(op, flat(tree, twice), 3).assemble()
        close(singles(H2, 1.0, X, np.zeros_like(X)), ref)


@pytest.mark.parametrize("shape", ["symmetric", "one-sided", "one-sided by row"])
@pytest.mark.parametrize("pde,leaf,panels", [("laplace", 16, (4, 5, 6)), ("helmholtz", 24, (4, 6, 8))])
def test_runs_of_panels(pde, leaf, panels, shape):
    """Runs of several coupling panels per warp.  At rank 125 the panels of a few KiB are 21 to 63 per
    block and 23000 to 82000 in all, which makes runs of one to seven panels where the default panels'
    are single; some lengths divide a block's panels and some do not.  Runs keep their sums over panels,
    change the row cluster and, with a partition that is not symmetric, go from blocks without a
    transposed partner to blocks with one of the same row cluster and back."""
    gr = hb.new_ellipsoid_surface3d(13, (1.0, 0.8, 1.3))
    tree = hb.build_tree(gr, K, K, leaf, 1.4)
    if shape != "symmetric":
        tree, alone, total = one_sided(tree, shape.endswith("row"))
        assert total // 8 < alone < total
    op = (hb.new_dlp_laplace_bem3d(gr, 2, 4, K, K, 0.5) if pde == "laplace"
          else hb.new_dlp_helmholtz_bem3d(2.0, gr, 2, 4, K, K, 0.5))
    H = hb.H2Matrix(op, tree, 5).assemble()
    A = parts(H)
    for kib in panels:
        H.set_matvec_shape(panel_kib=kib)
        for cols in (1, 3, 5, 8):
            X = vectors(H, H.cols, cols, cols)
            Y = np.zeros((cols, H.rows), dtype=H.dtype)
            multi(H, 1.0, cols, X, H.cols, Y, H.rows)
            close(Y.T, A @ X.T)
