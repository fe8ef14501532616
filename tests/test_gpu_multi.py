"""Products with several columns (h2b_h2matrix_addeval_multi) against products column by column and
against the matrix put together from its exported parts, which reads every coupling block where the
product reads one of two transposed ones.  Sums of at most a few thousand FP64 terms in another
order: 1e-13 on the norm."""
import ctypes as C

import numpy as np
import pytest

from h2lib_b200 import bem3d as hb
from h2lib_b200._lib import check, lib

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


@pytest.mark.parametrize("rb,cb", [(L, L), (K, K), (K, L)])
@pytest.mark.parametrize("pde,m", [("laplace", 2), ("laplace", 3), ("helmholtz", 5)])
def test_product_against_parts(pde, m, rb, cb):
    """rb != cb: the trees differ and no block stands for two."""
    H = matrix(pde, cb, m, rb)
    k = m ** 3
    rec = H.tree.block_records()
    trees = [H.tree.clusters(s) for s in (0, 1)]
    W = []
    for side, (cl, _, _) in enumerate(trees):
        V, E = H.export(2 * side), H.export(2 * side + 1)
        vo, eo, full, stack = 0, 0, {}, []
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
            parts = []
            for _ in range(cl[i][2]):
                s = at
                at = son_ids(s)
                parts.append(full[s] @ E[s])
            full[i] = np.concatenate(parts)
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
    X = vectors(H, H.cols, 3)
    Y = np.zeros((3, H.rows), dtype=H.dtype)
    multi(H, 1.0, 3, X, H.cols, Y, H.rows)
    close(Y.T, A @ X.T)
    close(singles(H, 1.0, X, np.zeros_like(Y)).T, A @ X.T)
