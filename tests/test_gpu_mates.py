"""Distant-pair kernels of the q = 2 rule against the oracle where they can go wrong: tile edges and
remainders, tiles filled together with their mates (equal row and column lists) and without (other
lists, mixed bases), the conjugate transpose, complex outputs aligned to 8 bytes, vertices with more
triangles than a warp's row table holds.  |a - b| <= 1e-12 * max(|b_ij|, max_j |b_ij|), the FP64
path's rule (sums of a few hundred terms in another order: below 1e-13)."""
import numpy as np
import pytest

from conftest import rel_entry_err
from h2lib_b200 import bem3d as hb
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
L, C = hb.BASIS_LINEAR_BEM3D, hb.BASIS_CONSTANT_BEM3D
KINDS = ["lslp", "ldlp", "ladlp", "hslp", "hdlp", "hadlp"]


def operator(kind, gr, rb, cb):
    make = {"slp": ("slp", ()), "dlp": ("dlp", (0.5,)), "adlp": ("adlp", (0.5,))}[kind[1:]]
    pde = "laplace" if kind[0] == "l" else "helmholtz"
    k = () if pde == "laplace" else (2.0,)
    return getattr(hb, f"new_{make[0]}_{pde}_bem3d")(*k, gr, 2, 4, rb, cb, *make[1])


def reference(kind, gr, rb, cb, ridx=None, cidx=None):
    layer = {"slp": orc.SLP, "dlp": orc.DLP, "adlp": orc.ADLP}[kind[1:]]
    pde = orc.LAPLACE if kind[0] == "l" else orc.HELMHOLTZ
    return orc.nearfield(orc.Mesh(gr.x, gr.t, gr.n, gr.g), pde, layer, rb, cb,
                         k=2.0 if kind[0] == "h" else 0.0,
                         alpha=0.0 if kind[1:] == "slp" else 0.5, ridx=ridx, cidx=cidx)


@pytest.fixture(scope="module")
def ball():
    return hb.new_ellipsoid_surface3d(5, (1.0, 0.8, 1.3))  # 200 triangles, 102 vertices


@pytest.mark.parametrize("basis", [C, L])
@pytest.mark.parametrize("kind", KINDS)
def test_equal_and_other_lists(ball, kind, basis):
    rng = np.random.default_rng(3)
    op = operator(kind, ball, basis, basis)
    for n in (1, 7, 8, 9, 63, 64, 65, min(op.rows, 130)):
        idx = rng.permutation(op.rows)[:n].astype(np.uint32)
        ref = reference(kind, ball, basis, basis, idx, idx)
        assert rel_entry_err(hb.nearfield(op, idx, idx), ref) < 1e-12, (n, "equal lists")
        other = rng.permutation(idx)
        ref2 = reference(kind, ball, basis, basis, idx, other)
        assert rel_entry_err(hb.nearfield(op, idx, other), ref2) < 1e-12, (n, "permuted list")
        nt = hb.nearfield(op, idx, idx, ntrans=True)
        assert rel_entry_err(nt, ref.conj().T) < 1e-12, (n, "ntrans")


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("rb,cb", [(C, L), (L, C)])
def test_mixed_bases(ball, kind, rb, cb):
    op = operator(kind, ball, rb, cb)
    ref = reference(kind, ball, rb, cb)
    assert rel_entry_err(hb.nearfield(op, None, None), ref) < 1e-12


@pytest.mark.parametrize("basis", [C, L])
def test_complex_output_on_8_bytes(ball, basis):
    import torch
    op = operator("hdlp", ball, basis, basis)
    n = op.rows
    buf = torch.zeros(2 * n * n + 1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()

    class At:
        def data_ptr(self):
            return buf.data_ptr() + 8
    hb.assemble_bem3d_amatrix(op, At())
    G = buf[1:].cpu().numpy().view(np.complex128).reshape(n, n).T
    assert rel_entry_err(G, reference("hdlp", ball, basis, basis)) < 1e-12


def bipyramid(n):
    """Two apices over a ring of n vertices: apices touched by n triangles each."""
    a = 2 * np.pi * np.arange(n) / n
    x = np.concatenate([np.stack([np.cos(a), np.sin(a), 0.1 * np.sin(3 * a)], 1),
                        [[0.1, 0.0, 1.2], [0.0, 0.2, -1.1]]])
    i, j = np.arange(n), (np.arange(n) + 1) % n
    t = np.concatenate([np.stack([i, j, np.full(n, n)], 1), np.stack([j, i, np.full(n, n + 1)], 1)])
    return hb.Surface3d(x, t)


@pytest.mark.parametrize("kind", ["lslp", "ldlp", "hdlp"])
@pytest.mark.parametrize("n", [9, 40, 150])
def test_many_triangles_around_a_vertex(kind, n):
    gr = bipyramid(n)
    op = operator(kind, gr, L, L)
    assert rel_entry_err(hb.nearfield(op, None, None), reference(kind, gr, L, L)) < 1e-12
    idx = np.arange(gr.vertices, dtype=np.uint32)[::-1].copy()  # apices first
    half = idx[:len(idx) // 2]
    ref = reference(kind, gr, L, L, half, idx)
    assert rel_entry_err(hb.nearfield(op, half, idx), ref) < 1e-12
