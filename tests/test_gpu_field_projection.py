"""Field evaluation and L2 projection against the oracle where their kernels can go wrong: point
counts around a warp and around what one pass of a CTA takes, damped wave numbers, meshes smaller
and larger than one stretch of sources; vertices above one per thread of the projection's launch,
vertices with more triangles than a thread keeps, meshes on both sides of the change (24576 vertices)
from one launch to a kernel per pass.

The field is a sum of n terms in another order: its error is at most n eps sum |terms|, and the sums
here stay below n eps * 100 |u| = 1e-10 for n = 5e3, in the root mean square below 1e-12.  The
projection solves a mass matrix of condition below 100 to the tolerance of its residual, 1e-15."""
import numpy as np
import pytest

from h2lib_b200 import bem3d as hb
from oracle import oracle as orc
from test_gpu_mates import bipyramid

pytestmark = pytest.mark.gpu
L, C = hb.BASIS_LINEAR_BEM3D, hb.BASIS_CONSTANT_BEM3D


def mesh(gr):
    return orc.Mesh(gr.x, gr.t, gr.n, gr.g)


def close(a, b, tol):
    assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)


@pytest.mark.parametrize("basis", [C, L])
@pytest.mark.parametrize("k", [2.0, 1.5 + 0.4j])
@pytest.mark.parametrize("split", [1, 5, 9])
def test_field(basis, k, split):
    gr = hb.new_ellipsoid_surface3d(split, (1.0, 0.8, 1.3))
    op = hb.new_slp_helmholtz_bem3d(k, gr, 2, 4, basis, basis)
    rng = np.random.default_rng(split)
    w = rng.standard_normal(op.rows) + 1j * rng.standard_normal(op.rows)
    d = rng.standard_normal((257, 3))
    pts = d / np.linalg.norm(d, axis=1)[:, None] * rng.uniform(1.6, 6.0, (257, 1))
    ref = orc.eval_brakhage_werner(mesh(gr), w, pts, k, 1.2 - 0.3j, basis == L)
    for n in (1, 2, 31, 32, 33, 64, 65, 257):
        close(hb.eval_brakhage_werner(op, w, pts[:n], 1.2 - 0.3j), ref[:n], 1e-12)


def field(gr, rule, w, pts, k, eta, real):
    """The field of a constant density in the arithmetic of the type `real`."""
    x, n, g = (a.astype(real) for a in (gr.x, gr.n, gr.g))
    A, B, D = (x[gr.t[:, j]] for j in range(3))
    u = np.zeros(len(pts), dtype=np.result_type(real, np.complex64))
    for q in range(rule["n"]):
        tx, sx, wq = real(rule["x0"][q]), real(rule["x1"][q]), real(rule["w"][3][q])
        y = A + tx * (B - A) + sx * (D - B)
        for i, p in enumerate(pts.astype(real)):
            d = p - y
            r2 = np.einsum("td,td->t", d, d)
            r = np.sqrt(r2)
            dn = np.einsum("td,td->t", d, n)
            ph = real(k) * r
            f = (np.cos(ph) + 1j * np.sin(ph)) / (r2 * r) * ((1 - 1j * ph) * dn - 1j * real(eta) * r2)
            u[i] += (f * (w * g * wq)).sum()
    return u / (4 * real(np.pi))


def test_field_rounding():
    """At k r to 200 the sines' arguments carry most of the error.  Against 80-bit arithmetic it is that of
    the same sums in plain FP64 with a rounded square root, 4.2e-15 (5 % for the order of the sums; with r
    from a reciprocal root alone it was 1.13 of it)."""
    if np.finfo(np.longdouble).eps > 1e-18:
        pytest.skip("no arithmetic wider than FP64")
    gr = hb.new_sphere_surface3d(9)
    k, eta = 20.0, 20.0
    op = hb.new_slp_helmholtz_bem3d(k, gr, 2, 4, C, C)
    rule = hb.quad_export(2, 4, C, C, 4)
    rng = np.random.default_rng(5)
    w = rng.standard_normal(op.rows) + 1j * rng.standard_normal(op.rows)
    d = rng.standard_normal((400, 3))
    pts = d / np.linalg.norm(d, axis=1)[:, None] * rng.uniform(1.6, 10.0, (400, 1))
    ref = field(gr, rule, w, pts, k, eta, np.longdouble)
    err = [np.linalg.norm((u - ref).astype(complex)) / np.linalg.norm(ref.astype(complex))
           for u in (hb.eval_brakhage_werner(op, w, pts, eta), field(gr, rule, w, pts, k, eta, np.float64))]
    assert err[0] <= 1.05 * err[1]


@pytest.mark.parametrize("gr", [lambda: hb.new_sphere_surface3d(1),
                                lambda: hb.new_sphere_surface3d(32),      # 4098 vertices
                                lambda: hb.new_cube_surface3d(38),        # 8666 vertices
                                lambda: hb.new_sphere_surface3d(78),      # 24338, one launch
                                lambda: hb.new_cube_surface3d(64),        # 24578, a kernel per pass
                                lambda: bipyramid(7), lambda: bipyramid(8), lambda: bipyramid(60)])
def test_projection(gr):
    gr = gr()
    dlp = hb.new_dlp_laplace_bem3d(gr, 2, 4, L, L, 0.5)
    z = (1.9, 2.1, -2.3)
    close(hb.project_l2_harmonic(dlp, z), orc.project_l2_harmonic(mesh(gr), z), 1e-12)


def test_projection_beside_other_work():
    """The CTAs of the projection's cluster write into each other's shared memory from the first sum on.
    Beside kernels that keep the SMs full they start one after the other, as SMs become free."""
    import torch
    gr = hb.new_sphere_surface3d(13)
    dlp = hb.new_dlp_laplace_bem3d(gr, 2, 4, L, L, 0.5)
    z = (1.9, 2.1, -2.3)
    ref = orc.project_l2_harmonic(mesh(gr), z)
    side = torch.cuda.Stream()
    a = torch.randn(1 << 24, device="cuda")
    torch.cuda.synchronize()
    for _ in range(40):
        with torch.cuda.stream(side):
            for _ in range(20):
                a.mul_(1.0000001)
        close(hb.project_l2_harmonic(dlp, z), ref, 1e-12)
    torch.cuda.synchronize()
