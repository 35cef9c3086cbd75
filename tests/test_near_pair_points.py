"""The free-space near field at evaluation points that lie on the mesh: at
vertices and on edges every output is finite, and the single layer's
displacement, which is continuous there, is its own limit.  Pair by pair on
the host (efmm_pair_eval_host), and the device kernels against sums of such
pairs."""
import ctypes

import numpy as np
import pytest

from conftest import rel
from elfmmlib3d_b200 import geometry as G

_dp = ctypes.POINTER(ctypes.c_double)
LAM, MU = 1.2, 0.9


def _pair(lib, tri, ssl, sdl, x, same=False):
    L = ctypes.CDLL(lib.library_path())
    u, e = np.zeros(3), np.zeros(6)
    keep = [None if a is None else np.ascontiguousarray(a, float) for a in (tri, ssl, sdl, x)]
    p = [None if a is None else a.ctypes.data_as(_dp) for a in keep]
    assert L.efmm_pair_eval_host(ctypes.c_double(LAM), ctypes.c_double(MU), p[0], p[1], p[2], p[3],
                                 ctypes.c_int(int(same)), u.ctypes.data_as(_dp), e.ctypes.data_as(_dp)) == 0
    return u, e


def _meshes():
    yield G.sphere_triangles(2)[0]
    yield G.planar_fault(6, 3)[0]
    yield G.planar_fault(5, 4, strike_deg=37.0, top_depth=1.3)[0]


def _off(tri, x):
    """x 1e-9 edge lengths above the triangle's plane."""
    n = np.cross(tri[1] - tri[0], tri[2] - tri[0])
    return x + 1e-9 * np.linalg.norm(tri[1] - tri[0]) * n / np.linalg.norm(n)


def _on_mesh(lib, weights):
    rng = np.random.default_rng(1)
    for mesh in _meshes():
        for tri in mesh:
            s = rng.normal(size=3)
            for k in range(3):
                for w in weights:
                    x = (1 - w) * tri[k] + w * tri[(k + 1) % 3]
                    us, es = _pair(lib, tri, s, None, x)
                    ud, ed = _pair(lib, tri, None, s, x)
                    for o in (us, es, ud, ed):
                        assert np.isfinite(o).all()
                    yield us, _pair(lib, tri, s, None, _off(tri, x))[0]


def test_vertices_are_finite(lib):
    for _ in _on_mesh(lib, (0.0, 1.0)):
        pass


def test_single_layer_displacement_is_its_limit_on_edges(lib):
    """The displacement 1e-9 edge lengths off the plane is 1e-9 times its
    gradient away, whose largest term there is log 1e9 = 21."""
    for on, off in _on_mesh(lib, (0.0, 0.25, 0.5, 1.0 / 3.0, 0.9, 1.0)):
        assert np.abs(on - off).max() < 1e-6 * np.abs(off).max()


def _device_points(gpu, weights):
    """Targets on a mesh through the direct sum, a plan's near field alone
    (iprec 5: one box), one and several right-hand sides, analytic and stored,
    against sums of host pairs: (layer, device result, sum) with strain."""
    import torch
    d = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")  # noqa: E731
    z = lambda *s: torch.zeros(s, dtype=torch.float64, device="cuda")  # noqa: E731
    for mesh in _meshes():
        mesh = mesh[:40]
        n, cen = len(mesh), mesh.mean(axis=1)
        nrm = np.cross(mesh[:, 1] - mesh[:, 0], mesh[:, 2] - mesh[:, 0])
        nrm /= np.linalg.norm(nrm, axis=1)[:, None]
        x = np.concatenate([(1 - w) * mesh[:9, k] + w * mesh[:9, (k + 1) % 3] for k in range(3) for w in weights])
        m = len(x)
        s = np.random.default_rng(m).normal(size=(5, n, 3))
        for layer in range(2):
            one = [(a, None) if layer == 0 else (None, a) for a in s[0]]
            ref = [sum(np.concatenate(_pair(gpu, t, *ab, y)) for t, ab in zip(mesh, one)) for y in x]
            ref = np.array(ref)
            host = (s[0], None) if layer == 0 else (None, s[0])
            six = lambda e: e.reshape(-1, 9)[:, [0, 4, 8, 1, 2, 5]]  # noqa: E731
            _, _, ut, et = gpu.el3dtriadirecttarg(LAM, MU, mesh, nrm, cen, *host, x)
            yield layer, np.concatenate([ut, six(et)], axis=1), ref
            P = gpu.Plan(0)
            P.set_geometry(d(mesh), d(nrm), d(cen), d(x), iprec=5, iter=True)
            for R in (1, 5):
                dens = [None if a is None else d(s[:R]) for a in host]
                for mode in (0, 1, 2):
                    u, e, ut, et = z(R, n, 3), z(R, n, 3, 3), z(R, m, 3), z(R, m, 3, 3)
                    P.evaluate_batch(LAM, MU, R, *dens, u, e, ut, et, mode=mode)
                    yield layer, np.concatenate([ut[0].cpu().numpy(), six(et[0].cpu().numpy())], axis=1), ref
            P.close()


@pytest.mark.gpu
def test_device_at_vertices(gpu):
    for _, got, ref in _device_points(gpu, (0.0,)):
        assert np.isfinite(got).all() and rel(got, ref) < 1e-12


@pytest.mark.gpu
def test_device_on_edges(gpu):
    """Off the vertices a point's distance from the edge rounds to 0 or not by
    the order of the operations, and what diverges there with it: only the
    displacement of the single layer is the same number on host and device."""
    for layer, got, ref in _device_points(gpu, (0.0, 0.25, 0.5)):
        assert np.isfinite(got).all()
        if layer == 0:
            assert rel(got[:, :3], ref[:, :3]) < 1e-12


@pytest.mark.parametrize("dist", [1e-2, 1e-4, 1e-6])
@pytest.mark.parametrize("height", [0.7, 0.02])
def test_close_to_a_corner_in_the_plane(lib, dist, height):
    """The pair does not depend on the order of the vertices (an odd one turns
    the normal, and the double layer's sign).  Close to a corner
    in the triangle's plane that holds only if the point's distances from the
    edges are measured from the nearer end: from the far one their rounding is
    that of the edge's length, 1e-16 / dist of the result and, in the strain of
    the double layer, its square root's worth more.  Some dozens of roundings
    of terms up to 1 / height times their sum: 1e-12."""
    rng = np.random.default_rng(7)
    worst = 0.0
    for _ in range(60):
        a = rng.normal(size=2)
        t = rng.uniform(0, 2 * np.pi)
        e, n = np.array([np.cos(t), np.sin(t)]), np.array([-np.sin(t), np.cos(t)])
        tri = np.zeros((3, 3))
        tri[:, :2] = a, a + e, a + rng.uniform(0.2, 0.8) * e + height * n
        phi = rng.uniform(0, 2 * np.pi)
        x = tri[rng.integers(3)] + dist * np.array([np.cos(phi), np.sin(phi), 0.0])
        s = rng.normal(size=3)
        for ab in ((s, None), (None, s)):
            f = 1.0 if ab[1] is None else -1.0
            o = _pair(lib, tri, *ab, x)
            for order in ((0, 2, 1), (1, 0, 2), (2, 1, 0)):
                worst = max(worst, *(rel(v, f * w) for v, w in zip(o, _pair(lib, tri[list(order)], *ab, x))))
    assert worst < 1e-12
