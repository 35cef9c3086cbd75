"""Calls without a far field add in a fixed order: the same call returns the
same bits.  Direct sums (whose parts meet in a cluster), plans with a near
field alone, and the near field alone of a plan with a tree."""
import ctypes

import numpy as np
import pytest

from conftest import rel
from elfmmlib3d_b200 import geometry as G

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _zeros(*s):
    import torch
    return torch.zeros(s, dtype=torch.float64, device="cuda")


def _equal(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


# one to eight parts of the triangles, remainders of the blocks of points and of the tiles
@pytest.mark.parametrize("n,m", [(1, 1), (15, 0), (33, 31), (317, 41), (1280, 1003), (5120, 25000), (20480, 1)])
@pytest.mark.parametrize("sl,dl", [(True, True), (True, False), (False, True)])
def test_direct_sum_repeats(gpu, n, m, sl, dl):
    level = next(k for k in range(8) if 20 * 4 ** k >= n)
    tri, nrm, cen = (a[:n] for a in G.sphere_triangles(level))
    tg = G.shell_targets(m, 3) if m else None
    rng = np.random.default_rng(n)
    dens = [rng.normal(size=(n, 3)) if on else None for on in (sl, dl)]
    outs = [gpu.el3dtriadirecttarg(1.2, 0.9, tri, nrm, cen, *dens, tg) for _ in range(3)]
    assert _equal(outs[0], outs[1]) and _equal(outs[0], outs[2])
    # a few points against the sum of host pairs
    L = ctypes.CDLL(gpu.library_path())
    dp = ctypes.POINTER(ctypes.c_double)
    p = lambda a: None if a is None else a.ctypes.data_as(dp)  # noqa: E731
    pick = rng.choice(n, min(n, 3), replace=False), rng.choice(m, min(m, 3), replace=False) if m else []
    for side, idx in enumerate(pick):
        for i in idx:
            u, e, x = np.zeros(3), np.zeros(6), np.ascontiguousarray(cen[i] if side == 0 else tg[i])
            du, de = np.zeros(3), np.zeros(6)
            for k in range(n):
                t, s, b = (None if a is None else np.ascontiguousarray(a[k]) for a in (tri, *dens))
                assert L.efmm_pair_eval_host(ctypes.c_double(1.2), ctypes.c_double(0.9), p(t), p(s), p(b), p(x),
                                             ctypes.c_int(int(side == 0 and i == k)), p(du), p(de)) == 0
                u += du
                e += de
            # (the displacement of one double layer at its own centroid is 0)
            got = np.concatenate([outs[0][2 * side][i], outs[0][2 * side + 1][i].reshape(9)[[0, 4, 8, 1, 2, 5]]])
            assert rel(got, np.concatenate([u, e])) < 1e-11


@pytest.mark.parametrize("n,m,iprec,surface", [(30, 7, 2, "sphere"), (317, 41, 5, "sphere"), (1280, 999, 5, "sphere"),
                                                (5120, 0, 5, "sphere"), (200, 20, 5, "fault")])
def test_near_field_alone_repeats(gpu, n, m, iprec, surface):
    if surface == "sphere":
        tri, nrm, cen = (a[:n] for a in G.sphere_triangles(next(k for k in range(8) if 20 * 4 ** k >= n)))
    else:
        tri, nrm, cen, _ = G.planar_fault(10, n // 20)
    n = len(cen)
    P = gpu.Plan(0)
    P.set_geometry(_dev(tri), _dev(nrm), _dev(cen), _dev(G.shell_targets(m, 3)) if m else None, iprec=iprec, iter=True)
    assert not P.info()["far"]
    dens = np.random.default_rng(n).normal(size=(2, 17, n, 3))
    direct = None
    for R in (1, 2, 3, 5, 17):
        d = [_dev(a[:R]) for a in dens]
        for mode in (0, 1, 2):
            outs = []
            for _ in range(3):
                o = [_zeros(R, n, 3), _zeros(R, n, 3, 3)] + ([_zeros(R, m, 3), _zeros(R, m, 3, 3)] if m else [])
                P.evaluate_batch(1.2, 0.9, R, *d, *o, mode=mode)
                outs.append([t.cpu().numpy() for t in o])
            assert _equal(outs[0], outs[1]) and _equal(outs[0], outs[2])
            if direct is None:
                direct = gpu.el3dtriadirecttarg(1.2, 0.9, tri, nrm, cen, dens[0, 0], dens[1, 0],
                                                G.shell_targets(m, 3) if m else None)
            for a, b in zip(outs[0], direct):
                assert rel(a[0], b) < 1e-11
    o = [[_zeros(n, 3), _zeros(n, 3, 3)] for _ in range(2)]
    for q in o:
        P.evaluate(1.2, 0.9, _dev(dens[0, 0]), _dev(dens[1, 0]), *q)
    assert _equal(*[[t.cpu().numpy() for t in q] for q in o])
    P.close()


def test_near_field_alone_of_a_tree_repeats(gpu):
    """icomp_type 5 of the ITER entry: a far field is there and not run."""
    tri, nrm, cen = G.sphere_triangles(4)
    tg = G.shell_targets(501, 3)
    dens = np.random.default_rng(1).normal(size=(2, len(cen), 3))
    outs = []
    for _ in range(3):
        w = np.zeros(8)
        ier, _, *o = gpu.elfmm3dtriatargiter(2, 1.2, 0.9, tri, nrm, cen, *dens, tg, icomp_type=5, wsave=w)
        assert ier == 0
        gpu.iter_release(w)
        outs.append(o)
    assert _equal(outs[0], outs[1]) and _equal(outs[0], outs[2])
