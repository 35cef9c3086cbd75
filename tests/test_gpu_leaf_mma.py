"""P2M and L2T of few right-hand sides on the FP64 tensor cores (leaf_mma.cu)
against the direct sums and against the many-right-hand-side product forms
(other kernels): free space and half-space image columns, orders 4 to 39
(every tile variant), one to seven right-hand sides, single layers, leaves of
one triangle and leaves past one batch of nodes, particles."""
import numpy as np
import pytest

from conftest import rel
from elfmmlib3d_b200 import geometry as G

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return None if a is None else torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _zeros(*s):
    import torch
    return torch.zeros(s, dtype=torch.float64, device="cuda")


@pytest.mark.parametrize("iprec,n,leaf,nrhs", [(-2, 400, 0, 1), (-1, 401, 3, 2), (0, 640, 0, 1), (1, 777, 1, 1), (1, 1280, 100, 7),
                                               (2, 1280, 0, 1), (2, 999, 17, 3), (3, 1280, 0, 1), (3, 700, 30, 2)])
@pytest.mark.parametrize("sl,dl", [(True, True), (True, False), (False, True)])
def test_few_right_hand_sides_equal_many(gpu, iprec, n, leaf, nrhs, sl, dl):
    """The same densities within a batch of 9 run the product forms."""
    level = next(k for k in range(8) if 20 * 4 ** k >= n)
    tri, nrm, cen = (a[:n] for a in G.sphere_triangles(level))
    tgt = G.box_targets(61, 5)
    rng = np.random.default_rng(n)
    big = 9
    ssl, sdl = (rng.normal(size=(big, n, 3)) if on else None for on in (sl, dl))
    P = gpu.Plan(0)
    if leaf:
        assert P._L.efmm_plan_set_leaf(P._h, leaf) == 0
    P.set_geometry(_dev(tri), _dev(nrm), _dev(cen), _dev(tgt), iprec=iprec)
    assert P.info()["far"]
    outs = []
    for R in (nrhs, big):
        o = [_zeros(R, n, 3), _zeros(R, n, 3, 3), _zeros(R, 61, 3), _zeros(R, 61, 3, 3)]
        P.evaluate_batch(1.3, 0.7, R, *(None if a is None else _dev(a[:R]) for a in (ssl, sdl)), *o)
        outs.append([t[:nrhs].cpu().numpy() for t in o])
    P.close()
    for a, b in zip(*outs):
        # both forms of the same sums in FP64; factorial-basis sums of up to
        # 1,640 terms, recombination amplified by about the size over a leaf
        assert rel(a, b) < 1e-11


@pytest.mark.parametrize("iprec,cells,nrhs", [(1, (20, 10), 1), (2, (24, 12), 1), (2, (15, 7), 4), (3, (24, 12), 2)])
def test_image_few_equal_many(gpu, iprec, cells, nrhs):
    tri, nrm, cen, _ = G.planar_fault(*cells, top_depth=0.7)
    n, big = len(cen), 5
    rng = np.random.default_rng(7)
    ssl, sdl = rng.normal(size=(2, big, n, 3))
    P = gpu.Plan(0)
    P.set_geometry(_dev(tri), _dev(nrm), _dev(cen), _dev(cen * np.array([1, 1, -1.0])), iprec=iprec, mindlin=True)
    assert P.info()["far"]
    outs = []
    for R in (nrhs, big):
        u, e = _zeros(R, n, 3), _zeros(R, n, 3, 3)
        P.evaluate_image(1.3, 0.7, R, _dev(ssl[:R]), _dev(sdl[:R]), u, e)
        outs.append([t[:nrhs].cpu().numpy() for t in (u, e)])
    P.close()
    for a, b in zip(*outs):
        assert rel(a, b) < 1e-11


@pytest.mark.parametrize("iprec,n,leaf", [(1, 777, 0), (2, 1280, 0), (2, 320, 1), (3, 1280, 0)])
@pytest.mark.parametrize("nrhs", [1, 2, 3, 4])
def test_mixed_few_right_hand_sides(gpu, iprec, n, leaf, nrhs):
    """Mixed passes of few right-hand sides, on both sides of the line
    between P2M one by one and the product form, are as close to the FP64
    pass at the same orders as the same densities in a batch of 9, whose P2M
    is the product form (half as much again allowed: FP32 rounding differs
    with the order of the sums)."""
    level = next(k for k in range(8) if 20 * 4 ** k >= n)
    tri, nrm, cen = (a[:n] for a in G.sphere_triangles(level))
    tgt = G.box_targets(61, 5)
    rng = np.random.default_rng(n)
    big = 9
    ssl, sdl = rng.normal(size=(2, big, n, 3))
    P = gpu.Plan(0)
    P.set_mixed_floor(0.0)
    if leaf:
        assert P._L.efmm_plan_set_leaf(P._h, leaf) == 0
    P.set_geometry(_dev(tri), _dev(nrm), _dev(cen), _dev(tgt), iprec=iprec)
    assert P.info()["far"]
    outs = []
    for R, precision in ((nrhs, 1), (big, 1), (big, 0)):
        o = [_zeros(R, n, 3), _zeros(R, n, 3, 3), _zeros(R, 61, 3), _zeros(R, 61, 3, 3)]
        P.evaluate_batch(1.3, 0.7, R, _dev(ssl[:R]), _dev(sdl[:R]), *o, precision=precision)
        outs.append([t[:nrhs].cpu().numpy() for t in o])
    P.close()
    for few, many, exact in zip(*outs):
        assert 0 < rel(few, exact) <= 1.5 * rel(many, exact) < 1e-4
