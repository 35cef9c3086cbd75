"""The near-field kernel of one right-hand side at the edges of its tiles:
numbers of evaluation points around the 128 threads of a block and of
triangles around its 32-triangle tiles, one and several leaves, each layer,
against the golden-checked direct sum (another kernel over the same pairs)
and, on a sample of points, the oracle's numerical integration."""
import numpy as np
import pytest

from conftest import rel
from elfmmlib3d_b200 import geometry as G

pytestmark = pytest.mark.gpu


def _soup(n, seed):
    """n separate triangles of unit size."""
    rng = np.random.default_rng(seed)
    tri = rng.uniform(-4, 4, (n, 1, 3)) + rng.uniform(-0.5, 0.5, (n, 3, 3))
    return G.triangles_from_mesh(tri.reshape(-1, 3), np.arange(3 * n).reshape(-1, 3))


@pytest.mark.parametrize("n,m", [(1, 0), (1, 1), (2, 126), (31, 97), (32, 96), (33, 96), (65, 200), (129, 0), (130, 300)])
@pytest.mark.parametrize("sl,dl,strain", [(True, True, True), (True, False, True), (False, True, False)])
def test_near_only_equals_direct(gpu, oracle, n, m, sl, dl, strain):
    import torch
    tri, nrm, cen = _soup(n, n)
    rng = np.random.default_rng(1)
    tgt = rng.uniform(-4, 4, (m, 3)) + 6.0
    d = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
    z = lambda *s: torch.zeros(s, dtype=torch.float64, device="cuda")
    P = gpu.Plan(0)
    P.set_geometry(d(tri), d(nrm), d(cen), d(tgt) if m else None, iprec=5)  # one box: near field only
    ssl, sdl = (rng.normal(size=(n, 3)) if on else None for on in (sl, dl))
    dens = [d(a) if a is not None else None for a in (ssl, sdl)]
    outs = []
    for direct in (False, True):
        o = [z(n, 3), z(n, 3, 3) if strain else None, z(m, 3) if m else None, z(m, 3, 3) if m and strain else None]
        P.evaluate(1.3, 0.7, *dens, *o, direct=direct)
        outs.append([None if t is None else t.cpu().numpy() for t in o])
    P.close()
    for a, b in zip(*outs):
        if a is not None:
            assert rel(a, b) < 1e-12  # at most 430 terms of the same closed forms in another order
    k = min(n, 3)
    pt, st, _, _ = oracle.direct(1.3, 0.7, tri, cen, ssl, sdl, None, rows=(0, k))
    assert rel(outs[0][0][:k], pt[:k]) < 1e-10
    if strain:
        assert rel(outs[0][1][:k], st[:k]) < 1e-10


@pytest.mark.parametrize("level,iprec", [(1, 1), (2, 2), (3, 1)])
def test_split_leaves_match_direct(gpu, level, iprec):
    """Few leaves: several blocks share a leaf's triangles."""
    tri, nrm, cen = G.sphere_triangles(level)
    rng = np.random.default_rng(2)
    ssl, sdl = rng.normal(size=(2,) + cen.shape)
    ier, u, e = gpu.elfmm3dtria(iprec, 1.0, 1.0, tri, nrm, cen, ssl, sdl)
    assert ier == 0
    ud, ed, _, _ = gpu.el3dtriadirecttarg(1.0, 1.0, tri, nrm, cen, ssl, sdl)
    tol = {1: 5e-4, 2: 5e-6}[iprec]
    assert rel(u, ud) < tol and rel(e, ed) < 10 * tol


@pytest.mark.parametrize("nrhs", [1, 4, 5, 16, 17])
@pytest.mark.parametrize("n,m", [(7, 0), (33, 9), (130, 50)])
@pytest.mark.parametrize("sl,dl,strain", [(True, True, True), (False, True, True), (True, False, False)])
def test_batch_equals_single_calls(gpu, nrhs, n, m, sl, dl, strain):
    """Both sides of the rule that runs few right-hand sides one by one."""
    import torch
    tri, nrm, cen = _soup(n, n + 1)
    rng = np.random.default_rng(3)
    d = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
    z = lambda *s: torch.zeros(s, dtype=torch.float64, device="cuda")
    P = gpu.Plan(0)
    P.set_geometry(d(tri), d(nrm), d(cen), d(rng.uniform(-5, 5, (m, 3))) if m else None, iprec=5)
    ssl, sdl = (d(rng.normal(size=(nrhs, n, 3))) if on else None for on in (sl, dl))
    mk = lambda *lead: [z(*lead, n, 3), z(*lead, n, 3, 3) if strain else None, z(*lead, m, 3) if m else None,
                        z(*lead, m, 3, 3) if m and strain else None]
    batch = mk(nrhs)
    P.evaluate_batch(1.3, 0.7, nrhs, ssl, sdl, *batch)
    for r in range(nrhs):
        one = mk()
        P.evaluate(1.3, 0.7, None if ssl is None else ssl[r], None if sdl is None else sdl[r], *one)
        for a, b in zip(batch, one):
            if a is not None:
                # the same closed forms; cancellation inside a pair's response up to about 1e4
                assert rel(a[r].cpu().numpy(), b.cpu().numpy()) < 1e-11
    P.close()
