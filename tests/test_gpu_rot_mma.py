"""The FP64 translations on the FP64 tensor cores (rot_mma.cu) against the
dense per-offset operators: a Plan made with ELFMM3D_TRANSLATIONS=dense runs
the same pass through other kernels.  Orders from 4 to 39 (iprec -2..3: blocks
of every remainder modulo 8 and 4, both tile heights of shared memory), column
counts around the tile widths of 8, 16 and 32, odd numbers of boxes."""
import numpy as np
import pytest

from conftest import rel
from elfmmlib3d_b200 import geometry as G

pytestmark = pytest.mark.gpu


def _run(gpu, monkeypatch, dense, geo, iprec, nrhs, ssl, sdl):
    import torch
    d = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
    monkeypatch.setenv("ELFMM3D_TRANSLATIONS", "dense" if dense else "factored")
    P = gpu.Plan(0)
    tri, nrm, cen, tgt = geo
    n, m = len(cen), len(tgt)
    P.set_geometry(d(tri), d(nrm), d(cen), d(tgt) if m else None, iprec=iprec)
    z = lambda *s: torch.zeros((nrhs,) + s, dtype=torch.float64, device="cuda")
    o = [z(n, 3), z(n, 3, 3), z(m, 3) if m else None, z(m, 3, 3) if m else None]
    P.evaluate_batch(1.3, 0.7, nrhs, d(ssl), d(sdl), *o)
    info = P.info()
    P.close()
    return [t.cpu().numpy() for t in o if t is not None], info


@pytest.mark.parametrize("iprec,nrhs,n,m", [(-2, 1, 300, 0), (-1, 1, 700, 33), (0, 2, 900, 0), (1, 1, 2000, 100), (1, 5, 1279, 7),
                                            (2, 1, 3001, 50), (2, 3, 1500, 0), (2, 17, 900, 21), (3, 1, 2500, 0),
                                            (3, 4, 1600, 40)])
def test_mma_translations_equal_dense(gpu, monkeypatch, iprec, nrhs, n, m):
    level = next(k for k in range(8) if 20 * 4 ** k >= n)
    tri, nrm, cen = (a[:n] for a in G.sphere_triangles(level))
    rng = np.random.default_rng(n)
    tgt = G.box_targets(m, 3) if m else np.zeros((0, 3))
    ssl, sdl = rng.normal(size=(2, nrhs, n, 3))
    geo = (tri, nrm, cen, tgt)
    a, info = _run(gpu, monkeypatch, False, geo, iprec, nrhs, ssl, sdl)
    b, _ = _run(gpu, monkeypatch, True, geo, iprec, nrhs, ssl, sdl)
    assert info["far"] and info["m2l_pairs"] > 0
    for x, y in zip(a, b):
        # factored and dense operators agree to 2e-14 in the normalised basis;
        # the recombination amplifies by about the size over a leaf
        assert rel(x, y) < 1e-11
