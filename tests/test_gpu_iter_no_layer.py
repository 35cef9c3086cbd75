"""Stored near field without a layer: nothing is stored, every replay returns
zeros, whatever the far field, the outputs and the number of points."""
import numpy as np
import pytest

from elfmmlib3d_b200 import geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level,iprec", [(0, 2), (3, 2), (2, 5)])  # one box, a tree, a near field only
@pytest.mark.parametrize("ntarg,strain", [(0, 1), (37, 1), (37, 0)])
def test_stored_calls_without_a_layer_return_zeros(gpu, level, iprec, ntarg, strain):
    tri, nrm, cen = G.sphere_triangles(level)
    tg = G.box_targets(ntarg, 3) if ntarg else None
    w = np.zeros(8)
    for icomp in (2, 3, 5, 3):
        ier, _, *out = gpu.elfmm3dtriatargiter(iprec, 1.2, 0.9, tri, nrm, cen, None, None, tg, icomp_type=icomp,
                                               wsave=w, ifstrain=strain, ifstraintarg=strain)
        assert ier == 0
        for o in out:
            assert not np.any(o)
    gpu.iter_release(w)


@pytest.mark.parametrize("nrhs", [1, 4, 5])
def test_stored_batches_without_a_layer_return_zeros(gpu, nrhs):
    import torch
    tri, nrm, cen = G.sphere_triangles(2)
    d = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")  # noqa: E731
    P = gpu.Plan(0)
    P.set_geometry(d(tri), d(nrm), d(cen), None, iprec=2, iter=True)
    for mode in (1, 2):
        u = torch.ones((nrhs, len(cen), 3), dtype=torch.float64, device="cuda")
        e = torch.ones((nrhs, len(cen), 3, 3), dtype=torch.float64, device="cuda")
        P.evaluate_batch(1.2, 0.9, nrhs, None, None, u, e, mode=mode)
        assert not u.any() and not e.any()
    P.close()
