"""Operation counts that the rates of the bench line are made from."""
import numpy as np
import pytest

from elfmmlib3d_b200 import geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iprec", [1, 2])
def test_fp64_translations_are_counted_in_the_form_that_runs(gpu, iprec):
    """At equal orders the FP64 and the FP32 translations run the same
    parity-split blocks: the same operations."""
    import torch
    d = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")  # noqa: E731
    tri, nrm, cen = G.sphere_triangles(4)
    P = gpu.Plan(0)
    P.set_mixed_floor(0.0)
    P.set_geometry(d(tri), d(nrm), d(cen), None, iprec=iprec)
    fp64, mixed, col = P.translation_flops(3, precision=0), P.translation_flops(3, precision=1), P.flops_per_column()
    for k in ("m2m", "m2l", "l2l"):
        assert fp64[k] > 0 and fp64[k] == pytest.approx(mixed[k], rel=1e-12)
        assert fp64[k] == pytest.approx(3 * 4 * col[k], rel=1e-12)
    P.close()
