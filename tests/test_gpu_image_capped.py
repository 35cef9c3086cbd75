"""Image near field of pairs whose adaptive quadrature reaches its last
halving: targets on the surface trace of a surface-breaking triangle, whose
image kernel is singular on the triangle's own edge.  The blocks that a plan
stores against the direct image sum, which halves sub-triangles by their
midpoints without a path code."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dip", [30.0, 65.0])
@pytest.mark.parametrize("layer", [0, 1])
@pytest.mark.parametrize("turn", [0, 1, 2])  # the trace on each edge: paths of other first digits
def test_targets_on_the_trace(gpu, dip, layer, turn):
    d = np.radians(dip)
    v = np.array([[0.0, 0.0, 0.0], [1.0, 0.3, 0.0], [0.4, 0.9 * np.cos(d), -0.9 * np.sin(d)]])
    x = np.stack([(1 - w) * v[0] + w * v[1] for w in (0.37, 0.61803, 0.88)])
    tri = np.roll(v, turn, axis=0)[None]
    nrm = np.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0])
    nrm /= np.linalg.norm(nrm, axis=1)[:, None]
    s = np.array([[0.3, -0.7, 0.5]])
    dens = (s, None) if layer == 0 else (None, s)
    gpu.hs_capped()
    ier, u0, e0 = gpu.hs_image_direct(1.2, 0.9, tri, nrm, *dens, x)
    assert ier == 0 and gpu.hs_capped() > 0
    ier, _, u, e = gpu.elhfmm3dtriatargiter(2, 1.2, 0.9, tri, nrm, tri.mean(axis=1), *dens, x)
    assert ier == 0 and gpu.hs_capped() > 0
    # both subdivide until a patch repeats to 1e-6 of itself or is capped; they
    # differ where one accepts a patch that the other halves again.  The image
    # cancels against itself at the surface, to about a hundredth of the patches
    for a, b in ((u, u0), (e, e0)):
        assert np.abs(a - b).max() < 1e-4 * np.abs(b).max()
