"""Other calls between two replays of a captured pass: they may refill the
work lists and move the buffers that it reads.  The next graph call returns
what the plain call returns, and does not capture anew where nothing moved."""
import numpy as np
import pytest

from conftest import rel
from elfmmlib3d_b200 import geometry as G

pytestmark = pytest.mark.gpu
SAME = 1e-12  # FP64 sums in another order


def _dev(a):
    import torch
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _zeros(*s):
    import torch
    return torch.zeros(s, dtype=torch.float64, device="cuda")


class Case:
    """A plan with stored near field, densities for up to 40 right-hand sides."""

    def __init__(self, gpu, kind, iprec=2):
        self.gpu, self.image, rng = gpu, kind == "image", np.random.default_rng(2)
        if self.image:
            tri, nrm, cen, _ = G.planar_fault(24, 12)
            tgt = cen * np.array([1, 1, -1.0])
        else:
            tri, nrm, cen = G.sphere_triangles(3)
            tgt = G.shell_targets(333, 4)
        self.n, self.m = len(cen), len(tgt)
        self.P = gpu.Plan(0)
        self.P.set_geometry(_dev(tri), _dev(nrm), _dev(cen), _dev(tgt), iprec=iprec, iter=True, mindlin=self.image)
        self.dens = rng.normal(size=(2, 40, self.n, 3))
        self.buf = {}

    def run(self, R, mode, precision=0, graph=False, lam=1.2, one=False):
        """Outputs of the call, from buffers kept per R (a graph's key)."""
        if R not in self.buf:
            o = [] if self.image else [_zeros(R, self.n, 3), _zeros(R, self.n, 3, 3)]
            self.buf[R] = ([_dev(a[:R]) for a in self.dens], o + [_zeros(R, self.m, 3), _zeros(R, self.m, 3, 3)])
        dens, out = self.buf[R]
        for t in out:
            t.fill_(7.0)
        if one:
            self.P.evaluate(lam, 0.9, dens[0][0], dens[1][0], *[t[0] for t in out], mode=mode)
        elif self.image:
            self.P.evaluate_image(lam, 0.9, R, *dens, *out, precision=precision, mode=mode, graph=graph)
        else:
            self.P.evaluate_batch(lam, 0.9, R, *dens, *out, precision=precision, mode=mode, graph=graph)
        return [t.cpu().numpy() for t in out]

    def graph(self, R, mode, precision=0, lam=1.2):
        """A graph call and the kernels it launched."""
        l0 = self.gpu.kernel_launches()
        return self.run(R, mode, precision, True, lam), self.gpu.kernel_launches() - l0


def _same(a, b, tol=SAME):
    for x, y in zip(a, b):
        assert rel(x, y) < tol


@pytest.mark.parametrize("iprec", [2, 5])  # a far field, a near field only
@pytest.mark.parametrize("R", [3, 16])
def test_plain_calls_of_the_other_mode_between_replays(gpu, iprec, R):
    c = Case(gpu, "free", iprec)
    c.run(R, 1)
    for mode in (2, 0):
        plain = c.run(R, mode)
        first, _ = c.graph(R, mode)
        _, once = c.graph(R, mode)
        _same(first, plain)
        c.run(R, 2 - mode)  # the other tiling of the near field's work items
        _same(c.graph(R, mode)[0], plain)
        c.run(R, 2 - mode)
        got, k = c.graph(R, mode)
        _same(got, plain)
        assert k == once  # both tilings are there, nothing moved: the captured pass has stayed
        c.run(R, 0, one=True)
        c.run(R, 1)
        _same(c.graph(R, mode)[0], plain)
        c.P.evaluate(1.2, 0.9, *[d[0] for d in c.buf[R][0]], *[t[0] for t in c.buf[R][1]], direct=True)
        _same(c.graph(R, mode)[0], plain)


@pytest.mark.parametrize("kind,mode", [("free", 0), ("free", 2), ("image", 2)])
@pytest.mark.parametrize("R,other", [(3, 9), (9, 3), (2, 40)])
def test_other_numbers_of_right_hand_sides_between_replays(gpu, kind, mode, R, other):
    c = Case(gpu, kind)
    c.run(R, 1)
    plain = c.run(R, mode)
    _same(c.graph(R, mode)[0], plain)
    want = c.run(other, mode)
    _same(c.graph(R, mode)[0], plain)
    _same(c.run(other, mode), want)
    _same(c.graph(R, mode)[0], plain)
    _same(c.graph(other, mode)[0], want)
    _same(c.graph(R, mode)[0], plain)


@pytest.mark.parametrize("kind", ["free", "image"])
def test_another_store_between_replays(gpu, kind):
    """Mode 2 needs the store of its own parameters, captured or not."""
    c = Case(gpu, kind)
    c.run(3, 1)
    plain = c.run(3, 2)
    _same(c.graph(3, 2)[0], plain)
    c.run(3, 1, lam=2.0)
    for graph in (False, True):
        with pytest.raises(gpu.ElfmmError):
            c.run(3, 2, graph=graph)
    other = c.run(3, 2, lam=2.0)
    _same(c.graph(3, 2, lam=2.0)[0], other)
    c.run(3, 1)
    _same(c.graph(3, 2)[0], plain)


@pytest.mark.parametrize("R", [3, 16])
def test_mixed_and_plain_calls_between_replays(gpu, R):
    """Mixed: the resident operands of a captured pass and those that a plain
    pass makes for itself share buffers; FP64 passes release them.  FP32 sums
    in another order: 1e-6."""
    c = Case(gpu, "free", 3)
    c.run(R, 1, 1)
    for mode in (2, 0):
        plain = c.run(R, mode, 1)
        _same(c.graph(R, mode, 1)[0], plain, 1e-6)
        for between in ((R, 2 - mode, 1), (R, mode, 0), (5, mode, 1), (R, 1, 1)):
            c.run(*between)
            _same(c.graph(R, mode, 1)[0], plain, 1e-6)
            _same(c.graph(R, mode, 1)[0], plain, 1e-6)
