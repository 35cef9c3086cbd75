"""The mixed form of few right-hand sides: the same arithmetic as in a batch
of many, and the same engine of the FP32 translations pass by pass."""
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


def _decide(L, p, nbox, cols, winner):
    """Let the tuner hold `winner` (0 tensor cores, 1 CUDA cores) for the
    three FP32 translation stages of a free-space plan."""
    L.efmm_tune_report.restype = None
    L.efmm_tune_report.argtypes = [ctypes.c_int] * 8 + [ctypes.c_float]
    for knob in range(3):
        for cand in (0, 0, 1, 1):
            L.efmm_tune_report(knob, p, nbox, cols, 1, 0, 2, cand, 1.0 if cand == winner else 9.0)
        assert L.efmm_tune_pick(knob, p, nbox, cols, 1, 0, 2) == winner


def _plan(gpu, n, iprec):
    level = next(k for k in range(8) if 20 * 4 ** k >= n)
    tri, nrm, cen = (a[:n] for a in G.sphere_triangles(level))
    P = gpu.Plan(0)
    P.set_mixed_floor(0.0)  # the orders of the FP64 pass
    P.set_geometry(_dev(tri), _dev(nrm), _dev(cen), _dev(G.shell_targets(500, 5)), iprec=iprec)
    assert P.info()["far"]
    return P


@pytest.mark.parametrize("iprec,n", [(1, 5120), (2, 5120), (2, 20480)])
@pytest.mark.parametrize("nrhs", [1, 2, 4])
def test_few_right_hand_sides_as_in_a_batch(gpu, iprec, n, nrhs):
    """Every right-hand side of a mixed pass has its multipoles from the unit
    multipoles' product, whatever the number of right-hand sides: a few alone
    differ from the same ones in a batch of 7 (the largest whose local
    expansions are evaluated point by point, as theirs are) by the order of the
    FP32 atomics of the translations only, which two passes over the same
    inputs show as well (four times that allowed; a P2M of other arithmetic
    differs by 5 to 10 times)."""
    P = _plan(gpu, n, iprec)
    info, big = P.info(), 7
    gpu.load().efmm_tune_reset()
    for R in (nrhs, big):
        _decide(gpu.load(), info["p"], info["nbox"], 4 * R, 1)
    rng = np.random.default_rng(n + iprec)
    ssl, sdl = rng.normal(size=(2, big, n, 3))
    outs = []
    for R in (nrhs, nrhs, big):
        o = [_zeros(R, n, 3), _zeros(R, n, 3, 3), _zeros(R, 500, 3), _zeros(R, 500, 3, 3)]
        P.evaluate_batch(1.3, 0.7, R, _dev(ssl[:R]), _dev(sdl[:R]), *o, precision=1)
        outs.append([t[:nrhs].cpu().numpy() for t in o])
    P.close()
    gpu.load().efmm_tune_reset()
    for few, again, many in zip(*outs):
        assert rel(few, many) < 4.0 * rel(few, again)


def _passes(gpu, P, n, R, count, seed=3, **more):
    rng = np.random.default_rng(seed)
    ssl, sdl = (_dev(a) for a in rng.normal(size=(2, R, n, 3)))
    outs = []
    for _ in range(count):
        o = [_zeros(R, n, 3), _zeros(R, n, 3, 3), _zeros(R, 500, 3), _zeros(R, 500, 3, 3)]
        P.evaluate_batch(1.3, 0.7, R, ssl, sdl, *o, precision=1, **more)
        outs.append([t.cpu().numpy() for t in o])
    return outs


@pytest.mark.parametrize("nrhs", [1, 5])
def test_first_passes_run_the_tuner_s_candidates(gpu, nrhs):
    """The passes of an undecided key run the tensor-core translations twice,
    then the CUDA-core ones twice, and a graph captured while undecided holds
    the tensor cores.  The engine of a pass shows in its rounding: its outputs
    are nearer to those of the same engine decided (they differ by the order of
    the FP32 atomics, 1e-7) than to the other's (4e-7 and more)."""
    n, L = 20480, gpu.load()
    P = _plan(gpu, n, 2)
    info = P.info()
    key = (info["p"], info["nbox"], 4 * nrhs)
    ref = []
    for cand in (0, 1):
        L.efmm_tune_reset()
        _decide(L, *key, cand)
        ref.append(_passes(gpu, P, n, nrhs, 1)[0])
    engine = lambda o: int(np.argmin([sum(rel(a, b) for a, b in zip(o, r)) for r in ref]))  # noqa: E731
    L.efmm_tune_reset()
    assert [engine(o) for o in _passes(gpu, P, n, nrhs, 4)] == [0, 0, 1, 1]
    L.efmm_tune_reset()
    assert engine(_passes(gpu, P, n, nrhs, 1, graph=True)[0]) == 0
    lines = [line.split() for line in gpu.tune_dump()]  # the pass before the capture reported, undecided
    assert [(int(q[0]), int(q[3]), int(q[6])) for q in lines] == [(knob, 4 * nrhs, -1) for knob in range(3)]
    P.close()
    L.efmm_tune_reset()
