"""The moment form of the half-space image kernels (image_moments.cuh, which
the image near field integrates: monomials of R over powers of r accumulated
per node, assembled once per pair) against the generated straight-line
kernels (mindlin_gen.cuh), on the host: single nodes, weighted sums of nodes,
deep and shallow targets and sources, near-vertical offsets (R1 = R2 = 0,
where the angular moments of U vanish).  No device is used."""
import ctypes

import numpy as np
import pytest

_dp = ctypes.POINTER(ctypes.c_double)
D = ctypes.c_double
I = ctypes.c_int


def _p(a):
    return a.ctypes.data_as(_dp)


@pytest.mark.parametrize("layer,strain", [(0, 1), (0, 0), (1, 1), (1, 0)])
@pytest.mark.parametrize("depth_x,depth_s,offset", [(1.0, 1.0, 2.0), (1e-3, 3.0, 1.0), (5.0, 1e-3, 1.0), (2.0, 1.0, 0.0),
                                                    (0.5, 0.5, 40.0)])
def test_moments_match_generated_kernels(lib, layer, strain, depth_x, depth_s, offset):
    L = ctypes.CDLL(lib.library_path())
    rng = np.random.default_rng(5)
    worst = 0.0
    for nnode in (1, 12):
        for _ in range(20):
            lam, mu = rng.uniform(0.2, 3.0, 2)
            x = np.array([*rng.uniform(-1, 1, 2) * offset, -depth_x * rng.uniform(0.5, 1)])
            s = np.stack([np.array([*(x[:2] + offset * rng.uniform(-1, 1, 2)), -depth_s * rng.uniform(0.5, 1)])
                          for _ in range(nnode)])
            w = rng.uniform(0.1, 1.0, nnode)
            n = rng.normal(size=3)
            n /= np.linalg.norm(n)
            ref, one, out = np.zeros(27), np.zeros(27), np.zeros(27)
            for q in range(nnode):
                assert L.efmm_mindlin_image_kernel(I(layer), D(lam), D(mu), _p(x), _p(s[q]), _p(n), _p(one)) == 0
                ref += w[q] * one
            assert L.efmm_mindlin_image_moments(I(layer), I(strain), D(lam), D(mu), _p(x), I(nnode), _p(s), _p(w), _p(n),
                                                _p(out)) == 0
            for k in range(3):
                for blk in [slice(9 * k, 9 * k + 3)] + ([slice(9 * k + 3, 9 * k + 9)] if strain else []):
                    worst = max(worst, np.abs(out[blk] - ref[blk]).max() / np.abs(ref[blk]).max())
    # both forms add a few hundred terms of the size of the largest response
    # of the pair (kernel size ~ 1 / r^n), each rounded to 2^-53
    assert worst < 1e-11, worst


def test_moments_reject_bad_arguments(lib):
    L = ctypes.CDLL(lib.library_path())
    x, out = np.array([0.0, 0.0, -1.0]), np.zeros(27)
    w = np.ones(1)
    assert L.efmm_mindlin_image_moments(I(2), I(1), D(1), D(1), _p(x), I(1), _p(x), _p(w), _p(x), _p(out)) == 16
    assert L.efmm_mindlin_image_moments(I(1), I(1), D(1), D(1), _p(x), I(0), _p(x), _p(w), _p(x), _p(out)) == 16
    assert L.efmm_mindlin_image_moments(I(1), I(1), D(1), D(1), _p(x), I(1), _p(x), _p(w), None, _p(out)) == 16
