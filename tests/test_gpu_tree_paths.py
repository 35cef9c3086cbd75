"""The tree and lists against the oracle's, bit for bit, where the builder
changes path: numbers of points around the partition's limit of 16,384 per
box (radix sort above), around its block sizes, boxes that hold nearly all
points at depth, list rows longer than a warp sorts (a coarse box of targets
beside hundreds of fine source boxes), and lists 3 and 4 that are empty."""
import numpy as np
import pytest

from elfmmlib3d_b200 import geometry as G

pytestmark = pytest.mark.gpu


def _check(gpu, oracle, src, tgt, iprec):
    import torch
    d = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
    P = gpu.Plan(0)
    n, m = len(src), len(tgt)
    P.set_geometry(d(np.zeros((n, 3, 3))), d(np.zeros((n, 3))), d(src), d(tgt) if m else None, iprec=iprec)
    T, nbox = P.tree(), P.info()["nbox"]
    P.close()
    O = oracle.Tree(src, tgt, nbox, False)
    assert len(T["boxes"]) == O.nboxes and np.array_equal(T["boxes"], O.boxes)
    assert np.array_equal(T["iz"], O.iz) and np.array_equal(T["iztarg"], O.iztarg)
    longest = 0
    for k in range(1, 6):
        for a, b in zip(T["lists"][k], O.lists[k]):
            assert np.array_equal(np.sort(a), np.sort(b))
            longest = max(longest, len(a))
    return longest


@pytest.mark.parametrize("n,m", [(33, 0), (64, 65), (96, 97), (513, 20), (1024, 1025), (16384, 100), (16385, 16384), (40001, 17000)])
def test_uniform_points(gpu, oracle, n, m):
    rng = np.random.default_rng(n)
    _check(gpu, oracle, rng.uniform(-1, 1, (n, 3)), rng.uniform(-1, 1, (m, 3)), 1)


def test_deep_cluster_above_the_partition_limit(gpu, oracle):
    rng = np.random.default_rng(3)
    src = np.vstack([rng.uniform(0, 1, (50, 3)), 0.3 + 1e-3 * rng.uniform(0, 1, (20000, 3))])
    _check(gpu, oracle, src, rng.uniform(0, 1, (40, 3)), 2)


def test_shell_and_few_targets(gpu, oracle):
    rng = np.random.default_rng(4)
    v = rng.normal(size=(60000, 3))
    src = v / np.linalg.norm(v, axis=1)[:, None]
    _check(gpu, oracle, src, rng.uniform(1.0, 1.9, (30, 3)), 1)


def sheet_beside_coarse_box():
    """Sources on a sheet along one face of an octant that holds 3 targets."""
    rng = np.random.default_rng(5)
    yz = rng.uniform(0, 0.5, (60000, 2))
    src = np.vstack([[[0, 0, 0], [1, 1, 1]], np.column_stack([np.full(len(yz), 0.5 + 1e-6), yz])])
    return src, rng.uniform(0.1, 0.4, (3, 3))


def test_long_list_rows(gpu, oracle):
    src, tgt = sheet_beside_coarse_box()
    assert _check(gpu, oracle, src, tgt, 1) > 512
