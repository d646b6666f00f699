"""Surface pass of triangles whose boxes are lines of voxels: lengths around
multiples of 32 and long ones, along each axis, cut by material subspaces and by
the grid, against the oracle; and the time of long ones.  Integer fields equal;
PartialNode ratios within the oracle's stated tolerance."""

import time

import numpy as np
import pytest

import oracle as O
from helpers import PARTIAL, RATIO_TOL, RATIO_UNSTABLE, masked, ratio_bad
from voxelizer_b200.api import LONG, SHORT, Voxelizer
from voxelizer_b200.scenes import Mesh, _box_shell

pytestmark = pytest.mark.gpu

KINDS = {"short": SHORT, "long": LONG, "partial": PARTIAL}


def _rod(axis, cells):
    v, f = _box_shell((0, 0, 0), tuple(1.0 if a == axis else 0.3 / cells for a in range(3)))
    return Mesh(v, f, (1 + np.arange(f.shape[0]) % 7).astype(np.uint8), 8)


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("cells,mat", [(1, 512), (30, 512), (31, 512), (32, 7), (63, 512), (64, 33), (1000, 100), (3001, 512)])
def test_lines(kind, axis, cells, mat):
    m, k, size, split = _rod(axis, cells), KINDS[kind], 1.0 / cells, (mat, mat, mat)
    want, _, conf = O.voxelize(m, k, 1, 1, size, (1024, 512, 512), split, want_conflicts=True)
    with Voxelizer(m.vertices, m.indices, m.materials, 8, node_type=k) as vx:
        got, _ = vx.voxelizeToNodesToRAM(size, (1024, 512, 512), split)
    got, want = masked(k, 1, got), masked(k, 1, want)
    if k != PARTIAL:
        assert np.array_equal(got, want)
        return
    low = np.uint64(0xFFFFFFFF)
    assert np.array_equal(got & low, want & low)
    stable = np.nonzero((conf & RATIO_UNSTABLE) == 0)[0]
    assert ratio_bad(got[stable], want[stable], RATIO_TOL).size == 0


def test_long_lines_are_shared_out():
    import torch

    m, took = _rod(1, 60_000), []
    for mats in (None, m.materials):
        with Voxelizer(m.vertices, m.indices, mats, 8, node_type=LONG) as vx:
            out = torch.empty(int(vx.plan(1, 60_000).bytes), dtype=torch.uint8, device="cuda")
            best = 1.0
            for _ in range(5):
                torch.cuda.synchronize()
                start = time.perf_counter()
                vx.voxelize_device(1, 60_000, out)
                torch.cuda.synchronize()
                best = min(best, time.perf_counter() - start)
        took.append(best)
    # One lane that takes a line of 60,000 voxels: 50 times as long.
    assert took[1] < 10 * took[0]
