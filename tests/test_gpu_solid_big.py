"""Solid pass of few triangles with very many candidates: three nested boxes of
8,192 x 8,192 rows list 0.8 M chunks of 64 candidates from 12 triangles.  Toggles
are exclusive-ors, so the grid of the three boxes is that of the single ones
combined, and its time about the sum of theirs."""

import time

import numpy as np
import pytest

from voxelizer_b200.api import LONG, Voxelizer
from voxelizer_b200.scenes import _box_shell

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _nested():
    vs, fs = [], []
    for k in range(3):
        v, f = _box_shell((0.0005 * k, 0.01 * k, 0.01 * k), (0.003 - 0.0005 * k, 1 - 0.01 * k, 1 - 0.01 * k))
        vs.append(v)
        fs.append(f + 8 * k)
    v = np.concatenate(vs)
    assert v.shape[0] == 24
    return v, fs


def test_few_triangles_many_candidates():
    v, boxes = _nested()

    def run(f):
        """The grid and the seconds of the fastest call.  All grids have
        all vertices, so they have the same bounding box."""
        with Voxelizer(v, f, node_type=LONG) as vx:
            out = torch.empty(int(vx.plan(0, 8192).count), dtype=torch.int32, device="cuda")
            best = 100.0
            for _ in range(3):
                torch.cuda.synchronize()
                start = time.perf_counter()
                vx.voxelize_device(0, 8192, out)
                torch.cuda.synchronize()
                best = min(best, time.perf_counter() - start)
        return out, best

    all_boxes, took = run(np.concatenate(boxes))
    alone = [run(f) for f in boxes]
    want = alone[0][0] ^ alone[1][0] ^ alone[2][0]
    assert int(torch.count_nonzero(want)) > 60_000_000
    assert torch.equal(all_boxes, want)
    # One warp that walked a triangle's four million candidates alone would
    # take a hundred times as long.
    assert took < 20 * sum(t for _, t in alone)
