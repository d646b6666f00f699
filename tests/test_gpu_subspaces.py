"""Solid pass over grids of yz subspaces of a few rows, uneven ones among them,
whose cuts fall inside and between 4x4 tiles and outside of most triangles:
bit arrays against the oracle, equal."""

import numpy as np
import pytest

import oracle as O
from voxelizer_b200.api import LONG, SHORT, Voxelizer
from voxelizer_b200.scenes import Mesh, _box_shell, icosphere, random_rotation, torus, transform

pytestmark = pytest.mark.gpu

MESHES = {
    "ico4": lambda: icosphere(4),
    "torus_turned": lambda: (transform(torus(24, 12)[0], random_rotation(np.random.default_rng(7))), torus(24, 12)[1]),
    "box_turned": lambda: (transform(_box_shell((0, 0, 0), (1, 2, 3))[0], random_rotation(np.random.default_rng(8))),
                           _box_shell((0, 0, 0), (1, 2, 3))[1]),
}


@pytest.mark.parametrize("mesh", list(MESHES))
@pytest.mark.parametrize("vox", [(1024, 1, 512), (1024, 512, 1), (1024, 3, 5), (64, 7, 4), (1024, 30, 512), (1024, 13, 29)])
@pytest.mark.parametrize("dim", [40, 151])
def test_bits_match_oracle(mesh, vox, dim):
    v, f = MESHES[mesh]()
    want = O.voxelize(Mesh(v, f), SHORT, 0, 0, dim, vox)[0]
    with Voxelizer(v, f, node_type=SHORT) as vx:
        got, _ = vx.voxelizeToRAM(dim, vox)
    assert np.array_equal(got, want)


def test_many_subspaces_cost_little():
    """A box wall of 4,096 rows each way: 4,225 subspaces against 81."""
    import time
    import torch

    v, f = _box_shell((0, 0, 0), (0.004, 1, 1))
    took = []
    with Voxelizer(v, f, node_type=LONG) as vx:
        for vox in ((1024, 512, 512), (1024, 64, 64)):
            out = torch.empty(int(vx.plan(0, 4096, vox).count), dtype=torch.int32, device="cuda")
            best = 1.0
            for _ in range(4):
                torch.cuda.synchronize()
                start = time.perf_counter()
                vx.voxelize_device(0, 4096, out, vox)
                torch.cuda.synchronize()
                best = min(best, time.perf_counter() - start)
            took.append(best)
    # With each subspace looked at per candidate, 50 times as long.
    assert took[1] < 12 * took[0]
