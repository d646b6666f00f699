"""The solid pass's work split against the oracle: batches of 1 to 32
triangles per warp, batches whose candidates are listed in chunks (few huge
triangles, many medium ones), subspaces that cut tiles, and units of
different meshes inside one batch of triangles.  Bit arrays are integers and
must be equal."""

import numpy as np
import pytest

import oracle as O
from voxelizer_b200.api import LONG, SHORT, Voxelizer, VoxelizerBatch
from voxelizer_b200.scenes import Mesh, icosphere, torus, transform, _box_shell

pytestmark = pytest.mark.gpu


def _turned(v, seed):
    from voxelizer_b200.scenes import random_rotation

    return transform(v, random_rotation(np.random.default_rng(seed)))


CASES = {
    # triangles per warp: 1 (12 and 576 triangles), 4, 8 and 32
    "box": (lambda: _box_shell((0, 0, 0), (3.0, 2.0, 1.0)), 301, (1024, 512, 512)),
    "box_split": (lambda: _box_shell((0, 0, 0), (1.0, 2.0, 3.0)), 203, (1024, 61, 37)),
    "tetra_turned": (lambda: (_turned(_box_shell((0, 0, 0), (1.0, 1.0, 1.0))[0], 5),
                              _box_shell((0, 0, 0), (1.0, 1.0, 1.0))[1]), 257, (512, 512, 512)),
    "torus_576": (lambda: (_turned(torus(24, 12)[0], 1), torus(24, 12)[1]), 33, (1024, 512, 512)),
    "ico4": (lambda: icosphere(4), 190, (192, 96, 100)),
    "ico5_listed": (lambda: icosphere(5), 611, (1024, 512, 512)),
    "ico6_small": (lambda: icosphere(6), 27, (1024, 512, 512)),
}


@pytest.mark.parametrize("name", list(CASES))
def test_bits_match_oracle(name):
    make, dim, vox = CASES[name]
    v, f = make()
    mesh = Mesh(v, f)
    want, _, _ = O.voxelize(mesh, SHORT, 0, 0, dim, vox)
    with Voxelizer(mesh.vertices, mesh.indices, node_type=SHORT) as vx:
        got, _ = vx.voxelizeToRAM(dim, vox)
    assert np.array_equal(got, want)


def test_batch_of_triangles_crosses_meshes():
    """Meshes of 12 and 80 triangles back to back beside one of 81,920 (32
    triangles per warp): a warp's triangles belong to several units."""
    import torch

    meshes = [icosphere(1), _box_shell((0, 0, 0), (1.0, 1.5, 0.7)), icosphere(6), icosphere(1),
              _box_shell((0, 0, 0), (2.0, 1.0, 1.0))]
    dims = [40, 150, 60, 25, 90]
    vx = [Voxelizer(v, f, node_type=LONG) for v, f in meshes]
    outs = []
    with VoxelizerBatch() as b:
        for x, d in zip(vx, dims):
            info = x.plan(0, d)
            outs.append(torch.zeros(int(info.count), dtype=torch.int32, device="cuda"))
            b.add(x, 0, d, outs[-1])
        b.run()
    for (v, f), d, out, x in zip(meshes, dims, outs, vx):
        want, _, _ = O.voxelize(Mesh(v, f), LONG, 0, 0, d)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
        x.close()
