"""Thin, tall grids and uneven batches against the oracle: more planes along z
than a launch may have blocks along y (65,535), by themselves, in a batch and
streamed to page-locked host memory, and batches whose units differ much in
planes and in words per plane.  Integer fields equal."""

import numpy as np
import pytest

import oracle as O
from helpers import masked
from voxelizer_b200.api import LONG, SHORT, Voxelizer, VoxelizerBatch
from voxelizer_b200.scenes import Mesh, _box_shell, icosphere

pytestmark = pytest.mark.gpu


def _rod(cells, width):
    v, f = _box_shell((0, 0, 0), (width / cells, width / cells, 1.0))
    return Mesh(v, f, (1 + np.arange(f.shape[0]) % 7).astype(np.uint8), 8)


def _ico(level):
    v, f = icosphere(level)
    return Mesh(v, f, (1 + np.arange(f.shape[0]) % 7).astype(np.uint8), 8)


def _open(m, kind, mats=1):
    return Voxelizer(m.vertices, m.indices, m.materials if mats else None, 8, node_type=kind)


@pytest.mark.parametrize("kind", [SHORT, LONG])
@pytest.mark.parametrize("mats", [1, 0])
def test_more_planes_than_blocks_along_y(kind, mats):
    m, dim = _rod(70_000, 2.4), 70_000
    want = O.voxelize(m, kind, 1, mats, dim)[0]
    with _open(m, kind, mats) as vx:
        got, info = vx.voxelizeToNodesToRAM(dim)
    assert info.dims[2] > 65_535
    assert np.array_equal(masked(kind, 1, got), masked(kind, 1, want))


def test_more_planes_than_blocks_along_y_streamed():
    """Page-locked output: four ranges of planes, each more than 65,535."""
    import torch

    m, dim = _rod(270_000, 0.4), 270_000
    want = O.voxelize(m, SHORT, 1, 1, dim)[0]
    with _open(m, SHORT) as vx:
        info = vx.plan(1, dim)
        out = torch.empty(int(info.bytes), dtype=torch.uint8).pin_memory()
        vx.voxelizeToNodesToRAM(dim, out=out.numpy())
    assert np.array_equal(masked(SHORT, 1, out.numpy()), masked(SHORT, 1, want))


@pytest.mark.parametrize("kind", [SHORT, LONG])
@pytest.mark.parametrize("tall", [4_000, 70_000])
def test_uneven_batch(kind, tall):
    import torch

    meshes = [_ico(1), _rod(tall, 1.7), _ico(2), _ico(4)] + [_ico(1)] * 12
    dims = [9, tall, 33, 150] + [8 + i for i in range(12)]
    vx = [_open(m, kind) for m in meshes]
    outs = []
    with VoxelizerBatch() as b:
        for x, d in zip(vx, dims):
            outs.append(torch.zeros(int(x.plan(1, d).bytes), dtype=torch.uint8, device="cuda"))
            b.add(x, 1, d, outs[-1])
        for graph in (False, True):
            b.run(graph=graph)
            for m, d, out in zip(meshes, dims, outs):
                want = O.voxelize(m, kind, 1, 1, d)[0]
                got = out.cpu().numpy().view(want.dtype)
                assert np.array_equal(masked(kind, 1, got), masked(kind, 1, want))
                out.zero_()
    for x in vx:
        x.close()
