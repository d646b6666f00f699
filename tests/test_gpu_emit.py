"""Node emission against the oracle where its words differ: rows of one word
and of several, flat faces whose words are all surface nodes, materials that
change from triangle to triangle, no materials, and partitions whose faces
are cleared.  Integer fields equal; PartialNode ratios within the oracle's
stated tolerance."""

import numpy as np
import pytest

import oracle as O
from helpers import PARTIAL, RATIO_TOL, RATIO_UNSTABLE, masked, ratio_bad
from voxelizer_b200.api import LONG, LONG_FCC, SHORT, SHORT_FCC, Voxelizer
from voxelizer_b200.scenes import Mesh, _box_shell, icosphere, random_rotation, torus, transform

pytestmark = pytest.mark.gpu

MESHES = {
    "box": lambda: _box_shell((0, 0, 0), (1.0, 0.7, 0.45)),
    "tall_box": lambda: _box_shell((0, 0, 0), (0.2, 1.0, 0.9)),
    "torus": lambda: (transform(torus(48, 24)[0], random_rotation(np.random.default_rng(3))), torus(48, 24)[1]),
    "ico": lambda: icosphere(3),
}
KINDS = {"short": SHORT, "long": LONG, "partial": PARTIAL, "short_fcc": SHORT_FCC, "long_fcc": LONG_FCC}


def _mesh(name):
    v, f = MESHES[name]()
    ext = float((v.max(0) - v.min(0)).max())
    return Mesh(v, f, (1 + np.arange(f.shape[0]) % 7).astype(np.uint8), 8), ext


def _check(kind, got, want, conf):
    got, want = masked(kind, 1, got), masked(kind, 1, want)
    if kind == PARTIAL and conf is not None:
        low = np.uint64(0xFFFFFFFF)
        assert np.array_equal(got & low, want & low)
        stable = np.nonzero((conf & RATIO_UNSTABLE) == 0)[0]
        assert ratio_bad(got[stable], want[stable], RATIO_TOL).size == 0
    else:
        assert np.array_equal(got, want)


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("mesh,cells", [("box", 25), ("box", 63), ("tall_box", 75), ("torus", 41), ("ico", 97)])
@pytest.mark.parametrize("mats", [1, 0])
def test_grid(kind, mesh, cells, mats):
    m, ext = _mesh(mesh)
    k, size, vox = KINDS[kind], ext / cells, (1024, 31, 512)
    want, _, conf = O.voxelize(m, k, 1, mats, size, vox, want_conflicts=True)
    with Voxelizer(m.vertices, m.indices, m.materials if mats else None, 8, node_type=k) as vx:
        got, _ = vx.voxelizeToNodesToRAM(size, vox)
    _check(k, got, want, conf if mats else None)


@pytest.mark.parametrize("kind", list(KINDS))
def test_partitions(kind):
    m, ext = _mesh("torus")
    k, size = KINDS[kind], ext / 45
    with Voxelizer(m.vertices, m.indices, m.materials, 8, node_type=k) as vx:
        parts = vx.voxelizePartsToRAM(1, size, (3, 2))
    for got, info in parts:
        want, _, conf = O.voxelize(m, k, 1, 1, size, part=tuple(int(x) for x in info.partition), want_conflicts=True)
        _check(k, got, want, conf)
