"""Surface pass against the oracle where its rows differ: rows of one and of
several 32-column segments, flat triangles (2D boxes), lines (1D boxes) and
tilted ones of each dominant axis, and material subspaces that cut the columns
and their depth ranges.  Integer fields equal; PartialNode ratios within the
oracle's stated tolerance.  Also: instances made and destroyed by several
threads, whose streams come from one list."""

import threading

import numpy as np
import pytest

import oracle as O
from helpers import PARTIAL, RATIO_TOL, RATIO_UNSTABLE, masked, ratio_bad
from voxelizer_b200 import _lib
from voxelizer_b200.api import LONG, SHORT, SHORT_FCC, Voxelizer
from voxelizer_b200.scenes import Mesh, _box_shell, icosphere, random_rotation, transform

pytestmark = pytest.mark.gpu


def _tilted(seed):
    v, f = _box_shell((0, 0, 0), (1.0, 0.8, 0.6))
    return transform(v, random_rotation(np.random.default_rng(seed))), f


MESHES = {
    "box": lambda: _box_shell((0, 0, 0), (1.0, 0.8, 0.6)),
    "tilted0": lambda: _tilted(0),
    "tilted5": lambda: _tilted(5),
    "rod_x": lambda: _box_shell((0, 0, 0), (1.0, 0.003, 0.002)),
    "rod_z": lambda: _box_shell((0, 0, 0), (0.003, 0.002, 1.0)),
}
KINDS = {"short": SHORT, "long": LONG, "partial": PARTIAL, "short_fcc": SHORT_FCC}


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("mesh", list(MESHES))
@pytest.mark.parametrize("cells,mat", [(31, 512), (32, 512), (33, 17), (64, 512), (65, 23)])
def test_rows(kind, mesh, cells, mat):
    v, f = MESHES[mesh]()
    m = Mesh(v, f, (1 + np.arange(f.shape[0]) % 7).astype(np.uint8), 8)
    k, size, split = KINDS[kind], float((v.max(0) - v.min(0)).max()) / cells, (mat, mat, mat)
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


@pytest.mark.parametrize("threads", [1, 6])
def test_streams_of_many_instances(threads):
    v, f = icosphere(3)
    m = Mesh(v, f, (1 + np.arange(f.shape[0]) % 7).astype(np.uint8), 8)
    sizes = [2.0 / 40, 2.0 / 150]
    want = [masked(LONG, 1, O.voxelize(m, LONG, 1, 1, s)[0]) for s in sizes]
    bad = []

    def work(t):
        for i in range(6):
            with Voxelizer(m.vertices, m.indices, m.materials, 8, node_type=LONG) as vx:
                got, _ = vx.voxelizeToNodesToRAM(sizes[(t + i) % 2])
            if not np.array_equal(masked(LONG, 1, got), want[(t + i) % 2]):
                bad.append((t, i))
            if i == 3 and t == 0:
                _lib.lib().vxb_trim_cache()

    pool = [threading.Thread(target=work, args=(t,)) for t in range(threads)]
    for p in pool:
        p.start()
    for p in pool:
        p.join()
    assert not bad
