"""An instance destroyed while a CUDA graph is being captured, in the capturing
thread (as when garbage collection runs then) or in another one: its streams go
back to the list of idle ones and the capture goes on."""

import threading

import numpy as np
import pytest

from voxelizer_b200.api import LONG, Voxelizer, VoxelizerBatch
from voxelizer_b200.scenes import icosphere

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _used_instance():
    v, f = icosphere(3)
    vx = Voxelizer(v, f, np.ones(f.shape[0], np.uint8), 2, node_type=LONG)
    vx.voxelizeToNodesToRAM(40)
    return vx


def _used_batch():
    v, f = icosphere(2)
    vx = Voxelizer(v, f, np.ones(f.shape[0], np.uint8), 2, node_type=LONG)
    b = VoxelizerBatch()
    b.add(vx, 1, 30, torch.zeros(int(vx.plan(1, 30).bytes), dtype=torch.uint8, device="cuda"))
    b.run(graph=True)
    return b


@pytest.mark.parametrize("make", [_used_instance, _used_batch])
@pytest.mark.parametrize("thread", ["same", "other"])
@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
def test_destroyed_during_a_capture(make, thread, mode):
    x = torch.ones(1000, device="cuda")
    used = make()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(torch.cuda.Stream()):
        g.capture_begin(capture_error_mode=mode)
        try:
            y = x + 1
            if thread == "same":
                used.close()
            else:
                t = threading.Thread(target=used.close)
                t.start()
                t.join()
            z = y + 1
        finally:
            g.capture_end()
    g.replay()
    torch.cuda.synchronize()
    assert float(z.sum()) == 3000.0
