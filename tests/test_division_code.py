"""The quotients and divisions of csrc/vxb_common.cuh and csrc/vxb_kernels.cuh
themselves, compiled into a program: operand ranges and set-up on the host, the
device functions against the plain operations over their whole ranges, and
meshes so small or large that the ranges do not hold, against the oracle."""

import os
import subprocess

import numpy as np
import pytest

import oracle as O
from helpers import masked
from voxelizer_b200.api import LONG, Voxelizer
from voxelizer_b200.build import ARCH
from voxelizer_b200.scenes import Mesh, _box_shell, icosphere, random_rotation, transform

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("division") / "division")
    subprocess.run(["nvcc", "-std=c++17", "-O2"] + ARCH + ["-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "voxelizer_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "division.cu"), "-o", exe], check=True)
    return exe


def _run(program, what):
    r = subprocess.run([program, what], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert " differ" in r.stdout


def test_ranges_and_set_up(program):
    _run(program, "host")


@pytest.mark.gpu
def test_device_functions(program):
    _run(program, "device")


MESHES = {"ico": lambda: icosphere(3),
          "tilted": lambda: (transform(_box_shell((0, 0, 0), (1.0, 0.8, 0.6))[0],
                                       random_rotation(np.random.default_rng(4))), _box_shell((0, 0, 0), (1, 1, 1))[1])}


# FP32: normals below 2^-60 from 1e-9 on, lengths below it from 1e-18 on, and
# above 2^60 for 1e10 and 1e18; FP64 ranges hold throughout.
@pytest.mark.gpu
@pytest.mark.parametrize("mesh", list(MESHES))
@pytest.mark.parametrize("scale", [1e-9, 1e-10, 1e-18, 1e-30, 1e10, 1e18])
@pytest.mark.parametrize("offset", [0.0, 3.0])
def test_meshes_out_of_range(mesh, scale, offset):
    v, f = MESHES[mesh]()
    v = ((np.asarray(v, np.float64) + offset) * scale).astype(np.float32)
    m = Mesh(v, f, (1 + np.arange(f.shape[0]) % 7).astype(np.uint8), 8)
    for nodes, mats in ((0, 0), (1, 1)):
        want = O.voxelize(m, LONG, nodes, mats, 40)[0]
        with Voxelizer(v, f, m.materials if mats else None, 8, node_type=LONG) as vx:
            got = (vx.voxelizeToNodesToRAM(40) if nodes else vx.voxelizeToRAM(40))[0]
        if nodes:
            got, want = masked(LONG, 1, got), masked(LONG, 1, want)
        assert np.array_equal(got, want)
