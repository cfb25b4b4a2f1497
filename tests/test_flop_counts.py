"""The operation counts that the benchmark's rooflines use, counted anew on the device
math with the benchmark's meshes."""
import json
import os
import shutil
import subprocess

import pytest

import bench
from pyquake3d_gb300 import mesh

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("half,shape,count", [(0, (80.0, 30.0, 200, 50), "GF_FLOP_PER_PAIR"),
                                              (1, (40.0, 20.0, 50, 25), "HS_FLOP_PER_PAIR")])
def test_tile_counts(tmp_path, half, shape, count):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.fail("no C++ compiler for the operation count")
    exe = str(tmp_path / "count")
    subprocess.run([cxx, "-O2", "-std=c++17", "-o", exe, os.path.join(REPO, "oracle", "count_tile_flops.cpp")], check=True)
    nodes, tris = mesh.rough_fault(*shape, hurst=0.8, ratio=1e-3, seed=0)
    inp = "%d %d\n" % (half, len(tris)) + "\n".join(" ".join("%.17g" % v for v in nodes[t - 1].ravel()) for t in tris)
    out = json.loads(subprocess.run([exe], input=inp, capture_output=True, text=True, check=True).stdout)
    assert round(out["flops_per_pair"]) == getattr(bench, count)
