"""The mesh build's edge angles on triangles that lie on one another, with every array index checked."""
import os
import subprocess

from rocketgpu_b200 import build
from tests.test_host_paths import CSRC, ROOT


def test_edges_of_coincident_triangles_stay_in_bounds(tmp_path):
    out = str(tmp_path / "mesh_edges")
    cuda = os.path.dirname(os.path.dirname(build.nvcc()))
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=bounds", "-fsanitize-undefined-trap-on-error", "-w", "-I", CSRC,
                    "-I", os.path.join(ROOT, "include"), "-I", os.path.join(cuda, "include"),
                    os.path.join(ROOT, "tests", "mesh_edges.cpp"), os.path.join(CSRC, "rg_mesh.cpp"), "-o", out,
                    "-L", os.path.join(cuda, "lib64"), "-lcudart", "-Wl,-rpath," + os.path.join(cuda, "lib64")],
                   check=True)
    assert subprocess.run([out]).returncode == 0
