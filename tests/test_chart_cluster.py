"""The cluster chart smoother's layout on the host (tests/native/
chart_cluster_check.cpp): slabs, pairs and stores into the neighbouring CTAs
against 4-colour Gauss-Seidel on the whole vector, bit for bit (the updates are
the same FMA chains), on atlases with one row per CTA up to the largest charts a
cluster holds, odd sizes, charts with holes and charts smaller than a cluster."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(built_lib, tmp_path_factory):
    pkg = os.path.join(ROOT, "gradientdomaintextureprocessing_b200")
    exe = str(tmp_path_factory.mktemp("native") / "chart_cluster_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(pkg, "csrc"), "-I", os.path.join(ROOT, "include"),
                    "-I/usr/local/cuda/include", os.path.join(ROOT, "tests", "native", "chart_cluster_check.cpp"), "-L", pkg, "-lgdtp",
                    "-Wl,-rpath," + pkg, "-L/usr/local/cuda/lib64", "-lcudart", "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("mesh,width,height", [("torus", 128, 128), ("torus", 301, 277), ("icosphere", 256, 256), ("icosphere", 725, 611),
                                              ("icosphere", 1024, 1024), ("genus2", 256, 256), ("genus2", 643, 905)])
def test_layout_gives_the_colour_passes_bits(check, tmp_path, mesh, width, height):
    from gradientdomaintextureprocessing_b200 import meshgen
    if mesh == "torus":
        m = meshgen.torus_atlas(width, height)
    elif mesh == "icosphere":
        m = meshgen.icosphere_atlas(width, height, subdiv=5)
    else:
        m = meshgen.genus2_atlas(width, height, nu=176, nv=72)
    path = str(tmp_path / "m.gdm")
    meshgen.write_gdm(path, m)
    for sweeps in (1, 3):
        r = subprocess.run([check, path, "5", str(sweeps)], capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
