"""The kernels that take a level where the cluster chart smoother does not: the launches, a
block per chart and the rows against each other with the clusters off, and that each
variant of the cluster smoother runs where it is meant to.  Every comparison is bitwise."""
import numpy as np
import pytest

from conftest import golden_mesh, load_golden

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["torus128", "ico256", "genus2lic512"])
def system(request, built_lib):
    from gradientdomaintextureprocessing_b200.hierarchy import InitializeHierarchy
    from gradientdomaintextureprocessing_b200.system import System
    g = load_golden(request.param)
    s = System(InitializeHierarchy(golden_mesh(g), levels=int(g["meta/size"][2])))
    s.update(1e-3, 1.0)
    s.set("chart_cluster", 0)
    return s


def results(s, b, precision="mixed"):
    x = s.vcycle(np.zeros_like(b, dtype=np.float32), b.astype(np.float32))
    y, rep = s.solve(b, tol=1e-30, max_iters=2, check=False, precision=precision)
    return x, y, rep["iterations"]


def routes(s, k, precision="mixed"):
    return s.array("levelRoutes", 0 if precision == "fp64" else k)[::3]


def compare(s, b, knob, values, precision="mixed"):
    old, out = s.get(knob), []
    try:
        for v in values:
            s.set(knob, v)
            out.append((*results(s, b, precision), routes(s, b.shape[1], precision)))
    finally:
        s.set(knob, old)
    for q in range(3):
        np.testing.assert_array_equal(out[0][q], out[1][q])
    return out[0][3], out[1][3]


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("k", [1, 3, 6])
def test_block_per_chart_matches_the_launches(system, k, precision):
    b = np.random.default_rng(k).standard_normal((system.n, k))
    off, on = compare(system, b, "chart_texels", (0, 1 << 30), precision)
    assert 2 not in off and 3 not in on and 2 in on


@pytest.mark.parametrize("k", [1, 3])
def test_rows_match_the_colour_passes(system, k):
    b = np.random.default_rng(k).standard_normal((system.n, k))
    old = system.get("chart_texels")
    try:
        system.set("chart_texels", 0)
        off, on = compare(system, b, "row_sweeps", (0, 1))
    finally:
        system.set("chart_texels", old)
    assert set(off) == {0} and 1 in on


@pytest.mark.parametrize("texels", [0, 1000])
@pytest.mark.parametrize("k", [1, 3, 6])
def test_first_sweeps_from_zero_match(system, k, texels):
    b = np.random.default_rng(k).standard_normal((system.n, k))
    old = system.get("chart_texels")
    try:
        system.set("chart_texels", texels)
        off, _ = compare(system, b, "zero_start_skip", (0, 1))
    finally:
        system.set("chart_texels", old)
    assert 3 not in off


# pairs of a row parity per CTA: up to 320, up to 512, up to 1024 (one wave), FP64
@pytest.mark.parametrize("mesh,width,height,k,precision,clustered", [
    ("torus", 256, 256, 3, "mixed", 3), ("torus", 256, 256, 15, "mixed", 3), ("icosphere", 725, 611, 1, "mixed", 4),
    ("icosphere", 1024, 1024, 3, "mixed", 4), ("icosphere", 1024, 1024, 1, "mixed", 4), ("torus", 256, 256, 3, "fp64", 3),
    ("icosphere", 1024, 1024, 3, "fp64", 3)])
def test_clusters_run_where_they_fit(built_lib, mesh, width, height, k, precision, clustered):
    """The levels meant for the cluster smoother take it (the comparisons elsewhere would pass
    without), and launch less than the kernels it replaces."""
    from gradientdomaintextureprocessing_b200 import meshgen
    from gradientdomaintextureprocessing_b200.hierarchy import InitializeHierarchy
    from gradientdomaintextureprocessing_b200.system import System
    m = meshgen.torus_atlas(width, height) if mesh == "torus" else meshgen.icosphere_atlas(width, height, subdiv=5)
    s = System(InitializeHierarchy(m, width, height, levels=4))
    s.update(1e-3, 1.0)
    s.set("chart_texels", 0)
    b = np.random.default_rng(0).standard_normal((s.n, k))
    kernels = {}
    for on in (1, 0):
        s.set("chart_cluster", on)
        s.solve(b, tol=1e-30, max_iters=2, check=False, precision=precision)
        got = routes(s, k, precision)
        deep = [s.hierarchy.counts(l)["numDeepTexels"] for l in range(len(got[:4]))]
        count = sum(r == 3 for r, d in zip(got, deep) if d > 0)
        assert count == 0 if not on else count >= clustered, got
        kernels[on] = s.array("profile")[3]
    if precision == "mixed":
        assert kernels[1] < kernels[0]
