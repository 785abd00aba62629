"""Atlases of many small charts: which kernels take their levels, and the same bits from all.

The FP32 V-cycle's arithmetic per right-hand side does not depend on how many are solved
together nor on which kernel variant runs, so every comparison is bitwise."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def grid_atlas(n, size, sub=2, gutter=2.0, seed=0):
    """n x n square charts of a wavy sheet, sub x sub quads each, corners moved by up to 0.3 texels."""
    from gradientdomaintextureprocessing_b200 import meshgen
    rng = np.random.default_rng(seed)
    m = n * sub
    i, j = np.meshgrid(np.arange(m + 1), np.arange(m + 1), indexing="xy")
    vertices = np.stack([i / m, j / m, 0.1 * np.sin(5 * i / m) * np.cos(4 * j / m)], -1).reshape(-1, 3)
    jitter = rng.uniform(-0.3, 0.3, (n, n, sub + 1, sub + 1, 2))
    inner = size / n - 2 * gutter
    triangles, uv = [], []
    for cy, cx, b, a in np.ndindex(n, n, sub, sub):
        quad = [(a, b), (a + 1, b), (a + 1, b + 1), (a, b + 1)]
        for t in ((0, 1, 2), (0, 2, 3)):
            triangles.append([(cy * sub + quad[q][1]) * (m + 1) + cx * sub + quad[q][0] for q in t])
            uv.append([[(c * size / n + gutter + p / sub * inner + jitter[cy, cx, quad[q][1], quad[q][0], x]) / size
                        for x, (c, p) in enumerate(((cx, quad[q][0]), (cy, quad[q][1])))] for q in t])
    uv = meshgen._keep_off_texel_grid(np.array(uv), size, size)
    return {"vertices": vertices, "triangles": np.array(triangles, dtype=np.int32), "uv": uv}


@pytest.fixture(scope="module", params=[(26, 832), (32, 1024), (12, 640)])
def atlas(request, built_lib):
    from gradientdomaintextureprocessing_b200.hierarchy import InitializeHierarchy
    from gradientdomaintextureprocessing_b200.system import System
    n, size = request.param
    s = System(InitializeHierarchy(grid_atlas(n, size), size, size, levels=4))
    s.update(1e-3, 1.0)
    s.charts = n * n
    return s


def vectors(n, k, seed=0):
    rng = np.random.default_rng(seed)
    return rng.standard_normal((n, k)), rng.standard_normal((n, k))


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("k", [1, 3, 9])
def test_charts_smooth_on_clusters(atlas, k, precision):
    """Up to 4 channels every level with deep texels smooths on clusters, however many charts
    it has; the launches give the same bits."""
    b, _ = vectors(atlas.n, k)
    got = {}
    try:
        for on, texels in ((1, 1000), (0, 1000), (0, 0)):
            atlas.set("chart_cluster", on)
            atlas.set("chart_texels", texels)
            got[on, texels] = atlas.solve(b, tol=1e-30, max_iters=2, check=False, precision=precision)[0]
            routes = atlas.array("levelRoutes", 0 if precision == "fp64" else k)[::3]
            deep = [atlas.hierarchy.counts(l)["numDeepTexels"] for l in range(min(4, len(routes)))]
            if on and k <= 4:
                assert all(r == 3 for r, d in zip(routes, deep) if d > 0), routes
            if not on:
                assert 3 not in routes
                assert texels == 0 or 2 in routes
    finally:
        atlas.set("chart_cluster", 1)
        atlas.set("chart_texels", 1000)
    np.testing.assert_array_equal(got[1, 1000], got[0, 0])
    np.testing.assert_array_equal(got[0, 1000], got[0, 0])


def test_boundary_products_run_where_they_are_faster(atlas):
    """The largest separators, more row groups than there are resident clusters, and the
    subdomains' product of one chunk take a CTA per chunk."""
    b, _ = vectors(atlas.n, 3)
    for precision, width in (("mixed", 3), ("fp64", 0)):
        atlas.set("max_block", atlas.get("max_block"))  # drops the multigrids of other widths
        atlas.solve(b, tol=1e-30, max_iters=1, check=False, precision=precision)
        routes = atlas.array("levelRoutes", width).reshape(-1, 3)
        if width:
            stats = atlas.array("levelStats").reshape(-1, 9)
            for (_, sub, schur), row in zip(routes, stats):
                rows = row[4]
                assert schur == (0 if rows == 0 else 1 if rows <= 1792 else 2) or 1792 < rows <= 2304
        assert routes[0][1] == 2 or atlas.charts < 400
        assert routes[0][2] == 2 or atlas.charts < 400


@pytest.mark.parametrize("k", [1, 3, 6, 9])
def test_boundary_products_give_the_same_bits(atlas, k):
    """A CTA per chunk against the coarse-level cluster kernel (the same chunks, added in the
    same order), and one column alone against k columns, whose products may run otherwise."""
    b, x = (v.astype(np.float32) for v in vectors(atlas.n, k))
    wide = atlas.vcycle(x, b)
    for c in {0, k - 1}:
        np.testing.assert_array_equal(wide[:, c], atlas.vcycle(x[:, c], b[:, c])[:, 0])
    if k > 4:
        return
    out = {}
    for precision in ("mixed", "fp64"):
        for texels in (0, 1 << 30):
            try:
                atlas.set("cluster_texels", texels)
                out[texels] = atlas.solve(b.astype(float), tol=1e-30, max_iters=2, check=False, precision=precision)[0]
            finally:
                atlas.set("cluster_texels", 0)
        np.testing.assert_array_equal(out[0], out[1 << 30])


@pytest.mark.parametrize("k", [1, 2, 3, 4])
def test_boundary_rows_give_the_same_sums(atlas, k):
    """A boundary row on one lane and on 8, by their number and the width: the operator's and
    the residual's columns alone and among 9 (several channel groups: a thread per row and
    group), with odd widths in between."""
    x, b = vectors(atlas.n, 9)
    y = atlas.apply(x)
    part = atlas.apply(np.ascontiguousarray(x[:, :k]))
    np.testing.assert_array_equal(part, y[:, :k])
    for precision in ("mixed", "fp64"):
        wide = atlas.solve(b, tol=1e-30, max_iters=2, check=False, precision=precision)[0]
        got = atlas.solve(np.ascontiguousarray(b[:, :k]), tol=1e-30, max_iters=2, check=False, precision=precision)[0]
        np.testing.assert_array_equal(got, wide[:, :k])


@pytest.mark.parametrize("k", [1, 3])
def test_norms_of_many_rows(atlas, k):
    """The norms add every row once: relative error at most n 2^-53 (n <= 1e6), so 1e-9."""
    b, x = vectors(atlas.n, k)
    r = b - atlas.apply(x)
    np.testing.assert_allclose(atlas.residual(b, x), np.sqrt((r * r).sum(0) / (b * b).sum(0)), rtol=1e-9)
