"""Edges of the solve kernels' launch rules on the device: widths, level sizes
and shapes where a kernel changes its variant or its last block is ragged.

Tolerances: the FP32 V-cycle's arithmetic per right-hand side does not depend on
how many are solved together nor on which kernel variant runs, so those
comparisons are bitwise.  Norms are FP64 sums of n x 2 non-negative terms:
relative error at most n 2^-53 (n <= 1e5 here), so 1e-11 with numpy's own.
"""
import numpy as np
import pytest

from conftest import golden_mesh, load_golden

pytestmark = pytest.mark.gpu


def make(name, levels=None, metric=False):
    from gradientdomaintextureprocessing_b200.hierarchy import InitializeHierarchy
    from gradientdomaintextureprocessing_b200.system import System
    g = load_golden(name)
    h = InitializeHierarchy(golden_mesh(g), levels=int(g["meta/size"][2]) if levels is None else levels)
    s = System(h)
    s.update(1e-3, 1.0)
    return s


@pytest.fixture(scope="module")
def torus(built_lib):
    return make("torus128")


@pytest.fixture(scope="module")
def ico(built_lib):
    return make("ico256")


def vectors(n, k, seed=0):
    rng = np.random.default_rng(seed)
    return rng.standard_normal((n, k)), rng.standard_normal((n, k))


@pytest.mark.parametrize("k", [1, 3, 4, 5, 8, 9, 16, 33, 64])
def test_norm_sums_at_every_width(torus, k):
    b, x = vectors(torus.n, k)
    r = b - torus.apply(x)
    expect = np.sqrt((r * r).sum(0) / (b * b).sum(0))
    np.testing.assert_allclose(torus.residual(b, x), expect, rtol=1e-11)
    np.testing.assert_array_equal(torus.residual(b, x), torus.residual(b, x))


@pytest.mark.parametrize("k", [1, 3, 5, 9, 13, 64])
def test_reported_residual_is_the_solutions(torus, k):
    b, _ = vectors(torus.n, k)
    for krylov in (0, 1):
        torus.set("krylov", krylov)
        try:
            x, rep = torus.solve(b, tol=1e-6, max_iters=200)
        finally:
            torus.set("krylov", 0)
        np.testing.assert_allclose(rep["rel_residual_max"], torus.residual(b, x).max(), rtol=1e-11)


@pytest.mark.parametrize("k", [2, 5, 9, 16, 40, 64])
def test_vcycle_columns_do_not_depend_on_the_width(ico, k):
    b, x = (v.astype(np.float32) for v in vectors(ico.n, k))
    wide = ico.vcycle(x, b)
    for c in (0, k // 2, k - 1):
        np.testing.assert_array_equal(wide[:, c], ico.vcycle(x[:, c], b[:, c])[:, 0])


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("max_coarse", [2600, 1000, 600, 300, 260])
def test_coarsest_solve_at_every_size(torus, ico, max_coarse, precision):
    """The coarsest level's rows per block follow its size; the coarse-level
    cluster kernel solves it a row per warp, with the same bits."""
    for s in (torus, ico):
        b, _ = vectors(s.n, 3)
        try:
            s.set("max_coarse", max_coarse)
            s.update(1e-3, 1.0)
            got, rep = s.solve(b, tol=1e-30, max_iters=2, check=False, precision=precision)
            s.set("cluster_texels", 1 << 30)
            ref, _ = s.solve(b, tol=1e-30, max_iters=2, check=False, precision=precision)
        finally:
            s.set("cluster_texels", 0)
            s.set("max_coarse", 2600)
            s.update(1e-3, 1.0)
        np.testing.assert_array_equal(got, ref)


@pytest.mark.parametrize("k", [6, 16, 40])
@pytest.mark.parametrize("max_coarse", [2600, 600, 260])
def test_coarsest_solve_of_wide_batches(torus, ico, max_coarse, k):
    """Right-hand sides staged in chunks of 32 rows: one column alone and among k."""
    for s in (torus, ico):
        b, x = (v.astype(np.float32) for v in vectors(s.n, k))
        try:
            s.set("max_coarse", max_coarse)
            s.update(1e-3, 1.0)
            wide = s.vcycle(x, b)
            for c in (0, k - 1):
                np.testing.assert_array_equal(wide[:, c], s.vcycle(x[:, c], b[:, c])[:, 0])
        finally:
            s.set("max_coarse", 2600)
            s.update(1e-3, 1.0)


@pytest.fixture(scope="module", params=[("torus", 256, 256), ("torus", 301, 277), ("icosphere", 512, 512), ("icosphere", 905, 643),
                                        ("icosphere", 1024, 1024), ("genus2", 643, 905)])
def atlas(request, built_lib):
    from gradientdomaintextureprocessing_b200 import meshgen
    from gradientdomaintextureprocessing_b200.hierarchy import InitializeHierarchy
    from gradientdomaintextureprocessing_b200.system import System
    name, w, h = request.param
    m = {"torus": lambda: meshgen.torus_atlas(w, h), "icosphere": lambda: meshgen.icosphere_atlas(w, h, subdiv=5),
         "genus2": lambda: meshgen.genus2_atlas(w, h, nu=176, nv=72)}[name]()
    s = System(InitializeHierarchy(m, w, h, levels=4))
    s.update(1e-3, 1.0)
    return s


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("k", [1, 3, 15])
def test_cluster_chart_smoother_matches_the_launches(atlas, k, precision):
    """All sweeps of a chart in one cluster launch: the bits of the row and colour launches."""
    b, _ = vectors(atlas.n, k)
    sweeps = {q: atlas.get(q) for q in ("coarse_pre_sweeps", "pre_sweeps", "post_sweeps")}
    got = {}
    for pre in (0, 2):
        try:
            atlas.set("coarse_pre_sweeps", pre)
            atlas.set("pre_sweeps", 3 - pre)
            atlas.set("post_sweeps", 1 + pre)
            for on in (1, 0):
                atlas.set("chart_cluster", on)
                atlas.set("chart_texels", 0 if on == 0 else 1000)
                got[on] = atlas.solve(b, tol=1e-30, max_iters=2, check=False, precision=precision)[0]
        finally:
            atlas.set("chart_cluster", 1)
            atlas.set("chart_texels", 1000)
            for q, v in sweeps.items():
                atlas.set(q, v)
        np.testing.assert_array_equal(got[1], got[0])


@pytest.mark.parametrize("k", [1, 3, 5, 16])
@pytest.mark.parametrize("knobs", [{"bs_blocks_per_sm": 1}, {"bs_blocks_per_sm": 16}, {"max_block": 64}, {"max_block": 17},
                                   {"dense_boundary_max": 8192}])
def test_boundary_products_at_every_chunking(ico, k, knobs):
    """Chunks per row group from 1 to the largest, ragged row groups, one whole
    block: the boundary products of the launches against those of the coarse-level
    cluster kernel (the same chunks, added in the same order)."""
    b, _ = vectors(ico.n, k)
    old = {q: ico.get(q) for q in knobs}
    out = {}
    try:
        for q, v in knobs.items():
            ico.set(q, v)
        for precision in ("mixed", "fp64"):
            ico.update(2e-3, 1.0)
            ico.set("max_block", ico.get("max_block"))  # lays the boundary solver out for the knobs
            for cluster in (0, 1 << 30):
                ico.set("cluster_texels", cluster)
                out[precision, cluster] = ico.solve(b, tol=1e-30, max_iters=2, check=False, precision=precision)[0]
    finally:
        ico.set("cluster_texels", 0)
        for q, v in old.items():
            ico.set(q, v)
        ico.set("max_block", ico.get("max_block"))
        ico.update(1e-3, 1.0)
    for precision in ("mixed", "fp64"):
        np.testing.assert_array_equal(out[precision, 0], out[precision, 1 << 30])


@pytest.mark.parametrize("k", [1, 2, 3, 4])
def test_brush_at_every_width(torus, ico, k):
    """A uniform mask is S f and masks that add up to one add up to it, per channel:
    both sides are FP64 sums of the same at most 64 products per texel, so they
    agree to 64 x 2^-53 of the largest product sum, taken as 1e-12 of the largest
    entry times the cancellation of a stiffness row (at most 10)."""
    from gradientdomaintextureprocessing_b200.system import STIFFNESS, Brush
    for s in (torus, ico):
        f, _ = vectors(s.n, k)
        brush = Brush(s, f)
        cells = s.hierarchy.counts(0)["numCells"]
        sf = s.apply(f, STIFFNESS)
        scale = np.abs(sf).max()
        assert np.abs(brush.apply(np.ones(cells)) - sf).max() <= 1e-11 * scale
        part = np.random.default_rng(3).integers(0, 3, cells)
        total = sum(brush.apply((part == i).astype(float)) for i in range(3))
        assert np.abs(total - sf).max() <= 1e-11 * scale
        single = Brush(s, f[:, k - 1]).apply((part == 1).astype(float))
        assert np.abs(single[:, 0] - brush.apply((part == 1).astype(float))[:, k - 1]).max() <= 1e-12 * scale


@pytest.mark.parametrize("k", [1, 3, 4, 6, 16, 64])
def test_host_vectors_of_every_size(torus, ico, k):
    """Host vectors below and above the staging size, with a ragged last chunk, pageable
    and pinned: the operator is linear and exact in powers of two, and the same call
    on pinned memory is a plain copy, so every comparison is bitwise."""
    import torch
    for s in (torus, ico):
        b, x = vectors(s.n, k)
        y = s.apply(x)
        pinned = torch.from_numpy(x).pin_memory().numpy()
        np.testing.assert_array_equal(s.apply(pinned), y)
        np.testing.assert_array_equal(s.apply(4.0 * x), 4.0 * y)
        np.testing.assert_array_equal(s.apply(x[:, k - 1])[:, 0], y[:, k - 1])
        np.testing.assert_array_equal(s.residual(b, x), s.residual(torch.from_numpy(b).pin_memory().numpy(), pinned))


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 12, 64])
def test_host_vcycle_and_sweeps(ico, k):
    """The V-cycle and the sweeps on host vectors, packed on the device: no sweeps give
    the vector back, and a column's result does not depend on the others."""
    b, x = (v.astype(np.float32) for v in vectors(ico.n, k))
    np.testing.assert_array_equal(ico.relax(x, b, sweeps=0), x)
    wide = ico.relax(x, b, sweeps=2)
    for c in (0, k - 1):
        np.testing.assert_array_equal(wide[:, c], ico.relax(x[:, c], b[:, c], sweeps=2)[:, 0])
    x0 = x.copy()
    ico.vcycle(x, b)
    np.testing.assert_array_equal(x, x0)


@pytest.mark.parametrize("k", [5, 8, 12, 16, 33, 48, 60, 64])
def test_operator_columns_do_not_depend_on_the_width(ico, k):
    """One column of A x alone and among k: the same products in the same order."""
    x, _ = vectors(ico.n, k, seed=k)
    y = ico.apply(x)
    for c in (0, k // 2, k - 1):
        np.testing.assert_array_equal(y[:, c], ico.apply(np.ascontiguousarray(x[:, c:c + 1]))[:, 0])


@pytest.mark.parametrize("k", [8, 12, 64])
def test_device_vectors_at_any_offset(ico, k):
    """Device vectors that start at an odd multiple of 8 bytes: the same iterate."""
    import ctypes as C

    import torch
    from gradientdomaintextureprocessing_b200 import _lib
    b, x = vectors(ico.n, k, seed=k)
    got = []
    for shift in (0, 1):
        buf = torch.zeros((2, b.size + 4), dtype=torch.float64, device="cuda")
        bd, xd = buf[0, shift:shift + b.size], buf[1, shift:shift + b.size]
        bd.copy_(torch.from_numpy(b.ravel()))
        xd.copy_(torch.from_numpy(x.ravel()))
        rep = _lib.Report()
        _lib.lib().gdtp_solve_device(ico.handle, C.c_void_p(bd.data_ptr()), C.c_void_p(xd.data_ptr()), k, 1e-300, 2,
                                     C.c_void_p(torch.cuda.current_stream().cuda_stream), C.byref(rep))  # not converged after 2
        assert rep.iterations == 2
        got.append(xd.cpu().numpy())
    np.testing.assert_array_equal(got[0], got[1])
