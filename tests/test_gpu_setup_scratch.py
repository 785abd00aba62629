"""Re-weighting at the limits of device memory: the levels' scratch side by side where there
is room for their sum, in turn where there is room for the largest."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

POOL_RELEASE, POOL_USED_HIGH = 0x4, 0x8  # cudaMemPoolAttrReleaseThreshold, cudaMemPoolAttrUsedMemHigh


@pytest.fixture(scope="module")
def rt():
    return C.CDLL("libcudart.so.12", mode=C.RTLD_GLOBAL)


def used_high(rt, pool, reset=False):
    v = C.c_uint64(0)
    if reset:
        assert rt.cudaMemPoolSetAttribute(pool, POOL_USED_HIGH, C.byref(v)) == 0
    assert rt.cudaMemPoolGetAttribute(pool, POOL_USED_HIGH, C.byref(v)) == 0
    return v.value


@pytest.mark.parametrize("share", [0.0, 0.75])
def test_update_with_room_for_one_level(built_lib, rt, share):
    """The values of an update whose levels ran in turn are those of one that ran them side by
    side.  share: of the scratch of all levels that fits; 0 leaves none and fails cleanly."""
    import torch
    from gradientdomaintextureprocessing_b200 import _lib, meshgen
    from gradientdomaintextureprocessing_b200.hierarchy import InitializeHierarchy
    from gradientdomaintextureprocessing_b200.system import System
    torch.zeros(1, device="cuda")
    s = System(InitializeHierarchy(meshgen.icosphere_atlas(1024, 1024, subdiv=5), 1024, 1024, levels=4))
    s.update(2e-3, 1.0)
    b = np.random.default_rng(0).standard_normal((s.n, 3))
    s.solve(b, tol=1e-30, max_iters=2, check=False)
    pool = C.c_void_p()
    assert rt.cudaDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    used_high(rt, pool, reset=True)
    s.update(1e-3, 1.0)
    expect = s.solve(b, tol=1e-30, max_iters=2, check=False)[0]
    need = used_high(rt, pool)
    s.update(2e-3, 1.0)
    torch.cuda.synchronize()
    assert rt.cudaMemPoolTrimTo(pool, C.c_size_t(0)) == 0
    free, total = C.c_size_t(), C.c_size_t()
    fill = []
    try:
        # leave that much: one large block, then smaller ones
        for unit in (1 << 30, 64 << 20, 2 << 20):
            assert rt.cudaMemGetInfo(C.byref(free), C.byref(total)) == 0
            size = (free.value - int(share * need)) // unit * unit
            p = C.c_void_p()
            if size > 0 and rt.cudaMalloc(C.byref(p), C.c_size_t(size)) == 0:
                fill.append(p)
            rt.cudaGetLastError()
        if share == 0.0:
            with pytest.raises(_lib.GDTPError, match="scratch"):
                s.update(1e-3, 1.0)
            return
        s.update(1e-3, 1.0)
        print("scratch of all levels %.1f MB, room for %.1f MB" % (need / 1e6, share * need / 1e6), s.array("profile.setup")[:8])
    finally:
        for p in fill:
            rt.cudaFree(p)
    np.testing.assert_array_equal(s.solve(b, tol=1e-30, max_iters=2, check=False)[0], expect)
