"""Host vectors on the device: handles in several threads that share a device."""
import ctypes as C
import threading

import numpy as np
import pytest

from conftest import golden_mesh, load_golden

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def geodesics(built_lib):
    from gradientdomaintextureprocessing_b200.geodesics import Geodesics
    from gradientdomaintextureprocessing_b200.hierarchy import InitializeHierarchy
    g = load_golden("geo256")
    return Geodesics(InitializeHierarchy(golden_mesh(g), levels=int(g["meta/size"][2])))


def test_handles_of_one_system_in_threads(geodesics):
    """Two geodesics handles on one system and the system's own handle, a thread each,
    on vectors that are staged (2 MB and more): every result is the serial one."""
    from gradientdomaintextureprocessing_b200 import _lib
    from gradientdomaintextureprocessing_b200.system import MASS
    L, s = _lib.lib(), geodesics.smooth
    k = -(-4 << 20) // (8 * s.n) + 1
    k = min(64, max(1, k))
    assert 8 * s.n * k >= 2 << 20
    rng = np.random.default_rng(0)
    second = C.c_void_p()
    _lib.check(L.gdtp_geodesics_create(s.handle, C.byref(second)))
    u = [rng.standard_normal((s.n, k)) for _ in range(3)]

    def rhs(handle, x):
        out = np.empty_like(x)
        _lib.check(L.gdtp_geodesic_rhs(handle, _lib.ptr(x), _lib.ptr(out), k))
        return out

    try:
        calls = [lambda: rhs(geodesics._g, u[0]), lambda: rhs(second, u[1]), lambda: s.apply(u[2], MASS)]
        serial = [c() for c in calls]
        wrong, errors = [0, 0, 0], []

        def work(i):
            try:
                for _ in range(20):
                    wrong[i] += not np.array_equal(calls[i](), serial[i])
            except Exception as e:  # noqa: BLE001 -- reported below, in the main thread
                errors.append(e)

        threads = [threading.Thread(target=work, args=(i,)) for i in range(3)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors and wrong == [0, 0, 0]
    finally:
        L.gdtp_geodesics_free(second)
