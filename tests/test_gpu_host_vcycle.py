"""The V-cycle and the sweeps on host vectors: what they allocate and what a failed one leaves."""
import numpy as np
import pytest

from conftest import golden_mesh, load_golden

pytestmark = pytest.mark.gpu


def make(name):
    from gradientdomaintextureprocessing_b200.hierarchy import InitializeHierarchy
    from gradientdomaintextureprocessing_b200.system import System
    g = load_golden(name)
    s = System(InitializeHierarchy(golden_mesh(g), levels=int(g["meta/size"][2])))
    s.update(1e-3, 1.0)
    return s


@pytest.mark.parametrize("call", ["vcycle", "relax"])
@pytest.mark.parametrize("k", [1, 3, 15])
def test_no_solve_vectors_are_allocated(built_lib, call, k):
    """The multigrid's own vectors are enough: the FP64 work vectors come with the first call
    that computes in FP64, and the results do not depend on them."""
    s = make("torus128")
    rng = np.random.default_rng(0)
    x, b = (rng.standard_normal((s.n, k)).astype(np.float32) for _ in range(2))
    first = getattr(s, call)(x, b)
    before = s.device_bytes()
    s.residual(b.astype(float), x.astype(float))
    assert s.device_bytes() - before >= 3 * 8 * s.n * k
    np.testing.assert_array_equal(getattr(s, call)(x, b), first)


@pytest.mark.parametrize("double", [False, True])
def test_a_failed_cycle_leaves_the_vector_alone(built_lib, double):
    """A grid barrier that timed out (its error word set from the host) fails the call; the
    caller's x keeps its values."""
    import ctypes as C
    from gradientdomaintextureprocessing_b200 import _lib
    L, s = _lib.lib(), make("torus128")
    s.set("grid_texels", 1 << 30)
    kind = np.float64 if double else np.float32
    call = L.gdtp_vcycle64 if double else L.gdtp_vcycle
    rng = np.random.default_rng(0)
    x, b = (rng.standard_normal((s.n, 3)).astype(kind) for _ in range(2))

    def run():
        y = x.copy()
        return call(s.handle, _lib.ptr(y), _lib.ptr(b), 3), y

    code, good = run()
    assert code == 0 and not np.array_equal(good, x)
    count = C.c_int64()
    assert L.gdtp_system_array(s.handle, b"fault.barrier", 0, None, C.byref(count)) == 0
    code, failed = run()
    assert code != 0
    np.testing.assert_array_equal(failed, x)
