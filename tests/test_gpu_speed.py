"""Routes that a size rule chooses, timed against what they replace: a route
that is slower than the other one by a wide margin is the wrong choice.  Times
are the least of several passes, on the device."""
import ctypes as C

import numpy as np
import pytest

from libgrid_b200 import capi, workloads

pytestmark = pytest.mark.gpu

MASS = 4.0 / workloads.GRID_AUTOAMU


def _ms(lib, call, repeats=9):
    """Least time of `repeats` calls, by the library's events."""
    lib.gb_event_elapsed_ms.restype = C.c_float
    lib.gb_event_elapsed_ms.argtypes = [C.c_int, C.c_int]
    best = float("inf")
    for _ in range(repeats):
        lib.gb_event_record(14)
        call()
        lib.gb_event_record(15)
        best = min(best, lib.gb_event_elapsed_ms(14, 15))
    return best


def _fluid(b200, shape, prop=capi.WF_2ND_ORDER_FFT):
    rng = np.random.default_rng(3)
    psi = rng.uniform(0.5, 1.0, shape) + 0j
    w = b200.wf(*shape, 0.3, MASS, capi.WF_PERIODIC_BOUNDARY, prop, values=psi)
    return w, b200.rgrid(*shape, 0.3, values=1e-3 * rng.uniform(-1, 1, shape))


@pytest.mark.parametrize("shape", [(16, 512, 512), (8, 256, 256), (128, 64, 64)])
def test_relaxation_steps_beat_single_calls(b200, shape):
    """Eight relaxation steps in one call save passes against eight steps with a
    normalisation after each (at 16 x 512 x 512 1.7 times faster)."""
    w, v = _fluid(b200, shape)
    tm = capi.Complex.of(-2j)

    def merged():
        b200.lib.grid_wf_relax_gp_n(w.ptr, v.ptr, 1e-3, tm, 8)

    def single():
        for _ in range(8):
            w.propagate_gp(v, 1e-3, -2j)
            w.normalize()

    b200.lib.grid_wf_relax_gp_n.restype = None
    b200.lib.grid_wf_relax_gp_n.argtypes = [C.POINTER(b200.WF), C.POINTER(b200.RGrid), C.c_double, capi.Complex, C.c_long]
    merged()
    single()
    assert _ms(b200.lib, merged) < 0.9 * _ms(b200.lib, single)
    b200.free(w)
    b200.free(v)


@pytest.mark.parametrize("shape", [(64, 512, 512), (512, 128, 128), (128, 64, 64)])
def test_overlapped_passes_beat_passes_apart(b200, shape):
    """A step whose launches may overlap against the same step with an event
    between any two of them, which keeps them apart: at most the spread of the
    least times slower (5%)."""
    w, v = _fluid(b200, shape)

    def steps():
        for _ in range(4):
            w.propagate_gp(v, 1e-3, 1.0)

    steps()
    b200.lib.gb_pass_timing(1)
    apart = _ms(b200.lib, steps)
    b200.lib.gb_pass_timing(0)
    assert _ms(b200.lib, steps) < 1.05 * apart
    b200.free(w)
    b200.free(v)
