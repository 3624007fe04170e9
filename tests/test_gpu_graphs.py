"""Tables kept between calls (kinetic factors, line-solver coefficients): the
tables of a captured step are the graph's own, whatever other steps run between
its replays, a replay leaves the tables of plain steps alone, and none outlives
gb_shutdown."""
import ctypes as C
import subprocess
import sys

import numpy as np
import pytest

from libgrid_b200 import capi, workloads

pytestmark = pytest.mark.gpu

MASS = 4.0 / workloads.GRID_AUTOAMU
# name: (shape, boundary, propagator, omega)
STEPS = {
    "cn-rotating": ((12, 10, 9), 2, capi.WF_2ND_ORDER_CN, 1e-4),
    "cn-rotating-2d": ((10, 14, 1), 1, capi.WF_2ND_ORDER_CN, 1e-4),
    "cn-rest": ((12, 10, 9), 3, capi.WF_2ND_ORDER_CN, 0.0),
    "fft": ((16, 8, 32), 3, capi.WF_2ND_ORDER_FFT, 0.0),
    "cfft-1d": ((1, 1, 64), 3, capi.WF_2ND_ORDER_CFFT, 0.0),
}


class _Runs:
    """Steps of one wave function, plain or captured, each from the same psi."""

    def __init__(self, api, name):
        shape, bc, prop, omega = STEPS[name]
        rng = np.random.default_rng(5)
        psi = rng.uniform(-1, 1, shape) + 1j * rng.uniform(-1, 1, shape)
        self.api, self.lib = api, api.lib
        self.w = api.wf(*shape, 0.3, MASS, bc, prop, values=psi)
        self.w.s.kmax = 6.0
        self.lib.cgrid_set_rotation(self.w.s.grid, omega)
        self.psi = api.cgrid(*shape, 0.3, values=psi)
        self.lib.gb_grid_device.restype = C.c_void_p
        self.lib.gb_grid_device.argtypes = [C.c_void_p, C.c_int]
        self.lib.gb_grid_device(self.psi.s.value, 0)  # reset() then copies on the device, as a replay needs
        self.v = api.cgrid(*shape, 0.3, values=1e-3 * rng.uniform(-1, 1, shape))
        self.plain(0.1)  # buffers on the device, scratch sized

    def reset(self):
        self.lib.cgrid_copy(self.w.s.grid, self.psi.ptr)

    def plain(self, dt):
        self.reset()
        self.w.propagate(self.v, dt)
        return self.w.grid.get()

    def capture(self, dt):
        self.reset()
        g = C.c_void_p()
        assert self.lib.gb_graph_begin() == 0
        self.w.propagate(self.v, dt)
        assert self.lib.gb_graph_end(C.byref(g)) == 0
        return g

    def replay(self, g):
        self.reset()
        assert self.lib.gb_graph_launch(g) == 0
        return self.w.grid.get()

    def free(self):
        for x in (self.w, self.psi, self.v):
            self.api.free(x)


def _graph_calls(lib):
    for name in ("gb_graph_begin", "gb_graph_end", "gb_graph_launch", "gb_graph_free"):
        getattr(lib, name).restype = C.c_int
    lib.gb_graph_begin.argtypes = []
    lib.gb_graph_end.argtypes = [C.POINTER(C.c_void_p)]
    lib.gb_graph_launch.argtypes = lib.gb_graph_free.argtypes = [C.c_void_p]


@pytest.mark.parametrize("last", ["same", "other"])
@pytest.mark.parametrize("name", STEPS)
def test_tables_of_graphs(b200, name, last):
    """`last`: the plain step before the capture has the captured step's
    parameters (tables at hand) or others (tables to be built)."""
    _graph_calls(b200.lib)
    r = _Runs(b200, name)
    want = {dt: r.plain(dt) for dt in (0.5, 0.3)}
    assert np.abs(want[0.5] - want[0.3]).max() > 1e-6
    r.plain(0.5 if last == "same" else 0.3)
    g = r.capture(0.5)
    for dt in (0.3, 0.3, 0.5, 0.3):
        assert np.array_equal(r.plain(dt), want[dt]), dt
        assert np.array_equal(r.replay(g), want[0.5])
    b200.lib.gb_graph_free(g)
    assert np.array_equal(r.plain(0.3), want[0.3])
    r.free()


def test_rotating_step_in_a_capture_of_the_stream(b200):
    """A capture that gb_graph_begin did not start owns no tables: a rotating
    step in it solves with per-line pivots, the same to rounding."""
    torch = pytest.importorskip("torch")
    lib = b200.lib
    lib.gb_stream_handle.restype = C.c_void_p
    r = _Runs(b200, "cn-rotating")
    want = {dt: r.plain(dt) for dt in (0.5, 0.3)}
    stream = torch.cuda.ExternalStream(lib.gb_stream_handle())
    g = torch.cuda.CUDAGraph()
    r.reset()
    with torch.cuda.graph(g, stream=stream, capture_error_mode="relaxed"):
        r.w.propagate(r.v, 0.5)
    for dt in (0.3, 0.5, 0.3):
        assert np.array_equal(r.plain(dt), want[dt])
        r.reset()
        with torch.cuda.stream(stream):
            g.replay()
        got = r.w.grid.get()
        # a few operations per element and sweep with condition numbers near 1
        assert np.abs(got - want[0.5]).max() <= 1e-13 * np.abs(want[0.5]).max()
    del g
    r.free()


_AFTER_SHUTDOWN = """
import sys; sys.path[:0] = [%r, %r]
import ctypes as C, numpy as np, libgrid_b200
from test_gpu_graphs import STEPS, _Runs
api = libgrid_b200.load(); lib = api.lib
lib.gb_device_alloc.restype = C.c_void_p
lib.gb_device_alloc.argtypes = [C.c_size_t]
lib.gb_device_free.argtypes = [C.c_void_p]
lib.gb_memset.argtypes = [C.c_void_p, C.c_int, C.c_size_t]
for name in STEPS:
    r = _Runs(api, name)
    want = r.plain(0.5)
    assert lib.gb_shutdown() == 0
    # what the freed tables held is overwritten
    blocks = [(lib.gb_device_alloc(1 << k), 1 << k) for k in range(12, 22) for _ in range(24)]
    for p, n in blocks:
        lib.gb_memset(p, 255, n)
    for p, n in blocks:
        lib.gb_device_free(p)
    assert np.array_equal(r.plain(0.5), want), name
print("same")
"""


def test_tables_after_shutdown():
    from conftest import ROOT

    p = subprocess.run([sys.executable, "-c", _AFTER_SHUTDOWN % (ROOT, ROOT + "/tests")], capture_output=True, text=True,
                       timeout=600)
    assert p.returncode == 0 and "same" in p.stdout, p.stderr[-2000:]
