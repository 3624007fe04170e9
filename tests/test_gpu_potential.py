"""Complex potentials through the fused steps against 64-bit numpy steps."""
import numpy as np
import pytest

from libgrid_b200 import capi

pytestmark = pytest.mark.gpu


def _step(psi, v, step, mass, dt):
    k2 = 0.0
    for d, n in enumerate(psi.shape):
        k = 2.0 * np.pi * np.fft.fftfreq(n, step)
        k2 = k2 + (k * k).reshape([-1 if a == d else 1 for a in range(3)])
    half = np.exp(-0.25j * dt / mass * k2)
    psi = np.fft.ifftn(np.fft.fftn(psi) * half) * np.exp(-1j * dt * v)
    return np.fft.ifftn(np.fft.fftn(psi) * half)


# line lengths of one to sixteen elements a thread, batches of V included;
# V with and without an imaginary part, phases on both sides of pi / 4
@pytest.mark.parametrize("shape", [(8, 4, 2), (4, 8, 16), (2, 4, 32), (2, 4, 128), (2, 2, 512), (1, 16, 64), (16, 16, 1)])
@pytest.mark.parametrize("vim", [0.0, 0.05])
@pytest.mark.parametrize("time", [0.3 + 0j, -0.2j, 0.2 - 0.1j])
def test_complex_potential_step(b200, shape, vim, time):
    rng = np.random.default_rng(sum(shape))
    psi = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    v = rng.uniform(-4.0, 4.0, shape) + 1j * vim * rng.standard_normal(shape)
    w = b200.wf(*shape, 0.5, 1.5, capi.WF_PERIODIC_BOUNDARY, capi.WF_2ND_ORDER_FFT, values=psi)
    pot = b200.cgrid(*shape, 0.5, values=v)
    b200.lib.grid_wf_propagate(w.ptr, pot.ptr, capi.Complex.of(time))
    want = _step(psi, v, 0.5, 1.5, time)
    # two transforms each way of log2 n stages and a phase, rounded at 1.1e-16
    assert np.linalg.norm(w.grid.get() - want) < 1e-14 * np.linalg.norm(want)
    b200.free(w)
    b200.free(pot)
