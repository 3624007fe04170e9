"""Finite-difference stencils and the FD kinetic energy against numpy, over
the boundary rules, odd sizes, axes of one and two points, and grids below and
above one chunk of a launch."""
import ctypes as C

import numpy as np
import pytest

from libgrid_b200 import capi

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (2, 1, 3), (1, 5, 2), (7, 2, 1), (5, 6, 33), (9, 17, 31), (3, 16, 64), (20, 15, 11)]


def _shift(a, axis, d, bc):
    n = a.shape[axis]
    i = np.arange(n) + d
    if bc == "dirichlet":
        out = np.zeros_like(a)
        ok = (i >= 0) & (i < n)
        dst = [slice(None)] * 3
        dst[axis] = ok
        out[tuple(dst)] = np.take(a, i[ok], axis)
        return out
    if bc == "periodic":
        return np.take(a, i % n, axis)
    i = np.where(i < 0, -i, i)
    i = np.where(i > n - 1, 2 * n - i - 2, i)
    return np.take(a, np.clip(i, 0, n - 1) if n > 1 else 0 * i, axis)


def _laplace(a, step, bc, axes=(2, 1, 0)):
    s = -2.0 * len(axes) * a
    for d in axes:
        s = s + _shift(a, d, 1, bc) + _shift(a, d, -1, bc)
    return s / step**2


def _close(got, want, scale):
    # up to eight terms of at most six times the largest value, scaled
    assert np.abs(got - want).max() <= 16 * 2.3e-16 * scale


@pytest.mark.parametrize("bc", ["dirichlet", "neumann", "periodic"])
@pytest.mark.parametrize("shape", SHAPES)
def test_stencils(b200, shape, bc):
    rng, step = np.random.default_rng(sum(shape)), 0.3
    a = rng.uniform(-1, 1, shape) + 1j * rng.uniform(-1, 1, shape)
    g, o = b200.cgrid(*shape, step, bc, values=a), b200.cgrid(*shape, step, bc)
    lib = b200.lib
    for axis, x in enumerate("xyz"):
        getattr(lib, "cgrid_fd_gradient_" + x)(g.ptr, o.ptr)
        _close(o.get(), (_shift(a, axis, 1, bc) - _shift(a, axis, -1, bc)) / (2 * step), 1 / step)
        getattr(lib, "cgrid_fd_laplace_" + x)(g.ptr, o.ptr)
        _close(o.get(), _laplace(a, step, bc, (axis,)), 4 / step**2)
    lib.cgrid_fd_laplace(g.ptr, o.ptr)
    _close(o.get(), _laplace(a, step, bc), 12 / step**2)
    r, q = b200.rgrid(*shape, step, bc, values=a.real), b200.rgrid(*shape, step, bc)
    lib.rgrid_fd_laplace(r.ptr, q.ptr)
    _close(q.get()[:, :, : shape[2]], _laplace(a.real.copy(), step, bc), 12 / step**2)
    for x in (g, o, r, q):
        b200.free(x)


@pytest.mark.parametrize("bc,boundary", [("dirichlet", 1), ("neumann", 2), ("periodic", 3)])
@pytest.mark.parametrize("shape", [(2, 3, 5), (9, 17, 31), (20, 16, 32), (64, 100, 101)])
def test_kinetic_energy(b200, shape, bc, boundary):
    rng, step, mass = np.random.default_rng(sum(shape)), 0.3, 1.5
    psi = rng.uniform(-1, 1, shape) + 1j * rng.uniform(-1, 1, shape)
    w = b200.wf(*shape, step, mass, boundary, capi.WF_2ND_ORDER_CN, values=psi)
    want = (-0.5 / mass * np.vdot(psi, _laplace(psi, step, bc)) * step**3).real
    kinetic = b200.lib.grid_wf_kinetic_energy_cn
    kinetic.restype = C.c_double
    assert abs(kinetic(w.ptr) - want) <= 1e-12 * abs(want)
    b200.free(w)
