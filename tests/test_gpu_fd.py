"""Finite-difference stencils and the FD kinetic energy against numpy, over
the boundary rules, odd sizes, axes of one and two points, grids below and above
one chunk of a launch, planes that go in bands, and more points than 32 bits."""
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


# the last two: planes above 20 MB, taken in bands of rows (the last one partial)
@pytest.mark.parametrize("bc", ["dirichlet", "neumann", "periodic"])
@pytest.mark.parametrize("shape", SHAPES + [(3, 1153, 1151), (1, 9, 150001)])
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


# below and above the sizes from which the sum goes over halo tiles (192 MB of
# psi in FP64, 64 MB in FP32), no extent there a multiple of a tile's
KINETIC = [((2, 3, 5), 0), ((9, 17, 31), 0), ((20, 16, 32), 0), ((64, 100, 101), 0), ((233, 235, 231), 0),
           ((9, 17, 31), 1), ((205, 207, 201), 1)]


@pytest.mark.parametrize("bc,boundary", [("dirichlet", 1), ("neumann", 2), ("periodic", 3)])
@pytest.mark.parametrize("shape,fp32", KINETIC)
def test_kinetic_energy(b200, shape, fp32, bc, boundary):
    rng, step, mass = np.random.default_rng(sum(shape)), 0.3, 1.5
    psi = rng.uniform(-1, 1, shape) + 1j * rng.uniform(-1, 1, shape)
    w = b200.wf(*shape, step, mass, boundary, capi.WF_2ND_ORDER_CN, values=psi)
    if fp32:
        w.precision(capi.GRID_PREC_FP32)
        psi = psi.astype(np.complex64).astype(complex)  # what the sum reads
    want = (-0.5 / mass * np.vdot(psi, _laplace(psi, step, bc)) * step**3).real
    kinetic = b200.lib.grid_wf_kinetic_energy_cn
    kinetic.restype = C.c_double
    assert abs(kinetic(w.ptr) - want) <= 1e-12 * abs(want)
    b200.free(w)


class _Geom(C.Structure):
    _fields_ = [("nx", C.c_long), ("ny", C.c_long), ("nz", C.c_long), ("step", C.c_double), ("prec", C.c_int)]


@pytest.mark.parametrize("bc", [1, 2])  # Neumann, periodic
@pytest.mark.parametrize("shape", [(131072, 128, 127), (2, 32771, 32769)])
def test_more_points_than_32_bits(b200, shape, bc):
    """Real FP32 grids of 2.1e9 stored elements, with small planes and with
    planes of 4.3 GB, checked on planes and rows at the edges and inside."""
    torch = pytest.importorskip("torch")
    nx, ny, nz = shape
    lib, row = b200.lib, 2 * (nz // 2 + 1)
    assert nx * ny * row >= 2**31
    lib.cuda_enable(b"\x01", 0, None)
    lib.gb_fd.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.POINTER(_Geom), C.c_int] + 3 * [C.c_double] + [C.c_int, C.c_long]
    gen = torch.Generator(device="cuda").manual_seed(7)
    a = torch.rand((nx, ny, row), generator=gen, device="cuda")
    out = torch.empty_like(a)
    g = _Geom(nx, ny, nz, 0.3, 1)
    ii = sorted({0, 1, nx // 2, nx - 1})
    jj = sorted({0, 1, ny // 2, ny - 1})

    def shift(c, n):  # coordinate that stands for c
        if bc == 2:
            return c % n
        return -c if c < 0 else (2 * n - 2 - c if c > n - 1 else c)

    kp = torch.tensor([shift(k + 1, nz) for k in range(nz)], device="cuda")
    km = torch.tensor([shift(k - 1, nz) for k in range(nz)], device="cuda")
    for op, axes, lap in ((1, (2, 1, 0), 1), (2, (0,), 1), (3, (1,), 1), (4, (2,), 1), (5, (0,), 0), (6, (1,), 0), (7, (2,), 0)):
        torch.cuda.synchronize()
        assert lib.gb_fd(op, out.data_ptr(), a.data_ptr(), C.byref(g), bc, 0.0, 0.0, 0.5, 1, row) == 0
        assert lib.gb_synchronize() == 0
        for i in ii:
            for j in jj:
                c = a[i, j, :nz].double()
                want = -2.0 * len(axes) * c if lap else torch.zeros_like(c)
                for d in axes:
                    if d == 2:
                        p, m = c[kp], c[km]
                    elif d == 1:
                        p, m = a[i, shift(j + 1, ny), :nz].double(), a[i, shift(j - 1, ny), :nz].double()
                    else:
                        p, m = a[shift(i + 1, nx), j, :nz].double(), a[shift(i - 1, nx), j, :nz].double()
                    want += p + m if lap else p - m
                # up to eight terms of at most six times the largest value
                assert (out[i, j, :nz].double() - 0.5 * want).abs().max() <= 16 * 6e-8 * 6 * 0.5
    del a, out
    torch.cuda.empty_cache()
