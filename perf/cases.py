"""Performance cases: the calls that programs built on this library spend their time in.

Each case makes one pass through the public entry points (the libgrid C API
through `libgrid_b200.load()`, and `libgrid_b200.warmstart` for the learned
start).  Fields and potentials come from the seeded families of the library's
own workloads, drawn on the GPU; the device copies of the grids are handed out
as tensors without a copy.
"""
import ctypes as C
import math

import numpy as np
import torch

import libgrid_b200
from libgrid_b200 import capi, warmstart

AMU = 1.0 / capi.GRID_AUTOAMU
DEV = "cuda"
CD, FD = torch.complex128, torch.float64

# ------------------------------------------------------------------ the cases


def listed():
    return [
        # the smallest everyday call: one real-time step of a wave packet on a
        # coarse grid (latency of the launches, not bandwidth)
        dict(name="packet-32", kind="step", nx=32, ny=32, nz=32, prec=64, pot="complex", imag=False, steps=1),
        # the library's main workload: a Gross-Pitaevskii step of a 256^3 fluid
        dict(name="gp-256", kind="step", nx=256, ny=256, nz=256, prec=64, pot="gp", imag=False, steps=1),
        # the same fluid in the single-precision mode, ten steps between two
        # analyses, the result read back as FP64
        dict(name="gp-256-fp32", kind="step", nx=256, ny=256, nz=256, prec=32, pot="gp", imag=False, steps=10),
        # ground-state search: ten imaginary-time steps with renormalisation
        # and one energy, as the relaxation loop runs them between two checks
        dict(name="relax-128", kind="relax", n=128, steps=10),
        # Crank-Nicolson Gross-Pitaevskii step in a box
        dict(name="cn-192", kind="cn", nx=192, ny=192, nz=192, boundary=1, pot="gp", omega=0.0, absorb=0),
        # Crank-Nicolson on a grid whose sizes no tile divides
        dict(name="cn-odd", kind="cn", nx=125, ny=99, nz=75, boundary=2, pot="complex", omega=0.0, absorb=0),
        # vortices: a rotating frame, which only Crank-Nicolson propagates
        dict(name="cn-rotating", kind="cn", nx=100, ny=100, nz=50, boundary=1, pot="complex", omega=1e-6, absorb=0),
        # many two-dimensional problems of four heights advanced together
        dict(name="batch-64", kind="batch", per_size=16, nz=256, prec=64, steps=20),
        # what a run prints and saves every so often: norm, energy, density
        # and the gradients that currents are made of
        dict(name="observe-odd", kind="observe", nx=200, ny=150, nz=101, boundary=3),
        # a density convolved with a kernel held in k-space (density functionals)
        dict(name="convolve-128", kind="convolve", nx=128, ny=128, nz=128),
        # training the learned start: one minibatch and one optimiser step
        dict(name="train-32", kind="train", n=32, batch=8),
        # the learned start itself: one inference at production size
        dict(name="infer-128", kind="infer", n=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pow2_shape(rng):
    while True:
        s = [2 ** rng.randint(4, 8) for _ in range(3)]
        if 2**13 <= s[0] * s[1] * s[2] <= 2**24:
            return dict(nx=s[0], ny=s[1], nz=s[2])


def _any_shape(rng, lo, hi):
    return dict(nx=_log_int(rng, lo, hi), ny=_log_int(rng, lo, hi), nz=_log_int(rng, lo, hi))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "relax", "cn", "cn", "batch", "observe", "convolve", "train", "infer"])
    if kind == "step":
        return dict(kind=kind, **_pow2_shape(rng), prec=rng.choice([64, 64, 32]), pot=rng.choice(["complex", "gp"]),
                    imag=rng.random() < 0.25, steps=rng.choice([1, 1, 2, 3, 5, 8]))
    if kind == "relax":
        return dict(kind=kind, n=rng.choice([32, 64, 128]), steps=rng.randint(3, 12))
    if kind == "cn":
        omega, absorb = rng.choice([0.0, 0.0, 0.0, 1e-6]), rng.choice([0, 0, 0, 4])
        return dict(kind=kind, **_any_shape(rng, 24, 128 if omega or absorb else 200), boundary=rng.randint(1, 3),
                    pot=rng.choice(["complex", "gp"]), omega=omega, absorb=absorb)
    if kind == "batch":
        return dict(kind=kind, per_size=rng.randint(2, 16), nz=rng.choice([64, 128, 256, 512]),
                    prec=rng.choice([64, 32]), steps=rng.randint(10, 20))
    if kind == "observe":
        return dict(kind=kind, **_any_shape(rng, 24, 220), boundary=rng.randint(1, 3))
    if kind == "convolve":
        return dict(kind=kind, **_pow2_shape(rng))
    if kind == "train":
        return dict(kind=kind, n=rng.choice([16, 24, 32]), batch=rng.randint(2, 16))
    return dict(kind=kind, n=8 * rng.randint(4, 16))


# ------------------------------------------------------- grids as GPU tensors


class _Owned:
    """Library objects freed when the last tensor on their memory is gone."""

    def __init__(self, api, *objs):
        self.api, self.objs = api, list(objs)

    def __del__(self):
        for o in self.objs:
            if isinstance(o, (warmstart.DeviceUNet, warmstart.DeviceSet)):
                o.free()
            else:
                self.api.free(o)


class _Memory:
    """Device memory of a library object for torch (keeps the object alive)."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr=typestr, data=(int(ptr), False), version=2)


def _tensor(owner, ptr, shape, typestr):
    return torch.as_tensor(_Memory(owner, ptr, shape, typestr), device=DEV)


def _api():
    api = libgrid_b200.load()
    lib = api.lib
    if lib.gb_stream_handle.restype is not C.c_void_p:
        lib.cuda_enable(b"\x01", 0, None)
        lib.gb_stream_handle.restype = C.c_void_p
        lib.gb_grid_device.restype = C.c_void_p
        lib.gb_grid_device.argtypes = [C.c_void_p, C.c_int]
        lib.grid_wf_relax_gp_n.restype = None
        lib.grid_wf_relax_gp_n.argtypes = [C.POINTER(api.WF), C.POINTER(api.RGrid), C.c_double, capi.Complex, C.c_long]
        lib.rgrid_copy.restype = None
        lib.rgrid_copy.argtypes = [C.POINTER(api.RGrid), C.POINTER(api.RGrid)]
    return api


class _View:
    """The FP64 device copy of a grid as a tensor."""

    def __init__(self, api, owner, grid):
        s = grid.s
        self.lib, self.owner, self.value, self.real = api.lib, owner, C.c_void_p(s.value), grid.real
        self.shape, self.nz = (s.nx, s.ny, s.nz2 if grid.real else s.nz), s.nz
        self.ptr, self.t = None, None

    def get(self, mode=0):
        p = self.lib.gb_grid_device(self.value, mode)
        if p != self.ptr:
            t = _tensor(self.owner, p, self.shape, "<f8" if self.real else "<c16")
            self.ptr, self.t = p, t[:, :, : self.nz] if self.real else t
        return self.t

    def put(self, values):
        self.get(1).copy_(values)
        torch.cuda.synchronize()


# ------------------------------------------------------------------ the inputs


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _u(g, lo, hi, n):
    return (lo + (hi - lo) * torch.rand(n, generator=g, device=DEV, dtype=FD)).tolist()


def _axes(shape, step):
    return [((torch.arange(n, device=DEV, dtype=FD) - n // 2) * step).reshape([-1 if a == d else 1 for a in range(3)])
            for d, n in enumerate(shape)]


def _wells(g, shape, step, nwells=8):
    """Random Gaussian wells: the external potential of the fluid workloads."""
    x, y, z = _axes(shape, step)
    half = max(shape) * step / 4
    d, w = _u(g, 1e-4, 1e-3, nwells), _u(g, 3.0, 10.0, nwells)
    c = [_u(g, -half, half, 3) for _ in range(nwells)]
    v = torch.zeros(shape, device=DEV, dtype=FD)
    for i in range(nwells):
        ex, ey, ez = (torch.exp(-((a - b) ** 2) / w[i] ** 2) for a, b in zip((x, y, z), c[i]))
        v -= d[i] * (ex * ey) * ez
    return v, max(d)


def _fluid(g, shape, step, coupling):
    """(psi, V): Thomas-Fermi fluid with 1% noise in random wells."""
    v, dmax = _wells(g, shape, step)
    xi = torch.randn(shape, generator=g, device=DEV, dtype=CD) * math.sqrt(2.0)
    psi = torch.sqrt(torch.clamp(2.0 * dmax - v, min=0.0) / coupling) * (1.0 + 0.01 * xi)
    return psi, v


def _packet(g, shape, step):
    """(psi, V): a Gaussian packet with momentum in a trap with random bumps."""
    x, y, z = _axes(shape, step)
    v, _ = _wells(g, shape, step)
    v = 0.005 * (x * x + y * y + z * z) + 10.0 * v
    c, k = _u(g, -1.0, 1.0, 3), _u(g, -0.5, 0.5, 3)
    r2 = (x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2
    psi = torch.exp(-r2 / 4.0) * torch.exp(1j * (k[0] * x + k[1] * y + k[2] * z))
    return psi, v


def _step_inputs(case, seed):
    """(psi, V, step, mass, coupling, time) of a propagation case."""
    g, shape = _gen(seed), (case["nx"], case["ny"], case["nz"])
    if case["pot"] == "gp":
        h, coupling, dt = (0.5, 0.0025, 1.0) if case["kind"] == "step" else (0.3, 0.001, 0.5)
        psi, v = _fluid(g, shape, h, coupling)
        mass = 4.0 * AMU
    else:
        h, coupling, dt, mass = 0.2, 0.0, 0.05, 1.0
        psi, v = _packet(g, shape, h)
        if case["kind"] == "cn" and (case["omega"] or case["absorb"]):
            mass, dt = 4.0 * AMU, 20.0  # helium in a rotating or absorbing box
    return psi, v, h, mass, coupling, (-1j * dt if case.get("imag") else dt + 0j)


def _trap(seed, n):
    """(V, g) of one ground-state problem: a harmonic trap with bumps."""
    g, h = _gen(seed), 3.2 / n
    x, y, z = _axes((n, n, n), h)
    k, coupling = _u(g, 0.005, 0.02, 1)[0], _u(g, 0.001, 0.01, 1)[0]
    v = 0.5 * k * (x * x + y * y + z * z)
    for _ in range(4):
        a, w, c = _u(g, -2e-3, 2e-3, 1)[0], _u(g, 0.2, 0.6, 1)[0], _u(g, -0.8, 0.8, 3)
        v = v + a * torch.exp(-((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2) / w**2)
    return v, coupling, h


def _relax_inputs(case, seed):
    v, coupling, h = _trap(seed, case["n"])
    x, y, z = _axes(v.shape, h)
    psi = torch.exp(-(x * x + y * y + z * z)).to(CD)
    return psi / torch.sqrt((psi.abs() ** 2).sum() * h**3), v, coupling, h


def _batch_inputs(case, seed):
    """[(psi, V)]: packets in traps with bumps, the heights in turn."""
    g, h = _gen(seed), 0.2
    out = []
    for n in (64, 128, 256, 512) * case["per_size"]:
        _, y, z = _axes((1, n, case["nz"]), h)
        k, bump, w, ky, kz = (_u(g, lo, hi, 1)[0] for lo, hi in ((0.005, 0.02), (1e-3, 1e-2), (1, 4), (-1, 1), (-1, 1)))
        r2 = y * y + z * z
        v = 0.5 * k * r2 + bump * torch.exp(-((y - w) ** 2 + z * z) / w**2)
        out.append((torch.exp(-r2 / 4.0) * torch.exp(1j * (ky * y + kz * z)), v))
    return out


def _observe_inputs(case, seed):
    return _fluid(_gen(seed), (case["nx"], case["ny"], case["nz"]), 0.5, 0.0025)


def _convolve_inputs(case, seed):
    """(density, kernel): a noisy fluid density and a soft-core kernel."""
    g, shape = _gen(seed), (case["nx"], case["ny"], case["nz"])
    psi, _ = _fluid(g, shape, 0.5, 0.0025)
    x, y, z = _axes(shape, 0.5)
    w = _u(g, 2.0, 5.0, 1)[0]
    return psi.abs() ** 2, torch.exp(-(x * x + y * y + z * z) / w**2) * (1.0 + 0.1 * torch.cos(x + 0.5 * y))


# the network: (layer, sources, output channels), in the parameter order
_NET = [("e0a", 3, 8), ("e0b", 8, 8), ("e1a", 8, 16), ("e1b", 16, 16), ("e2a", 16, 32), ("e2b", 32, 32), ("ba", 32, 64),
        ("bb", 64, 64), ("d2a", 96, 32), ("d2b", 32, 32), ("d1a", 48, 16), ("d1b", 16, 16), ("d0a", 24, 8),
        ("d0b", 8, 8), ("out", 8, 1)]


def _net_params(seed):
    rng, parts = np.random.default_rng(seed), []
    for name, ci, co in _NET:
        std = math.sqrt(2.0 / (27 * ci)) * (0.1 if name == "out" else 1.0)
        parts += [rng.standard_normal(co * ci * 27) * std, rng.standard_normal(co) * 0.02]
    return np.concatenate(parts).astype(np.float32)


def _net_inputs(seed, n, count):
    """Features [count][3][n^3] and targets [count][n^3] of random traps."""
    xs, ys = [], []
    for i in range(count):
        v, coupling, _ = _trap(seed * 1000 + i, n)
        mu = v.min() + 0.35 * (v.max() - v.min())
        amp = torch.sqrt(torch.clamp(mu - v, min=0.0) / (mu - v.min()))
        xs.append(torch.stack([torch.tanh((v - v.min()) / 0.01), torch.full_like(v, coupling / 0.01), amp]))
        ys.append(amp * (0.9 + 0.1 * torch.cos(3.0 * amp)))
    return torch.stack(xs).float(), torch.stack(ys).float()


# ------------------------------------------------------------- prepare and run


def _wf(api, shape, step, mass, boundary, propagator, psi, keep):
    w = api.wf(*shape, step, mass, boundary, propagator)
    keep.objs.append(w)
    view = _View(api, keep, w.grid)
    view.put(psi)
    return w, view


def _real(api, v, step, keep):
    r = api.rgrid(*v.shape, step)
    keep.objs.append(r)
    view = _View(api, keep, r)
    view.put(v)
    return r, view


def _complex(api, v, step, keep):
    c = api.cgrid(*v.shape, step)
    keep.objs.append(c)
    view = _View(api, keep, c)
    view.put(v.to(CD))
    return c, view


def prepare(case, seed):
    api, kind = _api(), case["kind"]
    lib, keep = api.lib, _Owned(api)
    if kind in ("step", "cn"):
        psi, v, h, mass, coupling, time = _step_inputs(case, seed)
        if kind == "step":
            w, view = _wf(api, v.shape, h, mass, capi.WF_PERIODIC_BOUNDARY, capi.WF_2ND_ORDER_FFT, psi, keep)
        else:
            w, view = _wf(api, v.shape, h, mass, case["boundary"], capi.WF_2ND_ORDER_CN, psi, keep)
            lib.cgrid_set_rotation(w.s.grid, case["omega"])
            if case["absorb"]:
                b = case["absorb"]
                lib.grid_wf_boundary(w.ptr, None, *(q for n in v.shape for q in (b, n - b)))
        pot, _ = (_real if coupling else _complex)(api, v, h, keep)
        if case.get("prec") == 32:
            w.precision(capi.GRID_PREC_FP32)
        t = capi.Complex.of(time)
        n = case.get("steps", 1)
        if coupling:
            args = (w.ptr, pot.ptr, coupling, t)
            call = (lib.grid_wf_propagate_gp, args) if n == 1 else (lib.grid_wf_propagate_gp_n, args + (n,))
        else:
            args = (w.ptr, pot.ptr, t)
            call = (lib.grid_wf_propagate, args) if n == 1 else (lib.grid_wf_propagate_n, args + (n,))
        return dict(kind=kind, call=call, view=view)
    if kind == "relax":
        psi, v, coupling, h = _relax_inputs(case, seed)
        lib.grid_wf_analyze_method(b"\x01")
        w, view = _wf(api, v.shape, h, 4.0 * AMU, capi.WF_PERIODIC_BOUNDARY, capi.WF_2ND_ORDER_FFT, psi, keep)
        pot, _ = _real(api, v, h, keep)
        rho, _ = _real(api, torch.zeros_like(v), h, keep)
        rho2, _ = _real(api, torch.zeros_like(v), h, keep)
        return dict(kind=kind, lib=lib, w=w, pot=pot, rho=rho.ptr, rho2=rho2.ptr, view=view, g=coupling,
                    time=capi.Complex.of(-2j), steps=case["steps"])
    if kind == "batch":
        wfs, pots, views = [], [], []
        for psi, v in _batch_inputs(case, seed):
            w, view = _wf(api, v.shape, 0.2, 1.0, capi.WF_PERIODIC_BOUNDARY, capi.WF_2ND_ORDER_FFT, psi, keep)
            pot, _ = _complex(api, v, 0.2, keep)
            if case["prec"] == 32:
                w.precision(capi.GRID_PREC_FP32)
            wfs, pots, views = wfs + [w], pots + [pot], views + [view]
        b = api.batch(wfs, pots, 0.05)
        keep.objs.insert(0, b)
        return dict(kind=kind, batch=b, views=views, steps=case["steps"])
    if kind == "observe":
        psi, v = _observe_inputs(case, seed)
        w, _ = _wf(api, v.shape, 0.5, 4.0 * AMU, case["boundary"], capi.WF_2ND_ORDER_CN, psi, keep)
        pot, _ = _real(api, v, 0.5, keep)
        rho, rview = _real(api, torch.zeros_like(v), 0.5, keep)
        grads = [_complex(api, torch.zeros_like(v), 0.5, keep) for _ in range(3)]
        return dict(kind=kind, lib=lib, w=w, pot=pot, rho=rho.ptr, rview=rview, grads=[g.ptr for g, _ in grads],
                    gviews=[x for _, x in grads])
    if kind == "convolve":
        rho, ker = _convolve_inputs(case, seed)
        a, _ = _real(api, rho, 0.5, keep)
        k, _ = _real(api, ker, 0.5, keep)
        work, view = _real(api, torch.zeros_like(rho), 0.5, keep)
        lib.rgrid_fft(k.ptr)  # the kernel stays in k-space for the whole run
        return dict(kind=kind, lib=lib, a=a.ptr, k=k.ptr, work=work.ptr, view=view)
    n = case["n"]
    if kind == "train":
        nb = case["batch"]
        net = warmstart.DeviceUNet(api, n, batch=nb)
        keep.objs.append(net)
        net.set_params(_net_params(seed))
        x, y = _net_inputs(seed, n, 2 * nb)
        ds = warmstart.DeviceSet(api.lib, 2 * nb, n**3)
        keep.objs.append(ds)
        _tensor(keep, ds.x, x.shape, "<f4").copy_(x)
        _tensor(keep, ds.y, y.shape, "<f4").copy_(y)
        torch.cuda.synchronize()
        net.prepare_training([2.0 / (n**3 * nb)], [nb])
        outs = [_tensor(keep, p, (net.nparam,), "<f4") for p in (net._p, net._m, net._v)]
        outs.append(_tensor(keep, net._act("out"), (nb, n, n, n), "<f4"))
        return dict(kind=kind, net=net, ds=ds, idx=_train_idx(seed, nb), scale=2.0 / (n**3 * nb), outs=outs)
    net = warmstart.DeviceUNet(api, n, batch=1)
    keep.objs.append(net)
    net.set_params(_net_params(seed))
    x, _ = _net_inputs(seed, n, 1)
    ds = warmstart.DeviceSet(api.lib, 1, n**3)
    keep.objs.append(ds)
    _tensor(keep, ds.x, x.shape, "<f4").copy_(x)
    torch.cuda.synchronize()
    net.infer_device(ds.xp(0))  # captures the inference graph
    return dict(kind=kind, net=net, x=ds.xp(0), out=_tensor(keep, net._act("out"), (1, n, n, n), "<f4"))


def _train_idx(seed, nb):
    return np.random.default_rng(seed + 1).permutation(2 * nb)[:nb].tolist()


def run(state):
    kind = state["kind"]
    if kind in ("step", "cn"):
        fn, args = state["call"]
        fn(*args)
        return state["view"].get()
    if kind == "relax":
        lib, w = state["lib"], state["w"]
        lib.grid_wf_relax_gp_n(w.ptr, state["pot"].ptr, state["g"], state["time"], state["steps"])
        e = w.energy(state["pot"])
        lib.grid_wf_density(w.ptr, state["rho"])
        lib.rgrid_product(state["rho2"], state["rho"], state["rho"])
        return state["view"].get(), e + 0.5 * state["g"] * lib.rgrid_integral(state["rho2"])
    if kind == "batch":
        state["batch"].propagate(state["steps"])
        return [v.get() for v in state["views"]]
    if kind == "observe":
        lib, w = state["lib"], state["w"]
        norm, e = w.norm(), w.energy(state["pot"])
        lib.grid_wf_density(w.ptr, state["rho"])
        gx, gy, gz = state["grads"]
        lib.cgrid_fd_gradient_x(w.s.grid, gx)
        lib.cgrid_fd_gradient_y(w.s.grid, gy)
        lib.cgrid_fd_gradient_z(w.s.grid, gz)
        return [norm, e, state["rview"].get()] + [v.get() for v in state["gviews"]]
    if kind == "convolve":
        lib, work = state["lib"], state["work"]
        lib.rgrid_copy(work, state["a"])
        lib.rgrid_fft(work)
        lib.rgrid_fft_convolute(work, work, state["k"])
        lib.rgrid_inverse_fft_norm2(work)
        return state["view"].get()
    if kind == "train":
        net = state["net"]
        net.train_set_batch(state["ds"], state["idx"], state["scale"])
        net.adam(2e-3)
        return state["outs"]
    state["net"].infer_device(state["x"])
    return state["out"]


# ----------------------------------------------------------- work and tolerance


def _conv_flops(n):
    lv = dict(e0=0, e1=1, e2=2, b=3, d2=2, d1=1, d0=0, out=0)
    return sum(2 * 27 * ci * co * (n >> lv[name if name == "out" else name[:-1]]) ** 3 for name, ci, co in _NET)


def work(case):
    kind = case["kind"]
    if kind in ("step", "cn", "observe", "convolve"):
        n = case["nx"] * case["ny"] * case["nz"]
    if kind == "step":
        pot = 8 if case["pot"] == "gp" else 16
        # psi and V in, psi out; the FP32 mode's result is read as FP64
        by = 32 + pot if case["prec"] == 64 else 8 + pot / 2 + 16
        return dict(bytes=n * by, flops=case["steps"] * n * (20 * math.log2(n) + 40))
    if kind == "relax":
        n = case["n"] ** 3
        return dict(bytes=n * 40, flops=case["steps"] * n * (20 * math.log2(n) + 45) + n * 5 * math.log2(n))
    if kind == "cn":
        return dict(bytes=n * (32 + (8 if case["pot"] == "gp" else 16)), flops=n * (3 * 60 + 2 * 40))
    if kind == "batch":
        n = case["per_size"] * 960 * case["nz"]
        by = 48 if case["prec"] == 64 else 24 + 24
        return dict(bytes=n * by, flops=case["steps"] * n * (10 * math.log2(n / case["per_size"] / 4) * 2 + 40))
    if kind == "observe":
        return dict(bytes=n * (16 + 8 + 8 + 48), flops=n * 45)
    if kind == "convolve":
        return dict(bytes=n * 24, flops=n * 5 * math.log2(n))
    n = case["n"]
    weights = sum(27 * ci * co + co for _, ci, co in _NET)
    if kind == "train":
        return dict(bytes=case["batch"] * n**3 * 20 + weights * 4 * 7, flops=3 * case["batch"] * _conv_flops(n))
    return dict(bytes=n**3 * 16 + weights * 2, flops=_conv_flops(n))


def tolerance(case):
    kind = case["kind"]
    if kind in ("step", "batch") and case["prec"] == 32:
        return {"rel": 5e-6, "max": 2e-4}
    if kind == "train" or kind == "infer":
        return {"rel": 1e-2, "max": 0.3}  # bf16 operands
    return {"rel": 2e-13, "max": 2e-11}  # FP64 throughout


# -------------------------------------------------------- plain 64-bit results


def _k2(shape, step):
    out = 0.0
    for d, n in enumerate(shape):
        i = torch.arange(n, device=DEV, dtype=FD)
        k = torch.where(i <= n // 2, i, i - n) * (2.0 * math.pi / (n * step))
        out = out + (k * k).reshape([-1 if a == d else 1 for a in range(3)])
    return out


def _split_steps(psi, v, coupling, step, mass, time, steps, norm_to=None):
    half = torch.exp(-0.5j * time / (2.0 * mass) * _k2(psi.shape, step))
    for _ in range(steps):
        psi = torch.fft.ifftn(torch.fft.fftn(psi) * half)
        psi = psi * torch.exp(-1j * time * (v + coupling * (psi.real**2 + psi.imag**2)))
        psi = torch.fft.ifftn(torch.fft.fftn(psi) * half)
        if norm_to:
            psi = psi * torch.sqrt(norm_to / ((psi.abs() ** 2).sum() * step**3))
    return psi


def _ramp(shape, b):
    t = 0.0
    for d, n in enumerate(shape):
        i = torch.arange(n, device=DEV, dtype=FD)
        r = torch.clamp(b - i, min=0.0) / b + torch.clamp(i - (n - b), min=0.0) / b
        t = t + r.reshape([-1 if a == d else 1 for a in range(3)])
    return torch.clamp(t * (2.0 / 3.0), max=1.0)


def _solve(sub, diag, sup, rhs):
    """Thomas elimination along dim 0; rhs [n, lines, systems]."""
    n = diag.shape[0]
    dp, rp = [diag[0]], [rhs[0]]
    for i in range(1, n):
        m = sub[i] / dp[-1]
        dp.append(diag[i] - m * sup[i - 1])
        rp.append(rhs[i] - m[:, None] * rp[-1])
    x = [rp[-1] / dp[-1][:, None]]
    for i in range(n - 2, -1, -1):
        x.append((rp[i] - sup[i][:, None] * x[-1]) / dp[i][:, None])
    return torch.stack(x[::-1])


def _cn_axis(psi, axis, step, mass, time, boundary, omega, ramp):
    """One Crank-Nicolson sweep: (cp - 2 +- c2) couplings, the boundary rows
    as the library defines them."""
    shape = psi.shape
    n = shape[axis]
    if n == 1:
        return psi
    xy = _axes(shape, step)
    turn = 1j * mass * omega * step  # the rotation couples x sweeps to y and y sweeps to x
    c3 = (turn * xy[1], -turn * xy[0], torch.zeros((1, 1, 1), device=DEV, dtype=CD))[axis].expand(shape)
    tim = torch.full(shape, complex(time), device=DEV, dtype=CD)
    if ramp is not None:
        tim = torch.complex((1.0 - ramp) * time.real, -time.real * ramp)
    lines = lambda t: t.movedim(axis, 0).reshape(n, -1)  # noqa: E731
    p, c, cp = lines(psi), lines(c3), lines(4j * mass * step * step / tim)
    up, dn = torch.roll(p, -1, 0), torch.roll(p, 1, 0)
    if boundary != capi.WF_PERIODIC_BOUNDARY:
        up[-1], dn[0] = 0.0, 0.0
    rhs = cp * p - (up - 2.0 * p + dn) - c * (up - dn)
    sub, sup, diag = 1.0 - c, 1.0 + c, cp - 2.0
    if boundary == capi.WF_NEUMANN_BOUNDARY:
        rhs[0] = cp[0] * p[0] - 2.0 * (p[1] - p[0])
        rhs[-1] = cp[-1] * p[-1] - 2.0 * (p[-2] - p[-1])
    if boundary != capi.WF_PERIODIC_BOUNDARY:
        sub, sup = sub.clone(), sup.clone()
        sub[-1], sup[0] = 2.0, 2.0
        x = _solve(sub, diag, sup, rhs[:, :, None])[:, :, 0]
    else:  # Sherman-Morrison for the two corner elements
        low, high, gamma = sup[0], sub[0], -diag[0]
        diag = diag.clone()
        diag[0] = diag[0] - gamma
        diag[-1] = diag[-1] - low * high / gamma
        u = torch.zeros_like(rhs)
        u[0], u[-1] = gamma, low
        s = _solve(sub, diag, sup, torch.stack([rhs, u], 2))
        y, z = s[:, :, 0], s[:, :, 1]
        x = y - z * (y[0] + high * y[-1] / gamma) / (1.0 + z[0] + high * z[-1] / gamma)
    return x.reshape([n] + [m for d, m in enumerate(shape) if d != axis]).movedim(0, axis)


def _cn_step(psi, v, coupling, step, mass, time, case):
    ramp = _ramp(psi.shape, case["absorb"]) if case["absorb"] else None
    for part in range(2):
        c = -0.5j * time
        if ramp is not None:
            c = torch.complex(-0.5 * time.real * ramp, -0.5 * time.real * (1.0 - ramp))
        if part == 1:
            for axis in range(3):
                psi = _cn_axis(psi, axis, step, mass, time, case["boundary"], case["omega"], ramp)
        psi = psi * torch.exp(c * (v + coupling * (psi.real**2 + psi.imag**2)))
    return psi


def _outside(psi, axis, shift, boundary):
    """Neighbour at +shift along an axis, with the grid's boundary rule."""
    out = torch.roll(psi, -shift, axis)
    if boundary != capi.WF_PERIODIC_BOUNDARY:
        n = psi.shape[axis]
        edge = n - 1 if shift > 0 else 0
        mirror = n - 2 if shift > 0 else 1
        val = psi.select(axis, mirror) if boundary == capi.WF_NEUMANN_BOUNDARY else 0.0
        out.select(axis, edge).copy_(torch.as_tensor(val, device=DEV, dtype=CD))
    return out


def _net_forward(x, flat, bf16):
    """The network in 64 bits; returns (output, weight leaves, bias leaves)."""
    F = torch.nn.functional
    ws, bs, off = {}, {}, 0
    for name, ci, co in _NET:
        w = flat[off : off + co * ci * 27].reshape(co, ci, 3, 3, 3)
        b = flat[off + co * ci * 27 : off + co * ci * 27 + co]
        ws[name] = (w.bfloat16() if bf16 else w).double().requires_grad_()
        bs[name] = b.double().requires_grad_()
        off += co * ci * 27 + co

    def conv(name, t, relu=True):
        t = F.conv3d(t, ws[name], bs[name], padding=1)
        return torch.relu(t) if relu else t

    e0 = conv("e0b", conv("e0a", x))
    e1 = conv("e1b", conv("e1a", F.avg_pool3d(e0, 2)))
    e2 = conv("e2b", conv("e2a", F.avg_pool3d(e1, 2)))
    t = conv("bb", conv("ba", F.avg_pool3d(e2, 2)))
    for lv, skip in (("d2", e2), ("d1", e1), ("d0", e0)):
        t = torch.cat([F.interpolate(t, scale_factor=2, mode="nearest"), skip], 1)
        t = conv(lv + "b", conv(lv + "a", t))
    return conv("out", t, False)[:, 0], ws, bs


def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        psi, v, h, mass, coupling, time = _step_inputs(case, seed)
        return _split_steps(psi, v, coupling, h, mass, time, case["steps"])
    if kind == "relax":
        psi, v, coupling, h = _relax_inputs(case, seed)
        psi = _split_steps(psi, v, coupling, h, 4.0 * AMU, -2j, case["steps"], 1.0)
        rho, n = psi.abs() ** 2, psi.numel()
        e = (_k2(psi.shape, h) * torch.fft.fftn(psi).abs() ** 2).sum() / n / (8.0 * AMU)
        return psi, float((e + (v * rho).sum() + 0.5 * coupling * (rho * rho).sum()) * h**3)
    if kind == "cn":
        psi, v, h, mass, coupling, time = _step_inputs(case, seed)
        return _cn_step(psi, v, coupling, h, mass, time, case)
    if kind == "batch":
        return [_split_steps(psi, v, 0.0, 0.2, 1.0, 0.05 + 0j, case["steps"]) for psi, v in _batch_inputs(case, seed)]
    if kind == "observe":
        psi, v = _observe_inputs(case, seed)
        b, h, rho = case["boundary"], 0.5, psi.abs() ** 2
        pairs = [(_outside(psi, d, 1, b), _outside(psi, d, -1, b)) for d in range(3)]
        lap = (sum(u + w for u, w in pairs) - 6.0 * psi) / h**2
        e = (-(psi.conj() * lap).real / (8.0 * AMU) + v * rho).sum() * h**3
        return [float(rho.sum() * h**3), float(e), rho] + [(u - w) / (2.0 * h) for u, w in pairs]
    if kind == "convolve":
        rho, ker = _convolve_inputs(case, seed)
        i, j, k = (torch.arange(n, device=DEV) for n in rho.shape)
        sign = 1.0 - 2.0 * ((i[:, None, None] + j[None, :, None] + k) % 2).to(FD)
        return torch.fft.ifftn(torch.fft.fftn(rho) * torch.fft.fftn(ker) * sign).real * 0.5**3
    n = case["n"]
    flat = torch.as_tensor(_net_params(seed), device=DEV)
    if kind == "infer":
        x, _ = _net_inputs(seed, n, 1)
        with torch.no_grad():
            return _net_forward(x.double(), flat, True)[0]
    nb = case["batch"]
    x, y = _net_inputs(seed, n, 2 * nb)
    idx = _train_idx(seed, nb)
    out, ws, bs = _net_forward(x[idx].double(), flat, True)
    (((out - y[idx].double()) ** 2).sum() / (n**3 * nb)).backward()
    g = torch.cat([t.grad.reshape(-1) for name, _, _ in _NET for t in (ws[name], bs[name])])
    p = flat.double() - 2e-3 * g / (g.abs() + 1e-8)
    return [p, 0.1 * g, 0.001 * g * g, out.detach()]
