"""The work whose speed is measured: what programs that use the dynamical core
have it do, through its public entry points.

* "step": a forecast leg on a device-resident core.  The program holds the
  state in page-locked host arrays, uploads it, takes some time steps and
  downloads the result (DynamicalCore.upload_state / driver_start / step /
  download_state), in FP64 or in the mixed form, with tracers or the subgrid
  model where a case says so;
* "ensemble": the same for independent domains of uneven sizes advanced
  together (Ensemble.step);
* "bicgstab", "mpdata": one call of a drop-in routine on host arrays, as the
  Fortran driver makes it;
* "columns": the sedimentation transport of many columns, on device arrays of
  the caller or on host arrays.

The flows are the package's own workloads (a shear layer, a warm bubble, a
sheared convection with tracers), built here on the GPU from the seed.
"""
import ctypes
import importlib
import math
import random

import numpy as np
import torch

pkg = importlib.import_module("dynamical-cloud-model_b200")
wl = importlib.import_module("dynamical-cloud-model_b200.cases")

Z0 = 0.1      # roughness length of the cases with the subgrid model, m
GRAV = 9.81
FIELDS = ("u", "v", "w", "zu", "zv", "zw", "th", "p")
SCRATCH = ("tu", "tv", "tw", "su", "sv", "sw", "psrc", "div", "sth")


def _step(name, flow, ip, jp, kp, steps, precision=0, precond=0, kord=3, tracers=0,
          viscous=False):
    c = {"kind": "step", "flow": flow, "ip": ip, "jp": jp, "kp": kp, "steps": steps,
         "precision": precision, "precond": precond, "kord": kord, "tracers": tracers,
         "viscous": viscous}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the 2-D shear layer of the CPU-runnable configuration: a domain so
        # small that launches and latencies are what its steps cost
        _step("shear_fp64_128x1x64", "shear", 128, 1, 64, 20, kord=2),
        # the headline: the 3-D warm bubble in the mixed form
        _step("bubble_mixed_256x256x128", "bubble", 256, 256, 128, 10, precision=1, precond=1),
        # the same domain on the FP64 path that parity with the reference asks for
        _step("bubble_fp64_256x256x128", "bubble", 256, 256, 128, 2),
        # a larger convective domain with columns of 256 levels: fields far above L2
        _step("convection_mixed_384x256x256", "convection", 384, 256, 256, 2, precision=1,
              precond=1),
        # tracers beside theta: most of a step is advection
        _step("tracers_mixed_192x160x96", "convection", 192, 160, 96, 4, precision=1,
              precond=1, tracers=6),
        # odd sizes, the mixed form's default options, one antidiffusive pass
        _step("bubble_mixed_97x75x61", "bubble", 97, 75, 61, 10, precision=1, kord=2),
        # the subgrid model in the step, odd sizes, FP64
        _step("subgrid_fp64_90x83x64", "convection", 90, 83, 64, 4, viscous=True),
        # an ensemble of uneven warm-bubble domains, mixed form
        {"name": "ensemble_mixed_10", "kind": "ensemble", "members": 10, "pick": 5, "steps": 3},
        # one pressure solve and one advection called on host arrays
        {"name": "bicgstab_128x96x64", "kind": "bicgstab", "ip": 128, "jp": 96, "kp": 64},
        {"name": "mpdata_256x256x128", "kind": "mpdata", "ip": 256, "jp": 256, "kp": 128,
         "nq": 1, "kord": 3},
        # the microphysics' sedimentation: many columns that live on the device
        {"name": "columns_device_65536x128", "kind": "columns", "ncol": 65536, "kp": 128,
         "nq": 2, "kord": 1, "monotone": False, "device": True},
        # and a few, on host arrays, with the limiter: the smallest call
        {"name": "columns_host_513x120", "kind": "columns", "ncol": 513, "kp": 120, "nq": 2,
         "kord": 3, "monotone": True, "device": False},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mixed", "mixed", "mixed", "fp64", "shear", "tracers", "subgrid",
                       "ensemble", "bicgstab", "mpdata", "columns", "columns"])
    if kind in ("mixed", "fp64", "tracers", "subgrid"):
        big = {"mixed": 320, "fp64": 200, "tracers": 160, "subgrid": 128}[kind]
        ip, jp, kp = _size(rng, 40, big), _size(rng, 40, big), _size(rng, 32, big // 2 + 32)
        n = ip * jp * kp
    if kind == "mixed":
        return _step(None, rng.choice(["bubble", "convection"]), ip, jp, kp,
                     max(2, min(12, int(2.5e7 / n))), precision=1, precond=rng.choice([0, 1, 1]),
                     kord=rng.choice([2, 3, 3]))
    if kind == "fp64":
        return _step(None, rng.choice(["bubble", "convection"]), ip, jp, kp,
                     max(1, min(8, int(1.2e7 / n))), kord=rng.choice([2, 3, 3]))
    if kind == "shear":
        return _step(None, "shear", _size(rng, 64, 512), 1, _size(rng, 48, 128),
                     rng.randint(5, 20), kord=2)
    if kind == "tracers":
        return _step(None, "convection", ip, jp, kp, rng.randint(2, 4), precision=1, precond=1,
                     tracers=rng.randint(1, 6))
    if kind == "subgrid":
        return _step(None, "convection", ip, jp, kp, rng.randint(2, 4), viscous=True,
                     kord=rng.choice([2, 3]))
    if kind == "ensemble":
        return {"kind": "ensemble", "members": rng.randint(3, 8), "pick": rng.randint(1, 9999),
                "steps": rng.randint(2, 3)}
    if kind == "bicgstab":
        return {"kind": "bicgstab", "ip": _size(rng, 24, 200), "jp": _size(rng, 24, 200),
                "kp": _size(rng, 24, 128)}
    if kind == "mpdata":
        return {"kind": "mpdata", "ip": _size(rng, 32, 200), "jp": _size(rng, 32, 200),
                "kp": _size(rng, 24, 128), "nq": rng.choice([1, 1, 3]),
                "kord": rng.choice([2, 3])}
    device = rng.random() < 0.5
    kord = rng.choice([1, 1, 3])
    return {"kind": "columns", "ncol": _size(rng, 512, 65536 if device else 8192),
            "kp": _size(rng, 30, 140), "nq": rng.randint(1, 3), "kord": kord,
            "monotone": kord > 1, "device": device}


# --- inputs -----------------------------------------------------------------

def _pinned(*shape):
    """A page-locked Fortran-ordered float64 array, zeroed."""
    t = torch.empty(tuple(reversed(shape)), dtype=torch.float64, pin_memory=True)
    t.zero_()
    return t.numpy().transpose(*range(len(shape) - 1, -1, -1))


def _put(a, t):
    """A GPU tensor (k, j, i) into the Fortran-ordered array a."""
    torch.from_numpy(a.transpose(2, 1, 0)).copy_(t.permute(2, 1, 0).contiguous())


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 11)


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _fill_full(a, lbc=0.0, ubc=0.0):
    """Periodic images in every halo cell, lbc / ubc on the bottom and top planes."""
    a[0], a[-1] = a[-2].clone(), a[1].clone()
    a[:, 0], a[:, -1] = a[:, -2].clone(), a[:, 1].clone()
    a[:, :, 0], a[:, :, -1] = a[:, :, -2].clone(), a[:, :, 1].clone()
    a[0, 1:-1, 1:-1] = lbc
    a[-1, 1:-1, 1:-1] = ubc


def _flow(flow, ip, jp, kp, gen, tracers=0, amp=2.0):
    """Grid, time step, and the initial u, theta' and tracers as GPU tensors."""
    kw = dict(dtype=torch.float64, device="cuda", generator=gen)
    th = torch.zeros(kp + 2, jp + 2, ip + 2, dtype=torch.float64, device="cuda")
    q = []
    if flow == "shear":
        d, dt = 20.0, 0.5
        zn = d * np.arange(kp + 2) - 0.5 * d
        mid = 0.5 * d * kp
        g = wl.make_grid(ip, jp, kp, d, d, d, zn, np.where(zn < mid, 300.0, 302.0))
        u = 10.0 * np.tanh((g.zn - mid) / 50.0)
        th[1:-1, 1:-1, 1:-1] = 0.2 * torch.rand(kp, jp, ip, **kw) - 0.1
    elif flow == "bubble":
        d, dt = 50.0, 1.0
        g = wl.make_grid(ip, jp, kp, d, d, d, [-1.0e4, 1.0e5], [300.0, 300.0])
        u = np.zeros(kp + 2)
        r0 = min(1000.0, 0.3 * d * min(ip, jp, kp))
        X, Y = _t(g.xn)[None, None, 1:-1], _t(g.yn)[None, 1:-1, None]
        Z = _t(g.zn)[1:-1, None, None]
        r = torch.sqrt(X * X + Y * Y + (Z - 1.5 * r0) ** 2)
        th[1:-1, 1:-1, 1:-1] = torch.where(
            r <= r0, amp * torch.cos(math.pi * r / (2.0 * r0)) ** 2,
            torch.zeros_like(r)) + 0.01 * torch.randn(kp, jp, ip, **kw)
    else:
        d, dt = 25.0, 0.5
        g = wl.make_grid(ip, jp, kp, d, d, d, [-1.0e4, 1.0e5], [300.0, 300.0])
        u = 5.0 * g.zn / 6400.0
        low = (_t(g.zn)[1:-1, None, None] < 500.0).double()
        th[1:-1, 1:-1, 1:-1] = low * (torch.rand(kp, jp, ip, **kw) - 0.5)
        for _ in range(tracers):
            a = torch.zeros_like(th)
            a[1:-1, 1:-1, 1:-1] = torch.rand(kp, jp, ip, **kw)
            _fill_full(a)
            q.append(a)
    u[:2], u[kp] = 0.0, 0.0
    uu = _t(u)[:, None, None].expand(kp + 2, jp + 2, ip + 2).clone()
    zu = uu.clone()
    _fill_full(uu)
    _fill_full(th)
    return g, dt, uu, zu, th, q


def _case_flow(case, seed):
    return _flow(case["flow"], case["ip"], case["jp"], case["kp"], _gen(seed), case["tracers"])


def _state(g, uu, zu, th, q):
    """The State of a flow that starts with v = w = p = 0 and equal time levels;
    the arrays are only read, so equal fields share one."""
    sh = g.shape
    U, TH, zero = _pinned(*sh), _pinned(*sh), _pinned(*sh)
    _put(U, uu)
    _put(TH, th)
    Z = U
    if not torch.equal(uu, zu):
        Z = _pinned(*sh)
        _put(Z, zu)
    st = wl.State(U, zero, zero, Z, zero, zero, Z, zero, zero, TH, zero)
    if q:
        st.q = [_pinned(*sh) for _ in q]
        for a, t in zip(st.q, q):
            _put(a, t)
    return st


def _buffers(g, keep=FIELDS):
    """Page-locked destinations of a download; the fields the program does not
    look at share one."""
    junk = _pinned(*g.shape)
    return {n: (_pinned(*g.shape) if n in keep else junk) for n in FIELDS + SCRATCH}


def _viscous(g):
    return dict(lamsq=wl.mixing_length_sq(g, 0.23, Z0), z0=Z0, z0th=Z0)


MEMBER_FIELDS = ("u", "v", "w", "th", "p")


def _members(case):
    r = random.Random(case["pick"])
    return [(r.choice([64, 96, 128, 192]), r.choice([64, 96, 128, 192]), r.choice([48, 64, 96]),
             r.uniform(1.0, 3.0)) for _ in range(case["members"])]


def _solve_input(case, seed):
    """A pressure source with zero mean, as the driver's has: smooth
    structures and noise."""
    ip, jp, kp = case["ip"], case["jp"], case["kp"]
    g = wl.make_grid(ip, jp, kp, 50.0, 50.0, 50.0, [-1.0e4, 1.0e5], [300.0, 300.0])
    gen = _gen(seed)
    kw = dict(dtype=torch.float64, device="cuda", generator=gen)
    ph = 2.0 * math.pi * torch.rand(3, **kw)
    X = 2.0 * math.pi * torch.arange(ip, device="cuda").double() / ip
    Y = 2.0 * math.pi * torch.arange(jp, device="cuda").double() / jp
    Z = math.pi * (torch.arange(kp, device="cuda").double() + 0.5) / kp
    r = (torch.cos(X + ph[0])[None, None, :] * torch.cos(2.0 * Y + ph[1])[None, :, None] +
         0.5 * torch.cos(3.0 * Z)[:, None, None] * torch.sin(2.0 * X + ph[2])[None, None, :])
    r = 1.0e-4 * (r + 0.1 * torch.randn(kp, jp, ip, **kw))
    b = torch.zeros(kp + 2, jp + 2, ip + 2, dtype=torch.float64, device="cuda")
    b[1:-1, 1:-1, 1:-1] = r - r.mean()
    return g, b


def _advection_input(case, seed):
    """A flow with rho-weighted divergence zero (a stream function in x-z, a
    shear along y) and positive fields."""
    ip, jp, kp = case["ip"], case["jp"], case["kp"]
    g = wl.make_grid(ip, jp, kp, 50.0, 50.0, 50.0, [-1.0e4, 1.0e5], [300.0, 300.0])
    gen = _gen(seed)
    kw = dict(dtype=torch.float64, device="cuda", generator=gen)
    ph = 2.0 * math.pi * torch.rand(2, **kw)
    i = torch.arange(ip + 2, device="cuda").double()
    k = torch.arange(kp + 2, device="cuda").double()
    psi = 1500.0 * torch.sin(2.0 * math.pi * i / ip + ph[0])[None, :] * \
        torch.sin(math.pi * k / kp)[:, None]
    rn, ra = _t(g.rhoan)[:, None], _t(g.rhoa)[:, None]
    u2, w2 = torch.zeros_like(psi), torch.zeros_like(psi)
    u2[1:] = (psi[1:] - psi[:-1]) / 50.0 / rn[1:]
    w2[:, 1:] = -(psi[:, 1:] - psi[:, :-1]) / 50.0 / ra
    shape = (kp + 2, jp + 2, ip + 2)
    u, w = (a[:, None, :].expand(shape).clone() for a in (u2, w2))
    v = (8.0 * torch.sin(2.0 * math.pi * i / ip + ph[1]))[None, None, :].expand(shape).clone()
    for a in (u, v, w):
        _fill_full(a)
    f = []
    for _ in range(case["nq"]):
        a = torch.zeros(shape, dtype=torch.float64, device="cuda")
        a[1:-1, 1:-1, 1:-1] = torch.rand(kp, jp, ip, **kw)
        _fill_full(a)
        f.append(a)
    return g, 1.0, u, v, w, f


def _column_input(case, seed):
    """Fall speeds up to 8 m/s, hydrometeor mixing ratios with clear layers,
    and the microphysics' number of sub-steps per column."""
    ncol, nq, kp = case["ncol"], case["nq"], case["kp"]
    gen = _gen(seed)
    kw = dict(dtype=torch.float64, device="cuda", generator=gen)
    z = np.linspace(0.0, 1.0, kp + 2)
    met = [_t(a) for a in (40.0 + 20.0 * z, 45.0 + 10.0 * z, 1.2 - 0.5 * z, 1.2 - 0.5 * z)]
    w = -8.0 * torch.rand(ncol, kp + 2, **kw) * torch.rand(ncol, 1, **kw)
    psi = 1e-3 * torch.rand(ncol, nq, kp + 2, **kw) * \
        (torch.rand(ncol, nq, kp + 2, **kw) > 0.3).double()
    dt = torch.full((ncol,), 2.0, dtype=torch.float64, device="cuda")
    ns = torch.clamp(torch.ceil(w.abs().amax(dim=1) * 2.0 / 40.0 * 2.0), min=1).to(torch.int32)
    return met, w, psi, dt, ns


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind == "step":
        g, dt, uu, zu, th, q = _case_flow(case, seed)
        s["core"] = pkg.DynamicalCore(g)
        s["state"] = _state(g, uu, zu, th, q)
        nq = case["tracers"]
        each = tuple(range(1, nq + 1))
        s["dt"], s["out"] = dt, _buffers(g)
        s["kw"] = dict(kord=case["kord"], precision=case["precision"], precond=case["precond"],
                       nq=nq, c_s=each, c_e=each,
                       viscous=_viscous(g) if case["viscous"] else None)
    elif kind == "ensemble":
        flows = [_flow("bubble", ip, jp, kp, _gen(1000 * seed + m), amp=amp)
                 for m, (ip, jp, kp, amp) in enumerate(_members(case))]
        s["ens"] = pkg.Ensemble([f[0] for f in flows])
        s["dt"] = flows[0][1]
        s["states"] = [_state(f[0], *f[2:]) for f in flows]
        s["outs"] = [_buffers(f[0], MEMBER_FIELDS) for f in flows]
    elif kind == "bicgstab":
        g, b = _solve_input(case, seed)
        s["core"] = pkg.DynamicalCore(g)
        s["b"], s["x"], s["sw"] = (np.zeros(g.shape, order="F") for _ in range(3))
        _put(s["b"], b)
    elif kind == "mpdata":
        g, s["dt"], u, v, w, f = _advection_input(case, seed)
        s["core"] = pkg.DynamicalCore(g)
        for n, t in (("u", u), ("v", v), ("w", w)):
            s[n] = np.zeros(g.shape, order="F")
            _put(s[n], t)
        s["psi"] = pkg.fortran_stack([np.zeros(g.shape, order="F") for _ in f])
        for n, t in enumerate(f):
            _put(s["psi"][n], t)
    else:
        met, w, psi, dt, ns = _column_input(case, seed)
        s["psi0"] = psi
        if case["device"]:
            s["args"] = [dt, ns] + met + [w]
            s["psi"] = psi.clone()
            s["lib"] = pkg.library()
        else:
            s["met"], s["w"] = [a.cpu().numpy() for a in met], w.cpu().numpy()
            s["nsub"], s["psi0"] = ns.cpu().numpy(), psi.cpu().numpy()
            s["psi"] = s["psi0"].copy()
    return s


def _inner(a):
    return a[..., 1:-1, 1:-1, 1:-1]


def run(s):
    kind = s["kind"]
    if kind == "step":
        core = s["core"]
        core.upload_state(s["state"], s["dt"], **s["kw"])
        core.driver_start()
        core.step(s["steps"])
        got = core.download_state(out=s["out"])
        return {n: _inner(got[n]) for n in FIELDS + (("q",) if s["tracers"] else ())}
    if kind == "ensemble":
        members = s["ens"].members
        for core, st in zip(members, s["states"]):
            core.upload_state(st, s["dt"], kord=3, precision=1, precond=1)
            core.driver_start()
        s["ens"].step(s["steps"])
        got = [core.download_state(out=o) for core, o in zip(members, s["outs"])]
        return [{n: _inner(f[n]) for n in MEMBER_FIELDS} for f in got]
    if kind == "bicgstab":
        s["x"].fill(0.0)
        s["core"].bicgstab(s["x"], s["b"], s["sw"], 1e-10)
        return _inner(s["x"])
    if kind == "mpdata":
        if s["nq"] == 1:
            s["core"].mpdata_3d(s["dt"], s["u"], s["v"], s["w"], s["psi"][0], 0.0, 0.0,
                                s["kord"], True)
        else:
            lb, ub = np.zeros(s["nq"]), np.zeros(s["nq"])
            s["core"].mpdata_vec_3d(s["dt"], s["u"], s["v"], s["w"], s["psi"], lb, ub,
                                    s["kord"], True)
        return s["psi"]
    if s["device"]:
        s["psi"].copy_(s["psi0"])
        p = [ctypes.c_void_p(t.data_ptr()) for t in s["args"]]
        st = s["lib"].dcm_mpdata_vec_1d_device(
            s["ncol"], s["kp"], s["nq"], 1, 1, p[0], p[1], *p[2:6], 0, p[6],
            ctypes.c_void_p(s["psi"].data_ptr()), s["kord"], int(s["monotone"]), 0,
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if st:
            raise RuntimeError("dcm_mpdata_vec_1d_device: status %d" % st)
        return s["psi"]
    np.copyto(s["psi"], s["psi0"])
    return pkg.mpdata_vec_1d_columns(2.0, s["nsub"], *s["met"], s["w"], s["psi"], kord=s["kord"],
                                     monotone=s["monotone"])


def work(case):
    """Each pass's inputs read once and outputs written once: the host copies of
    the state, and per time step the prognostic fields (u, v, w and their
    previous level, theta, p, tracers) in and out."""
    kind = case["kind"]
    if kind in ("step", "ensemble"):
        if kind == "step":
            n, q = case["ip"] * case["jp"] * case["kp"], case["tracers"]
            word = 4 if case["precision"] else 8
        else:
            n, q, word = sum(i * j * k for i, j, k, _ in _members(case)), 0, 4
        return {"bytes": n * (8 * (19 + 2 * q) + word * case["steps"] * (16 + 2 * q)),
                "flops": n * case["steps"] * (500 + 300 * (1 + q))}
    if kind == "columns":
        n = case["ncol"] * (case["kp"] + 2)
        return {"bytes": n * 8 * (2 * case["nq"] + 1),
                "flops": n * case["nq"] * (20 if case["kord"] == 1 else 150)}
    n = case["ip"] * case["jp"] * case["kp"]
    if kind == "bicgstab":
        return {"bytes": 16 * n, "flops": 100 * n}
    return {"bytes": 8 * n * (3 + 2 * case["nq"]), "flops": 300 * n * case["nq"]}


# --- the same in plain 64-bit torch -----------------------------------------

I, M, P = slice(1, -1), slice(0, -2), slice(2, None)  # interior, index - 1, index + 1
TINY = 1e-60


class _Grid:
    """1-D metrics as broadcastable tensors; kp levels along the first axis."""

    def __init__(self, g):
        self.g, self.kp, self.jp, self.ip = g, g.kp, g.jp, g.ip
        for n in ("rhoa", "rhoan", "theta", "thetan", "z"):
            setattr(self, n, _t(getattr(g, n))[:, None, None])
        self.dx, self.dy, self.dz = float(g.dx[1]), float(g.dy[1]), float(g.dz[1])

    def poisson(self, b):
        """The zero-mean solution of the 7-point equation, periodic in x and y
        and mirrored in z, by transforms in all three directions."""
        kp, jp, ip = self.kp, self.jp, self.ip
        kw = dict(dtype=torch.float64, device="cuda")
        m = torch.arange(kp, **kw)
        basis = torch.cos(math.pi * m[:, None] * (m[None, :] + 0.5) / kp) * math.sqrt(2.0 / kp)
        basis[0] /= math.sqrt(2.0)
        f = torch.fft.rfft2((basis @ b.reshape(kp, -1)).reshape(kp, jp, ip))
        lz = (2.0 * torch.cos(math.pi * m / kp) - 2.0) / self.dz ** 2
        ly = (2.0 * torch.cos(2.0 * math.pi * torch.arange(jp, **kw) / jp) - 2.0) / self.dy ** 2
        lx = (2.0 * torch.cos(2.0 * math.pi * torch.arange(ip // 2 + 1, **kw) / ip) - 2.0) / \
            self.dx ** 2
        lam = lz[:, None, None] + ly[None, :, None] + lx[None, None, :]
        lam[0, 0, 0] = 1.0
        f = f / lam
        f[0, 0, 0] = 0.0
        x = torch.fft.irfft2(f, s=(jp, ip)).reshape(kp, -1)
        return (basis.T @ x).reshape(kp, jp, ip)

    def donor(self, dt, u, v, w, a):
        ra, rn = self.rhoa, self.rhoan[I]
        c = a[I, I, I]

        def flux(vel, lo, hi):
            return torch.clamp(vel, min=0.0) * lo + torch.clamp(vel, max=0.0) * hi
        fx = flux(u[I, I, I], c, a[I, I, P]) - flux(u[I, I, M], a[I, I, M], c)
        fy = flux(v[I, I, I], c, a[I, P, I]) - flux(v[I, M, I], a[I, M, I], c)
        fz = flux(w[I, I, I] * ra[I], c, a[P, I, I]) - flux(w[M, I, I] * ra[M], a[M, I, I], c)
        return c - dt * (fx / self.dx + fy / self.dy + fz / (self.dz * rn))

    def antidiffusive(self, dt, u, v, w, p):
        ra, rn, rnp = self.rhoa, self.rhoan[I], self.rhoan[P]
        rk, rm, rp = ra[I], ra[M], ra[P]
        g3 = 0.5 * (rn + rnp)
        dx, dy, dz = self.dx, self.dy, self.dz

        def ratio(a, b, c, d):
            return (a + b - c - d) / (a + b + c + d + TINY)
        uc, vc, wc = u[I, I, I], v[I, I, I], w[I, I, I]
        d1 = (rk * (wc + w[I, I, P]) - rm * (w[M, I, I] + w[M, I, P])) / (dz * rn) + \
            (vc + v[I, I, P] - v[I, M, I] - v[I, M, P]) / dy
        d2 = (rk * (wc + w[I, P, I]) - rm * (w[M, I, I] + w[M, P, I])) / (dz * rn) + \
            (uc + u[I, P, I] - u[I, I, M] - u[I, P, M]) / dx
        d3 = (rn * (uc - u[I, I, M]) + rnp * (u[P, I, I] - u[P, I, M])) / (dx * g3) + \
            (rn * (vc - v[I, M, I]) + rnp * (v[P, I, I] - v[P, M, I])) / (dy * g3)
        b1 = (rk * (w[I, I, P] + wc) + rm * (w[M, I, P] + w[M, I, I])) / rn / dz * \
            ratio(p[P, I, P], p[P, I, I], p[M, I, P], p[M, I, I]) + \
            (v[I, I, P] + vc + v[I, M, P] + v[I, M, I]) / dy * \
            ratio(p[I, P, P], p[I, P, I], p[I, M, P], p[I, M, I])
        b2 = (rk * (w[I, P, I] + wc) + rm * (w[M, P, I] + w[M, I, I])) / rn / dz * \
            ratio(p[P, P, I], p[P, I, I], p[M, P, I], p[M, I, I]) + \
            (u[I, P, I] + uc + u[I, P, M] + u[I, I, M]) / dx * \
            ratio(p[I, P, P], p[I, I, P], p[I, P, M], p[I, I, M])
        b3 = (rnp * (v[P, I, I] + v[P, M, I]) + rn * (vc + v[I, M, I])) / g3 / dy * \
            ratio(p[P, P, I], p[I, P, I], p[P, M, I], p[I, M, I]) + \
            (rnp * (u[P, I, I] + u[P, I, M]) + rn * (uc + u[I, I, M])) / g3 / dx * \
            ratio(p[P, I, P], p[I, I, P], p[P, I, M], p[I, I, M])
        pc = p[I, I, I]
        us = (uc.abs() * dx - dt * uc * uc) * (p[I, I, P] - pc) / (p[I, I, P] + pc + TINY) / dx
        vs = (vc.abs() * dy - dt * vc * vc) * (p[I, P, I] - pc) / (p[I, P, I] + pc + TINY) / dy
        ws = (wc.abs() * dz - dt * (rk / g3) * wc * wc) * (p[P, I, I] - pc) / \
            (p[P, I, I] + pc + TINY) / dz
        us = us - 0.125 * dt * uc * b1 - 0.25 * dt * uc * ((u[I, I, P] - u[I, I, M]) / dx + d1)
        vs = vs - 0.125 * dt * vc * b2 - 0.25 * dt * vc * ((v[I, P, I] - v[I, M, I]) / dy + d2)
        ws = ws - 0.125 * dt * wc * b3 - \
            0.25 * dt * wc * ((rp * w[P, I, I] - rm * w[M, I, I]) / (dz * g3) + d3)
        return [self.filled(a) for a in (us, vs, ws)]

    def stress(self, inner):
        """A stress with zero top and bottom planes and periodic faces."""
        a = self.filled(inner)
        a[0], a[-1] = 0.0, 0.0
        return a

    def filled(self, inner, lbc=0.0, ubc=0.0):
        a = torch.zeros(self.kp + 2, self.jp + 2, self.ip + 2, dtype=torch.float64,
                        device="cuda")
        a[I, I, I] = inner
        _fill_full(a, lbc, ubc)
        return a

    def limited(self, dt, u, v, w, first, p):
        ra, rn = self.rhoa, self.rhoan[I]
        hi = lo = p[I, I, I]
        for f in (first, p):
            for n in ((I, I, I), (I, I, M), (I, I, P), (I, M, I), (I, P, I), (M, I, I),
                      (P, I, I)):
                hi, lo = torch.maximum(hi, f[n]), torch.minimum(lo, f[n])

        def pos(a):
            return torch.clamp(a, min=0.0)

        def neg(a):
            return torch.clamp(a, max=0.0)
        pc = p[I, I, I]
        into = (pos(u[I, I, M]) * p[I, I, M] - neg(u[I, I, I]) * p[I, I, P]) * rn / self.dx + \
            (pos(v[I, M, I]) * p[I, M, I] - neg(v[I, I, I]) * p[I, P, I]) * rn / self.dy + \
            (pos(w[M, I, I]) * ra[M] * p[M, I, I] - neg(w[I, I, I]) * ra[I] * p[P, I, I]) / self.dz
        out = (pos(u[I, I, I]) - neg(u[I, I, M])) * pc * rn / self.dx + \
            (pos(v[I, I, I]) - neg(v[I, M, I])) * pc * rn / self.dy + \
            (pos(w[I, I, I]) * ra[I] - neg(w[M, I, I]) * ra[M]) * pc / self.dz
        up, dn = torch.zeros_like(p), torch.zeros_like(p)
        up[I, I, I] = rn * (hi - pc) / (dt * into + TINY)
        dn[I, I, I] = rn * (pc - lo) / (dt * (out + TINY))
        for a in (up, dn):
            _fill_full(a)
        r = []
        for vel, n in ((u, (I, I, P)), (v, (I, P, I)), (w, (P, I, I))):
            c = vel[I, I, I]
            r.append(torch.clamp(torch.minimum(dn[I, I, I], up[n]), max=1.0) * pos(c) +
                     torch.clamp(torch.minimum(up[I, I, I], dn[n]), max=1.0) * neg(c))
        return [self.filled(a) for a in r]

    def mpdata(self, dt, u, v, w, fields, kord, whole):
        """The fields of one category with zero boundary values, the first
        field's velocities for all; whole: the shift counts the halo cells."""
        low = [min(float((f if whole else f[I, I, I]).min()), 0.0) for f in fields]
        f = [a - m for a, m in zip(fields, low)]
        first, vel = f[0], (u, v, w)
        for it in range(kord):
            if it:
                vel = self.antidiffusive(dt, *vel, f[0])
                vel = self.limited(dt, *vel, first, f[0])
            f = [self.filled(self.donor(dt, *vel, a), -m, -m) for a, m in zip(f, low)]
        return [a + m for a, m in zip(f, low)]


def _subgrid(G, u, v, w, zu, zv, zw, th, lamsq, su, sv, sw, sth):
    """The Smagorinsky model's stress and diffusion terms on su, sv, sw, sth."""
    g, kp, jp, ip = G.g, G.kp, G.jp, G.ip
    dx, dy, dz = G.dx, G.dy, G.dz

    def at(a, k=0, j=0, i=0):
        return a[1 + k:kp + 1 + k, 1 + j:jp + 1 + j, 1 + i:ip + 1 + i]

    def sq(a):
        return a * a
    t = sq((at(u, 1) - at(u, 1, 0, -1)) / dx) + sq((at(u) - at(u, 0, 0, -1)) / dx)
    t = t + sq((at(v, 1) - at(v, 1, -1)) / dy) + sq((at(v) - at(v, 0, -1)) / dy)
    t = t + sq((at(w) - at(w, -1)) / dz) + sq((at(w, 1) - at(w)) / dz)
    t = t + 0.5 * (sq((at(u, 1) - at(u)) / dz + (at(w, 0, 0, 1) - at(w)) / dx) +
                   sq((at(u, 1, 0, -1) - at(u, 0, 0, -1)) / dz +
                      (at(w) - at(w, 0, 0, -1)) / dx))
    t = t + 0.5 * (sq((at(w) - at(w, 0, -1)) / dy + (at(v, 1, -1) - at(v, 0, -1)) / dz) +
                   sq((at(w, 0, 1) - at(w)) / dy + (at(v, 1) - at(v)) / dz))

    def s12(k, i, j):  # i: -1 (west face pair) or 0; j: the j pair's lower index
        return sq((at(u, k, j + 1, i) - at(u, k, j, i)) / dy +
                  (at(v, k, j, i + 1) - at(v, k, j, i)) / dx)
    t = t + 0.125 * (s12(0, -1, -1) + s12(0, -1, 0) + s12(0, 0, -1) + s12(0, 0, 0) +
                     s12(1, -1, -1) + s12(0, -1, 0) + s12(1, 0, -1) + s12(1, 0, 0))
    ri = GRAV * (at(th, 1) / G.thetan[P] - at(th) / G.thetan[I]) / dz / \
        (t + float(np.float32(1.0e-15)))
    a = torch.clamp(ri, max=0.0)
    b = 1.0 - torch.clamp(ri, min=0.0, max=0.25) / 0.25
    stable = ri >= 0.0
    fm = torch.where(stable, b ** 4, torch.sqrt(1.0 - 16.0 * a))
    fh = torch.where(stable, b ** 4 * (1.0 - 1.2 * torch.clamp(ri, min=0.0)),
                     torch.sqrt(1.0 - 40.0 * a)) / 0.95
    lam = _t(lamsq)[I, None, None]
    nu, kh = torch.zeros_like(th), torch.zeros_like(th)
    nu[I, I, I] = lam * torch.sqrt(t) * fm
    kh[I, I, I] = lam * torch.sqrt(t) * fh * G.rhoa[I]
    nu[kp - 1:kp + 1] = 0.0
    kh[kp - 1:kp + 1] = 0.0
    # the surface layer
    z1, th0 = float(g.z[1]), float(g.theta[0])
    speed = 0.5 * torch.sqrt(sq(u[1, I, I] + u[1, I, M]) + sq(v[1, I, I] + v[1, M, I])) + 1e-10
    dth = th[1, I, I] + float(g.thetan[1]) - th0
    rib = GRAV * dth * (z1 - Z0) ** 2 / (th0 * sq(speed) * (z1 - Z0))
    lg = math.log(z1 / Z0)
    root = 0.16 * torch.sqrt((rib * z1 / Z0).abs()) / lg ** 2
    calm = 1.0 / sq(1.0 + 4.7 * torch.clamp(rib, min=0.0))
    gm = torch.where(rib <= 0.0, 1.0 - 9.4 * rib / (1.0 + 70.0 * root), calm)
    gh = torch.where(rib <= 0.0, 1.0 - 9.4 * rib / (1.0 + 50.0 * root), calm)
    ustar = 0.4 * speed / lg * torch.sqrt(gm)
    thstar = 0.16 * speed * dth / (ustar * 0.95 * lg ** 2) * gh
    floor = (sq(ustar) * (z1 - Z0) / speed, ustar * thstar / (dth / (z1 - Z0) + 1e-10))
    for a, f in zip((nu, kh), floor):
        top = a[-1, I, I].clone()
        _fill_full(a)
        a[0, I, I], a[-1, I, I] = f, top
    rn, ra = G.rhoan[I], G.rhoa[I]
    two = at(nu) + at(nu, -1)
    t11 = G.stress(rn * two * (at(zu) - at(zu, 0, 0, -1)) / dx)
    t22 = G.stress(rn * two * (at(zv) - at(zv, 0, -1)) / dy)
    t33 = G.stress(rn * two * (at(zw) - at(zw, -1)) / dz)
    eight = sum(at(nu, k, j, i) for k in (0, -1) for j in (0, 1) for i in (0, 1))
    t12 = G.stress(rn * 0.125 * eight * ((at(zu, 0, 1) - at(zu)) / dy +
                                         (at(zv, 0, 0, 1) - at(zv)) / dx))
    t13 = G.stress(ra * 0.5 * (at(nu) + at(nu, 0, 0, 1)) *
                   ((at(zu, 1) - at(zu)) / dz + (at(zw, 0, 0, 1) - at(zw)) / dx))
    t23 = G.stress(ra * 0.5 * (at(nu) + at(nu, 0, 1)) *
                   ((at(zw, 0, 1) - at(zw)) / dy + (at(zv, 1) - at(zv)) / dz))
    au = (at(t11, 0, 0, 1) - at(t11)) / dx + (at(t12) - at(t12, 0, -1)) / dy + \
        (at(t13) - at(t13, -1)) / dz
    av = (at(t22, 0, 1) - at(t22)) / dy + (at(t12) - at(t12, 0, 0, -1)) / dx + \
        (at(t23) - at(t23, -1)) / dz
    aw = (at(t33, 1) - at(t33)) / dz + (at(t13) - at(t13, 0, 0, -1)) / dx + \
        (at(t23) - at(t23, 0, -1)) / dy
    sw[1:kp, I, I] += aw[:kp - 1]
    su[2:kp, I, I] += au[1:kp - 1]
    sv[2:kp, I, I] += av[1:kp - 1]
    for a in (su, sv, sw):
        _fill_full(a)

    def flux(j, i):  # the horizontal diffusive flux through the face towards (j, i)
        k4 = at(kh) + at(kh, 0, j, i) + at(kh, -1) + at(kh, -1, j, i)
        return 0.25 * k4 * (at(th, 0, j, i) - at(th))
    d = (flux(0, -1) + flux(0, 1)) / dx ** 2 + (flux(-1, 0) + flux(1, 0)) / dy ** 2 + \
        (at(kh, -1) * (at(th, -1) - at(th)) + at(kh) * (at(th, 1) - at(th))) / dz ** 2
    sth[I, I, I] += d / rn
    _fill_full(sth)


def _steps(g, dt, uu, zu0, th, q, kord, steps, viscous=False):
    """model_driver's time loop from a state with v = w = p = 0."""
    G = _Grid(g)
    kp = g.kp
    rn, ra = G.rhoan, G.rhoa
    u, v, w = uu, torch.zeros_like(uu), torch.zeros_like(uu)
    zu, zv, zw = zu0.clone(), torch.zeros_like(uu), torch.zeros_like(uu)
    zu[1], zu[kp] = 0.0, 0.0
    p = torch.zeros_like(uu)
    lamsq = _viscous(g)["lamsq"]
    for _ in range(steps):
        tb = th[:, I, I].mean(dim=(1, 2))[:, None, None]
        sth = torch.zeros_like(th)

        def inner(a, b, c):  # rho-weighted centred flux differences along x, y, z
            return G.filled(a / (4.0 * G.dx) + b / (4.0 * G.dy) + c / (4.0 * G.dz))
        C = (I, I, I)
        su = inner(u[I, I, M] * (u[C] + u[I, I, M]) - u[I, I, P] * (u[C] + u[I, I, P]),
                   u[I, M, I] * (v[I, M, I] + v[I, M, P]) - u[I, P, I] * (v[C] + v[I, I, P]),
                   u[M, I, I] * (w[M, I, I] + w[M, I, P]) - u[P, I, I] * (w[C] + w[I, I, P])) * rn
        sv = inner(v[I, I, M] * (u[I, I, M] + u[I, P, M]) - v[I, I, P] * (u[C] + u[I, P, I]),
                   v[I, M, I] * (v[C] + v[I, M, I]) - v[I, P, I] * (v[C] + v[I, P, I]),
                   v[M, I, I] * (w[M, I, I] + w[M, P, I]) - v[P, I, I] * (w[C] + w[I, P, I])) * rn
        sw = inner(w[I, I, M] * (u[I, I, M] + u[P, I, M]) - w[I, I, P] * (u[C] + u[P, I, I]),
                   w[I, M, I] * (v[I, M, I] + v[P, M, I]) - w[I, P, I] * (v[C] + v[P, I, I]),
                   w[M, I, I] * (w[C] + w[M, I, I]) - w[P, I, I] * (w[C] + w[P, I, I]))
        sw[I, I, I] += GRAV * (th[C] + th[P, I, I]) / (2.0 * G.theta[I] + tb[I] + tb[P])
        sw = sw * ra
        for a in (su, sv, sw):
            _fill_full(a)
        if viscous:
            _subgrid(G, u, v, w, zu, zv, zw, th, lamsq, su, sv, sw, sth)
        su[0], sv[0], sw[0] = -su[1], -sv[1], 0.0
        for a in (su, sv, sw):
            a[kp:] = 0.0
        b = (su[C] - su[I, I, M]) / G.dx + (sv[C] - sv[I, M, I]) / G.dy + \
            (sw[C] - sw[M, I, I]) / G.dz
        p = G.filled(G.poisson(b))
        p[0], p[-1] = p[1], p[-2]
        # scalars
        t2 = th.clone()
        pr = G.thetan
        t2[I] -= dt * 0.5 / G.dz * (w[M] * ra[M] * (pr[I] - pr[M]) +
                                    w[I] * ra[I] * (pr[P] - pr[I])) / rn[I]
        _fill_full(t2)
        th = G.mpdata(dt, u, v, w, [t2], kord, True)[0] + sth * dt
        q = [G.mpdata(dt, u, v, w, [a], kord, False)[0] for a in q]
        # momentum, the time filter and the new roles
        tu, tv, tw = (torch.zeros_like(u) for _ in range(3))
        L = slice(0, kp + 1)
        tu[L, I, I] = zu[L, I, I] + 2.0 * dt * (su[L, I, I] - (p[L, I, P] - p[L, I, I]) / G.dx) / rn[L]
        tv[L, I, I] = zv[L, I, I] + 2.0 * dt * (sv[L, I, I] - (p[L, P, I] - p[L, I, I]) / G.dy) / rn[L]
        tw[L, I, I] = zw[L, I, I] + 2.0 * dt * (sw[L, I, I] - (p[1:, I, I] - p[:-1, I, I]) / G.dz) / ra[L]
        zu, zv, zw = (0.99 * a + 0.01 * z for a, z in ((u, zu), (v, zv), (w, zw)))
        u, v, w = tu, tv, tw
        for a in (u, v, w):
            _fill_full(a)
        w[0], u[0], v[0] = 0.0, -u[1], -v[1]
        w[-1], u[-1], v[-1] = 0.0, u[kp], v[kp]
    r = dict(u=u, v=v, w=w, zu=zu, zv=zv, zw=zw, th=th, p=p)
    if q:
        r["q"] = torch.stack(q)
    return {n: _inner(a) for n, a in r.items()}


def _columns_exact(case, seed):
    met, w, psi, dt, ns = _column_input(case, seed)
    dz, dzn, ra, rn = (a[None, :] for a in met)
    dts, passes = (dt / ns)[:, None], int(ns.max())

    def rows(a):
        a[:, 0], a[:, -2], a[:, -1] = a[:, 1].clone(), a[:, -3].clone(), a[:, -3].clone()
        return a

    for it in range(passes):
        low = psi[..., I].amin(dim=2, keepdim=True)
        f = psi - low
        start, vel = f[:, 0].clone(), w
        for k in range(case["kord"]):
            if k:
                p0, n = f[:, 0], torch.zeros_like(w)
                g3 = 0.5 * (rn[:, I] + rn[:, P])
                c = vel[:, I]
                n[:, I] = (c.abs() * dz[:, I] - dts * (ra[:, I] / g3) * c * c) * \
                    (p0[:, P] - p0[:, I]) / (p0[:, P] + p0[:, I] + TINY) / dzn[:, I] - \
                    0.25 * dts * c * (ra[:, P] * vel[:, P] - ra[:, M] * vel[:, M]) / \
                    dz[:, M] / g3
                vel = rows(n)
                hi = torch.stack([a[:, s] for a in (start, p0) for s in (M, I, P)])
                hi, lo = hi.amax(dim=0), hi.amin(dim=0)
                a, b = vel[:, M] * ra[:, M], vel[:, I] * ra[:, I]
                into = dts * (a.clamp(min=0.0) * p0[:, M] - b.clamp(max=0.0) * p0[:, P]) / \
                    dzn[:, I] + TINY
                out = dts * (b.clamp(min=0.0) - a.clamp(max=0.0)) * p0[:, I] / dzn[:, I] + TINY
                up, dn = torch.zeros_like(w), torch.zeros_like(w)
                up[:, I] = rn[:, I] * (hi - p0[:, I]) / into
                dn[:, I] = rn[:, I] * (p0[:, I] - lo) / out
                n = torch.zeros_like(w)
                n[:, I] = torch.minimum(dn[:, I], up[:, P]).clamp(max=1.0) * \
                    vel[:, I].clamp(min=0.0) + \
                    torch.minimum(up[:, I], dn[:, P]).clamp(max=1.0) * vel[:, I].clamp(max=0.0)
                vel = rows(n)
            m = (vel * ra)[:, None, :]
            flux = (m.clamp(min=0.0)[..., :-1] * f[..., :-1] + m.clamp(max=0.0)[..., :-1] *
                    f[..., 1:]) * dts[:, None]
            f = torch.nn.functional.pad(
                f[..., I] - (flux[..., 1:] - flux[..., :-1]) / (dzn * rn)[:, None, I],
                (1, 1))
        psi = torch.where((it < ns)[:, None, None], f + low, psi)
    return psi


def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        g, dt, uu, zu, th, q = _case_flow(case, seed)
        return _steps(g, dt, uu, zu, th, q, case["kord"], case["steps"], case["viscous"])
    if kind == "ensemble":
        r = []
        for m, (ip, jp, kp, amp) in enumerate(_members(case)):
            f = _steps(*_flow("bubble", ip, jp, kp, _gen(1000 * seed + m), amp=amp), 3,
                       case["steps"])
            r.append({n: f[n] for n in MEMBER_FIELDS})
        return r
    if kind == "bicgstab":
        g, b = _solve_input(case, seed)
        return _Grid(g).poisson(b[I, I, I])
    if kind == "mpdata":
        g, dt, u, v, w, f = _advection_input(case, seed)
        G = _Grid(g)
        return torch.stack(G.mpdata(dt, u, v, w, f, case["kord"], case["nq"] == 1))
    return _columns_exact(case, seed)
