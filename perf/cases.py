"""Performance cases: what a user of the two-phase step has the library do.

Every case goes through the public entry points: the device-resident time step
(``fmf.capi.Stepper`` over ``fmf_ctx_*``) in its three precisions, the host-buffer
step (``fmf_ctx_step_host``), the adjoint of the rollout (``fmf.adjoint.Adjoint``),
the single stages on device arrays (``fmf_dev_weno5_fused``, ``fmf_dev_csf_fused``)
and the drop-in Fortran subroutines on host arrays.
"""
from __future__ import annotations

import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "fel-multi-phase-flow_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

from fmf import adjoint as fadj  # noqa: E402
from fmf import capi  # noqa: E402
from fmf import config as fcfg  # noqa: E402

PRECISION = {"fp64": capi.FMF_FP64, "mixed": capi.FMF_MIXED, "fp64e": capi.FMF_FP64E}


def listed():
    return [
        # The smallest workload (two-phase Couette, 32x32x16, its 100 steps in calls of 20
        # with the fields looked at after each): launches and their latency count.
        {"name": "step couette 32x32x16", "kind": "step", "flow": "couette32", "ni": 32, "nj": 32, "nk": 16,
         "precision": "fp64", "steps": 20},
        # The rollout workload's grid, per-wall-cell contact angles.
        {"name": "step couette 128x64x64", "kind": "step", "flow": "couette128", "ni": 128, "nj": 64, "nk": 64,
         "precision": "fp64", "steps": 8},
        # Density and viscosity ratio 10, perturbed stripe: the middle of the range.
        {"name": "step couette 256x128x128", "kind": "step", "flow": "couette256", "ni": 256, "nj": 128, "nk": 128,
         "precision": "fp64", "steps": 4},
        # The sessile drop (density ratio 1000, checkerboard wall), the largest workload.
        {"name": "step drop 512x256x256", "kind": "step", "flow": "droplet512", "ni": 512, "nj": 256, "nk": 256,
         "precision": "fp64", "steps": 4},
        # The same flow at half the size in the other two precisions a caller chooses.
        {"name": "step drop 256x128x128 fp64e", "kind": "step", "flow": "droplet256", "ni": 256, "nj": 128,
         "nk": 128, "precision": "fp64e", "steps": 4},
        {"name": "step drop 256x128x128 mixed", "kind": "step", "flow": "droplet256", "ni": 256, "nj": 128,
         "nk": 128, "precision": "mixed", "steps": 4},
        # A caller whose state lives on the host: every step up from and back to pinned memory.
        {"name": "host step couette 128x64x64", "kind": "step_host", "flow": "couette128", "ni": 128, "nj": 64,
         "nk": 64, "precision": "fp64"},
        # The gradient of the contact-line objective: a short rollout on a coarse grid, and one
        # on the rollout workload's grid.
        {"name": "adjoint couette 32x16x16", "kind": "adjoint", "flow": "couette128", "ni": 32, "nj": 16, "nk": 16,
         "precision": "fp64", "steps": 8, "every": 4},
        {"name": "adjoint couette 128x64x64", "kind": "adjoint", "flow": "couette128", "ni": 128, "nj": 64, "nk": 64,
         "precision": "fp64", "steps": 16, "every": 8},
        # Single stages on a caller's own device arrays, on grids of another shape than the
        # workloads' (every grid size is a power of two, as in the reference).
        {"name": "weno5 64x256x64", "kind": "weno5", "ni": 64, "nj": 256, "nk": 64, "precision": "fp64"},
        {"name": "csf 128x64x256", "kind": "csf", "ni": 128, "nj": 64, "nk": 256, "precision": "fp64"},
        # The drop-in subroutines a Fortran program calls for its transport, advection, explicit
        # viscous term and pressure solve, arrays resident on the device between the calls.
        {"name": "drop-in 64x32x32", "kind": "dropin", "ni": 64, "nj": 32, "nk": 32},
    ]


def draw(rng):
    def pow2(lo, hi):
        return 1 << rng.randint(lo, hi)

    kind = rng.choice(["step", "step", "step", "step", "step_host", "adjoint", "weno5", "csf", "dropin"])
    if kind == "step":
        # any direction may be the longest
        ni, nj, nk = pow2(4, 8), pow2(3, 8), pow2(3, 8)
        return {"kind": kind, "flow": rng.choice(["couette32", "couette128", "couette256", "droplet256"]),
                "ni": ni, "nj": nj, "nk": nk, "precision": rng.choice(["fp64", "fp64", "mixed", "fp64e"]),
                "steps": rng.randint(2, 8)}
    if kind == "step_host":
        return {"kind": kind, "flow": rng.choice(["couette32", "couette128"]), "ni": pow2(4, 7), "nj": pow2(3, 7),
                "nk": pow2(3, 6), "precision": rng.choice(["fp64", "mixed", "fp64e"])}
    if kind == "adjoint":
        return {"kind": kind, "flow": rng.choice(["couette32", "couette128"]), "ni": pow2(5, 7), "nj": pow2(4, 6),
                "nk": pow2(4, 6), "precision": rng.choice(["fp64", "fp64", "mixed"]), "steps": rng.randint(4, 12),
                "every": rng.randint(2, 6)}
    if kind == "weno5":
        return {"kind": kind, "ni": pow2(3, 8), "nj": pow2(3, 8), "nk": pow2(3, 8),
                "precision": rng.choice(["fp64", "fp64", "mixed", "fp64e"])}
    if kind == "csf":
        return {"kind": kind, "ni": pow2(5, 8), "nj": pow2(3, 8), "nk": pow2(2, 8),
                "precision": rng.choice(["fp64", "fp64", "fp64e"])}
    return {"kind": kind, "ni": pow2(4, 7), "nj": pow2(3, 6), "nk": pow2(3, 6)}


# ---- inputs -------------------------------------------------------------------
def _config(case, seed):
    cfg = fcfg.get(case["flow"], ni=case["ni"], nj=case["nj"], nk=case["nk"], seed=seed % 100003)
    if cfg.checker_cells:
        cfg.checker_cells = max(1, case["ni"] // 16)  # squares of 0.125
    return cfg


def _coords(n, d, shift, dev):
    return (torch.arange(-2, n + 4, dtype=torch.float64, device=dev) - 0.5 + shift) * d


def _mesh(size, spacing, shift, dev):
    """Broadcastable (x, y, z) of a (nk+6, nj+6, ni+6) field whose points are shifted by
    `shift` cells from the cell centres."""
    x = _coords(size[0], spacing[0], shift[0], dev)[None, None, :]
    y = _coords(size[1], spacing[1], shift[1], dev)[None, :, None]
    z = _coords(size[2], spacing[2], shift[2], dev)[:, None, None]
    return x, y, z


def _velocity(size, spacing, length, rng, dev, wall=0.0):
    """Staggered velocities: a shear profile between the walls and a few smooth modes,
    periodic in x and z, zero wall-normal velocity on the walls."""
    out = []
    for c, shift in enumerate(((0.5, 0, 0), (0, 0.5, 0), (0, 0, 0.5))):
        x, y, z = _mesh(size, spacing, shift, dev)
        f = 0.5 * wall * (2.0 * y / length[1] - 1.0) * (c == 0) + torch.zeros_like(x + y + z)
        for _ in range(4):
            a = rng.uniform(0.02, 0.08)
            m, n, l = rng.integers(1, 4), rng.integers(1, 4), rng.integers(1, 4)
            p, q = rng.uniform(0, 2 * math.pi, 2)
            f = f + a * (torch.sin(2 * math.pi * m / length[0] * x + p) * torch.sin(math.pi * n / length[1] * y)
                         * torch.cos(2 * math.pi * l / length[2] * z + q))
        out.append(f)
    return out


def _phi(size, spacing, length, rng, dev, drop):
    """Volume fraction with a tanh profile of width 1.5 cells: a sessile drop, or a stripe
    with a perturbed interface."""
    x, y, z = _mesh(size, spacing, (0, 0, 0), dev)
    width = 1.5 * spacing[0]
    if drop:
        r0, cx, cz = 0.3 + rng.uniform(-0.03, 0.03), rng.uniform(0.45, 0.55), rng.uniform(0.45, 0.55)
        r = torch.sqrt((x - cx * length[0]) ** 2 + (y - 0.15) ** 2 + (z - cz * length[2]) ** 2)
        return 0.5 * (1.0 - torch.tanh((r0 - r) / width))
    s = torch.zeros_like(y + z)
    for m in range(3):
        a, n, p = rng.normal(0.0, 0.015), rng.integers(0, 3), rng.uniform(0, 2 * math.pi)
        s = s + a * torch.cos(2 * math.pi * (m * z / length[2] + n * y / length[1]) + p)
    d = 0.25 * length[0] - (x - 0.5 * length[0] - s).abs()
    return 0.5 * (1.0 + torch.tanh(d / width))


class _Device:
    """A (nk+6, nj+6, ni+6) double array at a device pointer; the tensor made from it keeps
    the owner of that memory alive."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False), "version": 2}


class _StepState:
    def __init__(self, cfg, precision):
        self.cfg = cfg
        self.step = capi.Stepper(cfg, precision)
        self.seen = {}

    def fields(self):
        """The 12 state fields as zero-copy tensors."""
        out = []
        p = ctypes.c_void_p()
        for f in range(12):
            capi.check(capi.lib().fmf_ctx_state_device_ptr(self.step.h, f, ctypes.byref(p)), "state pointer")
            if p.value not in self.seen:
                self.seen[p.value] = torch.as_tensor(_Device(p.value, self.cfg.shape, self.step), device="cuda")
            out.append(self.seen[p.value])
        return out


def _start(case, seed):
    """A context with a state a run has reached: both velocity levels, the interface of both
    volume-fraction slices, zero pressure, boundary values by the start-up pass."""
    cfg = _config(case, seed)
    rng = np.random.default_rng(seed)
    s = _StepState(cfg, PRECISION[case["precision"]])
    size, spacing = (cfg.ni, cfg.nj, cfg.nk), (cfg.dx, cfg.dy, cfg.dz)
    length = (cfg.xl, cfg.yl, cfg.zl)
    vel = _velocity(size, spacing, length, rng, "cuda", cfg.uwall)
    phi = _phi(size, spacing, length, rng, "cuda", cfg.init == "droplet")
    fields = s.fields()
    for f, q in zip(fields, vel + vel + [None, None] + [phi] * 4):
        f.zero_() if q is None else f.copy_(q)
    torch.cuda.synchronize()
    s.step.init_bc()
    s.step.sync()
    return s


class _HostState:
    pass


class _DropinState:
    """Host arrays of a Fortran caller and the argument lists of its calls."""

    def __init__(self):
        self.arrays, self.calls, self.results = [], [], []

    def __del__(self):
        try:
            for a in self.arrays:
                capi.lib().fmf_forget(capi.P(a))
        except Exception:
            pass


def _dropin(case, seed):
    ni, nj, nk = size = (case["ni"], case["nj"], case["nk"])
    length = (2.0, 1.0, 1.0)
    dx, dy, dz = spacing = tuple(l / n for l, n in zip(length, size))
    rng = np.random.default_rng(seed)
    s = _DropinState()
    shape = (nk + 6, nj + 6, ni + 6)

    def arr(t=None, shp=shape):
        a = np.zeros(shp) if t is None else np.ascontiguousarray(t.expand(shp).numpy())
        s.arrays.append(a)
        return a

    I, D, P = capi.I, capi.D, capi.P
    n3 = (I(ni), I(nj), I(nk))
    inv = (D(1 / dx), D(1 / dy), D(1 / dz))
    u, v, w = (arr(t) for t in _velocity(size, spacing, length, rng, "cpu", -1.0))
    phi = arr(_phi(size, spacing, length, rng, "cpu", False))
    mu = arr(torch.from_numpy(0.5 - 0.45 * phi))
    dyinv = arr(torch.full((nj + 6,), 1 / dy, dtype=torch.float64), (nj + 6,))
    gx, gy, gz, fx, fy, fz, phin, au, av, aw, vu, vv, vw, div, dp = (arr() for _ in range(15))
    sij, tau = arr(shp=(6,) + shape), arr(shp=(6,) + shape)
    pr, pi = arr(shp=(nk, nj, ni)), arr(shp=(nk, nj, ni))
    south, north, diag = (np.zeros(nj + 6) for _ in range(3))
    south[3:nj + 3] = north[3:nj + 3] = 1 / dy ** 2
    south[3] = north[nj + 2] = 0.0
    diag[:] = south + north
    south, north, diag = (arr(torch.from_numpy(a), (nj + 6,)) for a in (south, north, diag))
    dt, err, none = 1e-4, ctypes.c_double(), None
    sv = capi.IA([ni, nj, nk])
    s.keep = err
    s.calls = [
        ("bnd_periodic_", n3 + (P(phi),)),
        ("cal_grad_p2a_", (I(0), I(nj)) + n3 + (D(1 / dx), P(dyinv), D(1 / dz), P(phi), P(gx), P(gy), P(gz))),
        ("solphi_mthinc1_", n3 + inv + (D(dt), D(2.0), P(phi), P(gx), P(gy), P(gz), P(u), P(v), P(w), P(fx), P(fy),
                                        P(fz))),
        ("solphi_mthinc2_", n3 + inv + (D(dt), P(u), P(v), P(w), P(fx), P(fy), P(fz), P(phi), P(phin))),
        ("cal_advu_weno5_", n3 + inv + (P(u), P(v), P(w), P(au), P(av), P(aw))),
        ("calsij_", n3 + inv + (P(u), P(v), P(w), P(sij))),
        ("cal_arith_tau_", n3 + (P(sij), P(mu), P(tau))),
        ("cal_div_tensor_", n3 + inv + (P(tau), P(vu), P(vv), P(vw))),
        ("caldiv_", (I(0), I(1)) + n3 + inv + (D(dt), P(u), P(v), P(w), P(div), ctypes.byref(err))),
        ("solp_fft_tdma1_", n3 + (none, P(div), P(pr), P(pi))),
        ("solp_fft_tdma2_", (I(0), I(1), sv, D(1.0), D(1 / dx), D(1 / dz), P(south), P(north), P(diag), none, none,
                             none, P(pr), P(pi))),
        ("solp_fft_tdma3_", n3 + (none, P(pr), P(pi), P(dp))),
        ("bnd_avzero_", (I(0), I(1)) + n3 + (P(dp),)),
    ]
    s.results = [phin, au, av, aw, vu, vv, vw, dp]
    L = capi.lib()
    for a in s.arrays:
        L.fmf_forget(P(a))  # an earlier array at this address, if any
    return s


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        return kind, case["steps"], _start(case, seed)
    if kind == "step_host":
        s = _start(case, seed)
        h = _HostState()
        h.step = s.step
        h.pinned = [torch.empty((12,) + s.cfg.shape, dtype=torch.float64, pin_memory=True) for _ in range(2)]
        h.a, h.b = (p.numpy() for p in h.pinned)
        h.step.download(h.a)
        h.step.sync()
        return kind, 1, h
    if kind == "adjoint":
        cfg = _config(case, seed)
        rng = np.random.default_rng(seed)
        st = fcfg.raw_state(cfg)
        p = fcfg.STATE_FIELDS.index("phi1")
        st[p] = _phi((cfg.ni, cfg.nj, cfg.nk), (cfg.dx, cfg.dy, cfg.dz), (cfg.xl, cfg.yl, cfg.zl), rng, "cpu",
                     False).numpy()
        fcfg.periodic(st[p], cfg)
        a = fadj.Adjoint(cfg, sor_tol=1e-3, sor_max=21, adj_tol=1e-6, adj_max=200,
                         precision=PRECISION[case["precision"]])
        return kind, case["steps"], (a, st, fcfg.wall_arrays(cfg), case["every"])
    if kind == "dropin":
        return kind, 1, _dropin(case, seed)
    rng = np.random.default_rng(seed)
    size, length = (case["ni"], case["nj"], case["nk"]), (2.0, 1.0, 1.0)
    spacing = tuple(l / n for l, n in zip(length, size))
    if kind == "weno5":
        ins = _velocity(size, spacing, length, rng, "cuda", -1.0)
    else:
        ins = [_phi(size, spacing, length, rng, "cuda", bool(seed % 2))]
    return kind, 1, (dict(case), spacing, ins, [torch.zeros_like(ins[0]) for _ in range(3)])


def run(state):
    kind, n, s = state
    if kind == "step":
        s.step.step(n)
        return s.fields()
    if kind == "step_host":
        s.step.step_host(s.a, s.b)
        s.a, s.b = s.b, s.a
        return s.a
    if kind == "adjoint":
        a, st, walls, every = s
        J, grads = a.rollout(n, st, walls, every)
        return {"J": J, "theta0": grads[0], "zeta": grads[1], "l1": grads[2], "l2": grads[3], "phi": grads[4]}
    L = capi.lib()
    if kind == "dropin":
        for name, args in s.calls:
            getattr(L, name)(*args)
        for a in s.results:
            L.fmf_sync_to_host(capi.P(a))
        capi.check(L.fmf_last_error(), "drop-in")
        return list(s.results)
    case, (dx, dy, dz), ins, outs = s
    ptr = [ctypes.c_void_p(t.data_ptr()) for t in ins + outs]
    size = (case["ni"], case["nj"], case["nk"])
    if kind == "weno5":
        capi.check(L.fmf_dev_weno5_fused(PRECISION[case["precision"]], *size, 1 / dx, 1 / dy, 1 / dz, *ptr), "weno5")
    else:
        capi.check(L.fmf_dev_csf_fused(PRECISION[case["precision"]], *size, dx, dy, dz, 10.0, 1.0, 1.0, *ptr), "csf")
    return outs


# ---- what a pass cannot do without ----------------------------------------------
def work(case):
    cells = case["ni"] * case["nj"] * case["nk"]
    kind = case["kind"]
    if kind in ("step", "step_host"):
        n = case.get("steps", 1)
        return {"bytes": 8.0 * 24 * cells * n, "flops": 2000.0 * cells * n}
    if kind == "adjoint":
        # the forward step, its recomputation and the reverse of each
        return {"bytes": 8.0 * 24 * 3 * cells * case["steps"], "flops": 4 * 2000.0 * cells * case["steps"]}
    if kind == "weno5":
        return {"bytes": 8.0 * 6 * cells, "flops": 9 * 70.0 * cells}
    if kind == "csf":
        return {"bytes": 8.0 * 4 * cells, "flops": 250.0 * cells}
    return {"bytes": 8.0 * (5 + 8) * cells, "flops": 1500.0 * cells}


# ---- the same values in plain 64-bit arithmetic ----------------------------------
def _weno5_exact(case, seed):
    _, _, (_, spacing, q, out) = prepare(case, seed)
    ni, nj, nk = case["ni"], case["nj"], case["nk"]

    def at(a, o):  # a at (i, j, k) + o over the interior
        return a[3 + o[2]:3 + o[2] + nk, 3 + o[1]:3 + o[1] + nj, 3 + o[0]:3 + o[0] + ni]

    def side(a, b, c, d, e):
        # one-sided reconstruction from five differences, upwind end first
        s1 = 13 * (a - 2 * b + c) ** 2 + 3 * (a - 4 * b + 3 * c) ** 2
        s2 = 13 * (b - 2 * c + d) ** 2 + 3 * (b - d) ** 2
        s3 = 13 * (c - 2 * d + e) ** 2 + 3 * (3 * c - 4 * d + e) ** 2
        m1, m2, m3 = (s2 * s3) ** 2, 6 * (s1 * s3) ** 2, 3 * (s1 * s2) ** 2
        t = m1 + m2 + m3 + 1e-80
        w1, w3 = m1 / t, m3 / t
        return w1 * (2 * a - 7 * b + 11 * c) + (1 - w1 - w3) * (-b + 5 * c + 2 * d) + w3 * (2 * c + 5 * d - e)

    unit = ((1, 0, 0), (0, 1, 0), (0, 0, 1))
    res = []
    for c in range(3):
        tot = 0.0
        for d in range(3):
            e, s = unit[d], unit[c]
            lo = tuple(-x for x in e)
            z = (0, 0, 0)
            los = tuple(x + y for x, y in zip(lo, s))
            vel = 0.25 * ((at(q[d], lo) + at(q[d], los)) + (at(q[d], z) + at(q[d], s)))
            df = [at(q[c], tuple(m * x for x in e)) - at(q[c], tuple((m - 1) * x for x in e)) for m in range(-2, 4)]
            up = (vel + vel.abs()) * side(*df[:5]) + (vel - vel.abs()) * side(*df[:0:-1])
            tot = tot + up / 12.0 / spacing[d]
        full = torch.zeros_like(out[0])
        at(full, (0, 0, 0)).copy_(tot)
        res.append(full)
    return res


def _csf_exact(case, seed):
    _, _, (_, (dx, dy, dz), (phi,), out) = prepare(case, seed)
    ni, nj, nk = case["ni"], case["nj"], case["nk"]

    def sh(a, x=0, y=0, z=0):  # a(i + x, j + y, k + z); rolled values do not reach the interior
        return torch.roll(a, (-z, -y, -x), (0, 1, 2))

    def pairsum(a, **o):
        return a + sh(a, **o)

    gx = pairsum(pairsum(sh(phi, x=1) - phi, y=1), z=1) * (0.25 / dx)
    gy = pairsum(pairsum(sh(phi, y=1) - phi, x=1), z=1) * (0.25 / dy)
    gz = pairsum(pairsum(sh(phi, z=1) - phi, x=1), y=1) * (0.25 / dz)
    tiny = 1e-30 * math.sqrt(dx ** -2 + dy ** -2 + dz ** -2)

    def normal(*dirs):
        v = []
        for g in (gx, gy, gz):
            for d in dirs:
                g = 0.5 * pairsum(g, **{d: -1})
            v.append(g)
        m = 1.0 / (torch.sqrt(v[0] ** 2 + v[1] ** 2 + v[2] ** 2) + tiny)
        return [a * m for a in v]

    pp, n12, n13, n23 = normal("x", "y", "z"), normal("z"), normal("y"), normal("x")
    ku = (sh(pp[0], x=1) - pp[0]) / dx + (n12[1] - sh(n12[1], y=-1)) / dy + (n13[2] - sh(n13[2], z=-1)) / dz
    kv = (n12[0] - sh(n12[0], x=-1)) / dx + (sh(pp[1], y=1) - pp[1]) / dy + (n23[2] - sh(n23[2], z=-1)) / dz
    kw = (n13[0] - sh(n13[0], x=-1)) / dx + (n23[1] - sh(n23[1], y=-1)) / dy + (sh(pp[2], z=1) - pp[2]) / dz
    st = 2.0 / (10.0 + 1.0)
    res = []
    for k, g in ((ku, (sh(phi, x=1) - phi) / dx), (kv, (sh(phi, y=1) - phi) / dy), (kw, (sh(phi, z=1) - phi) / dz)):
        full = torch.zeros_like(out[0])
        full[3:3 + nk, 3:3 + nj, 3:3 + ni] = (-st * k * g)[3:3 + nk, 3:3 + nj, 3:3 + ni]
        res.append(full)
    return res


def exact(case, seed):
    """The single stages in plain 64-bit torch; a whole step or rollout has no short form."""
    if case["kind"] == "weno5":
        return _weno5_exact(case, seed)
    if case["kind"] == "csf":
        return _csf_exact(case, seed)
    return None
