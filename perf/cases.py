"""Timed workloads of the CUMC3D hot path, through its public entry points.

Each case is a stretch of a simulation as a program that uses the library runs
it: a time loop of a few RK3 steps on a context that is already set up, then
the output of the state into the program's own (pinned) host arrays, as
main.f90 does between two snapshots; or one gradient evaluation of an
optimisation loop over the initial state. The flows are the library's own
models: the Brio-Wu tube, the Orszag-Tang vortex, the spherical and
cylindrical tori, the curvilinear shells and the Fourier velocity box.

`listed` names the cases, `draw` gives further ones of the same ranges,
`prepare` builds the state of one, `run` is one pass, `work` the bytes and
operations a pass cannot do without, and `exact` the outputs of the first pass
in plain 64-bit torch.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from cumpic_b200 import _native as N
from cumpic_b200 import problems
from cumpic_b200.halo import LocalSlabs, ZSlabs

PRECISIONS = {"fp64": N.FP64, "fp64_fast": N.FP64_FAST, "mixed": N.MIXED}
RECONS = {"ppm": N.PPMC, "tvd": N.TVDMM}
OBJECTIVES = {"magnetic": N.OBJ_MAGNETIC, "kinetic": N.OBJ_KINETIC}
NO_END = 1.0e300  # total time of a loop bounded by its step count


def _case(name, flow, nx, ny, nz, steps, precision="fp64", recon="ppm", drive="device", **more):
    return {"name": name, "flow": flow, "nx": nx, "ny": ny, "nz": nz, "steps": steps, "precision": precision,
            "recon": recon, "drive": drive, **more}


def listed():
    return [
        # the 1-D shock-tube check a user runs first: tiny grid, main.f90's own
        # host loop (finddt, then RUNGEKUTTA, every step): launches and latency
        _case("brio_wu_512x4x4_host_loop", "brio_wu", 512, 4, 4, 20, drive="host"),
        # a development-size box in the device-side loop
        _case("orszag_tang_64", "orszag_tang", 64, 64, 64, 20),
        # the production size: the configuration the throughput is quoted on
        _case("orszag_tang_256", "orszag_tang", 256, 256, 256, 20),
        # the same box in the mixed-precision form
        _case("orszag_tang_256_mixed", "orszag_tang", 256, 256, 256, 20, precision="mixed"),
        # a survey-size box with the reciprocal form of the HLL solve
        _case("orszag_tang_128_fast", "orszag_tang", 128, 128, 128, 20, precision="fp64_fast"),
        # odd, unequal sides and the TVD reconstruction
        _case("orszag_tang_149x131x97_tvd", "orszag_tang", 149, 131, 97, 20, recon="tvd"),
        # the accretion torus at its configured grid: spherical-polar geometry,
        # gravity, floors, axis boundaries
        _case("torus_192x128x64", "torus", 192, 128, 64, 20),
        _case("torus_192x128x64_mixed", "torus", 192, 128, 64, 20, precision="mixed"),
        # a cylindrical torus of ragged size
        _case("torus_cyl_90x26x75", "torus_cyl", 90, 26, 75, 20),
        # one gradient of the final magnetic energy on the adjoint's check box
        _case("adjoint_fourier_128", "fourier_box", 128, 128, 128, 20, drive="adjoint", checkpoint=10,
              objective="magnetic"),
        # one gradient on a small curvilinear shell
        _case("adjoint_shell_48x40x33", "shell_sph", 48, 40, 33, 12, drive="adjoint", checkpoint=5,
              objective="kinetic"),
        # a box cut into z-slabs with the halo exchange between the stages
        _case("slabs_2_orszag_tang_128", "orszag_tang", 128, 128, 128, 20, drive="slabs", slabs=2),
    ]


def draw(rng):
    def size(lo, hi):  # spread over the logarithm of the range; odd and even alike
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["tube", "box", "box", "box", "mixed", "fast", "torus", "torus_cyl", "adjoint", "slabs"])
    steps = rng.randint(8, 20)
    recon = rng.choice(["ppm", "ppm", "ppm", "tvd"])
    if kind == "tube":
        c = _case("", "brio_wu", size(96, 2048), rng.randint(4, 8), rng.randint(4, 8), steps, recon=recon,
                  drive=rng.choice(["host", "device"]))
    elif kind in ("box", "mixed", "fast"):
        c = _case("", "orszag_tang", size(24, 250), size(24, 250), size(24, 250), steps, recon=recon,
                  precision={"box": "fp64", "mixed": "mixed", "fast": "fp64_fast"}[kind],
                  drive=rng.choice(["device", "device", "host"]))
    elif kind == "torus":
        c = _case("", "torus", size(48, 224), size(32, 144), size(16, 96), steps,
                  precision=rng.choice(["fp64", "mixed"]))
    elif kind == "torus_cyl":
        c = _case("", "torus_cyl", size(40, 160), size(6, 64), size(40, 160), steps)
    elif kind == "adjoint":
        flow = rng.choice(["fourier_box", "shell_sph", "shell_cyl"])
        n = size(24, 112)
        ny, nz = (n, n) if flow == "fourier_box" else (size(20, 64), size(20, 64))
        c = _case("", flow, n, ny, nz, rng.randint(4, 12), drive="adjoint", checkpoint=rng.randint(2, 8),
                  objective=rng.choice(["magnetic", "kinetic"]))
    else:
        c = _case("", "orszag_tang", size(32, 160), size(32, 160), size(32, 160), steps, drive="slabs",
                  slabs=rng.randint(2, 4))
    del c["name"]
    return c


def _problem(case, seed):
    """the flow's initial model; the seed moves its noise, phases or states"""
    nx, ny, nz, flow = case["nx"], case["ny"], case["nz"], case["flow"]
    recon, seed = RECONS[case["recon"]], int(seed) + 1
    if flow == "brio_wu":
        p = problems.brio_wu(nx, ny, nz, recon=recon)
        r = np.random.default_rng(seed)
        f = 1.0 + 0.05 * (2.0 * r.random(3) - 1.0)  # density, pressure and tangential field of both states
        p.prim[..., problems.IRHO] *= f[0]
        p.prim[..., problems.ITAU] *= f[1]
        p.prim[..., problems.IBY] *= f[2]
        p.eps *= f[1] / f[0]
    elif flow == "orszag_tang":
        p = problems.orszag_tang(nx, ny=ny, nz=nz, recon=recon, seed=seed)
    elif flow == "torus":
        p = problems.torus(nx, ny, nz, seed=seed)
    elif flow == "torus_cyl":
        p = problems.torus_cyl(nx, ny, nz, seed=seed)
    elif flow == "fourier_box":
        p = problems.fourier_box(nx, seed=seed)
    else:
        p = problems.shell(N.SPHERICAL if flow == "shell_sph" else N.CYLINDRICAL, nx, ny, nz, seed=seed, recon=recon)
    p.precision = PRECISIONS[case["precision"]]
    return p


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True)


def _ptr(t):
    return ctypes.cast(t.data_ptr(), N.POINTER(ctypes.c_double))


class _Context:
    """one library context and the program's host arrays"""

    def __init__(self, case, seed):
        self.case = case
        self.lib = N.lib()
        self.handle = None
        p = _problem(case, seed)
        full = (p.nz + 6, p.ny + 6, p.nx + 6)
        if case["drive"] == "slabs":
            self.slabs = LocalSlabs(p, case["slabs"])
            self.slabs.start()
            self.out = [_pinned((N.STATE_ARRAYS,) + s.shape) for s in self.slabs.sims]
            return
        h = ctypes.c_void_p()
        if self.lib.cumc_init(ctypes.byref(p.config()), ctypes.byref(h)) != N.CUMC_OK:
            raise RuntimeError(self.lib.cumc_last_error(None).decode())
        self.handle = h
        self.prim, self.eps = _pinned(full + (8,)), _pinned(full)
        if case["drive"] == "adjoint":  # every pass uploads its initial state
            self.prim0, self.eps0 = _pinned(full + (8,)), _pinned(full)
            self.prim0.copy_(torch.from_numpy(p.prim))
            self.eps0.copy_(torch.from_numpy(p.eps))
            return
        self.ok(self.lib.cumc_upload_state(h, p.prim.ctypes.data_as(N.POINTER(ctypes.c_double)),
                                           p.eps.ctypes.data_as(N.POINTER(ctypes.c_double))))
        self.ok(self.lib.cumc_initial_update(h))
        self.time = ctypes.c_double(0.0)

    def ok(self, status):
        if status != N.CUMC_OK:
            raise RuntimeError(self.lib.cumc_last_error(self.handle).decode())

    def __del__(self):
        if self.handle:
            self.lib.cumc_free(self.handle)
            self.handle = None


def prepare(case, seed):
    return _Context(case, seed)


def run(state):
    c, lib, h = state.case, state.lib, state.handle
    if c["drive"] == "slabs":
        for _ in range(c["steps"]):
            state.slabs.step()
        state.slabs.finish_exchange()
        for sim, buf in zip(state.slabs.sims, state.out):
            sim.snapshot_async(buf.numpy())
        for sim in state.slabs.sims:
            sim.snapshot_wait()
        return {"cons": [b[:8] for b in state.out], "prims": [b[8:] for b in state.out]}
    if c["drive"] == "adjoint":
        J = ctypes.c_double()
        dts = np.zeros(c["steps"])
        state.ok(lib.cumc_upload_state(h, _ptr(state.prim0), _ptr(state.eps0)))
        state.ok(lib.cumc_adjoint_run(h, c["steps"], c["checkpoint"], OBJECTIVES[c["objective"]], None, None,
                                      dts.ctypes.data_as(N.POINTER(ctypes.c_double)), ctypes.byref(J),
                                      _ptr(state.prim), _ptr(state.eps)))
        return {"J": J.value, "dts": dts, "grad_prim": state.prim, "grad_eps": state.eps}
    if c["drive"] == "host":
        dt = ctypes.c_double()
        for _ in range(c["steps"]):
            state.ok(lib.cumc_finddt(h, ctypes.byref(dt)))
            state.ok(lib.cumc_rungekutta(h, dt.value))
    else:
        state.ok(lib.cumc_advance(h, c["steps"], NO_END, ctypes.byref(state.time), None))
    state.ok(lib.cumc_download_state(h, _ptr(state.prim), None, _ptr(state.eps), None))
    return {"prim": state.prim, "eps": state.eps}


def work(case):
    """One RK3 step reads and writes the 8 conserved values of a cell once a
    stage and reads the step's old ones again at stages 2 and 3: 512 bytes in
    FP64; in the mixed form the old state is 64 bytes and the stage increments
    48. A gradient also runs every step in reverse, reading the step's state
    and reading and writing its adjoint. A stage reconstructs 7 fields (about
    35 operations each) and solves one Riemann problem (about 280) a face."""
    cells = case["nx"] * case["ny"] * case["nz"]
    full = (case["nx"] + 6) * (case["ny"] + 6) * (case["nz"] + 6)
    step_bytes = 448 if case["precision"] == "mixed" else 512
    step_flops = 3 * (3 * (7 * 35 + 280) + 150)
    updates = cells * case["steps"]
    if case["drive"] == "adjoint":
        return {"bytes": 3 * step_bytes * updates + 2 * 72 * full, "flops": 3 * step_flops * updates}
    out = 136 if case["drive"] == "slabs" else 72
    return {"bytes": step_bytes * updates + out * full, "flops": step_flops * updates}


# ---------------------------------------------------------------------------
# the first pass in plain 64-bit torch: the scheme of solver/*.f90 on whole
# arrays, index i of an axis at array position i + 2, axis d (x, y, z) = dim 2 - d
# ---------------------------------------------------------------------------
RHO, VX, VY, VZ, TAU, BX, BY, BZ = range(8)


def _shift(a, d, k):
    """value at index + k along axis d (the wrapped ends are never used)"""
    return torch.roll(a, -k, 2 - d)


class _Exact:
    def __init__(self, p):
        self.p, self.dev = p, "cuda" if torch.cuda.is_available() else "cpu"
        self.n = (p.nx, p.ny, p.nz)
        faces = [np.asarray(f, dtype=np.float64) for f in (p.xf, p.yf, p.zf)]
        self.tab = []
        for d, f in enumerate(faces):
            w = np.diff(f)  # width of cells -2..n+3
            wm, wp, wpp = (np.roll(w, 1), np.roll(w, -1), np.roll(w, -2))
            wm[0], wp[-1], wpp[-2:] = w[0], w[-1], w[-1]
            cc1, total = w / (wm + w + wp), wm + w + wp + wpp
            t = {"w": w, "f": f[1:], "fm": f[:-1], "c": 0.5 * (f[1:] + f[:-1]),
                 "b0": cc1 * (2 * wm + w) / (wp + w), "b1": cc1 * (w + 2 * wp) / (wm + w),
                 "a1": w / (w + wp) + 2 * wp * w / (wp + w) * ((wm + w) / (2 * w + wp) - (wpp + wp) / (2 * wp + w)) / total,
                 "a2": -w * (wm + w) / (2 * w + wp) / total, "a3": wp * (wpp + wp) / (2 * wp + w) / total,
                 "cf": (w + wp) / w, "cb": (w + wm) / w}
            self.tab.append({k: self.along(v, d) for k, v in t.items()})
        x, y = self.tab[0], self.tab[1]
        self.r3, self.r2, self.r2m = (x["f"] ** 3 - x["fm"] ** 3) / 3, x["f"] ** 2, x["fm"] ** 2
        self.rfac = 2 * self.r3 / (self.r2 - self.r2m)
        self.sin, self.sinm, self.sinc, self.tanc = (torch.sin(y["f"]), torch.sin(y["fm"]), torch.sin(y["c"]),
                                                     torch.tan(y["c"]))
        self.dcos = torch.cos(y["fm"]) - torch.cos(y["f"])
        self.inner = tuple(slice(3, 3 + m) for m in reversed(self.n))  # cells 1..n
        self.maps = [self.ghost_map(d) for d in range(3)]

    def along(self, v, d):
        shape = [1, 1, 1]
        shape[2 - d] = len(v)
        return torch.as_tensor(v, dtype=torch.float64, device=self.dev).reshape(shape)

    def ghost_map(self, d):
        """source position and the 8 parity signs of every position along axis d (solver/boundary.f90)"""
        n, src, sign = self.n[d], np.arange(self.n[d] + 6), np.ones((8, self.n[d] + 6))
        odd = {2: (VX + d, BX + d), 3: (VX + d, BX + d, VZ, BZ), 4: {1: (VY, BX, BZ), 2: (VZ, BX, BY)}.get(d, ())}
        for i in [-2, -1, 0, n + 1, n + 2, n + 3]:
            fl = self.p.boundary_flag[2 * d + (i > n)]
            src[i + 2] = 2 + ((i + n if i < 1 else i - n) if fl == 0 else (1 if i < 1 else n) if fl == 1 else
                              1 - i if i < 1 else 2 * n + 1 - i)
            for q in odd.get(fl, ()):
                sign[q, i + 2] = -1.0
        return torch.as_tensor(src, device=self.dev), [self.along(s, d) for s in sign]

    def fill(self, a, q, d):
        src, sign = self.maps[d]
        return a.index_select(2 - d, src) * (sign[q] if q is not None else 1.0)

    def boundary(self, s):
        p, n = self.p, self.n
        w = list(s["w"])
        for d in range(3):
            w = [self.fill(a, q, d) for q, a in enumerate(w)]
        bc = [self.fill(self.fill(self.fill(a, BX + q, 0), BX + q, 1), BX + q, 2) for q, a in enumerate(s["bc"])]
        eps = s["eps"]
        for d in range(3):
            eps = self.fill(eps, None, d)
        if p.model in (N.MODEL_TORUS_SPH, N.MODEL_TORUS_CYN):
            w[1] = torch.cat([w[1][..., :3].clamp(max=0.0), w[1][..., 3:n[0] + 3], w[1][..., n[0] + 3:].clamp(min=0.0)], 2)
        if p.model == N.MODEL_TORUS_CYN:
            w[3] = torch.cat([w[3][:3].clamp(max=0.0), w[3][3:n[2] + 3], w[3][n[2] + 3:].clamp(min=0.0)], 0)
        bf = []
        for c, a in enumerate(s["bf"]):  # only the components tangential to a ghost direction, on faces 0..n
            live = a.narrow(2 - c, 2, n[c] + 1)
            for d in range(3):
                if d != c:
                    live = self.fill(live, BX + c, d)
            bf.append(torch.cat([a.narrow(2 - c, 0, 2), live, a.narrow(2 - c, n[c] + 3, 3)], 2 - c))
        w = w[:4] + [w[0] * eps * (p.ggas - 1.0)]
        return {"w": w, "bc": bc, "eps": eps, "bf": bf}

    def put(self, full, part):
        """`part` on the cells 1..n, `full` around it"""
        pads = [(3, 3)] * 3
        mask = torch.zeros_like(full, dtype=torch.bool)
        mask[self.inner] = True
        return torch.where(mask, torch.nn.functional.pad(part, [q for pr in pads for q in pr]), full)

    def cons(self, s):
        w, bc = s["w"], s["bc"]
        v2, b2 = w[1] ** 2 + w[2] ** 2 + w[3] ** 2, bc[0] ** 2 + bc[1] ** 2 + bc[2] ** 2
        return [w[0], w[1] * w[0], w[2] * w[0], w[3] * w[0], w[0] * (s["eps"] + 0.5 * v2) + 0.5 * b2]

    def cell_field(self, bf):
        return [0.5 * (a + _shift(a, d, -1)) for d, a in enumerate(bf)]

    def floors(self, rho, e):
        p = self.p
        if p.model == N.MODEL_RIEMANN:
            return rho, e.clamp(min=0.0)
        if p.model in (N.MODEL_TORUS_SPH, N.MODEL_TORUS_CYN):
            return rho.clamp(min=p.rho_floor), e.clamp(min=p.eps_floor)
        return rho, e

    def initial(self, prim, eps):
        w = [prim[..., q] for q in range(5)]
        bf = [prim[..., BX + q] for q in range(3)]
        bc = [self.put(torch.zeros_like(b), b[self.inner]) for b in self.cell_field(bf)]
        rho, e = self.floors(w[0][self.inner], eps[self.inner])
        return self.boundary({"w": [self.put(w[0], rho)] + w[1:], "bc": bc, "eps": self.put(eps, e), "bf": bf})

    def primitives(self, u, bf, s):
        """from the hydro cons on cells 1..n and the face fields; s gives the arrays' other entries"""
        bcn = [b[self.inner] for b in self.cell_field(bf)]
        b2 = bcn[0] ** 2 + bcn[1] ** 2 + bcn[2] ** 2
        v = [u[q] / u[0] for q in (1, 2, 3)]
        rho, e = self.floors(u[0], (u[4] - 0.5 * b2) / u[0] - 0.5 * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2))
        return self.boundary({"w": [self.put(a, x) for a, x in zip(s["w"], [rho] + v)],
                              "bc": [self.put(a, x) for a, x in zip(s["bc"], bcn)], "eps": self.put(s["eps"], e),
                              "bf": bf})

    def states(self, a, d):
        """left and right states at the face between a cell and the next one (solver/reconstruct.f90)"""
        t = self.tab[d]
        up, dn = _shift(a, d, 1) - a, a - _shift(a, d, -1)
        if self.p.recon == N.TVDMM:
            f, b = 2 * up / t["cf"], 2 * dn / t["cb"]
            sl = torch.where(f * b > 0, torch.where(f.abs() < b.abs(), f, b), torch.zeros_like(f))
            vm, vp = a - 0.5 * sl, a + 0.5 * sl
        else:
            delta = t["b0"] * up + t["b1"] * dn
            lim = torch.minimum(torch.minimum(delta.abs(), 2 * dn.abs()), 2 * up.abs())
            lim = torch.where(up * dn > 0, torch.where(delta > 0, lim, -lim), torch.zeros_like(lim))
            face = a + t["a1"] * up + t["a2"] * _shift(lim, d, 1) + t["a3"] * lim
            vl, vr = _shift(face, d, -1), face
            flat = (vr - a) * (a - vl) <= 0
            vm = torch.where((vr - vl) * (vl - 3 * a + 2 * vr) < 0, 3 * a - 2 * vr, vl)
            vp = torch.where((vr - vm) * (3 * a - 2 * vl - vr) < 0, 3 * a - 2 * vl, vr)
            vm, vp = torch.where(flat, a, vm), torch.where(flat, a, vp)
        return vp, _shift(vm, d, 1)

    def fluxes(self, d, *prims):
        """HLL fluxes of the faces of axis d: rho, rho v, E and the three field components (solver/rsolver.f90)"""
        g, w, bc, bn = self.p.ggas, prims[:5], prims[5:8], prims[8]
        t1, t2 = (d + 1) % 3, (d + 2) % 3
        sides = []
        both = [self.states(a, d) for a in w]
        bt = {t1: self.states(bc[t1], d), t2: self.states(bc[t2], d)}
        for s in range(2):
            rho, v, pr = both[0][s], [both[1 + q][s] for q in range(3)], both[4][s]
            b = [bn if q == d else bt[q][s] for q in range(3)]
            a2, b2n = g * pr / rho, b[d] ** 2 / rho
            b2 = b2n + (b[t1] ** 2 + b[t2] ** 2) / rho
            disc = (a2 + b2) ** 2 - 4 * a2 * b2n
            root = torch.where(disc > 0, disc, torch.ones_like(disc)).sqrt() * (disc > 0)
            cf = (0.5 * (a2 + b2 + root)).sqrt()
            bsq, vb = b[0] ** 2 + b[1] ** 2 + b[2] ** 2, b[0] * v[0] + b[1] * v[1] + b[2] * v[2]
            e = pr / (g - 1.0) + 0.5 * rho * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2) + 0.5 * bsq
            u = [rho, rho * v[0], rho * v[1], rho * v[2], e] + b
            f = [x * v[d] for x in u]
            for q in range(3):
                f[1 + q] = f[1 + q] - b[d] * b[q]
                f[5 + q] = f[5 + q] - b[d] * v[q]
            f[1 + d] = f[1 + d] + pr + 0.5 * bsq
            f[4] = f[4] + (pr + 0.5 * bsq) * v[d] - b[d] * vb
            sides.append((u, f, v[d], cf, rho.sqrt()))
        (ul, fl, vl, cl, ql), (ur, fr, vr, cr, qr) = sides
        ubar, cbar = (ql * vl + qr * vr) / (ql + qr), (ql * cl + qr * cr) / (ql + qr)
        sl, sr = torch.minimum(vl - cl, ubar - cbar), torch.maximum(vr + cr, ubar + cbar)
        out = []
        for q in range(8):
            if q == 5 + d:
                continue
            mid = (sr * fl[q] - sl * fr[q] + sl * sr * (ur[q] - ul[q])) / (sr - sl)
            out.append(torch.where(sl >= 0, fl[q], torch.where(sr >= 0, mid, fr[q])))
        return tuple(out)

    def flux_geometry(self, d):
        x, y, z = self.tab
        one = torch.ones((1, 1, 1), dtype=torch.float64, device=self.dev)
        if self.p.coordinate == N.CARTESIAN:
            return one, one, self.tab[d]["w"]
        if self.p.coordinate == N.CYLINDRICAL:
            return [(x["f"], x["fm"], x["c"] * x["w"]), (one, one, x["c"] * y["w"]), (one, one, z["w"])][d]
        return [(self.r2, self.r2m, self.r3), (self.sin, self.sinm, self.rfac * self.dcos),
                (one, one, self.rfac * self.dcos * z["w"] / y["w"])][d]

    def sources(self, w, bc):
        p, (x, _, z) = self.p, self.tab
        I = self.inner
        rho, vx, vy, vz, pr, bx, by, bz = [a[I] for a in list(w) + list(bc)]
        r = x["c"][..., 3:3 + p.nx]
        b2, rep = bx ** 2 + by ** 2 + bz ** 2, p.geom_source_repeat
        sc = [torch.zeros_like(rho) for _ in range(5)]
        if p.coordinate == N.CYLINDRICAL:
            sc[1] = sc[1] + rep * (pr + rho * vy ** 2 + 0.5 * b2 - by ** 2) / r
            sc[2] = sc[2] - rep * (rho * vx * vy - bx * by) / r
        elif p.coordinate == N.SPHERICAL:
            tan = self.tanc[:, 3:3 + p.ny]
            sc[1] = sc[1] + rep * (2 * pr + bx ** 2 + rho * (vy ** 2 + vz ** 2)) / r
            sc[2] = sc[2] + rep * ((pr + rho * vz ** 2 + 0.5 * b2 - bz ** 2) / (r * tan) - (rho * vx * vy - bx * by) / r)
            sc[3] = sc[3] - rep * ((rho * vx * vz - bx * bz) / r + (rho * vy * vz - by * bz) / (r * tan))
        if p.model in (N.MODEL_TORUS_SPH, N.MODEL_TORUS_CYN):
            on = (rho >= p.rho_floor).double() * rho
            if p.model == N.MODEL_TORUS_SPH:
                gr, gz = 1.0 / (r - p.r_sh) ** 2, None
            else:
                zc = z["c"][3:3 + p.nz]
                rad = (r ** 2 + zc ** 2).sqrt()
                gr, gz = r / rad / (rad - p.r_sh) ** 2, zc / rad / (rad - p.r_sh) ** 2
            sc[1], sc[4] = sc[1] - on * gr, sc[4] - on * vx * gr
            if gz is not None:
                sc[3], sc[4] = sc[3] - on * gz, sc[4] - on * vz * gz
        return sc

    def spatial(self, s, keep):
        """l_rk: hydro on the cells 1..n and the curl of the edge EMFs on whole arrays"""
        w, bc, bf = s["w"], s["bc"], s["bf"]
        F = []
        for d in range(3):
            args = (d, *w, *bc, bf[d])
            F.append(self.fluxes(*args) if keep else checkpoint(self.fluxes, *args, use_reentrant=False))
        L = [0.0] * 5
        for d in range(3):
            gp, gm, gc = self.flux_geometry(d)
            for q in range(5):
                L[q] = L[q] - ((F[d][q] * gp - _shift(F[d][q], d, -1) * gm) / gc)[self.inner]
        L = [a + b for a, b in zip(L, self.sources(w, bc))]
        # x faces carry (by, bz) fluxes, y faces (bx, bz), z faces (bx, by)
        v = w[1:4]
        cell = [v[2] * bc[1] - v[1] * bc[2], v[0] * bc[2] - v[2] * bc[0], v[1] * bc[0] - v[0] * bc[1]]

        def edge(c, a, fa, b, fb):  # EMF along c: fluxes fa of the a faces and fb of the b faces
            e = 0.5 * (fa + _shift(fa, b, 1)) + 0.5 * (fb + _shift(fb, a, 1))
            m = cell[c] + _shift(cell[c], a, 1)
            return e - 0.25 * (m + _shift(m, b, 1))

        E = [edge(0, 1, -F[1][6], 2, F[2][6]), edge(1, 0, F[0][6], 2, -F[2][5]), edge(2, 0, -F[0][5], 1, F[1][5])]
        x, y, z = self.tab
        if self.p.coordinate == N.CARTESIAN:
            one = 1.0
            g = {"xz": (one, one, y["w"]), "xy": (one, one, z["w"]), "yx": (one, one, z["w"]),
                 "yz": (one, one, x["w"]), "zy": (one, one, x["w"]), "zx": (one, one, y["w"])}
        elif self.p.coordinate == N.CYLINDRICAL:
            g = {"xz": (1.0, 1.0, y["w"] * x["f"]), "xy": (1.0, 1.0, z["w"]), "yx": (1.0, 1.0, z["w"]),
                 "yz": (1.0, 1.0, x["w"]), "zy": (x["f"], x["fm"], x["c"] * x["w"]), "zx": (1.0, 1.0, x["c"] * y["w"])}
        else:
            g = {"xz": (self.sin, self.sinm, x["f"] * self.dcos), "xy": (1.0, 1.0, x["f"] * self.dcos * z["w"] / y["w"]),
                 "yx": (1.0, 1.0, x["c"] * self.sin * z["w"]), "yz": (x["f"], x["fm"], x["c"] * x["w"]),
                 "zy": (x["f"], x["fm"], x["c"] * x["w"]), "zx": (1.0, 1.0, x["c"] * y["w"])}

        def diff(e, d, k):
            gp, gm, gc = g[k]
            return (E[e] * gp - _shift(E[e], d, -1) * gm) / gc

        return L, [diff(1, 2, "xy") - diff(2, 1, "xz"), diff(2, 0, "yz") - diff(0, 2, "yx"),
                   diff(0, 1, "zx") - diff(1, 0, "zy")]

    def live(self, c, new, old):
        """new on the live faces of component c (0..n along c, 1..n across), old elsewhere"""
        mask = torch.zeros_like(old, dtype=torch.bool)
        at = list(self.inner)
        at[2 - c] = slice(2, 3 + self.n[c])
        mask[tuple(at)] = True
        return torch.where(mask, new, old)

    def stage(self, s, u0, b0, dt, stage, keep=True):
        k0, k1 = ((0.0, 1.0), (0.75, 0.25), (1.0 / 3.0, 2.0 / 3.0))[stage]
        u = [a[self.inner] for a in self.cons(s)]
        L, LB = self.spatial(s, keep)
        un = [k0 * a + k1 * (b + dt * c) for a, b, c in zip(u0, u, L)]
        bf = [self.live(c, k0 * b0[c] + k1 * (s["bf"][c] + dt * LB[c]), s["bf"][c]) for c in range(3)]
        return self.primitives(un, bf, s)

    def dt(self, s):
        p, (x, y, z) = self.p, self.tab
        rho, vx, vy, vz, pr = [a[self.inner] for a in s["w"]]
        b = [a[self.inner] for a in s["bc"]]
        a2, b2 = p.ggas * pr / rho, (b[0] ** 2 + b[1] ** 2 + b[2] ** 2) / rho
        speed = None
        for d, v in enumerate((vx, vy, vz)):
            c = (0.5 * (a2 + b2 + ((a2 + b2) ** 2 - 4 * a2 * b[d] ** 2 / rho).sqrt())).sqrt() + v.abs()
            speed = c if speed is None else torch.maximum(speed, c)
        dx, dy, dz = x["w"], y["w"], z["w"]
        if p.coordinate != N.CARTESIAN:
            dy = x["c"] * dy
        if p.coordinate == N.SPHERICAL:
            dz = x["c"] * self.sinc * dz
        least = torch.minimum(torch.minimum(dx, dy), dz).expand(s["eps"].shape)[self.inner]
        return float((least * p.cfl / speed).min())


def exact(case, seed):
    p = _problem(case, seed)
    e = _Exact(p)
    prim, eps = torch.from_numpy(p.prim).to(e.dev), torch.from_numpy(p.eps).to(e.dev)
    if case["drive"] == "adjoint":
        return _exact_gradient(case, e, prim, eps)
    with torch.no_grad():
        s = e.initial(prim, eps)
        for _ in range(case["steps"]):
            dt, b0 = e.dt(s), s["bf"]
            u0 = [a[e.inner] for a in e.cons(s)]
            for k in range(3):
                s = e.stage(s, u0, b0, dt, k)
        if case["drive"] == "slabs":
            # w, bcell and eps of each slab's planes; a slab's cons have no
            # value in its ghost planes, which nothing reads
            cuts = ZSlabs(p, case["slabs"])
            whole = torch.stack(list(s["w"]) + list(s["bc"]) + [s["eps"]]).cpu()
            return {"cons": None, "prims": [whole[:, o:o + m + 6] for o, m in zip(cuts.offsets, cuts.counts)]}
        return {"prim": torch.stack(list(s["w"]) + list(s["bf"]), 3).cpu(), "eps": s["eps"].cpu()}


def _exact_gradient(case, e, prim, eps):
    """the objective after the steps and its gradient by reverse-mode
    differentiation, each stage recomputed in the reverse pass"""
    prim.requires_grad_(True)
    eps.requires_grad_(True)
    s, dts = e.initial(prim, eps), []
    keys = [("w", 5), ("bc", 3), ("bf", 3)]

    def flat(s):
        return [*s["w"], *s["bc"], *s["bf"], s["eps"]]

    def state(a):
        return {"w": list(a[:5]), "bc": list(a[5:8]), "bf": list(a[8:11]), "eps": a[11]}

    for _ in range(case["steps"]):
        with torch.no_grad():
            dt = e.dt(s)
        dts.append(dt)
        b0, u0 = s["bf"], [a[e.inner] for a in e.cons(s)]
        for k in range(3):
            def one(*a, k=k, dt=dt):
                return tuple(flat(e.stage(state(a[:12]), a[12:17], a[17:20], dt, k, keep=False)))
            s = state(checkpoint(one, *flat(s), *u0, *b0, use_reentrant=False))
    p, (x, y, z) = e.p, e.tab
    vol = {N.CARTESIAN: x["w"] * y["w"] * z["w"], N.CYLINDRICAL: x["c"] * x["w"] * y["w"] * z["w"],
           N.SPHERICAL: e.r3 * e.dcos * z["w"]}[p.coordinate].expand(s["eps"].shape)[e.inner]
    if case["objective"] == "magnetic":
        J = (0.5 * sum(a[e.inner] ** 2 for a in s["bc"]) * vol).sum()
    else:
        J = (0.5 * s["w"][0][e.inner] * sum(a[e.inner] ** 2 for a in s["w"][1:4]) * vol).sum()
    J.backward()
    return {"J": float(J.detach()), "dts": np.array(dts), "grad_prim": prim.grad.cpu(), "grad_eps": eps.grad.cpu()}
