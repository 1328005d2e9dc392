"""The workloads that the framework's speed is judged by, each a pass through its public entry points.

A case is a dict of plain values. Three kinds, after what a user of the framework runs:

  mhd     a Yin-Yang shell handed over by the host (core upload from pinned memory), advanced by some RK4
          steps and taken back (core download): falcon_gb300.Falcon
  solve   an implicit solve to a tolerance and its solution on the host, heat conduction or a batch of PFSS
          fields: falcon_gb300.solver.Solver
  net     the learned coarse correction, a forward pass or a loss with its gradient: falcon_gb300.lcc.LCC

Grids are those of falcon_gb300.config, the command lines, bench.py and tests, or other tilings of the same form.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

import falcon_gb300 as fg
from falcon_gb300 import config, lcc, solver, synth

# 16^3 blocks cost this much work per cell: one RK4 step reads and writes the state 14 times (each of four stages
# reads u_s and u^n and writes u_s+1, the diffusion reads and writes) and forms its time step from v and B
STATE_PASSES, CFL_VALUES = 14, 6
STAGE_FLOPS, DIFFUSION_FLOPS = 600, 900     # per cell, all variables, from the formulas
EXACT_CELLS = 500_000                       # grids above take longer than 20 s in 64-bit torch


def _mhd(name, block, tiles_r, tiles_t, levels, amr, precision, steps, every_dt=False, divb=0):
    return {"kind": "mhd", "name": name, "block": block, "tiles_r": tiles_r, "tiles_t": tiles_t, "levels": levels,
            "amr": amr, "precision": precision, "steps": steps, "every_dt": every_dt, "divb": divb}


def _conduction(name, nr, nt, tol):
    return {"kind": "conduction", "name": name, "nr": nr, "nt": nt, "tol": tol}


def _pfss(name, problems, nr, nt, sizes_seed, tol):
    return {"kind": "pfss", "name": name, "problems": problems, "nr": nr, "nt": nt, "sizes_seed": sizes_seed, "tol": tol}


def _net(name, mode, n, D, H, W):
    return {"kind": "net", "name": name, "mode": mode, "n": n, "D": D, "H": H, "W": W}


def listed():
    return [
        # the production run: the 21,233,664-cell shell, 20 steps between two outputs
        _mhd("mixed_21m_20_steps", 16, 3, 3, 1, 2, "mixed", 20),
        # a driver that keeps the state on the host and hands it over every step (5,308,416 cells)
        _mhd("mixed_5m_host_step", 16, 3, 3, 1, 1, "mixed", 1, every_dt=True),
        # a development run: 442,368 cells in 108 blocks, the step's dt read by the driver each time
        _mhd("mixed_442k_10_steps", 16, 1, 3, 1, 0, "mixed", 10, every_dt=True),
        # the smallest shell (110,592 cells in 216 small blocks): launches and the dt read per step
        _mhd("mixed_tiny_20_steps", 8, 1, 3, 1, 0, "mixed", 20, every_dt=True),
        # div-B cleaning switched on, small blocks
        _mhd("mixed_glm_442k_10_steps", 8, 1, 3, 2, 1, "mixed", 10, divb=1),
        # the bit-exact path on its own shell, as a run that is compared with the CPU code
        _mhd("fp64_442k_10_steps", 8, 1, 3, 2, 1, "fp64", 10),
        # the bit-exact path on the production block size, Powell's source term
        _mhd("fp64_powell_442k_3_steps", 16, 1, 3, 1, 0, "fp64", 3, every_dt=True, divb=2),
        # the implicit conduction step of the 6,291,456-cell shell
        _conduction("conduction_6m", 64, 128, 1e-10),
        # eight magnetograms of uneven resolution in one batch
        _pfss("pfss_batch_8", 8, 0, 0, 5000, 1e-11),
        # one magnetogram at low resolution
        _pfss("pfss_24x45", 1, 24, 45, 0, 1e-11),
        # the correction of one V-cycle: both panels of the 6.3M-cell system's coarsest level
        _net("net_forward_2_panels", "forward", 2, 16, 32, 96),
        # one training step's loss and gradient on a batch of panels
        _net("net_gradient_8_panels", "gradient", 8, 16, 32, 96),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["mixed", "mixed", "mixed", "fp64", "conduction", "pfss", "pfss", "net"])
    if kind in ("mixed", "fp64"):
        cells = _log_uniform(rng, 1e5, 8e6 if kind == "mixed" else 6e5)
        while True:
            block, levels, amr = rng.choice([8, 16]), rng.randint(0, 2), rng.randint(0, 2)
            tiles_r, tiles_t = rng.randint(1, 3), rng.randint(1, 7)
            n = _cells(block, tiles_r, tiles_t, levels, amr)
            if 0.7 * cells < n < 1.4 * cells and tiles_t * 2 ** amr >= 3 and block * tiles_r * 2 ** levels >= 32:
                break    # coarser shells do not resolve the stratification
        c = _mhd("", block, tiles_r, tiles_t, levels, amr, kind, rng.randint(1, 12) if kind == "mixed" else rng.randint(1, 4),
                 rng.random() < 0.5, rng.choice([0, 0, 0, 1, 2]))
    elif kind == "conduction":
        c = _conduction("", 16 * rng.randint(2, 5), 16 * rng.randint(2, 9), 10.0 ** -rng.randint(9, 11))
    elif kind == "pfss":
        if rng.random() < 0.5:
            c = _pfss("", 1, rng.randint(24, 64), rng.randint(45, 180), 0, 10.0 ** -rng.randint(10, 11))
        else:
            c = _pfss("", rng.randint(2, 10), 0, 0, rng.randint(1, 9999), 10.0 ** -rng.randint(10, 11))
    else:
        c = _net("", rng.choice(["forward", "gradient"]), rng.randint(1, 8), 8 * rng.randint(1, 3), 8 * rng.randint(2, 6),
                 8 * rng.randint(4, 14))
    del c["name"]
    return c


# ---- grids -------------------------------------------------------------------

def _cells(block, tiles_r, tiles_t, levels, amr):
    return 2 * tiles_r * 3 * tiles_t * tiles_t * 2 ** levels * 4 ** amr * block ** 3


def _grid(case, device=0):
    return config.make_config(block=(case["block"],) * 3, root_tiles=(case["tiles_r"], case["tiles_t"], 3 * case["tiles_t"]),
                              radial_levels=case["levels"], radial_option=1, amr=((0, 1, 1),) * case["amr"], device=device,
                              precision=config.PREC_MIXED if case["precision"] == "mixed" else config.PREC_FP64,
                              divb_option=case["divb"])


def _spec(case, seed, device=0):
    if case["kind"] == "conduction":
        return solver.conduction_spec(nr=case["nr"], nt=case["nt"], np_=3 * case["nt"], seed=seed, device=device)
    sizes = [(case["nr"], case["nt"])] if case["nr"] else solver.random_pfss_sizes(case["problems"], case["sizes_seed"])
    return solver.pfss_spec(sizes, seed=seed, device=device)


def _psi(u):
    """GLM's psi of a state: a thousandth of the base sound speed times B_r."""
    c_b = synth.polytrope_constants(0.7 * synth.R_SUN, synth.R_SUN)["c_b"]
    u[:, 8] = 1e-3 * c_b * u[:, 4]


def _initial(case, f, seed, u):
    """The state a run starts from: entropy bump, dipole and a random-phase velocity at rms Mach 0.01."""
    f.init_synthetic(kind=1, seed=seed, mach=0.01)
    f.exchange()
    f.download_state_into(u)
    if case["divb"] == 1:
        _psi(u)


class Shell:
    """A shell on the GPU and the host arrays, pinned, that the driver hands over and takes back."""

    def __init__(self, case, seed):
        self.case = case
        self.f = fg.Falcon(_grid(case))
        self.pinned = []
        self.u = self._pinned()
        self.out = self._pinned()
        _initial(case, self.f, seed, self.u)
        self.f.upload_state_raw(self.u)
        self.f.download_state_into(self.out)

    def _pinned(self):
        a = fg.host_array(self.f.shape)
        self.f.pin_host(a)
        self.pinned.append(a)
        return a

    def __del__(self):
        if hasattr(self, "pinned"):
            for a in self.pinned:
                self.f.unpin_host(a)
        if hasattr(self, "f"):
            self.f.close()


def prepare(case, seed):
    if case["kind"] == "mhd":
        return Shell(case, seed)
    if case["kind"] == "net":
        x, t = _net_inputs(case, seed)
        return {"case": case, "net": lcc.LCC(seed=_net_seed(seed)), "x": x, "t": t}
    return {"case": case, "solver": solver.Solver(_spec(case, seed))}


def run(state):
    if isinstance(state, Shell):
        f, case, dts = state.f, state.case, []
        f.upload_state_core(state.u)
        if case["every_dt"]:
            dts = [f.advance_rk4() for _ in range(case["steps"])]
        else:
            f.run_steps(case["steps"])
        f.synchronize()
        f.download_state_core(state.out)
        return {"state": state.out, "dt": np.array(dts)}
    case = state["case"]
    if case["kind"] == "net":
        if case["mode"] == "forward":
            return {"y": state["net"].forward(state["x"])}
        loss, grad = state["net"].loss_grad(state["x"], state["t"])
        return {"loss": loss, "gradient": grad}
    s = state["solver"]
    s.solve(tol=case["tol"], max_iter=2000)
    return {"solution": s.solution()}


def work(case):
    if case["kind"] == "mhd":
        cells = _cells(case["block"], case["tiles_r"], case["tiles_t"], case["levels"], case["amr"])
        size = 4 if case["precision"] == "mixed" else 8
        nv = 9 if case["divb"] == 1 else 8
        core = 8 * nv * cells * (case["block"] + 4) / case["block"]     # handed over and taken back, each once
        return {"bytes": case["steps"] * cells * size * (STATE_PASSES * nv + CFL_VALUES) + 2 * core,
                "flops": case["steps"] * cells * (4.0 * STAGE_FLOPS + DIFFUSION_FLOPS)}
    if case["kind"] == "net":
        vox = case["n"] * case["D"] * case["H"] * case["W"]
        scale = [1, 1, 8, 8, 64, 512, 64, 8, 1, 1]
        flops = sum(2.0 * 27 * ci * co * vox / s for (ci, co), s in zip(NET_LAYERS, scale))
        back = 1 if case["mode"] == "forward" else 3
        return {"bytes": vox * 4.0 * (8 + 1) + 4.0 * (NET_PARAMS if back == 1 else 2 * NET_PARAMS), "flops": back * flops}
    # a solve reads its seven-point operator (four face arrays), its right-hand side and its guess, and writes the
    # solution; an iteration at the least applies the operator in its working precision, 10 of them to 1e-8
    cells = _solve_cells(case)
    its = (1.25 if case["kind"] == "conduction" else 4.6) * -math.log10(case["tol"])
    return {"bytes": cells * (7 * 8.0 + its * 6 * 8.0), "flops": cells * its * 2 * 7 * 4.0}


def _solve_cells(case):
    if case["kind"] == "conduction":
        return 2 * case["nr"] * case["nt"] * 3 * case["nt"]
    sizes = [(case["nr"], case["nt"])] if case["nr"] else solver.random_pfss_sizes(case["problems"], case["sizes_seed"])
    return sum(2 * 8 * -(-nr // 8) * 3 * (8 * -(-(nt // 2) // 8)) ** 2 for nr, nt in sizes)


# ---- what the passes compute, in 64 bits -------------------------------------

def exact(case, seed):
    if case["kind"] == "net":
        return _exact_net(case, seed)
    if case["kind"] == "mhd":
        if _cells(case["block"], case["tiles_r"], case["tiles_t"], case["levels"], case["amr"]) > EXACT_CELLS:
            return None
        f = fg.Falcon(_grid(case))
        u = np.empty(f.shape)
        _initial(case, f, seed, u)
        f.close()
        state, dts = ExactShell(case).run(u, case["steps"])
        return {"state": state, "dt": np.array(dts if case["every_dt"] else [])}
    if _solve_cells(case) > EXACT_CELLS:
        return None
    s = solver.Solver(_spec(case, seed, device=-1))
    return {"solution": _exact_solve(s)}


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _convert(theta, phi):
    """Yin-Yang transform of a direction."""
    st, ct, sp, cp = torch.sin(theta), torch.cos(theta), torch.sin(phi), torch.cos(phi)
    t = torch.acos(st * sp)
    p = torch.acos(-(st * cp) / torch.sqrt(st * st * cp * cp + ct * ct))
    return t, torch.copysign(p.abs(), ct)


class ExactShell:
    """The RK4 step of a shell as formulas on whole arrays u[block][variable][k][j][i] with two ghost layers."""

    def __init__(self, case):
        dev = _device()
        f = fg.Falcon(_grid(case, device=-1))
        put = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)
        n = self.n = case["block"]
        self.divb = case["divb"]
        nb = f.nblocks
        rg, flags, prof, gm = put(f.block_ranges()), put(f.block_flags()), put(f.background()), f.ghost_map()
        self.cfl = f.cfg.phys.cfl
        heating = f.cfg.phys.heating_ratio
        f.close()
        i = torch.arange(-1, n + 3, device=dev, dtype=torch.float64)
        x = [(rg[:, d, 0:1] * (n - i + 0.5) + rg[:, d, 1:2] * (i - 0.5)) / n for d in range(3)]
        self.dx = [((rg[:, d, 1] - rg[:, d, 0]) / n).view(nb, 1, 1, 1) for d in range(3)]
        self.c = [float(np.float32(1 / 12)) / d for d in self.dx]
        self.r, th = x[0].view(nb, 1, 1, -1), x[1].view(nb, 1, -1, 1)
        self.sin, self.cot = torch.sin(th), torch.cos(th) / torch.sin(th)
        g, rho0, p0, T0, g1, g3, dif, cool, xi = (prof[:, q].view(nb, 1, 1, -1) for q in range(9))
        self.rho0, self.xi2, self.g_rho0 = rho0, xi * xi, g / rho0
        self.a1, self.a2 = g1 * (p0 / rho0), (g3 - 1) * rho0 * T0
        self.heat = heating * (dif + cool) / (rho0 * T0)
        self.cs = torch.sqrt(g1 * (p0 / rho0)) / xi
        self.top, self.bottom = (flags & 2) != 0, (flags & 4) != 0
        # ghost map: base cell, weights and rotation of every entry
        tb, sb = put(gm["tblock"].astype(np.int64)), put(gm["sblock"].astype(np.int64))
        npad = n + 4
        self.tb, self.sb = tb, sb
        at = [put(gm[k].astype(np.int64)) + 1 for k in ("ti", "tj", "tk")]
        self.tc = (at[2] * npad + at[1]) * npad + at[0]
        src = put(gm["src_x"])
        base, self.w = [], []
        for d in range(3):
            xs = x[d][sb]
            p = (-1 + (src[:, d] - xs[:, 0]) / (xs[:, 3] - xs[:, 2])).clamp(1.0, float(n))
            base.append(p.floor())
            self.w.append((p - base[-1]).view(-1, 1))
        b = [q.long() + 1 for q in base]
        self.sc = (b[2] * npad + b[1]) * npad + b[0]
        self.step = (1, npad, npad * npad)
        yin = (flags & 1)
        self.rot = (yin[tb] != yin[sb]).nonzero().view(-1)
        _, back_p = _convert(src[self.rot, 1], src[self.rot, 2])
        back_t, _ = _convert(src[self.rot, 1], src[self.rot, 2])
        self.ra = torch.sin(src[self.rot, 2]) * torch.sin(back_p)
        self.rc = torch.cos(src[self.rot, 2]) / torch.sin(back_t)

    def at(self, f, axis=0, m=0):
        """The interior of f (blocks first, k, j, i last), shifted by m cells along axis (0: i, 1: j, 2: k)."""
        for a, dim in enumerate((-1, -2, -3)):
            if f.shape[dim] != 1:
                f = f.narrow(dim, 2 + (m if a == axis else 0), self.n)
        return f

    def d(self, f, axis):
        """Fourth-order derivative along an axis."""
        return self.c[axis] * (-self.at(f, axis, 2) + 8 * self.at(f, axis, 1) - 8 * self.at(f, axis, -1) + self.at(f, axis, -2))

    def exchange(self, u):
        flat = u.flatten(2)
        val = 0
        for q in range(8):
            w, off = 1.0, 0
            for d in range(3):
                w = w * (self.w[d] if q >> d & 1 else 1 - self.w[d])
                off += self.step[d] if q >> d & 1 else 0
            val = val + w * flat[self.sb, :, self.sc + off]
        for t, p in ((2, 3), (5, 6)):
            vt, vp = val[self.rot, t], val[self.rot, p]
            val[self.rot, t] = -(self.ra * vt) - self.rc * vp
            val[self.rot, p] = -(self.ra * vp) + self.rc * vt
        flat[self.tb, :, self.tc] = val

    def boundary(self, u):
        n = self.n
        for on, ghost, src, odd in ((self.top, (n + 2, n + 3), (n + 1, n), (1, 5, 6)), (self.bottom, (1, 0), (2, 3), (1, 4))):
            s = torch.ones(8, 1, 1, dtype=u.dtype, device=u.device)
            s[list(odd)] = -1
            b = on.nonzero().view(-1)
            for gi, si in zip(ghost, src):
                u[b, :8, :, :, gi] = s * u[b, :8, :, :, si]

    def speed(self, u):
        v = [self.at(u[:, q]) for q in range(1, 7)]
        r, sin = self.at(self.r), self.at(self.sin)
        w = self.at(self.cs) + torch.sqrt(v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
        w = w + torch.sqrt(v[3] ** 2 + v[4] ** 2 + v[5] ** 2) / torch.sqrt(self.at(self.rho0))
        return w, torch.minimum(torch.minimum(self.dx[0].expand_as(r), r * self.dx[1]), r * sin * self.dx[2])

    def rhs(self, u, u0):
        rho1, vr, vt, vp, br, bt, bp, s1, psi = (u[:, q] for q in range(9))
        at, d, r, sin, rho0 = self.at, self.d, self.r, self.sin, self.rho0
        ri, si, ci, rhoi = at(r), at(sin), at(self.cot), at(rho0)
        ur, ut, up, b1, b2, b3 = (at(f) for f in (vr, vt, vp, br, bt, bp))
        R = [None] * 9
        div = d(rho0 * vr * r * r, 0) / ri ** 2 + (d(rho0 * vt * sin, 1) + d(rho0 * vp, 2)) / si / ri
        R[0] = -div / at(self.xi2)
        adv = lambda f: ur * d(f, 0) + ut * d(f, 1) / ri + up * d(f, 2) / ri / si
        R[1] = -(adv(vr) - (ut * ut + up * up) / ri)
        R[2] = -(adv(vt) + (ut * ur - up * up * ci) / ri)
        R[3] = -(adv(vp) + (up * ur + up * ut * ci) / ri)
        p1 = self.a1 * rho1 + self.a2 * s1
        k1 = (d(bp * sin, 1) - d(bt, 2)) / ri / si
        k2 = (d(br / sin, 2) - d(bp * r, 0)) / ri
        k3 = (d(bt * r, 0) - d(br, 1)) / ri
        R[1] = R[1] + (k2 * b3 - k3 * b2 - d(p1, 0)) / rhoi - at(self.g_rho0) * at(rho1)
        R[2] = R[2] + (k3 * b1 - k1 * b3 - d(p1, 1) / ri) / rhoi
        R[3] = R[3] + (k1 * b2 - k2 * b1 - d(p1, 2) / ri / si) / rhoi
        e1, e2, e3 = vt * bp - vp * bt, vp * br - vr * bp, vr * bt - vt * br
        R[4] = (d(e3 * sin, 1) - d(e2, 2)) / ri / si
        R[5] = (d(e1 / sin, 2) - d(e3 * r, 0)) / ri
        R[6] = (d(e2 * r, 0) - d(e1, 1)) / ri
        R[7] = -adv(s1) + at(self.heat)
        R[8] = torch.zeros_like(R[0])
        if self.divb:
            divb = d(br * r * r, 0) / ri ** 2 + (d(bt * sin, 1) + d(bp, 2)) / si / ri
        if self.divb == 2:
            for q, v in ((4, ur), (5, ut), (6, up)):
                R[q] = R[q] - divb * v
        if self.divb == 1:
            R[4], R[5], R[6] = R[4] - d(psi, 0), R[5] - d(psi, 1) / ri, R[6] - d(psi, 2) / ri / si
            w, h = self.speed(u0)
            R[8] = -w * w * divb - w / h * at(psi)
        return torch.stack(R, 1)

    def slope(self, l, m, r):
        a, b, c = (r - l) * 0.5, 2 * (r - m), 2 * (m - l)
        zero = torch.zeros_like(a)
        t = torch.fmax(zero, a * b) * torch.fmax(zero, b * c) * 1e10 - float(np.float32(1e-30))
        s = torch.fmin(torch.fmin(a.abs(), b.abs()), c.abs())
        return torch.where(t >= 0, torch.copysign(s, a), zero)

    def flux(self, f, speed, axis, side):
        """Limited flux through the face between cells side-1 and side along an axis."""
        at = lambda m: self.at(f, axis, side + m)
        l, r = at(-1), at(0)
        num = ((r - self.slope(l, r, at(1)) * 0.5) - l) - self.slope(at(-2), l, r) * 0.5
        phi = torch.fmax(torch.zeros_like(num), 1 + 2 * (num / (r - l) - 1))
        c = self.at(speed, axis, side) + self.at(speed, axis, side - 1)
        return -(0.5 * phi * num) * c.unsqueeze(1) * 0.5

    def diffusion(self, u):
        ri = self.at(self.r)
        den = (self.dx[0], self.dx[1] * ri, self.dx[2] * ri * self.at(self.sin))
        R = 0
        for axis in range(3):
            speed = u[:, 1 + axis].abs() + self.cs
            R = R + (self.flux(u, speed, axis, 0) - self.flux(u, speed, axis, 1)) / den[axis].unsqueeze(1)
        return R

    def run(self, start, steps):
        n = self.n
        inner = (slice(None), slice(None)) + (slice(2, n + 2),) * 3
        u = torch.as_tensor(start, device=_device()).clone()
        core = (slice(None), slice(None), slice(2, n + 2), slice(2, n + 2))
        out, dts = u.clone(), []
        for _ in range(steps):
            w, h = self.speed(u)
            dt = min(float(np.float32(1e20)), self.cfl * float((h / w).min()))
            dts.append(dt)
            cur = u
            for s in range(1, 5):
                self.boundary(cur)
                new = cur if s > 1 else u.clone()
                new[inner] = u[inner] + dt * self.rhs(cur, u) / (5 - s)
                if s == 4:
                    u[inner] = new[inner]
                    new = u
                self.exchange(new)
                cur = new
            u[inner] = u[inner] + 0.5 * dt * self.diffusion(u)
            self.exchange(u)
        out[core] = u[core]
        return out, dts


def _exact_solve(s):
    """A x = b on every problem of a solver, by stabilised bi-conjugate gradients in 64 bits."""
    dev = _device()
    put = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)
    Aii, Ai, Aj, Ak = (put(a) for a in s.operator(0))
    b = put(s.rhs())
    idx, wx = s.halo_map(0)
    idx, wx = put(idx.astype(np.int64)), put(wx)
    nb, m2, m1, m0 = b.shape
    p0, p1 = m0 + 2, m1 + 2
    npad = p0 * p1 * (m2 + 2)
    tgt = idx[:, 0] * npad + (idx[:, 3] * p1 + idx[:, 2]) * p0 + idx[:, 1]
    src = idx[:, 4] * npad + (idx[:, 7] * p1 + idx[:, 6]) * p0 + idx[:, 5]
    step = (1, p0, p0 * p1)
    corners = []
    for q in range(8):
        w, off = 1.0, 0
        for d in range(3):
            w = w * (wx[:, d] if q >> d & 1 else 1 - wx[:, d])
            off = off + (torch.where(wx[:, d] != 0, step[d], 0) if q >> d & 1 else 0)
        corners.append((w, src + off))
    first = torch.as_tensor(s.problem_blocks().astype(np.int64), device=dev)
    prob = torch.bucketize(torch.arange(nb, device=dev), first[1:], right=True)
    pad = torch.zeros(nb, m2 + 2, p1, p0, dtype=torch.float64, device=dev)
    s.close()

    def apply(x):
        pad[:, 1:-1, 1:-1, 1:-1] = x
        flat = pad.view(-1)
        flat[tgt] = sum(w * flat[c] for w, c in corners)
        return (Aii * x + Ai[..., :-1] * pad[:, 1:-1, 1:-1, :-2] + Ai[..., 1:] * pad[:, 1:-1, 1:-1, 2:] +
                Aj[:, :, :-1] * pad[:, 1:-1, :-2, 1:-1] + Aj[:, :, 1:] * pad[:, 1:-1, 2:, 1:-1] +
                Ak[:, :-1] * pad[:, :-2, 1:-1, 1:-1] + Ak[:, 1:] * pad[:, 2:, 1:-1, 1:-1])

    np_ = len(first) - 1

    def dot(a, c):
        return torch.zeros(np_, dtype=torch.float64, device=dev).index_add_(0, prob, (a * c).flatten(1).sum(1))

    over = lambda a, c: torch.where(c != 0, a / torch.where(c != 0, c, 1.0), 0.0)
    each = lambda v: v[prob].view(-1, 1, 1, 1)
    x = torch.zeros_like(b)
    bb = dot(b, b)
    for _ in range(12):                                  # restarted from the true residual until it stands still
        r = b - apply(x)
        if bool((dot(r, r) <= 1e-29 * bb).all()):
            break
        r0, p = r.clone(), r.clone()
        rho, rr0 = dot(r0, r), dot(r, r)
        for _ in range(600):
            y = p / Aii
            v = apply(y)
            alpha = each(over(rho, dot(r0, v)))
            q = r - alpha * v
            z = q / Aii
            t = apply(z)
            omega = each(over(dot(t, q), dot(t, t)))
            x = x + alpha * y + omega * z
            r = q - omega * t
            rr = dot(r, r)
            if bool((rr <= torch.maximum(1e-16 * rr0, 1e-31 * bb)).all()):
                break
            new = dot(r0, r)
            beta = each(over(new, rho)) * torch.where(omega != 0, alpha / torch.where(omega != 0, omega, 1.0), 0.0)
            p = r + beta * (p - omega * v)
            rho = new
    return x


# ---- the learned correction ----------------------------------------------------

NET_LAYERS = [(8, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (64, 32), (32, 16), (16, 16), (16, 1)]
NET_PARAMS = sum(ci * co * 27 + co for ci, co in NET_LAYERS)


def _net_seed(seed):
    return 1 + seed % 1000


def _net_inputs(case, seed):
    g = np.random.Generator(np.random.PCG64(seed))
    shape = (case["n"], case["D"], case["H"], case["W"])
    x = g.standard_normal(shape + (8,), dtype=np.float32)
    return x, g.standard_normal(shape, dtype=np.float32)


def _exact_net(case, seed):
    dev = _device()
    net = lcc.LCC(seed=_net_seed(seed))
    p = torch.as_tensor(net.params(), device=dev).double().requires_grad_(case["mode"] == "gradient")
    net.close()
    layers, o = [], 0
    for ci, co in NET_LAYERS:
        layers.append((p[o:o + ci * co * 27].view(co, ci, 3, 3, 3), p[o + ci * co * 27:o + ci * co * 27 + co]))
        o += ci * co * 27 + co
    x, t = (torch.as_tensor(a, device=dev).double() for a in _net_inputs(case, seed))
    conv = lambda a, l: F.conv3d(a, layers[l][0], layers[l][1], padding=1)
    up = lambda a: F.interpolate(a, scale_factor=2, mode="nearest")
    with torch.backends.cudnn.flags(enabled=False), torch.set_grad_enabled(case["mode"] == "gradient"):
        a = x.permute(0, 4, 1, 2, 3).contiguous()
        s0 = conv(conv(a, 0).relu(), 1).relu()
        s1 = conv(conv(F.avg_pool3d(s0, 2), 2).relu(), 3).relu()
        s2 = conv(F.avg_pool3d(s1, 2), 4).relu()
        a = conv(F.avg_pool3d(s2, 2), 5).relu()
        a = conv(up(a) + s2, 6).relu()
        a = conv(up(a) + s1, 7).relu()
        a = conv(up(a) + s0, 8).relu()
        y = conv(a, 9)[:, 0]
        if case["mode"] == "forward":
            return {"y": y}
        loss = (y - t).square().mean()
        return {"loss": loss.detach(), "gradient": torch.autograd.grad(loss, p)[0]}
