"""The molecular-dynamics work that a user has this library do, as measurable cases.

Every case is a stretch of an MD run through the library's C ABI: `steps` iterations of the
reference's loop (integrator, charge spreading, field solve, forces, integrator) on one
prepared system, then the outputs that a program writes at its output stride (positions,
velocities, forces, energies) and, where `restart` says so, the potential of the restart
file. `driver` says how the program steps: "loop" makes the reference's own sequence of
calls once per step (the drop-in use), "md_step" hands the steps to solver_md_step, and
"batch" advances a set of replicas together with mzb_batch_step.

A case is a dict of plain values:

  method, precond, precision   the field solve (precision 0: the reference's FP64
                               algorithms, 1: FP32 multigrid with FP64 refinement, 2: the
                               same multigrid in FP64)
  n_ions, n_grid, density      a NaCl melt (Tosi-Fumi, Lennard-Jones or soft-core pairs) on
                               an n_grid^3 grid; "pb" cases are a solute of n_ions in a
                               box of implicit water instead
  tol, cas, pot, integrator    solver tolerance, charge assignment, pair potential, and
                               VERLET without or OVRVO with its thermostat
  steps, driver, restart       the stretch that one pass runs and what it writes

listed() holds the sizes of the library's own configurations (250 / 64^3, 2000 / 128^3,
16000 / 256^3, the served stream's 64^3 .. 256^3 grids, the 32-ion solute at 128^3 and the
uneven replica set) and some that no tuned path was made for; draw() spreads over the
ranges between them.
"""
import math
import os

import numpy as np
import torch

os.environ.setdefault("MZB_QUIET", "1")

from maze_poisson_b200 import systems  # noqa: E402
from maze_poisson_b200.c_api import CAPI  # noqa: E402
from maze_poisson_b200.md import MDRun, gamma_au  # noqa: E402

DT_FS, TEMPERATURE, FRICTION_PER_PS = 1.0, 1200.0, 1.0
PB_TEMPERATURE, PB_EPS_S, PB_EPS_INT = 300.0, 78.4, 1.0
BOX_PER_POINT_ANG = 0.3125  # the solute's box: 40 A at 128^3
BASE = dict(family="melt", method="LCG", precond="NONE", precision=0, n_ions=250, n_grid=64, density=1.379,
            tol=1e-10, cas="CIC", pot="TF", integrator="VERLET", steps=10, driver="loop", restart=True)


def _case(**changes):
    return dict(BASE, **changes)


def listed():
    return [
        # the reference's smallest configuration, driven as its Python drives it: CG field
        # solve at its default tolerance, one call at a time
        _case(name="lcg_250_64", tol=1e-7),
        # the smallest system as a served job: launches and latency are what it costs
        _case(name="refine_250_64", precision=1, steps=20, driver="md_step"),
        # MaZe with the Jacobi preconditioner and the thermostat on a grid that is not a
        # multiple of 16 points
        _case(name="maze_lcg_1024_100", method="MAZE-LCG", precond="JACOBI", n_ions=1024, n_grid=100, tol=1e-8,
              integrator="OVRVO", steps=5),
        # the reference's MaZe multigrid at its middle configuration
        _case(name="maze_multigrid_2000_128", method="MAZE-MULTIGRID", n_ions=2000, n_grid=128, density=1.329,
              integrator="OVRVO", steps=5),
        # a served job of middle size on a grid that is no power of two
        _case(name="refine_4394_192", precision=1, n_ions=4394, n_grid=192, integrator="OVRVO", driver="md_step"),
        # the headline configuration in the mixed-precision form
        _case(name="refine_16000_256", precision=1, n_ions=16000, n_grid=256, steps=20, driver="md_step"),
        # the headline configuration with the reference's FFT field solve
        _case(name="fft_16000_256", method="FFT", n_ions=16000, n_grid=256, steps=20, driver="md_step"),
        # FFT on a 2^a 3^b grid, cubic splines and Lennard-Jones pairs, one call at a time
        _case(name="fft_spline_2662_144", method="FFT", n_ions=2662, n_grid=144, cas="SPL_CUBIC", pot="LJ"),
        # the headline configuration with the reference's CG: the longest step there is
        _case(name="lcg_16000_256", n_ions=16000, n_grid=256, steps=1, driver="md_step"),
        # a solute in implicit solvent, CG and multigrid, the latter smaller and off the
        # power of two
        _case(name="pb_maze_lcg_32_128", family="pb", method="MAZE-LCG", n_ions=32, n_grid=128, steps=2),
        _case(name="pb_multigrid_14_96", family="pb", method="MULTIGRID", n_ions=14, n_grid=96, steps=2),
        # many uneven replicas advanced together
        _case(name="batch_32", family="batch", precision=1, n_ions=32, n_grid=0, density=0.0, integrator="OVRVO",
              steps=6, driver="batch", restart=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _ions_for(rng, n_grid, density):
    """An even number of ions whose box has a spacing of 0.26 to 0.34 A on this grid."""
    box_cm = n_grid * rng.uniform(0.26, 0.34) * 1e-8
    pairs = density * box_cm ** 3 * systems.N_AVOGADRO / systems.NACL_MOLAR_MASS
    return 2 * max(8, int(round(pairs)))


def draw(rng):
    kind = rng.choice(["lcg", "multigrid", "refine", "refine", "fft", "pb", "batch"])
    density = round(rng.uniform(1.30, 1.40), 3)
    integrator = rng.choice(["VERLET", "OVRVO"])
    driver = rng.choice(["loop", "md_step"])
    if kind == "batch":
        return _case(family="batch", precision=1, n_ions=_log_int(rng, 4, 32), n_grid=0, density=0.0,
                     integrator=integrator, steps=rng.randint(3, 8), driver="batch", restart=False)
    if kind == "pb":
        n = 2 * _log_int(rng, 32, 64)
        return _case(family="pb", method=rng.choice(["LCG", "MAZE-LCG", "MULTIGRID", "MAZE-MULTIGRID"]), n_grid=n,
                     n_ions=max(4, 2 * int(round(16 * (n / 128) ** 3))), steps=rng.randint(1, 3), driver=driver)
    if kind == "lcg":
        n = 2 * _log_int(rng, 24, 96)
        method, precond = rng.choice([("LCG", "NONE"), ("MAZE-LCG", "NONE"), ("MAZE-LCG", "JACOBI")])
        return _case(method=method, precond=precond, n_grid=n, density=density, n_ions=_ions_for(rng, n, density),
                     tol=rng.choice([1e-7, 1e-8, 1e-10]), cas=rng.choice(["CIC", "CIC", "SPL_QUADR"]),
                     integrator=integrator, steps=rng.randint(1, 5 if n <= 128 else 2), driver=driver)
    if kind == "multigrid":
        n = 2 * _log_int(rng, 24, 72)
        return _case(method=rng.choice(["MULTIGRID", "MAZE-MULTIGRID"]), n_grid=n, density=density,
                     n_ions=_ions_for(rng, n, density), integrator=integrator, steps=rng.randint(2, 5), driver=driver)
    if kind == "fft":
        n = rng.choice([54, 64, 72, 96, 108, 128, 144, 162, 192, 216, 256])
        return _case(method="FFT", n_grid=n, density=density, n_ions=_ions_for(rng, n, density),
                     cas=rng.choice(["CIC", "SPL_QUADR", "SPL_CUBIC"]), pot=rng.choice(["TF", "LJ", "SC"]),
                     integrator=integrator, steps=rng.randint(4, 12), driver=driver)
    n = 16 * _log_int(rng, 4, 16)
    return _case(method=rng.choice(["LCG", "MAZE-LCG", "MULTIGRID", "MAZE-MULTIGRID"]),
                 precision=rng.choice([1, 1, 1, 2]), n_grid=n, density=density, n_ions=_ions_for(rng, n, density),
                 integrator=integrator, steps=rng.randint(4, 12), driver=driver)


# -- inputs ----------------------------------------------------------------------------

def _replicas(case, seed):
    """(system, pb settings or None) of each system of the case, made from the seed."""
    if case["family"] == "batch":
        sizes = systems.replica_set(case["n_ions"], seed=2026)
        return [(systems.make_melt(n, g, density=rho, T=TEMPERATURE, seed=(seed, r)), None)
                for r, (n, g, rho, _) in enumerate(sizes)]
    if case["family"] == "pb":
        s = systems.make_pb_system(case["n_ions"], case["n_grid"], BOX_PER_POINT_ANG * case["n_grid"],
                                   T=PB_TEMPERATURE, seed=seed)
        return [(s, systems.pb_settings(s, eps_s=PB_EPS_S))]
    s = systems.make_melt(case["n_ions"], case["n_grid"], density=case["density"], T=TEMPERATURE, seed=seed)
    if case["pot"] == "LJ":
        s.pot_params = systems.lj_params_au()
    elif case["pot"] == "SC":
        s.pot_params = systems.sc_params_au()
    return [(s, None)]


def _forces(case):
    names = ["pos", "vel", "fcs_elec", "fcs_noel", "fcs_tot"]
    return names + ["fcs_db", "fcs_ib", "fcs_np"] if case["family"] == "pb" else names


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


class _State:
    """The systems of one case, initialised and bootstrapped, and the caller's output
    buffers."""
    capi = None

    def __init__(self, case, seed):
        if _State.capi is None:
            _State.capi = CAPI()
            _State.capi.solver_initialize()
        self.case, self.handles, self.runs = case, [], []
        c = _State.capi
        pb = case["family"] == "pb"
        for system, settings in _replicas(case, seed):
            self.handles.append(c.mzb_system_create())
            run = MDRun(c, system, method=case["method"], precond=case["precond"], tol=case["tol"],
                        integrator=case["integrator"], thermostat=case["integrator"] == "OVRVO",
                        T=system.T, gamma_per_ps=FRICTION_PER_PS, dt_fs=DT_FS, eps_s=PB_EPS_S if pb else 1.0,
                        eps_int=PB_EPS_INT, precision=case["precision"], cas=case["cas"], pot=case["pot"],
                        pb=settings)
            c.solver_initialize()
            c.mzb_set_seed(seed)
            run.initialize()
            self.runs.append(run)
        self.ids = np.array(self.handles, dtype=np.int32)
        total = sum(r.sys.n_ions for r in self.runs)
        self.out = {name: _pinned(total, 3) for name in _forces(case)}
        self.out["kinetic"] = np.zeros(len(self.runs))
        if case["restart"]:
            n = case["n_grid"]
            self.out["field"] = _pinned(n, n, n)

    def __del__(self):
        for h in self.handles:
            _State.capi.mzb_system_destroy(h)


def prepare(case, seed):
    return _State(dict(case), int(seed))


def run(state):
    c, case, out = state.capi, state.case, state.out
    if case["driver"] == "batch":
        if c.mzb_batch_step(state.ids, len(state.ids), case["steps"]) < 0:
            raise RuntimeError("a field solve did not converge")
    else:
        c.mzb_system_select(state.handles[0])
        if case["driver"] == "md_step":
            res = c.solver_md_step(case["steps"])
        else:
            state.runs[0].run(case["steps"])
            res = state.runs[0].n_iters
        if res < 0:
            raise RuntimeError("a field solve did not converge")
    at = 0
    for r, (handle, md) in enumerate(zip(state.handles, state.runs)):
        if len(state.handles) > 1:
            c.mzb_system_select(handle)
        n = md.sys.n_ions
        for name in _forces(case):
            getattr(c, "get_" + name)(out[name][at:at + n])
        out["kinetic"][r] = c.get_kinetic_energy()
        at += n
    if case["restart"]:
        c.get_field(out["field"])
    if case["driver"] == "loop":
        return dict(out, potential=state.runs[0].potential_notelec)
    return out


# -- what a pass cannot do without -------------------------------------------------------

def work(case):
    """Per step: the potential read and written once (and its predecessor read, where the
    method extrapolates from it), the ions' state read and written once with their stencil
    values, and each pair inside half the box evaluated once; the outputs once per pass."""
    if case["family"] == "batch":
        sizes = [(n, g) for n, g, _, _ in systems.replica_set(case["n_ions"], seed=2026)]
    else:
        sizes = [(case["n_ions"], case["n_grid"])]
    nbytes = flops = 0.0
    for n_ions, n in sizes:
        fields = 3 if case["method"] not in ("LCG", "FFT") else 2
        if case["family"] == "pb":
            fields += 4
        stencil = 8 if case["cas"] == "CIC" else 64
        step = 8.0 * fields * n ** 3 + n_ions * 8.0 * (3 * 6 + 2 + 2 * stencil)
        nbytes += case["steps"] * step + n_ions * 8.0 * 15 + (8.0 * n ** 3 if case["restart"] else 0.0)
        pairs = n_ions * (n_ions - 1) / 2 * math.pi / 6
        flops += case["steps"] * (60.0 * pairs + 5.0 * n ** 3 * math.log2(max(n, 2) ** 3))
    return {"bytes": nbytes, "flops": flops}


# -- the same stretch in 64 bits, as plain torch gives it ----------------------------------

_DEV = "cuda" if torch.cuda.is_available() else "cpu"
_KB = systems.KB


def _t(a):
    return torch.as_tensor(np.asarray(a), dtype=torch.float64, device=_DEV)


class _Exact:
    """One system advanced step by step with the field solved to rounding: by FFT with the
    7-point stencil's eigenvalues (or the continuous wave numbers, for the FFT method), or
    by conjugate gradients for the Poisson-Boltzmann operator."""

    def __init__(self, case, system, pb, seed):
        s = self.s = system
        self.case, self.pb, self.seed = case, pb, seed
        self.n, self.L, self.h = s.n_grid, s.L, s.h
        self.pos, self.vel, self.mass, self.chg = _t(s.pos), _t(s.vel), _t(s.mass)[:, None], _t(s.charges)
        self.types = torch.as_tensor(s.types, dtype=torch.int64, device=_DEV)
        self.dt, self.calls = DT_FS / systems.T_AU_FS, 0
        self.thermostat = case["integrator"] == "OVRVO"
        gamma = gamma_au(FRICTION_PER_PS)
        self.c1 = math.exp(-gamma * self.dt) if self.thermostat else 1.0
        self.c2 = math.sqrt(2 / (gamma * self.dt) * math.tanh(0.5 * gamma * self.dt)) if self.thermostat else 1.0
        self.field = torch.zeros((self.n,) * 3, dtype=torch.float64, device=_DEV)
        self.out = {}
        if pb is None:
            self._green()
        self.forces()          # the bootstrap: the forces of the start, then one step
        self.step()

    # the spectral factor of the Poisson solve, applied to the charges
    def _green(self):
        n, L, h = self.n, self.L, self.h
        m = torch.fft.fftfreq(n, 1.0 / n, device=_DEV, dtype=torch.float64)
        k = torch.arange(n // 2 + 1, device=_DEV, dtype=torch.float64)
        if self.case["method"] == "FFT":
            f, r = (2 * math.pi * m / L) ** 2, (2 * math.pi * k / L) ** 2
            g = 4 * math.pi / h ** 3 / (f[:, None, None] + f[None, :, None] + r[None, None, :] + 1e-10)
        else:
            f, r = 2 * torch.cos(2 * math.pi * m / n), 2 * torch.cos(2 * math.pi * k / n)
            lam = f[:, None, None] + f[None, :, None] + r[None, None, :] - 6
            lam[0, 0, 0] = 1.0
            g = -4 * math.pi / h / lam
        g[0, 0, 0] = 0.0
        self.green = g

    def _stencil(self):
        """Flat grid indices and weights (N, points) of the charge assignment."""
        n, h, cas = self.n, self.h, self.case["cas"]
        cell = torch.floor(self.pos / h)
        offs = torch.arange(0, 2, device=_DEV) if cas == "CIC" else torch.arange(-1, 3, device=_DEV)
        at = cell[:, :, None] + offs
        x = (self.pos[:, :, None] / h - at).abs()
        if cas == "CIC":
            w = (1 - x).clamp(min=0)
        elif cas == "SPL_QUADR":
            w = torch.where(x < 0.5, 0.75 - x * x, torch.where(x < 1.5, 0.5 * (1.5 - x) ** 2, torch.zeros_like(x)))
        else:
            w = torch.where(x < 1, (4 - 6 * x ** 2 + 3 * x ** 3) / 6,
                            torch.where(x < 2, (2 - x) ** 3 / 6, torch.zeros_like(x)))
        at = torch.remainder(at, n).to(torch.int64)
        flat = (at[:, 0, :, None, None] * n + at[:, 1, None, :, None]) * n + at[:, 2, None, None, :]
        ws = w[:, 0, :, None, None] * w[:, 1, None, :, None] * w[:, 2, None, None, :]
        return flat.reshape(len(flat), -1), ws.reshape(len(ws), -1)

    def _solve(self, q):
        if self.pb is None:
            self.field = torch.fft.irfftn(torch.fft.rfftn(q) * self.green, s=q.shape)
            return
        self._coefficients()
        b = -4 * math.pi * q / self.h
        x = self.field
        r = b - self._pb_op(x)
        z = r / -self.diag
        p, rz, top = z, (r * z).sum(), b.norm()
        for it in range(20000):
            ap = self._pb_op(p)
            alpha = rz / (p * ap).sum()
            x = x + alpha * p
            r = r - alpha * ap
            if it % 25 == 24 and r.norm() <= 1e-15 * top:
                break
            z = r / -self.diag
            new = (r * z).sum()
            p, rz = z + (new / rz) * p, new
        self.field = x

    def _pb_op(self, u):
        out = -self.diag * u
        for axis, e in enumerate(self.eps):
            out += torch.roll(u, -1, axis) * e + torch.roll(u * e, 1, axis)
        return out

    def _box(self, p, extra):
        """Grid indices and offsets from the ion, per axis, of the box of ion p."""
        reach = int(math.floor((self.pb.radii[p] + self.pb.w) / self.h)) + extra
        at = torch.floor(self.pos[p] / self.h)[:, None] + torch.arange(-reach, reach + 1, device=_DEV)
        d = self.pos[p][:, None] - at * self.h
        g = torch.remainder(at, self.n).to(torch.int64)
        n, (x, y, z) = self.n, d
        flat = (g[0][:, None, None] * n + g[1][None, :, None]) * n + g[2][None, None, :]
        return flat.reshape(-1), [v.expand_as(flat).reshape(-1)
                                  for v in (x[:, None, None], y[None, :, None], z[None, None, :])]

    def _coefficients(self):
        n, h, pb = self.n, self.h, self.pb
        arrays = [torch.full((n ** 3,), PB_EPS_S - PB_EPS_INT, dtype=torch.float64, device=_DEV) for _ in range(3)]
        arrays.append(torch.full((n ** 3,), float(pb.kbar2), dtype=torch.float64, device=_DEV))
        for p in range(len(self.pos)):
            flat, d = self._box(p, 1)
            rs, w = float(pb.radii[p]), pb.w
            for axis, a in enumerate(arrays):
                r2 = sum((v - (h / 2 if k == axis else 0.0)) ** 2 for k, v in enumerate(d))
                t = r2.sqrt() - rs + w
                f = -t ** 3 / (4 * w ** 3) + 3 * t ** 2 / (4 * w ** 2)
                f = torch.where(r2 >= (rs + w) ** 2, torch.ones_like(f), torch.where(r2 > (rs - w) ** 2, f, 0.0 * f))
                a[flat] *= f
        self.eps = [(a + PB_EPS_INT).reshape(n, n, n) for a in arrays[:3]]
        self.k2 = arrays[3].reshape(n, n, n)
        self.diag = self.k2 + sum(e + torch.roll(e, 1, axis) for axis, e in enumerate(self.eps))

    def _pb_forces(self):
        pb, h = self.pb, self.h
        back = [torch.roll(e, 1, axis) for axis, e in enumerate(self.eps)]
        grad = [e - b for e, b in zip(self.eps, back)]
        norm = torch.sqrt(sum(g * g for g in grad)) / h
        inv = torch.where(norm > 0, 1 / norm, torch.zeros_like(norm))
        fw = [torch.roll(self.field, -1, axis).reshape(-1) for axis in range(3)]
        bw = [torch.roll(self.field, 1, axis).reshape(-1) for axis in range(3)]
        phi, k2, inv = self.field.reshape(-1), self.k2.reshape(-1), inv.reshape(-1)
        db, ib, nop = (torch.zeros_like(self.pos) for _ in range(3))
        for p in range(len(self.pos)):
            flat, d = self._box(p, 2)
            rs, w = float(pb.radii[p]), pb.w

            def shell(sep):
                r2 = sum(v * v for v in sep)
                inside = (r2 < (rs + w) ** 2) & (r2 > (rs - w) ** 2)
                r = r2.sqrt() + 1e-12
                t = r - rs + w
                ratio = (-3 / (4 * w ** 3) * t ** 2 + 3 / (2 * w ** 2) * t) / \
                    (-t ** 3 / (4 * w ** 3) + 3 * t ** 2 / (4 * w ** 2))
                return torch.where(inside, ratio, torch.zeros_like(ratio)), torch.stack([v / r for v in sep], 1)

            ratio, u = shell(d)
            pc = phi[flat]
            ib[p] = ((k2[flat] * pc * pc * ratio)[:, None] * u).sum(0)
            for axis in range(3):
                for sign, face, near in ((-1.0, back, bw), (1.0, self.eps, fw)):
                    ratio, u = shell([v - sign * h / 2 if k == axis else v for k, v in enumerate(d)])
                    a = (face[axis].reshape(-1)[flat] - PB_EPS_INT) * ratio
                    db[p] -= ((a * (near[axis][flat] - pc) * pc)[:, None] * u).sum(0)
                    nop[p] += sign * ((a * inv[flat] * grad[axis].reshape(-1)[flat])[:, None] * u).sum(0)
        scale = h / (8 * math.pi)
        return db * scale, ib * scale, nop * (-pb.gamma_np * h / (PB_EPS_S - PB_EPS_INT))

    def _pair_terms(self, r, types):
        """Shifted pair force and energy at separations r of type pairs `types`."""
        rc, pot, par = self.L / 2, self.case["pot"], self.s.pot_params

        def bare(r, c):
            if pot == "TF":
                a, b, c6, d8, sg = c
                e = a * torch.exp(b * (sg - r))
                return b * e - 6 * c6 / r ** 7 - 8 * d8 / r ** 9, e - c6 / r ** 6 - d8 / r ** 8
            if pot == "LJ":
                sg, ep = c
                x = (sg / r) ** 6
                return 4 * ep * (12 * x * x - 6 * x) / r, 4 * ep * (x * x - x)
            nu, dd, bb = par
            x = bb * (dd / r) ** nu
            return nu * x / r, x

        width = {"TF": 5, "LJ": 2, "SC": 0}[pot]
        table = _t(par[:4 * width]).reshape(4, width)
        ends = [bare(torch.full((), rc, dtype=torch.float64, device=_DEV), table[t]) for t in range(4)]
        al, vs = (torch.stack([torch.as_tensor(e[k]) for e in ends]) for k in (0, 1))
        f, v = bare(r, [table[:, k][types] for k in range(width)])
        return f - al[types], v - vs[types] + al[types] * (r - rc)

    def _pairs(self):
        n, L, rc = len(self.pos), self.L, self.L / 2
        force, energy = torch.zeros_like(self.pos), 0.0
        rows = max(1, 24_000_000 // n)
        for at in range(0, n, rows):
            i = torch.arange(at, min(n, at + rows), device=_DEV)
            d = self.pos[i][:, None, :] - self.pos[None, :, :]
            d -= L * torch.round(d / L)
            r = d.square().sum(-1).sqrt()
            near = (r <= rc) & (i[:, None] != torch.arange(n, device=_DEV)[None, :])
            r = torch.where(near, r, torch.full_like(r, rc))
            f, v = self._pair_terms(r, self.types[i][:, None] * 2 + self.types[None, :])
            f = torch.where(near, f / r, torch.zeros_like(f))
            force[i] = (f[:, :, None] * d).sum(1)
            energy += float(torch.where(near, v, torch.zeros_like(v)).sum()) / 2
        return force, energy

    def forces(self):
        n, h = self.n, self.h
        flat, w = self._stencil()
        wq = w * self.chg[:, None]
        q = torch.zeros(n ** 3, dtype=torch.float64, device=_DEV)
        q.index_add_(0, flat.reshape(-1), wq.reshape(-1))
        self._solve(q.reshape(n, n, n))
        elec = [(wq * ((torch.roll(self.field, 1, a) - torch.roll(self.field, -1, a)) / (2 * h)).reshape(-1)[flat]).sum(1)
                for a in range(3)]
        o = self.out
        o["fcs_elec"] = torch.stack(elec, 1)
        o["fcs_noel"], o["potential"] = self._pairs()
        o["fcs_tot"] = o["fcs_elec"] + o["fcs_noel"]
        if self.pb is not None:
            o["fcs_db"], o["fcs_ib"], o["fcs_np"] = self._pb_forces()
            o["fcs_tot"] = o["fcs_tot"] + o["fcs_db"] + o["fcs_ib"] + o["fcs_np"]

    def _noise(self):
        """The thermostat's normals: Philox4x32-10 (Salmon et al., SC 2011) with counter
        (ion, draw, call) and the seed as key, by Box-Muller."""
        n = len(self.pos)
        ion, low = np.arange(n, dtype=np.uint64), np.uint64(0xFFFFFFFF)
        z = np.empty((n, 3))
        for k in (0, 1):
            c = [ion, np.full(n, k, np.uint64), np.full(n, self.calls, np.uint64), np.zeros(n, np.uint64)]
            key = [np.uint64(self.seed & 0xFFFFFFFF), np.uint64(self.seed >> 32)]
            for _ in range(10):
                p, q = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
                c = [(q >> np.uint64(32)) ^ c[1] ^ key[0], q & low, (p >> np.uint64(32)) ^ c[3] ^ key[1], p & low]
                key = [(key[0] + np.uint64(0x9E3779B9)) & low, (key[1] + np.uint64(0xBB67AE85)) & low]
            u, v = ((((c[a] << np.uint64(32)) | c[a + 1]) >> np.uint64(11)).astype(np.float64) + 0.5
                    for a in (0, 2))
            u, v = u * 2.0 ** -53, v * 2.0 ** -53
            z[:, 2 * k] = np.sqrt(-2 * np.log(u)) * np.cos(2 * np.pi * v)
            if k == 0:
                z[:, 1] = np.sqrt(-2 * np.log(u)) * np.sin(2 * np.pi * v)
        self.calls += 1
        return _t(z)

    def _bath(self):
        if self.thermostat:
            spread = torch.sqrt((1 - self.c1) * _KB * self.s.T / self.mass)
            self.vel = self.vel * math.sqrt(self.c1) + spread * self._noise()

    def step(self):
        self._bath()
        self.vel = self.vel + 0.5 * self.dt * self.c2 * self.out["fcs_tot"] / self.mass
        x = self.pos + self.c2 * self.dt * self.vel
        x = torch.where(x < 0, x + self.L, x)
        self.pos = torch.where(x >= self.L, x - self.L, x)
        self.forces()
        self.vel = self.vel + 0.5 * self.dt * self.c2 * self.out["fcs_tot"] / self.mass
        self._bath()

    def outputs(self):
        kinetic = 0.5 * (self.mass[:, 0] * self.vel.square().sum(1)).sum()
        return dict(self.out, pos=self.pos, vel=self.vel, kinetic=kinetic.reshape(1), field=self.field)


def exact(case, seed):
    """run()'s first answer for these inputs. The reference's multigrid leaves the
    potential's mean open, so its field has no one value; forces do not depend on it."""
    found = []
    for system, pb in _replicas(case, int(seed)):
        e = _Exact(case, system, pb, int(seed))
        for _ in range(case["steps"]):
            e.step()
        found.append(e.outputs())
    out = {name: torch.cat([f[name] for f in found]) for name in _forces(case) + ["kinetic"]}
    if case["restart"]:
        open_mean = case["family"] == "melt" and case["precision"] == 0 and "MULTIGRID" in case["method"]
        out["field"] = None if open_mean else found[0]["field"]
    if case["driver"] == "loop":
        out["potential"] = found[0]["potential"]
    return out
