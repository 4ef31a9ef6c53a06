"""The work that programs built on this engine have it do, case by case, for timing and for
comparing outputs: forward runs (one step graph per time step), the drop-in loop that calls
one hook per Domain method, single stiffness evaluations of a caller's field, batched sources
and the adjoint.

A case is a plain dict:

  drive       "run" (axg_run), "hooks" (the per-step hooks), "stiffness" (f = -K x of a caller's
              device field) or "adjoint" (checkpointed forward run and its adjoint sweep)
  mesh        "box" (Cartesian quads with the axis, a moment source and surface stations),
              "shell" (half annulus with a fluid layer, source and stations) or "block"
              (perturbed quads off the axis, uneven nr)
  precision   "fp32", "mixed" or "fp64"
  nx, nz      quads along s (theta on the shell) and z (solid layers of the shell; "fluid" more
              fluid layers below them)
  nr_lo, nr_hi  range of the Fourier order of the elements (box: nr_hi everywhere)
  rheology    "iso", "tiso" or "aniso" (21 Cij, in the RTZ frame on the shell)
  attenuation "none", "full" (SLS memory variables at 25 points) or "cg4" (at 4)
  three_d     moduli per azimuthal slice
  waves       independent sources advanced together
  steps       time steps of one pass
  absorbing   Clayton edges and a sponge (box)
  stations    receivers

Everything that does not depend on the inputs (mesh, moduli, masses) is built once per case and
process; the inputs are the wavefields, random with the amplitude falling as 1 / (1 + mode).
"""
import functools
import math

import numpy as np
import torch
import torch.utils.checkpoint

from axisem3d_b200 import meshgen
from axisem3d_b200.solver import Solver

DEV = "cuda"
AMP = 1e-3          # displacement amplitude of the initial wavefields (m)


def _case(name, drive, mesh, precision, nx, nz, nr_lo, nr_hi, rheology="iso", attenuation="none", three_d=False,
          waves=1, steps=1, fluid=0, absorbing=False, stations=0):
    c = dict(name=name, drive=drive, mesh=mesh, precision=precision, nx=nx, nz=nz, nr_lo=nr_lo, nr_hi=nr_hi,
             rheology=rheology, attenuation=attenuation, three_d=three_d, waves=waves, steps=steps, fluid=fluid,
             absorbing=absorbing, stations=stations)
    if name is None:
        del c["name"]
    return c


def listed():
    return [
        # the plain forward run at the size a reference CPU build runs: every step is a handful of
        # launches over 1600 small elements, the latency-bound end
        _case("box_run_fp32", "run", "box", "fp32", 40, 40, 5, 5, steps=100, stations=20),
        # the same engine behind the reference's own time loop: one call per Domain method, with
        # attenuation and absorbing edges, ragged grid
        _case("box_hooks_fp32", "hooks", "box", "fp32", 53, 31, 5, 5, attenuation="full", steps=25, absorbing=True,
              stations=20),
        # a global 1-D Earth model at a low order: axis, fluid layer, CG4 attenuation, many stations
        _case("globe_1d_cg4_fp32", "run", "shell", "fp32", 160, 36, 3, 5, attenuation="cg4", steps=50, fluid=4,
              stations=400),
        # 3-D transversely isotropic media with full SLS attenuation and uneven nr, in the three
        # precisions: the bulk of a regional 3-D run
        _case("block_3d_full_mixed", "run", "block", "mixed", 170, 140, 1, 64, "tiso", "full", True, steps=20),
        _case("block_3d_full_fp32", "run", "block", "fp32", 111, 83, 1, 64, "tiso", "full", True, steps=20),
        _case("block_3d_full_fp64", "run", "block", "fp64", 97, 89, 1, 64, "tiso", "full", True, steps=20),
        # the same mesh with 1-D moduli: stress and attenuation per Fourier mode
        _case("block_1d_full_mixed", "run", "block", "mixed", 160, 125, 1, 64, "tiso", "full", steps=20),
        # spherical shell with a random 3-D velocity field, high uneven nr, CG4, fluid layer
        _case("shell_3d_cg4_mixed", "run", "shell", "mixed", 150, 30, 3, 128, "iso", "cg4", True, steps=20, fluid=2,
              stations=20),
        # many sources on one 21-Cij mesh in one launch
        _case("shell_cij_batch_mixed", "run", "shell", "mixed", 60, 12, 3, 100, "aniso", "none", True, waves=16,
              steps=20, fluid=1),
        # waveform inversion: forward with checkpoints, then the adjoint sweep
        _case("box_adjoint_fp64", "adjoint", "box", "fp64", 100, 100, 9, 9, steps=24, stations=50),
        # one stiffness evaluation of a caller's field (a host program with its own time scheme)
        _case("stiffness_3d_fp32", "stiffness", "block", "fp32", 90, 70, 1, 64, "tiso", "none", True),
        # the same for few elements of very high order (near-source 3-D structure)
        _case("stiffness_high_nr_fp32", "stiffness", "block", "fp32", 14, 11, 120, 250, "iso", "none", True),
    ]


def draw(rng):
    def logint(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["box", "box", "globe", "block3", "block3", "block1", "shell", "batch", "adjoint", "stiffness",
                       "high"])
    prec = rng.choice(["fp32", "mixed", "fp64"])
    if kind == "box":
        return _case(None, rng.choice(["run", "hooks"]), "box", prec, logint(9, 80), logint(9, 80), 5,
                     rng.choice([3, 4, 5, 7, 8]), attenuation=rng.choice(["none", "full"]), steps=rng.choice([25, 40, 60]),
                     absorbing=rng.random() < 0.5, stations=rng.randint(1, 60))
    if kind == "globe":
        return _case(None, "run", "shell", prec, logint(24, 160), logint(8, 36), 3, rng.choice([3, 5, 7]),
                     attenuation=rng.choice(["none", "full", "cg4"]), steps=20, fluid=rng.randint(1, 4),
                     stations=logint(5, 400))
    if kind in ("block3", "block1"):
        return _case(None, "run", "block", prec, logint(12, 110), logint(12, 80), 1, rng.choice([9, 23, 40, 64, 72]),
                     rng.choice(["iso", "tiso"]), rng.choice(["none", "full", "full"]), kind == "block3", steps=20)
    if kind == "shell":
        return _case(None, "run", "shell", prec, logint(24, 110), logint(6, 24), 3, rng.choice([48, 100, 128]), "iso",
                     rng.choice(["cg4", "full", "none"]), True, steps=20, fluid=rng.randint(1, 3), stations=rng.randint(1, 40))
    if kind == "batch":
        return _case(None, "run", "shell", rng.choice(["fp32", "mixed"]), logint(16, 60), logint(4, 12), 3,
                     rng.choice([24, 64, 100]), "aniso", "none", True, waves=rng.randint(2, 16), steps=20, fluid=1)
    if kind == "adjoint":
        return _case(None, "adjoint", "box", "fp64", logint(12, 100), logint(12, 100), 9, rng.choice([5, 7, 9, 13]),
                     steps=rng.choice([13, 17, 24]), stations=rng.randint(2, 50))
    if kind == "stiffness":
        return _case(None, "stiffness", "block", rng.choice(["fp32", "fp64"]), logint(9, 90), logint(9, 70), 1,
                     rng.choice([5, 17, 33, 64, 90]), rng.choice(["iso", "tiso", "aniso"]), "none", rng.random() < 0.7)
    prec = rng.choice(["fp32", "fp64"])
    top = 250 if prec == "fp32" else 130        # the largest order whose modes one block's shared memory holds, about
    return _case(None, "stiffness", "block", prec, logint(3, 14), logint(3, 11), rng.randint(70, 100),
                 rng.randint(101, top), "iso", "none", True)


# ------------------------------------------------------------------ models ---
@functools.lru_cache(maxsize=6)
def _model(mesh, nx, nz, nr_lo, nr_hi, rheology, attenuation, three_d, waves, fluid, absorbing, stations):
    if mesh == "box":
        m = meshgen.cartesian_model(nx=nx, nz=nz, nr=nr_hi, nstations=max(stations, 1), nr_aware_dt=True,
                                    attenuation=dict(meshgen.default_sls(3), qkappa=57823.0, qmu=300.0)
                                    if attenuation == "full" else None, absorbing=absorbing)
        m.st_interval = 10
    elif mesh == "shell":
        m = meshgen.spherical_model(n_theta=nx, n_solid_layers=nz, n_fluid_layers=fluid, nr_min=nr_lo, nr_max=nr_hi,
                                    three_d=three_d, attenuation=None if attenuation == "none" else attenuation,
                                    rheology=rheology, nstations=max(stations, 1))
        m.st_interval = 10
        if waves > 1:
            m = meshgen.ensemble_model(m, nsrc=waves)
    else:
        m = meshgen.microbench_model(n_elem=nx * nz, nr_min=nr_lo, nr_max=nr_hi, rheology=rheology, aspect=nx / nz,
                                     attenuation=None if attenuation == "none" else attenuation, is3d=three_d)
    return m


def _of(case):
    return _model(*(case[k] for k in ("mesh", "nx", "nz", "nr_lo", "nr_hi", "rheology", "attenuation", "three_d", "waves",
                                      "fluid", "absorbing", "stations")))


def _modes(nr):
    """(owning point, mode) of every complex value of a field's modes."""
    nu = np.asarray(nr, np.int64) // 2 + 1
    pt = np.repeat(np.arange(len(nu)), nu)
    return pt, np.arange(len(pt)) - np.repeat(np.cumsum(nu) - nu, nu)


def _wave(case, m, seed, solid=True):
    """A random wavefield [waves][modes][components] that obeys the conditions on the axis and on
    the zeroth and Nyquist modes."""
    nr = np.asarray(m.sp_nr if solid else m.fp_nr)
    pt, al = _modes(nr)
    g = torch.Generator(DEV).manual_seed(int(seed) * 2 + int(solid))
    al_t = torch.from_numpy(al).to(DEV)
    u = torch.randn((case["waves"], len(al), 3 if solid else 1, 2), generator=g, device=DEV, dtype=torch.float64)
    u *= AMP / (1.0 + al_t)[None, :, None, None]
    nyq = torch.from_numpy((nr[pt] % 2 == 0) & (al == nr[pt] // 2)).to(DEV)
    u[:, (al_t == 0) | nyq, :, 1] = 0
    ax = m.sp_axial if solid else m.fp_axial
    if ax is not None and len(ax):
        on = torch.from_numpy(np.asarray(ax)[pt] != 0).to(DEV)
        if solid:
            u[:, on, :2] = 0
            u[:, on & (al_t > 0)] = 0
        else:
            u[:, on & (al_t > 0)] = 0
    return torch.view_as_complex(u)


def prepare(case, seed):
    m = _of(case)
    if case["drive"] == "stiffness":
        s = Solver(m, case["precision"])
        stream = torch.cuda.Stream()
        s.set_stream(stream.cuda_stream)
        x = _wave(case, m, seed)[0].to(torch.complex128 if case["precision"] == "fp64" else torch.complex64)
        x = torch.view_as_real(x).contiguous()
        f = torch.zeros_like(x)
        torch.cuda.current_stream().synchronize()
        return {"case": case, "solver": s, "stream": stream, "x": x, "f": f}
    s = Solver(m, case["precision"])
    u = _wave(case, m, seed)
    s.set_field(u.cpu().numpy().ravel(), "displ")
    v = _wave(case, m, seed + 7919) * (0.05 / m.dt)
    s.set_field(v.cpu().numpy().ravel(), "veloc")
    st = {"case": case, "solver": s}
    if case["drive"] != "adjoint":
        n = s.field_raw_bytes("displ")
        st["displ"] = torch.empty(n // (4 if case["precision"] == "fp32" else 8), pin_memory=True,
                                  dtype=torch.float32 if case["precision"] == "fp32" else torch.float64)
        st["bytes"] = n
    return st


def run(state):
    case, s = state["case"], state["solver"]
    n = case["steps"]
    if case["drive"] == "stiffness":
        with torch.cuda.stream(state["stream"]):
            state["f"].zero_()
        s.compute_stiffness_noalloc(state["x"].data_ptr(), state["f"].data_ptr())
        return state["f"]
    if case["drive"] == "adjoint":
        s.forward_checkpointed(n, max(1, (n + 1) // 2))
        seis = s.seismograms()
        g = s.adjoint(seis)
        return {"seismograms": seis, "moduli": g["moduli"], "mass": g["mass"], "displ0": g["displ0"],
                "veloc0": g["veloc0"]}
    if case["drive"] == "hooks":
        t0 = s.step if "t" not in state else state["t"]
        for t in range(t0, t0 + n):
            s.apply_sources(t)
            s.compute_stiffness()
            s.apply_bc_before_assembly()
            s.record_stations(t)
            s.apply_bc_after_assembly()
            s.stiff_to_accel()
            s.newmark_update()
        state["t"] = t0 + n
    else:
        s.run(n)
    s.get_field_raw(state["displ"].data_ptr(), state["bytes"], "displ")
    out = {"displ": state["displ"]}
    if case["stations"] and case["drive"] == "run":
        out["seismograms"] = s.seismograms()
    return out


def work(case):
    m = _of(case)
    s = 8 if case["precision"] == "fp64" else 4
    d = 4 if case["precision"] == "fp32" else 8       # displacement, velocity and SLS state
    nmod = {"iso": 2, "tiso": 5, "aniso": 21}[case["rheology"]]
    npa = {"none": 0, "full": 25, "cg4": 4}[case["attenuation"]]
    nr = np.asarray(m.se_nr, np.float64)
    nu = np.floor(nr / 2) + 1
    ns = nr if case["three_d"] else np.ones_like(nr)
    slots = nr * npa if case["three_d"] else 2 * nu * npa
    w = case["waves"]
    b = len(nr) * (150 * s + 108) + float(np.sum(nmod * ns * 25 + 2 * ns * npa)) * s
    b += w * float(np.sum(2 * (m.nsls + 1) * 6 * slots)) * d
    f = w * float(np.sum(nu)) * 25 * 600
    if case["three_d"]:
        f += w * float(np.sum(2 * 150 * 2.5 * nr * np.log2(np.maximum(nr, 2)) + 25 * nr * {2: 16, 5: 22, 21: 72}[nmod]))
        f += w * float(np.sum(nr * npa * (m.nsls * 24 + 14)))
    else:
        f += w * float(np.sum(nu)) * (25 * 2 * {2: 16, 5: 22, 21: 72}[nmod] + 2 * npa * (m.nsls * 24 + 14))
    modes = w * float(np.sum(np.asarray(m.sp_nr) // 2 + 1)) * 3
    if len(m.fe_nr):
        fu = float(np.sum(np.asarray(m.fe_nr) // 2 + 1))
        b += len(m.fe_nr) * (175 * s + 108)
        f += w * fu * 25 * 160
        modes += w * float(np.sum(np.asarray(m.fp_nr) // 2 + 1))
    if case["drive"] == "stiffness":
        return {"bytes": b + modes * 2 * 2 * s, "flops": f}
    # per step: displacement, velocity and acceleration read and written
    per = b + modes * (4 * 2 * d + 2 * 2 * s)
    n = case["steps"]
    if case["drive"] == "adjoint":
        # the forward run, its recomputation and the reverse steps (two wavefields each)
        return {"bytes": per * n * 4, "flops": f * n * 4}
    return {"bytes": per * n + modes * 2 * d, "flops": f * n + modes * 20 * n}


def tolerance(case):
    # about four times what two runs of the same inputs (the atomic adds in another order) differ by
    # after a few hundred steps, which is also about what either is off the 64-bit result
    if case["precision"] == "fp64":
        return {"rel": 1e-12, "max": 1e-10}
    if case["drive"] == "stiffness":
        return {"rel": 1e-6, "max": 1e-4}
    return {"rel": 1e-5, "max": 1e-3}


# ------------------------------------------------- the step in 64 bits, plain torch ---
def _derivative_table(nodes):
    """G[j, i] = l_j'(x_i) of the Lagrange basis on the nodes."""
    n = len(nodes)
    G = np.zeros((n, n))
    for j in range(n):
        p = np.poly1d([1.0])
        for k in range(n):
            if k != j:
                p = p * np.poly1d([1.0, -nodes[k]]) * (1.0 / (nodes[j] - nodes[k]))
        G[j] = np.polyval(np.polyder(p), nodes)
    return np.round(G, 12)


class _Exact:
    """The time step on the model's operands in float64: elements of one nr at a time, every
    transform by torch.fft, scatter by index_add."""

    CG4 = [6, 8, 16, 18]

    def __init__(self, m):
        self.m, self.dev = m, DEV
        t = self.t
        leg = np.polynomial.legendre
        gll = np.concatenate([[-1.0], np.sort(leg.legroots(leg.legder([0, 0, 0, 0, 1])).real), [1.0]])
        # interior GLJ nodes: roots of the Jacobi polynomial P_3^(1,2) = 12 - 54 ... in powers of (x - 1) / 2
        jac = np.poly1d([0.0])
        for k in range(4):
            c = math.comb(3, k) * math.gamma(7 + k) / math.gamma(7) * math.gamma(5) / math.gamma(2 + k) / 6.0
            jac = jac + c * np.poly1d([0.5, -0.5]) ** k
        glj = np.concatenate([[-1.0], np.sort(jac.roots.real), [1.0]])
        self.Gl, self.Gj = t(_derivative_table(gll)), t(_derivative_table(glj))
        self.solid = self._points(m.sp_nr, m.sp_axial, None, m.sp_mass)
        self.alpha, self.beta, self.gamma = ([float(x) for x in a][: m.nsls] for a in
                                             (m.att_alpha, m.att_beta, m.att_gamma))
        nmods = np.array([2, 5, 21])[np.asarray(m.se_rheo)]
        self.groups = []
        is3d = np.zeros(len(m.se_nr), bool) if m.se_is3d is None else np.asarray(m.se_is3d) != 0
        for nr in np.unique(m.se_nr):
            e = np.nonzero(np.asarray(m.se_nr) == nr)[0]
            ns, nm = int(nr) if is3d[e[0]] else 1, int(nmods[e[0]])
            g = self._group(m, int(nr), e, m.se_pts, m.se_axial, m.se_geom, self.solid)
            at = np.asarray(m.se_mat_off)[e][:, None] + np.arange(nm * ns * 25)
            g["mod"] = t(np.asarray(m.se_moduli)[at].reshape(len(e), nm, ns, 25))
            g["is3d"], g["e"] = bool(is3d[e[0]]), e
            g["rtz"] = m.se_rtz is not None and bool(m.se_rtz[e[0]]) and nm != 2
            if g["rtz"]:
                g["theta"] = t(m.se_theta[e])
            g["att"] = 0 if m.se_att is None else int(m.se_att[e[0]])
            if g["att"]:
                npa = 25 if g["att"] == 1 else 4
                at = np.asarray(m.se_att_off)[e][:, None] + np.arange(2 * ns * npa)
                g["dm"] = t(np.asarray(m.se_att_moduli)[at].reshape(len(e), 2, ns, npa))
                shape = (len(e), 6, int(nr) if g["is3d"] else g["nu"], npa)
                g["ds"] = torch.zeros(shape, dtype=torch.float64 if g["is3d"] else torch.complex128, device=self.dev)
                g["mem"] = [torch.zeros_like(g["ds"]) for _ in range(m.nsls)]
            self.groups.append(g)
        self.fluid, self.fgroups = None, []
        if len(m.fe_nr):
            self.fluid = self._points(m.fp_nr, m.fp_axial, m.fp_surface, m.fp_mass)
            for nr in np.unique(m.fe_nr):
                e = np.nonzero(np.asarray(m.fe_nr) == nr)[0]
                g = self._group(m, int(nr), e, m.fe_pts, m.fe_axial, m.fe_geom, self.fluid)
                g["K"] = t(np.asarray(m.fe_moduli)[np.asarray(m.fe_mat_off)[e][:, None] + np.arange(25)])
                self.fgroups.append(g)

    def t(self, a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)

    def _points(self, nr, axial, surface, mass):
        nr = np.asarray(nr, np.int64)
        pt, al = _modes(nr)
        nu = nr // 2 + 1
        ax = np.zeros(len(nr), bool) if axial is None else np.asarray(axial) != 0
        sf = np.zeros(len(nr), bool) if surface is None else np.asarray(surface) != 0
        return {"nu": self.t(nu), "off": self.t(np.cumsum(nu) - nu), "pt": self.t(pt), "n": len(pt),
                "keep": self.t(~(ax[pt] & (al >= 1))), "ax0": self.t(ax[pt] & (al == 0)), "ax1": self.t(ax[pt] & (al == 1)),
                "wet": self.t(~sf[pt]), "nyq": self.t((nr[pt] % 2 == 0) & (al == nr[pt] // 2)),
                "mass": self.t(np.asarray(mass, np.float64))}

    def _group(self, m, nr, e, pts, axial, geom, P):
        p = self.t(np.asarray(pts, np.int64).reshape(-1, 25)[e])
        nu = nr // 2 + 1
        al = torch.arange(nu, device=self.dev)
        idx = P["off"][p][:, None, :] + al[None, :, None]
        ok = al[None, :, None] < P["nu"][p][:, None, :]
        ax = self.t(np.asarray(axial)[e] != 0)
        ge = self.t(np.asarray(geom).reshape(-1, 6, 25)[e])
        plain = ge[:, :5].reshape(-1, 5, 1, 1, 5, 5)
        return {"nr": nr, "nu": nu, "idx": torch.where(ok, idx, 0), "ok": ok, "ax": ax[:, None, None, None, None],
                "plain": plain, "int": (ge[:, :5] * ge[:, 5:6]).reshape(-1, 5, 1, 1, 5, 5),
                "Gx": torch.where(ax[:, None, None], self.Gj, self.Gl).to(torch.complex128),
                "ia": (1j * al)[None, :, None, None].to(torch.complex128)}

    # gradients and their transposes; u [n][nu][c][5][5]
    def _dsz(self, g, u, geo):
        X = torch.einsum("nki,nackj->nacij", g["Gx"], u)
        Y = torch.einsum("nacik,kj->nacij", u, self.Gl.to(torch.complex128))
        return X * geo[:, 3] + Y * geo[:, 2], X * geo[:, 1] + Y * geo[:, 0]

    def _over_s(self, g, A, geo):
        lim = self._dsz(g, A, geo)[0]
        row0 = torch.zeros((5, 1), dtype=torch.bool, device=self.dev)
        row0[0] = True
        return torch.where(g["ax"] & row0, lim, A * geo[:, 4])

    def _div(self, g, X, Y, A, geo):
        """sum_k G(i, k) X(k, j) + Y(i, k) G(j, k) less the transpose of A / s."""
        gl = self.Gl.to(torch.complex128)
        f = torch.einsum("nik,nackj->nacij", g["Gx"], X) + torch.einsum("nacik,jk->nacij", Y, gl) - A * geo[:, 4]
        a0 = A[..., :1, :]
        f = f - torch.where(g["ax"], g["Gx"][:, None, None, :, :1] * (a0 * geo[:, 3][..., :1, :]), 0)
        low = torch.einsum("nacik,jk->nacij", a0 * geo[:, 2][..., :1, :], gl)
        return f - torch.where(g["ax"], torch.nn.functional.pad(low, (0, 0, 0, 4)), 0)

    def _strain(self, g, u):
        geo, ia = g["plain"], g["ia"][..., None]
        dS, dZ = self._dsz(g, u, geo)
        A = torch.stack([ia[:, :, 0] * u[:, :, 0] - u[:, :, 1], ia[:, :, 0] * u[:, :, 1] + u[:, :, 0],
                         ia[:, :, 0] * u[:, :, 2]], 2)
        o = self._over_s(g, A, geo)
        return torch.stack([dS[:, :, 0], o[:, :, 1], dZ[:, :, 2], dZ[:, :, 1] + o[:, :, 2], dZ[:, :, 0] + dS[:, :, 2],
                            dS[:, :, 1] + o[:, :, 0]], 2)

    def _force(self, g, s, geo):
        """computeQuad of a stress [n][nu][6][5][5]."""
        ia = g["ia"]
        z, x = geo[:, 3], geo[:, 2]
        se, sx = geo[:, 1], geo[:, 0]
        a, b = s[:, :, [0, 5, 4]], s[:, :, [4, 3, 2]]
        A = torch.stack([ia * s[:, :, 5] - s[:, :, 1], ia * s[:, :, 1] + s[:, :, 5], ia * s[:, :, 3]], 2)
        return self._div(g, a * z + b * se, a * x + b * sx, A, geo)

    @staticmethod
    def _elastic(e, c):
        """Stress of strains e = [6 tensors] for moduli c = [nmod tensors]."""
        if len(c) == 2:
            tr = (e[0] + e[1] + e[2]) * c[0]
            return [tr + 2 * c[1] * e[k] for k in range(3)] + [c[1] * e[k] for k in range(3, 6)]
        if len(c) == 5:
            A, C, F, Lm, N = c
            h = A * (e[0] + e[1]) + F * e[2]
            return [h - 2 * N * e[1], h - 2 * N * e[0], F * (e[0] + e[1]) + C * e[2], Lm * e[3], Lm * e[4], N * e[5]]
        at = {}
        k = 0
        for i in range(6):
            for j in range(i, 6):
                at[i, j] = at[j, i] = c[k]
                k += 1
        return [sum(at[i, j] * e[j] for j in range(6)) for i in range(6)]

    def _turn(self, e, th, back):
        """Voigt strains to the RTZ frame, or stresses back: the rotation by theta in the s-z plane."""
        c, s = torch.cos(th), torch.sin(th)
        if not back:
            e0 = c * c * e[0] + s * s * e[2] - c * s * e[4]
            e2 = s * s * e[0] + c * c * e[2] + c * s * e[4]
            return [e0, e[1], e2, c * e[3] + s * e[5], (c * c - s * s) * e[4] + 2 * c * s * (e[0] - e[2]), c * e[5] - s * e[3]]
        e0 = c * c * e[0] + s * s * e[2] + 2 * c * s * e[4]
        e2 = s * s * e[0] + c * c * e[2] - 2 * c * s * e[4]
        return [e0, e[1], e2, c * e[3] - s * e[5], (c * c - s * s) * e[4] - c * s * (e[0] - e[2]), c * e[5] + s * e[3]]

    def _stress(self, g, eps, mod):
        n, nu = eps.shape[:2]
        e = [eps[:, :, k].reshape(n, nu, 25) for k in range(6)]
        if g["rtz"]:
            e = self._turn(e, g["theta"][:, None], False)
        nr = g["nr"]
        if g["is3d"]:
            x = torch.stack(e, 1)
            if nr % 2 == 0:
                x = torch.cat([x[:, :, :-1], 2 * x[:, :, -1:]], 2)
            x = torch.fft.irfft(x, nr, dim=2, norm="forward")
            e = [x[:, k] for k in range(6)]
        s = self._elastic(e, [mod[:, k] for k in range(mod.shape[1])])
        if g["att"]:
            q = list(range(25)) if g["att"] == 1 else self.CG4
            s = torch.stack(s, 1)
            new = torch.stack(self._elastic([x[..., q] for x in e], [g["dm"][:, 0], g["dm"][:, 1]]), 1)
            s = s.index_add(3, torch.tensor(q, device=self.dev), -sum(g["mem"]))
            g["mem"] = [a * mm + b * g["ds"] + c * new for mm, a, b, c in
                        zip(g["mem"], self.alpha, self.beta, self.gamma)]
            g["ds"] = new
            s = [s[:, k] for k in range(6)]
        if g["is3d"]:
            x = torch.fft.rfft(torch.stack(s, 1), dim=2, norm="forward")
            if nr % 2 == 0:
                x = torch.cat([x[:, :, :-1], 0.5 * x[:, :, -1:]], 2)
            s = [x[:, k] for k in range(6)]
        if g["rtz"]:
            s = self._turn(s, g["theta"][:, None], True)
        return torch.stack(s, 2).reshape(n, nu, 6, 5, 5)

    def stiffness(self, u, f, mods=None):
        for i, g in enumerate(self.groups):
            uu = torch.where(g["ok"][..., None], u[g["idx"]], 0).permute(0, 1, 3, 2)
            uu = uu.reshape(*uu.shape[:3], 5, 5)
            s = self._stress(g, self._strain(g, uu), g["mod"] if mods is None else mods[i])
            r = self._force(g, s, g["int"]).reshape(*uu.shape[:3], 25).permute(0, 1, 3, 2)
            f = f.index_add(0, g["idx"][g["ok"]], -r[g["ok"]])
        return f

    def stiffness_fluid(self, u, f):
        for g in self.fgroups:
            x = torch.where(g["ok"], u[g["idx"]], 0)[:, :, None].reshape(*g["ok"].shape[:2], 1, 5, 5)
            dS, dZ = self._dsz(g, x, g["plain"])
            o = self._over_s(g, g["ia"][..., None] * x, g["plain"])
            K = g["K"].reshape(-1, 1, 1, 5, 5)
            dS, dZ, o = dS * K, dZ * K, o * K
            geo = g["int"]
            r = self._div(g, dS * geo[:, 3] + dZ * geo[:, 1], dS * geo[:, 2] + dZ * geo[:, 0], g["ia"][..., None] * o, geo)
            f = f.index_add(0, g["idx"][g["ok"]], -r.reshape(g["ok"].shape)[g["ok"]])
        return f

    def sources(self, f, t, wave):
        m = self.m
        for i, e in enumerate(np.asarray(m.ms_elem)):
            if (0 if m.ms_wave is None else int(m.ms_wave[i])) != wave:
                continue
            st = m.ms_stf[i]
            k = st.decay_factor / st.half_duration
            x = k * (t - st.time_shift)
            val = k ** 3 * math.exp(-x * x) * (4 * x * x - 2) / math.sqrt(math.pi)      # second derivative
            for g in self.groups:
                at = np.nonzero(g["e"] == e)[0]
                if not len(at):
                    continue
                nu = min(g["nu"], int(m.ms_nu[i]))
                o = int(m.ms_pat_off[i])
                pat = self.t(np.asarray(m.ms_pattern)[o:o + nu * 150].reshape(1, nu, 6, 5, 5))
                one = {k2: (v[int(at[0])][None] if torch.is_tensor(v) and k2 in ("idx", "ok", "ax", "plain", "Gx") else v)
                       for k2, v in g.items()}
                one["ia"] = g["ia"][:, :nu]
                r = self._force(one, pat * val, one["plain"]).reshape(1, nu, 3, 25).permute(0, 1, 3, 2)
                ok = one["ok"][:, :nu]
                f = f.index_add(0, one["idx"][:, :nu][ok], r[ok])
        return f

    def record(self, u):
        m, out = self.m, []
        nr = np.asarray(m.se_nr)
        for i, e in enumerate(np.asarray(m.st_elem)):
            nu = int(nr[e]) // 2 + 1
            p = self.t(np.asarray(m.se_pts, np.int64).reshape(-1, 25)[e])
            al = torch.arange(nu, device=self.dev)
            ok = al[:, None] < self.solid["nu"][p]
            x = torch.where(ok[..., None], u[torch.where(ok, self.solid["off"][p] + al[:, None], 0)], 0)
            w = self.t(np.asarray(m.st_w[i]))
            ph = torch.exp(1j * al * float(m.st_phi[i])) * torch.where(al == 0, 1.0, 2.0)
            out.append((x * w[None, :, None] * ph[:, None, None]).sum((0, 1)).real)
        return torch.stack(out)

    def point(self, f, P, solid, inv):
        if solid:
            h = 0.5 * (f[:, 0] - 1j * f[:, 1])
            f0 = torch.where(P["ax1"], h, torch.where(P["ax0"] | ~P["keep"], 0, f[:, 0]))
            f1 = torch.where(P["ax1"], 1j * h, torch.where(P["ax0"] | ~P["keep"], 0, f[:, 1]))
            f = torch.stack([f0, f1, torch.where(P["keep"], f[:, 2], 0)], 1)
        else:
            f = torch.where(P["keep"] & P["wet"], f, 0)
        ny = P["nyq"][:, None] if solid else P["nyq"]
        f = torch.where(ny, torch.complex(f.real, torch.zeros_like(f.real)), f)
        iv = inv[P["pt"]]
        return f * (iv[:, None] if solid else iv)

    def step(self, S, k, wave=0, mods=None, inv=None):
        """One step from S = (u, v, a[, fluid u, v, a]); returns the next S."""
        m = self.m
        u, v, a = S[:3]
        f = self.sources(torch.zeros_like(u), m.t0 + k * m.dt, wave)
        f = self.stiffness(u, f, mods)
        if m.cl_solid is not None:
            c = m.cl_solid
            for i, p in enumerate(c["point"]):
                o, n = int(self.solid["off"][p]), int(self.solid["nu"][p])
                ct, st = math.cos(c["theta"][i]), math.sin(c["theta"][i])
                sa, pa = c["rho_vs"][i] * c["area"][i], c["rho_vp"][i] * c["area"][i]
                C = torch.tensor([[sa * ct * ct + pa * st * st, 0, (pa - sa) * ct * st], [0, sa, 0],
                                  [(pa - sa) * ct * st, 0, sa * st * st + pa * ct * ct]], device=self.dev,
                                 dtype=torch.complex128)
                f[o:o + n] -= v[o:o + n] @ C
        if self.fluid is not None:
            fu, fv, fa = S[3:]
            ff = self.stiffness_fluid(fu, torch.zeros_like(fu))
            s, q = (self.t(np.asarray(x, np.int64)) for x in (m.sf_solid, m.sf_fluid))
            nu = self.solid["nu"][s]
            rep = torch.repeat_interleave(torch.arange(len(s), device=self.dev), nu)
            al = torch.arange(len(rep), device=self.dev) - (torch.cumsum(nu, 0) - nu)[rep]
            si, qi = self.solid["off"][s][rep] + al, self.fluid["off"][q][rep] + al
            w = [self.t(np.asarray(x, np.float64))[rep] for x in (m.sf_nsu, m.sf_nzu, m.sf_nsa, m.sf_nza, m.sf_mass_fluid)]
            ff[qi] += u[si, 0] * w[0] + u[si, 2] * w[1]
            f[si, 0] -= ff[qi] * w[2] / w[4]
            f[si, 2] -= ff[qi] * w[3] / w[4]
        f = self.point(f, self.solid, True, 1 / self.solid["mass"] if inv is None else inv)
        if m.sponge_solid is not None:
            gm = torch.zeros(len(self.solid["nu"]), dtype=torch.float64, device=self.dev)
            gm[self.t(np.asarray(m.sponge_solid[0], np.int64))] = self.t(np.asarray(m.sponge_solid[1]))
            gm = gm[self.solid["pt"]][:, None]
            f = f - (2 * gm * v + gm * gm * u)
        h = m.dt
        v = v + 0.5 * h * (a + f)
        out = (u + h * v + 0.5 * h * h * f, v, f)
        if self.fluid is not None:
            ff = self.point(ff, self.fluid, False, 1 / self.fluid["mass"])
            fv = fv + 0.5 * h * (fa + ff)
            out += (fu + h * fv + 0.5 * h * h * ff, fv, ff)
        return out


def exact(case, seed):
    m = _of(case)
    x = _Exact(m)
    u = _wave(case, m, seed)
    if case["drive"] == "stiffness":
        if case["precision"] == "fp32":
            u = u.to(torch.complex64).to(torch.complex128)
        f = x.stiffness(u[0], torch.zeros_like(u[0]))
        return torch.view_as_real(f)
    v = _wave(case, m, seed + 7919) * (0.05 / m.dt)
    if case["precision"] == "fp32":
        u, v = u.to(torch.complex64).to(torch.complex128), v.to(torch.complex64).to(torch.complex128)
    n, every = case["steps"], int(m.st_interval)
    if case["drive"] == "adjoint":
        return _exact_adjoint(x, m, u[0], v[0], n, every)
    ends, seis = [], []
    for w in range(case["waves"]):
        S = (u[w], v[w], torch.zeros_like(u[w]))
        if x.fluid is not None:
            z = torch.zeros(x.fluid["n"], dtype=torch.complex128, device=DEV)
            S += (z, z, z)
        for k in range(n):
            if case["stations"] and k % every == 0:
                seis.append(x.record(S[0]))
            S = x.step(S, k, w)
        ends.append(S[0])
    out = {"displ": torch.view_as_real(torch.stack(ends)).reshape(-1)}
    if case["stations"] and case["drive"] == "run":
        out["seismograms"] = torch.stack(seis)
    return out


def _exact_adjoint(x, m, u, v, n, every):
    """Gradients of the sum of squares / 2 of the seismograms by automatic differentiation, one
    recomputed step at a time."""
    mods = [g["mod"].clone().requires_grad_() for g in x.groups]
    mass = x.solid["mass"].clone().requires_grad_()
    u, v = u.clone().requires_grad_(), v.clone().requires_grad_()

    def advance(k, a, b, c, mass, *mods):
        return x.step((a, b, c), k, 0, mods, 1 / mass)

    S, seis = (u, v, torch.zeros_like(u)), []
    for k in range(n):
        if k % every == 0:
            seis.append(x.record(S[0]))
        S = torch.utils.checkpoint.checkpoint(advance, k, *S, mass, *mods, use_reentrant=False)
    seis = torch.stack(seis)
    (0.5 * (seis ** 2).sum()).backward()
    gm = torch.zeros((len(m.se_nr), mods[0].shape[1], 25), dtype=torch.float64, device=DEV)
    for g, md in zip(x.groups, mods):
        gm[torch.from_numpy(g["e"]).to(DEV)] = md.grad[:, :, 0]
    flat = lambda z: torch.view_as_real(z.resolve_conj()).reshape(-1)  # noqa: E731
    return {"seismograms": seis.detach(), "moduli": gm, "mass": mass.grad, "displ0": flat(u.grad), "veloc0": flat(v.grad)}
