"""The work that a user of this framework has it do, as cases that can be timed.

A case is one pass through the public entry points with the inputs in the
user's hands: advance a given state by some steps and take the result back
(`advance`), the reference driver's own loop with its per-step accessors
(`driver`), a batch of independent runs (`ensemble`), and the derivatives of
a run (`gradient`, `tangent`).  Mesh levels, solvers, precisions, parameters
and step sizes are those of the repository's workloads (hex(3) ... hex(9),
quad(3) ... quad(8); accretion on and off; steps that are and are not clipped by the
CFL bound).

`exact` evaluates the same runs in 64 bits with plain torch operations on the
mesh's geometric coefficients, which are inputs of the scheme.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "muscl-scheme-on-spherical-mesh-wip_gb300"))
import splash_gb300 as sg  # noqa: E402

GAM = 2 - 1 / (4 / 3)  # the 2-D index of a 4/3 gas
FP64, MIXED = "fp64", "mixed"
SOLVERS = {"hlle_p": sg.SOLVER_HLLE_P, "hllc": sg.SOLVER_HLLC, "hllcp": sg.SOLVER_HLLCPLUS, "hlle": sg.SOLVER_HLLE}


def listed():
    return [
        # the small plain run, driven as the reference's own main loop does it:
        # a step, the light curves and the stop check, step by step
        dict(name="driver_hex4_hllep_fp64", do="driver", mesh="hex", level=4, solver="hlle_p", precision=FP64,
             steps=10, dt=1e-3, start="blob", accretion=True, friction=True, rate=1e-2, tilt=0.2, omega=0.5),
        # the smallest mesh in use, mixed precision: launches and their latency
        dict(name="hex3_hllc_mixed", do="advance", mesh="hex", level=3, solver="hllc", precision=MIXED,
             steps=20, dt=1e-3, start="blob", accretion=True, friction=False, rate=1e-2, tilt=0.2, omega=0.5),
        # a parameter study's usual mesh, between two outputs
        dict(name="hex5_hllcp_mixed", do="advance", mesh="hex", level=5, solver="hllcp", precision=MIXED,
             steps=50, dt=5e-4, start="noise", accretion=True, friction=True, rate=1e-2, tilt=0.2, omega=0.5),
        # the accreting mid-size run, between two outputs
        dict(name="hex7_hllcp_mixed", do="advance", mesh="hex", level=7, solver="hllcp", precision=MIXED,
             steps=25, dt=2e-4, start="noise", accretion=True, friction=True, rate=1e-2, tilt=0.2, omega=0.5),
        # the same run coupled to a host code that holds the state: one step a call
        dict(name="hex7_hllcp_mixed_coupled", do="advance", mesh="hex", level=7, solver="hllcp", precision=MIXED,
             steps=1, dt=2e-4, start="noise", accretion=True, friction=True, rate=1e-2, tilt=0.2, omega=0.5),
        # the same run in the reference's own precision
        dict(name="hex7_hllcp_fp64", do="advance", mesh="hex", level=7, solver="hllcp", precision=FP64,
             steps=4, dt=2e-4, start="noise", accretion=True, friction=True, rate=1e-2, tilt=0.2, omega=0.5),
        # the large shear layer, every step clipped by the CFL bound
        dict(name="hex9_hllcp_mixed_shear", do="advance", mesh="hex", level=9, solver="hllcp", precision=MIXED,
             steps=8, dt=1e-2, start="shear", accretion=False, friction=True, rate=0.0, tilt=0.0, omega=0.0),
        # a shear layer on the quad sphere in full precision
        dict(name="quad8_hllc_fp64_shear", do="advance", mesh="quad", level=8, solver="hllc", precision=FP64,
             steps=3, dt=1e-2, start="shear", accretion=False, friction=True, rate=0.0, tilt=0.0, omega=0.0),
        # the isothermal solver in full precision
        dict(name="quad7_hlle_fp64", do="advance", mesh="quad", level=7, solver="hlle", precision=FP64,
             steps=8, dt=1e-4, start="shear", accretion=False, friction=True, rate=0.0, tilt=0.0, omega=0.0),
        # many small runs at once, each with its own parameters and CFL step
        dict(name="ensemble_48", do="ensemble", members=48, plan=3, low=3, high=7, steps=25, dt=1.0),
        # the gradient of a run with respect to its state and parameters
        dict(name="gradient_hex5_hllc", do="gradient", mesh="hex", level=5, solver="hllc", precision=FP64,
             steps=20, dt=5e-4, start="rough", accretion=True, friction=True, rate=1e-2, tilt=0.1, omega=0.5, keep=10),
        # the directional derivative of a run
        dict(name="tangent_hex5_hllc", do="tangent", mesh="hex", level=5, solver="hllc", precision=FP64,
             steps=20, dt=5e-4, start="rough", accretion=True, friction=True, rate=1e-2, tilt=0.1, omega=0.5, keep=10),
    ]


def draw(rng):
    do = rng.choice(["advance", "advance", "advance", "driver", "ensemble", "gradient", "tangent"])
    if do == "ensemble":
        low = rng.randint(3, 5)
        return dict(do=do, members=rng.randint(3, 60), plan=rng.randint(0, 999), low=low, high=low + rng.randint(0, 2), steps=rng.randint(3, 25),
                    dt=rng.choice([1.0, 5e-4, 1e-3]))
    mesh = rng.choice(["hex", "hex", "quad"])
    derive = do in ("gradient", "tangent")
    precision = FP64 if derive else rng.choice([FP64, MIXED])
    level = rng.randint(3, 6 if derive else 7 if do == "driver" else 8)
    solver = rng.choice(["hlle_p", "hllc", "hllcp"] if do != "advance" else ["hlle_p", "hllc", "hllcp", "hlle"])
    accretion = solver != "hlle" and rng.random() < 0.7
    most = {8: 6, 7: 12, 6: 20}.get(level, 50) if precision == FP64 else 50
    case = dict(do=do, mesh=mesh, level=level, solver=solver, precision=precision,
                steps=int(round(math.exp(rng.uniform(0, math.log(most))))),
                dt=10 ** rng.uniform(-4, -2), start="rough" if derive else rng.choice(["blob", "noise", "shear", "rough"]),
                accretion=accretion, friction=rng.random() < 0.7 or derive,
                rate=10 ** rng.uniform(-4, -1.5) if accretion else 0.0, tilt=rng.uniform(0.05, 1.5) if accretion else 0.0,
                omega=rng.uniform(0.05, 0.6) if accretion else 0.0)
    if derive:
        case["keep"] = rng.randint(1, 12)
    return case


# ---- inputs -----------------------------------------------------------
def mesh_of(case):
    return sg.icosphere_hex(case["level"]) if case["mesh"] == "hex" else sg.quad_sphere(case["level"])


def device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def start_state(kind, centres, seed):
    """(Sigma, l, E) per face, in 64 bits on the host: a rotating blob, quiet noise, an equatorial shear layer, or a
    shear layer with noise in every field (nowhere uniform, so that it has derivatives)."""
    g = torch.Generator().manual_seed(int(seed))
    r = torch.as_tensor(centres).to(device())
    n = r.shape[0]

    def noise(*shape):
        return (2 * torch.rand(*shape, generator=g, dtype=torch.float64) - 1).to(r.device)

    def swirl(speed):
        phi = torch.stack([-r[:, 1], r[:, 0], torch.zeros_like(r[:, 0])], 1)
        return speed[:, None] * phi / phi.norm(dim=1, keepdim=True).clamp_min(1e-300)

    if kind == "noise":
        sigma, pi, v = 1 + 1e-3 * noise(n), 1 + 1e-3 * noise(n), torch.zeros_like(r)
    elif kind == "blob":
        c = torch.randn(3, generator=g, dtype=torch.float64).to(r.device)
        sigma = 1 + 0.2 * torch.exp(-((r - c / c.norm()) ** 2).sum(1) / 0.05)
        pi, v = sigma**GAM, torch.linalg.cross(torch.tensor([0.0, 0.0, 0.3], dtype=r.dtype, device=r.device).expand_as(r), r)
        v = v + 1e-3 * noise(n, 3)
    else:
        k = 6 * torch.randn(8, 3, generator=g, dtype=torch.float64).to(r.device)
        wave = torch.cos(r @ k.T + k.sum(1)).sum(1) / 8
        sigma = 1 + 1e-2 * wave
        pi, v = sigma**GAM, swirl(0.5 * torch.tanh(torch.asin(r[:, 2].clamp(-1, 1)) / 0.05))
        if kind == "rough":
            sigma, pi, v = sigma * (1 + 1e-3 * noise(n)), pi * (1 + 1e-3 * noise(n)), v + 1e-3 * noise(n, 3)
    v = v - (v * r).sum(1, keepdim=True) * r
    ell = sigma[:, None] * torch.linalg.cross(r, v)
    e = pi / (GAM - 1) + sigma * (v * v).sum(1) / 2
    return torch.cat([sigma[:, None], ell, e[:, None]], 1).cpu().numpy()


def params_of(case):
    return sg.SolverParams(accretion_rate=case["rate"], e_acc=0.5, omega_acc_abs=case["omega"], tilt_angle=case["tilt"],
                           acc_width=0.1, alpha=1e-6, friction_on=case["friction"])


def host(n, dim):
    """A page-locked host array, as a code that exchanges states with the GPU holds them."""
    a = torch.empty(n, dim, dtype=torch.float64)
    return (a.pin_memory() if torch.cuda.is_available() else a).numpy()


def draws_of(case):
    """The members' meshes, solvers and parameters: the plan of the study, whatever states it starts from."""
    return sg.workloads.ensemble_draws(case["members"], seed=case["plan"], levels=tuple(range(case["low"], case["high"] + 1)))


def member_start(d, centres, seed):
    u = start_state("noise", centres, 1000 * int(seed) + d["index"])
    return np.ascontiguousarray(u[:, :4]) if d["dim"] == 4 else u


def rest(n, dim):
    """The state a solver is created with before its geometry is known: uniform and at rest."""
    u = np.zeros((n, dim))
    u[:, 0] = 1
    if dim == 5:
        u[:, 4] = 1 / (GAM - 1)
    return u


def theta_of(case):
    return np.array([case["rate"], case["tilt"], case["omega"]])


def prepare(case, seed):
    if case["do"] == "ensemble":
        centres, members = {}, []
        for d in draws_of(case):
            if d["level"] not in centres:
                centres[d["level"]] = sg.Geometry(sg.icosphere_hex(d["level"])).unit_face_centers()
            members.append(dict(mesh=sg.icosphere_hex(d["level"]), U_in=member_start(d, centres[d["level"]], seed), gam=GAM,
                                omega_ns=0.0, accretion_on=True, params=sg.SolverParams(**d["params"]),
                                solver=sg.SOLVER_HLLE if d["dim"] == 4 else sg.SOLVER_HLLCPLUS))
        return dict(case=case, ensemble=sg.Ensemble(members))
    mesh, dim = mesh_of(case), 4 if case["solver"] == "hlle" else 5
    n = sg.n_faces_of(mesh)
    solver = sg.Solver(mesh, rest(n, dim), dim, GAM, 0.0, case["accretion"], params=params_of(case),
                       solver=SOLVERS[case["solver"]], precision=sg.PREC_MIXED if case["precision"] == MIXED else sg.PREC_FP64)
    centres, area = solver.face_geometry()
    state = dict(case=case, solver=solver, U=host(n, dim), out=host(n, dim))
    state["U"][:] = start_state(case["start"], centres, seed)[:, :dim]
    if case["do"] in ("gradient", "tangent"):
        state["adjoint"] = sg.Adjoint(solver, checkpoint_every=case["keep"])
        rng = np.random.default_rng(seed)
        state["target"] = 1 + 0.05 * rng.standard_normal(n)
        state["dU"] = rng.standard_normal((n, 5)) * np.abs(state["U"]).max(axis=0)
        state["dtheta"] = rng.standard_normal(3) * theta_of(case)
    return state


def run(state):
    case = state["case"]
    if case["do"] == "ensemble":
        e = state["ensemble"]
        e.do_steps(case["steps"], case["dt"])
        return [e.get_state(i) for i in range(case["members"])]
    s = state["solver"]
    if case["do"] == "advance":
        return s.do_steps_host(state["U"], case["steps"], case["dt"], state["out"])
    if case["do"] == "driver":
        s.set_state(state["U"])
        curves, stops = [], []
        for _ in range(case["steps"]):
            s.do_step(case["dt"])
            curves.append(s.get_light_curves())
            stops.append(s.get_stop_check())  # latched: a log keeps it, the run goes on
        return {"state": s.get_state(state["out"]), "light_curves": np.array(curves), "stops": np.array(stops, dtype=np.int32)}
    a = state["adjoint"]
    if case["do"] == "gradient":
        loss, gU, gtheta = a.run(state["U"], theta_of(case), case["steps"], case["dt"], state["target"])
        return {"loss": loss, "dU": gU, "dtheta": gtheta}
    U, dU = a.tlm(state["U"], theta_of(case), state["dU"], state["dtheta"], case["steps"], case["dt"])
    return {"state": U, "derivative": dU}


def work(case):
    """Per stage the mesh's coefficients and the states once each (slots, interior edges, faces), per step the conserved
    state in and out; operations of the scheme's formulas, counting a transcendental as one."""
    if case["do"] == "ensemble":
        lv = np.arange(case["low"], case["high"] + 1)
        w = 2.0 ** -(lv - lv.min())
        f, slots, dim, word = case["members"] * float((10 * 4.0**lv + 2) @ (w / w.sum())), 6.0, 4.5, 4
    else:
        f = float(sg.n_faces_of(mesh_of(case)))
        slots, dim, word = (6.0 if case["mesh"] == "hex" else 4.0), (4 if case["solver"] == "hlle" else 5), 4 if case["precision"] == MIXED else 8
    stage = slots * (16 + 7 * word) + slots / 2 * 11 * word + 5 * 8 + 2 * dim * word
    flops = slots * (60 + 22 * dim) + slots / 2 * (40 * dim) + 100
    step_b, step_f = 2 * stage + 2 * dim * 8, 2 * flops
    many = {"gradient": 3.0, "tangent": 2.0}.get(case["do"], 1.0)  # forward, recomputation and reverse; values and tangents
    ends = 2 * dim * 8
    return {"bytes": f * (many * case["steps"] * step_b + ends), "flops": f * many * case["steps"] * step_f}


# ---- the scheme in 64 bits --------------------------------------------
class Scheme:
    """The MUSCL step on one mesh, as plain torch operations in 64 bits."""

    _made: dict = {}

    @classmethod
    def of(cls, mesh):
        key = (mesh.kind, mesh.level)
        if key not in cls._made:
            cls._made.clear() if mesh.level > 7 else None
            cls._made[key] = cls(mesh)
        return cls._made[key]

    def __init__(self, mesh):
        g = sg.Geometry(mesh)

        def dev(a):
            return torch.as_tensor(a).to(device())

        off = dev(g["face_off"]).long()
        self.n, self.count = g.n_faces, off[1:] - off[:-1]
        self.face = torch.repeat_interleave(torch.arange(self.n, device=off.device), self.count)
        nbr = dev(g["nbr_edge"]).long()
        key, back = self.face * self.n + nbr, nbr * self.n + self.face
        order = torch.argsort(key)
        self.reverse = order[torch.searchsorted(key[order], back)]
        va = dev(g["face_vtx"]).long()
        nxt = torch.arange(len(va), device=va.device) + 1
        last = off[1:] - 1
        nxt[last] = off[:-1]
        x = dev(g["vertices"])
        a, b = x[va], x[va[nxt]]
        ec = (a + b) / 2
        self.ec = ec / ec.norm(dim=1, keepdim=True)
        self.en = dev(g["edge_normals"])
        self.nxr = torch.linalg.cross(self.en, self.ec)
        self.area = dev(g["area"])
        chord = (a - b).norm(dim=1)
        ua, ub = a / a.norm(dim=1, keepdim=True), b / b.norm(dim=1, keepdim=True)
        arc = 2 * torch.asin(((ua - ub).norm(dim=1) / 2).clamp(max=1))
        self.arc_a = arc / self.area[self.face]
        self.coef = g.round_diff * chord / self.area[self.face]
        self.sp, self.sm = dev(g["ff_plus"]).long(), dev(g["ff_minus"]).long()
        self.bp, self.bm = dev(g["beta_plus"]), dev(g["beta_minus"])
        self.hp, self.hm, self.dist = dev(g["h_plus"]), dev(g["h_minus"]), dev(g["bm_dist"])
        self.twon = (2 * self.count[self.face]).double()
        fc = dev(g["face_centers"])
        self.centre = fc / fc.norm(dim=1, keepdim=True)
        self.h0 = g.h0

    def accretion(self, rate, tilt):
        sig = 0.1 / 2.355
        z = self.centre[:, 2]
        bell = torch.exp(-((torch.acos(z) - math.pi / 2) ** 2) / (2 * sig**2)) / math.sqrt(2 * math.pi * sig**2)
        coeff = (self.area * bell).sum() / (4 * math.pi)
        x = self.centre[:, 1] * torch.sin(tilt) + z * torch.cos(tilt)
        return rate / coeff / math.sqrt(2 * math.pi * sig**2) * torch.exp(-((torch.acos(x) - math.pi / 2) ** 2) / (2 * sig**2))


def hi(a, b):
    return torch.where(a < b, b, a)


def lo(a, b):
    return torch.where(b < a, b, a)


def dot(a, b):
    return (a * b).sum(-1)


def cross(a, b):
    return torch.linalg.cross(a, b)


class Run:
    """Steps of one run: the physics parameters on a Scheme."""

    def __init__(self, case, theta=None):
        self.m = Scheme.of(mesh_of(case))
        self.solver, self.on, self.friction = case["solver"], case["accretion"] and case["solver"] != "hlle", case["friction"]
        if theta is None:
            theta = torch.tensor(theta_of(case), dtype=torch.float64, device=self.m.area.device)
        self.rate, tilt, omega = theta[0], theta[1], theta[2]
        self.omega = torch.stack([torch.zeros_like(tilt), torch.sin(tilt), torch.cos(tilt)]) * omega
        self.profile = self.m.accretion(self.rate, tilt) if self.on else None
        self.mass = self.m.area.sum()  # of the uniform state that the solver is created with

    def pressure(self, u):
        l = cross(self.m.centre, u[:, 1:4])
        return hi(torch.full_like(u[:, 0], 1e-16), (u[:, 4] - dot(l, l) / u[:, 0] / 2) * (GAM - 1))

    def dt(self, u, dt0):
        m = self.m
        v = -cross(m.centre, u[:, 1:4]) / u[:, :1]
        speed = v.norm(dim=1)
        if self.solver == "hlle":
            fastest = speed.clamp(min=1.0).max()
            return min(dt0, 0.1 * m.h0 / float(fastest))
        p = self.pressure(u)
        fastest = torch.maximum(speed, torch.sqrt(GAM * p / u[:, 0])).max()
        g3 = 1 / (2 - GAM)
        rho = g3 / (2 * g3 - 1) * (0.217909 - speed**2) * u[:, 0] ** 2 / p
        extra = 0.01 * u[:, 0] / (1e-6 * rho * speed)
        extra = float(extra[~torch.isnan(extra)].min()) if bool((~torch.isnan(extra)).any()) else 1e20
        extra = 1e20 if extra < 0 else min(extra, 1e20)
        return min(dt0, 0.1 * m.h0 / float(fastest), extra)

    def source(self, w):
        m = self.m
        if not self.on:
            return torch.zeros_like(w)
        r, s, p = m.centre, w[:, 0], w[:, 4]
        v = -cross(r, w[:, 1:4]) / s[:, None]
        spin = cross(self.omega.expand_as(r), r)
        res0 = self.profile
        res_l = res0[:, None] * cross(r, spin)
        d = spin - v
        res_e = res0 * (0.5 + dot(d, d) / 2.0)
        v2 = dot(v, v)
        if not self.friction:
            loss = -(self.rate * 4 * math.pi) / self.mass * s
            res0 = res0 + loss
            res_l = res_l + loss[:, None] * cross(r, v)
            res_e = res_e + loss * (GAM / (GAM - 1) * p / s + v2 / 2.0)
        g_eff = 0.217909 - v2
        heat = 3.0 / 4 * 4.85e36 * g_eff * s  # below zero: not a number, and no derivative either
        root = torch.sqrt(torch.sqrt(torch.where(heat > 0, heat, torch.ones_like(heat))))
        c = torch.where(heat >= 0, 12.0 / 5 * 1.6e-13 * s / p * root * (heat > 0), torch.full_like(heat, math.nan))
        edge = -1 - 1 / (0.736194670678821 - 1)
        low = c <= edge
        safe = torch.where(low, torch.full_like(c, 2.0), c)
        beta = torch.where(low, 1 - 1 / (1 + torch.where(low, c, torch.ones_like(c))), 1 - (2 / safe) ** 4)
        beta = torch.where((beta < 1e-8) | torch.isnan(beta), torch.full_like(beta, 1e-8), beta)
        beta = torch.where(beta > 1 - 1e-8, torch.full_like(beta, 1 - 1e-8), beta)
        res_e = res_e - g_eff / 3.4e6 * (1 - beta)
        if self.friction:
            g3 = 1 / (2 - GAM)
            rho = g3 / (2 * g3 - 1) * g_eff * s * s / p
            dv = torch.sqrt(torch.where(v2 > 0, v2, torch.ones_like(v2))) * (v2 > 0)
            k = 1e-6 * rho * dv
            res_l = res_l + cross(r, -k[:, None] * v)
            res0 = res0 - k
            res_l = res_l - (k / s)[:, None] * w[:, 1:4]
            res_e = res_e - k * (v2 / 2.0 + p * GAM / ((GAM - 1) * s))
        return torch.cat([res0[:, None], res_l, res_e[:, None]], 1)

    def edges(self, w, dt):
        """The limited states at every slot's edge, (Sigma, l, Pi) or (Sigma, l)."""
        m = self.m
        here = w[m.face]
        up = m.bp[:, :1] * w[m.sp[:, 0]] + m.bp[:, 1:] * w[m.sp[:, 1]]
        um = m.bm[:, :1] * w[m.sm[:, 0]] + m.bm[:, 1:] * w[m.sm[:, 1]]
        pp, pm = (up - here) / m.hp[:, None], (here - um) / m.hm[:, None]
        flat = pp == 0
        r = pm / torch.where(flat, torch.ones_like(pp), pp)
        r = torch.where(flat, torch.where(pm == 0, torch.zeros_like(r), torch.sign(pm.detach()) * 1e300), r)
        v = -cross(m.ec, here[:, 1:4]) / here[:, :1]
        a = 1.0 if self.solver == "hlle" else torch.sqrt(GAM * here[:, 4] / here[:, 0])
        nu = ((a + dot(v, m.en)) * dt * m.arc_a)[:, None]
        one, zero = torch.ones_like(r), torch.zeros_like(r)
        eta_m, eta_p = (m.hm / m.dist)[:, None], (m.hp / m.dist)[:, None]
        if self.solver == "hlle":
            lim = hi(zero, hi(lo(one, eta_m * r * 2 / (m.twon[:, None] * nu)), lo(r, eta_m.expand_as(r))))
        else:
            sb = hi(zero, hi(lo(one, r * eta_m / (m.twon[:, None] * nu)), lo(r, eta_p.expand_as(r))))
            to = hi(zero, lo(sb, 1 + (1 + nu) / 3 * (r - 1)))
            mid, top = (r < 1) & (r > 0), r >= 1
            x = torch.where(mid, r, torch.full_like(r, 0.5))
            y = 4 * x * x * (1 - x) ** 0.1
            h = torch.where(mid, 2 / (1 + torch.exp(2 * y)), zero)
            z = torch.where(top & (r < 3), r, 1.5 * one) - 1
            h = torch.where(top, torch.where(r < 3, torch.tanh(10 * z**3) ** 6, one), h)
            lim = (1 - h) * to + h * sb
        lim = torch.where(flat & (pm == 0), zero, lim)
        return here + pp * lim * m.dist[:, None]

    def edge_side(self, u):
        m = self.m
        v = -cross(m.ec, u[:, 1:4]) / u[:, :1]
        return v, dot(v, m.en), hi(torch.full_like(u[:, 0], 1e-16), u[:, 4])

    def plain_flux(self, u, e, p, vn):
        return torch.cat([(u[:, 0] * vn)[:, None], u[:, 1:4] * vn[:, None] - self.m.nxr * p[:, None], ((e + p) * vn)[:, None]], 1)

    def flux(self, left):
        m = self.m
        right = left[m.reverse]
        if self.solver == "hlle":
            (vl, vr) = (dot(-cross(m.ec, u[:, 1:4]) / u[:, :1], m.en) for u in (left, right))
            sl, sr = (lo(vl, vr) - 1)[:, None], (hi(vl, vr) + 1)[:, None]
            fl, fr = (torch.cat([(u[:, 0] * n)[:, None], u[:, 1:4] * n[:, None] - m.nxr * u[:, :1], ], 1) for u, n in ((left, vl), (right, vr)))
            mid = (sr * fl - sl * fr + sr * sl * (right - left)) / (sr - sl)
            return torch.where(sl >= 0, fl, torch.where(sr > 0, mid, fr))
        (vl, nl, pl), (vr, nr, pr) = self.edge_side(left), self.edge_side(right)
        sl_, sr_ = left[:, 0], right[:, 0]
        el, er = (u[:, 4] / (GAM - 1) + u[:, 0] * dot(v, v) / 2 for u, v in ((left, vl), (right, vr)))
        ul, ur = torch.cat([left[:, :4], el[:, None]], 1), torch.cat([right[:, :4], er[:, None]], 1)
        al, ar = torch.sqrt(GAM * pl / sl_), torch.sqrt(GAM * pr / sr_)
        ps = hi(torch.zeros_like(pl), (pl + pr) / 2 - (nr - nl) * (sl_ + sr_) * (al + ar) / 8)

        def q(p):
            steep = ps > p
            return torch.where(steep, torch.sqrt(1 + (GAM + 1) / (2 * GAM) * (torch.where(steep, ps / p, torch.ones_like(p)) - 1)), torch.ones_like(p))

        SL, SR = nl - al * q(pl), nr + ar * q(pr)
        fl, fr = self.plain_flux(left, el, pl, nl), self.plain_flux(right, er, pr, nr)
        if self.solver == "hlle_p":
            a, b = SL[:, None], SR[:, None]
            return torch.where(a >= 0, fl, torch.where(b > 0, (b * fl - a * fr + a * b * (ur - ul)) / (b - a), fr))
        ml, mr = sl_ * (SL - nl), sr_ * (SR - nr)
        S = (pr - pl + nl * ml - nr * mr) / (ml - mr)
        plr = (pl + pr + ml * (S - nl) + mr * (S - nr)) / 2
        isl = S >= 0
        sk = torch.where(isl, SL, SR)
        uk, fk = torch.where(isl[:, None], ul, ur), torch.where(isl[:, None], fl, fr)
        d = torch.cat([torch.zeros_like(S)[:, None], -m.nxr, S[:, None]], 1)
        f = (S[:, None] * (sk[:, None] * uk - fk) + (sk * plr)[:, None] * d) / (sk - S)[:, None]
        if self.solver == "hllcp":
            M = hi(vl.norm(dim=1) / al, vr.norm(dim=1) / ar).clamp(max=1.0)
            turn = ((nl - al > 0) & (nr - ar < 0)) | ((nl + al > 0) & (nr + ar < 0)) | ((nr - ar > 0) & (nl - al < 0)) | ((nr + ar > 0) & (nl + al < 0))
            fs = torch.where(turn, torch.ones_like(M), M * torch.sqrt(4 + (1 - M * M) ** 2) / (1 + M * M))
            g = 1 - torch.exp(M * torch.log(lo(pl / pr, pr / pl)))
            dn, dv = nr - nl, vr - vl
            vff = ((fs - 1) * dn)[:, None] * m.en + (sk / (sk - S) * g)[:, None] * (dv - dn[:, None] * m.en)
            w = ml * mr / (mr - ml)
            am = cross(m.ec, vff) * w[:, None]
            f = f + torch.cat([torch.zeros_like(S)[:, None], am, ((fs - 1) * dn * S * w)[:, None]], 1)
        return torch.where(SL[:, None] >= 0, fl, torch.where(SR[:, None] >= 0, f, fr))

    def stage(self, u0, w, dt, dt_here):
        m = self.m
        change = dt_here * self.source(w)
        f = self.flux(self.edges(w, dt)) * (m.coef * dt_here)[:, None]
        u = u0 + change.index_add(0, m.face, -f)
        floor = torch.cat([torch.where(u[:, :1] < 1e-8, torch.full_like(u[:, :1], 1e-8), u[:, :1]), u[:, 1:]], 1)
        return floor

    def face(self, u):
        return u if self.solver == "hlle" else torch.cat([u[:, :4], self.pressure(u)[:, None]], 1)

    def step(self, u, dt0):
        dt = self.dt(u.detach(), dt0)
        w1 = self.face(self.stage(u, self.face(u), dt, dt / 2))
        return self.stage(u, w1, dt, dt)

    def light_curves(self, u):
        r = self.m.centre
        c = torch.stack([r[:, 0], (r[:, 0] + r[:, 2]) / math.sqrt(2), r[:, 2], -r[:, 2]], 1).clamp(min=0)
        return (c * (self.pressure(u) * self.m.area)[:, None]).sum(0)


def exact(case, seed):
    if case["do"] == "ensemble":
        out, centres = [], {}
        for d in draws_of(case):
            p = d["params"]
            one = dict(mesh="hex", level=d["level"], solver="hlle" if d["dim"] == 4 else "hllcp", accretion=True, friction=True,
                       rate=p["accretion_rate"], tilt=p["tilt_angle"], omega=p["omega_acc_abs"])
            r = Run(one)
            u = torch.as_tensor(member_start(d, r.m.centre.cpu().numpy(), seed)).to(device())
            for _ in range(case["steps"]):
                u = r.step(u, case["dt"])
            out.append(u.cpu().numpy())
        return out
    dim = 4 if case["solver"] == "hlle" else 5
    m = Scheme.of(mesh_of(case))
    u = torch.as_tensor(np.ascontiguousarray(start_state(case["start"], m.centre.cpu().numpy(), seed)[:, :dim])).to(device())
    if case["do"] in ("gradient", "tangent"):
        rng = np.random.default_rng(seed)
        target = 1 + 0.05 * rng.standard_normal(m.n)
        dU = rng.standard_normal((m.n, 5)) * np.abs(u.cpu().numpy()).max(axis=0)
        dtheta = rng.standard_normal(3) * theta_of(case)
        theta = torch.tensor(theta_of(case), dtype=torch.float64, device=u.device)

        def final(u, theta):
            r = Run(case, theta)
            for _ in range(case["steps"]):
                u = r.step(u, case["dt"])
            return u

        u.requires_grad_(True)
        theta.requires_grad_(True)
        end = final(u, theta)
        if case["do"] == "gradient":
            loss = 0.5 * (m.area * (end[:, 0] - torch.as_tensor(target).to(u.device)) ** 2).sum()
            gu, gt = torch.autograd.grad(loss, [u, theta], allow_unused=True)
            return {"loss": float(loss.detach()), "dU": gu.cpu().numpy(), "dtheta": (torch.zeros(3) if gt is None else gt).cpu().numpy()}
        # J d as the derivative of y -> J^T y, which is linear in y
        y = torch.zeros_like(end, requires_grad=True)
        gu, gt = torch.autograd.grad(end, [u, theta], y, create_graph=True, allow_unused=True)
        along = (gu * torch.as_tensor(dU).to(u.device)).sum()
        if gt is not None:
            along = along + (gt * torch.as_tensor(dtheta).to(u.device)).sum()
        return {"state": end.detach().cpu().numpy(), "derivative": torch.autograd.grad(along, y)[0].detach().cpu().numpy()}
    r = Run(case)
    curves = []
    with torch.no_grad():
        for _ in range(case["steps"]):
            u = r.step(u, case["dt"])
            if case["do"] == "driver":
                curves.append(r.light_curves(u).cpu().numpy())
    if case["do"] == "driver":
        return {"state": u.cpu().numpy(), "light_curves": np.array(curves), "stops": None}
    return u.cpu().numpy()
