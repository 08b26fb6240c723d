"""The workloads whose speed matters to a user of diskdyn_gb300, at the sizes users run them.

Each case is one call (or one forward and backward) through `diskdyn_gb300.engine.Engine` or
`diskdyn_gb300.adjoint.trajectory_image`, on state that stays on the GPU between calls:

- step      an RK4 step of star, planets, gravitating planetesimals and grains;
- images    the images of all tracers at several wavelengths;
- sed       their spectral energy distribution over every table wavelength;
- collide   the pairs of grains closer than h;
- adjoint   an image after n steps and the gradients of a loss on it.

The systems are drawn on the GPU from the case's seed: a debris belt (a 1.5 Msun star, two
planets, planetesimals and grains at 120-140 AU), the same belt with a wide halo disk and a
clump of grains, the solar system with a Kuiper belt of tracers.  Grains follow a log-uniform
size distribution from 1 to 1,000 um with the beta of their size, so the smallest ones are
blown out of the system as the run goes on.
"""
import math

import numpy as np
import torch

from diskdyn_gb300 import abi
from diskdyn_gb300.adjoint import trajectory_image
from diskdyn_gb300.engine import STATE_FIELDS, DeviceState, Engine, make_phys, make_view

DEV = "cuda:0"
PREC = {"fp64": abi.DDX_PREC_FP64, "mixed": abi.DDX_PREC_MIXED, "compensated": abi.DDX_PREC_COMPENSATED}

# Units of the state: AU, yr, mass x 4 pi^2 in Msun.
AU, MSUN, RSUN, YEAR, PC = 1.49598e11, 1.98892e30, 695700000.0, 3.1556926e7, 3.08567758149137e16
LIGHT_AU, CSPEED, KBOLTZ, HPLANK = 63239.6717367, 299792458.0, 1.3806503e-23, 6.626068e-34
GRAV = 4.0 * math.pi ** 2
RHO = 2700.0
N_BINS, N_THETA, N_WAV, N_R = 64, 181, 200, 100
# Bytes of a body's state that a step reads (x y z vx vy vz m N id) and writes (x y z vx vy vz).
READ_B, WRITE_B = 68, 48


def listed():
    return [
        # The main run: a belt of 4,096 gravitating planetesimals and a million grains, one
        # mixed-precision step (what bench.py times).
        {"name": "belt_mixed", "kind": "step", "system": "belt", "n_plsml": 4096, "n_dust": 1048576,
         "precision": "mixed", "lorentz": False, "steps": 1},
        # A shard of the same run, or a quick look at the same belt: few grains, all planetesimals.
        {"name": "belt_mixed_shard", "kind": "step", "system": "belt", "n_plsml": 4096, "n_dust": 16384,
         "precision": "mixed", "lorentz": False, "steps": 1},
        # A run that needs errors near FP64's at several times its speed.
        {"name": "belt_compensated", "kind": "step", "system": "belt", "n_plsml": 4096, "n_dust": 131072,
         "precision": "compensated", "lorentz": False, "steps": 1},
        # The default precision on the same belt.
        {"name": "belt_fp64", "kind": "step", "system": "belt", "n_plsml": 4096, "n_dust": 65536,
         "precision": "fp64", "lorentz": False, "steps": 1},
        # A belt with a wide halo disk and a clump of grains; odd sizes.
        {"name": "halo_mixed", "kind": "step", "system": "halo", "n_plsml": 3001, "n_dust": 500003,
         "precision": "mixed", "lorentz": False, "steps": 1},
        # The largest system: 65,536 planetesimals, two million grains.
        {"name": "scale_mixed", "kind": "step", "system": "belt", "n_plsml": 65536, "n_dust": 2097152,
         "precision": "mixed", "lorentz": False, "steps": 1},
        # Few planetesimals, charged grains in the stellar field, several steps between outputs.
        {"name": "few_planetesimals_lorentz", "kind": "step", "system": "belt", "n_plsml": 256, "n_dust": 262144,
         "precision": "mixed", "lorentz": True, "steps": 5},
        # The smallest call: one FP64 step of the solar system and a Kuiper belt.
        {"name": "solar_fp64", "kind": "step", "system": "solar", "n_plsml": 0, "n_dust": 16384,
         "precision": "fp64", "lorentz": False, "steps": 1},
        # The image output of a run: ten wavelengths at 1024 x 1024.
        {"name": "images_mixed", "kind": "images", "n_dust": 2097152, "n_img": 10, "xsize": 1024, "ysize": 1024,
         "inc": 30.0, "pa": 0.0, "precision": "mixed"},
        # The SED output of a run in the default precision.
        {"name": "sed_fp64", "kind": "sed", "n_dust": 262144, "inc": 30.0, "pa": 0.0, "precision": "fp64"},
        # The collision pass of a step of the main run.
        {"name": "collide", "kind": "collide", "system": "belt", "n_dust": 1048576, "h": 0.1},
        # Fitting an image: the image after 50 steps and its gradients in planets and grains.
        {"name": "adjoint", "kind": "adjoint", "n_dust": 65536, "steps": 50, "ckpt": 25, "xsize": 256, "ysize": 256},
    ]


def _spread(rng, lo, hi):
    """A whole number log-uniform in [lo, hi], odd half of the time."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    n |= rng.randrange(2)
    return max(lo, min(hi, n))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["images", "sed", "collide", "adjoint"])
    if kind == "step":
        system = rng.choice(["belt", "belt", "halo", "solar"])
        precision = rng.choice(["mixed", "mixed", "compensated", "fp64"])
        c = {"kind": kind, "system": system, "precision": precision, "lorentz": rng.random() < 0.25, "steps": 1}
        if system == "solar":
            return dict(c, n_plsml=0, n_dust=_spread(rng, 1000, 524288), steps=rng.randint(1, 4))
        c["n_plsml"] = _spread(rng, 200, 20000 if precision == "mixed" else 5000)
        top = {"mixed": 1048576, "compensated": 262144, "fp64": 65536}[precision]
        return dict(c, n_dust=_spread(rng, 2000, top))
    if kind == "images":
        return {"kind": kind, "n_dust": _spread(rng, 20000, 2097152), "n_img": rng.randint(1, 12),
                "xsize": rng.randint(100, 1024), "ysize": rng.randint(100, 1024), "inc": rng.uniform(0.0, 90.0),
                "pa": rng.uniform(0.0, 180.0), "precision": rng.choice(["mixed", "fp64"])}
    if kind == "sed":
        return {"kind": kind, "n_dust": _spread(rng, 5000, 524288), "inc": rng.uniform(0.0, 90.0),
                "pa": rng.uniform(0.0, 180.0), "precision": rng.choice(["mixed", "fp64"])}
    if kind == "collide":
        return {"kind": kind, "system": rng.choice(["belt", "halo"]), "n_dust": _spread(rng, 10000, 2097152),
                "h": rng.uniform(0.03, 0.15)}
    steps = rng.randint(10, 50)
    return {"kind": kind, "n_dust": _spread(rng, 4000, 65536), "steps": steps, "ckpt": rng.randint(5, steps),
            "xsize": rng.randint(64, 256), "ysize": rng.randint(64, 256)}


# ---- inputs ------------------------------------------------------------------------------

class _Draw:
    """Uniform and normal FP64 numbers on the GPU from one seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(int(seed))

    def uniform(self, lo, hi, n):
        return lo + (hi - lo) * torch.rand(n, dtype=torch.float64, device=DEV, generator=self.g)

    def normal(self, sigma, n):
        return sigma * torch.randn(n, dtype=torch.float64, device=DEV, generator=self.g)

    def bins(self, n):
        return torch.randint(0, N_BINS, (n,), dtype=torch.int32, device=DEV, generator=self.g)


def _orbit(mu, a, e, inc, w, o, nu):
    """Positions and velocities (6, n) of orbital elements about a central mu = m (1 - beta)."""
    p = a * (1.0 - e * e)
    cn, sn = torch.cos(nu), torch.sin(nu)
    r, h = p / (1.0 + e * cn), torch.sqrt(mu / p)
    xe, ye, vxe, vye = r * cn, r * sn, -h * sn, h * (e + cn)
    co, so, cw, sw, ci, si = torch.cos(o), torch.sin(o), torch.cos(w), torch.sin(w), torch.cos(inc), torch.sin(inc)
    r11, r12 = co * cw - so * sw * ci, -co * sw - so * cw * ci
    r21, r22 = so * cw + co * sw * ci, -so * sw + co * cw * ci
    r31, r32 = sw * si, cw * si
    return torch.stack([xe * r11 + ye * r12, xe * r21 + ye * r22, xe * r31 + ye * r32,
                        vxe * r11 + vye * r12, vxe * r21 + vye * r22, vxe * r31 + vye * r32])


def _ring(d, mu, n, a0, a1, emax, imax_deg):
    return _orbit(mu, d.uniform(a0, a1, n), d.uniform(0.0, emax, n), d.uniform(0.0, math.radians(imax_deg), n),
                  *(d.uniform(0.0, 2 * math.pi, n) for _ in range(3)))


def _sizes():
    """Radii (m), beta, beta_sw and charge of the size bins of the belt's grains."""
    s = np.logspace(-6.0, -3.0, N_BINS)
    beta = (0.57 * (8.7 / 1.5) / (s * 1e6) / (RHO / 1000.0)).astype(np.float32)
    betasw = (3.0 * 2e-14 * 2 * MSUN * YEAR * 400e3 / 32.0 / math.pi / (1.5 * GRAV) / RHO / AU ** 3 / s).astype(np.float32)
    return s, beta, betasw, np.linspace(1e-3, 2e-3, N_BINS).astype(np.float32)


def _bodies(system, n_plsml, n_dust, seed):
    """(n_grav, dt, phys, tables, state): the state as a dict of GPU tensors, massive bodies first."""
    d = _Draw(seed)
    vsw = 400e3 * YEAR / AU
    if system == "solar":
        M = torch.tensor(1.0 * GRAV, dtype=torch.float64, device=DEV)
        pm = torch.logspace(math.log10(1.7e-7), math.log10(9.5e-4), 8, dtype=torch.float64, device=DEV) * GRAV
        a = torch.logspace(math.log10(0.4), math.log10(30.0), 8, dtype=torch.float64, device=DEV)
        planets = _orbit(M + pm, a, d.uniform(0.0, 0.1, 8), d.uniform(0.0, math.radians(3.0), 8),
                         *(d.uniform(0.0, 2 * math.pi, 8) for _ in range(3)))
        massive, mass, n_planets = planets, pm, 9
        dust = _ring(d, M, n_dust, 30.0, 50.0, 0.1, 5.0)
        ids, dmass = d.bins(n_dust), torch.zeros(n_dust, dtype=torch.float64, device=DEV)
        dt, phys = 0.05, dict(radQ=0, SWQ=0, Wz=0.0, Rstar=RSUN / AU, Rmin=0.05)
        z = np.zeros(N_BINS, np.float32)
        tables = dict(size=_sizes()[0], beta=z, betasw=z, q=z)
    else:
        M = torch.tensor(1.5 * GRAV, dtype=torch.float64, device=DEV)
        pm = torch.tensor([1e-3 * GRAV, 3e-4 * GRAV], dtype=torch.float64, device=DEV)
        zero = torch.zeros(2, dtype=torch.float64, device=DEV)
        planets = _orbit(M + pm, torch.tensor([20.0, 60.0], dtype=torch.float64, device=DEV), zero, zero, zero, zero,
                         d.uniform(0.0, 2 * math.pi, 2))
        mm = 10 ** d.uniform(-10.0, -8.0, n_plsml) * GRAV
        s, beta, betasw, q = _sizes()
        tables = dict(size=s, beta=beta, betasw=betasw, q=q)
        ids = d.bins(n_dust)
        b = torch.as_tensor(beta.astype(np.float64) + betasw, device=DEV)
        b = torch.where(b >= 0.5, torch.zeros_like(b), b)[ids.long()]      # blown-out grains start on the belt
        dmass = torch.as_tensor(4.0 / 3.0 * math.pi * RHO * s ** 3 / MSUN * GRAV, device=DEV)[ids.long()]
        mu = M * (1.0 - b)
        if system == "belt":
            plsml = _ring(d, M + mm, n_plsml, 120.0, 140.0, 0.05, 3.0)
            dust = _ring(d, mu, n_dust, 120.0, 140.0, 0.05, 3.0)
        else:
            k = int(0.7 * n_plsml)
            plsml = torch.cat([_ring(d, M + mm[:k], k, 130.0, 145.0, 0.05, 3.0),
                               _ring(d, M + mm[k:], n_plsml - k, 30.0, 200.0, 0.15, 8.0)], dim=1)
            k, c = int(0.7 * n_dust), int(0.05 * n_dust)
            belt = _ring(d, mu[:k], k, 130.0, 145.0, 0.05, 3.0)
            halo = _ring(d, mu[k:n_dust - c], n_dust - c - k, 30.0, 200.0, 0.15, 8.0)
            r = torch.sqrt(mu[n_dust - c:] / 140.0)
            clump = torch.stack([140.0 + d.normal(3.0, c), d.normal(3.0, c), d.normal(1.0, c),
                                 0.02 * r * d.normal(1.0, c), r, 0.02 * r * d.normal(1.0, c)])
            dust = torch.cat([belt, halo, clump], dim=1)
        massive, mass, n_planets = torch.cat([planets, plsml], dim=1), torch.cat([pm, mm]), 3
        dt = math.sqrt(120.0 ** 3 / 1.5) / 300.0
        phys = dict(radQ=1, SWQ=1, Wz=365.2422 / 25.0, Rstar=2.0 * RSUN / AU, Rmin=0.5)
    phys = dict(phys, FLQ=0, Bstar=0.0, rho=RHO, vsw_AUyr=vsw, n_planets=n_planets)
    # planets and star about their centre of mass, as a run starts
    star = torch.zeros(6, 1, dtype=torch.float64, device=DEV)
    lead, lm = torch.cat([star, massive[:, :n_planets - 1]], dim=1), torch.cat([M.reshape(1), mass[:n_planets - 1]])
    lead[:3] -= (lm * lead[:3]).sum(1, keepdim=True) / lm.sum()
    lead[3:, 0] = -(lm[1:] * lead[3:, 1:]).sum(1) / lm[0]
    rv = torch.cat([lead, massive[:, n_planets - 1:], dust], dim=1)
    n_grav = n_planets + n_plsml
    state = {f: rv[k].contiguous() for k, f in enumerate(("x", "y", "z", "vx", "vy", "vz"))}
    state["m"] = torch.cat([M.reshape(1), mass, dmass])
    state["N"] = torch.ones(n_grav + n_dust, dtype=torch.float64, device=DEV)
    state["id"] = torch.cat([torch.full((n_grav,), -1, dtype=torch.int32, device=DEV), ids])
    return n_grav, dt, phys, tables, state


def _step_inputs(c, seed):
    n_grav, dt, phys, tables, state = _bodies(c["system"], c["n_plsml"], c["n_dust"], seed)
    if c["lorentz"]:
        phys.update(FLQ=1, Bstar=3e-38)
        if c["system"] == "solar":      # charged grains have a mass
            phys["Bstar"], tables["q"] = 5e-20, _sizes()[3]
            state["m"][n_grav:] = 1e-30
    return n_grav, dt, phys, tables, state


def _optics(Rmax, L, Teff, Rstar):
    """Henyey-Greenstein phase functions with g from 0.1 to 0.9 over the bins, grey grains at
    the blackbody temperature of their distance, a blackbody star at 10 pc."""
    w = np.logspace(math.log10(0.5e-6), math.log10(850e-6), N_WAV)
    mu = np.arange(N_THETA) * 2.0 / (N_THETA - 1) - 1.0
    g = np.linspace(0.1, 0.9, N_BINS)[:, None]
    P = (1 - g ** 2) / (4 * math.pi * (1 + g ** 2 - 2 * g * mu[None, :]) ** 1.5)
    one = np.ones((N_BINS, N_WAV))
    with np.errstate(over="ignore"):
        star = 2 * HPLANK * CSPEED ** 2 / (w ** 5 * (np.exp(HPLANK * CSPEED / (w * KBOLTZ * Teff)) - 1))
    R = 0.1 * np.exp(math.log(Rmax / 0.1) * np.arange(N_R) / (N_R - 1.0))
    Td = np.repeat((278.3 * L ** 0.25 * R ** -0.5)[None, :], N_BINS, axis=0)
    return dict(w=w, influx=math.pi * star * (Rstar / (10 * PC)) ** 2, Qabs=one, Qsca=one,
                Qpfunc=np.repeat(P[:, :, None], N_WAV, axis=2), Td=Td, Rmin=0.1, Rmax=float(Rmax))


def _flux_inputs(c, seed):
    """The Kuiper belt with size bins and 1e15 grains per tracer, seen from 10 pc."""
    n_grav, _, _, tables, state = _bodies("solar", 0, c["n_dust"], seed)
    state["N"][n_grav:] = 1e15
    view = dict(dist=10 * PC, fov=120.0, PA=math.radians(c["pa"]), inc=math.radians(c["inc"]), longitude=0.0,
                xsize=c.get("xsize", 512), ysize=c.get("ysize", 512))
    wj = [int(round(k)) for k in np.linspace(0, N_WAV - 2, c.get("n_img", 1))]
    return n_grav, tables, state, _optics(100.0, 1.0, 5770.0, RSUN), view, wj


def _adjoint_inputs(c, seed):
    n_grav, dt, phys, tables, state = _bodies("belt", 0, c["n_dust"], seed)
    massive = torch.stack([state[f][:n_grav] for f in ("x", "y", "z", "vx", "vy", "vz", "m")], dim=1)
    dust = torch.stack([state[f][n_grav:] for f in ("x", "y", "z", "vx", "vy", "vz")], dim=1)
    N, ids = 1e20 * state["N"][n_grav:], state["id"][n_grav:].contiguous()
    view = dict(dist=10 * PC, fov=300.0, PA=0.0, inc=math.radians(30.0), longitude=0.0, xsize=c["xsize"], ysize=c["ysize"])
    opt = _optics(400.0, 8.7, 7500.0, 2.0 * RSUN)
    wj = [int(np.argmin(abs(opt["w"] - 1.25e-6))), int(np.argmin(abs(opt["w"] - 100e-6)))]
    target = _Draw(seed + 1).uniform(0.0, 1e-3, 2 * c["xsize"] * c["ysize"]).reshape(2, c["xsize"], c["ysize"])
    return massive, dust, N, ids, dt, phys, tables, view, opt, wj, target


# ---- the calls -----------------------------------------------------------------------------

def _engine(tables, opt=None):
    eng = Engine(0)
    eng.set_size_table(**tables)
    if opt is not None:
        eng.set_optics(opt["w"], opt["influx"], opt["Qabs"], opt["Qsca"], opt["Qpfunc"], opt["Td"], opt["Rmin"], opt["Rmax"])
    return eng


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        n_grav, dt, phys, tables, state = _step_inputs(case, seed)
        return dict(case=case, eng=_engine(tables), st=DeviceState(**state), n_grav=n_grav, dt=dt, phys=make_phys(**phys))
    if kind in ("images", "sed"):
        n_grav, tables, state, opt, view, wj = _flux_inputs(case, seed)
        return dict(case=case, eng=_engine(tables, opt), st=DeviceState(**state), n_grav=n_grav, view=make_view(**view), wj=wj)
    if kind == "collide":
        n_grav, _, _, tables, state = _bodies(case["system"], 64, case["n_dust"], seed)
        # the run's list of pairs, which the next step reads: a buffer of one size, -1 past the end
        pairs = torch.empty((case["n_dust"], 2), dtype=torch.int32, device=DEV)
        return dict(case=case, eng=_engine(tables), st=DeviceState(**state), n_grav=n_grav, pairs=pairs)
    massive, dust, N, ids, dt, phys, tables, view, opt, wj, target = _adjoint_inputs(case, seed)
    return dict(case=case, eng=_engine(tables, opt), massive=massive.requires_grad_(), dust=dust.requires_grad_(), N=N,
                ids=ids, dt=dt, phys=make_phys(**phys), view=make_view(**view), wj=wj, target=target)


def run(s):
    c = s["case"]
    if c["kind"] == "step":
        s["eng"].evolve(s["st"], s["n_grav"], s["dt"], c["steps"], s["phys"], PREC[c["precision"]])
        return {f: getattr(s["st"], f) for f in STATE_FIELDS[:6] + ("N",)}
    if c["kind"] == "images":
        return s["eng"].image(s["st"], s["n_grav"], s["view"], s["wj"], precision=PREC[c["precision"]])
    if c["kind"] == "sed":
        return s["eng"].sed(s["st"], s["n_grav"], s["view"], precision=PREC[c["precision"]])
    if c["kind"] == "collide":
        found = s["eng"].collide(s["st"], s["n_grav"], s["st"].n_all, c["h"])
        k = min(found.shape[0], s["pairs"].shape[0])
        s["pairs"].fill_(-1)
        s["pairs"][:k] = found[:k]
        return s["pairs"]
    img = trajectory_image(s["eng"], s["massive"], s["dust"], s["N"], s["ids"], s["dt"], c["steps"], c["ckpt"],
                           s["phys"], s["view"], s["wj"])
    loss = ((img - s["target"]) ** 2).sum()
    gm, gd = torch.autograd.grad(loss, (s["massive"], s["dust"]))
    return {"image": img.detach(), "massive": gm, "dust": gd}


def work(case):
    kind, nd = case["kind"], case["n_dust"]
    if kind == "step":
        ng = case["n_plsml"] + (9 if case["system"] == "solar" else 3)
        # 20 flops a pair, four stages, every body against every massive one; 45 for a star term
        flops = case["steps"] * 4.0 * (20.0 * (ng - 1) * (ng + nd) + 45.0 * nd)
        return {"bytes": float(READ_B + WRITE_B) * (ng + nd), "flops": flops}
    if kind == "images":
        return {"bytes": 36.0 * nd + 8.0 * case["n_img"] * case["xsize"] * case["ysize"], "flops": 60.0 * nd * (1 + case["n_img"])}
    if kind == "sed":
        return {"bytes": 36.0 * nd + 8.0 * N_WAV, "flops": 60.0 * nd * (1 + N_WAV)}
    if kind == "collide":
        return {"bytes": 32.0 * nd, "flops": 8.0 * 8.0 * nd}
    # forward, recomputation and the reverse sweep (about twice a forward) of two planets and the star
    return {"bytes": (36.0 + 7 * 48.0) * nd + 48.0 * case["xsize"] * case["ysize"],
            "flops": 4.0 * case["steps"] * 4.0 * (20.0 * 2 + 45.0) * nd}


# ---- the same results from plain torch in 64 bits -------------------------------------------

def _pull(pos, src, mass, skip_self=False):
    """Gravity (3, n) of the sources (3, m) at the positions (3, n)."""
    out = torch.zeros_like(pos)
    chunk = max(1, (1 << 26) // max(1, src.shape[1]))
    for k in range(0, pos.shape[1], chunk):
        d = [src[a][None, :] - pos[a, k:k + chunk][:, None] for a in range(3)]
        rr = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        if skip_self:
            rr = torch.where(rr == 0.0, torch.ones_like(rr), rr)
        f = mass[None, :] / (rr * torch.sqrt(rr))
        for a in range(3):
            out[a, k:k + chunk] = (f * d[a]).sum(1)
    return out


def _star(d, r, m0, bet, bsw, ph, qm):
    RR = (d * d).sum(0)
    R3 = RR * torch.sqrt(RR)
    f1 = m0 / RR * (bet / LIGHT_AU + bsw / ph["vsw_AUyr"]) if ph["SWQ"] else bet * m0 / LIGHT_AU / RR
    a = -((1.0 - bet - bsw) * m0 / R3) * d - f1 * ((d * r).sum(0) / RR * d + r)
    if ph["FLQ"]:
        B = qm * (ph["Bstar"] * ph["Rstar"] ** 3) / R3
        a = a + torch.stack([B * (r[1] - ph["Wz"] * d[0]), -B * (r[0] + ph["Wz"] * d[1]), torch.zeros_like(B)])
    return a, RR > ph["Rmin"] ** 2


def _rk4(x, v, acc, dt):
    """One step; acc(stage, x, v) gives the acceleration.  Returns x, v and the stage positions."""
    h = dt * 0.5
    a1 = acc(0, x, v)
    r2, x2 = v + a1 * h, x + v * h
    a2 = acc(1, x2, r2)
    r3, x3 = v + a2 * h, x + r2 * h
    a3 = acc(2, x3, r3)
    r4, x4 = v + a3 * dt, x + r3 * dt
    a4 = acc(3, x4, r4)
    return x + dt / 6.0 * (v + 2.0 * (r2 + r3) + r4), v + dt / 6.0 * (a1 + 2.0 * (a2 + a3) + a4), (x, x2, x3, x4)


def _tables_of(tables, ids):
    on = (ids >= 0)
    k = ids.clamp(min=0).long()
    return [torch.where(on, torch.as_tensor(np.asarray(tables[t], np.float64), device=DEV)[k], torch.zeros((), dtype=torch.float64, device=DEV))
            for t in ("beta", "betasw", "q")]


def _exact_step(c, seed):
    ng, dt, ph, tables, st = _step_inputs(c, seed)
    x = torch.stack([st[f] for f in ("x", "y", "z")])
    v = torch.stack([st[f] for f in ("vx", "vy", "vz")])
    xm, vm, xd, vd, m, N = x[:, :ng], v[:, :ng], x[:, ng:], v[:, ng:], st["m"][:ng], st["N"].clone()
    bet, bsw, q = _tables_of(tables, st["id"][ng:])
    if not c["lorentz"]:
        q = torch.zeros_like(q)
    qm = q / torch.where(st["m"][ng:] == 0.0, torch.ones_like(q), st["m"][ng:])
    live = N[ng:] != 0
    for _ in range(c["steps"]):
        xm2, vm2, P = _rk4(xm, vm, lambda k, y, r: _pull(y, y, m, True), dt)
        out = torch.ones_like(live)

        def acc(k, y, r):
            nonlocal out
            a, ok = _star(y - P[k][:, :1], r, m[0], bet, bsw, ph, qm)
            out = out & ok
            return a + _pull(y, P[k][:, 1:], m[1:])

        xd2, vd2, _ = _rk4(xd, vd, acc, dt)
        live = live & out
        xd, vd, xm, vm = torch.where(live, xd2, xd), torch.where(live, vd2, vd), xm2, vm2
    N[ng:] = torch.where(live, N[ng:], torch.zeros_like(N[ng:]))
    x, v = torch.cat([xm, xd], dim=1), torch.cat([vm, vd], dim=1)
    return dict(zip(("x", "y", "z", "vx", "vy", "vz", "N"), [*x, *v, N]))


def _to_sky(pos, view):
    """Distance, scattering-angle cosine and image-plane coordinates in pixels from the corner."""
    x, y, z = pos
    ci, si, cp, sp = math.cos(view["inc"]), math.sin(view["inc"]), math.cos(view["PA"]), math.sin(view["PA"])
    psca = view["fov"] / max(view["xsize"], view["ysize"])
    R = torch.sqrt(x * x + y * y + z * z)
    ly, lz = -view["dist"] * si - y, view["dist"] * ci - z
    cosine = (x * x - y * ly - z * lz) / R / torch.sqrt(x * x + ly * ly + lz * lz)
    cosine = torch.clamp(cosine, min=-1.0, max=1.0 - 2.0 / N_THETA)
    y2 = y * ci + z * si
    return R, cosine, (x * cp - y2 * sp) / psca + 0.5 * view["xsize"], (x * sp + y2 * cp) / psca + 0.5 * view["ysize"]


def _fluxes(R, cosine, N, ids, size, opt, dist, wj):
    """Scattered and thermal flux (Jy) of each tracer, one wavelength after the other."""
    T64 = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=DEV)  # noqa: E731
    k = ids.long()
    lT, fR, lr = torch.log(T64(opt["Td"])), math.log(opt["Rmax"] / opt["Rmin"]) / (N_R - 1.0), torch.log(R / opt["Rmin"])
    j = torch.clamp(torch.floor(lr.detach() / fR).long() + 1, 1, N_R - 1)
    T = torch.exp(lT[k, j - 1] + (lT[k, j] - lT[k, j - 1]) * (lr - (j - 1).double() * fR) / fR)
    T = torch.where(R <= opt["Rmin"], T64(opt["Td"])[k, 0], torch.where(R >= opt["Rmax"], T64(opt["Td"])[k, N_R - 1], T))
    lQ, s = torch.log(T64(opt["Qpfunc"][:, :, wj])), T64(size)[k]
    cm = torch.floor(0.5 * (cosine.detach() + 1.0) * (N_THETA - 1)).long()
    wt = (cosine - (cm.double() * 2.0 / (N_THETA - 1) - 1.0)) / (2.0 / (N_THETA - 1))
    for n, jw in enumerate(wj):
        wvl = float(opt["w"][jw])
        xq = HPLANK * CSPEED / (wvl * KBOLTZ * T)
        planck = 2 * HPLANK * CSPEED ** 2 / (wvl ** 5 * torch.expm1(torch.clamp(xq, max=700.0))) * (xq < 700.0) * math.pi
        P = torch.exp(lQ[k, cm, n] + (lQ[k, cm + 1, n] - lQ[k, cm, n]) * wt)
        scat = float(opt["influx"][jw]) * math.pi * s * s * P / (R * R) / AU / AU     # Qsca = Qabs = 1
        yield N * (planck * s * s / dist / dist + scat) * 1e26 * wvl * wvl / CSPEED * (R > opt["Rmin"])


def _exact_flux(c, seed):
    ng, tables, st, opt, view, wj = _flux_inputs(c, seed)
    R, cosine, u, w = _to_sky([st[f][ng:] for f in ("x", "y", "z")], view)
    N, ids, size = st["N"][ng:], st["id"][ng:], tables["size"]
    if c["kind"] == "sed":
        out = []
        for j in range(0, N_WAV, 10):
            out += [F.sum() for F in _fluxes(R, cosine, N, ids, size, opt, view["dist"], list(range(j, min(j + 10, N_WAV))))]
        return torch.stack(out)
    nx, ny = view["xsize"], view["ysize"]
    i, j = torch.floor(u).long(), torch.floor(w).long()
    on = (i >= 0) & (i < nx) & (j >= 0) & (j < ny)
    pix = torch.where(on, i * ny + j, torch.zeros_like(i))
    out = [torch.zeros(nx * ny, dtype=torch.float64, device=DEV).index_add_(0, pix, F * on)
           for F in _fluxes(R, cosine, N, ids, size, opt, view["dist"], wj)]
    return torch.stack(out).reshape(len(wj), nx, ny)


def _exact_adjoint(c, seed):
    massive, dust, N, ids, dt, ph, tables, view, opt, wj, target = _adjoint_inputs(c, seed)
    massive, dust = massive.requires_grad_(), dust.requires_grad_()
    m = massive[:, 6]
    eye = torch.eye(massive.shape[0], dtype=torch.bool, device=DEV)
    bet, bsw, q = _tables_of(tables, ids)

    def massive_acc(k, y, r):
        d = y[:, None, :] - y[:, :, None]
        rr = torch.where(eye, torch.ones_like(d[0]), (d * d).sum(0))
        f = torch.where(eye, torch.zeros_like(rr), m[None, :] / (rr * torch.sqrt(rr)))
        return (f[None] * d).sum(2)

    xm, vm, xd, vd = massive[:, 0:3].T, massive[:, 3:6].T, dust[:, 0:3].T, dust[:, 3:6].T
    for _ in range(c["steps"]):
        xm2, vm2, P = _rk4(xm, vm, massive_acc, dt)

        def acc(k, y, r):
            a, _ = _star(y - P[k][:, :1], r, m[0], bet, bsw, ph, q)
            for b in range(1, massive.shape[0]):
                d = P[k][:, b:b + 1] - y
                rr = (d * d).sum(0)
                a = a + m[b] / (rr * torch.sqrt(rr)) * d
            return a

        xd, vd, _ = _rk4(xd, vd, acc, dt)
        xm, vm = xm2, vm2
    R, cosine, u, w = _to_sky([xd[0], xd[1], xd[2]], view)
    u, w = u - 0.5, w - 0.5
    nx, ny = view["xsize"], view["ysize"]
    i0, j0 = torch.floor(u.detach()), torch.floor(w.detach())
    fu, fw = u - i0, w - j0
    images = []
    for F in _fluxes(R, cosine, N, ids, tables["size"], opt, view["dist"], wj):
        flat = torch.zeros(nx * ny, dtype=torch.float64, device=DEV)
        for a in (0, 1):
            for b in (0, 1):
                px, py = (i0 + a).long(), (j0 + b).long()
                on = (px >= 0) & (px < nx) & (py >= 0) & (py < ny)
                at = torch.where(on, px * ny + py, torch.zeros_like(px))
                flat = flat.index_add(0, at, F * (fu if a else 1.0 - fu) * (fw if b else 1.0 - fw) * on)
        images.append(flat.reshape(nx, ny))
    img = torch.stack(images)
    gm, gd = torch.autograd.grad(((img - target) ** 2).sum(), (massive, dust))
    return {"image": img.detach(), "massive": gm, "dust": gd}


def exact(case, seed):
    kind = case["kind"]
    if kind == "collide":
        return None                      # whole numbers
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    with torch.no_grad():
        if kind == "step":
            pairs = 4.0 * case["steps"] * (case["n_plsml"] + 9) * (case["n_dust"] + case["n_plsml"])
            return _exact_step(case, seed) if pairs < 3e10 else None
        return _exact_flux(case, seed)
