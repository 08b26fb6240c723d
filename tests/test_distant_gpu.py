"""Tracers that take the planetesimals through one expansion about the star, six times their largest
distance away: which of them do, on their own state alone and with every near pull still in FP64."""
import numpy as np
import pytest
import torch

from diskdyn_gb300 import abi, synth
from diskdyn_gb300.engine import DeviceState, make_phys

pytestmark = pytest.mark.gpu
FIELDS = ("x", "y", "z", "vx", "vy", "vz", "N")


def heavy_ring(n_dust):
    """The dusty ring with planetesimals of 1 % of the star's mass together; every body at rest."""
    s = synth.dusty_ring(n_dust=n_dust, n_plsml=4096, seed=41, n_steps=1)
    s.state["m"][3:s.n_grav] = 0.01 * s.state["m"][0] / 4096
    for c in "xyz":
        s.state["v" + c][:] = 0.0
    return s


def shell(g, n, lo, hi):
    u = g.normal(size=(n, 3))
    return u * (g.uniform(lo, hi, n) / np.linalg.norm(u, axis=1))[:, None]


def stepped(engine, s, state, dt, prec=abi.DDX_PREC_MIXED):
    st = DeviceState.from_numpy(state)
    engine.step(st, s.n_grav, dt, make_phys(**s.phys), prec)
    torch.cuda.synchronize()
    return st.to_numpy()


def test_tracers_about_the_limit_step_alike_in_small_groups_and_together(engine):
    """The boxes of the ring's groups reach to 172 AU, so the limit lies at 1,034.  Where a tracer is expected
    leaves the planets out: one of the star's mass, and a step of 100 years, bring it some 0.2 AU further in than
    that.  Of 38,400 tracers from 1,024 to 1,044 AU some hundreds come out on the other side than expected."""
    n, batch = 38400, 64
    s = heavy_ring(n)
    ng = s.n_grav
    s.state["m"][1], s.state["m"][2] = s.state["m"][0], 0.0
    for c, p in zip("xyz", (0.0, 0.0, 400.0)):
        s.state[c][1] = p
    pos = shell(np.random.default_rng(7), n, 1024.0, 1044.0)
    for k, c in enumerate("xyz"):
        s.state[c][ng:] = pos[:, k]
    engine.set_size_table(**s.size_table)
    whole = stepped(engine, s, s.state, 100.0)
    for b in range(0, n, batch):
        rows = np.r_[0:ng, ng + b:ng + b + batch]
        part = stepped(engine, s, {k: v[rows] for k, v in s.state.items()}, 100.0)
        for f in FIELDS:
            np.testing.assert_array_equal(part[f][ng:], whole[f][ng + b:ng + b + batch], err_msg=f"{f} from {b}")


def test_near_radius_beyond_the_distant_limit(engine):
    """A system 200,000 AU from the coordinates' origin and a near radius of 0.02 of that, 4,000 AU: every pull is
    to be FP64's, those on distant tracers too.  Bound: 1e-11 dt A, with A the sum of the pulls' magnitudes (4,096
    FP64 roundings are 5e-13 of A; the expansion's FP32 terms of degree 2 are 1e-9 of it), and 1e-14 of the
    velocity, which the star's pull makes, for the roundings of that."""
    n = 2000
    s = heavy_ring(n)
    ng = s.n_grav
    pos = shell(np.random.default_rng(8), n, 950.0, 2500.0)
    for k, c in enumerate("xyz"):
        s.state[c][ng:] = pos[:, k]
        s.state[c] += (2.0e5, -1.0e5, 0.5e5)[k]
    engine.set_size_table(**s.size_table)
    try:
        abi.check(engine.lib.ddx_set_near_radius(engine.ctx, 0.02), "near")
        m = stepped(engine, s, s.state, s.dt)
    finally:
        abi.check(engine.lib.ddx_set_near_radius(engine.ctx, -1.0), "near")
    f = stepped(engine, s, s.state, s.dt, abi.DDX_PREC_FP64)
    src = np.stack([s.state[c][3:ng] for c in "xyz"], 1)
    A = np.array([(s.state["m"][3:ng] / ((src - [s.state[c][i] for c in "xyz"]) ** 2).sum(1)).sum()
                  for i in range(ng, ng + n)])
    vf, vm = (np.stack([q["v" + c][ng:] for c in "xyz"]) for q in (f, m))
    e = np.linalg.norm(vm - vf, axis=0)
    assert (e <= 1e-11 * s.dt * A + 1e-14 * np.linalg.norm(vf, axis=0)).all(), (e / (s.dt * A)).max()
