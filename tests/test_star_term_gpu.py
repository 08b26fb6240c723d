"""The star's pull, drags and Lorentz force of the step kernels (one rsqrt, per-tracer factors) against
the CPU oracle's expression, with and without stellar wind, charges and massive bodies, in
every precision, and tracers exactly on a planetesimal.

Tolerances: about 40 FP64 roundings of 1.1e-16 in an acceleration, whose share of the new
velocity is at most one here: 1e-13 leaves ten times that.  The planetesimals have no mass here
(test_pulls_gpu.py bounds their pulls): they only choose the kernel."""
import numpy as np
import pytest
import torch

import oracle.cpu as oc
from diskdyn_gb300 import abi, synth
from diskdyn_gb300.engine import DeviceState, make_phys

pytestmark = pytest.mark.gpu

PREC = [abi.DDX_PREC_FP64, abi.DDX_PREC_MIXED, abi.DDX_PREC_COMPENSATED]


def step(engine, s, st, prec):
    engine.set_size_table(**s.size_table)
    d = DeviceState.from_numpy(st)
    engine.step(d, s.n_grav, s.dt, make_phys(**s.phys), prec, abi.DDX_MODE_FIXED)
    torch.cuda.synchronize()
    return d.to_numpy()


@pytest.mark.parametrize("prec", PREC)
@pytest.mark.parametrize("n_plsml", [0, 40, 2500])
@pytest.mark.parametrize("swq,flq", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_star_term(engine, prec, n_plsml, swq, flq):
    s = synth.dusty_ring(n_dust=700, n_plsml=n_plsml, seed=19, n_steps=1)
    s.phys = dict(s.phys, SWQ=swq, FLQ=flq, Bstar=5e-20, Wz=14.6)
    s.size_table["q"] = np.linspace(1e-3, 2e-3, len(s.size_table["size"])).astype(np.float32)
    st = {k: np.array(v, copy=True) for k, v in s.state.items()}
    st["m"][3:s.n_grav] = 0.0
    st["m"][s.n_grav:] = 1e-30                   # with these charges the Lorentz force is some 1e-3 of the star's pull
    st["z"][s.n_grav::5] *= 40.0
    for c in "xyz":
        st[c][s.n_grav + 1::50] *= 0.02          # close to the star, a few inside its sublimation radius
        st[c][s.n_grav + 2::100] *= 0.002
    g = step(engine, s, st, prec)
    o = oc.step(st, s.n_grav, s.dt, s.size_table, s.phys, 1, ref_mode=False)
    np.testing.assert_array_equal(g["N"] == 0, o["N"] == 0)
    live = o["N"] != 0
    for f in ("", "v"):
        a = np.stack([g[f + c][live] for c in "xyz"])
        b = np.stack([o[f + c][live] for c in "xyz"])
        # a grain thrown out by the star within the step: its velocity change sets the scale
        scale = np.linalg.norm(b, axis=0) + np.linalg.norm(np.stack([st[f + c][live] for c in "xyz"]), axis=0)
        e = np.linalg.norm(a - b, axis=0) / scale
        near = np.linalg.norm(np.stack([st[c][live] for c in "xyz"]), axis=0) < 10.0
        assert e[~near].max() < 1e-13
        assert e[near].max() < 1e-10             # half an orbit and more in one step: stages amplify roundings


@pytest.mark.parametrize("prec", PREC)
@pytest.mark.parametrize("n_plsml", [256, 1100, 2500])
def test_tracer_on_a_planetesimal_is_removed(engine, prec, n_plsml):
    s = synth.dusty_ring(n_dust=3000, n_plsml=n_plsml, seed=3, n_steps=1)
    st = {k: np.array(v, copy=True) for k, v in s.state.items()}
    rows = s.n_grav + 10 * np.arange(5)
    for k, i in enumerate(rows):
        for f in ("x", "y", "z", "vx", "vy", "vz"):
            st[f][i] = st[f][3 + 7 * k]
    g = step(engine, s, st, prec)
    assert (g["N"][rows] == 0).all() and (g["N"][s.n_grav:] == 0).sum() == 5
