"""FP64 massive sums with a body that has no finite position, in each of their forms (a warp per body, pairs of
blocks from 1,664 to 4,352 bodies): a NaN position takes part in no pair, so the others move as if the body had
no mass, to rounding; an infinite one makes every other body's sum NaN (0 times an infinite separation)."""
import numpy as np
import pytest
import torch

from diskdyn_gb300 import abi, synth
from diskdyn_gb300.engine import DeviceState, make_phys

pytestmark = pytest.mark.gpu


def stepped(engine, s, state, prec):
    engine.set_size_table(**s.size_table)
    st = DeviceState.from_numpy(state)
    engine.step(st, s.n_grav, s.dt, make_phys(**s.phys), prec)
    torch.cuda.synchronize()
    return st.to_numpy()


@pytest.mark.parametrize("prec", [abi.DDX_PREC_FP64, abi.DDX_PREC_COMPENSATED])
@pytest.mark.parametrize("n_grav", [40, 1663, 1664, 2100, 4352, 4353])
@pytest.mark.parametrize("axis", ["x", "z"])
def test_body_without_a_position(engine, n_grav, prec, axis):
    s = synth.dusty_ring(n_dust=4, n_plsml=n_grav - 3, seed=61, n_steps=1)
    s.state["m"][3:n_grav] = 0.01 * s.state["m"][0] / n_grav
    bad = n_grav // 2
    others = np.delete(np.arange(n_grav), bad)
    massless = {k: v.copy() for k, v in s.state.items()}
    massless["m"][bad] = 0.0
    want = stepped(engine, s, massless, prec)
    nan = {k: v.copy() for k, v in s.state.items()}
    nan[axis][bad] = np.nan
    got = stepped(engine, s, nan, prec)
    for v in ("x", "y", "z"), ("vx", "vy", "vz"):
        a, b = (np.stack([q[f][others] for f in v]) for q in (got, want))
        # 5,000 roundings of sums whose terms are at most the star's pull
        assert (np.linalg.norm(a - b, axis=0) <= 1e-12 * np.linalg.norm(b, axis=0)).all()
    assert np.isnan(got[axis][bad])
    for v in ("vx", "vy", "vz"):                    # no pull on it either
        assert got[v][bad] == nan[v][bad]


@pytest.mark.parametrize("n_grav", [40, 1664, 4353])
def test_body_at_infinity(engine, n_grav):
    s = synth.dusty_ring(n_dust=4, n_plsml=n_grav - 3, seed=61, n_steps=1)
    state = {k: v.copy() for k, v in s.state.items()}
    state["y"][n_grav // 2] = np.inf
    got = stepped(engine, s, state, abi.DDX_PREC_FP64)
    assert np.isnan(np.delete(got["y"][:n_grav], n_grav // 2)).all()
