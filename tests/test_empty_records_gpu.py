"""A grain at exactly (0, 0, 0), away from the star and among the planetesimals of a last group that is not full:
the group's empty slots are no bodies that it could coincide with."""
import numpy as np
import pytest
import torch

from diskdyn_gb300 import abi, synth
from diskdyn_gb300.engine import DeviceState, make_phys

pytestmark = pytest.mark.gpu


# 2,048 fills its groups of 16 and spans of 32; one more, half a span, all but one slot
@pytest.mark.parametrize("n_plsml", [2048, 2049, 2064, 2065, 2079])
@pytest.mark.parametrize("prec", [abi.DDX_PREC_MIXED, abi.DDX_PREC_COMPENSATED])
def test_grain_at_the_origin_of_the_coordinates(engine, n_plsml, prec):
    s = synth.dusty_ring(n_dust=200, n_plsml=n_plsml, seed=91, n_steps=1)
    g = np.random.default_rng(2)
    ng = s.n_grav
    s.state["m"][3:ng] = 1e-6 * s.state["m"][0] / n_plsml
    s.state["x"][0] += 5.0                       # the planetesimals and grains: a clump 5 AU from the star
    for c in "xyz":
        s.state[c][3:] = 0.05 * g.normal(size=n_plsml + 200)
        s.state[c][ng] = 0.0
        s.state["v" + c][:] = 0.0
    got = {}
    for p in (prec, abi.DDX_PREC_FP64):
        engine.set_size_table(**s.size_table)
        st = DeviceState.from_numpy(s.state)
        engine.step(st, ng, 1e-4, make_phys(**s.phys), p)
        torch.cuda.synchronize()
        got[p] = st.to_numpy()
    np.testing.assert_array_equal(got[prec]["N"], got[abi.DDX_PREC_FP64]["N"])
    assert got[prec]["N"][ng] != 0
    x, want = (np.array([q[c][ng] for c in ("x", "y", "z", "vx", "vy", "vz")]) for q in (got[prec], got[abi.DDX_PREC_FP64]))
    assert np.abs(x - want).max() <= 1e-9 * np.abs(want).max()
