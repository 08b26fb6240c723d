"""Bounded waits so short that they run out while copies are on their way: some threads see a tile's copy
land and others, even lanes of one tracer, give up before.  The launch has to end and to leave every
block's tracers either stepped or as they were."""
import numpy as np
import pytest
import torch

from diskdyn_gb300 import abi, synth
from diskdyn_gb300.engine import DeviceState, make_phys

pytestmark = pytest.mark.gpu
FIELDS = ("x", "y", "z", "vx", "vy", "vz", "N")


# four lanes per tracer up to 6,144 (mixed) and 16,384 (compensated) tracers, one above
@pytest.mark.parametrize("prec,n_dust", [(abi.DDX_PREC_MIXED, 3000), (abi.DDX_PREC_MIXED, 9000),
                                         (abi.DDX_PREC_COMPENSATED, 3000), (abi.DDX_PREC_COMPENSATED, 20000)])
@pytest.mark.parametrize("wait_ns", [1, 400, 1500])
def test_waits_that_run_out_in_part_of_a_block(engine, prec, n_dust, wait_ns):
    s = synth.dusty_ring(n_dust=n_dust, n_plsml=1100, seed=5, n_steps=1)
    engine.set_size_table(**s.size_table)
    phys, ng = make_phys(**s.phys), s.n_grav

    def step(limited):
        st = DeviceState.from_numpy(s.state)
        if limited:       # no such tile: every copy is made, only the limit holds
            abi.check(engine.lib.ddx_debug_lose_tile_copy(engine.ctx, 1 << 20, wait_ns), "inject")
        engine.step(st, ng, s.dt, phys, prec)
        torch.cuda.synchronize()
        return st.to_numpy()

    whole = step(False)
    assert engine.sync_status() == 0
    for _ in range(5):
        got = step(True)
        status = engine.sync_status()
        assert status in (0, 6)
        as_before = np.all([got[f][ng:] == s.state[f][ng:] for f in FIELDS], axis=0)
        stepped = np.all([got[f][ng:] == whole[f][ng:] for f in FIELDS], axis=0)
        assert (as_before | stepped).all()
        if status == 0:
            assert stepped.all()
    again = step(False)                                  # the context stays usable
    assert engine.sync_status() == 0
    for f in FIELDS:
        np.testing.assert_array_equal(again[f], whole[f])
