"""A few planetesimals scattered far out leave the others' order alone: the belt's groups stay compact, and a cell
has about as many of them near as without those bodies (in one cell of a 30,000 AU order every group spans the
ring and is near every cell)."""
import ctypes as C

import numpy as np
import pytest
import torch

from diskdyn_gb300 import abi, synth
from diskdyn_gb300.engine import DeviceState, make_phys

pytestmark = pytest.mark.gpu


def cells_of_a_step(engine, s, state):
    engine.set_size_table(**s.size_table)
    st = DeviceState.from_numpy(state)
    engine.step(st, s.n_grav, s.dt, make_phys(**s.phys), abi.DDX_PREC_MIXED)
    nodes, room, dropped, near = C.c_longlong(), C.c_longlong(), C.c_int(), C.c_double()
    torch.cuda.synchronize()
    abi.check(engine.lib.ddx_debug_cell_nodes(engine.ctx, C.byref(nodes), C.byref(room), C.byref(dropped), C.byref(near),
                                              None), "cells")
    assert dropped.value == 0 and nodes.value <= room.value
    return near.value, st.to_numpy()


# the order in one block / by radix sort; one body in 32 at most may lie far out
@pytest.mark.parametrize("n_plsml", [4096, 9000])
@pytest.mark.parametrize("share", ["one", "some"])
def test_scattered_planetesimals_do_not_stretch_the_order(engine, n_plsml, share):
    s = synth.dusty_ring(n_dust=20000, n_plsml=n_plsml, seed=51, n_steps=1)
    want, _ = cells_of_a_step(engine, s, s.state)
    g = np.random.default_rng(3)
    state = {k: v.copy() for k, v in s.state.items()}
    n = 1 if share == "one" else n_plsml // 40
    rows = 3 + g.choice(n_plsml, n, replace=False)
    u = g.normal(size=(3, n))
    u *= (30000.0 if n == 1 else 10 ** g.uniform(2.8, 4.5, n)) / np.linalg.norm(u, axis=0)
    for k, c in enumerate("xyz"):
        state[c][rows] = u[k]
    got, out = cells_of_a_step(engine, s, state)
    # the groups of the bodies far out, and the one that they share with the ring's last, may be near every cell
    assert got <= 1.1 * want + n / 16 + 2, (got, want)
    live = out["N"][s.n_grav:] != 0
    assert np.isfinite(out["x"][s.n_grav:][live]).all()
