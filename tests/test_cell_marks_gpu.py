"""A tracer's mixed step with cell expansions hangs on its own state and the planetesimals alone, also where the
grids of the cells and of the visiting order end: the bits of a grain are the same alone, among grains beyond
that border, and on every run."""
import ctypes as C

import numpy as np
import pytest
import torch

from diskdyn_gb300 import abi, synth
from diskdyn_gb300.engine import DeviceState, make_phys

pytestmark = pytest.mark.gpu
FIELDS = ("x", "y", "z", "vx", "vy", "vz", "N")


def ring(n_dust, n_plsml=4096):
    """The dusty ring with planetesimals of 1 % of the star's mass together, whose cells' choice is
    seen in the last bits."""
    s = synth.dusty_ring(n_dust=n_dust, n_plsml=n_plsml, seed=31, n_steps=1)
    s.state["m"][3:s.n_grav] = 0.01 * s.state["m"][0] / n_plsml
    return s


def place(s, rows, pos, still=True):
    for k, c in enumerate("xyz"):
        s.state[c][rows] = pos[:, k]
        if still:
            s.state["v" + c][rows] = 0.0


def grains_of(engine, s, rows, phys=None, dt=None):
    """The grains `rows` of s after one step without the others."""
    ng = s.n_grav
    state = {k: np.concatenate([v[:ng], v[rows]]) for k, v in s.state.items()}
    st = DeviceState.from_numpy(state)
    engine.set_size_table(**s.size_table)
    engine.step(st, ng, s.dt if dt is None else dt, make_phys(**s.phys), abi.DDX_PREC_MIXED)
    torch.cuda.synchronize()
    g = st.to_numpy()
    return np.stack([g[f][ng:] for f in FIELDS])


def border_system(kind, n_in=2000, n_out=30000):
    """4,096 planetesimals in a ring of next to no height and a clump at the border of the order's grid; grains in
    the border layer at the clump, and others right beyond the border, which it clamps into that layer.

    height: the finest edge is 117 / 30 AU rounded to 4 and the order's cells, of half an edge, end 8 edges above
    the plane: the layer is z = 30 to 32 AU.  480 planetesimals in the clump leave the set flat.
    radius: with 1,600 in the clump at 508 AU they spread over more than half an octave, the finest edge is 206 / 24
    rounded to 8 and the order's grid ends at 64 edges: the layer is x = 508 to 512 AU."""
    s = ring(n_in + n_out)
    g = np.random.default_rng(4)
    ng, a = s.n_grav, s.n_grav + n_out
    s.state["z"][3:ng] *= 1e-4
    if kind == "height":
        clump = np.array([130.0, 0.0, 31.0]) + 3.0 * g.normal(size=(480, 3))
        inside = np.stack([130.0 + g.uniform(-8, 8, n_in), g.uniform(-8, 8, n_in), g.uniform(30.05, 31.9, n_in)], 1)
        beyond = np.stack([130.0 + g.uniform(-8, 8, n_out), g.uniform(-8, 8, n_out), g.uniform(33, 45, n_out)], 1)
    else:
        clump = np.array([508.0, 0.0, 0.0]) + 6.0 * g.normal(size=(1600, 3))
        inside = np.stack([g.uniform(508.2, 511.2, n_in), g.uniform(-16, 16, n_in), g.uniform(-16, 16, n_in)], 1)
        beyond = np.stack([g.uniform(516, 540, n_out), g.uniform(-16, 16, n_out), g.uniform(-16, 16, n_out)], 1)
    place(s, np.arange(3, 3 + len(clump)), clump)
    place(s, np.arange(ng, a), beyond)
    place(s, np.arange(a, a + n_in), inside)
    return s, np.arange(ng, a), np.arange(a, a + n_in)


def cells_built(engine):
    nodes, room, dropped, near = C.c_longlong(), C.c_longlong(), C.c_int(), C.c_double()
    abi.check(engine.lib.ddx_debug_cell_nodes(engine.ctx, C.byref(nodes), C.byref(room), C.byref(dropped), C.byref(near),
                                              None), "cells")
    return nodes.value


@pytest.mark.parametrize("kind", ["height", "radius"])
def test_grains_at_the_border_step_alike_alone_and_beside_clamped_ones(engine, kind):
    s, beyond, inside = border_system(kind)
    alone = grains_of(engine, s, inside)
    assert cells_built(engine) > 0
    for _ in range(3):
        np.testing.assert_array_equal(grains_of(engine, s, np.r_[beyond, inside])[:, len(beyond):], alone)
    # every other one of the grains removed before the step
    half = grains_of(engine, s, np.r_[beyond, inside[::2]])[:, len(beyond):]
    np.testing.assert_array_equal(half, alone[:, ::2])
