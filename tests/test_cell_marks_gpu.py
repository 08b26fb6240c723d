"""A tracer's mixed step with cell expansions hangs on its own state and the planetesimals alone, also where the
grids of the cells and of the visiting order end: the bits of a grain are the same alone, among grains beyond
that border, and on every run."""
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
    """4,096 planetesimals, 1,600 of them in a clump at the border of the order's grid; grains in the
    border layer at the clump, and others right beyond the border, which it clamps into that layer.

    flat: the ring has next to no height, so the finest edge is 121 / 30 AU rounded to 4 and the order's
    cells, of half an edge, end 8 edges above the plane: the layer is z = 30 to 32 AU.
    thick: the ring is 40 AU high; with the clump at 508 AU the planetesimals spread over more than half
    an octave, the finest edge is 206 / 24 rounded to 8 and the order's grid ends at 64 edges: the layer
    is x = 504 to 512 AU."""
    s = ring(n_in + n_out)
    g = np.random.default_rng(4)
    ng, a = s.n_grav, s.n_grav + n_out
    if kind == "flat":
        s.state["z"][3:ng] *= 1e-4
        clump = np.array([130.0, 0.0, 31.0]) + 3.0 * g.normal(size=(1600, 3))
        inside = np.stack([130.0 + g.uniform(-8, 8, n_in), g.uniform(-8, 8, n_in), g.uniform(30.05, 31.9, n_in)], 1)
        beyond = np.stack([130.0 + g.uniform(-8, 8, n_out), g.uniform(-8, 8, n_out), g.uniform(33, 45, n_out)], 1)
    else:
        s.state["z"][3:ng] = 40.0 * g.normal(size=4096)
        clump = np.array([508.0, 0.0, 0.0]) + 6.0 * g.normal(size=(1600, 3))
        inside = np.stack([g.uniform(504.2, 511.2, n_in), g.uniform(-16, 16, n_in), g.uniform(-16, 16, n_in)], 1)
        beyond = np.stack([g.uniform(516, 540, n_out), g.uniform(-16, 16, n_out), g.uniform(-16, 16, n_out)], 1)
    place(s, np.arange(3, 1603), clump)
    place(s, np.arange(ng, a), beyond)
    place(s, np.arange(a, a + n_in), inside)
    return s, np.arange(ng, a), np.arange(a, a + n_in)


@pytest.mark.parametrize("kind", ["flat", "thick"])
def test_grains_at_the_border_step_alike_alone_and_beside_clamped_ones(engine, kind):
    s, beyond, inside = border_system(kind)
    alone = grains_of(engine, s, inside)
    for _ in range(3):
        np.testing.assert_array_equal(grains_of(engine, s, np.r_[beyond, inside])[:, len(beyond):], alone)
    # every other one of the grains removed before the step
    half = grains_of(engine, s, np.r_[beyond, inside[::2]])[:, len(beyond):]
    np.testing.assert_array_equal(half, alone[:, ::2])
