"""Which planetesimals act through cells: flat sets (at any tilt) that fill little room.  The others are taken
one by one, with the bits of a context that has no memory for cells.  The choice is the planetesimals' alone: a grain's
step is the same among few tracers and many."""
import ctypes as C

import numpy as np
import pytest
import torch

from diskdyn_gb300 import abi, synth
from diskdyn_gb300.engine import DeviceState, Engine, make_phys

pytestmark = pytest.mark.gpu
FIELDS = ("x", "y", "z", "vx", "vy", "vz", "N")


def disk(g, n, lo, hi, inc, log=False):
    a = 10 ** g.uniform(np.log10(lo), np.log10(hi), n) if log else g.uniform(lo, hi, n)
    t, w = g.uniform(0.0, 2 * np.pi, n), g.uniform(0.0, 2 * np.pi, n)
    z = a * np.sin(np.deg2rad(inc) * g.uniform(0.0, 1.0, n)) * np.sin(w)
    return np.stack([a * np.cos(t), a * np.sin(t), z])


def ball(g, n):
    u = g.normal(size=(3, n))
    return u * (100.0 * g.uniform(0.01, 1.0, n) ** (1 / 3) / np.linalg.norm(u, axis=0))


def tilted(p, degrees):
    c, s = np.cos(np.deg2rad(degrees)), np.sin(np.deg2rad(degrees))
    return np.stack([c * p[0] + s * p[2], p[1], -s * p[0] + c * p[2]])


# root of the smallest eigenvalue of the directions' mean of r r^T times the octaves of distance, against 7e-3 where
# these are few (1.4e-3, 5.4e-3, 7.9e-3, 3.6e-3; 9.6e-3 for the wide ring; 0 for one clump) and 6.2e-2 where they are many
# (4.8e-2, 7.7e-2, 2.1e-2); 1.92 octaves, against 1.25, for two decades
SETS = {"ring": (lambda g, n: disk(g, n, 120, 140, 3), True),
        "inclined 12": (lambda g, n: disk(g, n, 120, 140, 12), True),
        "inclined 17": (lambda g, n: disk(g, n, 120, 140, 17), False),
        "tilted 90": (lambda g, n: tilted(disk(g, n, 120, 140, 8), 90), True),
        "tilted 37": (lambda g, n: tilted(disk(g, n, 120, 140, 8), 37), True),
        "wide": (lambda g, n: disk(g, n, 100, 160, 7), False),
        "clump": (lambda g, n: np.array([[90.0], [90.0], [20.0]]) + g.normal(size=(3, n)), True),
        "ball": (ball, False),
        "disk 8": (lambda g, n: disk(g, n, 20, 200, 8), True),
        "disk 13": (lambda g, n: disk(g, n, 20, 200, 13), False),
        "decade": (lambda g, n: disk(g, n, 30, 300, 3, log=True), True),
        "two decades": (lambda g, n: disk(g, n, 3, 300, 3, log=True), False)}


def system(make, n_plsml, n_dust):
    s = synth.dusty_ring(n_dust=n_dust, n_plsml=n_plsml, seed=81, n_steps=1)
    g = np.random.default_rng(12)
    s.state["m"][3:s.n_grav] = 0.01 * s.state["m"][0] / n_plsml
    s.state["z"][1] += 0.5                               # planets off the planetesimals' plane
    p, d = make(g, n_plsml), make(g, n_dust) + 0.1 * g.normal(size=(3, n_dust))
    for k, c in enumerate("xyz"):
        s.state[c][3:s.n_grav], s.state[c][s.n_grav:] = p[k], d[k]
        s.state["v" + c][:] = 0.0
    return s


def stepped(e, s, n):
    e.set_size_table(**s.size_table)
    st = DeviceState.from_numpy({k: v[:s.n_grav + n].copy() for k, v in s.state.items()})
    e.step(st, s.n_grav, s.dt, make_phys(**s.phys), abi.DDX_PREC_MIXED)
    torch.cuda.synchronize()
    return st.to_numpy()


@pytest.fixture(scope="module")
def without_cells(built_lib):
    e = Engine(0)
    abi.check(e.lib.ddx_debug_limit_cells(e.ctx, 0), "limit")
    yield e
    e.close()


@pytest.mark.parametrize("n_plsml", [2048, 2065, 9001])
@pytest.mark.parametrize("kind", list(SETS))
def test_flat_sets_take_cells(engine, without_cells, kind, n_plsml):
    make, flat = SETS[kind]
    s = system(make, n_plsml, 9000)
    got = stepped(engine, s, 9000)
    nodes, room, dropped, near = C.c_longlong(), C.c_longlong(), C.c_int(), C.c_double()
    abi.check(engine.lib.ddx_debug_cell_nodes(engine.ctx, C.byref(nodes), C.byref(room), C.byref(dropped), C.byref(near),
                                              None), "cells")
    assert (nodes.value > 0) == flat
    one_by_one = stepped(without_cells, s, 9000)
    assert all(np.array_equal(got[f], one_by_one[f]) for f in FIELDS) != flat
    few = stepped(engine, s, 100)                        # four or eight lanes a tracer here
    ng = s.n_grav
    for f in FIELDS:
        np.testing.assert_array_equal(few[f][:ng + 100], got[f][:ng + 100])
