"""Room for the cells where planetesimals need the most of them and tracers are everywhere: no level is left out,
and the first grains step alike alone and among three million.

The finest cell edge is a share of the planetesimals' mean distance, rounded to a power of two or three times
one; the systems are scaled to just below the thresholds at which it is rounded down the farthest."""
import ctypes as C

import numpy as np
import pytest
import torch

from diskdyn_gb300 import abi, synth
from diskdyn_gb300.engine import DeviceState, make_phys

pytestmark = pytest.mark.gpu
FIELDS = ("x", "y", "z", "vx", "vy", "vz", "N")
N_DUST, N_FIRST = 3_000_000, 4000


def directions(g, n):
    u = g.normal(size=(n, 3))
    return u / np.linalg.norm(u, axis=1)[:, None]


def planetesimals(kind, n, g):
    """Of the sets that take cells those that need the most of them: a tilted ring inclined up to 11 degrees, and
    clumps of some 24 groups."""
    if kind == "ring":
        a, t = g.uniform(120.0, 140.0, n), g.uniform(0.0, 2 * np.pi, n)
        z = a * np.sin(np.deg2rad(11.0) * g.uniform(0.0, 1.0, n)) * np.sin(g.uniform(0.0, 2 * np.pi, n))
        x, y = a * np.cos(t), a * np.sin(t)
        return np.stack([0.8 * x - 0.6 * z, y, 0.6 * x + 0.8 * z], 1)
    t = 2 * np.pi * g.integers(0, 8, n) / 8
    return np.stack([130.0 * np.cos(t), 130.0 * np.sin(t), 0.0 * t], 1) + g.normal(size=(n, 3))


# n planetesimals with star and planets a multiple of 1,024; phase: of the finest edge before rounding
@pytest.mark.parametrize("kind,n,phase,power", [("clumps", 3069, 0.285, 0.25), ("clumps", 3069, 0.785, 0.25),
                                                ("ring", 6141, 0.285, 0.125), ("ring", 8189, 0.285, 0.125),
                                                ("ring", 8189, 0.785, 0.125)])
def test_no_level_is_left_out(engine, kind, n, phase, power):
    g = np.random.default_rng(n)
    s = synth.dusty_ring(n_dust=N_DUST, n_plsml=n, seed=71, n_steps=1)
    ng = s.n_grav
    s.state["m"][3:ng] = 0.01 * s.state["m"][0] / n
    p = planetesimals(kind, n, g)
    want = np.log2(np.exp2(np.log2(np.abs(p).max(1)).mean()) / 30.0 * (4096.0 / n) ** power)
    p *= 2.0 ** (phase - (want - np.floor(want)))
    edge = 2.0 ** np.floor(want) * (1.0 if phase < 0.5 else 1.5)
    # half of the grains near planetesimals, half anywhere
    k = N_DUST // 2
    near = p[g.integers(0, n, k)] + directions(g, k) * (10.0 * edge * g.uniform(0.0, 1.0, k) ** (1 / 3))[:, None]
    far = directions(g, N_DUST - k) * (3.0 * np.linalg.norm(p, axis=1).max() * g.uniform(0.0, 1.0, N_DUST - k) ** 0.5)[:, None]
    d = np.concatenate([near, far])[g.permutation(N_DUST)]
    for j, c in enumerate("xyz"):
        s.state[c][3:ng], s.state[c][ng:] = p[:, j], d[:, j]
        s.state["v" + c][:] = 0.0
    engine.set_size_table(**s.size_table)
    out = []
    for m in (N_FIRST, N_DUST):
        st = DeviceState.from_numpy({f: v[:ng + m] for f, v in s.state.items()})
        engine.step(st, ng, s.dt, make_phys(**s.phys), abi.DDX_PREC_MIXED)
        torch.cuda.synchronize()
        got = st.to_numpy()
        out.append(np.stack([got[f][ng:ng + N_FIRST] for f in FIELDS]))
    nodes, room, dropped, near = C.c_longlong(), C.c_longlong(), C.c_int(), C.c_double()
    abi.check(engine.lib.ddx_debug_cell_nodes(engine.ctx, C.byref(nodes), C.byref(room), C.byref(dropped), C.byref(near),
                                              None), "cells")
    assert dropped.value == 0 and 0 < nodes.value <= room.value, (nodes.value, room.value, dropped.value)
    np.testing.assert_array_equal(out[0], out[1])
