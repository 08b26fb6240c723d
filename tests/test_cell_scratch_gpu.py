"""Device memory of the cell expansions: refused on growth, grown under a captured step, and not there when a
step is captured.  Where a step has no cells it takes every planetesimal one by one, which a
context that never gets the memory does too: its bits are the expected ones."""
import numpy as np
import pytest
import torch

from diskdyn_gb300 import abi, synth
from diskdyn_gb300.engine import DeviceState, Engine, make_phys

pytestmark = pytest.mark.gpu
FIELDS = ("x", "y", "z", "vx", "vy", "vz", "N")


def ring(n_plsml):
    return synth.dusty_ring(n_dust=3000, n_plsml=n_plsml, seed=21, n_steps=1)


@pytest.fixture
def contexts(built_lib):
    made = []

    def make(s, most=-1):
        e = Engine(0)
        e.set_size_table(**s.size_table)
        abi.check(e.lib.ddx_debug_limit_cells(e.ctx, most), "limit")
        made.append(e)
        return e

    yield make
    torch.cuda.synchronize()
    for e in made:
        e.close()


def stepped(e, s, prec=abi.DDX_PREC_MIXED):
    st = DeviceState.from_numpy(s.state)
    e.step(st, s.n_grav, s.dt, make_phys(**s.phys), prec)
    torch.cuda.synchronize()
    return st.to_numpy()


def same(a, b):
    return all(np.array_equal(a[f], b[f]) for f in FIELDS)


def captured(e, s, prec=abi.DDX_PREC_MIXED):
    """A graph of one step and the state that it works on."""
    st = DeviceState.from_numpy(s.state)
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        e.step(st, s.n_grav, s.dt, make_phys(**s.phys), prec)
    return g, st


# 2,100 and 4,000 share the massive scratch of 4,096 bodies, 8,000 does not
@pytest.mark.parametrize("more", [4000, 8000])
def test_refused_growth_takes_every_planetesimal(contexts, more):
    few, many = ring(2100), ring(more)
    with_cells = contexts(few)
    cells = stepped(with_cells, few)
    all_pairs = stepped(contexts(many, 0), many)
    assert not same(cells, stepped(contexts(few, 0), few))
    assert not same(all_pairs, stepped(contexts(many), many))
    abi.check(with_cells.lib.ddx_debug_limit_cells(with_cells.ctx, 2200), "limit")
    for _ in range(2):
        assert same(stepped(with_cells, many), all_pairs)
        assert same(stepped(with_cells, few), cells)


def test_captured_step_replays_after_growth(contexts):
    few, many = ring(2100), ring(4000)
    e = contexts(few)
    want = stepped(e, few)
    graph, st = captured(e, few)
    stepped(e, many)                              # grows within the same massive scratch
    graph.replay()
    torch.cuda.synchronize()
    assert same(st.to_numpy(), want)


def test_captured_step_replays_after_more_tracers(contexts):
    """The room for cells goes by the tracers too while they are few."""
    few = ring(2100)
    many = synth.dusty_ring(n_dust=200000, n_plsml=2100, seed=21, n_steps=1)
    e = contexts(few)
    want = stepped(e, few)
    graph, st = captured(e, few)
    got = stepped(e, many)
    assert same(got, stepped(contexts(many), many))
    graph.replay()
    torch.cuda.synchronize()
    assert same(st.to_numpy(), want)
    assert same(stepped(e, few), want)


def test_capture_without_cells_takes_every_planetesimal(contexts):
    """After a compensated step everything but the cells is there."""
    s = ring(2100)
    e = contexts(s)
    stepped(e, s, abi.DDX_PREC_COMPENSATED)
    graph, st = captured(e, s)
    graph.replay()
    torch.cuda.synchronize()
    assert same(st.to_numpy(), stepped(contexts(s, 0), s))
    assert same(stepped(e, s), stepped(contexts(s), s))
