"""Steps whose kernels overlap their start with the end of the one before, against the same steps
captured in a CUDA graph and replayed, on another stream, and with every kernel waited for: the
same bits."""
import numpy as np
import pytest
import torch

from diskdyn_gb300 import abi, synth
from diskdyn_gb300.engine import DeviceState, make_phys

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "z", "vx", "vy", "vz", "N")


# without planetesimals everything overlaps, up to 512 massive bodies the massive passes, beyond
# that the short kernels
@pytest.mark.parametrize("n_plsml", [0, 200, 600, 2100])
@pytest.mark.parametrize("prec", [abi.DDX_PREC_FP64, abi.DDX_PREC_MIXED, abi.DDX_PREC_COMPENSATED])
def test_captured_steps_give_the_same_bits(engine, prec, n_plsml):
    s = synth.dusty_ring(n_dust=3000, n_plsml=n_plsml, seed=8, n_steps=4)
    engine.set_size_table(**s.size_table)
    phys = make_phys(**s.phys)

    def steps(st, n, wait=False):
        for _ in range(n):
            engine.step(st, s.n_grav, s.dt, phys, prec, abi.DDX_MODE_FIXED)
            if wait:
                torch.cuda.synchronize()

    a, b, c, d = (DeviceState.from_numpy(s.state) for _ in range(4))
    steps(a, 4, wait=True)
    steps(b, 4)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        steps(c, 4)
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        steps(d, 2)
    graph.replay()
    graph.replay()
    torch.cuda.synchronize()
    for f in FIELDS:
        for other in (b, c, d):
            assert torch.equal(getattr(a, f), getattr(other, f)), f


def test_repeated_seds_and_collisions_give_the_same_values(engine):
    s = synth.imaging(n_dust=20000, xsize=64, ysize=64)
    engine.set_size_table(**s.size_table)
    o = s.optics
    engine.set_optics(o["w"], o["in"], o["Qabs"], o["Qsca"], o["Qpfunc"], o["Td"], o["Rmin"], o["Rmax"])
    from diskdyn_gb300.engine import make_view
    st = DeviceState.from_numpy(s.state)
    view = make_view(**s.view)
    first = engine.sed(st, s.n_grav, view).clone()
    for _ in range(5):
        assert torch.equal(engine.sed(st, s.n_grav, view), first)
    pairs = engine.collide(st, s.n_grav, st.n_all, 0.3).clone()
    for _ in range(5):
        assert torch.equal(engine.collide(st, s.n_grav, st.n_all, 0.3), pairs)
    assert np.isfinite(first.cpu().numpy()).all()
