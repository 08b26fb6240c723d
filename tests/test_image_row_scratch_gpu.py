"""Device memory of the mixed images' table rows: not taken for few tracers, not asked for on every call when it is
refused, and kept while a captured call may replay with it."""
import numpy as np
import pytest
import torch

from diskdyn_gb300 import abi, synth
from diskdyn_gb300.engine import DeviceState, Engine, make_view

pytestmark = pytest.mark.gpu
N = 100000                       # from here on the rows are used


@pytest.fixture(scope="module")
def system():
    return synth.imaging(n_dust=N, xsize=60, ysize=60)


@pytest.fixture
def context(built_lib, system):
    e = Engine(0)
    o = system.optics
    e.set_size_table(**system.size_table)
    e.set_optics(o["w"], o["in"], o["Qabs"], o["Qsca"], o["Qpfunc"], o["Td"], o["Rmin"], o["Rmax"])
    yield e
    torch.cuda.synchronize()
    e.close()


def wavelengths(n):
    return [int(k) for k in np.linspace(0, 199, n)]


def image(e, s, st, n_img, size=60, out=None):
    return e.image(st, s.n_grav, make_view(**dict(s.view, xsize=size, ysize=size)), wavelengths(n_img), out=out,
                   precision=abi.DDX_PREC_MIXED)


def close(a, b):
    lit = a > 1e-30 * a.amax(dim=(1, 2), keepdim=True)
    return ((b[lit] / a[lit] - 1.0).abs() < 1e-5).all()


def test_few_tracers_take_no_rows(context, system):
    """64 wavelengths of 60 x 60 pixels are 0.9 MB of sums; the rows would be 64 bins x 180 angles x 64 x 8 bytes = 5.9 MB."""
    s = system
    st = DeviceState.from_numpy({k: np.asarray(v)[:s.n_grav + 1000] for k, v in s.state.items()})
    out = image(context, s, st, 1)
    out = torch.empty((64, 60, 60), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    image(context, s, st, 64, out=out)
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] <= 4 << 20


def captured(e, s, st, n_img, size=60):
    out = torch.empty((n_img, size, size), dtype=torch.float64, device="cuda")
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        image(e, s, st, n_img, size, out=out)
    return g, out


def test_refused_rows_are_not_asked_for_again(context, system):
    """With the rows refused a second call allocates nothing, so it can be captured."""
    s, e = system, context
    st = DeviceState.from_numpy(s.state)
    want = image(e, s, st, 8).clone()
    o = s.optics                              # new optics: the rows are gone
    e.set_optics(o["w"], o["in"], o["Qabs"], o["Qsca"], o["Qpfunc"], o["Td"], o["Rmin"], o["Rmax"])
    abi.check(e.lib.ddx_debug_limit_image_rows(e.ctx, 0), "limit")
    assert close(want, image(e, s, st, 8))
    g, out = captured(e, s, st, 8)
    g.replay()
    torch.cuda.synchronize()
    assert close(want, out)


def test_captured_images_replay_after_the_rows_grew(context, system):
    s, e = system, context
    st = DeviceState.from_numpy(s.state)
    want = image(e, s, st, 4, 300).clone()
    g, out = captured(e, s, st, 4, 300)
    image(e, s, st, 64)                       # fewer sums, more rows
    g.replay()
    torch.cuda.synchronize()
    assert close(want, out)


def test_images_captured_first_do_without_rows(context, system):
    s, e = system, context
    st = DeviceState.from_numpy(s.state)
    few = DeviceState.from_numpy({k: np.asarray(v)[:s.n_grav + 1000] for k, v in s.state.items()})
    image(e, s, few, 8)                       # the sums are there, the rows are not
    g, out = captured(e, s, st, 8)
    g.replay()
    torch.cuda.synchronize()
    assert close(image(e, s, st, 8), out)
