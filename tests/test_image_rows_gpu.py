"""Mixed images with the wavelengths' table rows side by side (100,000 tracers and more) and without, at
the numbers of wavelengths where a row's groups of four and the passes of eight end, against
the FP64 images.  Tolerance 1e-5 as for the other mixed images: the FP32 photometry of a pixel's
tracers, 2e-6 each, and its FP32 sum."""
import numpy as np
import pytest
import torch

from diskdyn_gb300 import abi, synth
from diskdyn_gb300.engine import DeviceState, make_view

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def many():
    return synth.imaging(n_dust=100000, xsize=60, ysize=44)


@pytest.mark.parametrize("n_dust", [99999, 100000])
@pytest.mark.parametrize("n_img", [1, 3, 4, 5, 8, 9, 12, 64])
def test_mixed_images_match_fp64(engine, many, n_img, n_dust):
    s, o = many, many.optics
    engine.set_size_table(**s.size_table)
    engine.set_optics(o["w"], o["in"], o["Qabs"], o["Qsca"], o["Qpfunc"], o["Td"], o["Rmin"], o["Rmax"])
    st = DeviceState.from_numpy({k: np.asarray(v)[:s.n_grav + n_dust] for k, v in s.state.items()})
    wj = [int(round(k)) for k in np.linspace(0, len(o["w"]) - 1, n_img)][::-1]
    view = make_view(**s.view)
    a = engine.image(st, s.n_grav, view, wj, precision=abi.DDX_PREC_FP64).cpu().numpy()
    b = engine.image(st, s.n_grav, view, wj, precision=abi.DDX_PREC_MIXED).cpu().numpy()
    torch.cuda.synchronize()
    # pixels without tracers are 0 in both; an image whose brightest tracer FP32 scales to 1 may lose
    # tracers 2^-126 below it, far under the tolerance of any lit pixel
    scale = a.reshape(n_img, -1).max(1).reshape(-1, 1, 1)
    lit = a > 1e-30 * scale
    assert (b[a == 0] == 0).all()
    assert np.abs(b[lit] / a[lit] - 1.0).max() < 1e-5
