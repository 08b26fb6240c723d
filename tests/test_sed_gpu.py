"""The FP64 SED at the sizes where its batches of 32 tracers, its threads (a wavelength and a
slice of the batch each, up to 512) and its rows of block sums end, against the CPU oracle.
Tolerance 1e-11 as for the images: the factors are the oracle's in another order (some 20
roundings), and a Planck exponent of up to 700 carries its own rounding, 2e-13."""
import numpy as np
import pytest
import torch

import oracle.cpu as oc
from diskdyn_gb300 import abi, synth
from diskdyn_gb300.engine import DeviceState, make_view

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_wav,n_dust", [(1, 1), (2, 31), (31, 32), (33, 33), (200, 1000), (200, 45000), (511, 100),
                                          (512, 65), (513, 65), (700, 200)])
def test_sed_sizes(engine, n_wav, n_dust):
    s = synth.imaging(n_dust=n_dust, xsize=16, ysize=16)
    o = synth.hg_optics(n_grid=len(s.size_table["size"]), n_wav=n_wav)
    o["size"] = s.size_table["size"]
    engine.set_size_table(**s.size_table)
    engine.set_optics(o["w"], o["in"], o["Qabs"], o["Qsca"], o["Qpfunc"], o["Td"], o["Rmin"], o["Rmax"])
    st = DeviceState.from_numpy(s.state)
    F = engine.sed(st, s.n_grav, make_view(**s.view), mode=abi.DDX_MODE_FIXED).cpu().numpy()
    G = engine.sed(st, s.n_grav, make_view(**s.view), mode=abi.DDX_MODE_FIXED).cpu().numpy()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(F, G)
    Fo = oc.sed(s.state, s.n_grav, o, s.size_table["size"], s.view, ref_mode=False)
    np.testing.assert_allclose(F, Fo, rtol=1e-11)
