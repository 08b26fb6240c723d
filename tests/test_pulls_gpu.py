"""One mixed step's pulls between many bodies against FP64, at the sizes where the kernels'
tiles, slices and orders end.

The planetesimals of a ring get equal masses, together 1 % of the star's, so that one pull
left out or taken twice is seen: among n bodies the weakest (from the far side of the ring)
is about 0.1 / n of A, the sum of the magnitudes of a body's pulls.  Bound: a pull from rsqrt.approx and FP32
arithmetic is off by 6e-7 of itself (2 ulp of rsqrt cubed, and the roundings of the separation
and the product), its sum by less, so a velocity after one step is off by at most
2e-6 dt A, plus FP64 roundings of the velocity itself (1e-14 |v|)."""
import numpy as np
import pytest
import torch

from diskdyn_gb300 import abi, synth
from diskdyn_gb300.engine import DeviceState, make_phys

pytestmark = pytest.mark.gpu


def heavy_ring(n_plsml, n_dust, seed=77):
    s = synth.dusty_ring(n_dust=n_dust, n_plsml=n_plsml, seed=seed, n_steps=1)
    st = {k: np.array(v, copy=True) for k, v in s.state.items()}
    st["m"][3:s.n_grav] = 0.01 * st["m"][0] / n_plsml
    return synth.System(s.name, s.n_grav, st, s.dt, 1, s.phys, s.size_table)


def one_step(engine, s, state, prec):
    engine.set_size_table(**s.size_table)
    d = DeviceState.from_numpy(state)
    engine.step(d, s.n_grav, s.dt, make_phys(**s.phys), prec, abi.DDX_MODE_FIXED)
    torch.cuda.synchronize()
    return d.to_numpy()


def pull_sums(state, ng, rows):
    """Sum over the planetesimals of m / d^2 for the bodies `rows` (FP64, on the CPU)."""
    src = np.stack([state[f][3:ng] for f in "xyz"], 1)
    m = state["m"][3:ng]
    out = np.empty(len(rows))
    for k, i in enumerate(rows):
        d2 = ((src - [state[f][i] for f in "xyz"]) ** 2).sum(1)
        w = np.where(d2 > 0, m / np.where(d2 > 0, d2, 1.0), 0.0)
        out[k] = w.sum()
    return out


def check_velocities(s, f, m, rows, rel=2e-6):
    a = np.maximum(pull_sums(s.state, s.n_grav, rows), pull_sums(f, s.n_grav, rows))
    vf = np.stack([f["v" + c][rows] for c in "xyz"])
    vm = np.stack([m["v" + c][rows] for c in "xyz"])
    bound = rel * s.dt * a + 1e-14 * np.linalg.norm(vf, axis=0)
    e = np.linalg.norm(vm - vf, axis=0)
    assert (e <= bound).all(), (e / bound).max()


# a slice block's 256 targets and 128 threads, a tile's pairs, the one-launch order's threshold
# 1,024 and its list of 1,024 keys a block, and 8,192, where the order goes to the radix sort
@pytest.mark.parametrize("n_plsml", [2, 125, 126, 253, 254, 1023, 1024, 1025, 2047, 2049, 8191, 8192, 8193])
def test_massive_set_pulls(engine, n_plsml):
    s = heavy_ring(n_plsml, 64)
    f = one_step(engine, s, s.state, abi.DDX_PREC_FP64)
    m = one_step(engine, s, s.state, abi.DDX_PREC_MIXED)
    rows = np.arange(3, s.n_grav)
    rows = rows if len(rows) <= 1024 else np.concatenate([rows[:300], rows[300:-300:13], rows[-300:]])
    check_velocities(s, f, m, rows)
