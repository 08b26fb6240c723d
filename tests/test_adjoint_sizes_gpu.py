"""The gradient kernels where their paths change: five massive bodies (a lane per pair of bodies up to
there) and six, tracers around a block of 64, and scratch memory kept from a larger and a smaller
call on another stream.  Against torch.autograd over the same model on the CPU, with the
tolerances of the two-planet comparison (the same FP64 operations in another order)."""
import numpy as np
import pytest
import torch

import oracle.torch_ref as tr
from diskdyn_gb300 import adjoint as adj
from diskdyn_gb300.engine import Engine, make_phys, make_view

pytestmark = pytest.mark.gpu

STEPS = 8


@pytest.fixture(scope="module")
def sys65():
    s = adj.adjoint_system(n_dust=200, xsize=48, ysize=40, n_steps=STEPS, seed=5)
    eng = Engine(0)
    eng.set_size_table(**s.size_table)
    o = s.optics
    eng.set_optics(o["w"], o["in"], o["Qabs"], o["Qsca"], o["Qpfunc"], o["Td"], o["Rmin"], o["Rmax"])
    yield s, eng
    eng.close()


def inputs(s, n_massive, n_dust):
    m = np.stack([s.state[k][:s.n_grav] for k in ("x", "y", "z", "vx", "vy", "vz", "m")], axis=1)
    extra = m[np.arange(max(n_massive - len(m), 0)) % (len(m) - 1) + 1].copy()
    for k in range(len(extra)):                   # more planets, turned and moved out
        c, q = np.cos(1.0 + k), np.sin(1.0 + k)
        for a in (0, 3):
            extra[k, a], extra[k, a + 1] = c * extra[k, a] - q * extra[k, a + 1], q * extra[k, a] + c * extra[k, a + 1]
        extra[k, :3] *= 1.3 + 0.1 * k
        extra[k, 3:6] /= np.sqrt(1.3 + 0.1 * k)
    m = np.concatenate([m, extra])[:n_massive]
    rows = slice(s.n_grav, s.n_grav + n_dust)
    d = np.stack([s.state[k][rows] for k in ("x", "y", "z", "vx", "vy", "vz")], axis=1)
    return m, d, s.state["N"][rows], s.state["id"][rows].astype(np.int32)


def gpu_gradients(s, eng, m, d, N, ids, ckpt=3):
    m, d = (torch.tensor(a, device="cuda", dtype=torch.float64, requires_grad=True) for a in (m, d))
    img = adj.trajectory_image(eng, m, d, torch.tensor(N, device="cuda"), torch.tensor(ids, device="cuda"), s.dt, STEPS, ckpt,
                               make_phys(**dict(s.phys, n_planets=len(m))), make_view(**s.view), s.image_wj)
    gm, gd = torch.autograd.grad((img ** 2).sum(), (m, d))
    return gm, gd


@pytest.mark.parametrize("n_massive", [1, 2, 5, 6])
@pytest.mark.parametrize("n_dust", [1, 63, 64, 65, 200])
def test_gradients_match_torch(sys65, n_massive, n_dust):
    s, eng = sys65
    m, d, N, ids = inputs(s, n_massive, n_dust)
    gm, gd = gpu_gradients(s, eng, m, d, N, ids)
    mc, dc = (torch.tensor(a, dtype=torch.float64, requires_grad=True) for a in (m, d))
    k = torch.tensor(ids, dtype=torch.int64)
    beta, betasw = (torch.tensor(s.size_table[f].astype(np.float64))[k] for f in ("beta", "betasw"))
    final = tr.trajectory(mc, dc, beta, betasw, s.dt, STEPS, s.phys["SWQ"], s.phys["vsw_AUyr"])
    img = tr.splat_image(final[:, :3], torch.tensor(N, dtype=torch.float64), k, s.optics, s.optics["size"], s.view, s.image_wj)
    cm, cd = torch.autograd.grad((img ** 2).sum(), (mc, dc))
    for a, b in ((gm, cm), (gd, cd)):
        a, b = a.cpu().numpy(), b.numpy()
        np.testing.assert_allclose(a, b, rtol=1e-7, atol=1e-9 * np.abs(b).max())


def test_kept_scratch_gives_the_same_gradients(sys65):
    s, eng = sys65
    want = {}
    for n in (200, 3, 64):
        fresh, o = Engine(0), s.optics
        fresh.set_size_table(**s.size_table)
        fresh.set_optics(o["w"], o["in"], o["Qabs"], o["Qsca"], o["Qpfunc"], o["Td"], o["Rmin"], o["Rmax"])
        want[n] = [g.clone() for g in gpu_gradients(s, fresh, *inputs(s, 3, n))]
        fresh.close()
    for k, n in enumerate((64, 200, 3, 200, 64)):
        stream = torch.cuda.Stream() if k % 2 else torch.cuda.current_stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            got = gpu_gradients(s, eng, *inputs(s, 3, n))
        torch.cuda.synchronize()
        # the image is summed by atomics: its last bits vary from run to run
        for a, b in zip(got, want[n]):
            np.testing.assert_allclose(a.cpu().numpy(), b.cpu().numpy(), rtol=1e-10,
                                       atol=1e-12 * b.abs().max().item())
