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
# 1,024 and its list of 1,024 keys a block, 6,144 and 8,192 bodies, where the slices become more, and 8,192
# planetesimals, where the order goes to the radix sort
@pytest.mark.parametrize("n_plsml", [2, 125, 126, 253, 254, 1023, 1024, 1025, 2047, 2049, 6141, 6142, 8189, 8190, 8191, 8192,
                                     8193])
def test_massive_set_pulls(engine, n_plsml):
    s = heavy_ring(n_plsml, 64)
    f = one_step(engine, s, s.state, abi.DDX_PREC_FP64)
    m = one_step(engine, s, s.state, abi.DDX_PREC_MIXED)
    rows = np.arange(3, s.n_grav)
    rows = rows if len(rows) <= 1024 else np.concatenate([rows[:300], rows[300:-300:13], rows[-300:]])
    check_velocities(s, f, m, rows)


# Cell expansions of far planetesimals.  Their series stops at degree 10; for one source at the
# least far distance of 4.5 cell edges and a tracer at the corner of the reach of 0.55 edges
# (ratio 0.21) the rest is at most sum over n > 10 of n 0.21^(n - 1) = 2.6e-6 of the pull;
# with the FP32 roundings above 4e-6.
CELLS = 4e-6


def scattered(n_plsml, n_dust, seed=78):
    """The heavy ring with grains everywhere: half in the ring, the rest at 15 to 5,000 AU in
    all directions, and every 100th planetesimal moved to 300 to 30,000 AU."""
    s = heavy_ring(n_plsml, n_dust, seed)
    g = np.random.default_rng(seed)
    ng = s.n_grav

    def move(rows, lo, hi):
        u = g.normal(size=(3, len(rows)))
        u *= 10 ** g.uniform(np.log10(lo), np.log10(hi), len(rows)) / np.linalg.norm(u, axis=0)
        for k, c in enumerate("xyz"):
            s.state[c][rows] = u[k]
            s.state["v" + c][rows] *= 0.1
    move(np.arange(ng + 1, ng + n_dust, 2), 15.0, 5000.0)
    move(np.arange(3, ng, 100), 300.0, 30000.0)
    return s


# 2,048 planetesimals is where the cells begin, 8,192 where the grid becomes finer
@pytest.mark.parametrize("n_plsml", [2047, 2048, 2049, 4096, 8192, 8193, 16385])
@pytest.mark.parametrize("make", [heavy_ring, scattered])
def test_tracer_pulls(engine, n_plsml, make):
    s = make(n_plsml, 3000)
    f = one_step(engine, s, s.state, abi.DDX_PREC_FP64)
    m = one_step(engine, s, s.state, abi.DDX_PREC_MIXED)
    np.testing.assert_array_equal(m["N"] == 0, f["N"] == 0)
    rows = np.arange(s.n_grav, s.n_grav + 3000)
    check_velocities(s, f, m, rows[f["N"][rows] != 0], CELLS)


def test_lanes_per_tracer_give_the_same_bits(engine):
    """Few tracers are shared by 8 or 4 lanes each; the first 100 grains come out the same
    among 100, 7,999, 8,000, 33,999, 34,000 and 48,000."""
    s = scattered(3000, 48000)
    ng = s.n_grav
    first = None
    for n in (100, 7999, 8000, 33999, 34000, 48000):
        state = {k: np.asarray(v)[:ng + n].copy() for k, v in s.state.items()}
        m = one_step(engine, s, state, abi.DDX_PREC_MIXED)
        got = np.stack([m[c][:ng + 100] for c in ("x", "y", "z", "vx", "vy", "vz", "N")])
        if first is None:
            first = got
        np.testing.assert_array_equal(got, first)


@pytest.mark.parametrize("far", [0.0, 1e12, 1e30])
def test_star_and_planetesimals_far_from_the_origin(engine, far):
    """The whole system displaced by 2^20 AU and more, or a planetesimal at a huge distance or
    with no finite position: tracers take every planetesimal when no cell serves them, and stay as
    close to FP64 as its own rounding allows."""
    s = heavy_ring(2500, 2000)
    st = {k: v.copy() for k, v in s.state.items()}
    if far == 0.0:
        for c, d in (("x", 2.0 ** 21), ("y", -2.0 ** 21), ("z", 2.0 ** 20)):
            st[c] += d
    else:
        st["x"][s.n_grav - 1] = far
    f = one_step(engine, s, st, abi.DDX_PREC_FP64)
    m = one_step(engine, s, st, abi.DDX_PREC_MIXED)
    np.testing.assert_array_equal(m["N"] == 0, f["N"] == 0)
    rows = np.arange(s.n_grav, s.n_grav + 2000)
    rows = rows[f["N"][rows] != 0]
    # hi + lo hold a coordinate to 2^-48 of itself: 7.5e-9 AU at 2^21 AU against separations beyond
    # the near radius (which is there larger than the ring): every pull is FP64's
    a = pull_sums(st, s.n_grav, rows)
    e = np.linalg.norm(np.stack([m["v" + c][rows] - f["v" + c][rows] for c in "xyz"]), axis=0)
    v = np.linalg.norm(np.stack([f["v" + c][rows] for c in "xyz"]), axis=0)
    assert (e <= CELLS * s.dt * a + 1e-14 * v + (1e-12 * v if far == 0.0 else 0.0)).all()


def test_fp64_lanes_per_tracer_give_the_same_bits(engine):
    """Four lanes share a tracer of the FP64 step up to 4,864 tracers, or 131,072 with 128 massive
    bodies and more; the first 50 grains come out the same on either side."""
    for n_plsml, counts in ((3, (50, 4864, 4865)), (123, (50, 4864, 4865)), (127, (50, 131072, 131073))):
        s = synth.dusty_ring(n_dust=counts[-1], n_plsml=n_plsml, seed=12, n_steps=1)
        first = None
        for n in counts:
            state = {k: np.asarray(v)[:s.n_grav + n].copy() for k, v in s.state.items()}
            m = one_step(engine, s, state, abi.DDX_PREC_FP64)
            got = np.stack([m[c][:s.n_grav + 50] for c in ("x", "y", "z", "vx", "vy", "vz", "N")])
            first = got if first is None else first
            np.testing.assert_array_equal(got, first)


# massive bodies at the ends of a group of four sources and of a tile of 256
@pytest.mark.parametrize("n_plsml", [1, 2, 3, 4, 5, 253, 254, 255, 256, 257])
def test_fp64_tracer_pulls(engine, n_plsml):
    """Against the same sums in FP64 on the CPU: velocities after one step to 1e-13 (some 50
    roundings of a sum whose terms are at most the star's pull)."""
    import oracle.cpu as oc
    s = heavy_ring(n_plsml, 300)
    f = one_step(engine, s, s.state, abi.DDX_PREC_FP64)
    o = oc.step(s.state, s.n_grav, s.dt, s.size_table, s.phys, 1, ref_mode=False)
    np.testing.assert_array_equal(f["N"] == 0, o["N"] == 0)
    vf, vo = (np.stack([q["v" + c][s.n_grav:] for c in "xyz"]) for q in (f, o))
    live = o["N"][s.n_grav:] != 0
    assert (np.linalg.norm(vf - vo, axis=0) / np.linalg.norm(vo, axis=0))[live].max() < 1e-13


# index order and spatial order, few and many spans; four lanes up to 6,144 and 16,384 tracers
@pytest.mark.parametrize("n_plsml", [127, 128, 300, 1500])
@pytest.mark.parametrize("prec,counts", [(abi.DDX_PREC_MIXED, (70, 6144, 6145)),
                                         (abi.DDX_PREC_COMPENSATED, (70, 16384, 16385))])
def test_span_lanes_per_tracer_give_the_same_bits(engine, prec, counts, n_plsml):
    s = scattered(n_plsml, counts[-1])
    ng = s.n_grav
    first = None
    for n in counts:
        state = {k: np.asarray(v)[:ng + n].copy() for k, v in s.state.items()}
        m = one_step(engine, s, state, prec)
        got = np.stack([m[c][:ng + 70] for c in ("x", "y", "z", "vx", "vy", "vz", "N")])
        first = got if first is None else first
        np.testing.assert_array_equal(got, first)


@pytest.mark.parametrize("n_plsml", [127, 128, 129, 511, 512, 513, 1500])
def test_few_tracers_pulls(engine, n_plsml):
    s = heavy_ring(n_plsml, 500)
    f = one_step(engine, s, s.state, abi.DDX_PREC_FP64)
    rows = np.arange(s.n_grav, s.n_grav + 500)
    for prec, rel in ((abi.DDX_PREC_MIXED, 2e-6), (abi.DDX_PREC_COMPENSATED, 6e-7)):
        m = one_step(engine, s, s.state, prec)
        np.testing.assert_array_equal(m["N"] == 0, f["N"] == 0)
        check_velocities(s, f, m, rows[f["N"][rows] != 0], rel)


# FP64 all-pairs over pairs of bodies from 1,664 to 4,352 massive bodies (3 of them star and planets), in
# blocks of 128
@pytest.mark.parametrize("n_grav", [1663, 1664, 1665, 1791, 1792, 1793, 4223, 4351, 4352, 4353])
@pytest.mark.parametrize("prec", [abi.DDX_PREC_FP64, abi.DDX_PREC_COMPENSATED])
def test_massive_set_in_fp64(engine, n_grav, prec):
    """Against the sums in FP64 on the CPU, without the later stages: a step so short that the
    velocity's change is dt times the first acceleration.  4,000 roundings are 4e-13 of the pulls'
    magnitudes, and the bodies' motion within the step, a dt^2 against the nearest at some 0.01 AU, is
    as much: 1e-9 leaves room for pairs a thousand times nearer, and one pull left out is 2e-4 / 10."""
    s = heavy_ring(n_grav - 3, 8)
    st = {k: v.copy() for k, v in s.state.items()}
    for c in "xyz":
        st["v" + c][:n_grav] = 0.0               # so that the change of velocity is the velocity
    dt = 1e-6
    engine.set_size_table(**s.size_table)
    d = DeviceState.from_numpy(st)
    engine.step(d, s.n_grav, dt, make_phys(**s.phys), prec, abi.DDX_MODE_FIXED)
    torch.cuda.synchronize()
    got = d.to_numpy()
    x, m = np.stack([st[c][:n_grav] for c in "xyz"], 1), st["m"][:n_grav]
    rows = np.r_[0:40, 100:n_grav:37, n_grav - 40:n_grav]
    for i in rows:
        dx = x - x[i]
        r2 = (dx ** 2).sum(1)
        r2[i] = 1.0
        w = m / (r2 * np.sqrt(r2))
        w[i] = 0.0
        want = dt * (w[:, None] * dx).sum(0)
        mag = dt * (w * np.sqrt(r2)).sum()
        v = np.array([got["v" + c][i] for c in "xyz"])
        assert np.abs(v - want).max() <= 1e-9 * mag, (i, np.abs(v - want).max() / mag)


def test_grains_in_a_ball_step_alike_alone_and_among_many(engine):
    """A ball of planetesimals with tracers everywhere in it needs the most cells; all of them fit, so
    the first 5,000 grains come out the same alone and among 1,500,000."""
    n_dust = 1_500_000
    s = heavy_ring(8100, n_dust)
    g = np.random.default_rng(6)
    ng = s.n_grav
    for rows in (slice(3, ng), slice(ng, None)):
        n = len(s.state["x"][rows])
        u = g.normal(size=(3, n))
        u *= 140.0 * g.uniform(0.01, 1.0, n) ** (1 / 3) / np.linalg.norm(u, axis=0)
        for k, c in enumerate("xyz"):
            s.state[c][rows] = u[k]
            s.state["v" + c][rows] *= 0.3
    got = []
    for n in (5000, n_dust):
        m = one_step(engine, s, {k: np.asarray(v)[:ng + n].copy() for k, v in s.state.items()}, abi.DDX_PREC_MIXED)
        got.append(np.stack([m[c][:ng + 5000] for c in ("x", "y", "z", "vx", "vy", "vz", "N")]))
    np.testing.assert_array_equal(got[0], got[1])


# 100,000 tracers: blocks and tiles of half the size
@pytest.mark.parametrize("n_plsml", [100, 257, 1100])
@pytest.mark.parametrize("prec", [abi.DDX_PREC_MIXED, abi.DDX_PREC_COMPENSATED])
def test_blocks_of_half_the_size_give_the_same_bits(engine, prec, n_plsml):
    s = scattered(n_plsml, 100000)
    ng = s.n_grav
    got = []
    for n in (99999, 100000):
        m = one_step(engine, s, {k: np.asarray(v)[:ng + n].copy() for k, v in s.state.items()}, prec)
        got.append(np.stack([m[c][:ng + 99999] for c in ("x", "y", "z", "vx", "vy", "vz", "N")]))
    np.testing.assert_array_equal(got[0], got[1])
