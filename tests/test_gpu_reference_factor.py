"""REFERENCE math's factors ((m r) r) r, r = 1 / sqrt(d2) with both operations correctly
rounded, for every mantissa of d2: one source of mass 1 and massless targets whose squared
distances from it are the floats of a range, so that each target's acceleration is one term.
The wanted bits are NumPy's float32 root, quotient and products.

The kernels make two consecutive sources' factors together: the source's neighbour stands
elsewhere, at distances in range, so that only the target's own value decides how it is taken."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
REF = dict(simulation_time=1.0, gravitational_const=1.0)


def _offsets(x):
    """(dx, dy) with fma(dx, dx, fma(dy, dy, eps2)) == x for any eps2 below 2^-40 x."""
    x64 = x.astype(np.float64)
    dx = np.sqrt(x64).astype(np.float32)
    dx = np.where(dx.astype(np.float64) ** 2 > x64, np.nextafter(dx, np.float32(0)), dx)
    dy = np.sqrt(x64 - dx.astype(np.float64) ** 2).astype(np.float32)  # at most sqrt(2^-22 x)
    return np.stack([dx, dy], axis=1)


def _wanted(x, offsets, m):
    r = np.float32(1) / np.sqrt(x)
    with np.errstate(over="ignore", invalid="ignore"):  # r^3 beyond FP32 with mass 1: infinities, and NaN for dy = 0
        return -offsets * (((np.float32(m) * r) * r) * r)[:, None]


def _wrong(gs, x, n, source, scale, softening, m=1.0, batched=False):
    """The squared distances of x (times scale^2) whose term differs from the wanted one."""
    x = (x * np.float32(scale * scale)).astype(np.float32)
    partner = source ^ 1
    targets = np.setdiff1d(np.arange(n), [source, partner])
    pos = np.zeros((n, 2), np.float32)
    pos[partner] = np.array((1.5, 0.9) if scale > 1 else (-1.25, 0.4)) * scale
    mass = np.zeros(n, np.float32)
    mass[source] = m
    vel = np.zeros_like(pos)
    wrong = []
    params = gs.default_params(algorithm=gs.DIRECT_SUM, math_mode=gs.MATH_REFERENCE, softening_len=softening,
                               flags=gs.FLAG_RECORD_ACCEL, **REF)
    pos[targets, 0] = np.float32(scale)
    with gs.Simulation(pos, vel, mass, params=params) as sim:
        batch = gs.Batch([sim]) if batched else None
        for at in range(0, len(x), len(targets)):
            part = x[at:at + len(targets)]
            off = _offsets(part)
            pos[targets[:len(part)]] = off
            sim.set_particles(pos, vel, mass)
            if batched:
                batch.run(1)
                batch.sync()
            else:
                sim.run(1)
            got = sim.get_accel()[targets[:len(part)]]
            want = _wanted(part, off, m)
            wrong += list(part[((got != want) & ~(np.isnan(got) & np.isnan(want))).any(axis=1)])
        if batch:
            batch.close()
    return [hex(int(w.view(np.uint32))) for w in wrong]


def test_every_mantissa(gs):
    """Both exponent parities."""
    for first in range(0x3f800000, 0x40800000, 1 << 20):
        x = np.arange(first, first + (1 << 20), dtype=np.uint32).view(np.float32)
        assert _wrong(gs, x, 4096, 0, 1.0, 1e-10) == []


# the split kernel, the one for large systems, and the batched one; either lane of the packed
# pair; the ends of the range of the kernels' own root and reciprocal, [2^-100, 2^100]
@pytest.mark.parametrize("n,batched", [(4096, False), (16448, False), (4096, True)])
@pytest.mark.parametrize("source", [0, 1, 3])
@pytest.mark.parametrize("scale,softening,m", [(1.0, 1e-10, 1.0), (2.0 ** -50, 2.0 ** -72, 1.0),
                                               (2.0 ** -50, 2.0 ** -72, 2.0 ** -60), (2.0 ** 49, 1e-10, 1.0)])
def test_all_ones_mantissas_and_a_sample(gs, n, batched, source, scale, softening, m):
    tails = np.concatenate([np.arange(e - 64, e + 64) for e in (0x3f800040, 0x40000000, 0x40800000 - 64)])
    some = np.random.default_rng(7).integers(0x3f800000, 0x40800000, 100000)
    x = np.concatenate([tails, some]).astype(np.uint32).view(np.float32)
    assert _wrong(gs, x, n, source, scale, softening, m, batched) == []


@pytest.mark.parametrize("bits", [0x3f7ffffe, 0x3f7fffff, 0x407ffffe, 0x407fffff, 0x4f7ffffe])
def test_two_particles_as_oracle(gs, orc, bits):
    x = np.array([bits], np.uint32).view(np.float32)
    pos = np.concatenate([np.zeros((1, 2), np.float32), _offsets(x)])
    vel, mass = np.zeros_like(pos), np.array([1, 0], np.float32)
    st = orc.State(pos, vel, mass)
    orc.direct_step(st, dt=1.0, softening=1e-10)
    with gs.Simulation(pos, vel, mass, algorithm=gs.DIRECT_SUM, math_mode=gs.MATH_REFERENCE, softening_len=1e-10,
                       **REF) as sim:
        sim.run(1)
        for g, o in zip(sim.get_particles(), st.current()):
            np.testing.assert_array_equal(g, o)
