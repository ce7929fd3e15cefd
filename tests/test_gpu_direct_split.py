"""The direct sum's kernels at the edges of their ranges: small systems (32 targets a block,
source tiles split over its warps), large ones (i-tiles x j-chunks), the form of 1/sqrt that
also takes subnormal distances, and REFERENCE math's factors outside the range of its own
root and reciprocal.

FAST math: the oracle's FP64 sum within the 2e-6 RMS of the other direct-sum tests;
REFERENCE math: the oracle's bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rms(acc, a64):
    den = np.linalg.norm(a64, axis=1)
    return np.sqrt(np.mean((np.linalg.norm(acc.astype(np.float64) - a64, axis=1) / den) ** 2))


# one tile; fewer tiles than parts; parts of uneven length; the last small and the first
# large system; a last i-tile that is not full
@pytest.mark.parametrize("n", [64, 960, 1088, 12288, 12289, 13000, 33333])
@pytest.mark.parametrize("plain", [False, True])
def test_fast_sizes(gs, orc, n, plain):
    pos, vel, mass = gs.generate(gs.GEN_EXP_DISK_COLLISION, n, size=100.0, seed=900 + n)
    flags = gs.FLAG_RECORD_ACCEL | (gs.FLAG_PLAIN_SUM if plain else 0)
    targets = np.unique(np.r_[0:min(n, 64), np.arange(0, n, max(1, n // 500)), n - 1]).astype(np.uint32)
    with gs.Simulation(pos, vel, mass, algorithm=gs.DIRECT_SUM, flags=flags) as sim:
        sim.run(1)
        acc = sim.get_accel()[targets]
    P, _, M = orc.pad_state(pos, vel, mass)
    assert _rms(acc, orc.direct_accel_f64(P, M, targets=targets)) < 2e-6


@pytest.mark.parametrize("n", [100, 13000])
def test_fast_subnormal_softening(gs, orc, n):
    """eps^2 = 1e-40 is subnormal: a particle's own term is its mass times (1e20)^3, finite for
    these masses, and must not become an infinity times zero."""
    pos, vel, _ = gs.generate(gs.GEN_UNIFORM_DISK, n, size=100.0, seed=5)
    mass = np.full(n, 1e-25, np.float32)
    with gs.Simulation(pos, vel, mass, algorithm=gs.DIRECT_SUM, softening_len=1e-20,
                       flags=gs.FLAG_RECORD_ACCEL) as sim:
        sim.run(1)
        acc = sim.get_accel()
        sim.set_particles(pos, vel, mass)
        t = np.arange(0, n, max(1, n // 200), dtype=np.uint32)
        a64 = sim.accel_f64(t)
    assert np.isfinite(acc).all()
    assert _rms(acc[t], a64) < 2e-6


@pytest.mark.parametrize("n", [64, 4160, 16448])
@pytest.mark.parametrize("scale,mass_scale,softening", [(1.0, 1.0, 0.2), (1e13, 1.0, 0.2), (1e17, 1.0, 0.2),
                                                        (1e19, 1.0, 0.2), (1e-17, 1e-25, 1e-19)])
def test_reference_ranges_bit_exact(gs, orc, n, scale, mass_scale, softening):
    """Distances squared around 2^100 and 2^-100, where the library's root and reciprocal take
    over, and beyond the FP32 range."""
    pos, vel, mass = gs.generate(gs.GEN_UNIFORM_DISK, n, size=100.0, seed=17)
    pos = (pos * np.float32(scale)).astype(np.float32)
    mass = (mass * np.float32(mass_scale)).astype(np.float32)
    st = orc.State(pos, vel, mass)
    with gs.Simulation(pos, vel, mass, algorithm=gs.DIRECT_SUM, math_mode=gs.MATH_REFERENCE,
                       softening_len=softening) as sim:
        for _ in range(2):
            sim.run(1)
            orc.direct_step(st, softening=softening)
        for g, o in zip(sim.get_particles(), st.current()):
            np.testing.assert_array_equal(g, o)


def test_steps_chained_and_single_agree(gs):
    """Steps launched behind one another and steps submitted one by one: the same bits."""
    for n in (1000, 13000):
        pos, vel, mass = gs.generate(gs.GEN_GALAXY, n, size=100.0, seed=3)
        with gs.Simulation(pos, vel, mass, algorithm=gs.DIRECT_SUM) as a, \
                gs.Simulation(pos, vel, mass, algorithm=gs.DIRECT_SUM) as b:
            a.run(40)
            for _ in range(40):
                b.run(1)
                b.sync()
            for x, y in zip(a.get_particles(), b.get_particles()):
                np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32))
