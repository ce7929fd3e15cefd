"""The reference rule's walk at the edges of its kernels: a tree copied into shared memory, a
small system whose tree does not fit there, systems walked through windows, a last block
that is not full, and a softening whose square is subnormal.

REFERENCE math: the oracle's bits and counts; FAST math as in the other Barnes-Hut tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 8192 particles with 15 bits per axis: more than 10,240 records, walked through windows
@pytest.mark.parametrize("n,box,bits", [(1, 1, 12), (40, 0, 12), (129, 1, 12), (5000, 0, 12), (8192, 0, 12), (8192, 1, 15),
                                        (8193, 1, 12), (20000, 0, 12)])
@pytest.mark.parametrize("count", [False, True])
def test_rule_walk_bit_exact(gs, orc, n, box, bits, count):
    pos, vel, mass = gs.generate(gs.GEN_RANDOM if n > 1000 else gs.GEN_UNIFORM_DISK, n, size=100.0, seed=n)
    st = orc.State(pos, vel, mass)
    prm = gs.default_params(algorithm=gs.BARNES_HUT, box_mode=box, math_mode=gs.MATH_REFERENCE, key_bits=bits,
                            flags=gs.FLAG_COUNT_INTERACTIONS if count else 0)
    with gs.Simulation(pos, vel, mass, params=prm) as sim:
        for _ in range(2):
            sim.reset_stats()
            sim.run(1)
            o = orc.bh_step(st, box_mode=box, key_bits=bits if box else 0)
            if count:
                s = sim.stats()
                assert (s.interactions, s.warp_visits) == (o["interactions"], o["warp_visits"])
        for g, c in zip(sim.get_particles(), st.current()):
            np.testing.assert_array_equal(g, c)


@pytest.mark.parametrize("n", [500, 20000])
def test_rule_walk_subnormal_softening(gs, orc, n):
    """eps^2 = 1e-40: a particle's own leaf term is finite for these masses."""
    pos, vel, _ = gs.generate(gs.GEN_UNIFORM_DISK, n, size=100.0, seed=8)
    mass = np.full(n, 1e-25, np.float32)
    acc = {}
    for mm in (gs.MATH_FAST, gs.MATH_REFERENCE):
        prm = gs.default_params(algorithm=gs.BARNES_HUT, math_mode=mm, softening_len=1e-20,
                                flags=gs.FLAG_RECORD_ACCEL)
        with gs.Simulation(pos, vel, mass, params=prm) as sim:
            sim.run(1)
            acc[mm] = sim.get_accel().astype(np.float64)
    ref = acc[gs.MATH_REFERENCE]
    assert np.isfinite(acc[gs.MATH_FAST]).all()
    den = np.linalg.norm(ref, axis=1)
    assert np.max(np.linalg.norm(acc[gs.MATH_FAST] - ref, axis=1) / den) < 1e-4
