"""The group walk on one and on two warps per group: sizes around the bound between them, a
walk whose stack outgrows its shared-memory window, in both lists lengths, alone and in
batches.  REFERENCE math against the oracle, bit for bit; FAST math on two warps against
the counting kernels, which walk a group on one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ACC, REL = 0x70, 0x170


def _prm(gs, **kw):
    base = dict(algorithm=gs.BARNES_HUT, box_mode=1, math_mode=gs.MATH_REFERENCE, accuracy_parameter=1.0,
                relative_accuracy=0.006, relative_theta_floor=0.2, flags=REL)
    base.update(kw)
    return gs.default_params(**base)


@pytest.mark.parametrize("n", [1, 63, 65, 136192, 136193])
def test_sizes_bit_exact(gs, orc, n):
    pos, vel, mass = gs.generate(gs.GEN_UNIFORM_DISK, n, size=100.0, seed=n)
    st = orc.State(pos, vel, mass)
    with gs.Simulation(pos, vel, mass, params=_prm(gs)) as sim:
        for _ in range(2):
            sim.run(1)
            orc.bh_step(st, box_mode=1, theta=1.0, flags=orc.ACCURATE | orc.RELATIVE_MAC, rel_alpha=0.006,
                        rel_floor=0.2, keep_tree=False)
        for g, c in zip(sim.get_particles(), st.current()):
            np.testing.assert_array_equal(g, c)


@pytest.mark.parametrize("warps,short", [(1, 0), (2, 0), (2, 1), (4, 0)])
@pytest.mark.parametrize("count", [False, True])
def test_deep_stack_bit_exact(gs, orc, warps, short, count):
    """theta = 0 opens every node: a stack of more records than the 256 that shared memory
    holds."""
    n = 16000
    pos, vel, mass = gs.generate(gs.GEN_UNIFORM_DISK, n, size=100.0, seed=77)
    st = orc.State(pos, vel, mass)
    flags = ACC | (gs.FLAG_COUNT_INTERACTIONS if count else 0)
    with gs.Simulation(pos, vel, mass, params=_prm(gs, accuracy_parameter=0.0, flags=flags)) as sim:
        sim.set_shape(force_warps=warps, force_short_lists=short)
        sim.run(1)
        o = orc.bh_step(st, box_mode=1, theta=0.0, flags=orc.ACCURATE, keep_tree=False)
        assert o["max_stack"] > 256
        if count:
            assert sim.stats().interactions == o["interactions"]
        for g, c in zip(sim.get_particles(), st.current()):
            np.testing.assert_array_equal(g, c)


@pytest.mark.parametrize("sizes", [[300, 5000, 20000], [140000, 7000, 100]])
def test_batches_as_alone(gs, sizes):
    """FAST math, batches whose groups take two warps each and one: each member as alone."""
    inputs = [gs.generate(gs.GEN_SPIRAL, n, size=100.0, seed=n) for n in sizes]
    prm = _prm(gs, math_mode=gs.MATH_FAST)
    alone = []
    for p in inputs:
        with gs.Simulation(*p, params=prm) as s:
            s.run(3)
            alone.append(s.get_particles())
    sims = [gs.Simulation(*p, params=prm) for p in inputs]
    with gs.Batch(sims) as b:
        b.run(3)
        b.sync()
    for s, want in zip(sims, alone):
        for g, c in zip(s.get_particles(), want):
            np.testing.assert_array_equal(g.view(np.uint32), c.view(np.uint32))
        s.close()
