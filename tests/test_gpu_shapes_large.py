"""Launch shapes at sizes whose kernels read every field: trees above 8,192 (3,072 with
quadrupoles) particles, sort tiles above 131,072, the moments launch from 313,344, direct sums
above 12,288.  Barnes-Hut in REFERENCE math bit-identical to the oracle, direct sums as with the
other number of targets per thread, members of a batch as alone."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
REL = dict(box_mode=1, relative_accuracy=0.006, relative_theta_floor=0.2, flags=0x170)
FORCE = ((1, 0), (2, 0), (2, 1), (4, 0))


def _words(sim):
    return np.concatenate([a.ravel() for a in sim.padded_state()[:3]]).view(np.uint32)


# 10,000: 1024-key tiles whatever the shape says; 140,000: the shape's; 320,000: a moments launch
# whose size is the shape's
@pytest.mark.parametrize("n,rule", [(10000, True), (10000, False), (140000, True), (140000, False), (320000, True)])
def test_every_field_bit_exact(gs, orc, n, rule):
    pos, vel, mass = gs.generate(gs.GEN_SPIRAL, n, size=100.0, seed=61)
    prm = gs.default_params(algorithm=1, math_mode=1, **({} if rule else REL))
    okw = dict(box_mode=0) if rule else dict(box_mode=1, flags=orc.ACCURATE | orc.RELATIVE_MAC, rel_alpha=0.006,
                                             rel_floor=0.2)
    st = orc.State(pos, vel, mass)
    want = []
    for _ in range(2):
        orc.bh_step(st, theta=1.0, keep_tree=False, **okw)
        want.append(np.concatenate([a.ravel() for a in (st.pos[st.inp], st.vel[st.inp], st.mass[st.inp])])
                    .view(np.uint32).copy())
    for j, (kpt, lb, scan, mom) in enumerate(itertools.product((8, 16), (8, 16, 32), (32, 64, 128), (1, 2))):
        warps, short = FORCE[j % len(FORCE)]
        with gs.Simulation(pos, vel, mass, params=prm) as sim:
            sim.set_shape(sort_keys_per_thread=kpt, sort_lookback=lb, scan_lookback=scan, force_warps=warps,
                          force_short_lists=short, moment_blocks_per_sm=mom)
            for k in range(2):
                sim.run(1)
                assert np.array_equal(_words(sim), want[k]), (kpt, lb, scan, mom, warps, short, k)


@pytest.mark.parametrize("n", [12289, 33333])
@pytest.mark.parametrize("plain,softening", [(False, 0.2), (True, 0.2), (False, 1e-20)])
def test_direct_targets_change_no_bit(gs, orc, n, plain, softening):
    """Alone and in a batch, for every j-split that the creation shape's scratch holds; each within
    FP32 tolerance of the oracle's sequential sum."""
    pos, vel, mass = gs.generate(gs.GEN_UNIFORM_DISK, n, size=100.0, seed=62)
    if softening < 0.1:
        mass[:] = 1e-25  # a particle's own term, its mass times (1e20)^3, stays finite
    kw = dict(algorithm=gs.DIRECT_SUM, softening_len=softening, flags=gs.FLAG_PLAIN_SUM if plain else 0)
    other = gs.generate(gs.GEN_UNIFORM_DISK, 2000, size=100.0, seed=63)
    st = orc.State(pos, vel, mass)
    for _ in range(2):
        orc.direct_step(st, softening=softening)
    ov = st.current()[1]
    for bps in (4, 8, 12):
        got = []
        for ipt in (2, 4):
            with gs.Simulation(pos, vel, mass, **kw) as sim:
                sim.set_shape(direct_targets=ipt, direct_blocks_per_sm=bps)
                sim.run(2)
                got.append(_words(sim))
                assert np.max(np.abs(sim.get_particles()[1] - ov)) <= 1e-4 * np.abs(ov).max()
            with gs.Simulation(pos, vel, mass, **kw) as a, gs.Simulation(*other, **kw) as b:
                a.set_shape(direct_blocks_per_sm=bps)
                with gs.Batch([a, b]) as batch:
                    batch.set_shape(direct_targets=ipt)
                    batch.run(2)
                    batch.sync()
                got.append(_words(a))
        for g in got[1:]:
            assert np.array_equal(g, got[0]), bps
