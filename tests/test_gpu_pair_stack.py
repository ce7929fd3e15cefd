"""Costly groups (relative criterion, 2^18 particles) whose warp pair's stack outgrows its 512
entries in shared memory more than once, alone and in a batch: bit-identical to the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_deep_pair_stack_bit_exact(gs, orc):
    """A disk that is its own mirror image: the field nearly cancels at its centre, so the groups
    there are costly, and a small alpha makes them open most of the tree."""
    n, alpha, floor = 262144, 1e-4, 0.02
    rng = np.random.default_rng(1)
    r, a = 100 * np.sqrt(rng.uniform(size=n // 2 - 32)), rng.uniform(0, 2 * np.pi, n // 2 - 32)
    half = np.concatenate([np.stack([r * np.cos(a), r * np.sin(a)], 1), rng.normal(0, 1e-3, (32, 2))])
    pos = np.concatenate([half, -half]).astype(np.float32)
    vel, mass = np.zeros_like(pos), np.ones(n, np.float32)
    st = orc.State(pos, vel, mass)
    okw = dict(box_mode=1, theta=1.0, flags=orc.ACCURATE | orc.RELATIVE_MAC, rel_alpha=alpha, rel_floor=floor,
               keep_tree=False)
    prm = gs.default_params(algorithm=gs.BARNES_HUT, box_mode=1, math_mode=gs.MATH_REFERENCE, accuracy_parameter=1.0,
                            relative_accuracy=alpha, relative_theta_floor=floor, flags=0x170)
    with gs.Simulation(pos, vel, mass, params=prm) as sim, gs.Simulation(pos, vel, mass, params=prm) as member:
        sim.run(2)
        with gs.Batch([member]) as batch:
            batch.run(2)
            batch.sync()
        stacks = [orc.bh_step(st, **okw)["max_stack"] for _ in range(2)]
        # the second step has known |a|, hence pairs; single walks stay below 512 (the first step)
        assert stacks[0] < 512 and stacks[1] > 512 + 256
        for s in (sim, member):
            for g, o in zip(s.get_particles(), st.current()):
                np.testing.assert_array_equal(g, o)
