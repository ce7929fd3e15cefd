"""Group walks whose last groups take two warps: the same bits as with every group on one warp
(blocks of four), around the sizes where the number of such groups changes, odd numbers of
groups, costly groups on warp pairs, and the first step's estimate pass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
GROUP, ACC, REL = 0x40, 0x70, 0x170


@pytest.mark.parametrize("n", [136193, 136257, 194560, 194561, 300000])
@pytest.mark.parametrize("flags", [GROUP, ACC, REL])
def test_as_on_one_warp(gs, n, flags):
    assert flags == ACC or flags in (gs.FLAG_GROUP_WALK, gs.FLAGS_ACCURATE | gs.FLAG_RELATIVE_MAC)
    pos, vel, mass = gs.generate(gs.GEN_SPIRAL, n, size=100.0, seed=n)
    got = []
    for warps in (2, 4):
        prm = gs.default_params(algorithm=gs.BARNES_HUT, box_mode=1, accuracy_parameter=0.6, relative_accuracy=0.006,
                                relative_theta_floor=0.2, flags=flags)
        with gs.Simulation(pos, vel, mass, params=prm) as sim:
            sim.set_shape(force_warps=warps)
            sim.run(3)
            got.append(sim.get_particles())
    for g, c in zip(*got):
        np.testing.assert_array_equal(g.view(np.uint32), c.view(np.uint32))
