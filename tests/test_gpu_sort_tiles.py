"""Sort tiles of a system sorted alone: sizes around one tile and around the bound between
the tiles of 1024 keys and the shape's.  Every record bit-identical to the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 33000, 131072, 131073])
def test_tree_bit_exact(gs, orc, n):
    pos, vel, mass = gs.generate(gs.GEN_SPIRAL, n, size=100.0, seed=n)
    st = orc.State(pos, vel, mass)
    prm = gs.default_params(algorithm=gs.BARNES_HUT, math_mode=gs.MATH_REFERENCE)
    with gs.Simulation(pos, vel, mass, params=prm) as sim:
        sim.run(1)
        o = orc.bh_step(st)
        t = sim.bh_tree()
    assert t["tree_size"] == o["tree_size"]
    for k in ("skip", "radius", "pos", "mass"):
        np.testing.assert_array_equal(t[k], o[k], err_msg=k)
