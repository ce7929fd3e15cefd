"""The tree's separate kernels (above the 8,192 particles that one block takes) on removed
particles, NaN positions, an empty system, one full cell and pairs with a node per level; and
the largest one-block system beside the next.  Every record bit-identical to the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(gs, kind, n):
    rng = np.random.default_rng(n)
    vel, ones = np.zeros((n, 2), np.float32), np.ones(n, np.float32)
    if kind == "outside":  # a third beyond the fixed box: removed
        return rng.uniform(-750, 750, (n, 2)).astype(np.float32), vel, rng.uniform(1, 10, n).astype(np.float32)
    if kind == "nan":  # outside the fixed box by the shader's comparisons
        pos = rng.uniform(-90, 90, (n, 2)).astype(np.float32)
        pos[::100, 0] = np.nan
        pos[50::1000] = np.nan
        return pos, vel, ones
    if kind == "gone":  # nothing left
        return np.full((n, 2), 900, np.float32), vel, ones
    if kind == "point":  # every particle in one finest cell
        return np.full((n, 2), 3.25, np.float32), vel, ones
    if kind == "pairs":
        pos = np.repeat(rng.uniform(-90, 90, ((n + 1) // 2, 2)), 2, axis=0)[:n].astype(np.float32)
        pos[1::2] += np.float32(1e-3)
        return pos, vel, ones
    return gs.generate(gs.GEN_SPIRAL, n, size=100.0, seed=n)


SYSTEMS = [("spiral", 8192), ("spiral", 8193), ("outside", 8193), ("outside", 40000), ("nan", 8192), ("nan", 9000),
           ("gone", 9000), ("point", 8193), ("point", 20000), ("pairs", 8193), ("pairs", 30001)]
MODES = [(0, 0, 0), (1, 12, 0), (1, 15, 0x20), (0, 0, 0x40), (0, 0, 0x70), (1, 12, 0x70)]


# a NaN position has no cell in the bounding box
@pytest.mark.parametrize("kind,n,box,bits,flags",
                         [s + m for s in SYSTEMS for m in MODES if s[0] != "nan" or m[0] == 0])
def test_tree_bit_exact(gs, orc, kind, n, box, bits, flags):
    pos, vel, mass = _inputs(gs, kind, n)
    st = orc.State(pos, vel, mass)
    prm = gs.default_params(algorithm=gs.BARNES_HUT, box_mode=box, math_mode=gs.MATH_REFERENCE, key_bits=bits,
                            flags=flags)
    oflags = ((orc.QUADRUPOLE if flags & gs.FLAG_QUADRUPOLE else 0) | (orc.SAFE_RADIUS if flags & gs.FLAG_SAFE_RADIUS else 0)
              | (orc.GROUP_WALK if flags & gs.FLAG_GROUP_WALK else 0))
    with gs.Simulation(pos, vel, mass, params=prm) as sim:
        for _ in range(2):  # the second step on the first one's buffers
            sim.run(1)
            o = orc.bh_step(st, box_mode=box, key_bits=bits, flags=oflags)
        t = sim.bh_tree()
        got = sim.get_particles()
    assert t["tree_size"] == o["tree_size"]
    for k in ("keys", "sorted_src", "skip", "radius", "pos", "mass") + (("quad",) if flags & gs.FLAG_QUADRUPOLE else ()):
        np.testing.assert_array_equal(t[k], o[k], err_msg=k)
    for g, r in zip(got, st.current()):
        np.testing.assert_array_equal(g, r)
