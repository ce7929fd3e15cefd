"""The one-block tree of small systems: sizes around its vectors and its largest system, both
boxes, removed particles, every key length, monopole and quadrupole moments.  Every record
bit-identical to the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(gs, kind, n):
    rng = np.random.default_rng(n)
    if kind == "outside":  # a third beyond the fixed box: removed
        pos = rng.uniform(-750, 750, (n, 2)).astype(np.float32)
        return pos, np.zeros_like(pos), rng.uniform(1, 10, n).astype(np.float32)
    if kind == "gone":  # nothing left
        return np.full((n, 2), 900, np.float32), np.zeros((n, 2), np.float32), np.ones(n, np.float32)
    if kind == "point":  # every particle in one finest cell
        return np.full((n, 2), 3.25, np.float32), np.zeros((n, 2), np.float32), np.ones(n, np.float32)
    if kind == "pairs":  # pairs that share every cell but the finest: a node per level each
        p = rng.uniform(-90, 90, ((n + 1) // 2, 2))
        pos = np.repeat(p, 2, axis=0)[:n].astype(np.float32)
        pos[1::2] += np.float32(1e-3)
        return pos, np.zeros_like(pos), np.ones(n, np.float32)
    return gs.generate(gs.GEN_SPIRAL, n, size=100.0, seed=n)


@pytest.mark.parametrize("kind,n", [("spiral", 1), ("spiral", 2), ("outside", 65), ("gone", 100), ("point", 500),
                                    ("outside", 2048), ("pairs", 2049), ("outside", 3072),
                                    ("spiral", 3073), ("spiral", 4096), ("outside", 4097), ("pairs", 5000),
                                    ("point", 8192), ("pairs", 8192), ("spiral", 8193)])
@pytest.mark.parametrize("box,bits,quad", [(0, 0, False), (1, 12, False), (0, 0, True), (1, 12, True), (1, 15, True)])
def test_tree_bit_exact(gs, orc, kind, n, box, bits, quad):
    pos, vel, mass = _inputs(gs, kind, n)
    st = orc.State(pos, vel, mass)
    flags = gs.FLAGS_ACCURATE if quad else 0
    prm = gs.default_params(algorithm=gs.BARNES_HUT, box_mode=box, math_mode=gs.MATH_REFERENCE, key_bits=bits,
                            flags=flags)
    with gs.Simulation(pos, vel, mass, params=prm) as sim:
        for _ in range(2):  # the second step on the first one's buffers
            sim.run(1)
            o = orc.bh_step(st, box_mode=box, key_bits=bits,
                            flags=(orc.QUADRUPOLE | orc.SAFE_RADIUS | orc.GROUP_WALK) if quad else 0)
        t = sim.bh_tree()
        gp, gv, gm = sim.get_particles()
    assert t["tree_size"] == o["tree_size"]
    for k in ("keys", "sorted_src", "skip", "radius", "pos", "mass") + (("quad",) if quad else ()):
        np.testing.assert_array_equal(t[k], o[k], err_msg=k)
    op, ov, om = st.current()
    for g, r in ((gp, op), (gv, ov), (gm, om)):
        np.testing.assert_array_equal(g, r)
