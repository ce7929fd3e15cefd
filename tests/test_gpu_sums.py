"""Monopole moments of the reference rule: the largest system that one block sums and the next
larger, finest cells of many particles, and a small system with more records than the block's
shared memory holds.  Every record bit-identical to the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(gs, kind, n):
    if kind == "clumps":  # finest cells of hundreds of particles
        rng = np.random.default_rng(n)
        pos = (rng.uniform(-90, 90, (40, 2))[rng.integers(0, 40, n)] + rng.normal(0, 0.05, (n, 2))).astype(np.float32)
        return pos, np.zeros_like(pos), rng.uniform(1, 10, n).astype(np.float32)
    if kind == "pairs":  # pairs that share every cell but the finest: a node per level each
        rng = np.random.default_rng(n)
        p = rng.uniform(-90, 90, ((n + 1) // 2, 2))
        pos = np.repeat(p, 2, axis=0)[:n].astype(np.float32)
        pos[1::2] += np.float32(1e-3)
        return pos, np.zeros_like(pos), np.ones(n, np.float32)
    return gs.generate(gs.GEN_SPIRAL, n, size=100.0, seed=n)


@pytest.mark.parametrize("kind,n", [("spiral", 3072), ("spiral", 3073), ("spiral", 30000), ("clumps", 2000),
                                    ("clumps", 20000), ("pairs", 3000), ("pairs", 12000), ("spiral", 100000)])
@pytest.mark.parametrize("box,bits,safe", [(0, 0, False), (1, 12, False), (1, 15, True)])
def test_sums_bit_exact(gs, orc, kind, n, box, bits, safe):
    pos, vel, mass = _inputs(gs, kind, n)
    st = orc.State(pos, vel, mass)
    prm = gs.default_params(algorithm=gs.BARNES_HUT, box_mode=box, math_mode=gs.MATH_REFERENCE, key_bits=bits,
                            flags=gs.FLAG_SAFE_RADIUS if safe else 0)
    with gs.Simulation(pos, vel, mass, params=prm) as sim:
        sim.run(1)
        o = orc.bh_step(st, box_mode=box, key_bits=bits, flags=orc.SAFE_RADIUS if safe else 0)
        t = sim.bh_tree()
    assert t["tree_size"] == o["tree_size"]
    for k in ("skip", "radius", "pos", "mass"):
        np.testing.assert_array_equal(t[k], o[k], err_msg=k)
