"""gs_footprint of Barnes-Hut systems: what a server with a budget admits.  A change of the
kernels' scratch must not make systems larger than these."""
import pytest

# particles: monopoles in the fixed box; relative criterion with 24-bit and with 30-bit keys
BYTES = {64: (46756, 67492, 77476), 1024: (342436, 616868, 734628), 2048: (641448, 1182632, 1417128),
         20000: (5025736, 10008008, 12301768), 131072: (28004004, 59319972, 74327716),
         131073: (28018084, 59348644, 74364580), 500000: (92021876, 207546996, 264801396)}


@pytest.mark.parametrize("n", BYTES)
def test_no_larger(gs, n):
    for want, prm in zip(BYTES[n], (dict(), dict(box_mode=1, flags=0x170), dict(box_mode=1, key_bits=15, flags=0x170))):
        p = gs.default_params(algorithm=gs.BARNES_HUT, **prm)
        assert 0 < gs.footprint(p, n) <= want
