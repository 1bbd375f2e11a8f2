"""The separable solve (field_mode 2) at the edges of its forms: clusters of 8 and of 16 CTAs with odd strips and
CTAs without one, every padded row length, and one launch per product past a cluster's range.  Every output of a
product is a sum in k order, so all of them give the oracle's bits."""
import numpy as np
import pytest

import hpic
import oracle
from hpic.decks import ccp_deck

pytestmark = pytest.mark.gpu

SIZES = [
    (5, 6),      # fewer columns than CTAs
    (33, 34),    # rows of exactly 32 unknowns, the last CTA's strip one column
    (128, 40),   # the widest strips of an 8-CTA cluster, rows padded from 38 to 64
    (129, 41),   # one column over: 16 CTAs
    (40, 82),    # rows padded to 96
    (96, 106),   # near the most unknowns of a cluster, rows padded to 128
    (12, 130),   # the longest rows of a cluster
    (12, 131),   # past them: one launch per product, one column of tiles
    (130, 82),   # just past the most unknowns of a cluster: tiles cut along both edges
    (202, 101),
    (20, 1060),  # many rows of tiles
]


@pytest.mark.parametrize("nx,ny", SIZES)
def test_separable_solve_bit_exact(nx, ny):
    deck = ccp_deck(nx, ny, (nx - 1) * 3.125e-4, (ny - 1) * 3.125e-4, ppc=3, voltage=150.0)
    kw = dict(seed=9, field_mode=2, gas_temp_mode=1)
    S = hpic.Setup(deck, **kw)
    case = hpic.Case(setup=S, **kw)
    assert case.info.field_mode == 2
    o = oracle.Oracle(S.table, S.info, case.opts, 32)
    for s in range(S.info.nsp):
        counts, arrs = S.particles(s, layout=0)
        o.set_particles(s, counts, *arrs)
    o.DepositBasic()
    for t in (1, 2):
        case.set_tstep(t)
        case.Field()
        o.Field(t)
        for g in ("PHI_POIS", "PHI", "EX", "EY"):
            a, b = case.grid(g), o.grid(g)
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (t, g)
    assert case.status() == 0
    assert 0 <= case.field_residual() < 1e-8
    case.close()


def test_sizes_together_in_one_batch():
    """The forms side by side in one launch sequence give each case's own bits."""
    decks = [ccp_deck(nx, ny, (nx - 1) * 3.125e-4, (ny - 1) * 3.125e-4, ppc=3) for nx, ny in ((33, 17), (129, 40), (202, 101))]
    alone, mixed = [[hpic.Case(d, seed=3 + k, field_mode=2, move_mode=1) for k, d in enumerate(decks)] for _ in range(2)]
    b = hpic.Batch(mixed)
    b.step(3)
    for c in alone:
        c.step(3)
    for a, m in zip(alone, mixed):
        assert np.array_equal(a.grid("PHI").view(np.uint32), m.grid("PHI").view(np.uint32))
        assert a.field_residual() == m.field_residual()
    b.close()
