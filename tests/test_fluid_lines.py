"""The sweeps of the continuity solve at the edges of their loops: lines of a few cells, of whole and broken batches of
8 cells (the back substitution) and of 32 and 128 cells (the loads), against the oracle, bit for bit."""
import pytest

import hpic
import oracle
from hpic.decks import ccp_deck
from test_gpu_fluid import check, fluid_deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(5, 6), (10, 9), (11, 18), (33, 34), (130, 32), (129, 35), (258, 8)])
def test_sweeps_bit_exact(nx, ny):
    deck = fluid_deck(ccp_deck(nx, ny, (nx - 1) * 3.125e-4, (ny - 1) * 3.125e-4, ppc=6, pressure_torr=0.1,
                               voltage=200.0), average_iter=2)
    kw = dict(seed=21, field_mode=2, move_mode=1, cap_per_cell=256)
    S = hpic.Setup(deck, **kw)
    case = hpic.Case(setup=S, **kw)
    o = oracle.Oracle(S.table, S.info, case.opts, 32)
    for s in range(S.info.nsp):
        counts, arrs = S.particles(s, layout=0)
        o.set_particles(s, counts, *arrs)
    o.DepositBasic()
    for k in range(2):
        case.step(4)
        o.run(4 * k, 4, accumulate=True)
        check(case, o, f"{nx}x{ny}, step {4 * (k + 1)}")
    case.close()
