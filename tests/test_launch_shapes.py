"""Every launch shape that hp_tune accepts has to launch, and to give the oracle's bits: Move's ring of chunks asks for
up to 70 KB of shared memory at 16 warps per CTA, which a launch gets only after asking for it.  The autotuner tries
such shapes on a batch and has to leave the batch where it stood."""
import numpy as np
import pytest

import hpic
import oracle
from hpic.decks import ccp_deck
from test_gpu_fluid import fluid_deck

pytestmark = pytest.mark.gpu

GRIDS = ("EX", "EY", "PHI", "PHI_POIS", "DEN", "SOURCE", "PCG_X", "PCG_B", "AVE_DEN", "AVE_PHI", "COND_CHARGE", "MCC_COUNT",
         "EEDF", "AVE_SOURCE", "AVE_EX", "AVE_EY", "FLUID_CELL_DEN", "FLUID_DEN", "FLUID_SOURCE", "FLUID_FLUX_X",
         "FLUID_FLUX_Y")


def raw(a):
    return np.ascontiguousarray(a).tobytes()


@pytest.mark.parametrize("unroll", [1, 2, 4])
@pytest.mark.parametrize("warps", [1, 4, 8, 10, 11, 15, 16])  # 48 KB of rings: between 10 and 11 (unroll 4), 15 and 16 (unroll 1) warps
def test_move_shapes_bit_exact(warps, unroll):
    deck = ccp_deck(33, 17, 0.01, 0.005, ppc=70, voltage=200.0)  # cells of two to four chunks
    kw = dict(seed=12, field_mode=2, move_mode=1)
    S = hpic.Setup(deck, **kw)
    case = hpic.Case(setup=S, **kw)
    case.set_tune(warps_per_block_particles=warps, move_unroll=unroll)
    o = oracle.Oracle(S.table, S.info, case.opts, 32)
    for s in range(S.info.nsp):
        counts, arrs = S.particles(s, layout=0)
        o.set_particles(s, counts, *arrs)
    o.DepositBasic()
    case.step(3)
    o.run(0, 3, accumulate=True)
    for s in range(S.info.nsp):
        gc, ga = case.particles(s)
        oc, oa = o.particles(s)
        assert np.array_equal(gc, oc)
        for a, b in zip(ga, oa):
            assert raw(a) == raw(b), s
    for g in ("EX", "EY", "DEN"):
        assert raw(case.grid(g)) == raw(o.grid(g)), g
    assert case.status() == 0
    case.close()


def batch(field_mode):
    decks = [fluid_deck(ccp_deck(nx, ny, (nx - 1) * 3.125e-4, (ny - 1) * 3.125e-4, ppc=ppc, pressure_torr=0.1,
                                 voltage=200.0)) for nx, ny, ppc in ((33, 17, 20), (66, 34, 9))]
    cases = [hpic.Case(d, seed=5 + k, field_mode=field_mode, move_mode=1, eedf_every=2) for k, d in enumerate(decks)]
    b = hpic.Batch(cases)
    b.step(9)  # past two averaging windows: the continuity solve runs in every trial's steps
    return b


def same_state(a, b):
    for c, d in zip(a.cases, b.cases):
        for g in GRIDS:
            assert raw(c.grid(g)) == raw(d.grid(g)), g
        for s in range(c.info.nsp):
            (nc, ac), (nd, ad) = c.particles(s), d.particles(s)
            assert np.array_equal(nc, nd)
            assert all(raw(u) == raw(v) for u, v in zip(ac, ad))
        assert c.info.tstep == d.info.tstep and c.pushes() == d.pushes()
        assert c.status() == d.status() == 0


@pytest.mark.parametrize("field_mode", [0, 2])
def test_autotune_leaves_the_batch_where_it_stood(field_mode):
    tuned, plain = batch(field_mode), batch(field_mode)
    same_state(tuned, plain)
    tuned.autotune()
    same_state(tuned, plain)
    if field_mode == 2:  # the PCG's sums follow its launch shape, so there the next steps may round differently
        tuned.step(5)
        plain.step(5)
        same_state(tuned, plain)
    tuned.close()
    plain.close()
