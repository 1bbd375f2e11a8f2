"""Move, the re-binning and the deposit where their chunks of 32, groups of cells and rare paths meet: cells of 0, 1,
31, 32, 33, 63 to 65 and 96 to 130 particles, cells that all leave, stay or leave after a chunk of stayers, offsets of
exactly 0, -0 and just below 1, and cells whose movers come without movers in the step before.  Against the oracle,
bit for bit."""
import numpy as np
import pytest

import hpic
import oracle
from hpic.decks import ccp_deck

pytestmark = pytest.mark.gpu

COUNTS = [0, 1, 31, 32, 33, 63, 64, 65, 96, 97, 127, 128, 130, 5]


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


@pytest.mark.parametrize("move_mode", [0, 1])
# 96 and 182 (species, cell) items: whole and cut groups of four in the deposit, one item per warp in the sort's push;
# 10,706 and 19,866 items: groups of three and of four there too, the last one cut (4,736 warps are resident)
@pytest.mark.parametrize("cells", [(8, 6), (13, 7), (101, 53), (129, 77)])
def test_operators_bit_exact(move_mode, cells):
    ncx, ncy = cells
    cs = 3.125e-4
    deck = ccp_deck(ncx + 1, ncy + 1, ncx * cs, ncy * cs, ppc=4)
    kw = dict(seed=3, field_mode=1, move_mode=move_mode, cap_per_cell=1024)
    S = hpic.Setup(deck, **kw)
    case = hpic.Case(setup=S, **kw)
    o = oracle.Oracle(S.table, S.info, case.opts, 32, pcg_cluster=case.info.pcg_cluster, pcg_block=case.info.pcg_block)
    rng = np.random.default_rng(11)
    C = ncx * ncy
    for s in range(2):
        counts = np.array([COUNTS[(k + 3 * s) % len(COUNTS)] for k in range(C)], np.int32)
        n = int(counts.sum())
        x, y = (rng.random(n, dtype=np.float32) for _ in range(2))
        cell = np.repeat(np.arange(C), counts)
        k = np.arange(n) - np.repeat(np.cumsum(counts) - counts, counts)
        step = cs / float(S.info.dt)  # one cell per step
        v = [(rng.random(n, dtype=np.float32) * 2 - 1) * np.float32(step) for _ in range(3)]
        kind = cell % 5
        stay = (kind == 1) | ((kind == 2) & (k < 40))          # stayers only; movers after a chunk of stayers
        v = [np.where(stay, np.float32(0), a) for a in v]
        v[0] = np.where(kind == 3, np.float32(1.5 * step), v[0])  # the whole cell leaves
        x = np.where(stay & (k % 7 == 0), np.float32(0), x)
        y = np.where(stay & (k % 11 == 0), np.float32(-0.0), y)
        x = np.where(stay & (k % 13 == 0), np.nextafter(np.float32(1), np.float32(0)), x)
        arrs = [np.ascontiguousarray(a, np.float32) for a in (x, y, *v)]
        case.set_particles(s, counts, *arrs)
        o.set_particles(s, counts, *arrs)
    case.Deposit()
    o.Deposit()
    for t in (1, 2, 3):  # later steps start from the movers of the one before
        case.set_tstep(t)
        case.Field()
        o.Field(t)
        case.Move()
        o.Move()
        for s in range(2):
            gc, ga, gk = case.movers(s)
            oc, oa, ok = o.movers(s)
            assert np.array_equal(gc, oc) and np.array_equal(gk, ok), (t, s)
            for a, b in zip(ga, oa):
                assert np.array_equal(bits(a), bits(b)), (t, s, "movers")
        case.SortBoundary()
        o.SortBoundary()
        for s in range(2):
            gc, ga = case.particles(s)
            oc, oa = o.particles(s)
            assert np.array_equal(gc, oc), (t, s)
            for q, (a, b) in enumerate(zip(ga, oa)):
                assert np.array_equal(bits(a), bits(b)), (t, s, q)
        case.Deposit()
        o.Deposit()
        assert np.array_equal(case.grid("DEN").view(np.uint64), o.grid("DEN").view(np.uint64)), t
    assert case.status() == 0
    case.close()


def test_sorts_in_a_row():
    """SortBoundary once more with no Move in between files the parked movers again, source cells in increasing
    order, and stays inside the cells however often it is called."""
    ncx, ncy, cs = 9, 7, 3.125e-4
    deck = ccp_deck(ncx + 1, ncy + 1, ncx * cs, ncy * cs, ppc=4)
    case = hpic.Case(deck, seed=3, field_mode=1, move_mode=1, cap_per_cell=1024)
    rng = np.random.default_rng(5)
    C = ncx * ncy
    counts = np.array([COUNTS[k % 6] for k in range(C)], np.int32)
    n = int(counts.sum())
    x, y, *v = (rng.random(n, dtype=np.float32) for _ in range(5))
    v = [(a * 2 - 1) * np.float32(0.9 * cs / float(case.info.dt)) for a in v]  # under one cell per step: near movers only
    for s in range(2):
        case.set_particles(s, counts, x, y, *v)
    case.Move()
    moved = [case.movers(s) for s in range(2)]
    assert all(m[0].sum() > 0 for m in moved)
    case.SortBoundary()
    want = [case.particles(s) for s in range(2)]
    for _ in range(12):
        case.SortBoundary()
        for s in range(2):
            mc, ma, code = moved[s]
            at = np.concatenate([[0], np.cumsum(mc)])
            pc, pa = want[s]
            start = np.concatenate([[0], np.cumsum(pc)])
            new_c, new_a = np.zeros_like(pc), [[] for _ in range(5)]
            for c in range(C):
                i, j = divmod(c, ncy)
                own = np.arange(start[c], start[c + 1])
                add = []
                for si in range(max(i - 1, 0), min(i + 2, ncx)):
                    for sj in range(max(j - 1, 0), min(j + 2, ncy)):
                        src = si * ncy + sj
                        q = np.arange(at[src], at[src + 1])
                        add.append(q[code[q] == (i - si + 1) * 3 + (j - sj + 1)])
                add = np.concatenate(add)
                new_c[c] = own.size + add.size
                for a in range(5):
                    new_a[a] += [pa[a][own], ma[a][add]]
            want[s] = new_c, [np.concatenate(a) for a in new_a]
            got_c, got_a = case.particles(s)
            assert np.array_equal(got_c, want[s][0])
            for a in range(5):
                assert np.array_equal(bits(got_a[a]), bits(want[s][1][a]))
    assert case.status() == 0
    case.close()


def test_mcc_groups_of_cells():
    """Collision groups of 5 cells (16,200 cells, the last group cut short), against the oracle, and a group that
    holds the end of one case and the start of the next in a batch."""
    cs = 3.125e-4
    deck = ccp_deck(181, 91, 180 * cs, 90 * cs, ppc=6, pressure_torr=0.2, voltage=300.0)
    kw = dict(seed=21, field_mode=2, move_mode=1)
    S = hpic.Setup(deck, **kw)
    case = hpic.Case(setup=S, **kw)
    o = oracle.Oracle(S.table, S.info, case.opts, 32)
    for s in range(2):
        counts, arrs = S.particles(s, layout=0)
        o.set_particles(s, counts, *arrs)
    for t in (1, 2):
        case.set_tstep(t)
        case.MCC()
        o.MCC(t)
        for s in range(2):
            gc, ga = case.particles(s)
            oc, oa = o.particles(s)
            assert np.array_equal(gc, oc)
            for a, b in zip(ga, oa):
                assert np.array_equal(bits(a), bits(b)), (t, s)
    assert np.array_equal(case.grid("MCC_COUNT"), o.counters()[1])
    assert case.grid("MCC_COUNT").sum() > 0
    case.close()
    small = ccp_deck(34, 18, 33 * cs, 17 * cs, ppc=9, pressure_torr=0.2, voltage=300.0)
    alone, mixed = [[hpic.Case(d, seed=4 + k, field_mode=2, move_mode=1) for k, d in enumerate((small, deck, small))]
                    for _ in range(2)]
    b = hpic.Batch(mixed)
    b.step(4)
    for a, m in zip(alone, mixed):
        a.step(4)
        assert np.array_equal(a.grid("MCC_COUNT"), m.grid("MCC_COUNT"))
        for s in range(2):
            for u, v in zip(a.particles(s)[1], m.particles(s)[1]):
                assert np.array_equal(bits(u), bits(v))
    b.close()
