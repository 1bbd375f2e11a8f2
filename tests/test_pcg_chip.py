"""The solve with its state on chip (csrc/pcg.cu) at the edges of its range: one to eight nodes per thread, one
CTA to a 16-CTA cluster to the whole GPU, halos of one and two nodes per thread, and the launch shapes just past
it that keep k_pcg.  Every solve has to give the oracle's bits (the oracle repeats the reduction tree of the same
number of CTAs and threads)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import hpic
import oracle
from hpic.decks import ccp_deck

pytestmark = pytest.mark.gpu

SHAPES = [  # nodes, threads per CTA, largest cluster
    (17, 9, 512, 16),     # one node per thread, one CTA
    (33, 17, 96, 16),     # 6 nodes per thread, three warps
    (33, 17, 64, 16),     # 9 nodes per thread: k_pcg
    (64, 64, 512, 16),    # 4096 nodes: 8 per thread, one CTA
    (65, 64, 512, 16),    # just past it: two CTAs, 5 per thread
    (129, 65, 512, 16),   # four CTAs
    (129, 65, 512, 2),    # two CTAs of 9 nodes per thread: k_pcg
    (9, 500, 512, 16),    # a halo of two nodes per thread
    (9, 520, 512, 16),    # a halo past that: k_pcg
    (257, 129, 512, 16),  # a 16-CTA cluster, the last CTA not full
    (263, 251, 512, 16),  # whole GPU, 65 CTAs
    (263, 251, 128, 16),  # whole GPU, 8 nodes per thread
    (263, 251, 64, 16),   # whole GPU past the range: k_pcg
]


@pytest.mark.parametrize("nx,ny,block,cluster", SHAPES)
@pytest.mark.parametrize("mode", [0, 1])
def test_solve_bit_exact(nx, ny, block, cluster, mode):
    deck = ccp_deck(nx, ny, (nx - 1) * 3.125e-4, (ny - 1) * 3.125e-4, ppc=3, voltage=150.0)
    kw = dict(seed=9, field_mode=mode, gas_temp_mode=1)
    S = hpic.Setup(deck, **kw)
    case = hpic.Case(setup=S, **kw)
    case.set_tune(pcg_block=block, pcg_cluster_max=cluster)
    info = hpic.CaseInfo()
    hpic._check(hpic.lib().hp_case_get_info(case.h, C.byref(info)))
    o = oracle.Oracle(S.table, S.info, case.opts, 32, pcg_cluster=info.pcg_cluster, pcg_block=info.pcg_block)
    for s in range(S.info.nsp):
        counts, arrs = S.particles(s, layout=0)
        o.set_particles(s, counts, *arrs)
    o.DepositBasic()
    for t in (1, 2):  # the second solve starts from the first one's solution
        case.set_tstep(t)
        case.Field()
        o.Field(t)
        for g in ("PHI_POIS", "PHI", "EX", "EY"):
            a, b = case.grid(g), o.grid(g)
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (t, g)
        assert case.pcg_iters()[0] == o.counters()[2][0]
    assert case.status() == 0
    case.close()


def test_solve_after_one_whose_waits_gave_up(tmp_path):
    """The whole-GPU solve with no polls allowed returns with HP_STATUS_WAIT_TIMEOUT, and the solve after it takes none
    of the words that such a solve can leave behind (tests/pcg_words.cu)."""
    here = os.path.dirname(os.path.abspath(__file__))
    src = os.path.join(here, "..", "hybrid-final_b200", "csrc")
    exe = str(tmp_path / "pcg_words")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "--fmad=false", "-I", src,
                    "-I", os.path.join(here, "..", "include"), os.path.join(here, "pcg_words.cu"),
                    os.path.join(src, "prof.cu"), "-o", exe], check=True)
    lines = subprocess.run([exe], capture_output=True, text=True, timeout=120).stdout.splitlines()
    assert len(lines) == 2, lines
    for line in lines:
        f = line.split()
        assert f[2:9] == ["ran", "1", "gave_up", "1", "same", "1", "iterations"], line
        assert f[9] == f[10] and int(f[9]) > 5, line
        assert f[11:] == ["nonzero", "1", "status", "0", "0"], line
