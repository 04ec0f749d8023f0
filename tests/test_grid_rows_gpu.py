"""The grid team's rows (csrc/group_sys.cuh): several elements a thread, each
row as long as its compartment has neighbours, on a lone system of any size
that the team takes."""
import numpy as np
import pytest

import gbrkc as G
import morph as M
from gpu_cases import jitter_for

pytestmark = pytest.mark.gpu


def star_purkinje(ncomp, branches, seed=4):
    """A synthetic Purkinje cell whose soma carries `branches` more dendrites: the
    dendrite ends that come first in the numbering hang on the soma."""
    rows = M.pkj_synthetic(seed, ncomp)
    soma = ncomp - 1
    parents = set(rows[:, 1].astype(int))
    ends = [i for i in range(ncomp - 1) if i not in parents][:branches]
    rows[ends, 1] = soma
    return rows


@pytest.mark.parametrize("branches,bw,ctas", [(13, 32, 5), (14, 32, 5), (15, 64, 3), (16, 32, 4), (40, 64, 2), (40, 128, 2)])
def test_long_rows_several_a_thread(oracle, monkeypatch, branches, bw, ctas):
    """Rows of 14 to 41 neighbours with two to eight elements a thread."""
    monkeypatch.setenv("GBRKC_GRID_MIN_NC", "300")
    monkeypatch.setenv("GBRKC_GRID_BW", str(bw))
    monkeypatch.setenv("GBRKC_GRID_CTAS", str(ctas))
    rows = star_purkinje(700, branches)
    stim = (699, 0.4e-3, 0.0, 1e9)
    jit = jitter_for(oracle, M.PKJ, 1)
    s = oracle.System(M.PKJ, 1, 1, rows, jit, stim=stim, canon=True)
    assert s.init() == 0
    eng = G.Engine(G.FP64)
    sid = eng.add_system(M.PKJ, 1, 1, rows, jit, stim=stim)
    eng.build()
    assert eng.type_team(M.PKJ) == "grid" and eng.launch_layout()[1][M.PKJ] == ctas
    at = 0.0
    for chunk in (1, 7):
        eng.advance(at, chunk)
        for _ in range(chunk):
            assert s.advance(at) == 0
            at += G.H_MAX
        np.testing.assert_array_equal(eng.vnew(sid), s.vnew())
    ctl, st, status = eng.ctl(sid)
    assert status == 0 and st == s.stats()
    eng.close()


@pytest.mark.parametrize("ncomp,bw", [(9, 0), (32, 0), (250, 32), (700, 128), (700, 256)])
def test_grid_of_one_cta(oracle, monkeypatch, ncomp, bw):
    """The grid team on one CTA -- a system of a warp at most, or a forced shape
    -- has its tables like any other, with nothing to receive."""
    monkeypatch.setenv("GBRKC_GRID_MIN_NC", "9")
    if bw:
        monkeypatch.setenv("GBRKC_GRID_BW", str(bw))
        monkeypatch.setenv("GBRKC_GRID_CTAS", "1")
    t, rows, stim = M.PKJ, M.pkj_synthetic(2, ncomp), (ncomp - 1, 0.02e-3, 0.0, 1e9)
    jit = jitter_for(oracle, t, 1)
    s = oracle.System(t, 1, 1, rows, jit, stim=stim, canon=True)
    assert s.init() == 0
    eng = G.Engine(G.FP64)
    sid = eng.add_system(t, 1, 1, rows, jit, stim=stim)
    eng.build()
    assert eng.type_team(t) == "grid" and eng.launch_layout()[1][t] == 1
    for k in range(4):
        eng.advance(k * G.H_MAX, 1)
        assert s.advance(k * G.H_MAX) == 0
        np.testing.assert_array_equal(eng.vnew(sid), s.vnew())
    ctl, st, status = eng.ctl(sid)
    assert status == 0 and st == s.stats()
    eng.close()


def test_large_system_with_a_long_row_takes_the_grid():
    """5 x 5 Purkinje cells of 1600 compartments whose somas have 17 dendrites and
    more (two elements a thread on every SM)."""
    rows = star_purkinje(1600, 16)
    eng = G.Engine(G.FP64)
    eng.add_system(M.PKJ, 5, 5, rows, np.zeros(25), gj_pairs=M.PKJ_GJ_PAIRS, gap=True)
    eng.build()
    assert eng.type_team(M.PKJ) == "grid"
    eng.advance(0.0, 2)
    eng.close()
