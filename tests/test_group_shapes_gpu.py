"""Every form of the group teams (csrc/group_sys.cuh) by a forced shape: one,
two and four elements a thread, in a CTA and in a cluster of CTAs, with ragged
last chunks, chunks that differ by one between CTAs, values received from
several CTAs, and gap junctions across them.  The team that ran is the one
asked for; the bits are the oracle's in FP64, and in both precisions those of
the teams with their vectors in memory."""
import numpy as np
import pytest

import gbrkc as G
import morph as M
import test_group_gpu as T
from test_grid_rows_gpu import star_purkinje

pytestmark = pytest.mark.gpu

go = lambda k: M.go_synthetic(2000 + k % 3)
pkj = lambda n: lambda k: M.pkj_synthetic(7 + k, n)
io = lambda k: M.io_rows()

# (type, systems, nx, ny, rows by system), shape, team, elements a thread
FORMS = [
    ((M.IO, 2, 2, 2, io), "cta:32", "pool", 1),                # 12 compartments: less than a warp
    ((M.IO, 3, 8, 8, io), "cta:192", "pool", 1),               # exactly its threads
    ((M.IO, 3, 8, 8, io), "cta:160", "pool", 2),               # 32 compartments over
    ((M.GO, 5, 1, 1, go), "cta:160", "pool", 1),
    ((M.GO, 5, 1, 1, go), "cta:96", "pool", 2),
    ((M.PKJ, 2, 1, 1, pkj(511)), "cta:256", "pool", 2),
    ((M.GO, 5, 1, 1, go), "cluster:32x5", "cluster", 1),       # the last CTA owns three compartments
    ((M.GO, 5, 1, 1, go), "cluster:64x2", "cluster", 2),
    ((M.GR, 2, 1, 1, lambda k: M.gr_synthetic(11 + k)), "cluster:64x10", "cluster", 1),
    ((M.GR, 2, 1, 1, lambda k: M.gr_synthetic(11 + k)), "cluster:64x6", "cluster", 2),
    ((M.IO, 2, 11, 11, io), "cluster:32x12", "cluster", 1),
    ((M.IO, 2, 11, 11, io), "cluster:32x7", "cluster", 2),
    ((M.IO, 1, 16, 16, io), "cluster:64x12", "cluster", 1),
    ((M.PKJ, 3, 1, 1, pkj(977)), "cluster:64x16", "cluster", 1),
    ((M.PKJ, 3, 1, 1, pkj(977)), "cluster:128x4", "cluster", 2),
    ((M.PKJ, 3, 1, 1, pkj(977)), "cluster:256x2", "cluster", 2),     # 46 KB of shared memory beside the kernel's own 4
    ((M.PKJ, 2, 1, 1, lambda k: star_purkinje(440, 6, 2 + k)), "cta:224", "pool", 2),      # the same
    ((M.PKJ, 3, 1, 1, pkj(977)), "cluster:128x3", "cluster", 4),     # three and two chunks a CTA
    ((M.PKJ, 3, 1, 1, pkj(977)), "cluster:64x4", "cluster", 4),
    ((M.PKJ, 20, 1, 1, pkj(1599)), "cluster:128x13", "cluster", 1),
    ((M.PKJ, 2, 2, 1, pkj(1600)), "cluster:256x4", "cluster", 4),    # a system's own operator, linear gap junctions
]


@pytest.mark.parametrize("precision", [G.FP64, G.MIXED])
@pytest.mark.parametrize("form,shape,team,rows", FORMS, ids=lambda x: x if isinstance(x, str) else "")
def test_forced_shape_same_bits(oracle, monkeypatch, form, shape, team, rows, precision):
    threads, _, ctas = shape.split(":")[1].partition("x")
    chunks = -(-form[2] * form[3] * form[4](0).shape[0] // int(threads))
    most = -(-chunks // int(ctas or 1))
    assert {1: (1,), 2: (2,), 4: (3, 4)}[rows].count(most) == 1      # the kernel of that many elements a thread
    monkeypatch.setitem(T.SHAPES, "forced", form)
    intervals = 2 if form[0] == M.GR or form[1] > 10 else 6
    use = oracle if precision == G.FP64 else None
    monkeypatch.setenv("GBRKC_GROUP", shape)
    ran, got, stats, refs = T._run("forced", precision, intervals, use)
    assert ran == team
    for s, v, (_, st, status) in zip(refs, got, stats):
        np.testing.assert_array_equal(v, s.vnew())
        assert status == 0 and st == s.stats()
    monkeypatch.setenv("GBRKC_GROUP", "0")
    other, want, wstats, _ = T._run("forced", precision, intervals)
    assert other in ("mega", "pool")
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
    assert stats == wstats


def test_a_shape_that_does_not_fit_is_not_taken(monkeypatch):
    """More elements than the team's registers hold, fewer chunks than CTAs,
    or no shape at all: the pool keeps its other teams."""
    for shape in ("cta:32", "cluster:32x16", "cluster:96x2", "cta:33", "cta:512", "cluster:64"):
        monkeypatch.setenv("GBRKC_GROUP", shape)
        eng = G.Engine(G.MIXED)
        eng.add_system(M.GO, 1, 1, M.go_synthetic(2000), [0.0])
        eng.build()
        if shape != "cluster:64":        # (not a shape: the estimate's)
            assert eng.type_team(M.GO) == "mega"
        eng.advance(0.0, 1)
        eng.close()
