"""Group teams (csrc/group_sys.cuh): a pool alone in its engine takes one
system per CTA, per cluster of CTAs or over the whole grid where that is
shorter.  Bit for bit the same as the warp and block teams it takes the place
of (GBRKC_GROUP=0), in both precisions, and as the oracle in FP64: cells of
less than a warp, ragged last chunks, one and two elements a thread, several
systems per CTA in turn, gap junctions across CTAs."""
import numpy as np
import pytest

import gbrkc as G
import morph as M

pytestmark = pytest.mark.gpu

SHAPES = {
    # name: (type, systems, nx, ny, rows by system)
    "io_1x1": (M.IO, 3, 1, 1, lambda k: M.io_rows()),
    "io_4x4": (M.IO, 1, 4, 4, lambda k: M.io_rows()),
    "io_4x4_many": (M.IO, 700, 4, 4, lambda k: M.io_rows()),
    "io_11x11": (M.IO, 2, 11, 11, lambda k: M.io_rows()),
    "io_16x16": (M.IO, 1, 16, 16, lambda k: M.io_rows()),
    "go_few": (M.GO, 5, 1, 1, lambda k: M.go_synthetic(2000 + k)),
    "go_more": (M.GO, 200, 1, 1, lambda k: M.go_synthetic(2000 + k % 3)),
    "go_2x2": (M.GO, 3, 2, 2, lambda k: M.go_synthetic(3)),
    "pkj_one": (M.PKJ, 1, 1, 1, lambda k: M.pkj_synthetic(2)),
    "pkj_odd": (M.PKJ, 3, 1, 1, lambda k: M.pkj_synthetic(7 + k, 977)),
    "pkj_2x1": (M.PKJ, 2, 2, 1, lambda k: M.pkj_synthetic(4)),
    "gr_full": (M.GR, 2, 1, 1, lambda k: M.gr_synthetic(11 + k)),
}


def _run(shape, precision, intervals, oracle=None):
    t, n, nx, ny, rows = SHAPES[shape]
    rng = np.random.default_rng(3)
    eng = G.Engine(precision)
    amp = {M.GR: 0.01e-3, M.GO: 0.4e-3, M.PKJ: 0.4e-3, M.IO: 5.5}[t]
    ids, refs, cells = [], [], nx * ny
    for k in range(n):
        r = rows(k)
        jit = rng.uniform(-0.5, 0.5, cells)
        comp = {M.GR: 16, M.GO: 30, M.PKJ: r.shape[0] - 1, M.IO: 0}[t]
        stim = (np.full(cells, comp), rng.uniform(0, amp, cells), rng.uniform(0, 0.3, cells), np.full(cells, 1e9))
        gj = M.PKJ_GJ_PAIRS if t == M.PKJ and cells > 1 else None
        ids.append(eng.add_system(t, nx, ny, r, jit, stim=stim, gap=cells > 1, gj_pairs=gj))
        if oracle is not None and k < 3:
            s = oracle.System(t, nx, ny, r, jit, stim=stim, gj_pairs=gj, io_gap=cells > 1, go_gj=cells > 1,
                              pkj_gj=cells > 1, canon=True)
            assert s.init() == 0
            refs.append(s)
    eng.build()
    team = eng.type_team(t)
    eng.record_soma(intervals)
    eng.record_spikes(1 << 16)
    at = 0.0
    for chunk in (1, intervals - 1):
        eng.advance(at, chunk)
        for s in refs:
            for i in range(chunk):
                assert s.advance(at + i * G.H_MAX) == 0
        at += chunk * G.H_MAX
    out = [eng.vnew(i) for i in ids] + [eng.read(i, G.F_V) for i in ids] + [eng.read(i, G.F_B) for i in ids]
    out += [eng.read(i, G.F_ION, 3) for i in ids[:4]]
    soma = np.empty((intervals, eng.type_cells(t)))
    out += [eng.read_soma_type(t, intervals, soma), eng.read_spikes(t)[0]]
    stats = [eng.ctl(i) for i in ids]
    eng.close()
    return team, out, stats, refs


@pytest.mark.parametrize("precision", [G.FP64, G.MIXED])
@pytest.mark.parametrize("shape", SHAPES)
def test_group_team_same_bits(oracle, monkeypatch, shape, precision):
    intervals = 2 if SHAPES[shape][0] == M.GR or SHAPES[shape][1] > 100 else 12
    use = oracle if precision == G.FP64 else None
    monkeypatch.delenv("GBRKC_GROUP", raising=False)
    _, got, stats, refs = _run(shape, precision, intervals, use)
    for s, v, (_, st, status) in zip(refs, got, stats):
        np.testing.assert_array_equal(v, s.vnew())
        assert status == 0 and st == s.stats()
    monkeypatch.setenv("GBRKC_GROUP", "0")
    other, want, wstats, _ = _run(shape, precision, intervals)
    assert other in ("mega", "pool")    # (a pool of Golgi or granule systems too large for a warp has its own launch)
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
    assert stats == wstats


def _uneven(precision, n=170):
    """Rounds of 2 and 20 intervals with few and with all of the slots at work."""
    rng = np.random.default_rng(8)
    eng = G.Engine(precision)
    for k in range(n):
        r = M.pkj_synthetic(2 + k % 2, 1599 if k % 2 else 801)
        stim = ([r.shape[0] - 1], [rng.uniform(0, 0.4e-3)], [0.0], [1e9])
        eng.add_system(M.PKJ, 1, 1, r, rng.uniform(-0.5, 0.5, 1), stim=stim)
    eng.build()
    eng.record_spikes(1 << 16)
    at, teams = 0.0, []
    for busy, intervals in ((n, 2), (3, 2), (3, 2), (n, 20), (n, 2), (70, 2), (70, 2)):
        eng.set_budget(0, n, 0)
        eng.set_budget(0, busy, -1)
        teams.append(eng.type_team(M.PKJ))
        eng.advance(at, intervals)
        at += intervals * G.H_MAX
    out = [eng.read(i, f) for i in range(n) for f in (G.F_V, G.F_B)] + [eng.read_spikes(M.PKJ)[0]]
    stats = [eng.ctl(i) for i in range(n)]
    eng.close()
    return teams, out, stats


@pytest.mark.parametrize("precision", [G.FP64, G.MIXED])
def test_wide_teams_same_bits(monkeypatch, precision):
    """A pool whose chains were uneven in the last launch goes on in cluster
    teams that take systems from the line, and back; the same bits as in the
    persistent launch alone."""
    monkeypatch.delenv("GBRKC_GROUP", raising=False)
    teams, got, stats = _uneven(precision)
    assert teams[0] == "mega" and teams[3] == "cluster" and teams[4] == "mega"
    monkeypatch.setenv("GBRKC_GROUP", "0")
    other, want, wstats = _uneven(precision)
    assert set(other) == {"mega"}
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
    assert stats == wstats


@pytest.mark.parametrize("precision", [G.FP64, G.MIXED])
def test_granule_turns_same_bits(monkeypatch, precision):
    """More granule cells than the persistent launch's quads (8 warps of 8 on
    each SM): quads take turns between intervals; the same bits as cells run to
    their end one after another in the type's own launch."""
    n, intervals = 9900, 3
    rng = np.random.default_rng(5)
    jit, amp = rng.uniform(-0.5, 0.5, (n, 1)), rng.uniform(0, 0.012e-3, n)
    ids = np.arange(0, n, 37)

    def run():
        eng = G.Engine(precision)
        for k in range(n):
            eng.add_system(M.GR, 1, 1, M.gr_reduced4(), jit[k], stim=([1], [amp[k]], [0.0], [1e9]))
        eng.build()
        team = eng.type_team(M.GR)
        eng.set_budget(50, 400, 2)       # budgets that end within the launch
        eng.record_soma(intervals)
        eng.advance(0.0, intervals)
        soma = np.empty((intervals, eng.type_cells(M.GR)))
        out = [eng.read_soma_type(M.GR, intervals, soma)] + [eng.read(i, f) for i in ids for f in (G.F_V, G.F_B)]
        stats = [eng.ctl(i) for i in ids]
        eng.close()
        return team, out, stats

    monkeypatch.delenv("GBRKC_NO_MEGA", raising=False)
    team, got, stats = run()
    assert team == "mega"
    monkeypatch.setenv("GBRKC_NO_MEGA", "1")
    other, want, wstats = run()
    assert other == "pool"
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
    assert stats == wstats
