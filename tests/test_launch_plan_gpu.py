"""How the next launch of a pool is planned (csrc/engine.cpp): the teams it may
take, the systems it counts, and what idle slots cost it."""
import os
import subprocess
import sys

import numpy as np
import pytest

import configs
import gbrkc as G
import morph as M

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def comb_purkinje(teeth=700, soma_dendrites=9):
    """A Purkinje cell of 2 * teeth compartments: a trunk whose every
    compartment carries one tooth, the teeth numbered before the trunk, so that
    on two CTAs nearly every tooth reads and is read across them; and a soma
    with several dendrites of one compartment beside the trunk."""
    n = 2 * teeth
    rows = np.zeros((n, 7))
    rng = np.random.default_rng(1)
    for i in range(n):
        along = rng.standard_normal(3)
        length = rng.uniform(5.0, 20.0) / np.linalg.norm(along)
        parent = i + teeth if i < teeth else i + 1
        rows[i] = [i, parent, *(length * along), 3.0 if i < teeth else 6.0, 3 if i < teeth else 2]
    soma = n - 1
    for i in range(soma_dendrites - 2):       # (the trunk's end and the soma's own tooth are two)
        rows[i, 1] = soma
    rows[soma] = [soma, -1, 0.0, 0.0, 0.0, 29.8, 0]
    return rows


def uneven_comb(others):
    """170 comb cells, of which one has 20 intervals to do in the second launch
    and the others fewer; the third launch's team and the last voltages."""
    n, r = 170, comb_purkinje()
    eng = G.Engine(G.MIXED)
    for k in range(n):
        eng.add_system(M.PKJ, 1, 1, r, [0.0])
    eng.build()
    eng.advance(0.0, 4)
    eng.set_budget(0, n, others)
    eng.set_budget(0, 1, -1)
    eng.advance(4 * G.H_MAX, 20)
    team = eng.type_team(M.PKJ)
    eng.set_budget(0, n, -1)
    eng.advance(24 * G.H_MAX, 2)
    out = np.concatenate([eng.vnew(i) for i in range(n)])
    eng.close()
    return team, out


def _alone(others, group):
    """uneven_comb in a process of its own: a kernel's shared-memory limit is the
    process's, and other tests raise it."""
    env = dict(os.environ)
    env.pop("GBRKC_GROUP", None)
    if group is not None:
        env["GBRKC_GROUP"] = group
    code = ("import sys; sys.path[:0] = %r; import numpy as np, test_launch_plan_gpu as t; team, v = t.uneven_comb(%d); "
            "print('TEAM', team); print('BITS', v.tobytes().hex())" % ([p for p in sys.path if p] + [HERE], others))
    p = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stderr[-2000:]
    line = {w.split(" ", 1)[0]: w.split(" ", 1)[1] for w in p.stdout.splitlines() if w.startswith(("TEAM", "BITS"))}
    return line["TEAM"], np.frombuffer(bytes.fromhex(line["BITS"]))


@pytest.mark.parametrize("others", [6, 7])
def test_wide_rows_on_a_cluster(others):
    """A cluster team whose rows and hand-overs take more shared memory than
    the estimate's (rows of nine neighbours, 640 received values) is
    launched with what it needs: the same bits as in the persistent launch."""
    team, got = _alone(others, None)
    assert team == "cluster"
    other, want = _alone(others, "0")
    assert other == "mega"
    np.testing.assert_array_equal(got, want)


def test_granule_places_follow_the_work():
    """Granule cells alone take a place each: as many CTAs after all of them
    were refilled as before (999 cells, FP64: 8 to a warp, a warp a CTA), and
    as many as there are cells with work after budgets ended and were raised."""
    n = 999
    eng = G.Engine(G.FP64)
    for k in range(n):
        eng.add_system(M.GR, 1, 1, M.gr_reduced4(), [0.0])
    eng.build()
    eng.advance(0.0, 1)
    first = eng.launch_layout()
    eng.reset_systems(0, n, np.zeros(n))
    eng.advance(G.H_MAX, 1)
    assert eng.launch_layout() == first
    eng.set_budget(0, 900, 0)
    eng.advance(2 * G.H_MAX, 1)
    few = eng.launch_layout()
    assert few[1][M.GR] < first[1][M.GR] / 4
    eng.set_budget(0, 900, -1)
    eng.advance(3 * G.H_MAX, 1)
    assert eng.launch_layout() == first
    eng.close()


def test_idle_slots_cost_a_role_nothing():
    """A role of the persistent launch whose slots have no work ends at once: the
    systems without work are not in the line that its teams take systems from.
    (Within half a millisecond, where the granule cells beside them take 14 or
    more; the split leaves such a role one CTA or two after a few launches.)"""
    eng = G.Engine(G.MIXED)
    for k in range(3000):
        eng.add_system(M.GR, 1, 1, M.gr_reduced4(), [1e-4 * k])
    go = [eng.add_system(M.GO, 1, 1, M.go_synthetic(2000), [0.0], idle=k > 0) for k in range(2000)]
    eng.build()
    for k in range(12):
        if k == 2:
            eng.set_budget(go[0], 1, 0)
        eng.advance(8 * k * G.H_MAX, 8)
    assert eng.type_team(M.GO) == "mega"
    assert eng.last_kernel_ms(M.GO) < 0.5 < eng.last_kernel_ms(M.GR)
    eng.close()


def test_autotune_keeps_the_line():
    """Budgets change between an advance and autotune, which restores the
    device's state: the next launch still takes the systems with work."""
    def run(tune):
        eng = G.Engine(G.MIXED)
        for k in range(64):
            eng.add_system(M.GR, 1, 1, M.gr_reduced4(), [0.0])
        go = [eng.add_system(M.GO, 1, 1, M.go_synthetic(2000), [0.0]) for k in range(40)]
        eng.build()
        eng.advance(0.0, 2)
        eng.set_budget(go[0], 30, 0)
        eng.advance(2 * G.H_MAX, 2)
        eng.set_budget(go[0], 40, -1)
        if tune:
            eng.autotune(4 * G.H_MAX, 2)
        eng.advance(4 * G.H_MAX, 2)
        out = [eng.vnew(i) for i in go] + [eng.ctl(i) for i in go]
        eng.close()
        return out

    for a, b in zip(run(True), run(False)):
        np.testing.assert_equal(a, b)


def test_split_follows_the_work():
    """Granule cells that come beside other types get the CTAs they need in
    their first launch, not after the split has crept there: it takes less
    than three times the launch of the same cells eight launches later."""
    eng = G.Engine(G.MIXED)
    n = 3400
    for k in range(n):
        eng.add_system(M.GR, 1, 1, M.gr_reduced4(), [1e-4 * k])
    for k in range(40):
        eng.add_system(M.GO, 1, 1, M.go_synthetic(2000), [0.0])
    eng.build()
    at = 0.0

    def advance():
        nonlocal at
        eng.advance(at, 8)
        at += 8 * G.H_MAX
        return eng.last_advance_ms()

    eng.set_budget(1, n - 1, 0)
    for _ in range(6):
        advance()
    assert eng.launch_layout()[1][M.GR] == 1
    eng.set_budget(1, n - 1, -1)
    first = advance()
    for _ in range(8):
        later = advance()
    assert first < 3.0 * later, (first, later)
    eng.set_budget(n, 40, 0)
    advance()
    advance()
    assert eng.launch_layout()[1][M.GO] == 1      # (and of a type with no work left they go to the others)
    eng.close()


def test_autotune_restores_before_the_next_launch():
    """A batch whose state takes longer to copy back than a launch to begin:
    every launch of the tuning, and the advance after it, starts from the
    restored state -- the same bits as without the tuning."""
    def run(tune):
        eng = G.Engine(G.MIXED)
        specs = configs.scaled_stated_batch(0.5)
        ids = configs.add_to(eng, specs)
        eng.build()
        eng.advance(0.0, 2, tolerate_retire=True)
        for _ in range(2 if tune else 0):
            eng.autotune(2 * G.H_MAX, 8)
        eng.advance(2 * G.H_MAX, 8, tolerate_retire=True)
        out = [eng.vnew(i) for i in ids[::7]] + [eng.ctl(i) for i in ids[::7]]
        eng.close()
        return out

    for a, b in zip(run(True), run(False)):
        np.testing.assert_equal(a, b)


def _many_golgi(n=5600):
    """Golgi cells that outnumber the persistent launch's teams some 37 times,
    alike but for a few currents: the third launch, planned from the second."""
    rng = np.random.default_rng(6)
    eng = G.Engine(G.MIXED)
    rows = M.go_synthetic(2000)
    for k in range(n):
        eng.add_system(M.GO, 1, 1, rows, rng.uniform(-0.5, 0.5, 1), stim=([30], [1e-5 * (k % 7)], [0.0], [1e9]))
    eng.build()
    eng.set_budget(17, 9, 5)
    eng.record_soma(6)
    for k in range(3):
        eng.advance(2 * k * G.H_MAX, 2)
    team = eng.type_team(M.GO)
    soma = np.empty((6, eng.type_cells(M.GO)))
    out = [eng.read_soma_type(M.GO, 6, soma)] + [eng.read(i, f) for i in range(0, n, 41) for f in (G.F_V, G.F_B, G.F_YN)]
    stats = [eng.ctl(i) for i in range(0, n, 41)]
    ms = eng.last_advance_ms()
    eng.close()
    return team, out, stats, ms


def test_golgi_cells_beyond_their_teams_take_warps(monkeypatch):
    """The next launch takes a warp per cell where that does more: the same bits
    as with warps alone (GBRKC_GROUP=0), and about their time (the launches of
    two seeds of the same work differ by less than a sixth; a launch in teams
    takes a third longer)."""
    monkeypatch.delenv("GBRKC_GROUP", raising=False)
    team, got, stats, ms = _many_golgi()
    monkeypatch.setenv("GBRKC_GROUP", "0")
    other, want, wstats, wms = _many_golgi()
    assert team == other == "mega"
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
    assert stats == wstats
    assert ms < 1.17 * wms, (ms, wms)


def test_no_intervals_leave_the_plan():
    """An advance of no intervals -- a refill's initialisation -- keeps what the
    last launch said of the next one's teams."""
    n = 170
    eng = G.Engine(G.MIXED)
    for k in range(n):
        eng.add_system(M.PKJ, 1, 1, M.pkj_synthetic(2, 801), [0.0])
    eng.build()
    eng.set_budget(3, n - 3, 0)
    eng.advance(0.0, 2)
    assert eng.type_team(M.PKJ) == "cluster"
    eng.reset_systems(0, 3, np.zeros(3))
    eng.advance(0.0, 0)
    assert eng.type_team(M.PKJ) == "cluster"
    eng.advance(0.0, 2)
    assert eng.type_team(M.PKJ) == "cluster"
    eng.close()
