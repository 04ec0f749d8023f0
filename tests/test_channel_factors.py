"""Channel-density factors of multi-cell systems (Engine.add_system,
Engine.reset_systems): the C ABI reads one row per cell, whatever the caller
passes."""
import os
import re

import numpy as np
import pytest

import gbrkc as G
import morph as M


def test_channels_of_the_types():
    src = open(os.path.join(os.path.dirname(G.__file__), "csrc", "model.h")).read()
    counts = [len(re.findall(r"\b%s_g_\w+" % t, src)) for t in ("GR", "GO", "PK", "IO")]
    assert tuple(counts) == G.NCOND


@pytest.mark.parametrize("t,systems,cells", [(M.GO, 1, 1), (M.GO, 1, 4), (M.GO, 3, 12), (M.IO, 2, 32)])
def test_factors_by_system_and_by_cell(t, systems, cells):
    k = G.NCOND[t]
    by_cell = np.random.default_rng(1).uniform(0.8, 1.2, (cells, k))
    np.testing.assert_array_equal(G._channel_factors(by_cell, t, systems, cells), by_cell.reshape(-1))
    by_system = by_cell[:systems]
    want = np.repeat(by_system, cells // systems, axis=0)
    np.testing.assert_array_equal(G._channel_factors(by_system, t, systems, cells), want.reshape(-1))


@pytest.mark.parametrize("t,systems,cells,n", [(M.GO, 1, 4, 14), (M.GO, 3, 12, 3), (M.IO, 2, 32, 8), (M.GR, 5, 5, 49)])
def test_too_few_factors_are_refused(t, systems, cells, n):
    with pytest.raises(ValueError):
        G._channel_factors(np.ones(n), t, systems, cells)


@pytest.mark.gpu
def test_system_factors_are_its_cells_factors():
    f = np.random.default_rng(2).uniform(0.8, 1.2, (2, G.NCOND[M.GO]))
    by_cell = np.repeat(f, 4, axis=0)
    out = []
    for first, again in ((f[0], f), (by_cell[:4], by_cell)):
        eng = G.Engine(G.FP64)
        a = eng.add_system(M.GO, 2, 2, M.go_synthetic(3), np.zeros(4), cond_scale_ch=first)
        b = eng.add_system(M.GO, 2, 2, M.go_synthetic(3), np.zeros(4), cond_scale_ch=first)
        eng.build()
        eng.advance(0.0, 2)
        v = [eng.vnew(a), eng.vnew(b)]
        eng.reset_systems(a, 2, np.zeros(8), cond_scale_ch=again)
        eng.advance(0.0, 2)
        out.append(v + [eng.vnew(a), eng.vnew(b)])
        eng.close()
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
    assert np.any(out[0][2] != out[0][3])
