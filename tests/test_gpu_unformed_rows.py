"""Metropolis sequences on trees whose expansion rows no pass, or only one, has
formed: such rows are zero and change by the accepted moves alone, so every way
to run the sequence gives the energy shifts of the graphs of single moves.

The shifts differ by the order of fewer than 2e5 terms below 1e3 in size, each
rounded to 1.2e-16 of that with either sign: sqrt(2e5) * 1.2e-13 = 5e-11."""
import numpy as np
import pytest

import pdmk4mc_b200 as P

pytestmark = pytest.mark.gpu

N, L = 4000, 16.0
ABS_DE = 2e-10
PASSES = {"nothing": "", "outgoing": "o", "incoming": "i", "incoming_first": "io"}


def system():
    rng = np.random.default_rng(31)
    return rng.uniform(0, L, 3 * N), np.where(np.arange(N) % 2 == 0, 1.0, -1.0)


def proposals(m, seed):
    rng = np.random.default_rng(seed)
    # half of them forced, so that rows change; the others meet the changes
    return rng.integers(0, N, m), rng.uniform(-0.3, 0.3, (m, 3)), np.where(np.arange(m) % 2 == 0, -1.0, np.inf)


def dirty_pool(prm):
    # memory that an earlier tree of the same shape has written
    t = P.HPDMKPtTree(prm, *system())
    t.form_outgoing_pw()
    t.form_incoming_pw()
    t.eval_energy()
    t.close()


def open_tree(prm, passes):
    t = P.HPDMKPtTree(prm, *system())
    for p in passes:
        t.form_outgoing_pw() if p == "o" else t.form_incoming_pw()
    return t


def params(digits):
    return P.HPDMKParams(n_per_leaf=20, digits=digits, L=L, init=P.DIRECT)


def close(a, b):
    return np.all(np.abs(a - b) <= ABS_DE * np.maximum(1.0, np.abs(b)))


@pytest.mark.parametrize("digits", [3, 9])
@pytest.mark.parametrize("moves", [5, 300])
@pytest.mark.parametrize("formed", sorted(PASSES))
def test_sequence_on_unformed_rows(formed, moves, digits):
    prm = params(digits)
    idx, disp, u = proposals(moves, moves)
    got = []
    for mode in (P.MC_PERSISTENT, P.MC_GRAPH):
        dirty_pool(prm)
        t = open_tree(prm, PASSES[formed])
        try:
            t.set_mc_mode(mode)
            got.append([t.mc_run(idx, disp, u, 1.0) for _ in range(2)])  # again on the rows of the first
        finally:
            t.close()
    for a, b in zip(*got):
        np.testing.assert_array_equal(a[1], b[1])
        assert close(a[0], b[0])


@pytest.mark.parametrize("digits", [3, 9])
@pytest.mark.parametrize("formed", sorted(PASSES))
def test_sequence_that_empties_boxes(formed, digits):
    # a few particles on many boxes: a box left by its last particle keeps a row
    n, l = 64, 4.0
    rng = np.random.default_rng(5)
    r, q = rng.uniform(0, l, 3 * n), np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    prm = P.HPDMKParams(n_per_leaf=1, digits=digits, L=l, init=P.DIRECT)
    idx, disp = rng.integers(0, n, 150), rng.uniform(-2.0, 2.0, (150, 3))
    got = []
    for mode in (P.MC_PERSISTENT, P.MC_GRAPH):
        t = P.HPDMKPtTree(prm, r, q)
        try:
            for p in PASSES[formed]:
                t.form_outgoing_pw() if p == "o" else t.form_incoming_pw()
            t.set_mc_mode(mode)
            got.append([t.mc_run(idx, disp, np.full(150, -1.0), 1.0)[0] for _ in range(3)] + [t.eval_energy_parts()])
        finally:
            t.close()
    for a, b in zip(*got):
        assert close(a, b)


@pytest.mark.parametrize("sets", [["nothing"] * 2, ["outgoing", "formed"], ["incoming_first", "formed"], ["incoming"]])
def test_replicas_with_unformed_rows(sets):
    # more moves than a replica lists, then a second call on the rows of the first
    m, prm = 150, params(6)
    passes = dict(PASSES, formed="oi")
    prop = [proposals(m, 7 + k) for k in range(len(sets))]
    want = []
    for name, p in zip(sets, prop):
        dirty_pool(prm)
        t = open_tree(prm, passes[name])
        try:
            t.set_mc_mode(P.MC_GRAPH)
            want.append([t.mc_run(*p, 1.0) for _ in range(2)])
        finally:
            t.close()
    dirty_pool(prm)
    ts = [open_tree(prm, passes[name]) for name in sets]
    try:
        for call in range(2):
            dE, acc = P.replicas_mc_run(ts, *(np.stack([p[k] for p in prop]) for k in range(3)), 1.0)
            for k in range(len(sets)):
                np.testing.assert_array_equal(acc[k], want[k][call][1])
                assert close(dE[k], want[k][call][0])
    finally:
        for t in ts:
            t.close()
