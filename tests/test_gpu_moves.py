"""Metropolis sequences with deferred row updates (the persistent kernel's long
form) against the move-by-move form (CUDA graphs of shift and update launches),
at the sizes where the deferred form can go wrong: every digits setting, more
moves than one launch lists, a particle moved many times in a row, full leaves
(every arrival parked in the overflow pool), uniform and clustered trees, and the
shortest sequence that is deferred. Both forms evaluate the same sums in another
order: each of the about 1e5 terms of an energy shift carries a rounding of
1e-16 of a term below 1e3, so the shifts agree within ABS_DE, and a row that
sums m moves within REL_PW of its largest coefficient."""
import numpy as np
import pytest

import pdmk4mc_b200 as P

pytestmark = pytest.mark.gpu

ABS_DE = 2e-10
REL_PW = 1e-11


def system(n, L, kind, seed):
    rng = np.random.default_rng(seed)
    r = rng.uniform(0, L, (n, 3))
    if kind == "clustered":
        c = rng.uniform(0, L, (8, 3))
        m = int(0.8 * n)
        r[:m] = np.mod(c[rng.integers(0, 8, m)] + rng.normal(0, L / 40, (m, 3)), L)
        r[r >= L] = 0.0
    return r.reshape(-1), np.where(np.arange(n) % 2 == 0, 1.0, -1.0)


@pytest.mark.parametrize("n,npl,digits,kind,moves,few,slack", [
    (3000, 20, 3, "uniform", 300, 0, 8),
    (3000, 20, 6, "uniform", 1500, 0, 8),       # two launches
    (6000, 30, 9, "uniform", 300, 0, 0),        # no free slots: the overflow pool
    (4000, 16, 9, "clustered", 300, 0, 2),
    (4000, 16, 12, "clustered", 200, 0, 4),
    (2000, 10, 6, "uniform", 400, 3, 4),        # three particles take all the moves
    (30000, 20, 6, "uniform", 2100, 0, 1),      # a tree of more than 1024 expansion rows
    (1000, 10, 6, "uniform", 18, 1, 8),         # one particle, few moves
])
def test_deferred_updates_match_move_by_move(n, npl, digits, kind, moves, few, slack):
    L = n ** (1 / 3)
    r, q = system(n, L, kind, n + digits)
    rng = np.random.default_rng(moves)
    idx = rng.integers(0, few if few else n, moves)
    disp = rng.uniform(-0.4, 0.4, (moves, 3))
    disp[::7] *= 1e-2  # short moves: the particle's own old place is a near source (terms up to 1e3)
    u = rng.uniform(0, 1, moves)
    out = []
    for mode in (P.MC_PERSISTENT, P.MC_GRAPH):
        t = P.HPDMKPtTree(P.HPDMKParams(n_per_leaf=npl, digits=digits, L=L, init=P.DIRECT), r, q, leaf_slack=slack)
        try:
            t.form_outgoing_pw()
            t.form_incoming_pw()
            t.set_mc_mode(mode)
            dE, acc = t.mc_run(idx, disp, u, 1.0)
            lv, _, leaf, _ = t.tree_nodes()
            inner = np.flatnonzero((lv >= 2) & (lv <= t.max_depth - 2) & (leaf == 0))
            some = inner[:: max(1, len(inner) // 6)]
            rows = [t.pw(0)] + [t.pw(int(b), w) for b in some for w in ("out", "inc")]
            dE2, acc2 = t.mc_run(idx[:3], disp[:3], u[:3], 1.0)  # the rows serve the next sequence
            out.append((dE, acc, t.positions(), rows, dE2, acc2))
        finally:
            t.close()
    a, b = out
    np.testing.assert_array_equal(a[1], b[1])
    assert 0 < a[1].sum()
    assert np.all(np.abs(a[0] - b[0]) <= ABS_DE * np.maximum(1.0, np.abs(b[0])))
    np.testing.assert_array_equal(a[2], b[2])
    for x, y in zip(a[3], b[3]):
        assert np.max(np.abs(x - y)) <= REL_PW * np.max(np.abs(y))
    assert np.all(np.abs(a[4] - b[4]) <= ABS_DE * np.maximum(1.0, np.abs(b[4])))
    np.testing.assert_array_equal(a[5], b[5])
