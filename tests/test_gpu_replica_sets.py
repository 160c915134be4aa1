"""Sets of uneven trees, whose row updates share launches: one without expansion
levels beside shallow and deep ones, more moves than a list holds, some trees
without an accepted move. Each tree's energy shifts, then those of a second call on
its rows, and the rows themselves are those of the graphs of single moves.

The shifts differ by the order of fewer than 2e5 terms below 1e3, each rounded to
1.2e-16 of that with either sign: sqrt(2e5) * 1.2e-13 = 5e-11; a row of 150 moves
by 150 roundings of its terms of size one."""
import numpy as np
import pytest

import pdmk4mc_b200 as P

pytestmark = pytest.mark.gpu

ABS_DE = 2e-10


@pytest.mark.parametrize("digits", [3, 6, 9, 12])
def test_uneven_sets(digits):
    sizes = [(150, 200), (700, 8), (4000, 60), (2500, 6)]  # particles, n_per_leaf
    moves = 150
    systems, prop = [], []
    for k, (n, npl) in enumerate(sizes):
        rng = np.random.default_rng(60 + k)
        L = n ** (1 / 3)
        r = rng.uniform(0, L, (n, 3))
        if k == 3:
            r[:1200] = np.mod(0.3 * L + rng.normal(0, L / 60, (1200, 3)), L)
        systems.append((P.HPDMKParams(n_per_leaf=npl, digits=digits, L=L, init=P.DIRECT), r.reshape(-1),
                        np.where(np.arange(n) % 2 == 0, 1.0, -1.0)))
        u = np.where(np.arange(moves) % 2 == 0, -1.0, np.inf)
        prop.append((rng.integers(0, n, moves), rng.uniform(-0.3, 0.3, (moves, 3)), u if k != 2 else np.full(moves, np.inf)))

    def opened(k):
        t = P.HPDMKPtTree(*systems[k])
        t.form_outgoing_pw()
        t.form_incoming_pw()
        return t

    def rows(t):
        lv, _, leaf, _ = t.tree_nodes()
        inner = np.flatnonzero((lv >= 2) & (lv <= t.max_depth - 2) & (leaf == 0))
        return [t.pw(0)] + [t.pw(int(b), w) for b in inner[:: max(1, len(inner) // 8)] for w in ("out", "in")]

    want = []
    for k in range(len(sizes)):
        t = opened(k)
        t.set_mc_mode(P.MC_GRAPH)
        want.append([t.mc_run(*prop[k], 1.0), t.mc_run(*prop[k], 1.0), rows(t)])
        t.close()
    ts = [opened(k) for k in range(len(sizes))]
    try:
        for call in range(2):
            dE, acc = P.replicas_mc_run(ts, *(np.stack([p[c] for p in prop]) for c in range(3)), 1.0)
            for k in range(len(sizes)):
                np.testing.assert_array_equal(acc[k], want[k][call][1])
                assert np.all(np.abs(dE[k] - want[k][call][0]) <= ABS_DE * np.maximum(1.0, np.abs(want[k][call][0])))
        for k, t in enumerate(ts):
            for a, b in zip(rows(t), want[k][2]):
                assert np.max(np.abs(a - b)) <= 1e-11 * np.max(np.abs(b))
    finally:
        for t in ts:
            t.close()
