"""Energy shifts next to particles that wait in the overflow pool: hundreds of
arrivals at full leaves are parked, then trial moves beside them are evaluated by
the persistent kernel's deferred form and by the graphs of single moves.

Tolerance: a shift sums fewer than 2e5 terms, each rounded to 1.2e-16 of at
most 1e3 (no two particles of the crowd are closer than 1e-3), with errors of
either sign: sqrt(2e5) * 1.2e-13 = 5e-11 a side. A pair of the crowd that is left
out or taken twice shows with its residual energy, about 1 / r = 0.1 to 10."""
import numpy as np
import pytest

import pdmk4mc_b200 as P

pytestmark = pytest.mark.gpu

ABS_DE = 2e-10


@pytest.mark.parametrize("digits", [3, 6, 9, 12])
@pytest.mark.parametrize("parked", [40, 140, 700])
def test_shifts_beside_parked_arrivals(digits, parked):
    n = 6000
    L = n ** (1 / 3)
    rng = np.random.default_rng(digits + parked)
    r = rng.uniform(0, L, (n, 3))
    q = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    # the crowd: a lattice over a corner of the box, spacing L / 4 / 9, a leaf's
    # neighbourhood wide; its particles come from outside that corner
    side = L / 4
    inside = np.all(r < side, axis=1)
    far = rng.permutation(np.flatnonzero(~inside))
    cell = rng.permutation(729)[:parked]
    goal = (np.stack([cell % 9, cell // 9 % 9, cell // 81], 1) + 0.5 + rng.uniform(-0.2, 0.2, (parked, 3))) * side / 9
    near = r[inside]
    gap = np.min(np.linalg.norm(goal[:, None] - near[None], axis=2))
    assert gap > 1e-3
    who = far[:parked]
    trials = np.concatenate([rng.choice(who, 100), rng.choice(np.flatnonzero(inside), 50), rng.choice(far[parked:], 50)])
    small = rng.uniform(-0.05, 0.05, (200, 3))
    small[150:] = rng.uniform(0, side, (50, 3)) - r[trials[150:]]  # from outside into the crowd
    idx = np.concatenate([who, trials])
    disp = np.concatenate([goal - r[who], small])
    u = np.concatenate([np.full(parked, -1.0), np.full(200, np.inf)])  # all of the first accepted, none of the others
    got = []
    for mode in (P.MC_PERSISTENT, P.MC_GRAPH):
        t = P.HPDMKPtTree(P.HPDMKParams(n_per_leaf=30, digits=digits, L=L, init=P.DIRECT), r.reshape(-1), q, leaf_slack=0)
        try:
            t.form_outgoing_pw()
            t.form_incoming_pw()
            t.set_mc_mode(mode)
            dE, acc = t.mc_run(idx, disp, u, 1.0)
            assert acc[:parked].all() and not acc[parked:].any()
            got.append(dE)
        finally:
            t.close()
    a, b = got
    assert np.all(np.abs(a - b) <= ABS_DE * np.maximum(1.0, np.abs(b)))
