"""Large batches of candidates and points run in groups that share expansion
rows, small ones one by one: the same particles give the same numbers bit for
bit either way (a point's sums are formed in the same order in any group), at
every digits setting, for batches that do not divide into groups, with many
candidates of one particle, and with arrivals in the overflow pool; and they
agree with the single-move kernel within its parity tolerance."""
import numpy as np
import pytest

import pdmk4mc_b200 as P

pytestmark = pytest.mark.gpu

ABS_DE = 2e-10  # energy shifts, absolute (as in the parity tests)


@pytest.mark.parametrize("n,npl,digits,m,few,slack", [
    (3000, 20, 3, 1184, 0, 8),
    (3000, 20, 6, 1185, 5, 0),
    (6000, 20, 9, 1187, 0, 0),
    (2500, 12, 12, 1301, 0, 4),
    (150, 200, 9, 1190, 0, 8),   # no expansion levels
])
def test_groups_match_single_candidates(n, npl, digits, m, few, slack):
    rng = np.random.default_rng(n + digits)
    L = n ** (1 / 3)
    r = rng.uniform(0, L, 3 * n)
    q = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    t = P.HPDMKPtTree(P.HPDMKParams(n_per_leaf=npl, digits=digits, L=L, init=P.DIRECT), r, q, leaf_slack=slack)
    try:
        t.form_outgoing_pw()
        t.form_incoming_pw()
        k = 60  # some accepted moves first
        t.mc_run(rng.integers(0, n, k), rng.uniform(-0.4, 0.4, (k, 3)), np.full(k, -1.0), 1.0)
        idx = rng.integers(0, few if few else n, m)
        disp = rng.uniform(-0.5, 0.5, (m, 3))
        whole = t.eval_shift_energy_batch(idx, disp)
        parts = np.concatenate([t.eval_shift_energy_batch(idx[a:a + 500], disp[a:a + 500]) for a in range(0, m, 500)])
        np.testing.assert_array_equal(whole, parts)
        np.testing.assert_array_equal(whole, t.eval_shift_energy_batch_static(idx, disp))
        for c in range(0, m, 97):
            one = t.eval_shift_energy(int(idx[c]), *disp[c])
            assert abs(whole[c] - one) <= ABS_DE * max(1.0, abs(one)), (c, whole[c], one)
        phi, field = t.potential(idx)
        some = [t.potential(idx[a:a + 500]) for a in range(0, m, 500)]
        np.testing.assert_array_equal(phi, np.concatenate([s[0] for s in some]))
        np.testing.assert_array_equal(field, np.concatenate([s[1] for s in some]))
    finally:
        t.close()
