"""Crystals whose spacing divides the leaf's side have pairs at the cut-off itself,
where the residual kernel ends with the method's error: every form of a move has to
count them alike, whatever the last bit of the spacing. (A pair counted in one form
and not in the other shows with about 1e-4 over the spacing at 3 digits; the forms'
sums of fewer than 1e5 terms below 10 differ by sqrt(1e5) * 1.2e-15 = 4e-13.)"""
import numpy as np
import pytest

import pdmk4mc_b200 as P

pytestmark = pytest.mark.gpu


def test_pairs_at_the_cut_off():
    m, moves = 8, 120
    rng = np.random.default_rng(4)
    g = np.arange(m)
    site = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    n = len(site)
    q = np.where(site.sum(1) % 2 == 0, 1.0, -1.0)
    for L in np.concatenate([[8.0], rng.uniform(6.0, 10.0, 40)]):
        r = np.minimum(site * (L / m), np.nextafter(L, 0))
        # off the lattice, then on it again: pairs at all lattice distances, with other last bits
        off = rng.uniform(-0.4, 0.4, (moves // 2, 3)) * (L / m)
        who = rng.permutation(n)[: moves // 2]
        idx = np.concatenate([who, who])
        disp = np.concatenate([off, -off])
        got = []
        for mode in (P.MC_PERSISTENT, P.MC_GRAPH):
            t = P.HPDMKPtTree(P.HPDMKParams(n_per_leaf=4, digits=3, L=L, init=P.DIRECT), r.reshape(-1), q)
            try:
                t.form_outgoing_pw()
                t.form_incoming_pw()
                t.set_mc_mode(mode)
                got.append(t.mc_run(idx, disp, np.full(moves, -1.0), 1.0)[0])
            finally:
                t.close()
        assert np.all(np.abs(got[0] - got[1]) <= 1e-10 * np.maximum(1.0, np.abs(got[1]))), L
