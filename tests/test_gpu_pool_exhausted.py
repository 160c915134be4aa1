"""An overflow pool that runs full: the call reports it, however the moves are run,
and the moves that found no room leave every particle in one place, so later calls
(which report it again) and a rebuild stay sound."""
import numpy as np
import pytest

import pdmk4mc_b200 as P

pytestmark = pytest.mark.gpu

N, L = 600, 600 ** (1 / 3)


def check_particles(t):
    lv, _, leaf, cnt = t.tree_nodes()
    assert cnt[0] == N and cnt[leaf != 0].sum() == N and cnt.min() >= 0
    pos = t.positions()
    assert np.all((pos >= 0) & (pos < L))
    assert len(np.unique(pos.reshape(-1, 3), axis=0)) == N  # nobody lost: a lost one would read as zeros or as another


@pytest.mark.parametrize("digits", [3, 9])
@pytest.mark.parametrize("form", ["short", "long", "unformed", "graph", "replicas", "single"])
def test_full_pool_is_reported_and_harmless(form, digits):
    rng = np.random.default_rng(9)
    r = rng.uniform(0, L, 3 * N)
    q = np.where(np.arange(N) % 2 == 0, 1.0, -1.0)
    prm = P.HPDMKParams(n_per_leaf=6, digits=digits, L=L, init=P.DIRECT)
    ts = [P.HPDMKPtTree(prm, r, q, leaf_slack=0, pool_capacity=5) for _ in range(2 if form == "replicas" else 1)]
    t = ts[0]
    try:
        for x in ts:
            if form != "unformed":
                x.form_outgoing_pw()
                x.form_incoming_pw()
        if form == "graph":
            t.set_mc_mode(P.MC_GRAPH)
        m = {"short": 6, "long": 300, "unformed": 300, "graph": 300, "replicas": 200, "single": 1}[form]

        def run():
            idx, disp, u = rng.integers(0, N, (2, m)), rng.uniform(-1.5, 1.5, (2, m, 3)), np.full((2, m), -1.0)
            if form == "replicas":
                P.replicas_mc_run(ts, idx, disp, u, 1.0)
            elif form == "single":
                t.eval_shift_energy(int(idx[0, 0]), *disp[0, 0])
                t.update_shift(int(idx[0, 0]), *disp[0, 0])
            else:
                t.mc_run(idx[0], disp[0], u[0], 1.0)

        errors = 0
        for _ in range(400 if m < 100 else 4):
            try:
                run()
                assert errors == 0  # the word stays set
            except P.HPDMKError as e:
                assert "overflow pool" in str(e)
                errors += 1
        assert errors >= 3
        for x in ts:
            check_particles(x)
            x.rebuild()
            e = x.eval_energy()
            f = P.HPDMKPtTree(prm, x.positions(), q)
            f.form_outgoing_pw()
            f.form_incoming_pw()
            assert abs(e - f.eval_energy()) <= 1e-11 * max(abs(e), 1.0) * N
            f.close()
    finally:
        for x in ts:
            x.close()
