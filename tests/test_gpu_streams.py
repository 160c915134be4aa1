"""Streams and small buffers handed from one tree to the next: trees made,
used and closed by several threads at once give the energies that one after
another gives."""
import threading

import numpy as np
import pytest

import pdmk4mc_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads,held", [(1, 1), (6, 1), (3, 8)])
def test_trees_of_many_threads(threads, held):
    # held: trees a thread keeps open at once (24 trees return more streams than are kept)
    def system(k):
        rng = np.random.default_rng(100 + k)
        n = 400 + 60 * k
        q = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
        return rng.uniform(0, 6.0, 3 * n), q

    prm = P.HPDMKParams(n_per_leaf=20, digits=3, L=6.0, init=P.DIRECT)

    def energies(ks):
        ts = [P.HPDMKPtTree(prm, *system(k)) for k in ks]
        for t in ts:
            t.form_outgoing_pw()
            t.form_incoming_pw()
        out = [t.eval_energy() for t in ts]
        for t in ts:
            t.close()
        return out

    keys = list(range(held))
    want = energies(keys)
    got = [None] * threads

    def work(i):
        got[i] = [energies(keys) for _ in range(5)]

    ts = [threading.Thread(target=work, args=(i,)) for i in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for g in got:
        assert g is not None and all(e == want for e in g)


def test_single_moves_of_more_trees_than_result_slots():
    # 70 trees at once: the first 64 read their results from mapped memory, the
    # others copy them; an accepted move's new position shows in the next trial
    rng = np.random.default_rng(8)
    n, L = 60, 4.0
    r = rng.uniform(0, L, 3 * n)
    q = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    prm = P.HPDMKParams(n_per_leaf=10, digits=3, L=L, init=P.DIRECT)
    ts = [P.HPDMKPtTree(prm, r, q) for _ in range(70)]
    try:
        for t in ts:
            t.form_outgoing_pw()
            t.form_incoming_pw()
        first = [t.eval_shift_energy(5, 0.3, -0.2, 0.1) for t in ts]
        assert first == first[:1] * len(ts)
        for t in ts:
            t.update_shift(5, 0.3, -0.2, 0.1)
        back = [t.eval_shift_energy(5, -0.3, 0.2, -0.1) for t in ts]
        assert back == back[:1] * len(ts)
        # the way back undoes the move: two differences of the same two states
        assert abs(back[0] + first[0]) <= 1e-9 * max(1.0, abs(first[0]))
    finally:
        for t in ts:
            t.close()
