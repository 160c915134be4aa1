"""The device-side layout of the outgoing pass: boxes cut into many items,
several blocks of nodes, empty boxes and trees without expansion levels give
the rows that uncut boxes give, and the energy follows."""
import numpy as np
import pytest

import pdmk4mc_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [P.PRECISION_FP64, P.PRECISION_MIXED])
@pytest.mark.parametrize("n,npl,kind", [
    (600, 700, "uniform"),     # no level with expansions
    (5000, 12, "uniform"),     # many blocks of nodes, boxes below the cut
    (20001, 40, "point"),      # deep tree, boxes of one to many items, empty boxes
    (16640, 2000, "uniform"),  # boxes of 256 and 257 particles and a few more
])
def test_cut_boxes_match_whole_ones(n, npl, kind, precision):
    L = 9.0
    rng = np.random.default_rng(n)
    r = rng.uniform(0, L, (n, 3))
    if kind == "point":
        r[: n // 2] = np.mod(L * 0.4 + rng.normal(0, L * 4e-3, (n // 2, 3)), L)
    q = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    prm = P.HPDMKParams(n_per_leaf=npl, digits=6, L=L, init=P.DIRECT)
    t = P.HPDMKPtTree(prm, r.reshape(-1), q, precision=precision)
    try:
        lv, _, _, cnt = t.tree_nodes()
        rows = [0] + [int(b) for b in np.nonzero((lv >= 2) & (lv <= t.max_depth - 2))[0]]
        got = []
        for k in (16384, 256):
            t.set_tuning(ksplit=k, ksplit_root=k)
            t.form_outgoing_pw()
            t.form_incoming_pw()
            got.append(([t.pw(b) for b in rows], t.eval_energy()))
        for b, x, y in zip(rows, got[0][0], got[1][0]):
            # two orders of a sum of m terms of size one, an m u m error each
            m = int(cnt[b])
            assert np.abs(x - y).max() <= 2 * m * m * 2.0 ** -53 + 1e-300, b
        # the row errors above reach the energy through its quadratic form: eight
        # digits are far above them and far below any missing item
        assert abs(got[0][1] - got[1][1]) <= 1e-8 * abs(got[0][1])
    finally:
        t.close()


@pytest.mark.parametrize("first", ["shift", "captured", "incoming", "rows"])
def test_rows_are_zero_until_a_pass_forms_them(first):
    # the pool hands out memory that an earlier tree has written
    import torch
    n, L = 4000, 8.0
    rng = np.random.default_rng(3)
    r = rng.uniform(0, L, 3 * n)
    r[: 3 * 1500] = np.mod(4.0 + rng.normal(0, 0.1, 3 * 1500), L)  # leaves on the expansion levels
    q = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    prm = P.HPDMKParams(n_per_leaf=20, digits=3, L=L, init=P.DIRECT)
    old = P.HPDMKPtTree(prm, r, q)
    old.form_outgoing_pw()
    old.form_incoming_pw()
    e_old = old.eval_energy()
    idx, disp = np.arange(64) * 60, rng.uniform(-0.3, 0.3, (64, 3))
    d_old = np.array(old.eval_shift_energy_batch(idx, disp))
    old.close()
    t = P.HPDMKPtTree(prm, r, q)
    try:
        lv, _, leaf, _ = t.tree_nodes()
        rows = np.nonzero((lv >= 2) & (lv <= t.max_depth - 2))[0]
        if first == "shift":
            t.eval_shift_energy(0, 0.1, 0.1, 0.1)
        elif first == "captured":
            s = torch.cuda.ExternalStream(t.stream_ptr())
            di = torch.tensor(idx.astype(np.int32), device="cuda")
            dd = torch.tensor(disp, device="cuda")
            de = torch.zeros(64, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=s):
                t.eval_shift_energy_batch_device(64, di.data_ptr(), dd.data_ptr(), de.data_ptr())
        elif first == "incoming":
            t.form_incoming_pw()
        if first in ("shift", "rows"):
            for b in rows[:: max(1, len(rows) // 50)]:
                assert not t.pw(int(b), "out").any() and not t.pw(int(b), "in").any()
        t.form_outgoing_pw()
        t.form_incoming_pw()
        if first == "captured":
            t.synchronize()  # the replay runs on another stream
            graph.replay()
            torch.cuda.synchronize()
            np.testing.assert_array_equal(de.cpu().numpy(), d_old)
        assert t.eval_energy() == e_old
        np.testing.assert_array_equal(np.array(t.eval_shift_energy_batch(idx, disp)), d_old)
        for b in rows[leaf[rows] != 0][:20]:
            assert not t.pw(int(b), "in").any()
    finally:
        t.close()
