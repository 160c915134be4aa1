"""Device calls captured on a tree's stream and replayed: the energy afterwards is
that of a tree built from the positions read back, and other calls beside a
replay give what they give alone."""
import numpy as np
import pytest

import pdmk4mc_b200 as P

pytestmark = pytest.mark.gpu

N, L = 4000, 16.0


def params(digits=6):
    return P.HPDMKParams(n_per_leaf=20, digits=digits, L=L, init=P.DIRECT)


def system():
    rng = np.random.default_rng(3)
    return rng.uniform(0, L, 3 * N), np.where(np.arange(N) % 2 == 0, 1.0, -1.0)


def energy(t):
    t.form_outgoing_pw()
    t.form_incoming_pw()
    return t.eval_energy()


class Sequence:
    def __init__(self, m, seed):
        import torch
        rng = np.random.default_rng(seed)
        self.m = m
        self.i = torch.as_tensor(rng.integers(0, N, m).astype(np.int32), device="cuda")
        self.d = torch.as_tensor(rng.uniform(-0.5, 0.5, 3 * m), device="cuda")
        self.u = torch.full((m,), -1.0, dtype=torch.float64, device="cuda")  # every move accepted
        self.dE = torch.zeros(m, dtype=torch.float64, device="cuda")
        self.acc = torch.zeros(m, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()

    def run(self, t):
        t.mc_run_device(self.m, self.i.data_ptr(), self.d.data_ptr(), self.u.data_ptr(), 1.0, self.dE.data_ptr(),
                        self.acc.data_ptr())


def capture(t, f):
    import torch
    t.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.ExternalStream(t.stream_ptr())):
        f()
    return g


def replay(t, g):
    import torch
    t.synchronize()
    g.replay()
    torch.cuda.synchronize()


@pytest.mark.parametrize("precision", [P.PRECISION_FP64, P.PRECISION_MIXED])
@pytest.mark.parametrize("slack", [8, 0])  # 0: arrivals go to the overflow pool
@pytest.mark.parametrize("moves", [8, 200])  # rows updated move by move, and deferred
def test_energy_after_replayed_moves(moves, slack, precision):
    r, q = system()
    t = P.HPDMKPtTree(params(), r, q, precision=precision, leaf_slack=slack)
    try:
        e = energy(t)
        s = Sequence(moves, moves)
        s.run(t)
        g = capture(t, lambda: s.run(t))
        for _ in range(3):
            e = energy(t)
            replay(t, g)
            assert s.acc.all()
            e2 = energy(t)
            f = P.HPDMKPtTree(params(), t.positions(), q, precision=precision)
            want = energy(f)
            f.close()
            # two trees' sums of one system at 6 digits: each is within 1e-6 of the
            # energy, of size 1e3 here, and its shifts add up to the same
            assert abs(e2 - want) <= 2e-6 * max(1e3, abs(want))
            assert abs(e2 - e - float(s.dE.sum())) <= 2e-6 * max(1e3, abs(want))
        del g
    finally:
        t.close()


@pytest.mark.parametrize("warm,captured,after", [(8, 200, 600), (200, 8, 30), (20, 600, 600), (600, 600, 20)])
def test_captured_and_direct_sequences_share_a_tree(warm, captured, after):
    # neither leaves the other with memory that belongs to a graph. Shifts as in
    # the move-by-move form: under 2e5 terms below 1e3, rounded to 1.2e-16 of that
    r, q = system()
    parts = [Sequence(m, 50 + k) for k, m in enumerate((warm, captured, after))]
    order = (0, 1, 2, 1)
    want = []
    t = P.HPDMKPtTree(params(), r, q)
    try:
        energy(t)
        t.set_mc_mode(P.MC_GRAPH)
        for k in order:
            parts[k].run(t)
            t.synchronize()
            want.append(parts[k].dE.cpu().numpy())
    finally:
        t.close()
    t = P.HPDMKPtTree(params(), r, q)
    try:
        energy(t)
        parts[0].run(t)
        t.synchronize()
        got = [parts[0].dE.cpu().numpy()]
        g = capture(t, lambda: parts[1].run(t))
        for k in order[1:]:
            if k == 1:
                replay(t, g)
            else:
                parts[k].run(t)
                t.synchronize()
            got.append(parts[k].dE.cpu().numpy())
        del g
    finally:
        t.close()
    for a, b in zip(got, want):
        assert np.all(np.abs(a - b) <= 2e-10 * np.maximum(1.0, np.abs(b)))


def test_captured_batch_beside_direct_ones():
    # the graph runs on another stream while the tree's own evaluates other batches
    import torch
    r, q = system()
    t = P.HPDMKPtTree(params(), r, q)
    try:
        energy(t)
        a, b = Sequence(3000, 1), Sequence(1500, 2)

        def batch(s):
            t.eval_shift_energy_batch_device(s.m, s.i.data_ptr(), s.d.data_ptr(), s.dE.data_ptr())

        want = []
        for s in (a, b):
            batch(s)
            t.synchronize()
            want.append(s.dE.clone())
        g = capture(t, lambda: batch(a))
        other = torch.cuda.Stream()
        for _ in range(20):
            a.dE.zero_()
            b.dE.zero_()
            torch.cuda.synchronize()
            with torch.cuda.stream(other):
                g.replay()
            batch(b)
            torch.cuda.synchronize()
            t.synchronize()
            assert torch.equal(a.dE, want[0]) and torch.equal(b.dE, want[1])  # whatever the groups
        del g
    finally:
        t.close()
