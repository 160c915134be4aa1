"""Boxes at the edges of the outgoing pass's cut (256 particles an item): boxes of
0, 1, 255, 256, 257, 512 and 513 particles and their children, against the sums
written out on the host.

A row entry is a sum of m phases of size one. FP64: an axis factor comes out of
at most 26 roundings after its sincos, and the host's argument (below 120) is
rounded once per axis, 400 u a term in all. Mixed: operands in fixed point with
2^-25 of their range each and products dropped below 1e-9 of it, 3e-9 a term. A
particle that is left out or taken twice shows with one."""
import numpy as np
import pytest

import pdmk4mc_b200 as P

pytestmark = pytest.mark.gpu

COUNTS = (0, 1, 255, 256, 257, 512, 513)


@pytest.mark.parametrize("precision,term", [(P.PRECISION_FP64, 400 * 2.0 ** -53), (P.PRECISION_MIXED, 3e-9)])
@pytest.mark.parametrize("cut", [256, 16384])
def test_rows_of_boxes_at_the_cut(precision, term, cut):
    L, digits, n_diff, n_win = 16.0, 6, 12, 8
    rng = np.random.default_rng(41)
    size = [COUNTS[k % len(COUNTS)] for k in range(64)]
    r = np.concatenate([np.array([k % 4, k // 4 % 4, k // 16]) * 4.0 + rng.uniform(0, 4.0, (c, 3)) for k, c in enumerate(size)])
    r = np.minimum(r, np.nextafter(L, 0))
    n = len(r)
    q = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    order = rng.permutation(n)
    r, q = np.ascontiguousarray(r[order]), q[order]
    t = P.HPDMKPtTree(P.HPDMKParams(n_per_leaf=20, digits=digits, L=L, init=P.DIRECT), r.reshape(-1), q, precision=precision)
    try:
        t.set_tuning(ksplit=cut, ksplit_root=cut)
        t.form_outgoing_pw()
        lv, prefix, _, cnt = t.tree_nodes()
        level2 = np.flatnonzero(lv == 2)
        assert t.max_depth >= 5 and sorted(cnt[level2].tolist()) == sorted(size)  # boxes with rows
        pick = [int(b) for b in level2[:14]] + [int(b) for b in np.flatnonzero(lv == 3)[::37]]

        def host(inside, dk, m):
            k = np.arange(-m, m + 1) * dk
            f = [np.exp(-1j * np.outer(r[inside, a], k)) for a in range(3)]
            return np.einsum("j,jz,jy,jx->zyx", q[inside], f[2][:, : m + 1], f[1], f[0], optimize=True).reshape(-1)

        for b in pick:
            l = int(lv[b])
            p = int(prefix[b])
            box = np.array([sum(((p >> (3 * i + a)) & 1) << i for i in range(l)) for a in range(3)])
            inside = np.flatnonzero(np.all(np.floor(r / L * 2 ** l) == box, axis=1))
            assert len(inside) == cnt[b]
            want = host(inside, 2 * np.pi / (3 * L / 2 ** l), n_diff)
            assert np.abs(t.pw(b) - want).max() <= term * max(1, len(inside)), (l, len(inside))
        want = host(np.arange(n), 2 * np.pi / L, n_win)
        assert np.abs(t.pw(0) - want).max() <= term * n
    finally:
        t.close()
