"""The tree build at the sizes where its sort and its level passes change form:
one block's sort up to 4096 pairs, radix passes above it (for the leaves the
passes whose digits can differ), bitmaps of the shallow levels in one launch and
of the deeper ones level by level. Nodes, neighbour lists and the particle order
are bit-exact with the oracle's."""
import numpy as np
import pytest

import pdmk4mc_b200 as P
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,npl,kind", [
    (2, 1, "uniform"), (33, 2, "uniform"), (4095, 30, "uniform"), (4096, 30, "uniform"), (4097, 30, "uniform"),
    (9001, 1, "uniform"),      # more than 4096 leaves
    (5000, 4, "point"),        # one tight cluster: levels beyond the shallow ones
    (4096, 30, "twins"),       # many equal keys: the order of equals is the input's
])
def test_build_matches_the_oracle(n, npl, kind):
    L = 7.0
    rng = np.random.default_rng(n + npl)
    r = rng.uniform(0, L, (n, 3))
    if kind == "point":
        r[: n // 2] = np.mod(L * 0.37 + rng.normal(0, L * 2e-3, (n // 2, 3)), L)
    if kind == "twins":
        r = r[rng.integers(0, 40, n)]
    r = r.reshape(-1)
    q = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    g = P.HPDMKPtTree(P.HPDMKParams(n_per_leaf=npl, digits=3, L=L, init=P.DIRECT), r, q)
    o = O.OracleTree(L, npl, 3, r, q)
    try:
        assert (g.max_depth, g.n_nodes) == (o.max_depth, o.n_nodes)
        for a, b in zip(g.tree_nodes(), o.tree_nodes()):
            np.testing.assert_array_equal(a, b)
        for a, b in zip(g.tree_neighbors(), o.tree_neighbors()):
            np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(g.sorted_order(), o.sorted_order())
    finally:
        g.close()


@pytest.mark.parametrize("n", [4097, 6144, 20481, 300001])
@pytest.mark.parametrize("kind", ["uniform", "line", "equal"])
def test_large_sorts_are_stable(n, kind):
    # tiles of 2048 keys: whole, one over, many; one digit value for all keys of a pass
    L = 5.0
    rng = np.random.default_rng(n)
    r = rng.uniform(0, L, (n, 3))
    if kind == "line":
        r[:, 1:] = 1.25
    if kind == "equal":
        r = r[rng.integers(0, 7, n)]
    q = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    # leaf sizes that keep the trees shallow: the order is what is tested
    g = P.HPDMKPtTree(P.HPDMKParams(n_per_leaf=n, digits=3, L=L, init=P.DIRECT), r.reshape(-1), q)
    try:
        cell = np.minimum(np.floor(r / L * 2.0 ** 21), 2 ** 21 - 1).astype(np.uint64)
        key = np.zeros(n, np.uint64)
        for b in range(21):
            for a in range(3):
                key |= ((cell[:, a] >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b + a)
        np.testing.assert_array_equal(g.sorted_order(), np.argsort(key, kind="stable"))
    finally:
        g.close()
