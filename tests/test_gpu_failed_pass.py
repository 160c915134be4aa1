"""An outgoing pass that cannot get its memory raises and leaves box rows that read
as zero, not as the memory's last contents; a later pass works."""
import ctypes

import numpy as np
import pytest

import pdmk4mc_b200 as P

pytestmark = pytest.mark.gpu


def empty_pool():
    # what earlier trees left in the device's pool would serve the pass
    import torch
    torch.cuda.synchronize()
    rt = ctypes.CDLL("libcudart.so.12")  # the one torch has loaded
    pool = ctypes.c_void_p()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert rt.cudaMemPoolTrimTo(pool, ctypes.c_size_t(0)) == 0


def test_rows_stay_zero_when_a_pass_fails():
    import torch
    empty_pool()
    n = 400000
    L = n ** (1 / 3)
    rng = np.random.default_rng(5)
    r = rng.uniform(0, L, 3 * n)
    q = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    prm = P.HPDMKParams(n_per_leaf=200, digits=9, L=L, init=P.DIRECT)
    t = P.HPDMKPtTree(prm, r, q)
    try:
        t.form_outgoing_pw()  # its rows stay behind in the memory that the next tree gets
        t.form_incoming_pw()
        e = t.eval_energy()
    finally:
        t.close()
    t = P.HPDMKPtTree(prm, r, q, precision=P.PRECISION_MIXED)
    try:
        # the mixed pass needs tables of 0.5 GB for the root and 1.3 GB for the boxes
        torch.cuda.synchronize()
        hold = torch.empty(torch.cuda.mem_get_info()[0] - 1000000000, dtype=torch.uint8, device="cuda")
        with pytest.raises(P.HPDMKError):
            t.form_outgoing_pw()
        del hold
        torch.cuda.empty_cache()
        try:
            t.eval_shift_energy(0, 0.1, 0.1, 0.1)
        except P.HPDMKError:
            pass  # the runtime's last error is still the failed allocation's
        lv = t.tree_nodes()[0]
        for b in np.flatnonzero((lv >= 2) & (lv <= t.max_depth - 2))[::40]:
            assert not t.pw(int(b), "out").any()
        t.form_outgoing_pw()
        t.form_incoming_pw()
        assert abs(t.eval_energy() - e) <= 1e-7 * abs(e)
    finally:
        t.close()
