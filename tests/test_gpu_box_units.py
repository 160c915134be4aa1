"""The energy scales with the unit of length: a system shrunk or stretched by a
power of two has all positions scaled exactly, so its energy parts are the
unscaled ones times that power, to the rounding of each (1e-12 covers sums of 1e4
terms). Leaf sides reach from 1e-31 to 1e30, far beyond what single precision can
square."""
import numpy as np
import pytest

import pdmk4mc_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [P.PRECISION_FP64, P.PRECISION_MIXED])
@pytest.mark.parametrize("digits", [3, 9])
def test_energy_parts_scale_with_the_box(digits, precision):
    n, L = 1500, 8.0
    rng = np.random.default_rng(17)
    r = rng.uniform(0, L, 3 * n)
    q = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)

    def parts(s):
        t = P.HPDMKPtTree(P.HPDMKParams(n_per_leaf=20, digits=digits, L=L * s, init=P.DIRECT), r * s, q, precision=precision)
        try:
            t.form_outgoing_pw()
            t.form_incoming_pw()
            return t.eval_energy_parts() * s
        finally:
            t.close()

    want = parts(1.0)
    for k in (-100, -75, -62, 40, 58, 64, 100):
        np.testing.assert_allclose(parts(2.0 ** k), want, rtol=1e-12, atol=1e-12 * np.abs(want).max(), err_msg=str(k))
