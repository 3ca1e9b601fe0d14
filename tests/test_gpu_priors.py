"""Posterior -> prior on both sides of the record count from which one block forms the alpha total
ahead of the others, against the oracle; a total that is negative or not a number leaves alpha_o
as it was, on either side."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("total", ["given", "positive", "negative", "nan", "none"])
@pytest.mark.parametrize("n", [1, 257, 65535, 65536, 70001])
def test_priors_around_the_total_of_its_own(cuda_ok, n, total):
    from tgmm_b200 import _lib as L
    from tgmm_b200 import engine as E
    rng = np.random.default_rng(n)
    g = np.zeros(n, L.GAUSS_DTYPE)
    for k in ("beta_k", "nu_k", "alpha_k"):
        g[k] = rng.uniform(60, 400, n)
    for k in ("beta_o", "nu_o", "alpha_o"):
        g[k] = rng.uniform(3, 30, n)
    g["W_k"], g["m_k"] = rng.uniform(0.01, 0.1, (n, 6)), rng.uniform(0, 900, (n, 3))
    if total == "negative":
        g["alpha_k"] *= -1
    elif total == "nan":
        g["alpha_k"][n // 2] = np.nan
    gm = E.gauss_to_device(g)
    E.update_priors(gm, n, 0.01, 1.0, 0.8, 1234.5 if total == "given" else -1.0, total != "none")
    got, want = E.gauss_from_device(gm), g.copy()
    atot = {"given": 1234.5, "positive": float(np.sum(g["alpha_k"]))}.get(total, -1.0)
    O.lib().or_update_priors(want.ctypes.data, n, 0.01, 1.0, 0.8, atot)
    if atot < 0:
        want["alpha_o"] = g["alpha_o"]
    for k in g.dtype.names:
        if k == "alpha_o" and total == "positive":
            # a sum of n positive terms in another order
            np.testing.assert_allclose(got[k], want[k], rtol=n * 2.3e-16 + 4e-16)
        elif k == "W_o":  # a product and a quotient: two roundings each
            np.testing.assert_allclose(got[k], want[k], rtol=5e-16)
        else:
            np.testing.assert_array_equal(got[k], want[k], err_msg=k)
