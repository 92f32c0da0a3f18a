"""What mixed precision and the coefficient fields of a line search may not cost: powers are rounded once, a run does
not drift from the state it stores, and trials stay as exact as fields formed anew."""
import numpy as np
import pytest

import maxlq_b200 as mlq

pytestmark = pytest.mark.gpu


def _power_norm_fp32(a, q, base32):
    """||u||_q^{q/2} of the constant field u = (a, 0, 0) for 4 < q < 6 as the FP32 path rounds it: S = |u|^2, A = g^2 and
    the product A g^(q/2 - 2), g = sqrt(S); every transform of a constant is exact for a power-of-two size."""
    f = np.float32
    s = f(f(a) * f(a))
    g = np.sqrt(s)  # FP32
    A = f(g * g)
    base = float(g) if base32 else np.sqrt(float(s))
    return float(f(A * f(base ** (q / 2.0 - 2.0))))


# The power's base stays in 64 bits: one rounding of g^k, one of the product.  The norm of a constant field then is the
# value above to the accuracy of the FP64 pow of the norm's root, some 1e-16; a base rounded to FP32 first moves it by up
# to 6e-8 k.
@pytest.mark.parametrize("q", [4.5, 5.0, 5.9])
def test_norm_power_of_a_constant_field_is_rounded_once(q):
    n = 16
    rng = np.random.default_rng(5)
    a = rng.uniform(0.5, 2.0, 512).astype(np.float32)
    differ = [x for x in a if _power_norm_fp32(x, q, False) != _power_norm_fp32(x, q, True)]
    assert len(differ) >= 8
    with mlq.MaxLq(n, q, 1.0, precision="mixed") as c:
        for x in differ[:8]:
            u = np.zeros((3, n, n, n))
            u[0] = float(x)
            want = _power_norm_fp32(x, q, False) ** (2.0 / q)
            assert abs(c.calc_global_Lq_norm(u) - want) <= 1e-14 * want
