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


# At q != 4 every gradient transforms the stored state, so an evaluation between two iterations (which overwrites the
# physical fields of u) changes no bit of what follows.  A run that carried its fields from one retraction to the next
# would drift from its state instead.
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,q", [(32, 6.0), (32, 8.0), (24, 5.0), (48, 3.0)])
def test_gradient_of_a_run_is_that_of_its_state(n, q, precision):
    def run(evaluate):
        with mlq.MaxLq(n, q, 1.0, precision=precision, optim_tol=0.0) as c:
            c.state_load(c.seed_field(3, 2.0, n / 12))
            rec = []
            for _ in range(6):
                _, st, r = c.state_iterate(1)
                rec += r
                if st:
                    break
                if evaluate:
                    c.state_R()
            return rec, c.state_store()

    a, ua = run(False)
    b, ub = run(True)
    assert len(a) == len(b) >= 4
    for x, y in zip(a, b):
        for k in ("alpha", "beta", "norm_grad", "tau", "J1", "n_evals"):
            assert x[k] == y[k], (x["iter"], k)
    assert np.array_equal(ua, ub)
