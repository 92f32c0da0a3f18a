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


# A direction that undoes the base field: phi + tau d near tau = T is 64 times smaller than phi.  Sums of coefficient
# fields lose 64^2 there, polynomials of degree q 64^q; such trials evaluate R whole.  Those carry some q 64 roundings,
# 1e-13 of J at most, which moves Brent's minimum by some sqrt(1e-13) = 3e-7 of the bracket; the bound leaves a
# factor of 300.
@pytest.mark.parametrize("n,q", [(32, 6.0), (32, 8.0), (24, 8.0)])
def test_search_along_a_direction_that_undoes_the_field(n, q, monkeypatch):
    def search(reuse):
        monkeypatch.setenv("MLQ_REUSE", reuse)
        with mlq.MaxLq(n, q, 1.0) as c:
            v = c.rescaleLqNorm(c.seed_field(2, 2.0, n / 12))
            w = c.divAvg_free(c.HilbertGradient(c.GradL2ForLq(v), 1.5 - 1.0 / q))
            w *= np.sqrt((v * v).sum() / (w * w).sum())
            tb, flag = c.mnbrak(v, w, 0.0, 1.0)
            assert flag == 0
            T = 64.0
            return tb, c.brent(v - T * w, w, T + tb) - T, c.kernel_config()

    tb, x0, _ = search("0")
    _, x1, cfg = search("1")
    assert tb[0] < x0 < tb[1]
    assert abs(x1 - x0) <= 1e-4 * (tb[1] - tb[0])
    assert cfg["line_search_trials_whole"] > 0


# and a search of a run, whose directions are tangent to the constraint, needs none of them
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,q", [(32, 3.0), (32, 5.0), (48, 6.0), (32, 8.0)])
def test_searches_of_a_run_use_the_coefficient_fields(n, q, precision):
    with mlq.MaxLq(n, q, 1.0, precision=precision, optim_tol=0.0) as c:
        c.state_load(c.seed_field(3, 2.0, n / 12))
        c.state_iterate(6)
        cfg = c.kernel_config()
    assert cfg["line_search_trials_whole"] == 0
    if q in (6.0, 8.0):
        assert cfg["line_search_trials_polynomial"] > 0


# All trials of one search are formed one way: mnbrak along the full gradient (which undoes the field) brackets as with
# whole evaluations, also where steps are so small that J changes by the rounding of FP32.
@pytest.mark.parametrize("n,q", [(64, 5.0), (64, 3.0), (64, 8.0)])
def test_bracket_along_the_full_gradient_in_mixed_precision(n, q, monkeypatch):
    def search(reuse):
        monkeypatch.setenv("MLQ_REUSE", reuse)
        with mlq.MaxLq(n, q, 1.0, precision="mixed") as c:
            u = c.rescaleLqNorm(c.seed_field(0, 2.0, n / 12))
            d = c.divAvg_free(c.HilbertGradient(c.GradL2ForLq(u), 1.5 - 1.0 / q))
            d *= np.sqrt((u * u).sum() / (d * d).sum())
            tb, flag = c.mnbrak(u, d, 0.0, 1.0)
            return tb, flag, c.kernel_config()

    _, f0, c0 = search("0")
    _, f1, c1 = search("1")
    assert f0 == f1
    n0, n1 = c0["line_search_trials_whole"], c1["line_search_trials_whole"]
    assert n1 > 0 and c1["line_search_trials_polynomial"] == c1["line_search_trials_transform"] == 0


# and such a search takes no coefficient fields: 42 or more of a field's size
@pytest.mark.parametrize("n,q", [(32, 6.0), (24, 3.0)])
def test_whole_evaluations_need_no_search_fields(n, q):
    with mlq.MaxLq(n, q, 1.0) as c:
        u = c.rescaleLqNorm(c.seed_field(0, 2.0, n / 12))
        d = c.divAvg_free(c.HilbertGradient(c.GradL2ForLq(u), 1.5 - 1.0 / q))
        d *= np.sqrt((u * u).sum() / (d * d).sum())
        c.calc_global_dLqdt_inclParts(u)
        before = c.device_bytes
        tb, flag = c.mnbrak(u, d, 0.0, 1.0)
        assert flag == 0
        c.brent(u, d, tb)
        assert c.kernel_config()["line_search_trials_whole"] > 0
        assert c.device_bytes - before < 30 * 8 * n**3
