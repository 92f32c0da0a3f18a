"""Compile-time pass kernels at N = 16, 32 and 3 2^a: against the oracle up to
N = 96, and above against the shared-memory Stockham kernels with run-time
plans (MLQ_PASS_KERNELS=reg selects those).  N = 16 and 32 are the shortest
lines, 48 the two-stage plan with the fewest threads per column, 96, 192 and
384 the three- and four-stage plans; N/3 + 1 columns leave a ragged last tile
at every size."""
import numpy as np
import pytest

import maxlq_b200 as mlq
from oracle.oracle import Oracle
from oracle.seedfield import seed_field

pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = np.asarray(a), np.asarray(b)
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


# tolerances of the parity tests: FP64 1e-10 for R and the gradient, 1e-12 for
# one round trip; mixed 2e-5 and 1e-3
@pytest.mark.parametrize("n,q", [(16, 4.0), (16, 3.0), (32, 6.0), (48, 4.0), (48, 3.0), (96, 6.0)])
def test_R_and_gradient_against_oracle(n, q):
    o = Oracle(n, q, 1.0)
    u = o.rescale(seed_field(n, 0, 2.0, n / 16))
    R, g = o.R_parts(u), o.grad_l2(u)
    with mlq.MaxLq(n, q, 1.0) as c:
        assert c.kernel_config()["pass_kernels"] == "compile-time"
        assert rel(c.calc_global_dLqdt_inclParts(u), R) < 1e-10
        assert rel(c.GradL2ForLq(u), g) < 1e-10
    with mlq.MaxLq(n, q, 1.0, precision="mixed") as m:
        assert rel(m.calc_global_dLqdt_inclParts(u), R) < 2e-5
        assert rel(m.GradL2ForLq(u), g) < 1e-3


@pytest.mark.parametrize("n", [16, 32, 48, 96])
def test_full_band_operators_and_dealias(n):
    """The full band reads the Nyquist column and keeps every row; the order
    1.5 cut is wider than the state band."""
    rng = np.random.default_rng(n)
    f = rng.standard_normal((n, n, n))
    u = rng.standard_normal((3, n, n, n))
    o = Oracle(n, 4.0)
    with mlq.MaxLq(n, 4.0, 1.0) as c:
        assert rel(c.gradient(f), o.gradient(f)) < 1e-12
        assert rel(c.divergence(u), o.divergence(u)) < 1e-12
        assert rel(c.laplacian(u), o.laplacian(u)) < 1e-12
        for order in (2.0, 1.5, 3.0):
            assert rel(c.dealias_scalar(f, order), o.dealias_scalar(f, order)) < 1e-12


def _run(n, precision, q, env, monkeypatch):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    with mlq.MaxLq(n, q, 1.0, precision=precision, optim_tol=1e-14) as c:
        u = c.seed_field(1, 2.0, n / 16)
        g = c.GradL2ForLq(u)
        out = {"g": g, "dealias": c.dealias_scalar(np.random.default_rng(3).standard_normal((n, n, n)), 2.0)}
        c.state_load(u)
        out["R"] = c.state_R()[0]
        _, st, rec = c.state_iterate(2)
        out["J1"] = [r["J1"] for r in rec]
        out["cfg"] = c.kernel_config()
    for k in env:
        monkeypatch.delenv(k)
    return out


def _same(b, a, precision):
    for k in ("dealias", "R"):
        assert rel(b[k], a[k]) < (1e-12 if precision == "fp64" else 2e-6), k
    assert rel(b["g"], a["g"]) < (1e-10 if precision == "fp64" else 1e-3)
    assert b["J1"] == pytest.approx(a["J1"], rel=1e-10 if precision == "fp64" else 1e-5)


@pytest.mark.parametrize("n,precision", [(96, "mixed"), (192, "fp64"), (192, "mixed"), (384, "mixed")])
def test_match_run_time_plans(n, precision, monkeypatch):
    a = _run(n, precision, 4.0, {"MLQ_PASS_KERNELS": "reg"}, monkeypatch)
    assert a["cfg"]["pass_kernels"] == "shared-memory"
    b = _run(n, precision, 4.0, {"MLQ_AUTOTUNE": "0"}, monkeypatch)
    assert b["cfg"]["pass_kernels"] == "compile-time"
    _same(b, a, precision)


@pytest.mark.parametrize("n,precision", [(16, "fp64"), (48, "fp64"), (48, "mixed"), (96, "fp64"), (192, "mixed")])
def test_reductions_of_the_z_stage(n, precision, monkeypatch):
    """Every trial of the line search by a transform, whose z stage sums the
    spectrum's squares and its products with three others: the chunks of a
    column's loads have to divide its elements (12 at 3 2^a)."""
    monkeypatch.setenv("MLQ_LS_TRANSFORM_TRIALS", "1")
    J = {}
    for kernels in ("reg", "compile-time"):
        monkeypatch.setenv("MLQ_PASS_KERNELS", kernels)
        with mlq.MaxLq(n, 4.0, 1.0, precision=precision, optim_tol=1e-14) as c:
            c.state_load(c.seed_field(1, 2.0, n / 16))
            _, _, rec = c.state_iterate(3)
            J[kernels] = [r["J1"] for r in rec]
    # FP32 trial values carry noise of 1e-7, which enters J once per iteration
    assert J["compile-time"] == pytest.approx(J["reg"], rel=1e-9 if precision == "fp64" else 1e-4)


@pytest.mark.parametrize("n,precision,variant", [(192, "fp64", 2), (192, "mixed", 1), (192, "mixed", 2),
                                                 (192, "mixed", 8), (384, "mixed", 8)])
def test_tile_variants_match_default(n, precision, variant, monkeypatch):
    a = _run(n, precision, 4.0, {"MLQ_AUTOTUNE": "0"}, monkeypatch)
    b = _run(n, precision, 4.0, {"MLQ_YZ_VARIANT": str(variant)}, monkeypatch)
    assert b["cfg"]["yz_variants"] == f"fixed by MLQ_YZ_VARIANT={variant}"
    _same(b, a, precision)
