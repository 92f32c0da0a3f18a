"""Line searches at q != 4 and on the e_u branch: trials formed from the
coefficient fields of the search's setup against trials that evaluate R whole
(MLQ_REUSE=0 runs every program in its plain transform sequence).  The cases
cover each form that the |u|^k chain takes: a4 = A and an odd power in the
norm (q = 6), a4 and the norm the same field (q = 8), a fractional cut in the
norm (q = 3), raw powers (q = 5), a fractional power below the branch point
(q = 3.5), q = 4 with unit vectors, q < 4 without (negative powers), and
sizes with and without 3c = N on compile-time and run-time kernels."""
import numpy as np
import pytest

import maxlq_b200 as mlq

pytestmark = pytest.mark.gpu


def _trajectory(n, q, prec, iters, env, monkeypatch, **params):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    with mlq.MaxLq(n, q, 1.0, precision=prec, optim_tol=1e-14, **params) as c:
        c.state_load(c.seed_field(2, 2.0, n / 12))
        _, st, rec = c.state_iterate(iters)
        l = c.kernel_launches
    for k in env:
        monkeypatch.delenv(k)
    assert st == 0 and len(rec) == iters
    return rec, l


CASES = [(16, 6.0, {}), (64, 6.0, {}), (48, 8.0, {}), (64, 3.0, {}), (36, 3.0, {}), (32, 5.0, {}), (24, 3.5, {}),
         (32, 4.0, {"use_e_u_auto": 0, "use_e_u": 1}), (32, 3.0, {"use_e_u_auto": 0, "use_e_u": 0})]


# J1, R and the norm to 1e-9, the step and what follows from it to Brent's
# resolution of a flat minimum, 1e-7, as for q = 4 (test_gpu_reuse.py)
@pytest.mark.parametrize("transform_trials", ["0", "1"])
@pytest.mark.parametrize("n,q,params", CASES)
def test_trials_from_coefficient_fields_match_whole_evaluations(n, q, params, transform_trials, monkeypatch):
    plain, l0 = _trajectory(n, q, "fp64", 3, {"MLQ_REUSE": "0"}, monkeypatch, **params)
    fields, l1 = _trajectory(n, q, "fp64", 3, {"MLQ_LS_TRANSFORM_TRIALS": transform_trials}, monkeypatch, **params)
    assert l1 < l0  # the other path ran
    for a, b in zip(plain, fields):
        for k in ("J1", "R", "u_norm_q"):
            assert b[k] == pytest.approx(a[k], rel=1e-9), (a["iter"], k)
        for k in ("tau", "norm_grad", "norm_d1"):
            assert b[k] == pytest.approx(a[k], rel=1e-7), (a["iter"], k)
        assert b["beta"] == pytest.approx(a["beta"], rel=1e-7, abs=1e-7), a["iter"]


# FP32 trial values carry noise of some 1e-7 relative, which Brent resolves
# the minimum to the square root of (tau) and adds to J once
@pytest.mark.parametrize("n,q", [(64, 6.0), (48, 8.0), (64, 3.0)])
def test_mixed_precision_first_iteration(n, q, monkeypatch):
    (a,), _ = _trajectory(n, q, "fp64", 1, {}, monkeypatch)
    (b,), _ = _trajectory(n, q, "mixed", 1, {}, monkeypatch)
    assert b["J1"] == pytest.approx(a["J1"], rel=2e-5)
    assert b["tau"] == pytest.approx(a["tau"], rel=5e-3)


@pytest.mark.parametrize("q", [3.0, 6.0])
def test_nan_in_the_direction_is_reported(q):
    n = 32
    with mlq.MaxLq(n, q, 1.0) as c:
        u = c.seed_field(0, 2.0, 2.0)
        tb, flag = c.mnbrak(u, 0.1 * c.seed_field(1, 2.0, 2.0), 0.0, 0.1)
        assert np.isfinite(tb).all()
        bad = u.copy()
        bad[1, 2, 3, 4] = np.nan
        with pytest.raises(mlq.MlqError) as e:
            c.mnbrak(u, bad, 0.0, 0.1)
        assert e.value.status == mlq.MLQ_ERR_NAN
        assert np.isfinite(c.eval_J(u, "LineMin"))
