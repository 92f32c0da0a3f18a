"""What a context does after a failure inside an iteration.  The failures are made on the host (MLQ_INJECT)."""
import numpy as np
import pytest

import maxlq_b200 as mlq

pytestmark = pytest.mark.gpu



# A NaN met in the transport leaves the state as it was, and the next iteration is the one that failed, done again.  Its
# gradient transforms the state where the run that did not fail forms u from the retraction: 1e-13 apart, which Brent's
# flat minimum turns into 1e-7 of the step and the cancellation of deltaJ into 1e-9 of J.
@pytest.mark.parametrize("n,q", [(64, 4.0), (48, 4.0), (32, 6.0)])
def test_iteration_after_a_nan_in_the_transport(n, q, monkeypatch):
    def start():
        c = mlq.MaxLq(n, q, 1.0, optim_tol=0.0)
        c.state_load(c.seed_field(1, 2.0, n / 12))
        return c

    with start() as c:
        c.state_iterate(1)
        u1 = c.state_store()
        _, st, good = c.state_iterate(1)
        assert st == 0
        u2 = c.state_store()
    monkeypatch.setenv("MLQ_INJECT", "transport-nan=2")
    with start() as c:
        c.state_iterate(1)
        with pytest.raises(mlq.MlqError) as e:
            c.state_iterate(1)
        assert e.value.status == mlq.MLQ_ERR_NAN
        assert np.array_equal(c.state_store(), u1)
        _, st, again = c.state_iterate(1)
        assert st == 0
        a, g = again[0], good[0]
        for k in ("alpha", "beta", "norm_grad", "norm_d1", "J0", "J1"):
            assert abs(a[k] - g[k]) <= 1e-9 * abs(g[k]), k
        assert abs(a["tau"] - g["tau"]) <= 1e-6 * g["tau"]
        assert np.abs(c.state_store() - u2).max() <= 1e-6 * np.abs(u2).max()


# Where the device search's graph cannot be built the search runs on the host, and the iteration's record holds this
# update's scalars.  The field is smooth enough that every trial is a polynomial, so that no trial's fetch brings them.
@pytest.mark.parametrize("iters", [1, 3])
def test_record_of_a_search_without_its_graph(iters, monkeypatch):
    def run():
        with mlq.MaxLq(64, 4.0, 1.0, optim_tol=0.0) as c:
            u = c.seed_field(1, 2.0, 0.7)
            c.state_load(u)
            _, st, rec = c.state_iterate(iters)
            assert st == 0
            return rec, c.kernel_config()

    dev, cfg = run()
    assert cfg["line_searches_on_device"] == iters and cfg["line_search_trials_transform"] == 0
    monkeypatch.setenv("MLQ_INJECT", "ls-graph")
    host, cfg = run()
    assert cfg["line_searches_on_device"] == 0 and cfg["line_search_trials_transform"] == 0
    for a, b in zip(host, dev):
        for k in ("alpha", "beta", "norm_grad", "norm_td0", "norm_d1", "tau", "J1"):
            assert abs(a[k] - b[k]) <= 1e-9 * abs(b[k]), (b["iter"], k)


# A search at q != 4 that cannot have its fields (the k-th allocation fails: the block of fields, a spectrum of the setup
# or one of a trial) evaluates R whole, and the next run asks again.  Trials both ways agree as in
# test_gpu_general_line_search.py.
@pytest.mark.parametrize("n,q,k", [(n, q, k) for n, q in ((32, 6.0), (24, 8.0), (32, 3.0)) for k in (1, 2, 6, 12)
                                   if (q, k) != (3.0, 12)])  # a search at q = 3 makes fewer than 12
def test_search_without_memory_for_its_fields(n, q, k, monkeypatch):
    def run(c):
        c.state_load(c.seed_field(2, 2.0, n / 12))
        _, st, rec = c.state_iterate(2)
        assert st == 0
        return rec

    with mlq.MaxLq(n, q, 1.0, optim_tol=0.0) as c:
        good = run(c)
    monkeypatch.setenv("MLQ_INJECT", f"search-oom={k}")
    with mlq.MaxLq(n, q, 1.0, optim_tol=0.0) as c:
        first = run(c)
        whole = c.kernel_config()["line_search_trials_whole"]
        assert whole > 0
        again = run(c)
        assert c.kernel_config()["line_search_trials_whole"] == whole
    for rec in (first, again):
        for a, b in zip(rec, good):
            assert abs(a["J1"] - b["J1"]) <= 1e-9 * abs(b["J1"])
            assert abs(a["tau"] - b["tau"]) <= 1e-7 * max(b["tau"], 1e-2)


# The fields of a search stay with their context, but not against another context's need: with memory for a second
# context only where the first gives its fields back, the second runs, and the first goes on.
def test_a_context_gives_its_search_fields_back():
    import torch

    n, q = 128, 6.0

    def run(c, iters):
        _, st, rec = c.state_iterate(iters)
        assert st == 0
        return rec

    with mlq.MaxLq(n, q, 1.0, optim_tol=0.0) as c:
        u = c.seed_field(2, 2.0, n / 12)
        c.state_load(u)
        good = run(c, 2)
        held = c.device_bytes
    with pytest.MonkeyPatch.context() as mp:
        mp.setenv("MLQ_REUSE", "0")
        with mlq.MaxLq(n, q, 1.0, optim_tol=0.0) as c:
            c.state_load(u)
            run(c, 1)
            plain = c.device_bytes
    fields = held - plain
    assert fields > 40 * 8 * n**3
    with mlq.MaxLq(n, q, 1.0, optim_tol=0.0) as a:
        a.state_load(u)
        ra = run(a, 1)
        full = a.device_bytes
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        ballast = torch.empty(free - (plain - fields // 2), dtype=torch.uint8, device="cuda")
        try:
            with mlq.MaxLq(n, q, 1.0, optim_tol=0.0) as b:
                b.state_load(u)
                rb = run(b, 2)
                assert a.device_bytes < full - 40 * 8 * n**3
                ra += run(a, 1)
        finally:
            del ballast
            torch.cuda.empty_cache()
    for rec in (ra, rb):
        for x, y in zip(rec, good):
            assert abs(x["J1"] - y["J1"]) <= 1e-9 * abs(y["J1"])
