"""Dependent launches (a kernel's set-up overlaps its predecessor's end) against plain ones (MLQ_PDL=0): the same kernels
on the same data, so every record and the stored field agree to the last bit.  Sizes: 32 and 64 release their successor
early, 36 runs the run-time kernels, 96 and 128 the late release."""
import numpy as np
import pytest

import maxlq_b200 as mlq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,q,precision", [(32, 4.0, "fp64"), (32, 6.0, "mixed"), (36, 5.0, "fp64"), (64, 4.0, "mixed"),
                                           (64, 8.0, "fp64"), (64, 3.0, "fp64"), (96, 4.0, "mixed"), (96, 6.0, "fp64"),
                                           (128, 4.0, "fp64")])
def test_dependent_and_plain_launches_agree_to_the_bit(n, q, precision, monkeypatch):
    monkeypatch.setenv("MLQ_AUTOTUNE", "0")

    def run(pdl):
        monkeypatch.setenv("MLQ_PDL", pdl)
        with mlq.MaxLq(n, q, 1.0, precision=precision, optim_tol=0.0) as c:
            u = c.seed_field(4, 2.0, n / 12)
            c.state_load(u)
            _, st, rec = c.state_iterate(4)
            R, norm = c.state_R()
            for r in rec:
                del r["seconds"]
            return st, rec, R, norm, c.state_store(), c.GradL2ForLq(u)

    a, b = run("1"), run("0")
    assert a[0] == b[0] and a[1] == b[1] and a[3] == b[3]
    for i in (2, 4, 5):
        assert np.array_equal(a[i], b[i])
