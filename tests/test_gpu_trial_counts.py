"""kernel_config counts a trial as a polynomial one only where it transforms nothing but, at q = 6, its norm."""
import pytest

import maxlq_b200 as mlq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q,polynomial", [(3.0, False), (5.0, False), (6.0, True), (7.0, False), (8.0, True), (10.0, False)])
def test_trials_are_counted_by_how_they_are_formed(q, polynomial):
    with mlq.MaxLq(32, q, 1.0, optim_tol=0.0) as c:
        c.state_load(c.seed_field(3, 2.0, 32 / 12))
        c.state_iterate(3)
        k = c.kernel_config()
    assert (k["line_search_trials_polynomial"] > 0) == polynomial
    assert k["line_search_trials_polynomial"] + k["line_search_trials_transform"] > 0


# FP32 at q < 4 without unit vectors: the power |phi|^{q-4} amplifies what separately rounded coefficients leave at small
# |phi|
def test_negative_powers_evaluate_whole_in_mixed_precision():
    with mlq.MaxLq(32, 3.0, 1.0, precision="mixed", optim_tol=0.0, use_e_u_auto=0, use_e_u=0) as c:
        c.state_load(c.seed_field(3, 2.0, 32 / 12))
        c.state_iterate(3)
        k = c.kernel_config()
    assert k["line_search_trials_polynomial"] == k["line_search_trials_transform"] == 0
    assert k["line_search_trials_whole"] > 0
