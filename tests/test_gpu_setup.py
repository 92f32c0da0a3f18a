"""What mlq_init does and does not do."""
import pytest

import maxlq_b200 as mlq

pytestmark = pytest.mark.gpu


# the y/z tile shapes of 3 2^a follow a rule; a tuned context reports the times of the shapes that it launched
@pytest.mark.parametrize("n", [96, 192, 384])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_sizes_with_a_factor_3_are_not_tuned(n, precision):
    with mlq.MaxLq(n, 4.0, 1.0, precision=precision) as c:
        assert " ms" not in c.kernel_config()["yz_variants"]
