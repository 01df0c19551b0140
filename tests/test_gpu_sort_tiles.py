"""The key sort on both sides of the last number of tiles that are sorted in
two launches a pass (28 of 4,096 keys)."""
import pytest

import test_gpu_sort

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("equal", [False, True])
@pytest.mark.parametrize("n", [49153, 28 * 4096, 28 * 4096 + 1])
def test_order(pkg, oracle, n, equal):
    test_gpu_sort.test_order(pkg, oracle, n, equal)
