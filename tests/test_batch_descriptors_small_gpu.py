"""The smallest set of descriptors that a rate-dematching launch carries in its arguments (20), and one more."""
import pytest

from test_batch_descriptors_gpu import test_rate_dematch_batches as check_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [19, 20, 21])
def test_smallest_argument_set(n):
    check_batch(n)
