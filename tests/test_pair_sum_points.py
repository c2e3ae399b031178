"""The pair sums where a CTA holds more than four targets (fewer than 24 points
a fiber): one target less and more than a CTA's, idle lanes, a shard's ragged
end through the last CTA."""
import pytest

from test_pair_sum import test_against_oracle as against_oracle

pytestmark = pytest.mark.gpu


# targets of a CTA at 3, 6, 9, 12, 15, 18 and 21 points: 32, 16, 7, 8, 4, 5, 4
@pytest.mark.parametrize("M,N,NoQI", [(31, 5, 1), (33, 2, 1), (65, 8, 1), (17, 5, 2), (8, 3, 3), (20, 6, 3),
                                      (9, 5, 4), (15, 5, 4), (11, 5, 6), (9, 1, 7)])
@pytest.mark.parametrize("analytic", [1, 0])
def test_targets_per_cta(M, N, NoQI, analytic):
    against_oracle(M, N, NoQI, analytic)
