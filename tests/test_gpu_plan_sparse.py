"""The row plan of few slots over thousands of bins (one CTA, two words per bin) at the ends of its range, against a stable
sort on the CPU."""

import pytest

from tests.test_gpu_plan import test_plan_matches_a_stable_sort as matches_a_stable_sort

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K,E,cap,lo,n_local", [
    (1, 1, 4000, 0, 0, 4000),       # one slot
    (400, 8, 1024, 5, 0, 1024),     # capacity per (expert, k)
    (512, 8, 4500, 0, 0, 4500),     # the most slots of this launch
    (513, 8, 4500, 0, 0, 4500),     # one token more: the general launches
    (200, 4, 6144, 0, 0, 6144),     # exactly 48 KiB of shared memory
    (37, 4, 9000, 0, 1000, 5000),   # experts of one rank only
    (100, 2, 40000, 0, 0, 40000),   # bins beyond shared memory
])
def test_few_slots_over_many_bins(N, K, E, cap, lo, n_local):
    matches_a_stable_sort(N, K, E, cap, lo, n_local)
