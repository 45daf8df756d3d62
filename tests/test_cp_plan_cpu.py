"""Whether sequences are cut: the uncut scan starts the longest sequences first, each on the SM that is free first."""
import random

import pytest

from flashqla_b200 import cp


@pytest.mark.parametrize("chunks, heads, sms, makespan", [
    ([7], 3, 148, 7),
    ([10, 10], 2, 3, 20),            # four chains of ten on three SMs
    ([9, 5, 4, 1], 1, 2, 10),        # 9 + 1 | 5 + 4
    ([33] + [5] * 20, 8, 148, 33),   # the short ones beside the long one
])
def test_makespan(chunks, heads, sms, makespan):
    assert cp._uncut_makespan(chunks, heads, sms) == makespan


def test_unequal_lengths_that_fill_the_machine_are_not_cut():
    rng = random.Random(7)
    lens = [rng.randint(40, 2100) for _ in range(24)]
    assert not cp.plan_segments(lens, 8, 148).use_cp
    assert cp.plan_segments([2100] * 24, 4, 148).use_cp == (cp._uncut_makespan([33] * 24, 4, 148) > 33)
    assert cp.plan_segments([32768], 8, 148).use_cp and cp.plan_segments([32768, 100], 4, 148).use_cp
