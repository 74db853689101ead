"""A plan of a decode projection is one that its kernel takes, at widths that no model has too."""
import pytest

from them_bones_b200.utils.decode import rows_plan


def _taken(n, k, nt, splits, sms):
    """The argument checks of bones_decode_rows, and the one wave that the plan is for."""
    return (k % 128 == 0 and 16 <= nt <= 64 and nt % 8 == 0 and n > 0 and n % nt == 0 and splits in (1, 2, 4, 8) and splits <= k // 128
            and n // nt * splits <= sms)


@pytest.mark.parametrize("sms", [64, 132, 148])
def test_plans_are_taken(sms):
    plans = 0
    for n in [*range(1, 200), *range(900, 1100), 1288, 1290, 2000, 3848, 5128, 10000]:
        for k in (128, 256, 384, 1000, 1280, 5120, 16384):
            plan = rows_plan(16, n, k, sms)
            assert plan is None or _taken(n, k, *plan, sms), (n, k, plan)
            plans += plan is not None
    assert plans > 100
