"""Which kernel and which split a decode step's projections take."""
import pytest

from them_bones_b200.utils.decode import rows_plan, use_rows


@pytest.mark.parametrize("sms", [64, 132, 148, 160])
def test_rows_plans_are_one_wave_that_covers_the_device(sms):
    for width in range(128, 4097, 128):
        for n, k in ((3 * width, width), (width, width), (4 * width, width), (width, 4 * width)):
            for b in (1, 16, 17, 64):
                plan = rows_plan(b, n, k, sms)
                if plan is None:
                    continue
                nt, s = plan
                assert n % nt == 0 and nt in (16, 32, 40, 48, 64) and s in (1, 2, 4, 8) and s <= k // 128
                assert n // nt * s <= (sms if s < 4 else 0.9 * sms) and (k <= 1536 * s or s == 8)
                assert n // nt * s >= sms // 2 or n <= 16 * sms       # few CTAs only where there are few columns
            assert rows_plan(65, n, k, sms) is None and rows_plan(64, n, k + 64, sms) is None


def test_a_step_takes_one_kernel_for_all_its_layers():
    assert use_rows(64, 1280, 1280, 5120, 148) and use_rows(4, 1280, 1280, 5120, 148) and use_rows(64, 1024, 1024, 4096, 148)
    assert not use_rows(65, 1280, 1280, 5120, 148) and not use_rows(64, 2048, 2048, 8192, 148) and not use_rows(16, 768, 768, 3072, 148) and use_rows(64, 256, 256, 1024, 148)
