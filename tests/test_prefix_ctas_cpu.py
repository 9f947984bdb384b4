"""How many SMs the shared-prompt attention phase gets, and into how many parts long keys are split (host rules, no GPU)."""

import pytest


@pytest.mark.parametrize("units,tiles,own_us,want", [
    (192, 8, 251.0, 64),  # the per-row phase is the longer one
    (128, 2, 91.0, 64),
    (48, 8, 36.0, 64),  # fewer units than SMs set aside
    (72, 7, 15.0, 72),  # one unit each instead of a second round
    (80, 4, 8.0, 80),
    (480, 8, 20.0, 148),  # the prompt phase is most of the work
    (1, 1, 0.0, 64),
])
def test_prefix_ctas(units, tiles, own_us, want):
    from diff_gpt_b200.model import gpt

    assert gpt.prefix_ctas(units, tiles, own_us, 148) == want
    assert gpt.prefix_ctas(units, tiles, own_us, 40) <= 40


@pytest.mark.parametrize("pairs,keys", [(1, 512), (8, 1000), (512, 3682), (1040, 1400), (1184, 4000), (1185, 4000), (2368, 4000)])
def test_splits_leave_one_wave(pairs, keys):
    from diff_gpt_b200.model import gpt

    n = gpt._pick_splits(pairs, keys)
    room = gpt._sm_count() * 16
    assert 1 <= n <= 64 and n <= keys // 256 and (n == 1 or n * pairs <= room)
