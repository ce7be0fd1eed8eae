"""How a portion of tokens is cut into passes."""
import random

import pytest

from mi50grad_b200.engine.engine import portion_passes


def check(n, want, few, wide, logit_rows, many):
    got, at = portion_passes(n, want, few, wide, logit_rows, many), 0
    for i, c, hit in got:
        assert i == at and c >= 1 and hit == any(i <= w < i + c for w in want)
        few_row = c <= few and (i + c == n or not many)
        assert few_row or (many and c <= (min(wide, logit_rows) if hit else wide))
        at += c
    assert at == n
    return got


@pytest.mark.parametrize("n,want,passes", [(3000, [2999], [2999, 1]), (5000, [4999], [4096, 903, 1]), (3000, [], [3000]), (9000, [], [4096, 4096, 808]),
                                           (1000, [10, 999], [10, 8, 981, 1]), (1000, [7], [8, 992]), (8, [0, 7], [8]), (20, [3], [8, 12])])
def test_rows_in_front_of_a_wanted_place_run_at_full_width(n, want, passes):
    assert [c for _, c, _ in check(n, want, 8, 4096, 8, True)] == passes


def test_many_wanted_places_and_other_limits():
    assert [c for _, c, _ in check(1200, range(0, 1200, 7), 8, 4096, 512, True)] == [512, 512, 176]
    assert [c for _, c, _ in check(20, [19], 8, 4096, 8, False)] == [8, 8, 4]
    r = random.Random(1)
    for _ in range(500):
        n = r.randint(1, 700)
        check(n, [r.randrange(n) for _ in range(r.randint(0, 5))], r.randint(1, 8), r.choice([64, 512, 4096]), r.choice([8, 64, 512]), r.random() < 0.8)
