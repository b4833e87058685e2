"""The straight-line FP64 division over the whole range in which the kernels use it (B200 required).

The optical-depth bound of a step divides by rates down to 2^-200 and the RK45 step controller by errors up to
2^400, so the self-test has to take such divisors as its own and not count them as out of range."""
import pytest

from engine_fixtures import dms_b200

pytestmark = pytest.mark.gpu


def test_division_equals_ieee_over_its_whole_range():
    n = 1 << 24
    with dms_b200.Engine(0) as e:
        bad, outside = e.check_certified_math(n, seed=3)[:2]
    assert bad == 0
    # A quarter of the pairs are arbitrary bit patterns: 600 of 2 048 exponents of the divisor and 1 100 of the
    # dividend are in range, so 0.21 of all pairs are outside; 0.24 with divisors from 2^-100 to 2^100 only.
    assert 0.18 * n < outside < 0.225 * n
