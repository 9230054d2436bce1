"""The bounds that the range kernel's windows rest on (range.cu), in exact integers: after i steps, F of
them odd, a seed n is at C n + rho with C = 3^F / 2^i, and D = 485 F - 306 i stands for C."""
import math
import random

import pytest

JW = 13


def test_sign_of_d_is_that_of_the_coefficient():
    """D > 0 exactly when 3^F > 2^i, for every F and 0 < i < 485."""
    for i in range(1, 485):
        for f in range(i + 1):
            assert (485 * f - 306 * i > 0) == (3 ** f > 1 << i), (i, f)


def test_seeds_from_which_the_coefficient_decides():
    """At the first i < 485 with C < 1, T^i(n) < n as soon as n (1 / C - 1) > F / 3 with F the odd steps; the negative
    map stays above m while C > 1 and m (1 - 1 / C) > F / 3.  Both hold from 2^16 on (with F at most the
    largest that the sign of C allows)."""
    below = above = 0
    for i in range(1, 485):
        f = (306 * i) // 485  # the largest F with C < 1
        lo, hi = 3 ** f, 3 ** (f + 1)
        below = max(below, f * lo / (3 * ((1 << i) - lo)))
        above = max(above, (f + 1) * hi / (3 * (hi - (1 << i))))
    assert below < 27_100 and above < 8_600
    # the distance of D / 306 from log2 C, which the limits' margins cover
    assert max(abs((485 * f - 306 * i) / 306 - (f * math.log2(3) - i)) for i in range(1, 485) for f in (0, (306 * i) // 485, i)
               if 485 * f - 306 * i >= -306) < 0.0024


def _step(x, neg):
    return ((3 * x - 1 if neg else 3 * x + 1) >> 1) if x & 1 else x >> 1


@pytest.mark.parametrize("neg", [False, True])
@pytest.mark.parametrize("bits", [17, 20, 32, 47, 64, 80, 95])
def test_windows_of_whole_trajectories(bits, neg):
    """Windows as the kernel takes them, against single steps: the value at a window's end, a seed called
    fallen has fallen, and D bounds every value until then."""
    rng = random.Random(bits * 2 + neg)
    for _ in range(400):
        n = rng.getrandbits(bits) | 1 << (bits - 1)
        n += max(0, (1 << 16) - n)
        x, d, steps, lg = n, 0, 0, math.log2(n)
        while steps + JW < 485:
            r, f, low, dd, y = x & ((1 << JW) - 1), 0, 0, 0, x
            fell, t = False, r
            for j in range(JW):
                dd += (179 if y & 1 else -306)
                f += y & 1
                y, t = _step(y, neg), _step(t, neg)
                low = min(low, dd)
                if d + low > 0 or not fell:
                    fell = fell or y < n
                if not fell:
                    assert 306 * (math.log2(y) - lg) <= d + dd + 1.83  # 306 (0.0024 + log2(1 + F / (3 n))) with F < 485; the kernel allows 2
                    assert d + dd > 0 or y == n
            assert y == (x >> JW) * 3 ** f + t  # the table's multiply-add
            steps += JW
            called = d < 128 * min(-low >> 7, 15) or d + dd < 0
            assert fell if called else True
            if called or fell:
                break
            x, d = y, d + dd
