"""CPU check of the 64-bit headroom of the digit-slice ring products, for every ring length that
takes them (limits read from ss_digit.h)."""
import os
import re

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _limits():
    text = open(os.path.join(ROOT, "springsteel.jl_gb300", "csrc", "ss_digit.h")).read()
    return [int(re.search(r"constexpr int %s = (\d+);" % name, text).group(1))
            for name in ("kDigitFullRing", "kDigitMaxRing")]


def test_no_ring_sum_reaches_the_sign_bit():
    """In units of the columns' fixed point a term of a ring point is at most 2^53 in its cosine and
    in its sine part (2^52 at k = 0); |cos| + |sin| ≤ √2.  A quadrant part holds the cosine or the
    sine terms of one parity of k ≤ n − 1; rings above kDigitFullRing store it halved, rounded."""
    full, most = _limits()
    for n in range(2, most + 1):
        point = (0.5 + np.sqrt(2.0) * (n - 1)) * 2.0 ** 53
        part = (n // 2 + 1) * 2.0 ** 53
        forward = n * 2.0 ** 53
        assert part < 2.0 ** 63 and forward < 2.0 ** 63
        assert (point if n <= full else point / 2 + 4) < 2.0 ** 63, n


def test_the_bound_is_met_by_equal_parts():
    """re = ± im = c at every k comes within 0.9 of the bound: rings of more than 805 points a quadrant
    would wrap at full scale."""
    full, _ = _limits()
    n = 805
    theta = 2 * np.pi * (np.arange(n) + (n & 1) / 2) / (4 * n)
    a = np.outer(theta, np.arange(1, n))
    point = (0.5 + np.abs(np.cos(a)).sum(1) + np.abs(np.sin(a)).sum(1)).max()
    assert 2.0 ** 10 < point < np.sqrt(2.0) * n and n > full
