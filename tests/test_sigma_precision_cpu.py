"""Significance of a power (accel_sigma_of_power) to double precision, against
the same equation solved with 40 digits.

Bound: log P(Gamma(n, 1) > x) and the logarithm of the Gaussian tail are each
within a few units of 2^-53 of their value, at most 8 together; with d sigma =
d log P / m and the inverse Mills ratio m above max(0.8, sigma), sigma moves by
at most 8 2^-53 max(|log P| / sigma^2, 1 / (0.8 sigma)) of itself: 4e-15 from
sigma = 0.5 on, tested at 1e-14.  (From 30 on the tail is an asymptotic series,
good to 3e-11.)"""
import random

import pytest

mp = pytest.importorskip("mpmath")


def exact(power, numharm, numindep, start):
    x = mp.mpf(power)
    logp = -x + mp.log(mp.fsum(x ** k / mp.factorial(k) for k in range(numharm)))
    if numindep > 1:
        logp += mp.log(numindep)
    return mp.findroot(lambda s: mp.log(mp.erfc(s / mp.sqrt(2)) / 2) - logp, start)


def test_sigma_to_double_precision():
    from gpu_accelsearch_gb300 import native as N
    f = N.lib().accel_sigma_of_power
    rng = random.Random(4)
    cases = [(3.92618399598226, 2, 1.0)]
    cases += [(10.0 ** rng.uniform(0.0, 3.0), rng.choice([1, 2, 4, 8, 16]), rng.choice([0.0, 1e3, 1e7, 1e12]))
              for _ in range(500)]
    tested = 0
    with mp.workdps(40):
        for case in cases:
            s = f(*case)
            if not 0.5 <= s <= 29.99:
                continue
            want = exact(*case, s)
            assert abs(s - want) <= 1e-14 * want, (case, s, float(want))
            tested += 1
    assert tested > 150
