"""The margin of the step's rounding test (nhf_math.cuh) against the errors of the
short evaluations that rely on it, from the documented bounds of the hardware's
approximations: log2 to 2^-22 of its value (absolute between 1/2 and 2), exp2 to
2^-22. Where the margin is wider than the error, a value that it lets pass has
the full evaluation's F32 bits."""
import re
from pathlib import Path

import numpy as np

CSRC = Path(__file__).resolve().parents[1] / 'nh-flood-2d_b200' / 'csrc'
TEXT = (CSRC / 'nhf_math.cuh').read_text()
LD, F = np.longdouble, np.float32
EXPONENT = F(7.0 / 3.0)
LN2 = np.log(LD(2))


def margin():
    """The test's half width, relative to a value whose unit is 2^-53 of it at least."""
    named = re.search(r'kOpenUnits = (\d+)', TEXT)
    units = int(named.group(1)) if named else int(re.search(r'0x10000000u - (\d+)u', TEXT).group(1))
    return units * 2.0 ** -53


def test_margin_covers_the_friction_power():
    c = abs(7.0 / 3.0 - float(EXPONENT))
    low, high = 1e-5, 2.0 ** 20
    w = c * max(abs(np.log(low)), np.log(high))
    logarithm, roundings = 2.0 ** -22, 3 * 2.0 ** -24       # constant, product, sum of w and w^2 / 2
    s = 2.0 ** -18                                            # of the estimate of x^(-1/3)
    series = 14 / 81 * (3 * s) ** 3 * 2                       # its third term enters squared
    bound = w * (logarithm + roundings) + w ** 3 / 6 + series + 12 * 2.0 ** -53
    assert bound < margin()


def test_margin_covers_the_horton_exponential():
    r = float(LN2) / 2 + 80 / float(LN2) * 2 * 2.0 ** -24    # the quotient is rounded in F32
    remainder = r ** 11 / 39916800 * 1.03 / np.exp(-r)
    reduction = 116 * float(LN2) * 2.0 ** -54
    assert remainder + reduction + 12 * 2.0 ** -53 < margin()


def short_power(x, log_error, exp_error):
    """friction_pow with the approximations off by their bounds."""
    exact = np.log2(x.astype(LD))
    lg = np.where((x > 0.5) & (x < 2), exact + log_error, exact * (1 + log_error)).astype(F)
    s = (np.exp2((lg * F(float.fromhex('-0x1.555556p-2'))).astype(LD)) * (1 + exp_error)).astype(F).astype(float)
    xd = x.astype(float)
    t = (1 - xd.astype(LD) * s.astype(LD) ** 3).astype(float)
    r = s + s * t * (1 / 3 + t * 2 / 9)
    v = (xd * xd) * ((xd * r) * r)
    w = lg * F(-(7.0 / 3.0 - float(EXPONENT)) * 0.693147180559945309)
    return v + v * (F(0.5) * w * w + w).astype(float)


def test_short_power_stays_inside_the_margin():
    rng = np.random.default_rng(3)
    x = np.exp(rng.uniform(np.log(1e-5), np.log(2.0 ** 20), 20000)).astype(F)
    x = np.concatenate([x, np.float32(2.0 ** 20) - np.arange(1, 2000, dtype=F) / 16, [F(1e-5), F(1), F(2), F(0.5)]])
    exact = np.exp(x.astype(LD) * 0 + LD(EXPONENT) * np.log(x.astype(LD)))
    for log_error in (-2.0 ** -22, 0, 2.0 ** -22):
        for exp_error in (-2.0 ** -22, 2.0 ** -22):
            off = np.abs(short_power(x, LD(log_error), LD(exp_error)) / exact - 1).max()
            assert off < margin(), float(np.log2(off))
