"""The logarithm's short evaluation hands inputs whose rounding it leaves open
to the full one: the correctly rounded value where ln x lies next to the middle
of two doubles (found with the 64-bit mantissa of long double), around the
ends of the table's intervals, and at powers of two."""
import numpy as np
import pytest

from test_exp_sampler import correctly_rounded_ln


def check(oracle, x):
    got = oracle.ln(x)
    want = np.array([correctly_rounded_ln(float(v)) for v in x])
    bad = np.flatnonzero(got.view(np.uint64) != want.view(np.uint64))
    assert bad.size == 0, [(float(x[i]).hex(), got[i], want[i]) for i in bad[:5]]


@pytest.mark.parametrize("near", [-1, 0, 1])
def test_next_to_the_middle_of_two_doubles(oracle, near):
    if np.finfo(np.longdouble).nmant != 63:
        pytest.skip("long double has no 64-bit mantissa here")
    rng = np.random.default_rng(11 + near)
    x = (rng.integers(0, 2 ** 53, size=3_000_000, dtype=np.uint64) + np.uint64(1)).astype(np.float64) * 2.0 ** -53
    x = x[x < 1.0]
    m, _ = np.frexp(np.log(x.astype(np.longdouble)))
    low = (np.abs(m) * np.longdouble(2) ** 64).astype(np.uint64) & np.uint64(0x7FF)  # the bits past a double's
    hard = x[low == np.uint64(0x400 + near)]
    assert len(hard) > 800
    check(oracle, hard[:800])


def test_interval_ends_and_powers_of_two(oracle):
    ends = 0.701171875 + np.arange(0, 78) / 256.0
    x = np.concatenate([np.nextafter(ends, 0), ends, np.nextafter(ends, 2)] +
                       [2.0 ** -np.arange(1.0, 54.0), np.nextafter(2.0 ** -np.arange(1.0, 53.0), 1)])
    x = x[(x > 0) & (x < 1)]
    check(oracle, x)
