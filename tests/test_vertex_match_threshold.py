"""The classifier compares squared vertex distances: d2 < dtol^2 must decide like sqrt(d2) < dtol."""
import math


def test_square_of_the_tolerance_is_the_exact_threshold():
    dtol = 2.220446049250313e-16 * 1.0e3
    t = dtol * dtol
    assert math.sqrt(t) >= dtol and math.sqrt(math.nextafter(t, 0.0)) < dtol
