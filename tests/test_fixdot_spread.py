"""The rule by which an entry of the stiffness integral stays on the integer pipes (csrc/element.cu,
k_int_tensor4_fix), restated in Python integers: the largest exponent of the entry's own terms against
those of the largest values of the element. Where the rule holds, the entry is within one rounding of its
largest term of the exact sum; values whose large partners never meet do not pass it."""

import random
from fractions import Fraction as F

import pytest

from test_fixdot_algebra import _exponent, limbs, mad, sum_limbs, to_double

NONE, SPREAD = -(1 << 14), 18


def _bound(d):
    return (_exponent(d) or 1) if d else NONE


def _entry(gv, C, g, ec, eg, ev):
    """(value on integers, largest exponent of a term): gv [q][i], C [q][i][l], g [q][l]."""
    acc, top = (0, 0, 0), NONE
    for v, c, n in zip(gv, C, g):
        for j, gl in enumerate(n):
            s, w = (0, 0, 0), NONE
            for vi, row in zip(v, c):
                s = mad(s, limbs(vi, ev), limbs(row[j], ec))
                w = max(w, _bound(vi) + _bound(row[j]))
            acc = mad(acc, sum_limbs(s), limbs(gl, eg))
            top = max(top, w + _bound(gl))
    return to_double(acc, ec + ev + eg - 3 * 1022 + 2), top


def _exact(gv, C, g):
    terms = [F(vi) * F(row[j]) * F(gl) for v, c, n in zip(gv, C, g) for j, gl in enumerate(n) for vi, row in zip(v, c)]
    return sum(terms), max(map(abs, terms))


def _values(r, nd, q):
    def one(*shape):
        if not shape:
            return r.choice([1, -1]) * r.uniform(0.01, 1.0)
        return [one(*shape[1:]) for _ in range(shape[0])]

    return one(q, nd), one(q, nd, nd), one(q, nd)


def _scales(gv, C, g):
    return (max(_exponent(x) for c in C for row in c for x in row), max(_exponent(x) for n in g for x in n),
            max(_exponent(x) for v in gv for x in v))


@pytest.mark.parametrize("nd", [2, 3])
def test_entry_at_the_limit_of_the_rule(nd):
    """The scales of the element as far above the entry's terms as the rule lets them lie."""
    r = random.Random(nd)
    for trial in range(60):
        gv, C, g = _values(r, nd, 2 ** nd)
        ec, eg, ev = _scales(gv, C, g)
        _, top = _entry(gv, C, g, ec, eg, ev)
        lift = SPREAD - (ec + eg + ev - top)
        a, b = sorted(r.randint(0, lift) for _ in range(2)) if trial % 3 else (lift, lift)
        got, again = _entry(gv, C, g, ec + a, eg + b - a, ev + lift - b)
        assert again == top
        exact, largest = _exact(gv, C, g)
        assert abs(F(got) - exact) <= F(2) ** -53 * (largest + abs(exact))


def test_points_of_different_scale_do_not_pass():
    """A tensor large at the point whose volume is small: blocks, directions and their largest values look
    alike, but no term comes near the product of the largest."""
    r = random.Random(3)
    for s in (12, 30, 60):
        gv, C, g = _values(r, 3, 8)
        gv[0] = [x * 2.0 ** -s for x in gv[0]]
        C[0] = [[x * 2.0 ** s for x in row] for row in C[0]]
        scales = _scales(gv, C, g)
        got, top = _entry(gv, C, g, *scales)
        exact, largest = _exact(gv, C, g)
        if top >= sum(scales) - SPREAD:
            assert abs(F(got) - exact) <= F(2) ** -53 * (largest + abs(exact))
        else:
            assert s > 12
    assert abs(F(got) - exact) > F(2) ** -40 * abs(exact)  # s = 60 on integers: what the rule keeps out


def test_zeros_have_no_term():
    gv, C, g = _values(random.Random(4), 3, 8)
    scales = _scales(gv, C, g)
    got, top = _entry(gv, [[[0.0] * 3 for _ in range(3)] for _ in range(8)], g, *scales)
    assert got == 0.0 and top < 0
