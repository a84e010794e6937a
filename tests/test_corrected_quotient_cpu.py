"""The codes of 16-bit inputs come from x y (y close to 1 / t) corrected once by the residual.  That quotient is far closer to x / t than
any rounding boundary is, except where x / t lies within a few units in the last place of one; there x and the boundary times t are
integers a few units apart, and this file goes through all such cases: divisors t of every significand for which 4, 5, 6 or 7 times it
(the boundaries' significands) lies next to a number of eleven significant bits (float16's, and so bfloat16's eight).
Reciprocals up to two units in the last place off are allowed, the device's is off by one at most."""
import numpy as np
import pytest

from oracle import ck_oracle as oc

# boundary significand -> powers of two that bring x / t to the boundaries of E2M1: 0.25 | 1.25, 2.5, 5 | 0.75 | 1.75, 3.5
SHIFTS = {4: (16.0,), 5: (1.0, 2.0, 4.0), 6: (8.0,), 7: (2.0, 4.0)}


def _f32(exact_head, error):
    """exact_head + error (float64 and the rest of an exact sum) rounded once to float32."""
    f = exact_head.astype(np.float32)
    tie = (exact_head.view(np.uint64) & np.uint64((1 << 29) - 1)) == np.uint64(1 << 28)
    toward = np.where(error > 0, np.inf, -np.inf)
    moved = np.nextafter(exact_head, toward).astype(np.float32)
    return np.where(tie & (error != 0), moved, f)


def _corrected(x, t, y):
    x, t, y = (v.astype(np.float64) for v in (x, t, y))
    p = (x * y).astype(np.float32).astype(np.float64)       # 48 bits: exact before it is rounded
    r = (t * p - x).astype(np.float32).astype(np.float64)   # neighbours: the difference is exact
    step = -(r * y)                                         # exact
    head = p + step
    back = head - p
    return _f32(head, (p - (head - back)) + (step - back))


@pytest.mark.parametrize("c", sorted(SHIFTS))
def test_every_divisor_with_a_boundary_next_to_a_short_number(c):
    m = np.arange(1 << 23, 1 << 24, dtype=np.int64)
    v = c * m
    short = (v + (1 << 14)) >> 15 << 15
    near = np.abs(v - short) <= 64
    if c == 4:
        near &= m != (1 << 24) - 1  # the significand of all ones, which the kernels send to the divisions
    m, short = m[near], short[near].astype(np.float32)
    assert m.size > 10_000
    for shift in SHIFTS[c]:
        t = (m * shift).astype(np.float32)
        exact = oc.f32_to_e2m1((short / t).astype(np.float32))
        y0 = (np.float32(1.0) / t).astype(np.float32)
        for ulps in (-2, -1, 0, 1, 2):
            y = (y0.view(np.int32) + np.int32(ulps)).view(np.float32)
            assert np.array_equal(oc.f32_to_e2m1(_corrected(short, t, y)), exact), (shift, ulps)


def test_the_significand_of_all_ones_is_the_exception():
    t = np.array([((1 << 24) - 1) * 16.0], dtype=np.float32)
    x = np.array([2.0 ** 26], dtype=np.float32)
    y = ((np.float32(1.0) / t).astype(np.float32).view(np.int32) - np.int32(1)).view(np.float32)
    assert oc.f32_to_e2m1(_corrected(x, t, y)) != oc.f32_to_e2m1((x / t).astype(np.float32))
