"""The straight NVFP4 blocks bracket the E4M3 scale RN(RN(amax / 6) / g) by amax * c(1 +- 2^-21), c = RN(1 / RN(6 g)), and
the codes with a reciprocal that may be one unit in the last place off.  Both rules in float32 numpy against the
exact chains, on random operands and a few ulps around every rounding boundary."""
import numpy as np
import pytest

from oracle import ck_oracle as oc

F = np.float32
HI, LO = F(1.0 + 2.0 ** -21), F(1.0 - 2.0 ** -21)


def _scale_byte(s):
    return oc.f32_to_e4m3(np.minimum(s, F(448.0)).astype(F))


def _check_scale(amax, g):
    amax, g = amax.astype(F), g.astype(F)
    exact = _scale_byte(((amax / F(6.0)).astype(F) / g).astype(F))
    c = (F(1.0) / (F(6.0) * g).astype(F)).astype(F)
    hi = _scale_byte((amax * (c * HI).astype(F)).astype(F))
    lo = _scale_byte((amax * (c * LO).astype(F)).astype(F))
    agree = hi == lo
    assert np.array_equal(hi[agree], exact[agree])
    return 1.0 - agree.mean()


def test_scale_of_random_blocks():
    rng = np.random.default_rng(3)
    g = np.exp(rng.uniform(-20, 20, 1_000_000)).astype(F)
    amax = (g * 6.0 * np.exp(rng.uniform(-8, 7, g.size))).astype(F)
    assert _check_scale(amax, g) < 1e-3
    amax[::5] = 0.0
    _check_scale(amax, g)


def test_scale_next_to_every_boundary():
    rng = np.random.default_rng(4)
    values = oc.e4m3_to_f32(np.arange(127, dtype=np.uint8))
    middles = np.concatenate([(values[1:] + values[:-1]) / 2, [448.0, 464.0]]).astype(F)
    g = np.exp(rng.uniform(-15, 15, 4000)).astype(F)
    for m in middles:
        at = (g.astype(np.float64) * 6.0 * float(m)).astype(F).view(np.uint32).astype(np.int64)
        for delta in range(-6, 7):
            _check_scale((at + delta).astype(np.uint32).view(F), g)


@pytest.mark.parametrize("ulp", [-1, 0, 1])
def test_codes_with_a_reciprocal_one_ulp_off(ulp):
    rng = np.random.default_rng(5)
    t = np.exp(rng.uniform(-8, 3, 100_000)).astype(F)
    y = ((F(1.0) / t).astype(F).view(np.int32) + ulp).view(F)

    def codes(q):
        return oc.f32_to_e2m1(np.clip(q, F(-6.0), F(6.0)))

    for b in (0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0):
        bits = (t * F(b)).astype(F).view(np.uint32).astype(np.int64)
        for delta in range(-6, 7):
            x = (bits + delta).astype(np.uint32).view(F)
            hi, lo = codes((x * (y * HI).astype(F)).astype(F)), codes((x * (y * LO).astype(F)).astype(F))
            agree = hi == lo
            assert np.array_equal(hi[agree], codes((x / t).astype(F))[agree])
