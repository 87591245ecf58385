"""Tone mapping: every way the percentile selection can end, both saturation paths, window edges."""

import numpy as np
import pytest

import gradient_domain_b200 as gd
from oracle import hdr

pytestmark = pytest.mark.gpu


def _radiance(kind, shape, rng):
    if kind == "noise":
        return np.exp(rng.standard_normal(shape + (3,)))
    if kind == "zeros":
        r = np.exp(rng.standard_normal(shape + (3,)))
        r[..., 0][rng.random(shape) < 0.3] = 0.0
        return r
    # values crowd into one slice of an octave: nothing (one value), a slice of 2^-12
    # and one of 2^-24 hold more of them than the candidate list
    spread = {"flat": 0.0, "crowded": 1e-5, "packed": 1e-9}[kind]
    return 0.7 * (1.0 + spread * rng.random(shape + (3,)))


@pytest.mark.parametrize("kind", ["noise", "zeros", "flat", "crowded", "packed"])
@pytest.mark.parametrize("shape,levels,saturation", [((160, 181), 8, 0.5), ((161, 160), 1, 0.7),
                                                     ((17, 33), 8, 0.5)])
def test_tone_map_matches_the_oracle(kind, shape, levels, saturation):
    rad = _radiance(kind, shape, np.random.default_rng(7))
    config = gd.ToneMapConfig(levels=levels, saturation=saturation)
    out, factor = gd.tone_map(rad, config)
    ref, ref_factor = hdr.tone_map(rad, hdr.ToneMapConfig(levels=levels, saturation=saturation))
    # logarithm, power and exponential differ by a few ulp; the transform solve spreads
    # them over the image
    np.testing.assert_allclose(factor, ref_factor, rtol=1e-10, atol=0)
    np.testing.assert_allclose(out, ref, rtol=1e-9, atol=1e-12)
