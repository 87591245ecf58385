"""Tone mapping: every way the percentile selection can end, both saturation paths, window edges."""

import numpy as np
import pytest
import torch

import gradient_domain_b200 as gd
from gradient_domain_b200 import _lib
from gradient_domain_b200 import hdr as hdr_gpu
from oracle import hdr

pytestmark = pytest.mark.gpu


def _radiance(kind, shape, rng):
    if kind == "noise":
        return np.exp(rng.standard_normal(shape + (3,)))
    if kind == "zeros":
        r = np.exp(rng.standard_normal(shape + (3,)))
        r[..., 0][rng.random(shape) < 0.3] = 0.0
        return r
    # values crowd into one slice of an octave: nothing (one value), slices of 2^-12, 2^-24,
    # 2^-36 and 2^-48 hold more of them than the candidate list
    spread = {"flat": 0.0, "crowded": 1e-5, "packed": 1e-9, "tight": 1e-12, "ulps": 4e-15}[kind]
    return 0.7 * (1.0 + spread * rng.random(shape + (3,)))


@pytest.mark.parametrize("kind", ["noise", "zeros", "flat", "crowded", "packed", "tight", "ulps"])
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


@pytest.mark.parametrize("shape,most", [((1440, 2160), 4.0), ((128, 160), 2.5)])
def test_percentile_time_does_not_depend_on_the_values(shape, most):
    """A nearly flat image, whose values crowd within 2^-24 of the percentile, is selected by
    the whole grid too: at most `most` times as long as noise (four histograms more on top of
    two and a collection; one CTA alone took 70 times as long, and three times for the 61440
    values of the small image when they all fitted its list)."""
    h, w = shape
    lib = _lib.lib()
    g = torch.Generator(device="cuda")
    g.manual_seed(2)

    def rand(*shape):
        return torch.rand(*shape, generator=g, dtype=torch.float64, device="cuda")

    def compose_ms(spread):
        rad, lum = rand(h, w, 3) + 0.5, rand(h, w) + 0.5
        comp = rand(h, w) * spread
        image, out = torch.empty_like(rad), torch.empty_like(rad)
        scratch = hdr_gpu._scratch(rad.device)
        best = np.inf
        for _ in range(4):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            # saturation 0: the image is exp(comp - max comp) in all channels
            _lib.check(lib.gd_tm_compose(_lib.ptr(out), _lib.ptr(image), _lib.ptr(rad),
                                         _lib.ptr(lum), _lib.ptr(comp), h, w, 0.0, 99.5,
                                         _lib.ptr(scratch), _lib.stream_handle()), "compose")
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        peak = torch.from_numpy(np.percentile(image.cpu().numpy(), [99.5])).cuda()
        assert torch.equal(out, (image / peak).clamp(0, 1))
        return best

    assert compose_ms(1e-13) <= most * compose_ms(1.0)


@pytest.mark.parametrize("shape", [(2000, 17), (17, 2000), (900, 33), (600, 65), (400, 129),
                                   (300, 257)])
def test_attenuation_of_narrow_images_matches_the_oracle(shape):
    """Widths around the powers of two that a CTA's columns take."""
    logl = np.random.default_rng(sum(shape)).standard_normal(shape)
    want = hdr.attenuation_field(logl, hdr.ToneMapConfig())
    got = gd.attenuation_field(logl, gd.ToneMapConfig())
    # a logarithm, a power and the mean's order of sums differ by a few ulp
    np.testing.assert_allclose(got, want, rtol=1e-12, atol=0)


def test_attenuation_time_of_a_narrow_image():
    """20000 x 20 has a seventh of the cells of 1440 x 2000: its attenuation takes at most half
    as long (as long, when every row took a CTA of 256 columns)."""
    def device_us(h, w):
        logl = torch.randn((h, w), dtype=torch.float64, device="cuda")
        scratch = hdr_gpu._scratch(logl.device)
        best = np.inf
        for _ in range(10):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda._sleep(3_000_000)  # the launches are queued before the device reaches them
            a.record()
            hdr_gpu._attenuation_dev(logl, gd.ToneMapConfig(levels=2), scratch)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 1e3)
        return best

    assert device_us(20000, 20) <= 0.5 * device_us(1440, 2000)
