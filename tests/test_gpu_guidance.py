"""Guidance divergence: both kernels at the edges of their tiles, and small windows' time."""

import ctypes as C

import numpy as np
import pytest
import torch

from gradient_domain_b200 import _lib
from oracle import operators as ops

pytestmark = pytest.mark.gpu


def _launch(div, kind, target, window, edges, source=None, select=None, weights=None):
    h, w, c = target.shape
    r0, c0, hh, ww = window
    ptr = lambda t: _lib.ptr(t) if t is not None else None
    d = _lib.FieldDesc(kind, h, w, c, c - 1, edges, ptr(target), ptr(source), ptr(select),
                       ptr(weights), 0.0, 0.0, 0.0)
    _lib.check(_lib.lib().gd_guidance_divergence(_lib.ptr(div), C.byref(d), r0, c0, hh, ww,
                                                 _lib.stream_handle()), "gd_guidance_divergence")


# narrow windows on 4, 8, 16 and 32 lanes, one row and one column, remainders of 31 columns
# and of 8, 17, 35 and 71 rows; two that are walked (8250 and 8214 walks) beside one that is not
@pytest.mark.parametrize("shape", [(1, 1), (1, 40), (40, 1), (2, 2), (71, 3), (72, 3), (73, 4),
                                   (35, 7), (36, 8), (17, 15), (18, 16), (8, 31), (9, 32),
                                   (7, 33), (16, 62), (25, 63), (2000, 1000), (65712, 20),
                                   (1984, 999)])
def test_windows_match_the_oracle(shape):
    h, w = shape
    rng = np.random.default_rng(h * 100 + w)
    whole = (0, 0, h, w)
    target, source = rng.random((h, w, 2)), rng.random((h, w, 2))
    select, weights = rng.random((h, w)) < 0.5, rng.random((h, w))
    dev = [torch.as_tensor(a).cuda() for a in (target, source, select.astype(np.uint8), weights)]
    gx, gy = ops.gradient(target[..., 1])
    sx, sy = ops.gradient(source[..., 1])
    fields = {_lib.GD_FIELD_WEIGHTED: (gx * weights, gy * weights),
              _lib.GD_FIELD_IMPORT: (np.where(select, sx, gx), np.where(select, sy, gy))}
    for kind, (fx, fy) in fields.items():
        want = ops.divergence(fx, fy)
        div = torch.full((h, w), np.nan, dtype=torch.float64, device="cuda")
        _launch(div, kind, dev[0], whole, 1, dev[1], dev[2], dev[3])
        assert np.array_equal(div.cpu().numpy(), want), kind
        if min(h, w) > 2:  # a window writes zeros on its ring
            want[0], want[-1], want[:, 0], want[:, -1] = 0, 0, 0, 0
            _launch(div, kind, dev[0], whole, 0, dev[1], dev[2], dev[3])
            assert np.array_equal(div.cpu().numpy(), want), kind


@pytest.mark.parametrize("shape", [(64, 64), (300, 200), (4000, 6)])
def test_small_windows_take_one_short_launch(shape):
    """A small window's launch is a chain of latencies, not longer than 1.4 times that of the
    masked right-hand side of the same cells (1.7 times and more when a warp walked eight
    rows; event times of single launches)."""
    h, w = shape
    target = torch.rand((h, w, 1), dtype=torch.float64, device="cuda")
    weights, div, rhs = (torch.rand((h, w), dtype=torch.float64, device="cuda") for _ in range(3))
    unknown = torch.ones((h, w), dtype=torch.uint8, device="cuda")

    def guidance():
        _launch(div, _lib.GD_FIELD_WEIGHTED, target, (0, 0, h, w), 1, weights=weights)

    def masked():
        _lib.check(_lib.lib().gd_masked_rhs(_lib.ptr(rhs), _lib.ptr(div), _lib.ptr(weights),
                                            _lib.ptr(unknown), h, w, 1.0, _lib.stream_handle()),
                   "gd_masked_rhs")

    def device_us(run):
        run()
        best = np.inf
        for _ in range(30):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda._sleep(1_000_000)  # the launch is queued before the device reaches it
            a.record()
            run()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 1e3)
        return best

    assert device_us(guidance) <= 1.4 * device_us(masked)
