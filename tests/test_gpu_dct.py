"""DCT Neumann solver: every radix, the power-of-two kernels, odd grids, unaligned rows."""

import numpy as np
import pytest
import torch
from scipy import fft

from gradient_domain_b200.solvers import DctPlan
from oracle import solvers

pytestmark = pytest.mark.gpu

# every in-register radix as a length of its own, two and three passes, a prime
# above 13 alone and next to other factors, and both directions of the
# power-of-two kernels (64 .. 8192) beside each kind of the other axis
SHAPES = [(2, 3), (4, 5), (6, 7), (8, 9), (10, 11), (12, 13), (14, 15), (16, 64), (17, 256),
          (64, 128), (256, 64), (33, 128), (128, 70), (90, 143), (19 * 4, 23 * 17), (1080, 480), (512, 1024), (1024, 513), (2048, 6),
          (7, 2048), (4096, 5), (3, 4096), (8192, 3), (2, 8192)]


@pytest.mark.parametrize("shape", SHAPES)
def test_dct_solve_matches_the_oracle(shape):
    h, w = shape
    b = np.random.default_rng(h * 10000 + w).standard_normal(shape)
    ref = solvers.solve_neumann(b)
    plan = DctPlan(h, w)
    bd = torch.as_tensor(b).cuda()
    u = plan.solve(bd, torch.full_like(bd, np.nan))
    # FP64 transforms: a few eps per pass, four transforms of at most 13 octaves; the
    # smallest eigenvalue, about (pi / n)^2 of terms near 4, amplifies only modes that
    # the right-hand side's noise gives no more than 1 / sqrt(h w) of its norm
    assert np.linalg.norm(u.cpu().numpy() - ref) <= 1e-12 * np.linalg.norm(ref)
    # an odd pitch and an 8-byte aligned first row, solved in place: the same bits
    buf = torch.zeros((h, w + 3), dtype=torch.float64, device="cuda")
    view = buf[:, 1:w + 1]
    view.copy_(bd)
    plan.solve(view, view)
    assert torch.equal(view, u)
    assert not buf[:, 0].any() and not buf[:, w + 1:].any()


@pytest.mark.parametrize("shape", [(720, 1280), (1000, 1000), (375, 1125), (1024, 1024)])
def test_transform_error_in_the_smoothest_modes(shape):
    """A right-hand side whose solution is white noise is strongest in its highest modes, and
    the transform's rounding of those is what its smoothest modes carry, divided by their
    small eigenvalues.  That error, times the eigenvalue, against 80-bit transforms with the
    solver's own eigenvalues: at most six passes (three a direction) of six roundings (four
    additions, a product by a twiddle of the table) and four of the DCT's own twiddles, each
    of rms eps / sqrt(12) - 1.27 is measured, 1.9 to 2.2 with twiddles by repeated products."""
    h, w = shape
    wide = np.longdouble
    eig = ((2 * np.cos(np.pi * np.arange(h) / h))[:, None]
           + (2 * np.cos(np.pi * np.arange(w) / w))[None] - 4).astype(wide)
    g = np.random.default_rng(h + w).standard_normal(shape).astype(wide)
    g[0, 0] = 0
    b = fft.idctn(g * eig, type=2, norm="ortho").astype(np.float64)
    ref = fft.dctn(b.astype(wide), type=2, norm="ortho")
    ref[0, 0] = 0
    bd = torch.as_tensor(b).cuda()
    u = DctPlan(h, w).solve(bd, torch.empty_like(bd)).cpu().numpy()
    err = fft.dctn(u.astype(wide), type=2, norm="ortho") * eig - ref
    low = err[:h // 16, :w // 16].ravel()[1:].astype(np.float64)
    eps = np.finfo(np.float64).eps
    bound = eps / np.sqrt(12) * np.sqrt(6 * 6 + 4)
    assert np.sqrt(np.mean(low ** 2)) <= bound * np.sqrt(np.mean(b ** 2))


def _device_us(run, passes=20, rounds=10):
    """Shortest device time of one of `passes` back-to-back calls, in microseconds."""
    run()
    best = np.inf
    for _ in range(rounds):
        start, stop = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda._sleep(2_000_000)  # the calls are queued before the device reaches them
        start.record()
        for _ in range(passes):
            run()
        stop.record()
        stop.synchronize()
        best = min(best, start.elapsed_time(stop) * 1e3 / passes)
    return best


def test_small_powers_of_two_are_not_slower_than_larger_ones():
    """Launches of few short lines are as long as one thread's chain: a side of 64 to 256
    must not take longer than one of 512 (25 to 28 us against 25 by the run-time passes)."""
    def solve_us(n):
        plan = DctPlan(n, n)
        b = torch.randn((n, n), dtype=torch.float64, device="cuda")
        u = torch.empty_like(b)
        return _device_us(lambda: plan.solve(b, u))

    larger = solve_us(512)
    for n in (64, 128, 256):
        assert solve_us(n) <= 0.95 * larger, n
