"""DCT Neumann solver: every radix, the power-of-two kernels, odd grids, unaligned rows."""

import numpy as np
import pytest
import torch

from gradient_domain_b200.solvers import DctPlan
from oracle import solvers

pytestmark = pytest.mark.gpu

# every in-register radix as a length of its own, two and three passes, a prime
# above 13 alone and next to other factors, and both directions of the
# power-of-two kernels (512 .. 8192) beside each kind of the other axis
SHAPES = [(2, 3), (4, 5), (6, 7), (8, 9), (10, 11), (12, 13), (14, 15), (16, 64), (17, 256),
          (90, 143), (19 * 4, 23 * 17), (1080, 480), (512, 1024), (1024, 513), (2048, 6),
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
