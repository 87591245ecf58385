"""Fused reference V-cycle against the one-kernel-per-operation form, bit for bit."""

import numpy as np
import pytest
import torch

from gradient_domain_b200.multigrid import MultigridOptions, RefWorkspace
from oracle import operators

pytestmark = pytest.mark.gpu

# (coarsest grids of one warp, of one CTA with and without a cell per thread, beyond the
# small kernel's shared memory; even, odd and narrow sides)
SHAPES = [(5, 5), (7, 7), (8, 9), (33, 47), (64, 64), (200, 131), (9, 400), (511, 300), (8, 700)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("pre,post", [(2, 2), (1, 0), (0, 3), (5, 2)])
@pytest.mark.parametrize("spacing,coarsest", [(1.0, 8), (0.3, 40)])
def test_fused_cycle_is_the_cycle_by_operation(shape, pre, post, spacing, coarsest):
    g = torch.Generator(device="cuda")
    g.manual_seed(shape[0] * 1000 + shape[1])
    b = torch.randn(shape, generator=g, dtype=torch.float64, device="cuda")
    u0 = torch.randn(shape, generator=g, dtype=torch.float64, device="cuda")
    options = MultigridOptions(pre_smoothing=pre, post_smoothing=post, coarsest_size=coarsest)
    ws = RefWorkspace(shape, coarsest, b.device)
    got, want = u0.clone(), u0.clone()
    for _ in range(2):
        ws.vcycle(got, b, spacing, options)
        ws.vcycle(want, b, spacing, options, by_operation=True)
    assert torch.equal(got, want)
    r = b.cpu().numpy() - operators.laplacian(got.cpu().numpy(), spacing)
    # sums of at most 2^18 squares in another order: far below 1e-12
    assert abs(ws.residual_norm(got, b, spacing) - np.linalg.norm(r)) <= 1e-12 * np.linalg.norm(r)
