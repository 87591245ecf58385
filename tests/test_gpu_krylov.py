"""Krylov kernels at the edges of their tiles: residual against plain torch, batch against alone."""

import numpy as np
import pytest
import torch

from gradient_domain_b200.plan import Instance, PoissonPlan, SolveParams

pytestmark = pytest.mark.gpu

# sides around the 128-column strips and the 32 / 64 / 128-row tiles, one grid with the tall tiles
SHAPES = [(33, 127), (64, 128), (65, 129), (31, 641), (1, 300), (1025, 513), (3600, 4100)]


def _true_residual(x, f, boundary, on):
    """||f - A x|| / ||f|| with A the positive five-point operator of the boundary type."""
    p = torch.nn.functional.pad(x, (1, 1, 1, 1))
    nb = p[2:, 1:-1] + p[:-2, 1:-1] + p[1:-1, 2:] + p[1:-1, :-2]
    d = torch.full_like(x, 4.0)
    if boundary == "neumann":
        d[0] -= 1
        d[-1] -= 1
        d[:, 0] -= 1
        d[:, -1] -= 1
    r = f - (d * x - nb)
    if on is not None:
        r = torch.where(on, r, torch.zeros_like(r))
    return float(r.norm() / f.norm())


@pytest.mark.parametrize("boundary", ["neumann", "dirichlet", "masked"])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_krylov_tiles(boundary, precision):
    shapes = SHAPES if precision == "mixed" else SHAPES[:-1]
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    insts, fs, ons = [], [], []
    for h, w in shapes:
        f = torch.randn((h, w), generator=g, dtype=torch.float64, device="cuda")
        on = None
        if boundary == "neumann":
            f -= f.mean()
        if boundary == "masked":
            on = torch.rand((h, w), generator=g, device="cuda") < 0.8
            f = torch.where(on, f, torch.zeros_like(f))
        insts.append(Instance(h, w, boundary, boundary == "neumann"))
        fs.append(f)
        ons.append(on)
    params = SolveParams(precision=precision, tolerance=1e-8, zero_start=True)

    def solve(ids):
        plan = PoissonPlan([insts[i] for i in ids], params)
        for k, i in enumerate(ids):
            if ons[i] is not None:
                plan.set_mask(k, ons[i].to(torch.uint8))
        xs = [torch.full_like(fs[i], np.nan) for i in ids]
        res = plan.solve([fs[i] for i in ids], xs)
        assert all(r.converged for r in res), res
        return xs

    together = solve(range(len(shapes)))
    for i in range(len(shapes)):
        # the solver's own residual is the true one; 2x for the order of the norm's sum
        assert _true_residual(together[i], fs[i], boundary, ons[i]) <= 2e-8, shapes[i]
    for i in (0, 2, 5):
        assert torch.equal(solve([i])[0], together[i]), shapes[i]


@pytest.mark.parametrize("shape", [(64, 2), (64, 3), (256, 2), (256, 3)])
def test_last_columns_square_in_fp64(shape):
    """The columns of a width that is no multiple of four square their residual in FP64.

    A smooth f of 1e-23 has search directions far above it, so p.Ap is a normal number of
    the iteration, but every square of r is below FP32's smallest, 1.4e-45.  Summed in FP32
    r.r would be zero and ask for a refresh at once; in FP64 the residual stays above
    reliable_delta and the tolerance, and the only refresh is the one that ends the solve."""
    h, w = shape
    y = torch.arange(h, dtype=torch.float64, device="cuda")[:, None]
    f = 1e-23 * torch.cos(np.pi * (y + 0.5) / h).expand(h, w).contiguous()
    params = SolveParams(tolerance=1e-4, reliable_delta=1e-8, max_iterations=2, zero_start=True)
    plan = PoissonPlan([Instance(h, w, "neumann", True)], params)
    for _ in range(2):  # direct launches, then the graph
        res = plan.solve([f], [torch.empty_like(f)], scale=-1.0)[0]
        assert res.iterations >= 1 and res.refreshes == 1, res
