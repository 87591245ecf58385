"""Mask set-up and the tiles it lets the kernels skip."""

import pytest
import torch

from gradient_domain_b200.plan import Instance, PoissonPlan, SolveParams

pytestmark = pytest.mark.gpu


def _masks(h, w, g):
    y = torch.arange(h, device="cuda")[:, None]
    x = torch.arange(w, device="cuda")[None, :]
    disc = (y - h * 0.6) ** 2 + (x - w * 0.3) ** 2 < (0.22 * min(h, w)) ** 2
    corner = (y < 3) & (x >= w - 5)
    two = ((y - 7).abs() < 5) & ((x - 9).abs() < 6) | (y >= h - 2) & (x < w // 2)
    holes = (torch.rand((h, w), generator=g, device="cuda") < 0.97) & (y > h // 2)
    single = (y == h // 3) & (x == w // 2)
    return {"disc": disc, "corner": corner, "two": two, "holes": holes, "single": single}


def _residual(x, f, on):
    p = torch.nn.functional.pad(x, (1, 1, 1, 1))
    r = f - (4 * x - (p[2:, 1:-1] + p[:-2, 1:-1] + p[1:-1, 2:] + p[1:-1, :-2]))
    return float(torch.where(on, r, torch.zeros_like(r)).norm() / f.norm())


# grids with strips, large and small tiles and a bottom, one with every level above 6,
# one that is a bottom alone
@pytest.mark.parametrize("shape", [(700, 1100), (301, 97), (60, 60), (5, 900), (2050, 2100)])
@pytest.mark.parametrize("precision,zero_start", [("mixed", True), ("fp64", True),
                                                  ("mixed", False)])
def test_masks_one_after_another_on_one_plan(shape, precision, zero_start):
    """A plan that had another mask, another solution and NaN in its buffers before gives
    bitwise what a fresh plan gives, zeros outside the mask and a true residual."""
    h, w = shape
    g = torch.Generator(device="cuda")
    g.manual_seed(h + w)
    params = SolveParams(precision=precision, tolerance=1e-9, zero_start=zero_start)
    insts = [Instance(h, w, "masked"), Instance(h, w, "dirichlet")]
    used = PoissonPlan(insts, params)
    rect = torch.randn(shape, generator=g, dtype=torch.float64, device="cuda")
    masks = _masks(h, w, g)
    # a solve that breaks down leaves NaN behind
    used.set_mask(0, torch.ones(shape, dtype=torch.uint8, device="cuda"))
    bad = [torch.full_like(rect, float("nan")), rect]
    used.solve(bad, [torch.zeros_like(rect) for _ in bad])
    for name, on in masks.items():
        f = torch.where(on, torch.randn(shape, generator=g, dtype=torch.float64, device="cuda"),
                        torch.zeros_like(rect))
        start = torch.full_like(f, 3.0) if not zero_start else torch.full_like(f, float("nan"))
        got = []
        for plan in (used, PoissonPlan(insts, params)):
            plan.set_mask(0, on.to(torch.uint8))
            x = [start.clone(), torch.zeros_like(rect)]
            res = plan.solve([f, rect], x)
            assert all(r.converged for r in res), (name, res)
            got.append(x)
        assert torch.equal(got[0][0], got[1][0]), name
        assert torch.equal(got[0][1], got[1][1]), name
        x = got[0][0]
        assert not x[~on].any(), name
        # the reported residual is the true one; 2x for the order of the sums
        assert _residual(x, f, on) <= 2e-9, name


# strips and tiles with parts that hold no unknown, and a grid that is a bottom alone
@pytest.mark.parametrize("shape", [(700, 1100), (301, 97), (60, 60)])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_residual_outside_the_mask_is_not_read(shape, precision):
    """What apply_vcycle's residual holds where there is no unknown changes neither its
    result nor a later solve on the plan."""
    h, w = shape
    g = torch.Generator(device="cuda")
    g.manual_seed(h * w)
    params = SolveParams(precision=precision, tolerance=1e-9, zero_start=True)
    for name, on in _masks(h, w, g).items():
        f = torch.where(on, torch.randn(shape, generator=g, dtype=torch.float64, device="cuda"),
                        torch.zeros(shape, dtype=torch.float64, device="cuda"))
        clean, dirty = [PoissonPlan([Instance(h, w, "masked")], params) for _ in range(2)]
        for plan in (clean, dirty):
            plan.set_mask(0, on.to(torch.uint8))
        z = clean.apply_vcycle(0, f)
        assert not z[~on].any(), name
        for junk in (float("nan"), float("inf"), -1e300):
            r = torch.where(on, f, torch.full_like(f, junk))
            assert torch.equal(dirty.apply_vcycle(0, r), z), (name, junk)
            x = [torch.empty_like(f) for _ in range(2)]
            for plan, out in zip((clean, dirty), x):
                assert plan.solve([f], [out])[0].converged, (name, junk)
            assert torch.equal(x[0], x[1]), (name, junk)


@pytest.mark.parametrize("shape", [(700, 1100), (301, 297)])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_persistent_coarse_launch_skips_the_same_tiles(shape, precision):
    """The persistent coarse launch leaves out tiles without unknowns as the level launches
    do: the same bits, on direct launches and in the solve graph, beside a rectangle."""
    h, w = shape
    g = torch.Generator(device="cuda")
    g.manual_seed(h + 2 * w)
    insts = [Instance(h, w, "masked"), Instance(h, w, "neumann", True)]
    plans = [PoissonPlan(insts, SolveParams(precision=precision, tolerance=1e-9, zero_start=True,
                                            persistent_coarse=p)) for p in (False, True)]
    for name, on in _masks(h, w, g).items():
        f = [torch.randn(shape, generator=g, dtype=torch.float64, device="cuda") for _ in insts]
        f[0] = torch.where(on, f[0], torch.zeros_like(f[0]))
        for _ in range(2):
            got = []
            for plan in plans:
                plan.set_mask(0, on.to(torch.uint8))
                x = [torch.full_like(q, float("nan")) for q in f]
                assert all(r.converged for r in plan.solve(f, x, scale=-1.0)), name
                got.append(x)
            assert all(torch.equal(p, q) for p, q in zip(*got)), name
