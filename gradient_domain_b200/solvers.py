"""Linear solvers for the Poisson system, on the GPU.

Drop-in for gradient-domain/src/gradient_domain/solvers.py: the same
``SolverReport`` (:50-75), ``SOLVERS`` registry (:163-168) with the same
signature ``f(b, spacing, tolerance, max_iterations) -> (u, iterations,
converged)``, ``solve_system`` (:171-221) and ``solve_neumann`` (:224-262).
Every method runs on the device; there is no CPU path.

``mgcg``
    The B200 solver: batched cell-centred MGPCG, FP32 V-cycle with FP64
    residual refresh, solution accumulator and scalars.  It converges to the
    same solution as the reference's ``mgcg`` (same system, same tolerance on
    the true residual) in fewer iterations, because its hierarchy coarsens
    every grid size exactly.
``multigrid``
    The reference's vertex-centred V-cycle, reproduced operation by operation
    in FP64 kernels; same cycle counts as the reference.
``cg``
    The reference's Jacobi-PCG loop on the device (FP64).
``direct``
    The reference factorises the operator with SuperLU.  Here it is the FP64
    B200 MGPCG driven to a relative residual of 1e-13, which reproduces the
    factorised solution to rounding level on the grids this path serves.
``mgcg_fp64``
    The B200 kernels with every array in FP64 (the precision baseline).
``mgcg_port``
    A literal GPU port of the reference's ``mgcg``: its vertex-centred V-cycle
    as preconditioner, one kernel per operation, scalars read back to the host
    every iteration (the port-equivalent baseline).
"""

from __future__ import annotations

import ctypes as C
import threading
import time
from collections import OrderedDict
from dataclasses import dataclass, replace

import numpy as np
import torch

from . import _lib
from ._host import download, upload
from .autotune import resolve
from .multigrid import MultigridOptions, RefWorkspace
from .plan import Instance, PoissonPlan, SolveParams, cached_plan

__all__ = ["SolverReport", "SOLVERS", "solve_system", "solve_neumann", "solve_neumann_batch",
           "solve_neumann_batch_async", "NeumannBatchFuture"]


@dataclass
class SolverReport:
    """Cost and accuracy of one solve (solvers.py:50-75), plus the exit status."""

    method: str
    iterations: int
    relative_residual: float
    seconds: float
    converged: bool
    status: str = "converged"

    def __str__(self) -> str:
        return (f"{self.method}: {self.iterations} iterations, "
                f"residual {self.relative_residual:.2e}, {self.seconds * 1e3:.0f} ms")


def _dev_array(a, dev: torch.device) -> torch.Tensor:
    return upload(a, dev, np.float64)


def _plan_solve(b: np.ndarray, spacing: float, boundary: str, params: SolveParams,
                zero_mean: bool = False):
    dev = _lib.device()
    m, n = b.shape
    plan = cached_plan((Instance(m, n, boundary, zero_mean),), replace(params, zero_start=True))
    f = _dev_array(b, dev)
    x = torch.empty_like(f)
    (res,) = plan.solve([f], [x], scale=-(spacing * spacing))
    return download(x), res


def _solve_mgcg(b, spacing, tolerance, max_iterations):
    params = SolveParams(tolerance=tolerance, max_iterations=max_iterations)
    u, res = _plan_solve(b, spacing, "dirichlet", params)
    return u, res.iterations, res.converged


def _solve_mgcg_fp64(b, spacing, tolerance, max_iterations):
    params = SolveParams(precision="fp64", tolerance=tolerance, max_iterations=max_iterations)
    u, res = _plan_solve(b, spacing, "dirichlet", params)
    return u, res.iterations, res.converged


def _solve_direct(b, spacing, tolerance, max_iterations):
    params = SolveParams(precision="fp64", tolerance=1e-13, max_iterations=max(max_iterations,
                                                                               500))
    u, res = _plan_solve(b, spacing, "dirichlet", params)
    return u, 0, True


def _ref_pcg_dev(b_d: torch.Tensor, spacing, tolerance, max_iterations, precondition_kind: str):
    """The reference's PCG loop (solvers.py:99-118, :142-160) on a device right-hand
    side; returns the device solution, the iteration count and convergence."""
    dev = b_d.device
    ws = RefWorkspace(tuple(b_d.shape), 8, dev)
    opts = MultigridOptions(pre_smoothing=1, post_smoothing=1)
    zeros = torch.zeros_like(b_d)
    diag = 4.0 / (spacing * spacing)

    def precondition(r: torch.Tensor) -> torch.Tensor:
        if precondition_kind == "jacobi":
            z = r.clone()
            ws.axpby(z, r, 1.0 / diag, 0.0)
            return z
        z = torch.zeros_like(r)
        neg = torch.zeros_like(r)
        ws.axpby(neg, r, -1.0, 0.0)
        ws.vcycle(z, neg, spacing, opts, by_operation=True)
        return z

    rhs = torch.zeros_like(b_d)
    ws.axpby(rhs, b_d, -1.0, 0.0)
    u = torch.zeros_like(b_d)
    r = rhs.clone()
    p = precondition(r)
    rz = ws.dot(r, p)
    target = tolerance * float(np.sqrt(ws.dot(rhs, rhs)))
    q = torch.empty_like(b_d)
    for it in range(1, max_iterations + 1):
        ws.residual(q, p, zeros, spacing)          # q = 0 - laplacian(p) = -L p
        alpha = rz / ws.dot(p, q)
        ws.axpby(u, p, alpha, 1.0)
        ws.axpby(r, q, -alpha, 1.0)
        if float(np.sqrt(ws.dot(r, r))) <= target:
            return u, it, True
        z = precondition(r)
        rz_new = ws.dot(r, z)
        ws.axpby(p, z, 1.0, rz_new / rz)
        rz = rz_new
    return u, max_iterations, False


def _ref_pcg(b, spacing, tolerance, max_iterations, precondition_kind: str):
    """The reference's PCG loop with device arrays, from and to NumPy."""
    u, it, ok = _ref_pcg_dev(_dev_array(b, _lib.device()), spacing, tolerance, max_iterations,
                             precondition_kind)
    return download(u), it, ok


def _solve_cg(b, spacing, tolerance, max_iterations):
    return _ref_pcg(b, spacing, tolerance, max_iterations, "jacobi")


def _solve_mgcg_port(b, spacing, tolerance, max_iterations):
    return _ref_pcg(b, spacing, tolerance, max_iterations, "vcycle")


def _solve_multigrid(b, spacing, tolerance, max_iterations):
    """Stand-alone reference V-cycles (solvers.py:121-131)."""
    dev = _lib.device()
    opts = MultigridOptions(max_cycles=max_iterations, tolerance=tolerance)
    b_d = _dev_array(b, dev)
    ws = RefWorkspace(tuple(b_d.shape), opts.coarsest_size, dev)
    u = torch.zeros_like(b_d)
    scale = float(np.sqrt(ws.dot(b_d, b_d))) or 1.0
    for cycle in range(1, max_iterations + 1):
        ws.vcycle(u, b_d, spacing, opts)
        if ws.residual_norm(u, b_d, spacing) / scale < tolerance:
            return download(u), cycle, True
    return download(u), max_iterations, False


SOLVERS = {
    "direct": _solve_direct,
    "cg": _solve_cg,
    "multigrid": _solve_multigrid,
    "mgcg": _solve_mgcg,
    "mgcg_fp64": _solve_mgcg_fp64,
    "mgcg_port": _solve_mgcg_port,
}


def relative_residual(u: np.ndarray, b: np.ndarray, spacing: float) -> float:
    """||b - laplacian(u)|| / ||b|| evaluated on the device (solvers.py:78-82)."""
    dev = _lib.device()
    b_d, u_d = _dev_array(b, dev), _dev_array(u, dev)
    ws = RefWorkspace(tuple(b_d.shape), 8, dev)
    scale = float(np.sqrt(ws.dot(b_d, b_d)))
    if scale == 0.0:
        return 0.0
    return ws.residual_norm(u_d, b_d, spacing) / scale


def solve_system(b, method: str = "mgcg", spacing: float = 1.0, tolerance: float = 1e-8,
                 max_iterations: int = 2000) -> tuple[np.ndarray, SolverReport]:
    """Solve ``laplacian(u) = b`` with zero Dirichlet values (solvers.py:171-221).

    Raises
    ------
    KeyError
        If ``method`` is not a key of :data:`SOLVERS`.
    """
    if method not in SOLVERS:
        raise KeyError(f"unknown solver {method!r}; choose from {sorted(SOLVERS)}")
    b = np.asarray(b, dtype=float)
    if not np.any(b):
        return np.zeros_like(b), SolverReport(method, 0, 0.0, 0.0, True)
    started = time.perf_counter()
    u, iterations, converged = SOLVERS[method](b, spacing, tolerance, max_iterations)
    elapsed = time.perf_counter() - started
    return u, SolverReport(method, iterations, relative_residual(u, b, spacing), elapsed,
                           converged, "converged" if converged else "max_iterations")


NEUMANN_EXACT_TOLERANCE = 1e-14


DCT_MAX_SIDE = 8192  # longest line a DCT pass holds in shared memory


class DctPlan:
    """DCT Neumann solver for one grid shape (gd_dct_* of the C ABI): the library's own
    FFT kernels, three passes over the grid, sides of 2 to 8192 cells.

    The coefficients between the passes live in the plan's workspace, so solves of one plan
    run one after another: a solve on another stream than the last one's waits for that one
    (threads may share a plan; each enqueues its solve whole).  Under graph capture, and for
    replays of such a graph, the order is the caller's."""

    def __init__(self, h: int, w: int):
        self.shape = (h, w)
        self.device = _lib.device()
        self._lock = threading.Lock()
        self._done = torch.cuda.Event()  # after the latest solve, and the stream it ran on
        self._ran_on: int | None = None
        lib = _lib.lib()
        handle = C.c_void_p()
        _lib.check(lib.gd_dct_plan_create(h, w, C.byref(handle)), "gd_dct_plan_create")
        self._handle = handle
        nbytes = int(lib.gd_dct_workspace_bytes(handle))
        self.workspace = torch.empty(nbytes, dtype=torch.uint8, device=self.device)
        _lib.check(lib.gd_dct_plan_bind(handle, _lib.ptr(self.workspace), nbytes,
                                        _lib.stream_handle()), "gd_dct_plan_bind")

    def solve(self, b: torch.Tensor, u: torch.Tensor) -> torch.Tensor:
        """u = zero-mean solution of laplacian(u) = b (FP64 device tensors, one row pitch)."""
        for t in (b, u):
            if (t.dtype != torch.float64 or t.device != self.device or tuple(t.shape) != self.shape
                    or t.stride(1) != 1):
                raise ValueError(f"expected {self.shape} float64 tensors on {self.device}")
        if b.stride(0) != u.stride(0):
            raise ValueError("b and u must share a row pitch (u may be b: solved in place)")
        stream = torch.cuda.current_stream(self.device)
        handle = _lib.stream_handle(stream)
        with self._lock:
            ordered = not torch.cuda.is_current_stream_capturing()
            if ordered and self._ran_on not in (None, handle):
                stream.wait_event(self._done)
            _lib.check(_lib.lib().gd_dct_solve_neumann(self._handle, _lib.ptr(b), _lib.ptr(u),
                                                       u.stride(0), handle),
                       "gd_dct_solve_neumann")
            if ordered:
                self._done.record(stream)
                self._ran_on = handle
        return u

    def __del__(self):
        if getattr(self, "_handle", None):
            try:
                torch.cuda.current_stream(self.device).synchronize()
                if self._ran_on is not None:
                    self._done.synchronize()  # the last solve, whichever stream it ran on
                _lib.lib().gd_dct_plan_destroy(self._handle)
            except Exception:
                pass
            self._handle = None


_DCT_PLANS: OrderedDict = OrderedDict()


def _dct_plan(h: int, w: int) -> DctPlan:
    key = (h, w, torch.cuda.current_device())
    with _PIPELINE_LOCK:
        plan = _DCT_PLANS.pop(key, None)
        if plan is None:
            plan = DctPlan(h, w)
        _DCT_PLANS[key] = plan
        while len(_DCT_PLANS) > 8:
            _DCT_PLANS.popitem(last=False)
    return plan


def solve_neumann(b, tolerance: float = NEUMANN_EXACT_TOLERANCE,
                  max_iterations: int = 2000, method: str = "mgcg") -> np.ndarray:
    """Zero-mean solution of ``laplacian(u) = b`` with homogeneous Neumann boundaries.

    ``method="mgcg"`` (default) replaces the DCT solve of solvers.py:224-262
    with the B200 MGPCG on the edge-replicated operator; the default tolerance
    drives the true relative residual to 1e-14, so that even the smoothest
    error mode is reduced to the rounding level of the exact transform solve.
    ``method="dct"`` runs the reference's own algorithm (forward DCT-II,
    division by the eigenvalues, inverse) on the device with this library's
    FFT kernels (sides up to 8192; larger grids raise ``ValueError``).  Either
    way any constant component of ``b`` is discarded and the solution has
    zero mean.
    """
    b = np.asarray(b, dtype=float)
    if b.ndim != 2:
        raise ValueError("solve_neumann expects a 2-D right-hand side")
    if method == "dct":
        if min(b.shape) < 2 or max(b.shape) > DCT_MAX_SIDE:
            raise ValueError(f"the DCT solver takes sides of 2 to {DCT_MAX_SIDE} cells, "
                             f"not {b.shape}")
        dev = _lib.device()
        bd = _dev_array(b, dev)
        return download(_dct_plan(*b.shape).solve(bd, torch.empty_like(bd)))
    if method != "mgcg":
        raise KeyError(f"unknown Neumann method {method!r}; choose 'mgcg' or 'dct'")
    params = SolveParams(tolerance=tolerance, max_iterations=max_iterations)
    u, _ = _plan_solve(b, 1.0, "neumann", params, zero_mean=True)
    return u


def solve_neumann_batch(b, tolerance: float = NEUMANN_EXACT_TOLERANCE, max_iterations: int = 2000,
                        precision: str = "mixed", out: torch.Tensor | None = None,
                        method: str = "mgcg"):
    """:func:`solve_neumann` for a stack of right-hand sides ``(n, h, w)`` in one batched solve.

    ``b`` may be a NumPy array or a (preferably pinned) CPU torch tensor; with
    ``out`` (a CPU tensor of the same shape) the solutions are copied there and
    ``out`` is returned, otherwise a new NumPy array is.  All ``n`` problems go
    through the same kernel launches (they are instances of one plan), except
    when ``b`` and ``out`` are both pinned FP64 tensors: then each problem has
    its own plan and stream, so host-device copies overlap the solves (the
    results are bitwise the same either way).  ``method="dct"`` solves each
    right-hand side with the exact transform solver instead.
    """
    dev = _lib.device()
    if method == "dct":
        f = (b.to(device=dev, dtype=torch.float64) if isinstance(b, torch.Tensor)
             else upload(b, dev, np.float64))
        if f.dim() != 3 or min(f.shape[1:]) < 2:
            raise ValueError("solve_neumann_batch expects an (n, h, w) stack with h, w >= 2")
        f = f.contiguous()
        plan = _dct_plan(f.shape[1], f.shape[2])
        x = torch.empty_like(f)
        for k in range(f.shape[0]):
            plan.solve(f[k], x[k])
        solve_neumann_batch.last_results = []
        if out is not None:
            out.copy_(x, non_blocking=True)
            torch.cuda.current_stream().synchronize()
            return out
        return download(x)
    if method != "mgcg":
        raise KeyError(f"unknown Neumann method {method!r}; choose 'mgcg' or 'dct'")
    if (isinstance(b, torch.Tensor) and isinstance(out, torch.Tensor) and b.dim() == 3
            and b.shape[0] > 1 and b.dtype == torch.float64 and out.dtype == torch.float64
            and b.device.type == "cpu" and out.device.type == "cpu" and b.is_pinned()
            and out.is_pinned() and out.shape == b.shape):
        params = SolveParams(precision=precision, tolerance=tolerance,
                             max_iterations=max_iterations, zero_start=True)
        solve_neumann_batch.last_results = _pipelined_neumann(b, out, params)
        return out
    if isinstance(b, torch.Tensor):
        f = b.to(device=dev, dtype=torch.float64, non_blocking=True)
    else:
        f = upload(b, dev, np.float64)
    if f.dim() != 3:
        raise ValueError("solve_neumann_batch expects an (n, h, w) stack")
    n, h, w = f.shape
    params = SolveParams(precision=precision, tolerance=tolerance, max_iterations=max_iterations,
                         zero_start=True)
    plan = cached_plan(tuple(Instance(h, w, "neumann", True) for _ in range(n)), params)
    x = torch.empty_like(f)
    results = plan.solve(list(f), list(x), scale=-1.0)
    if out is not None:
        out.copy_(x, non_blocking=True)
        torch.cuda.current_stream().synchronize()
        solve_neumann_batch.last_results = results
        return out
    solve_neumann_batch.last_results = results
    return download(x)


solve_neumann_batch.last_results = []

_PIPELINES: OrderedDict = OrderedDict()
_PIPELINE_LOCK = threading.Lock()


def _take_pipeline(h: int, w: int, params: SolveParams, n: int):
    """``n`` single-instance plans, each with its own stream and device buffers.

    A pipeline is removed from the pool while in use, so concurrent callers of
    the same shape (or calls still in flight) each get their own.
    """
    key = (h, w, params, n)
    with _PIPELINE_LOCK:
        idle = _PIPELINES.get(key)
        if idle:
            _PIPELINES.move_to_end(key)
            return key, idle.pop()
    dev = _lib.device()
    pipe = []
    inst = Instance(h, w, "neumann", True)
    params = resolve([inst], params)
    for _ in range(n):
        stream = torch.cuda.Stream(dev)
        with torch.cuda.stream(stream):
            plan = PoissonPlan([inst], params, stream=stream)
            f = torch.empty((h, w), dtype=torch.float64, device=dev)
            x = torch.empty_like(f)
        pipe.append((plan, stream, f, x))
    return key, pipe


_PIPELINES_KEPT = 8  # idle pipelines kept over all shapes


def _return_pipeline(key, pipe) -> None:
    closing = []
    with _PIPELINE_LOCK:
        _PIPELINES.setdefault(key, []).append(pipe)
        _PIPELINES.move_to_end(key)
        while sum(len(v) for v in _PIPELINES.values()) > _PIPELINES_KEPT:
            old_key = next(iter(_PIPELINES))
            closing.append(_PIPELINES[old_key].pop(0))
            if not _PIPELINES[old_key]:
                del _PIPELINES[old_key]
    for old in closing:
        for plan, *_ in old:
            plan.close()


class NeumannBatchFuture:
    """A :func:`solve_neumann_batch_async` call in flight.  ``result()`` waits for
    its solves and downloads and returns ``out``; ``reports`` then holds one
    result per right-hand side."""

    def __init__(self, out: torch.Tensor, key, pipe):
        self.out = out
        self.reports: list = []
        self._key, self._pipe = key, pipe

    def done(self) -> bool:
        return self._pipe is None

    def result(self) -> torch.Tensor:
        if self._pipe is None:
            return self.out
        pipe, self._pipe = self._pipe, None
        try:
            for plan, stream, f, x in pipe:
                self.reports.extend(plan.finish())
                stream.synchronize()
        except BaseException:
            for plan, *_ in pipe:
                plan.close()
            raise
        _return_pipeline(self._key, pipe)
        return self.out


def _launch_pipelined(b: torch.Tensor, out: torch.Tensor, params: SolveParams):
    """Channel k's upload, solve and download run on stream k: the copy of one
    channel overlaps the solves of the others (copy engines and SMs work at the
    same time), and each solve is one graph with a device-side loop.  Returns
    without waiting."""
    n, h, w = b.shape
    key, pipe = _take_pipeline(h, w, params, n)
    try:
        caller = torch.cuda.current_stream()
        for k, (plan, stream, f, x) in enumerate(pipe):
            stream.wait_stream(caller)
            with torch.cuda.stream(stream):
                f.copy_(b[k], non_blocking=True)
                plan.solve_async([f], [x], scale=-1.0)
                out[k].copy_(x, non_blocking=True)
    except BaseException:
        for plan, *_ in pipe:
            plan.close()
        raise
    return NeumannBatchFuture(out, key, pipe)


def _pipelined_neumann(b: torch.Tensor, out: torch.Tensor, params: SolveParams):
    fut = _launch_pipelined(b, out, params)
    fut.result()
    return fut.reports


def solve_neumann_batch_async(b: torch.Tensor, out: torch.Tensor,
                              tolerance: float = NEUMANN_EXACT_TOLERANCE,
                              max_iterations: int = 2000,
                              precision: str = "mixed") -> NeumannBatchFuture:
    """:func:`solve_neumann_batch` without waiting, for callers that keep several
    batches in flight (the next batch's uploads then overlap this one's solves
    and downloads).  ``b`` and ``out`` are pinned FP64 CPU tensors of one shape
    ``(n, h, w)``; neither may be touched until ``result()`` has returned.  The
    solutions are bitwise those of :func:`solve_neumann_batch`."""
    if not (isinstance(b, torch.Tensor) and isinstance(out, torch.Tensor) and b.dim() == 3
            and b.dtype == torch.float64 and out.dtype == torch.float64
            and b.device.type == "cpu" and out.device.type == "cpu" and b.is_pinned()
            and out.is_pinned() and out.shape == b.shape):
        raise ValueError("solve_neumann_batch_async takes pinned FP64 CPU tensors b and out "
                         "of one (n, h, w) shape")
    params = SolveParams(precision=precision, tolerance=tolerance,
                         max_iterations=max_iterations, zero_start=True)
    return _launch_pipelined(b, out, params)
