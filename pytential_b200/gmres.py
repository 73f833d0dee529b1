"""Batched GMRES for many right-hand sides through one apply per iteration.

The iteration is the reference's (``pytential/linalg/gmres.py:143-315``): a
residual-minimizing method that keeps orthonormal images ``Ae[k]`` and their
preimages ``e[k]``, double-orthogonalizes each new direction ``A r`` against the
last ``restart`` images, recomputes the true residual every 10 iterations, and
fails on non-monotonic residuals or stalls.  Here every quantity carries a leading
density axis: one call of ``op`` applies the operator to all unconverged densities
at once (one traversal of the FMM lists per iteration for all of them), and the
inner products, norms and updates are per density, in float64 / complex128 on the
device.  A density stops changing once its residual meets the tolerance.

On a GPU the orthogonalization and the updates of an iteration are one kernel launch
(``qbxfmm_gmres_step``), which takes plain contiguous float64 or complex128 tensors
outside of autograd; anything else, and few densities of very many unknowns, goes through
the tensor operations below.
"""

from __future__ import annotations

import ctypes
from dataclasses import dataclass, field

import torch


class GMRESError(RuntimeError):
    pass


@dataclass
class GMRESResult:
    """Mirror of ``GMRESResult`` (pytential/linalg/gmres.py:124-141) for a batch:
    ``residual_norms[i]`` holds the residual norms of all densities at iteration i."""
    solution: torch.Tensor
    residual_norms: list = field(default_factory=list)
    iteration_count: int = 0
    success: bool = False
    state: str = ""
    converged: torch.Tensor | None = None          # per density


def _dot(a, b):
    """Per-density inner product sum(conj(a) * b) over the last axis."""
    return torch.sum(a.conj() * b, dim=-1)


def _plain(*tensors):
    """Whether the kernel can take the tensors: same shape, type and GPU, contiguous, and
    nothing that records or transforms operations on them."""
    t0 = tensors[0]
    if not t0.is_cuda or t0.dtype not in (torch.float64, torch.complex128):
        return False
    # modes that see every operation (counters, recorders, tracers) would miss the kernel's
    if torch.jit.is_tracing() or torch._C._len_torch_dispatch_stack() > 0:
        return False
    return all(
        type(t) is torch.Tensor and t.shape == t0.shape and t.dtype == t0.dtype
        and t.device == t0.device and t.is_contiguous() and not t.is_conj() and not t.is_neg()
        and not (torch.is_grad_enabled() and t.requires_grad)
        and not torch._C._functorch.is_functorch_wrapped_tensor(t)
        and torch.autograd.forward_ad.unpack_dual(t).tangent is None
        for t in tensors) and t0.shape[0] <= 65535


def _step_wins(nd, n):
    """Whether the kernel is faster than the tensor operations.  It gives a density eight
    SMs, which wait on one another at every inner product; the tensor operations use the
    whole GPU but read and write every vector at every step.  Kernel against operations,
    float64 and complex128, 2 to 40 kept images, 1 to 64 densities: 6224 unknowns 37-374
    against 410-3933 us, 65 536 (the slowest for the kernel: 4 densities, 40 images, float64)
    2.5 against 3.2 ms; 131 072, 40 images: 1 density 3.9-5.8 against 3.3-4.1 ms, 64 densities
    9.4-14.7 against 13.9-28.6; 307 200, 40 images: 1 density 11.1-13.5 against 3.3-4.1 ms, 16
    16.4-22.3 against 8.3-17.5, 64 21.7-34.8 against 30.9-64.0."""
    return n <= 65536 or nd >= 64


def _step(Ae, e, w, r, x, active, update_r):
    """One iteration's orthogonalization and update: ``w``, its preimage, the next residual
    (``r`` itself unless ``update_r``) and the next ``x`` as new tensors (an operator or a
    callback may have kept the ones it was given)."""
    from . import native
    nd, n = r.shape
    w1, v, x1 = torch.empty_like(w), torch.empty_like(r), x.clone()
    r1 = torch.empty_like(r) if update_r else None
    arr = ctypes.c_void_p * max(len(Ae), 1)
    with torch.cuda.device(r.device):
        native.call("qbxfmm_gmres_step", int(r.dtype == torch.complex128), nd, n, len(Ae),
                    arr(*[t.data_ptr() for t in Ae]), arr(*[t.data_ptr() for t in e]),
                    w.data_ptr(), r.data_ptr(), w1.data_ptr(), v.data_ptr(), active.data_ptr(),
                    None if r1 is None else r1.data_ptr(), x1.data_ptr(),
                    torch.cuda.current_stream(r.device).cuda_stream)
    return w1, v, r if r1 is None else r1, x1


def gmres(op, rhs: torch.Tensor, restart: int | None = None, tol: float | None = None,
          x0: torch.Tensor | None = None, maxiter: int | None = None,
          hard_failure: bool | None = None, no_progress_factor: float | None = None,
          stall_iterations: int | None = None, callback=None,
          require_monotonicity: bool = True) -> GMRESResult:
    """Solve ``op(X) = rhs`` for every row of ``rhs`` (shape ``(ndens, n)``)."""
    rhs = torch.atleast_2d(rhs)
    nd, n = rhs.shape
    if restart is None:
        restart = min(n, 20)
    if tol is None:
        tol = 1e-5
    if maxiter is None:
        maxiter = 2 * n
    if hard_failure is None:
        hard_failure = True
    if stall_iterations is None:
        stall_iterations = 10
    if no_progress_factor is None:
        no_progress_factor = 1.25

    def norm(x):
        return torch.sqrt(torch.abs(_dot(x, x)))

    if x0 is None:
        x = torch.zeros_like(rhs)
        r = rhs.clone()
        recalc_r = False
    else:
        x = x0.clone()
        recalc_r = True
    Ae = [None] * restart
    e = [None] * restart
    k = 0
    # the norms are on the host anyway: so are the decisions, one read an iteration
    norm_b = norm(rhs).detach().cpu()
    last = None
    residual_norms = []
    done = torch.zeros(nd, dtype=torch.bool)
    active = ~done
    active_dev = active.to(rhs.device)

    def finish(success, state, iteration):
        if not success and hard_failure:
            raise GMRESError(state)
        return GMRESResult(solution=x, residual_norms=residual_norms, iteration_count=iteration,
                           success=success, state=state, converged=done.to(rhs.device, copy=True))

    for iteration in range(maxiter):
        if k == restart:
            k = 0
            orth_count = restart
        else:
            orth_count = k
        if recalc_r:
            r = rhs - op(x)
        norm_r = norm(r).detach().cpu()
        residual_norms.append(norm_r)
        if callback is not None:
            callback(r)
        done = done | (norm_r < tol * norm_b) | (norm_r == 0)
        if bool(done.all()):
            return finish(True, "success", iteration)
        if not torch.equal(active, ~done):
            active = ~done
            active_dev = active.to(rhs.device)
        if last is not None:
            if require_monotonicity and bool(((norm_r > 1.25 * last) & active).any()):
                return finish(False, "non-monotonic residuals", iteration)
            if stall_iterations and len(residual_norms) > stall_iterations:
                old = residual_norms[-stall_iterations]
                if bool(((norm_r > old / no_progress_factor) & active).all()):
                    return finish(False, "stalled", iteration)
        last = norm_r

        w = op(r)
        recalc_r = (iteration + 1) % 10 == 0
        if _step_wins(nd, rhs.shape[1]) and _plain(w, r, x, *Ae[:orth_count], *e[:orth_count]):
            Ae[k], e[k], r, x = _step(Ae[:orth_count], e[:orth_count], w, r, x, active_dev,
                                      not recalc_r)
            k += 1
            continue
        rp = r
        for _ in range(2):
            for j in range(orth_count):
                d = _dot(Ae[j], w)[:, None]
                w = w - d * Ae[j]
                rp = rp - d * e[j]
            nw = norm(w)
            inv = torch.where(active_dev & (nw > 0), 1.0 / torch.where(nw > 0, nw, 1.0),
                              torch.zeros_like(nw))[:, None]
            w = inv * w
            rp = inv * rp
        Ae[k] = w
        e[k] = rp
        d = _dot(Ae[k], r)[:, None]
        d = torch.where(active_dev[:, None], d, torch.zeros_like(d))   # converged densities stay
        if not recalc_r:
            r = r - d * Ae[k]
        x = x + d * e[k]
        k += 1
    return finish(False, "max iterations", maxiter)
