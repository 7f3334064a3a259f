"""Rectangular spectral Helmholtz solves by transform-matrix products on
the tensor cores.

``solve_helmholtz_dst(rhs, dx, dy, lambda_)`` is the drop-in for
spectraldiffx's ``solve_helmholtz_dst`` that finitevolX re-exports
(solvers/spectral.py:14-98): it solves (nabla^2 - lambda) psi = rhs on the
interior-only array ``rhs`` [..., Ny, Nx] with psi = 0 outside.
``solve_helmholtz_dct`` (Neumann, DCT-II) and ``solve_helmholtz_fft``
(periodic) are the other two solvers that finitevolX's ``_spectral_solve``
dispatches on (spectral.py:105-128); they take the whole [..., Ny, Nx]
array and return the zero-mean solution when the problem has a null mode
(lambda = 0).  The periodic solve uses the real Hartley transform pair, the
same linear map as the FFT solve on real data.

* float32 input: 3xBF16-split tcgen05 GEMM chain, FP32 accumulation
  (relative error ~1e-5 of the FP64 answer);
* float64 input: the FP64 chain (``method="fp64"``, default) or the
  split chain with FP64 iterative refinement (``method="refine"``) to a
  normwise backward error ``tol``.
``lambda_`` may be a scalar or one value per layer (shape [nl], matching
``rhs.shape[-3]``, as ``pv_inversion`` uses it).
"""

from __future__ import annotations

import ctypes
import math
import threading

import numpy as np
import torch

from finitevolx_b200 import _lib as L
from finitevolx_b200._lib import D, I, P, check, fn, stream_ptr

I64 = ctypes.c_longlong


KINDS = {"dst": 0, "dct": 1, "fft": 2}


class DSTHelmholtzPlan:
    """Pre-built transform matrices, eigenvalue grids and workspaces for one
    size and boundary condition (``bc``: "dst" Dirichlet, "dct" Neumann,
    "fft" periodic).

    Creating a plan allocates device memory once; ``solve`` allocates
    nothing on the device besides its output (pass ``out=`` to avoid that).
    A plan has one set of workspaces: threads may share it on one stream, but
    a stream of its own needs a plan of its own (as the solve_* functions have).
    """

    def __init__(self, ny: int, nx: int, dx: float, dy: float, lambdas=(0.0,), batch_max: int = 1,
                 fp64: bool = True, bc: str = "dst"):
        L.require_cuda()
        if bc not in KINDS:
            raise ValueError(f"bc must be 'fft', 'dst', or 'dct'; got {bc!r}")
        lam = np.atleast_1d(np.asarray(lambdas, dtype=np.float64))
        self.ny, self.nx, self.dx, self.dy = int(ny), int(nx), float(dx), float(dy)
        self.bc = bc
        self.lambdas = lam
        self.batch_max = int(batch_max)
        self._lock = threading.Lock()  # a solve's launches stay together
        self._h = ctypes.c_void_p()
        lam_c = (ctypes.c_double * len(lam))(*lam.tolist())
        check(fn("fvx_spectral_plan_create")(I(KINDS[bc]), I(self.ny), I(self.nx), D(self.dx), D(self.dy),
                                             I(self.batch_max), lam_c, I(len(lam)), I(int(fp64)),
                                             ctypes.byref(self._h)),
              "SpectralHelmholtzPlan")
        self.split_ok = (self.nx % 8 == 0) and (self.ny % 8 == 0)
        self.fp64 = bool(fp64) or not self.split_ok  # has the FP64 chain

    def __del__(self):
        h = getattr(self, "_h", None)
        if h is not None and h.value:
            try:
                fn("fvx_dst_plan_destroy")(h)
            except Exception:
                pass
            self._h = None

    @property
    def handle(self):
        return self._h

    def _views(self, rhs):
        if rhs.shape[-2:] != (self.ny, self.nx):
            raise ValueError(f"rhs interior shape {tuple(rhs.shape[-2:])} != plan {(self.ny, self.nx)}")
        b = math.prod(rhs.shape[:-2])
        if b > self.batch_max:
            raise ValueError(f"batch {b} exceeds the plan's batch_max {self.batch_max}")
        return b

    def solve(self, rhs, out=None, method: str = "fp64") -> torch.Tensor:
        rhs = L.as_field(rhs)
        b = self._views(rhs)
        out = torch.empty_like(rhs) if out is None else out
        plane = self.ny * self.nx
        if rhs.dtype == torch.float32:
            with self._lock:
                st = fn("fvx_dst_solve_f32")(self._h, P(rhs), I64(plane), I64(self.nx), P(out), I64(plane),
                                             I64(self.nx), I(b), stream_ptr())
            check(st, "solve_helmholtz_dst")
        elif rhs.dtype == torch.float64:
            m = {"fp64": 0, "refine": 1}[method]
            info = (ctypes.c_double * 3)()
            with self._lock:
                st = fn("fvx_dst_solve_f64")(self._h, P(rhs), I64(plane), I64(self.nx), P(out), I64(plane),
                                             I64(self.nx), I(b), I(m), D(1e-12), I(8), info, stream_ptr())
            check(st, "solve_helmholtz_dst")
        else:
            raise TypeError(f"unsupported dtype {rhs.dtype}")
        return out

    def solve_refined(self, rhs, tol: float = 1e-12, max_iter: int = 8, out=None):
        """Split-BF16 solve + FP64 iterative refinement (Dirichlet plans).

        Returns (psi, info) with info = {passes, backward_error, rel_residual};
        backward_error = ||r|| / (||A|| ||psi|| + ||rhs||).
        """
        if self.bc != "dst":
            raise ValueError("iterative refinement is provided for the Dirichlet (DST) plan only")
        rhs = L.as_field(rhs, dtype=torch.float64)
        b = self._views(rhs)
        out = torch.empty_like(rhs) if out is None else out
        plane = self.ny * self.nx
        info = (ctypes.c_double * 3)()
        with self._lock:
            st = fn("fvx_dst_solve_f64")(self._h, P(rhs), I64(plane), I64(self.nx), P(out), I64(plane), I64(self.nx),
                                         I(b), I(1), D(tol), I(max_iter), info, stream_ptr())
        res = dict(passes=int(info[0]), backward_error=float(info[1]), rel_residual=float(info[2]),
                   converged=st == 0)
        if st not in (0, 5):
            check(st, "solve_helmholtz_dst (refined)")
        return out, res

    def check_device(self):
        """Raises if a bounded device wait of the plan's products gave up
        since the last check (the flag is cleared once reported)."""
        check(fn("fvx_dst_plan_check")(self._h, stream_ptr()), "DST kernels")

    def set_wait_limit(self, cycles: int) -> None:
        """Bound, in SM clock cycles, on each barrier wait of the products."""
        check(fn("fvx_dst_plan_set_wait_limit")(self._h, ctypes.c_longlong(int(cycles))), "wait limit")

    def hold(self, stream: int) -> None:
        """Counts the graph being captured on ``stream`` as a holder."""
        check(fn("fvx_dst_plan_hold")(self._h, ctypes.c_void_p(stream)), "plan in a capture")

    def holds(self) -> int:
        """Graphs that hold the plan: it has to live while there are any."""
        return fn("fvx_dst_plan_holds")(self._h)

    def set_kernel(self, kind: int) -> None:
        """Even/odd product kernel of this plan (an index of autotune's
        DST_KERNELS); -1: the process's choice."""
        check(fn("fvx_dst_plan_kernel")(self._h, I(int(kind))), "dst kernel")


class _PlanPool:
    """The plans behind ``get_plan``: one per problem and stream, because a plan's
    workspaces serve one stream at a time, each as large as the largest batch
    asked of it.  A problem keeps the plans of at most ``STREAMS`` streams (all
    that PyTorch hands out, and the default one); the oldest goes first.

    A capture gets plans of its own, made during it: its graph runs on any
    stream, at any time, so it shares no workspace with calls outside.  They
    live until their graph is gone, and serve the next capture after that.

    ``make(key, batch, fp64)`` creates a plan."""

    STREAMS = 33

    def __init__(self, make):
        self._make, self._plans, self._lock = make, {}, threading.Lock()
        self._held: list = []  # ((key, stream, capture), plan) of graphs

    @staticmethod
    def _serves(p, batch, fp64) -> bool:
        return p is not None and p.batch_max >= batch and (p.fp64 or not fp64)

    def get(self, key, stream: int, batch: int, fp64: bool, capture: int = 0):
        """``capture``: the id of the capture ``stream`` is in, or 0."""
        if capture:
            return self._for_graph(key, stream, batch, fp64, capture)
        p = self._plans.get((key, stream))
        if self._serves(p, batch, fp64):
            return p
        with self._lock:
            p = self._plans.get((key, stream))
            if self._serves(p, batch, fp64):
                return p
            self._held = [(k, h) for k, h in self._held if h.holds()]
            others = [k for k in self._plans if k[0] == key and k[1] != stream]
            if p is None and len(others) >= self.STREAMS:
                del self._plans[others.pop(0)]
            if p is not None:  # replaced by one that serves its callers too
                batch, fp64 = max(batch, p.batch_max), fp64 or p.fp64
            try:
                p = self._make(key, batch, fp64)
            except L.FvxError:
                if not others:
                    raise
                for k in others:  # give the other streams' memory back and try again
                    del self._plans[k]
                p = self._make(key, batch, fp64)
            self._plans[(key, stream)] = p
            return p

    def _for_graph(self, key, stream, batch, fp64, capture):
        with self._lock:
            for k, p in self._held:
                if k == (key, stream, capture) and self._serves(p, batch, fp64):
                    return p
            free = [h for h in self._held if h[0][0] == key and not h[1].holds() and self._serves(h[1], batch, fp64)]
            if free:
                self._held.remove(free[0])
                p = free[0][1]
            else:
                try:
                    p = self._make(key, batch, fp64)
                except L.FvxError:  # no memory for another: the graph takes one over
                    k = next((k for k, e in self._plans.items() if k[0] == key and self._serves(e, batch, fp64)), None)
                    if k is None:
                        raise
                    p = self._plans.pop(k)
            p.hold(stream)
            self._held.append(((key, stream, capture), p))
            return p


_POOL = _PlanPool(lambda key, batch, fp64: DSTHelmholtzPlan(*key[1:6], batch_max=max(batch, 1), fp64=fp64, bc=key[0]))


SpectralHelmholtzPlan = DSTHelmholtzPlan


def _lambda_tuple(lam) -> tuple:
    """The lambda values as a tuple of floats (one for a scalar)."""
    if isinstance(lam, (float, int)):
        return (float(lam),)
    if isinstance(lam, torch.Tensor):
        lam = lam.cpu()
    return tuple(np.atleast_1d(np.asarray(lam, dtype=np.float64)).tolist())


def get_plan(ny, nx, dx, dy, lambdas, batch, fp64=True, bc: str = "dst") -> DSTHelmholtzPlan:
    """The current stream's plan of a problem, for up to ``batch`` fields; during
    a capture, one that belongs to its graph."""
    dev = torch.cuda.current_device()
    key = (bc, ny, nx, float(dx), float(dy), _lambda_tuple(lambdas), dev)
    stream, capture = torch._C._cuda_getCurrentRawStream(dev), 0
    if L.capturing():
        cid = ctypes.c_ulonglong()
        check(fn("fvx_capture_id")(ctypes.c_void_p(stream), ctypes.byref(cid)), "capture")
        capture = cid.value
    return _POOL.get(key, stream, batch, fp64, capture)


def _solve(rhs, dx, dy, lambda_, method, bc):
    rhs = L.as_field(rhs)
    if rhs.ndim < 2:
        raise ValueError("rhs must be at least 2-D")
    lam = _lambda_tuple(lambda_)
    if len(lam) > 1 and (rhs.ndim < 3 or rhs.shape[-3] != len(lam)):
        raise ValueError(f"rhs.shape[-3] must match the {len(lam)} lambda values")
    ny, nx = rhs.shape[-2:]
    b = math.prod(rhs.shape[:-2])
    return get_plan(ny, nx, dx, dy, lam, b, bc=bc).solve(rhs, method=method)


def solve_helmholtz_dct(rhs, dx: float, dy: float, lambda_=0.0) -> torch.Tensor:
    """(nabla^2 - lambda) psi = rhs with homogeneous Neumann walls (cell-centred,
    DCT-II); zero-mean psi when lambda = 0."""
    return _solve(rhs, dx, dy, lambda_, "fp64", "dct")


def solve_helmholtz_fft(rhs, dx: float, dy: float, lambda_=0.0) -> torch.Tensor:
    """(nabla^2 - lambda) psi = rhs on a doubly periodic grid; zero-mean psi
    when lambda = 0."""
    return _solve(rhs, dx, dy, lambda_, "fp64", "fft")


def solve_poisson_dct(rhs, dx: float, dy: float) -> torch.Tensor:
    return solve_helmholtz_dct(rhs, dx, dy, 0.0)


def solve_poisson_fft(rhs, dx: float, dy: float) -> torch.Tensor:
    return solve_helmholtz_fft(rhs, dx, dy, 0.0)


def spectral_solve(rhs, dx: float, dy: float, lambda_, bc: str) -> torch.Tensor:
    """The rectangular solver for ``bc`` (spectral.py:105-128 ``_spectral_solve``)."""
    if bc not in KINDS:
        raise ValueError(f"base_bc must be 'fft', 'dst', or 'dct'; got {bc!r}")
    return _solve(rhs, dx, dy, lambda_, "fp64", bc)


def make_spectral_preconditioner(dx: float, dy: float, lambda_: float = 0.0, bc: str = "fft"):
    """M_inv(r) = the rectangular spectral solve of (nabla^2 - lambda)
    (preconditioners.py:44-84); default periodic."""
    if bc not in KINDS:
        raise ValueError(f"bc must be 'fft', 'dst', or 'dct'; got {bc!r}")
    return lambda r: spectral_solve(r, dx, dy, lambda_, bc)


def dct2_eigenvalues(n: int, d: float) -> np.ndarray:
    k = np.arange(n)
    return -4.0 / d ** 2 * np.sin(np.pi * k / (2 * n)) ** 2


def fft_eigenvalues(n: int, d: float) -> np.ndarray:
    k = np.arange(n)
    return -4.0 / d ** 2 * np.sin(np.pi * k / n) ** 2


def solve_helmholtz_dst(rhs, dx: float, dy: float, lambda_=0.0, method: str = "fp64") -> torch.Tensor:
    """(nabla^2 - lambda) psi = rhs with psi = 0 outside the interior array."""
    return _solve(rhs, dx, dy, lambda_, method, "dst")


def solve_poisson_dst(rhs, dx: float, dy: float) -> torch.Tensor:
    return solve_helmholtz_dst(rhs, dx, dy, 0.0)


def dst1_eigenvalues(n: int, d: float) -> np.ndarray:
    k = np.arange(n)
    return -4.0 / d ** 2 * np.sin(np.pi * (k + 1) / (2 * (n + 1))) ** 2
