"""Drop-in replacement for the reference's ``src/bem/solver.py``.

Same public names, argument meaning, dtypes, shapes and return types as the
reference (``BEM_Solver`` solver.py:69-147, ``solve_linear_equation``
:61-66, ``map_triangle2vertex`` :150-154, ``preprocess`` :40-58,
``check_tensor`` :34-37); every computation runs in ``libbemb200.so``
(hand-written sm_100a kernels) through its C ABI.  Differences a caller can
see:

* the default linear solver is the device-resident GMRES with FP64
  refinement (same stopping test as the reference's BiCGSTAB:
  ``||b - A x||^2 < tol ||b||^2``); ``solver="bicgstab"`` runs the
  reference's BiCGSTAB iteration instead;
* new keyword-only options: ``precision`` of the Krylov matvec ("fp32":
  CUDA cores; "fp16x3": tensor cores with fp16 hi/lo splits and scales,
  FP32-level accuracy; "bf16x3" / "bf16": tensor cores with bf16 splits,
  ~3e-5 / ~1e-3, refined in FP64), ``solver``, ``restart``, ``rtol``;
  right-hand sides may be (N,) or (N, m);
* ``boundary2potential``/``single_potential``/``double_potential`` evaluate
  listeners without building the P x N potential matrices;
* mesh errors raise ``BEMError`` (the reference has no checks).

The geometry (normals, curls, quadrature points, tiles, touching pairs) is
built once per ``BEM_Solver`` and reused by every call.
"""
from __future__ import annotations

import contextlib
import ctypes
import math

import numpy as np
import torch

from .. import _lib as L
from .bicgstab import BiCGSTAB

_LAYERS = {
    "single": L.SINGLE_LAYER,
    "double": L.DOUBLE_LAYER,
    "adjointdouble": L.ADJOINT_DOUBLE_LAYER,
    "hypersingular": L.HYPERSINGULAR,
    "bm_lhs": L.BM_LHS,
    "bm_rhs": L.BM_RHS,
}
_PRECISIONS = {"fp32": L.PREC_FP32, "bf16x3": L.PREC_BF16X3, "bf16": L.PREC_BF16, "fp16x3": L.PREC_FP16X3}


def _vp(t) -> int:
    """Device address for a ``void*`` argument (the bindings declare the type)."""
    return 0 if t is None else t.data_ptr()


def _stream(device=None) -> int:
    return torch.cuda.current_stream(device).cuda_stream


_HERE = contextlib.nullcontext()


def _on(device: torch.device):
    """``torch.cuda.device(device)`` where another device is current, else
    nothing (entering and leaving it takes microseconds of a short call)."""
    return _HERE if device.index == torch.cuda.current_device() else torch.cuda.device(device)


def check_tensor(tensor, dtype):
    """Same contract as the reference (solver.py:34-37)."""
    assert tensor.dtype == dtype
    assert tensor.is_cuda
    assert tensor.is_contiguous()


class Geometry:
    """Device workspace holding the preprocessed mesh (C ABI ``bem_geometry_*``)."""

    def __init__(self, vertices: torch.Tensor, triangles: torch.Tensor):
        lib = L.lib()
        self.device = vertices.device
        self.nv = int(vertices.shape[0])
        self.nt = int(triangles.shape[0])
        with _on(self.device):
            st = _stream(self.device)
            nbytes = ctypes.c_size_t(0)
            L.check(lib.bem_geometry_bytes(_vp(vertices), self.nv, _vp(triangles), self.nt, ctypes.byref(nbytes), st),
                    "bem_geometry_bytes")
            self.buffer = torch.empty(int(nbytes.value), dtype=torch.uint8, device=self.device)
            L.check(lib.bem_geometry_build(_vp(vertices), self.nv, _vp(triangles), self.nt, _vp(self.buffer),
                                           int(nbytes.value), st), "bem_geometry_build")

    @property
    def ptr(self) -> ctypes.c_void_p:
        return ctypes.c_void_p(self.buffer.data_ptr())

    def check_status(self) -> None:
        """Raise ``BEMError`` (BEM_ERR_CUDA) if a bounded wait of an assembly
        kernel expired on this geometry since the last check (the matrices
        assembled meanwhile may be wrong); synchronises the current stream."""
        with _on(self.device):
            L.check(L.lib().bem_geometry_status(_vp(self.buffer), _stream(self.device)), "assembly on this geometry")

    def __del__(self):
        # the library caches the header per workspace address: forget it
        # before the allocator can hand the address to another buffer
        try:
            buf = self.__dict__.get("buffer")
            if buf is not None:
                L.lib().bem_geometry_release(_vp(buf))
        except Exception:
            pass

    def normals_and_curls(self):
        normals = torch.empty((self.nt, 3), dtype=torch.float32, device=self.device)
        curls = torch.empty((self.nt, 3, 3), dtype=torch.float32, device=self.device)
        with _on(self.device):
            L.check(L.lib().bem_geometry_normals(_vp(self.buffer), _vp(normals), _vp(curls), _stream(self.device)),
                    "bem_geometry_normals")
        return normals, curls


def preprocess(vertices, triangles):
    """Unit triangle normals (T,3) and surface curls (T,3,3) (solver.py:40-58)."""
    g = Geometry(vertices, triangles)
    return g.normals_and_curls()


def cmatmul(A: torch.Tensor, X: torch.Tensor) -> torch.Tensor:
    """Y = A X for complex64 A (n,n) and X (n,) or (n,m), on the library's kernel."""
    check_tensor(A, torch.complex64)
    n = A.shape[0]
    Xc = X.contiguous()
    m = 1 if Xc.dim() == 1 else Xc.shape[1]
    Y = torch.empty_like(Xc)
    with _on(A.device):
        L.check(L.lib().bem_cmatmul(_vp(A), n, _vp(Xc), m, _vp(Y), _stream(A.device)), "bem_cmatmul")
    return Y


class SolveInfo(dict):
    pass


def gmres(A: torch.Tensor, b: torch.Tensor, x=None, *, rtol=1e-5, atol=0.0, max_iters=1000, restart=200,
          precision="fp32", max_refine=None, inner_rtol=None, info: dict | None = None, raise_on_failure=False):
    """Device GMRES (+ FP64 refinement) for complex64 A and b of shape (n,) or (n, m)."""
    check_tensor(A, torch.complex64)
    n = int(A.shape[0])
    vec = b.dim() == 1
    B = b.reshape(n, -1).to(torch.complex64).contiguous()
    m = int(B.shape[1])
    X = torch.zeros_like(B) if x is None else x.reshape(n, m).to(torch.complex64).contiguous().clone()
    prec = _PRECISIONS[precision]
    p = L.SolverParams()
    p.precision = prec
    p.restart = int(min(restart, 255, max(1, max_iters)))  # Krylov dimension per cycle
    p.max_iters = int(max_iters)
    p.max_refine = int(max_refine if max_refine is not None else (2 if prec in (L.PREC_FP32, L.PREC_FP16X3) else 6))
    p.rtol = float(rtol)
    p.atol = float(atol)
    p.inner_rtol = float(inner_rtol if inner_rtol is not None else (3e-2 if prec == L.PREC_BF16 else 1e-3))
    lib = L.lib()
    ws_bytes = int(lib.bem_gmres_workspace_bytes(n, m, ctypes.byref(p)))
    if ws_bytes == 0:
        raise L.BEMError(L.BEM_ERR_INVALID_ARGUMENT, "bem_gmres_workspace_bytes")
    ws = torch.empty(ws_bytes, dtype=torch.uint8, device=A.device)
    out = L.SolverInfo()
    with _on(A.device):
        st = lib.bem_gmres_solve(_vp(A), n, _vp(B), m, _vp(X), 0 if x is None else 1, ctypes.byref(p), _vp(ws),
                                 ws_bytes, ctypes.byref(out), _stream(A.device))
    if info is not None:
        info.update(status=out.status, iterations=out.iterations, refinements=out.refinements, matvecs=out.matvecs,
                    rel_residual=out.rel_residual)
    if st not in (L.BEM_OK, L.BEM_ERR_NOT_CONVERGED) or (raise_on_failure and st != L.BEM_OK):
        raise L.BEMError(st, "bem_gmres_solve")
    return X[:, 0] if vec else X


def solve_linear_equation(A_func, b, x=None, nsteps=500, tol=1e-10, atol=1e-16, *, solver="gmres",
                          precision="fp32", restart=200, info: dict | None = None):
    """Solve A x = b (solver.py:61-66).

    ``A_func`` is a complex64 (n, n) tensor or a callable x -> A x.  Stops when
    ||b - A x||^2 < tol ||b||^2 or ||b - A x||^2 < atol, as the reference.
    Matrices go to the device GMRES (``solver="gmres"``, default) or to the
    reference's BiCGSTAB iteration (``solver="bicgstab"``); callables always
    use BiCGSTAB.
    """
    if callable(A_func) and not isinstance(A_func, torch.Tensor):
        return BiCGSTAB(A_func).solve(b, x=x, nsteps=nsteps, tol=tol, atol=atol)
    if solver == "bicgstab":
        return BiCGSTAB(lambda v: cmatmul(A_func, v)).solve(b, x=x, nsteps=nsteps, tol=tol, atol=atol)
    if solver != "gmres":
        raise ValueError(f"unknown solver {solver!r}")
    return gmres(A_func, b, x, rtol=math.sqrt(max(tol, 0.0)), atol=math.sqrt(max(atol, 0.0)), max_iters=nsteps,
                 restart=restart, precision=precision, info=info)


def _order(approx):
    """Quadrature order of the reference's ``approx`` argument."""
    if not approx:
        return L.ORDER_EXACT
    return L.ORDER_APPROX_1 if approx in ("1", 1) and approx is not True else L.ORDER_APPROX


class BEM_Solver:
    """Mesh holder and operator facade (solver.py:69-147)."""

    def __init__(self, vertices, triangles):
        if isinstance(vertices, np.ndarray):
            vertices = torch.from_numpy(vertices).cuda().float()
        if isinstance(triangles, np.ndarray):
            triangles = torch.from_numpy(triangles).cuda().int()
        check_tensor(vertices, torch.float32)
        check_tensor(triangles, torch.int32)
        self.vertices = vertices
        self.triangles = triangles
        self.device = vertices.device
        self.geometry = Geometry(vertices, triangles)
        self.normals, self.surface_curls_trans = self.geometry.normals_and_curls()

    # ---- assembly ---------------------------------------------------------
    def _new_matrix(self, rows=None):
        n = self.geometry.nv
        return torch.empty((n if rows is None else rows, n), dtype=torch.complex64, device=self.device)

    def assemble_boundary_matrix(self, wavenumber, layer_type, approx=False):
        """Dense (N, N) complex64 matrix; ``approx`` as in the reference
        (False: <4,6>, True: <2,3>, "1" or 1 (beyond the reference's bool): <2,1>)."""
        order = _order(approx)
        out = self._new_matrix()
        with _on(self.device):
            L.check(L.lib().bem_boundary_matrix(_vp(self.geometry.buffer), _LAYERS[layer_type], order,
                                                float(wavenumber), _vp(self.normals), _vp(self.surface_curls_trans),
                                                _vp(out), _stream(self.device)), f"assemble {layer_type}")
        return out

    def assemble_vk(self, wavenumber, single=True, lhs=True, *, check=True):
        """Fused assembly: (V, 0.5 I - K); either may be skipped (None).

        With ``check`` (default) the call synchronises and raises
        ``BEMError`` if a bounded wait of the assembly kernel expired;
        ``check=False`` leaves that to a later ``self.geometry.check_status()``
        (the solve paths check once after their solver has synchronised)."""
        V = self._new_matrix() if single else None
        A = self._new_matrix() if lhs else None
        with _on(self.device):
            L.check(L.lib().bem_boundary_matrices_vk(_vp(self.geometry.buffer), float(wavenumber), _vp(V), _vp(A),
                                                     0.5, -1.0, _stream(self.device)), "bem_boundary_matrices_vk")
        if check:
            self.geometry.check_status()
        return V, A

    def assemble_bm(self, wavenumber, approx=True, *, check=True):
        """Fused Burton-Miller matrices (bm_lhs + 1/2 I, bm_rhs - (i/(2k)) I),
        one pass; ``approx`` as in ``assemble_boundary_matrix`` (True: the
        <2,3> rules of ``neumann2dirichlet``; False: <4,6>, which is the
        ``HBIE`` system).  ``check`` as in ``assemble_vk``."""
        lhs, rhs = self._new_matrix(), self._new_matrix()
        with _on(self.device):
            L.check(L.lib().bem_boundary_matrices_bm(_vp(self.geometry.buffer), _order(approx), float(wavenumber),
                                                     _vp(lhs), _vp(rhs), _stream(self.device)),
                    "bem_boundary_matrices_bm")
        if check:
            self.geometry.check_status()
        return lhs, rhs

    def identity_matrix(self):
        out = self._new_matrix()
        with _on(self.device):
            L.check(L.lib().bem_identity_matrix(_vp(self.geometry.buffer), _vp(out), _stream(self.device)),
                    "bem_identity_matrix")
        return out

    # ---- boundary integral equations -------------------------------------
    def CBIE(self, k, neumann, *, precision="fp32", solver="gmres", rtol=1e-5, restart=200, max_iters=1000,
             info: dict | None = None):
        """Exterior Neumann CBIE (solver.py:97-104): (0.5 I - K) u = -V g."""
        V, lhs = self.assemble_vk(k, check=False)
        rhs = -cmatmul(V, neumann.to(torch.complex64))
        del V
        if solver == "bicgstab":
            u = solve_linear_equation(lhs, rhs, solver="bicgstab", tol=rtol * rtol)
        else:
            u = gmres(lhs, rhs, rtol=rtol, max_iters=max_iters, restart=restart, precision=precision, info=info)
        self.geometry.check_status()  # the solver has synchronised: a cheap read
        return u

    def HBIE(self, k, neumann, **kw):
        """Hypersingular BIE (solver.py:106-116): 1/2 I - K + (i/k) W and
        -V - (i/k)(K' + 1/2 I) are the Burton-Miller pair at the <4,6>
        rules, assembled in one fused pass."""
        lhs, rhs_m = self.assemble_bm(k, approx=False, check=False)
        rhs = cmatmul(rhs_m, neumann.to(torch.complex64))
        del rhs_m
        u = solve_linear_equation(lhs, rhs, **kw)
        self.geometry.check_status()
        return u

    def neumann2dirichlet(self, k, neumann, **kw):
        """Burton-Miller with the <2,3> rules (solver.py:118-126): the fused
        assembly of (bm_lhs + 1/2 I, bm_rhs - (i/(2k)) I), then
        ``solve_linear_equation`` (same options)."""
        lhs, rhs_m = self.assemble_bm(k, check=False)
        rhs = cmatmul(rhs_m, neumann.to(torch.complex64))
        del rhs_m
        u = solve_linear_equation(lhs, rhs, **kw)
        self.geometry.check_status()
        return u

    # ---- listeners ----------------------------------------------------------
    def potential_matrix(self, k, points, layer_type="single"):
        """Explicit (P, N) potential matrix (bind.cu:156-176)."""
        check_tensor(points, torch.float32)
        out = self._new_matrix(rows=points.shape[0])
        with _on(self.device):
            L.check(L.lib().bem_potential_matrix(_vp(self.geometry.buffer), _LAYERS[layer_type], _vp(points),
                                                 int(points.shape[0]), float(k), _vp(out), _stream(self.device)),
                    "bem_potential_matrix")
        return out

    def _b2p(self, k, neumann, dirichlet, points):
        if points.dtype is not torch.float32 or not points.is_contiguous():
            points = points.to(torch.float32).contiguous()
        ref = neumann if neumann is not None else dirichlet
        vec = ref.dim() == 1
        n, nt = self.geometry.nv, self.geometry.nt

        def prep(u):
            if u is None or (u.dtype is torch.complex64 and u.dim() == 2 and u.shape[0] == n and u.is_contiguous()):
                return u
            return u.reshape(n, -1).to(torch.complex64).contiguous()

        nu, du = prep(neumann), prep(dirichlet)
        m = (nu if nu is not None else du).shape[1]
        P = int(points.shape[0])
        out = torch.empty((P, m), dtype=torch.complex64, device=self.device)
        lib = L.lib()
        with _on(self.device):
            # without the scratch tensor where the library takes it so (same kernels; 2 us of a 25 us call)
            if 6 * nt * m <= lib.bem_boundary2potential_noalloc_max():
                L.check(lib.bem_boundary2potential_noalloc(_vp(self.geometry.buffer), _vp(points), P, float(k), _vp(nu),
                                                           _vp(du), m, _vp(out), _stream(self.device)),
                        "bem_boundary2potential")
            else:
                sb = int(lib.bem_boundary2potential_scratch_bytes(nt, m))
                scratch = torch.empty(sb, dtype=torch.uint8, device=self.device)
                L.check(lib.bem_boundary2potential(_vp(self.geometry.buffer), _vp(points), P, float(k), _vp(nu),
                                                   _vp(du), m, _vp(out), _vp(scratch), sb, _stream(self.device)),
                        "bem_boundary2potential")
        return out[:, 0] if vec else out

    def single_potential(self, k, neumann, points):
        """S neumann at the listeners (solver.py:128-132)."""
        return -self._b2p(k, neumann, None, points)

    def double_potential(self, k, dirichlet, points):
        """D dirichlet at the listeners (solver.py:134-138)."""
        return self._b2p(k, None, dirichlet, points)

    def boundary2potential(self, k, neumann, dirichlet, points):
        """-S neumann + D dirichlet at the listeners (solver.py:140-147)."""
        return self._b2p(k, neumann, dirichlet, points)

    # ---- the whole path ------------------------------------------------------
    def solve_and_evaluate(self, k, neumann, points, *, precision="fp16x3", rtol=1e-6, restart=200, max_iters=1000,
                           info: dict | None = None):
        """Assemble (fused V, 0.5 I - K), solve the CBIE for every column of
        ``neumann`` and evaluate the listener pressures.  Returns (u, p)."""
        u = self.CBIE(k, neumann, precision=precision, rtol=rtol, restart=restart, max_iters=max_iters, info=info)
        return u, self.boundary2potential(k, neumann, u, points)


def map_triangle2vertex(vertices, triangles, features):
    """Average per-triangle complex values onto vertices (solver.py:150-154)."""
    check_tensor(vertices, torch.float32)
    check_tensor(triangles, torch.int32)
    check_tensor(features, torch.complex64)
    g = Geometry(vertices, triangles)
    out = torch.empty(g.nv, dtype=torch.complex64, device=vertices.device)
    counts = torch.empty(g.nv, dtype=torch.int32, device=vertices.device)
    with _on(vertices.device):
        L.check(L.lib().bem_triangle2vertex(g.ptr, _vp(features), _vp(out), _vp(counts), _stream(vertices.device)),
                "bem_triangle2vertex")
    return out
